"""Buffers made on a handle's first use, when one of their allocations fails:
the call reports it, nothing half made stays behind, and the next call starts
afresh (on the host, over a stand-in for the CUDA runtime: no GPU)."""

from __future__ import annotations

import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
CSRC = ROOT / "apple_gb300" / "csrc"

ADJOINT = r"""
#include "host_fakes.h"
using namespace agb;
static int launches = 0, bad = 0;
static bool has(const void* p) { return p && fake::live.count((void*)p); }
static agb::CgState* g_state = nullptr;
namespace agb {
cudaError_t resident_prepare(const SolveArgs&, ResidentPlan* p) { p->shape = 0; return cudaSuccess; }
cudaError_t cg_resident_prepare(const SolveArgs&, ResidentPlan* p) { p->shape = 1; return cudaSuccess; }
cudaError_t launch_cg_init(const CgArgs& c, const void*, const int32_t*, cudaStream_t) {
  ++launches;
  if (!has(c.lam) || !c.res || !c.q || !c.minv || !c.p0 || !c.p1 || !has(c.part) || !has(c.cnt) || !has(c.cs) ||
      c.a.n_points == 0)
    ++bad;
  g_state = c.cs;
  return cudaSuccess;
}
cudaError_t launch_cg_set_limit(const CgArgs&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_cg_resident(const CgArgs&, const ResidentPlan& p, void* part_p, void* part_v, unsigned* counters,
                               cudaStream_t) {
  if (p.shape != 1 || !has(part_p) || part_v <= part_p || !has(counters) || counters[0] != 0) ++bad;
  return cudaSuccess;
}
cudaError_t launch_cg_unpack(const CgArgs&, const int32_t*, void*, cudaStream_t) { return cudaSuccess; }
}

int main() {
  FakeMesh m(2);
  agb_space* s = nullptr; agb_fem* f = nullptr; agb_model* md = nullptr;
  if (agb_space_create(m.n_points(), m.points.data(), &s)) return 1;
  if (agb_fem_create(s, AGB_STABLE_NEO_HOOKEAN, AGB_F32, m.n_cells(), m.cells.data(), m.points.data(), nullptr, nullptr,
                     nullptr, m.mu.data(), m.lam.data(), 0, &f)) return 2;
  if (agb_model_create(s, AGB_F32, 1, &f, nullptr, nullptr, 0, nullptr, nullptr, &md)) return 3;
  std::vector<float> rhs(3 * m.n_points()), lam(3 * m.n_points());
  for (int k = 1;; ++k) {
    agb_solver* sv = nullptr;
    if (agb_solver_create(md, nullptr, &sv)) return 4;
    const size_t before = fake::live.size();
    fake::fail_at = k;
    const int rc = agb_solver_adjoint(sv, rhs.data(), lam.data(), nullptr, nullptr, nullptr);
    const bool failed = fake::fail_at == 0;
    fake::fail_at = 0;
    if (failed && (rc == AGB_OK || launches)) { printf("allocation %d: rc %d\n", k, rc); return 5; }
    if (failed && fake::live.size() != before) { printf("allocation %d: buffers left\n", k); return 6; }
    if (agb_solver_adjoint(sv, rhs.data(), lam.data(), nullptr, nullptr, nullptr) || bad || !launches) {
      printf("allocation %d: the next call ran on half-made buffers (%d launches, %d bad)\n", k, launches, bad);
      return 7;
    }
    launches = 0;
    agb_solver_destroy(sv);
    if (!failed) return k > 6 ? 0 : 8;  // every allocation of the set-up has failed once
  }
}
"""

MATERIAL_GRADIENT = r"""
#include "host_fakes.h"
using namespace agb;
static int launches = 0, bad = 0;
static bool has(const void* p) { return p && fake::live.count((void*)p); }
namespace agb {
cudaError_t launch_param_vjp(const FemView& fv, int precision, const void*, const void*, const void* vol,
                             const int32_t* elem_user, void*, void*, cudaStream_t) {
  ++launches;
  if (!has(vol) || !has(elem_user)) ++bad;
  else if (elem_user[0] < 0 || elem_user[0] >= fv.n_cells) ++bad;
  else if ((precision == AGB_F64 ? *(const double*)vol : *(const float*)vol) <= 0) ++bad;
  return cudaSuccess;
}
}

int main() {
  FakeMesh m(2);
  for (int precision : {AGB_F32, AGB_F64})
    for (int k = 1;; ++k) {
      agb_space* s = nullptr; agb_fem* f = nullptr;
      if (agb_space_create(m.n_points(), m.points.data(), &s)) return 1;
      if (agb_fem_create(s, AGB_STABLE_NEO_HOOKEAN, precision, m.n_cells(), m.cells.data(), m.points.data(), nullptr,
                         nullptr, nullptr, m.mu.data(), m.lam.data(), 0, &f)) return 2;
      double x[1] = {0};
      launches = 0;
      fake::fail_at = k;
      const int rc = agb_fem_grad_param_vjp(f, x, x, x, x, nullptr);
      const bool failed = fake::fail_at == 0;
      fake::fail_at = 0;
      if (failed && (rc == AGB_OK || launches)) { printf("allocation %d: rc %d\n", k, rc); return 5; }
      if (agb_fem_grad_param_vjp(f, x, x, x, x, nullptr) || bad || !launches) {
        printf("allocation %d: the next call ran on half-made tables\n", k);
        return 7;
      }
      agb_fem_destroy(f);
      agb_space_destroy(s);
      if (!fake::live.empty()) return 6;
      if (!failed) {
        if (k < 3) return 8;
        break;
      }
    }
  return 0;
}
"""


def _run(tmp_path, program):
    cpp = tmp_path / "check.cpp"
    cpp.write_text(program)
    exe = tmp_path / "check"
    cmd = ["g++", "-O1", "-std=c++17", "-no-pie", "-Wl,-z,lazy", "-Wl,--unresolved-symbols=ignore-all",
           f"-I{ROOT / 'tests'}", f"-I{CSRC}", f"-I{ROOT / 'include'}", "-I/usr/local/cuda/include", str(cpp),
           str(CSRC / "capi.cpp"), str(CSRC / "prep.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)


@pytest.mark.parametrize("program", [ADJOINT, MATERIAL_GRADIENT], ids=["adjoint", "material_gradient"])
def test_a_failed_allocation_leaves_nothing_half_made(tmp_path, program):
    _run(tmp_path, program)
