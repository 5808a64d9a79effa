"""Tiles are cut and paired for the SMs that the device has, and where no
resident form fits, the iterations run over the whole tiles (on the host, over
a stand-in for the CUDA runtime: no GPU)."""

from __future__ import annotations

import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parent.parent
CSRC = ROOT / "apple_gb300" / "csrc"

PROGRAM = r"""
#include "host_fakes.h"
using namespace agb;
static int shape = 0, prepared = 0, wrong = 0;
static SolveArgs iter_args, whole_args;
namespace agb {
cudaError_t resident_prepare(const SolveArgs& a, ResidentPlan* p) {
  ++prepared;
  iter_args = a;
  p->shape = shape;
  if (p->sms != fake::sms || a.fv.n_tiles > 2 * fake::sms) wrong |= 1;
  if (p->whole != 0 && p->whole != fake::sms) wrong |= 2;
  if (p->order) {  // every tile once, at most two a CTA, over as many CTAs as SMs
    std::vector<int> seen(a.fv.n_tiles, 0);
    for (int k = 0; k < 2 * fake::sms; ++k)
      if (p->order[k] >= 0) ++seen[p->order[k]];
    for (int s : seen)
      if (s != 1) wrong |= 4;
  } else if (a.precision == AGB_F64 && a.fv.n_tiles > fake::sms) {
    wrong |= 8;
  }
  return cudaSuccess;
}
cudaError_t launch_solver_init(const SolveArgs& a, const void*, const void*, const int32_t*, cudaStream_t) {
  whole_args = a;
  return cudaSuccess;
}
cudaError_t launch_solver_force_refresh(const SolveArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_solver_first(const SolveArgs&, cudaStream_t) { return cudaSuccess; }
// the reset's refresh runs on the iterations' tiles
cudaError_t launch_solver_refresh(const SolveArgs& a, cudaStream_t, bool) {
  iter_args = a;
  return cudaSuccess;
}
}

int main() {
  for (int n : {16, 30}) {
    FakeMesh m(n);
    for (int sms : {152, 132, 40})
      for (int precision : {AGB_F32, AGB_F64})
        for (int s : {1, 0}) {
          fake::sms = sms;
          shape = s;
          prepared = wrong = 0;
          agb_space* sp = nullptr; agb_fem* f = nullptr; agb_model* md = nullptr; agb_solver* sv = nullptr;
          if (agb_space_create(m.n_points(), m.points.data(), &sp)) return 1;
          if (agb_fem_create(sp, AGB_STABLE_NEO_HOOKEAN, precision, m.n_cells(), m.cells.data(), m.points.data(),
                             nullptr, nullptr, nullptr, m.mu.data(), m.lam.data(), 0, &f)) return 2;
          if (f->pieces.n_tiles > 2 * sms) return 3;
          if (agb_model_create(sp, precision, 1, &f, nullptr, nullptr, 0, nullptr, nullptr, &md)) return 4;
          if (agb_solver_create(md, nullptr, &sv)) return 5;
          const int tiles = f->plan.n_tiles;
          if (prepared != (tiles <= 2 * sms) || wrong) {
            printf("n %d sms %d precision %d: %d tiles, wrong %d\n", n, sms, precision, tiles, wrong);
            return 6;
          }
          std::vector<double> u(3 * m.n_points(), 0.0);
          if (agb_solver_reset(sv, u.data(), nullptr)) return 7;
          if (whole_args.fv.n_tiles != tiles) return 8;
          if (precision == AGB_F32 && (s == 0 || !prepared)) {
            if (iter_args.fv.n_tiles != tiles || iter_args.fv.tv_vid != whole_args.fv.tv_vid ||
                iter_args.slot_of_tv != whole_args.slot_of_tv || iter_args.off != whole_args.off ||
                iter_args.n_slots != whole_args.n_slots) {
              printf("n %d sms %d: no resident form, but %d tiles in place of %d\n", n, sms, iter_args.fv.n_tiles,
                     tiles);
              return 9;
            }
          } else if (precision == AGB_F32 && n == 16 && iter_args.fv.n_tiles <= tiles) {
            return 10;  // this mesh's tiles are cut
          }
          agb_solver_destroy(sv);
          agb_model_destroy(md);
          agb_fem_destroy(f);
          agb_space_destroy(sp);
          if (!fake::live.empty()) return 11;
        }
  }
  return 0;
}
"""


def test_tiles_follow_the_device(tmp_path):
    cpp = tmp_path / "check.cpp"
    cpp.write_text(PROGRAM)
    exe = tmp_path / "check"
    cmd = ["g++", "-O1", "-std=c++17", "-no-pie", "-Wl,-z,lazy", "-Wl,--unresolved-symbols=ignore-all",
           f"-I{ROOT / 'tests'}", f"-I{CSRC}", f"-I{ROOT / 'include'}", "-I/usr/local/cuda/include", str(cpp),
           str(CSRC / "capi.cpp"), str(CSRC / "prep.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
