// Host-callable kernel launchers (fem_eval.cu, solver.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "agb_internal.h"

namespace agb {

// bytes of one reduction partial for a precision
inline size_t partial_bytes(int precision) { return precision == AGB_F64 ? 8 : 8; }
inline size_t real_bytes(int precision) { return precision == AGB_F64 ? 8 : 4; }
inline size_t v4_bytes(int precision) { return 4 * real_bytes(precision); }

// Fused element pass over all tiles of `fv` (AGB_* flags); u and p in the
// caller's order; with p_slot (one entry per component: its index among the
// free ones, or -1) p holds the free components.  Vector results go to the slots of slot_of_tv[tv], packed
// as the requested vectors' 3 reals each in the order gradient, diagonal,
// product (at most 9 reals of each of n_slots); scalar results are added to
// *energy / *quad by the last block, or with `assign` stored there.
cudaError_t launch_fem_eval(int precision, const FemView& fv, unsigned flags, const void* u, const void* p,
                            const int32_t* p_slot, const int32_t* slot_of_tv, void* slots, int32_t n_slots,
                            void* partials, unsigned* counter, double* energy, double* quad, int assign,
                            cudaStream_t stream);

// After launch_fem_eval with the same vector flags, in the same stream: sum
// slots per vertex (CSR `off`) and add them to the caller's (n_points, 3)
// arrays, or with `assign` store them (with out_slot, only the free
// components, at their index among them); with `force` (V4, device order) add -f
// to grad and, with AGB_FUN, -f.u to *energy.
cudaError_t launch_unpack(int precision, int n_points, const int32_t* user_of_internal, const int32_t* off,
                          const void* slots, int32_t n_slots, unsigned flags, void* grad, void* diag, void* prod,
                          const int32_t* out_slot, int assign, const void* force, const void* u, void* partials,
                          unsigned* counter, double* energy, cudaStream_t stream);

int unpack_blocks(int n_points);

// muscle: rewrite the element records (D A in place of D) and the S stream
// `act` (FemView layouts) for the activation act_user (n_cells x 6 doubles,
// the caller's cell order); D is TilePlan::D, elem_user the cell of each element
cudaError_t launch_muscle_records(int precision, int n_cells, const int32_t* elem_user, const double* D,
                                  const double* act_user, void* rec, void* act, cudaStream_t stream);

// free/fixed DOF maps: free[i] = full[free_idx[i]];
// full[j] = slot[j] >= 0 ? free[slot[j]] : (fill ? fill[j] : 0)
cudaError_t launch_dof_to_free(int precision, int64_t n_free, const int64_t* free_idx, const void* full,
                               void* free_out, cudaStream_t stream);
cudaError_t launch_dof_to_full(int precision, int64_t n_full, const int32_t* slot, const void* free_in,
                               const void* fill, void* full_out, cudaStream_t stream);

}  // namespace agb
