// elastic3d.cu -- 3-D isotropic elastic (velocity-stress, staggered grid)
// forward and boundary-saving adjoint for sm_100a, at spatial orders 2, 4, 6
// and 8 (this file: order 8 and the dispatch by order; elastic3d_orders.cu:
// orders 2, 4, 6; the body of every order is elastic3d_impl.cuh).
//
// Restates the reference's elastic3d path (src/sweep/csrc/cuda/equations/
// elastic3d/kernels.cuh, driver_traits.cuh; common/sg_driver.cuh):
//
//   forward, per step:
//     vel3      velocity update; the nine stress-derivative CPML memories
//               outside the physical box shrunk by one cell  kernels.cuh:104-248
//     str3      stress update with the nine velocity-derivative memories
//                                                             kernels.cuh:290-483
//     src3 / strips3 / rec3   source injection per source field, the nine
//               fields' boundary strips, the receiver gather  driver_traits.cuh:265-300
//   reverse, per step (driver_traits.cuh:680-905):
//     res3      signed residual injection (stress -1, velocity +1); src3 with
//               -w takes the forward source back out
//     stress_rev   stress reconstruction on the box minus one cell
//               (kernels.cuh:653-768) and the vp / vs imaging of the
//               stress-adjoint prepare                        kernels.cuh:1367-1615
//     strips3   stress strips of step it - 1 restored
//     adj_vel   the stress step's transpose (adjoint velocities)
//                                                             kernels.cuh:1367-1780
//     adj_str   the velocity step's transpose (adjoint stresses)
//                                                             kernels.cuh:959-1236
//     vel_rev   velocity reconstruction (kernels.cuh:536-652) with the rho
//               image of the step it takes back; the reference images v(it) -
//               v(it + 1) and corrects it at the receivers and body-force
//               sources (common/common.cu:40-116)
//     restore_velocity   velocity strips of step it - 1
//
// Four x cells per thread on pitched rows (vec4.cuh).  Layout: fields
// (B, nz, ny, P), x fastest, P = nx rounded up to 8; CPML memories in per-axis
// slabs covering the cells outside the box shrunk by one cell along their
// axis.  Cells in the CPML branch because of another axis have zero
// coefficients on this one and keep no memory (as the reference's stored()
// gating).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <vector>

#include "common.cuh"
#include "elastic3d.cuh"

#define EL3D_M 4
#define EL3D_NS el3d_m4
#include "elastic3d_impl.cuh"
#undef EL3D_NS
#undef EL3D_M

namespace sweep {
namespace el3d {

// the entry points of the order the descriptor asks for
#define SWEEP_EL3D_BY_ORDER(CALL)                                                                          \
    switch (d->M) {                                                                                          \
    case 1: el3d_m1::CALL; break;                                                                            \
    case 2: el3d_m2::CALL; break;                                                                            \
    case 3: el3d_m3::CALL; break;                                                                            \
    case 4: el3d_m4::CALL; break;                                                                            \
    default: SWEEP_REQUIRE(false, "elastic3d: spatial orders 2, 4, 6 and 8 are built (got order %d)", 2 * d->M); \
    }

void sizes(const sweep_elastic3d_desc* d, int mem_mode, int ckpt_every, int64_t* ws_bytes, int64_t* tape_bytes)
{
    SWEEP_REQUIRE(d != nullptr, "null descriptor");
    SWEEP_EL3D_BY_ORDER(sizes(d, mem_mode, ckpt_every, ws_bytes, tape_bytes))
}

void forward(const sweep_elastic3d_desc* d, int mem_mode, int ckpt_every, float* record, void* tape, void* ws,
             int64_t ws_bytes, cudaStream_t st)
{
    SWEEP_REQUIRE(d != nullptr, "null descriptor");
    SWEEP_EL3D_BY_ORDER(forward(d, mem_mode, ckpt_every, record, tape, ws, ws_bytes, st))
}

void backward(const sweep_elastic3d_desc* d, int mem_mode, int ckpt_every, const float* adj, const void* tape,
              float* grad_vp, float* grad_vs, float* grad_rho, void* ws, int64_t ws_bytes, cudaStream_t st)
{
    SWEEP_REQUIRE(d != nullptr, "null descriptor");
    SWEEP_EL3D_BY_ORDER(backward(d, mem_mode, ckpt_every, adj, tape, grad_vp, grad_vs, grad_rho, ws, ws_bytes, st))
}

#undef SWEEP_EL3D_BY_ORDER

}  // namespace el3d
}  // namespace sweep
