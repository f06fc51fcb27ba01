// vti3d.cu -- 3-D first-order acoustic VTI (Duveneck et al. 2008: vx, vy, vz
// and the horizontal / vertical stresses sH = s11 = s22, sV = s33 on a
// staggered grid) forward and boundary-saving adjoint with vp / epsilon /
// delta / rho gradients, at every even spatial order 2..14, for sm_100a.
//
// The C descriptor's checks and the instances of the path of vti_impl.cuh
// (reference src/sweep/csrc/cuda/equations/acoustic_vti_1st_3d/kernels.cuh,
// forward.cu, backward.cu).  Fields vx, vy, vz, sH, sV.
#include "vti3d.cuh"
#include "vti_impl.cuh"

namespace sweep {
namespace vti3 {

static vtik::Desc unpack(const sweep_vti3d_desc* d)
{
    SWEEP_REQUIRE(d != nullptr, "null descriptor");
    SWEEP_REQUIRE(d->B >= 1 && d->nt >= 1 && d->nz >= 1 && (long long)d->B * d->nz <= 65535,
                  "vti3d: B * nz must be 1 to 65535 and nt >= 1");
    vtik::Desc e{};
    e.B = d->B; e.nz = d->nz; e.ny = d->ny; e.nx = d->nx; e.nt = d->nt; e.M = d->M;
    for (int f = 0; f < 6; ++f) e.pad[f] = d->pad[f];
    e.dt = d->dt; e.dz = d->dz; e.dy = d->dy; e.dx = d->dx;
    const float* prof[3][4] = {{d->ax, d->bx, d->axh, d->bxh}, {d->ay, d->by, d->ayh, d->byh},
                               {d->az, d->bz, d->azh, d->bzh}};
    for (int a = 0; a < 3; ++a)
        for (int k = 0; k < 4; ++k) e.prof[a][k] = prof[a][k];
    e.m = vtik::Models{d->vp, d->epsilon, d->delta, d->rho};
    e.model_stride = d->model_stride;
    e.nsrc = d->nsrc; e.nrec = d->nrec; e.nsf = d->nsrc_fields; e.nrf = d->nrec_fields;
    e.sf = d->src_fields; e.rf = d->rec_fields;
    e.src = d->src_loc; e.rec = d->rec_loc; e.wavelet = d->wavelet;
    return e;
}

void sizes(const sweep_vti3d_desc* d, int mem_mode, int, int64_t* ws_bytes, int64_t* tape_bytes)
{
    const vtik::Desc e = unpack(d);
    vtik::sizes<3>(vtik::make_plan<3>(e, mem_mode, "vti3d"), ws_bytes, tape_bytes);
}

void forward(const sweep_vti3d_desc* d, int mem_mode, int, float* record, void* tape, void* ws, int64_t ws_bytes,
             cudaStream_t st)
{
    const vtik::Desc e = unpack(d);
    vtik::Plan pl = vtik::make_plan<3>(e, mem_mode, "vti3d");
#define SWEEP_VTI_FWD(m) vtik::forward<m, 3>(e, pl, record, tape, ws, ws_bytes, st)
    SWEEP_VTI_DISPATCH(e.M, SWEEP_VTI_FWD)
#undef SWEEP_VTI_FWD
}

void backward(const sweep_vti3d_desc* d, int mem_mode, int, const float* adj, const void* tape, float* grad_vp,
              float* grad_eps, float* grad_dlt, float* grad_rho, void* ws, int64_t ws_bytes, cudaStream_t st)
{
    const vtik::Desc e = unpack(d);
    vtik::Plan pl = vtik::make_plan<3>(e, mem_mode, "vti3d");
    const vtik::Grads out{{grad_vp, grad_eps, grad_dlt, grad_rho}};
#define SWEEP_VTI_BWD(m) vtik::backward<m, 3>(e, pl, adj, tape, out, ws, ws_bytes, st)
    SWEEP_VTI_DISPATCH(e.M, SWEEP_VTI_BWD)
#undef SWEEP_VTI_BWD
}

}  // namespace vti3
}  // namespace sweep
