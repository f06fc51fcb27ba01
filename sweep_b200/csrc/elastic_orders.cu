// elastic_orders.cu -- the 2-D isotropic elastic forward and boundary-saving
// adjoint at every spatial order but 8 (M = 1..7: orders 2, 4, 6, 10, 12,
// 14), for sm_100a.  Order 8 runs through elastic2d.cu: its forward on tiled
// kernels, its reverse on those of elastic_vec.cuh as here.  The reference's
// Elastic defaults to order 4, so a drop-in caller lands here unless it asks
// for order 8.
//
// Restates the reference's templated elastic2d path (src/sweep/csrc/cuda/
// equations/elastic2d/kernels.cuh, common/sg_driver.cuh step order,
// common/elastic_free_surface.cuh for traction-free faces), order by order,
// with the staggered weights of that order (operators/staggered.cuh):
//   forward, per step: velocity step (four stress derivatives, CPML memories
//     outside the physical box), stress step (Robertsson corrections and
//     zeroing on free faces), source injection per source field, the five
//     fields' boundary bands (width M + 1 from M cells outside the box),
//     receivers;
//   reverse, per step it = nt - 1 .. 1: signed residuals (stress -1, velocity
//     +1), source removal, stress reconstruction on the box minus one cell,
//     stress bands restored, the stress step's transpose with the vp / vs /
//     rho imaging, the velocity step's transpose, velocity reconstruction,
//     velocity bands restored.
//
// Four x cells per thread (vec4.cuh) on pitched rows, a warp over 32 x 4 (x, z)
// cells.  A reverse step is five launches: the stress reconstruction with its
// image and the transpose into the adjoint velocities touch different fields
// and share one (`rev_a`, by block), the velocity reconstruction and the
// transpose into the adjoint stresses another (`rev_b`).  The transposes read
// q = dt C lambda_s and p = kv lambda_v as their producers left them, through
// the adjoint CPML memory in the layers only, which is double-buffered.  The
// rho image of step `it` is lambda_v . (v(it - 1) - v(it)): inside, minus kv
// lambda_v . div s (what the reconstruction takes back), on the box's
// outermost layer at an absorbing face the difference the restored bands make
// (the reference carries v(it + 1) along and corrects for the residuals and
// the body forces in it); the image of the update of step 1 is left out, as
// by the reference's staggered reverse.
//
// Measured at order 4: 8 shots of 187 x 331 with a free top face, 300 steps,
// 18.5 ms a gradient (51 ms on fourteen launches of one cell per thread a
// reverse step): 14 + 12 us the two reverse kernels, 7 + 9 us the forward's.
// The small grid is bound by latency and launches.
// Memory: boundary saving with fp32 bands in device memory (SWEEP_MEM_BOUNDARY).
#include <cuda_runtime.h>

#include <algorithm>

#include "bands.cuh"
#include "common.cuh"
#include "elastic_orders.cuh"
#include "elastic_vec.cuh"

namespace sweep {
namespace eord {

using namespace evec;

__global__ void inject(const Geo G, const Fields F, int it)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < G.B * G.nsrc) inject_at(G, F, e, it, 1.f);
}

// record[b, it, r, k] = field rf[k] at receiver r, and the bands of every
// field into one step slot (B, 5, ns); either may be absent
__global__ void save(const Geo G, const Fields F, float* record, float* slot, int it)
{
    long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nr = record ? (long long)G.B * G.nrec : 0;
    if (e < nr) {
        const int b = (int)(e / G.nrec), r = (int)(e - (long long)b * G.nrec);
        const int c = loc(G, G.rec + 2 * e);
        if (c < 0) return;
        float* out = record + (((long long)b * G.nt + it) * G.nrec + r) * G.nrf;
        for (int k = 0; k < G.nrf; ++k) out[k] = F.f[G.rf[k]][b * G.S + c];
        return;
    }
    e -= nr;
    if (!slot || e >= (long long)G.B * G.ns) return;
    const int b = (int)(e / G.ns), n = (int)(e - (long long)b * G.ns);
    const long long i = b * G.S + __ldg(G.cells + n);
#pragma unroll
    for (int f = 0; f < 5; ++f) slot[(b * 5LL + f) * G.ns + n] = F.f[f][i];
}

// Field f0 + blockIdx.y of the bands from a step slot.  Velocities add the rho
// image of the box cells outside the reverse box: the difference this makes in
// the two of them.
__global__ void restore(const Geo G, const Rev R, const float* __restrict__ slot, int f0)
{
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)G.B * G.ns) return;
    const int b0 = (int)(e / G.ns), n = (int)(e - (long long)b0 * G.ns);
    const int c = __ldg(G.cells + n), z = c / G.P, x = c - z * G.P;
    const bool img = f0 == VX && R.it > 1 && zbox(G, z) && xbox(G, x) &&
                     !(z >= G.rz0 && z < G.rz1 && x >= G.rx0 && x < G.rx1);
    if (!img) {
        const int f = f0 + blockIdx.y;
        R.f.f[f][b0 * G.S + c] = __ldg(slot + (b0 * 5LL + f) * G.ns + n);
        return;
    }
    const int nb = image_shots(G, b0, blockIdx.y);
    float s = 0.f;
    for (int b = b0; b < b0 + nb; ++b) {
        const long long i = b * G.S + c;
        for (int f = VX; f <= VZ; ++f) {
            const float v = __ldg(slot + (b * 5LL + f) * G.ns + n);
            s += R.p[f][i] / G.kv[b * G.ms + c] * (v - R.f.f[f][i]);
            R.f.f[f][i] = v;
        }
    }
    if (nb) R.g[2][b0 / G.group * G.S + c] += s;
}

// ------------------------------------------------------------- per call
// Lame parameters and dt / rho per model copy, pitched (reference
// derived_models.cu:27-37 rounding)
__global__ void prep(const float* __restrict__ vp, const float* __restrict__ vs, const float* __restrict__ rho,
                     long long rows, int nx, int P, float dt, float* lam, float* mu, float* kv)
{
    const long long n = rows * P;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long row = k / P;
        const int x = (int)(k - row * P);
        if (x >= nx) { lam[k] = mu[k] = kv[k] = 0.f; continue; }
        const long long i = row * nx + x;
        const float v = vp[i], s = vs[i], r = rho[i];
        mu[k] = (r * s) * s;
        lam[k] = r * ((v * v) - ((2.f * s) * s));
        kv[k] = dt * (1.f / r);
    }
}

// ------------------------------------------------------------------- host
struct Plan {
    Geo G;
    int nm;                         // model copies
    bands::Bands bands;
};

static Plan make_plan(const sweep_elastic_desc* d, int mem_mode)
{
    SWEEP_REQUIRE(d != nullptr, "null descriptor");
    SWEEP_REQUIRE(d->M >= 1 && d->M <= MAXM, "elastic: spatial orders 2 to %d are built (got order %d)", 2 * MAXM,
                  2 * d->M);
    SWEEP_REQUIRE(d->M != 4, "elastic: order 8 runs on kernels of its own");
    SWEEP_REQUIRE(mem_mode == SWEEP_MEM_BOUNDARY,
                  "elastic order %d: boundary saving with fp32 strips in device memory is built for orders other "
                  "than 8 (mem_mode %d; checkpoints, reduced strip formats and the host tape run at order 8)",
                  2 * d->M, mem_mode);
    SWEEP_REQUIRE(d->B >= 1 && d->B <= 65535 && d->nt >= 1, "elastic: 1 to 65535 shots and nt >= 1");
    SWEEP_REQUIRE(d->nsrc >= 0 && d->nrec >= 0, "elastic: negative source/receiver count");
    SWEEP_REQUIRE(d->nsrc_fields >= 1 && d->nsrc_fields <= 5, "elastic: 1 to 5 source fields");
    SWEEP_REQUIRE(d->nrec_fields >= 1 && d->nrec_fields <= 5, "elastic: 1 to 5 receiver fields");
    for (int k = 0; k < d->nsrc_fields; ++k) {
        SWEEP_REQUIRE(d->src_fields[k] >= 0 && d->src_fields[k] < 5, "elastic: bad source field %d", d->src_fields[k]);
        for (int j = 0; j < k; ++j)
            SWEEP_REQUIRE(d->src_fields[j] != d->src_fields[k], "elastic: source field %d repeated", d->src_fields[k]);
    }
    for (int k = 0; k < d->nrec_fields; ++k)
        SWEEP_REQUIRE(d->rec_fields[k] >= 0 && d->rec_fields[k] < 5, "elastic: bad receiver field %d",
                      d->rec_fields[k]);
    Plan pl{};
    Geo& G = pl.G;
    const int M = d->M;
    G.B = d->B; G.nz = d->nz; G.nx = d->nx; G.nt = d->nt; G.M = M;
    const long long cells = (long long)d->nz * d->nx;
    G.P = (d->nx + 7) / 8 * 8;
    G.S = (long long)d->nz * G.P;
    SWEEP_REQUIRE(cells < (1LL << 31) && G.S < (1LL << 31), "elastic: one shot's grid must hold < 2^31 cells");
    G.fs = 0;
    for (int f = 0; f < 4; ++f) {
        if (d->free_surface[f]) {
            SWEEP_REQUIRE(d->pad[f] == 0, "elastic: a free face has no PML pad (face %d has %d)", f, d->pad[f]);
            G.fs |= 1 << f;
        } else {
            SWEEP_REQUIRE(d->pad[f] >= 1, "elastic: every absorbing face needs a PML pad >= 1 (face %d has %d)", f,
                          d->pad[f]);
        }
    }
    G.z0 = d->pad[0] + M; G.z1 = G.nz - d->pad[1] - M;
    G.x0 = d->pad[2] + M; G.x1 = G.nx - d->pad[3] - M;
    SWEEP_REQUIRE(G.z1 - G.z0 >= 2 && G.x1 - G.x0 >= 2, "elastic: the physical box must be at least 2 cells per axis");
    G.dt = d->dt; G.ihz = 1.f / d->dz; G.ihx = 1.f / d->dx;
    for (int k = 0; k <= MAXM; ++k) G.c[k] = 0.f;
    v4::staggered_weights(M, G.c);
    G.az = d->az; G.bz = d->bz; G.azh = d->azh; G.bzh = d->bzh;
    const bool per_shot = d->model_stride != 0;
    SWEEP_REQUIRE(!per_shot || d->model_stride == cells, "elastic: model_stride must be 0 or nz * nx");
    G.ms = per_shot ? G.S : 0;
    pl.nm = per_shot ? G.B : 1;
    G.nsrc = d->nsrc; G.nrec = d->nrec; G.nsf = d->nsrc_fields; G.nrf = d->nrec_fields;
    for (int k = 0; k < 5; ++k) { G.sf[k] = d->src_fields[k]; G.rf[k] = d->rec_fields[k]; }
    G.src = d->src_loc; G.rec = d->rec_loc; G.wavelet = d->wavelet;
    // the boundary bands (boundary/strip.cuh:46-123: width M + 1 from M cells
    // outside the box, each band over the box tangentially)
    pl.bands = bands::make<2>(M, G.z0, G.z1, 0, 1, G.x0, G.x1);
    G.ns = pl.bands.count;
    layout(G, per_shot ? 1 : 4);
    return pl;
}

struct Ws {
    float *lam, *mu, *kv;
    float* xprof;                   // a, b, a_half, b_half along x, padded
    int* cells;
    float* f[5];
    float* m[2][NMEM];              // forward memories ([0]) / adjoint memories, double-buffered
    float* a[2];
    float* q[3];
    float* p[2];
    float* g[3];
    char *zero0, *zero1;
};

static void carve(Carve& c, const Plan& pl, bool rev, Ws& w)
{
    const Geo& G = pl.G;
    const long long n = (long long)G.B * G.S, mc = (long long)pl.nm * G.S;
    w = Ws{};
    w.lam = c.take<float>(mc); w.mu = c.take<float>(mc); w.kv = c.take<float>(mc);
    w.xprof = c.take<float>(4LL * xprof_len(G));
    w.cells = c.take<int>(std::max(G.ns, 1));
    c.take<char>(0);
    w.zero0 = c.base ? c.base + c.off : nullptr;
    for (float*& p : w.f) p = c.take<float>(n);
    for (int s = 0; s < (rev ? 2 : 1); ++s)
        for (int k = 0; k < NMEM; ++k) w.m[s][k] = c.take<float>(mem_floats(G, k));
    if (rev) {
        for (float*& p : w.a) p = c.take<float>(n);
        for (float*& p : w.q) p = c.take<float>(n);
        for (float*& p : w.p) p = c.take<float>(n);
        for (float*& p : w.g) p = c.take<float>(G.nslot * G.S);
    }
    c.take<char>(0);
    w.zero1 = c.base ? c.base + c.off : nullptr;
}

static long long slot_floats(const Plan& pl) { return (long long)pl.G.B * 5 * pl.G.ns; }

void sizes(const sweep_elastic_desc* d, int mem_mode, int, int64_t* ws_bytes, int64_t* tape_bytes)
{
    const Plan pl = make_plan(d, mem_mode);
    Carve f(nullptr), r(nullptr);
    Ws w;
    carve(f, pl, false, w);
    carve(r, pl, true, w);
    *ws_bytes = std::max(f.off, r.off);
    *tape_bytes = ((long long)pl.G.nt * slot_floats(pl) + 5LL * pl.G.B * pl.G.nz * pl.G.nx) * 4;
}

static unsigned blocks(long long n) { return (unsigned)std::max<long long>((n + 255) / 256, 1); }

static void setup(const sweep_elastic_desc* d, Plan& pl, const Ws& w, cudaStream_t st)
{
    Geo& G = pl.G;
    G.lam = w.lam; G.mu = w.mu; G.kv = w.kv; G.cells = w.cells;
    const long long rows = (long long)pl.nm * G.nz;
    prep<<<std::min(blocks(rows * G.P), 4096u), 256, 0, st>>>(d->vp, d->vs, d->rho, rows, G.nx, G.P, d->dt, w.lam, w.mu,
                                                              w.kv);
    const int len = xprof_len(G);
    prep_profiles<<<8, 256, 0, st>>>(d->ax, d->bx, d->axh, d->bxh, G.nx, len, w.xprof);
    G.ax = w.xprof + kGuard; G.bx = G.ax + len; G.axh = G.bx + len; G.bxh = G.axh + len;
    // on the device: a list in host memory would have to outlive a captured call
    bands::band_table<2><<<std::min(blocks(G.ns), 1024u), 256, 0, st>>>(pl.bands, G.P, G.P, w.cells);
    SWEEP_LAUNCH_CHECK();
    SWEEP_CUDA(cudaMemsetAsync(w.zero0, 0, w.zero1 - w.zero0, st));
}

template <int M, bool FS>
static void forward_m(const sweep_elastic_desc* d, Plan& pl, float* record, void* tape, void* ws, int64_t ws_bytes,
                      cudaStream_t st)
{
    Carve c(ws);
    Ws w;
    carve(c, pl, false, w);
    SWEEP_REQUIRE(ws != nullptr && c.off <= ws_bytes, "elastic forward: workspace too small (%lld < %lld bytes)",
                  (long long)ws_bytes, (long long)c.off);
    setup(d, pl, w, st);
    const Geo& G = pl.G;
    if (G.nrec == 0) record = nullptr;
    if (record) SWEEP_CUDA(cudaMemsetAsync(record, 0, sizeof(float) * (size_t)G.B * G.nt * G.nrec * G.nrf, st));
    Fields F{};
    Mems W{};
    for (int k = 0; k < 5; ++k) F.f[k] = w.f[k];
    for (int k = 0; k < NMEM; ++k) W.m[k] = w.m[0][k];
    float* tp = static_cast<float*>(tape);
    const dim3 grid = grid_of(G, 1), block(8, (unsigned)G.rows);
    const long long nsave = (record ? (long long)G.B * G.nrec : 0) + (tp ? (long long)G.B * G.ns : 0);
    StepGraphs sg(st, resolve_graph_steps(-1));
    for (int it = 0; it < G.nt; ++it) {
        cudaStream_t s = sg.stream();
        vel<M, FS><<<grid, block, 0, s>>>(G, F, W);
        str<M, FS><<<grid, block, 0, s>>>(G, F, W);
        if (G.nsrc > 0) inject<<<(G.B * G.nsrc + 127) / 128, 128, 0, s>>>(G, F, it);
        if (nsave > 0) save<<<blocks(nsave), 256, 0, s>>>(G, F, record, tp ? tp + it * slot_floats(pl) : nullptr, it);
        SWEEP_LAUNCH_CHECK();
        sg.step_done();
    }
    sg.flush();
    if (tp) {
        // the final state, (5, B, nz, nx)
        float* last = tp + (long long)G.nt * slot_floats(pl);
        const long long rows = (long long)G.B * G.nz;
        for (int f = 0; f < 5; ++f) copy_rows(last + f * rows * G.nx, G.nx, w.f[f], G.P, G.nx, rows, st);
    }
}

template <int M, bool FS>
static void backward_m(const sweep_elastic_desc* d, Plan& pl, const float* adj, const void* tape, const Out& out,
                       void* ws, int64_t ws_bytes, cudaStream_t st)
{
    SWEEP_REQUIRE(tape != nullptr, "elastic backward: the forward's tape is required");
    Carve c(ws);
    Ws w;
    carve(c, pl, true, w);
    SWEEP_REQUIRE(ws != nullptr && c.off <= ws_bytes, "elastic backward: workspace too small (%lld < %lld bytes)",
                  (long long)ws_bytes, (long long)c.off);
    setup(d, pl, w, st);
    const Geo& G = pl.G;
    const float* tp = static_cast<const float*>(tape);
    const float* last = tp + (long long)G.nt * slot_floats(pl);
    const long long rows = (long long)G.B * G.nz;
    for (int f = 0; f < 5; ++f) copy_rows(w.f[f], G.P, last + f * rows * G.nx, G.nx, G.nx, rows, st);
    Rev R{};
    for (int k = 0; k < 5; ++k) R.f.f[k] = w.f[k];
    for (int k = 0; k < 3; ++k) { R.q[k] = w.q[k]; R.g[k] = w.g[k]; }
    for (int k = 0; k < 2; ++k) { R.a[k] = w.a[k]; R.p[k] = w.p[k]; }
    R.adj = adj;
    const long long ne = (long long)G.B * G.nsrc + (long long)G.B * G.nrec;
    const unsigned bb = blocks((long long)G.B * G.ns);
    int cur = 0;
    StepGraphs sg(st, resolve_graph_steps(-1));
    for (int it = G.nt - 1; it >= 1; --it) {
        cudaStream_t s = sg.stream();
        R.it = it;
        for (int k = 0; k < NMEM; ++k) { R.ai.m[k] = w.m[cur][k]; R.ao.m[k] = w.m[cur ^ 1][k]; }
        cur ^= 1;
        const float* prev = tp + (long long)(it - 1) * slot_floats(pl);
        if (ne > 0) events<<<(unsigned)((ne + 127) / 128), 128, 0, s>>>(G, R);
        launch_a<M, FS>(G, R, s);
        restore<<<dim3(bb, 3), 256, 0, s>>>(G, R, prev, SXX);
        launch_b<M, FS>(G, R, s);
        restore<<<dim3(bb, 2), 256, 0, s>>>(G, R, prev, VX);
        SWEEP_LAUNCH_CHECK();
        sg.step_done();
    }
    sg.flush();
    finalize<<<std::min(blocks((long long)pl.nm * G.nz * G.nx), 8192u), 256, 0, st>>>(G, R, out);
    SWEEP_LAUNCH_CHECK();
}

#define SWEEP_EORD_DISPATCH(M_, CALL) \
    switch (M_) {                     \
    case 1: CALL(1); break;           \
    case 2: CALL(2); break;           \
    case 3: CALL(3); break;           \
    case 5: CALL(5); break;           \
    case 6: CALL(6); break;           \
    default: CALL(7); break;          \
    }

void forward(const sweep_elastic_desc* d, int mem_mode, int, float* record, void* tape, void* ws, int64_t ws_bytes,
             cudaStream_t st)
{
    Plan pl = make_plan(d, mem_mode);
#define SWEEP_EORD_FWD(m)                                                   \
    (pl.G.fs ? forward_m<m, true>(d, pl, record, tape, ws, ws_bytes, st)    \
             : forward_m<m, false>(d, pl, record, tape, ws, ws_bytes, st))
    SWEEP_EORD_DISPATCH(d->M, SWEEP_EORD_FWD)
#undef SWEEP_EORD_FWD
}

void backward(const sweep_elastic_desc* d, int mem_mode, int, const float* adj, const void* tape, float* grad_vp,
              float* grad_vs, float* grad_rho, void* ws, int64_t ws_bytes, cudaStream_t st)
{
    Plan pl = make_plan(d, mem_mode);
    const Out out{d->vp, d->vs, d->rho, {grad_vp, grad_vs, grad_rho}};
#define SWEEP_EORD_BWD(m)                                                       \
    (pl.G.fs ? backward_m<m, true>(d, pl, adj, tape, out, ws, ws_bytes, st)     \
             : backward_m<m, false>(d, pl, adj, tape, out, ws, ws_bytes, st))
    SWEEP_EORD_DISPATCH(d->M, SWEEP_EORD_BWD)
#undef SWEEP_EORD_BWD
}

}  // namespace eord
}  // namespace sweep
