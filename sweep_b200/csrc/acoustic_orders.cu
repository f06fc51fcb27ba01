// acoustic_orders.cu -- the acoustic forward and boundary-saving adjoint at
// every spatial order but 8 (M = 1..7: orders 2, 4, 6, 10, 12, 14), 2-D and
// 3-D, for sm_100a.  Order 8 runs the TMA-tiled kernels of acoustic2d.cu /
// acoustic3d.cu; the reference's Acoustic / Acoustic3D default to order 4, so
// a drop-in caller lands here unless it asks for order 8.
//
// Restates the reference's templated acoustic path (src/sweep/csrc/cuda/
// equations/acoustic2d/forward_split.cu:40-250, adjoint_split.cu:27-300,
// acoustic3d/forward_split.cu:79-372, adjoint_split.cu:14-320,
// driver_traits.cuh step order), order by order:
//   * forward and reconstruction Laplacian in difference form
//     sum_k c_k ((u_k - u0) + (u_-k - u0)) / h^2, except order 4, which keeps
//     the summed form (c1 (u_1 + u_-1) + c2 (u_2 + u_-2) - 5/2 u0) / h^2
//     (operators/laplace.cuh:68-100, 145-200); the adjoint in difference
//     form at every order;
//   * CPML per axis in the compute band: 2-D with the fused d(a psi) term
//     (pad + 2M band), 3-D with the product-rule split a d(psi) + d(a) psi on
//     the band plus one cell; the exact transposes in the adjoint;
//   * boundary saving: the strip cells (width M + 1 inside the physical box)
//     of u(it) every step, the last two states at the end; the reverse
//     reconstructs the box minus the strips, restores the strips, takes the
//     source back out of a strip cell, images, re-injects.
//
// One launch per step and pass carries the stencils, the strips and the
// image (`fwd`, `rev`), a second one the sources and receivers.  Four x cells
// per thread (vec4.cuh) on pitched rows; a warp covers 32 x 4 (x, y) cells in
// 3-D and 32 x 4 (x, z) in 2-D, shots fastest in the grid so that the cells of
// one model tile meet in L2.  An axis's CPML runs, and its memories are read
// and written, only where its profile reaches.
//
// Measured, order 4: the 16-shot 256 x 768 survey's steps 24 us forward and
// 48 us reverse (31 and 66 + 31 + 14 us in nine launches with one cell per
// thread; 8.5 and 26 us of field traffic at the copy rate), a 101 x 119 x 141
// grid's with two shots 71 and 123 us (123 and 296 us; 20 and 50 us).  Bound
// by latency at 64 registers a thread (`rev` spills 84 bytes in 2-D and 136 in
// 3-D for them) and, in the layers, by the memories' taps.
// Memory: boundary saving with fp32 strips in device memory (SWEEP_MEM_BOUNDARY).
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "acoustic_orders.cuh"
#include "acoustic_vec.cuh"

namespace sweep {
namespace aord {

using namespace avec;

constexpr int kThreads = 256;
// blocks per SM the step kernels are compiled for: what the taps' registers
// leave (at order 4, no bound / 3 / 4 / 5 / 6 blocks took 27.3 / 24.8 / 22.0 / 26.5
// / 30.0 ms on the 2-D survey's gradient, 43 / 36.7 / 33.8 / 44.8 / 58.7 ms on a
// 101 x 119 x 141 grid's)
constexpr int blocks_for(int m) { return m <= 2 ? 4 : m <= 4 ? 3 : 2; }

// the forward step on the core, and the strips of u
template <int M, int ND>
__global__ void __launch_bounds__(kThreads, blocks_for(M)) fwd(const Geo G, const Step A)
{
    const Cell<ND> q(G);
    if (!q.core) return;
    const long long k = q.b * G.S + q.i;
    F4 u0;
    const F4 un = step_cells<M, ND>(G, q, A, k, u0);
    store_core(G, q, A.unx + k, un);
    if (!A.slot) return;
    bool phys[4], rec[4], any;
    lanes<ND>(G, q, phys, rec, any);
    if (!any) return;
    float* slot = A.slot + (long long)q.b * G.ns;
#pragma unroll
    for (int l = 0; l < 4; ++l)
        if (phys[l] && !rec[l]) slot[strip_index<ND>(G, q.c[2], q.c[1], q.c[0] + l)] = u0.v[l];
}

// lambda(it) on the core; u(it-1) on the physical box -- rebuilt in the
// reconstruction box, the saved strips around it -- and its image with
// lambda(it), before the step's residuals and source (`rev_events` adds what
// these change).
template <int M, int ND>
__global__ void __launch_bounds__(kThreads, blocks_for(M)) rev(const Geo G, const Rev A)
{
    const Cell<ND> q(G);
    if (!q.core) return;
    const long long k = q.b * G.S + q.i, mi = q.b * G.ms + q.i;
    const F4 lx = adj_cells<M, ND>(G, q, A, k, mi);
    store_core(G, q, A.lx + k, lx);
    if (!A.rx) return;
    bool phys[4], rec[4], any;
    lanes<ND>(G, q, phys, rec, any);
    if (!any) return;
    const F4 u0 = v4::ldg(A.rn + k), up = v4::ldg(A.rp + k);
    F4 un = u0;
    if (rec[0] || rec[1] || rec[2] || rec[3]) un = recon_cells<M, ND>(G, A.rn, k, coef<ND>(G, q), u0, up);
    const float* slot = A.slot + (long long)q.b * G.ns;
    F4 g = v4::ld(A.g + k);
    bool all = true;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        all &= phys[l];
        if (!phys[l]) continue;
        if (!rec[l]) un.v[l] = __ldg(slot + strip_index<ND>(G, q.c[2], q.c[1], q.c[0] + l));
        g.v[l] += ((un.v[l] - 2.f * u0.v[l]) + up.v[l]) * lx.v[l];
    }
    v4::st(A.g + k, g);
    if (all) {
        v4::st(A.rx + k, un);
    } else {
#pragma unroll
        for (int l = 0; l < 4; ++l)
            if (phys[l]) A.rx[k + l] = un.v[l];
    }
}

// ---------------------------------------------------- sources and receivers
// cell of location l (x[, y], z) as z, y, x, or false off the grid
__device__ __forceinline__ bool cell_at(const Geo& G, const int* l, int& z, int& y, int& x)
{
    x = l[0];
    y = G.nd == 3 ? l[1] : 0;
    z = l[G.nd - 1];
    return x >= 0 && x < G.nx && y >= 0 && y < G.ny && z >= 0 && z < G.nz;
}
__device__ __forceinline__ long long offset(const Geo& G, int b, int z, int y, int x)
{
    return b * G.S + ((long long)z * G.SZ + y * G.SY + x);
}
__device__ __forceinline__ bool in_box_nd(const Geo& G, const int* lo, const int* hi, int z, int y, int x)
{
    return G.nd == 3 ? in_box<3>(lo, hi, z, y, x) : in_box<2>(lo, hi, z, y, x);
}

// Forward: u(cell) += wavelet[b, s, it] at the shot's sources, then (after a
// block barrier when `part` asks for both) record[b, it, r] = u(cell) at its
// receivers; records start zeroed, off-grid receivers stay 0.  One block per
// shot and part 3, or blocks over part 1 / part 2.
enum { PART_SRC = 1, PART_REC = 2 };

__global__ void fwd_events(const Geo G, float* u, float* record, int it, int part)
{
    const int b = blockIdx.y;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    int z, y, x;
    if (part & PART_SRC)
        for (int s = t0; s < G.nsrc; s += step) {
            const long long e = (long long)b * G.nsrc + s;
            if (cell_at(G, G.src + e * G.nd, z, y, x)) atomicAdd(u + offset(G, b, z, y, x), G.wavelet[e * G.nt + it]);
        }
    if (part == (PART_SRC | PART_REC)) __syncthreads();
    if (part & PART_REC)
        for (int r = t0; r < G.nrec; r += step)
            if (cell_at(G, G.rec + ((long long)b * G.nrec + r) * G.nd, z, y, x))
                record[((long long)b * G.nt + it) * G.nrec + r] = __ldcg(u + offset(G, b, z, y, x));
}

// Reverse, after `rev`: the residuals into lambda(it) and what they add to the
// image; then the wavelet gradient, and the source put back: into u(it-1) in
// the reconstruction box; a strip cell was restored with it, so there its
// share leaves the image.
struct RevEv {
    float *lx, *rx;                 // rx null at it = 0
    const float *rn, *rp, *adj;
    float *g, *gwav;                // gwav null: no wavelet gradient
    int add_src;
};

__global__ void rev_events(const Geo G, const RevEv A, int it, int part)
{
    const int b = blockIdx.y;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    int z, y, x;
    if (part & PART_REC)
        for (int r = t0; r < G.nrec; r += step) {
            if (!cell_at(G, G.rec + ((long long)b * G.nrec + r) * G.nd, z, y, x)) continue;
            const long long o = offset(G, b, z, y, x);
            const float res = __ldg(A.adj + ((long long)b * G.nt + it) * G.nrec + r);
            atomicAdd(A.lx + o, res);
            if (A.rx && in_box_nd(G, G.lo, G.hi, z, y, x))
                atomicAdd(A.g + o, ((A.rx[o] - 2.f * A.rn[o]) + A.rp[o]) * res);
        }
    if (part == (PART_SRC | PART_REC)) __syncthreads();
    if (part & PART_SRC)
        for (int s = t0; s < G.nsrc; s += step) {
            const long long e = (long long)b * G.nsrc + s;
            if (!cell_at(G, G.src + e * G.nd, z, y, x)) continue;
            const long long o = offset(G, b, z, y, x);
            const float l = __ldcg(A.lx + o);
            if (A.gwav) A.gwav[e * G.nt + it] = l;
            if (!A.rx) continue;
            const float w = G.wavelet[e * G.nt + it];
            const bool strip = in_box_nd(G, G.lo, G.hi, z, y, x) && !in_box_nd(G, G.rlo, G.rhi, z, y, x);
            if (strip) atomicAdd(A.g + o, -w * l);
            else if (A.add_src) atomicAdd(A.rx + o, w);
        }
}

// u(cell) += sign * wavelet[b, s, it] at every source in a strip (strip) or
// outside the strips
__global__ void add_src(const Geo G, float* u, int it, float sign, int strip)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= G.B * G.nsrc) return;
    const int b = e / G.nsrc;
    int z, y, x;
    if (!cell_at(G, G.src + (long long)e * G.nd, z, y, x)) return;
    const bool s = in_box_nd(G, G.lo, G.hi, z, y, x) && !in_box_nd(G, G.rlo, G.rhi, z, y, x);
    if (s == (strip != 0)) atomicAdd(u + offset(G, b, z, y, x), sign * G.wavelet[(long long)e * G.nt + it]);
}

// illumination on the physical box: ir += lambda^2; is += u_tt^2 (is null:
// the it = 0 tail, lambda only)
__global__ void illum(const Geo G, const float* rx, const float* rn, const float* rp, const float* ln, float* is,
                      float* ir)
{
    const long long n = (long long)G.B * G.S;
    const float dt2 = G.dt * G.dt;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(k % G.S), x = c % G.P, r = c / G.P;
        if (!in_box_nd(G, G.lo, G.hi, r / G.ny, r % G.ny, x)) continue;
        ir[k] += ln[k] * ln[k];
        if (is) {
            const float utt = ((rx[k] - 2.f * rn[k]) + rp[k]) / dt2;
            is[k] += utt * utt;
        }
    }
}

// per-shot slots (B, S) -> out, unpitched: (B, cells) for per-shot models, else
// the sum over shots in shot order; image: times 2 / v (the factor 2 dt^2 / v
// of the reference's image and the 1 / dt^2 of its u_tt)
__global__ void finalize(const Geo G, const float* __restrict__ slots, int image, float* out)
{
    const long long cells = (long long)G.nz * G.ny * G.nx;
    const bool per_shot = G.ms != 0;
    const long long n = per_shot ? G.B * cells : cells;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long row = e / G.nx, k = row * G.P + (e - row * G.nx);
        float v = slots[k];
        if (!per_shot)
            for (int b = 1; b < G.B; ++b) v += slots[b * G.S + k];
        out[e] = image ? 2.f * v / G.vp[e] : v;
    }
}

// the model field of a pass, pitched: cf of the forward, ca of the reverse (whose
// reconstruction takes cf from the caller's models: a field less per model)
__global__ void prep(const Geo G, long long rows, int rev, float* __restrict__ c)
{
    const long long n = rows * G.P;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long row = k / G.P;
        const int x = (int)(k - row * G.P);
        const float v = x < G.nx ? G.vp[row * G.nx + x] : 0.f;
        c[k] = rev ? (v * v) * (G.dt * G.dt) : ((v * v) * G.dt) * G.dt;
    }
}

// ------------------------------------------------------------------- host
struct Plan {
    Geo G;
    int nm;                         // model copies
};

static Plan make_plan(const sweep_acoustic_desc* d, int mem_mode)
{
    SWEEP_REQUIRE(d != nullptr, "null descriptor");
    SWEEP_REQUIRE(d->ndim == 2 || d->ndim == 3, "acoustic: ndim %d is not built", d->ndim);
    SWEEP_REQUIRE(d->M >= 1 && d->M <= MAXM, "acoustic: spatial orders 2 to %d are built (got order %d)", 2 * MAXM,
                  2 * d->M);
    SWEEP_REQUIRE(d->M != 4, "acoustic: order 8 runs on kernels of its own");
    SWEEP_REQUIRE(mem_mode == SWEEP_MEM_BOUNDARY,
                  "acoustic order %d: boundary saving with fp32 strips in device memory is built for orders other "
                  "than 8 (mem_mode %d; checkpoints, reduced strip formats and the host tape run at order 8)",
                  2 * d->M, mem_mode);
    SWEEP_REQUIRE(d->B >= 1 && d->nt >= 1, "acoustic: B and nt must be >= 1");
    SWEEP_REQUIRE(d->nsrc >= 0 && d->nrec >= 0, "acoustic: negative source/receiver count");
    for (int f = 0; f < 6; ++f)
        SWEEP_REQUIRE(d->pad[f] >= 0, "acoustic: negative PML pad on face %d", f);
    Plan pl{};
    Geo& G = pl.G;
    const int M = d->M;
    G.nd = d->ndim; G.B = d->B; G.nz = d->nz; G.nx = d->nx; G.nt = d->nt; G.M = M;
    G.ny = d->ndim == 3 ? d->ny : 1;
    G.P = (G.nx + 7) / 8 * 8;
    G.SY = G.P; G.SZ = G.ny * G.P;
    G.S = (long long)G.nz * G.ny * G.P;
    const long long cells = (long long)G.nz * G.ny * G.nx;
    SWEEP_REQUIRE(cells < (1LL << 31) && G.S < (1LL << 31), "acoustic: one shot's grid must hold < 2^31 cells");
    SWEEP_REQUIRE(d->ndim == 2 || (long long)G.nz * G.B <= 65535, "acoustic: nz x shots must be <= 65535");
    SWEEP_REQUIRE(d->ndim == 3 || G.B <= 65535, "acoustic: at most 65535 shots per call");
    const int n[3] = {G.nx, G.ny, G.nz};
    const int plo[3] = {d->pad[4], d->pad[2], d->pad[0]}, phi[3] = {d->pad[5], d->pad[3], d->pad[1]};
    const float h[3] = {d->dx, d->dy, d->dz};
    // strip cells: the physical box within M + 1 of its faces (widths clipped
    // on a thin box: boundary/strip.cuh:63-67)
    for (int a = 0; a < 3; ++a) {
        if (G.nd == 2 && a == 1) { G.lo[a] = G.rlo[a] = 0; G.hi[a] = G.rhi[a] = 1; continue; }
        G.lo[a] = plo[a] + M; G.hi[a] = n[a] - phi[a] - M;
        G.rlo[a] = G.lo[a] + M + 1; G.rhi[a] = G.hi[a] - (M + 1);
        G.wl[a] = std::min(M + 1, std::max(G.hi[a] - G.lo[a], 0));
        G.wh[a] = std::min(M + 1, std::max(G.hi[a] - G.lo[a] - G.wl[a], 0));
        G.ih2[a] = 1.f / (h[a] * h[a]);
        G.ih[a] = 1.f / h[a];
    }
    SWEEP_REQUIRE(G.hi[2] > G.lo[2] && G.hi[0] > G.lo[0] && G.hi[1] > G.lo[1], "acoustic: the physical box is empty");
    const long long bx = G.hi[0] - G.lo[0], by = G.hi[1] - G.lo[1], bz = G.hi[2] - G.lo[2];
    const long long byi = std::max(0LL, by - G.wl[1] - G.wh[1]), bzi = std::max(0LL, bz - G.wl[2] - G.wh[2]);
    G.n_top = (int)(G.wl[2] * by * bx);
    G.n_bot = (int)(G.wh[2] * by * bx);
    G.nring = (int)((G.wl[1] + G.wh[1]) * bx + byi * (G.wl[0] + G.wh[0]));
    G.ns = (int)(G.n_top + G.n_bot + bzi * G.nring);
    G.dt = d->dt;
    for (int k = 0; k <= MAXM; ++k) { G.lc[k] = k <= M ? d->lap[k] : 0.f; G.gc[k] = k <= M ? d->grad[k] : 0.f; }
    G.vp = d->vp;
    SWEEP_REQUIRE(d->vp_stride == 0 || d->vp_stride == cells, "acoustic: vp_stride must be 0 or the cells per shot");
    G.ms = d->vp_stride ? G.S : 0;
    pl.nm = d->vp_stride ? G.B : 1;
    G.nsrc = d->nsrc; G.nrec = d->nrec;
    G.src = d->src_loc; G.rec = d->rec_loc; G.wavelet = d->wavelet;
    G.nbx = (G.nx + 31) / 32;
    return pl;
}

struct Ws {
    float* model;
    float* prof[3];
    float* u[3];                    // forward: u_prev, u, u_next; backward: reconstruction
    float* l[2];                    // backward: adjoint, two times of which the older is written over
    float* ps[2][3];                // CPML psi (forward) / adjoint psi, double-buffered
    float* zt[2][3];                // zeta (forward: [0] only) / adjoint zeta, double-buffered
    float *g, *is, *ir;             // backward: per-shot image, illumination slots
    char *zero0, *zero1;
};

static void carve(Carve& c, const Plan& pl, bool rev, Ws& w)
{
    const Geo& G = pl.G;
    const long long n = (long long)G.B * G.S;
    w = Ws{};
    w.model = c.take<float>(pl.nm * G.S);
    const int len[3] = {G.P + 2 * kGuard, G.ny + 2 * kGuard, G.nz + 2 * kGuard};
    for (int a = 0; a < 3; ++a) w.prof[a] = c.take<float>(4LL * len[a]);
    c.take<char>(0);
    w.zero0 = c.base ? c.base + c.off : nullptr;
    for (int k = 0; k < 3; ++k) w.u[k] = c.take<float>(n);
    for (int s = 0; s < 2; ++s)
        for (int a = 0; a < 3; ++a)
            if (a != 1 || G.nd == 3) w.ps[s][a] = c.take<float>(n);
    for (int s = 0; s < (rev ? 2 : 1); ++s)
        for (int a = 0; a < 3; ++a)
            if (a != 1 || G.nd == 3) w.zt[s][a] = c.take<float>(n);
    if (rev) {
        for (float*& p : w.l) p = c.take<float>(n);
        w.g = c.take<float>(n);
        w.is = c.take<float>(n);
        w.ir = c.take<float>(n);
    }
    c.take<char>(0);
    w.zero1 = c.base ? c.base + c.off : nullptr;
}

static long long slot_floats(const Plan& pl) { return (long long)pl.G.B * pl.G.ns; }

// cells of the state of a tape
static long long state_floats(const Geo& G) { return (long long)G.B * G.nz * G.ny * G.nx; }

static void copy_state(const Geo& G, float* dst, int dst_pitch, const float* src, int src_pitch, cudaStream_t st)
{
    copy_rows(dst, dst_pitch, src, src_pitch, G.nx, (long long)G.B * G.nz * G.ny, st);
}

void sizes(const sweep_acoustic_desc* d, int mem_mode, int, int64_t* ws_bytes, int64_t* tape_bytes)
{
    const Plan pl = make_plan(d, mem_mode);
    Carve f(nullptr), r(nullptr);
    Ws w;
    carve(f, pl, false, w);
    carve(r, pl, true, w);
    *ws_bytes = std::max(f.off, r.off);
    *tape_bytes = ((long long)pl.G.nt * slot_floats(pl) + 2 * state_floats(pl.G)) * 4;
}

// Rows of a 2-D block: 32, or 8 where that leaves the GPU with less than two
// blocks per SM (a small grid's step is one round of memory latency, and lasts
// as long as its fullest SM).
static int rows_of(const Geo& G)
{
    return (long long)G.nbx * G.B * ((G.nz + 31) / 32) >= 2 * 148 ? 32 : 8;
}

static dim3 cell_grid(const Geo& G)
{
    if (G.nd == 2) return dim3((unsigned)(G.nbx * G.B), (unsigned)((G.nz + rows_of(G) - 1) / rows_of(G)));
    return dim3((unsigned)(G.nbx * G.B), (G.ny + kBY - 1) / kBY, (G.nz + kBZ - 1) / kBZ);
}

static dim3 cell_block(const Geo& G) { return G.nd == 2 ? dim3(8, (unsigned)rows_of(G)) : dim3(8, kBY, kBZ); }

static unsigned blocks_of(long long n, int per)
{
    return (unsigned)std::max<long long>(std::min<long long>((n + per - 1) / per, 8192), 1);
}

static void setup(const sweep_acoustic_desc* d, Plan& pl, const Ws& w, bool rev, cudaStream_t st)
{
    Geo& G = pl.G;
    (rev ? G.ca : G.cf) = w.model;
    const long long rows = (long long)pl.nm * G.nz * G.ny;
    prep<<<blocks_of(rows * G.P, 256), 256, 0, st>>>(G, rows, rev, w.model);
    const float* in[3][3] = {{d->ax, d->bx, d->dbx}, {d->ay, d->by, d->dby}, {d->az, d->bz, d->dbz}};
    const int n[3] = {G.nx, G.ny, G.nz};
    for (int a = 0; a < 3; ++a) {
        if (a == 1 && G.nd == 2) continue;
        const int len = (a == 0 ? G.P : n[a]) + 2 * kGuard;
        prep_profiles<<<blocks_of(len, 256), 256, 0, st>>>(in[a][0], in[a][1], in[a][2], n[a], G, G.ih[a], kGuard, len,
                                                           w.prof[a]);
        G.a[a] = w.prof[a] + kGuard; G.b[a] = G.a[a] + len; G.db[a] = G.b[a] + len; G.da[a] = G.db[a] + len;
    }
    SWEEP_LAUNCH_CHECK();
    SWEEP_CUDA(cudaMemsetAsync(w.zero0, 0, w.zero1 - w.zero0, st));
}

// Sources and receivers of a step: one launch with a block per shot while a
// block walks the receivers in a few rounds, else one launch per kind.
constexpr int kEventBlock = 512;
static bool one_launch(const Geo& G) { return G.nrec <= 4 * kEventBlock && G.nsrc <= 4 * kEventBlock; }
static dim3 event_grid(const Geo& G, int n)
{
    return dim3((unsigned)std::max(1, (n + kEventBlock - 1) / kEventBlock), (unsigned)G.B);
}

template <int M, int ND>
static void forward_m(const sweep_acoustic_desc* d, Plan& pl, float* record, void* tape, void* ws, int64_t ws_bytes,
                      cudaStream_t st)
{
    Carve c(ws);
    Ws w;
    carve(c, pl, false, w);
    SWEEP_REQUIRE(ws != nullptr && c.off <= ws_bytes, "acoustic forward: workspace too small (%lld < %lld bytes)",
                  (long long)ws_bytes, (long long)c.off);
    setup(d, pl, w, false, st);
    const Geo& G = pl.G;
    if (G.nrec == 0) record = nullptr;
    if (record) SWEEP_CUDA(cudaMemsetAsync(record, 0, sizeof(float) * (size_t)G.B * G.nt * G.nrec, st));
    float* tp = static_cast<float*>(tape);
    float *up = w.u[0], *un = w.u[1], *unx = w.u[2];
    int cur = 0;
    const dim3 grid = cell_grid(G), block = cell_block(G);
    const int parts = (G.nsrc > 0 ? PART_SRC : 0) | (record ? PART_REC : 0);
    StepGraphs sg(st, resolve_graph_steps(-1));
    for (int it = 0; it < G.nt; ++it) {
        cudaStream_t s = sg.stream();
        Step A{};
        A.un = un; A.up = up; A.unx = unx;
        for (int a = 0; a < 3; ++a) { A.ps[a] = w.ps[cur][a]; A.psn[a] = w.ps[cur ^ 1][a]; A.zt[a] = w.zt[0][a]; }
        A.slot = tp ? tp + (long long)it * slot_floats(pl) : nullptr;
        fwd<M, ND><<<grid, block, 0, s>>>(G, A);
        if (parts && one_launch(G)) {
            fwd_events<<<dim3(1, G.B), kEventBlock, 0, s>>>(G, unx, record, it, parts);
        } else {
            if (parts & PART_SRC) fwd_events<<<event_grid(G, G.nsrc), kEventBlock, 0, s>>>(G, unx, record, it, PART_SRC);
            if (parts & PART_REC) fwd_events<<<event_grid(G, G.nrec), kEventBlock, 0, s>>>(G, unx, record, it, PART_REC);
        }
        SWEEP_LAUNCH_CHECK();
        sg.step_done();
        float* t = up; up = un; un = unx; unx = t;
        cur ^= 1;
    }
    sg.flush();
    if (tp) {
        float* tail = tp + (long long)G.nt * slot_floats(pl);
        copy_state(G, tail, G.nx, up, G.P, st);
        copy_state(G, tail + state_floats(G), G.nx, un, G.P, st);
    }
}

template <int M, int ND>
static void backward_m(const sweep_acoustic_desc* d, Plan& pl, const float* adj, const void* tape, float* grad_vp,
                       float* grad_wavelet, float* illum_src, float* illum_rec, void* ws, int64_t ws_bytes,
                       cudaStream_t st)
{
    Carve c(ws);
    Ws w;
    carve(c, pl, true, w);
    SWEEP_REQUIRE(ws != nullptr && c.off <= ws_bytes, "acoustic backward: workspace too small (%lld < %lld bytes)",
                  (long long)ws_bytes, (long long)c.off);
    SWEEP_REQUIRE(tape != nullptr, "acoustic backward: the forward's tape is required");
    setup(d, pl, w, true, st);
    const Geo& G = pl.G;
    if (G.nsrc == 0) grad_wavelet = nullptr;
    if (grad_wavelet)
        SWEEP_CUDA(cudaMemsetAsync(grad_wavelet, 0, sizeof(float) * (size_t)G.B * G.nsrc * G.nt, st));
    const float* tp = static_cast<const float*>(tape);
    const long long n = (long long)G.B * G.S;
    const bool il = illum_src || illum_rec;
    float *rp = w.u[0], *rn = w.u[1], *rx = w.u[2];
    const float* tail = tp + (long long)G.nt * slot_floats(pl);
    copy_state(G, rp, G.P, tail + state_floats(G), G.nx, st);
    copy_state(G, rn, G.P, tail, G.nx, st);
    float *lp = w.l[0], *ln = w.l[1];
    int cur = 0;
    const dim3 grid = cell_grid(G), block = cell_block(G);
    const unsigned cb = blocks_of(n, 256), srcb = (unsigned)(G.B * G.nsrc + 127) / 128;
    const int parts = (G.nsrc > 0 ? PART_SRC : 0) | (G.nrec > 0 ? PART_REC : 0);
    StepGraphs sg(st, resolve_graph_steps(-1));
    for (int it = G.nt - 1; it >= 0; --it) {
        cudaStream_t s = sg.stream();
        const bool recon = it > 0;
        Rev A{};
        A.ln = ln; A.lp = A.lx = lp;
        for (int a = 0; a < 3; ++a) {
            A.ps[a] = w.ps[cur][a]; A.zt[a] = w.zt[cur][a];
            A.pso[a] = w.ps[cur ^ 1][a]; A.zto[a] = w.zt[cur ^ 1][a];
        }
        A.rn = rn; A.rp = rp; A.rx = recon ? rx : nullptr;
        A.slot = recon ? tp + (long long)(it - 1) * slot_floats(pl) : nullptr;
        A.g = w.g;
        rev<M, ND><<<grid, block, 0, s>>>(G, A);
        const RevEv E{lp, recon ? rx : nullptr, rn, rp, adj, w.g, grad_wavelet, il ? 0 : 1};
        if (parts && one_launch(G)) {
            rev_events<<<dim3(1, G.B), kEventBlock, 0, s>>>(G, E, it, parts);
        } else {
            if (parts & PART_REC) rev_events<<<event_grid(G, G.nrec), kEventBlock, 0, s>>>(G, E, it, PART_REC);
            if (parts & PART_SRC) rev_events<<<event_grid(G, G.nsrc), kEventBlock, 0, s>>>(G, E, it, PART_SRC);
        }
        if (il) {
            // u_tt without the source: out of the restored strips for the
            // illumination's read, then back everywhere
            if (recon && G.nsrc > 0) add_src<<<srcb, 128, 0, s>>>(G, rx, it, -1.f, 1);
            illum<<<cb, 256, 0, s>>>(G, rx, rn, rp, lp, recon ? w.is : nullptr, w.ir);
            if (recon && G.nsrc > 0) {
                add_src<<<srcb, 128, 0, s>>>(G, rx, it, 1.f, 1);
                add_src<<<srcb, 128, 0, s>>>(G, rx, it, 1.f, 0);
            }
        }
        SWEEP_LAUNCH_CHECK();
        sg.step_done();
        std::swap(lp, ln);
        { float* t = rp; rp = rn; rn = rx; rx = t; }
        cur ^= 1;
    }
    sg.flush();
    finalize<<<cb, 256, 0, st>>>(G, w.g, 1, grad_vp);
    if (illum_src) finalize<<<cb, 256, 0, st>>>(G, w.is, 0, illum_src);
    if (illum_rec) finalize<<<cb, 256, 0, st>>>(G, w.ir, 0, illum_rec);
    SWEEP_LAUNCH_CHECK();
}

#define SWEEP_AORD_DISPATCH(M_, CALL)                                              \
    switch (M_) {                                                                  \
    case 1: CALL(1); break;                                                        \
    case 2: CALL(2); break;                                                        \
    case 3: CALL(3); break;                                                        \
    case 5: CALL(5); break;                                                        \
    case 6: CALL(6); break;                                                        \
    default: CALL(7); break;                                                       \
    }

void forward(const sweep_acoustic_desc* d, int mem_mode, int, float* record, void* tape, void* ws, int64_t ws_bytes,
             cudaStream_t st)
{
    Plan pl = make_plan(d, mem_mode);
#define SWEEP_AORD_FWD(m)                                                                        \
    (d->ndim == 2 ? forward_m<m, 2>(d, pl, record, tape, ws, ws_bytes, st)                       \
                  : forward_m<m, 3>(d, pl, record, tape, ws, ws_bytes, st))
    SWEEP_AORD_DISPATCH(d->M, SWEEP_AORD_FWD)
#undef SWEEP_AORD_FWD
}

void backward(const sweep_acoustic_desc* d, int mem_mode, int, const float* adj, const void* tape, float* grad_vp,
              float* grad_wavelet, float* illum_src, float* illum_rec, void* ws, int64_t ws_bytes, cudaStream_t st)
{
    Plan pl = make_plan(d, mem_mode);
#define SWEEP_AORD_BWD(m)                                                                                        \
    (d->ndim == 2 ? backward_m<m, 2>(d, pl, adj, tape, grad_vp, grad_wavelet, illum_src, illum_rec, ws, ws_bytes, st) \
                  : backward_m<m, 3>(d, pl, adj, tape, grad_vp, grad_wavelet, illum_src, illum_rec, ws, ws_bytes, st))
    SWEEP_AORD_DISPATCH(d->M, SWEEP_AORD_BWD)
#undef SWEEP_AORD_BWD
}

}  // namespace aord
}  // namespace sweep
