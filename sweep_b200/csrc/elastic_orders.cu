// elastic_orders.cu -- the 2-D isotropic elastic forward and boundary-saving
// adjoint at every spatial order but 8 (M = 1..7: orders 2, 4, 6, 10, 12,
// 14), for sm_100a.  Order 8 runs the tiled kernels of elastic2d.cu; the
// reference's Elastic defaults to order 4, so a drop-in caller lands here
// unless it asks for order 8.
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
// 18.6 ms a gradient (51 ms on fourteen launches of one cell per thread a
// reverse step): 14 + 13 us the two reverse kernels, 7 + 9 us the forward's;
// 16 shots of 400 x 1200: 189 + 165 and 61 + 75 us.  The small grid is bound
// by latency and launches, the large one by latency at 64 registers.
// Memory: boundary saving with fp32 bands in device memory (SWEEP_MEM_BOUNDARY).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "elastic_orders.cuh"
#include "vec4.cuh"

namespace sweep {
namespace eord {

using v4::F4;

constexpr int MAXM = 7;
constexpr int kGuard = 16;          // zero floats before and after a packed x profile
constexpr int kThreads = 256;
enum { VX = 0, VZ = 1, SXX = 2, SZZ = 3, SXZ = 4 };
// CPML memories: the field differenced and the axis
enum { M_VXX, M_VZZ, M_VXZ, M_VZX, M_SXXX, M_SZZZ, M_SXZX, M_SXZZ, NMEM };

struct Geo {
    int B, nz, nx, nt, M;
    int P;                          // row pitch
    long long S;                    // shot stride
    int fs;                         // bit f: traction-free face f (z_lo, z_hi, x_lo, x_hi; pad 0)
    int z0, z1, x0, x1;             // physical box
    int rz0, rz1, rx0, rx1;         // reverse box: the physical box minus one cell at an absorbing face
    int nbx, rows;                  // x blocks, rows of a block
    float dt, ihz, ihx;
    float c[MAXM + 1];              // staggered weights c[1..M]
    // profiles a, b at integer and at half positions; the x ones are padded
    // with zeros (kGuard floats before their start and past their end)
    const float *az, *bz, *azh, *bzh, *ax, *bx, *axh, *bxh;
    const float *lam, *mu, *kv;     // derived, pitched, kv = dt (1 / rho)
    long long ms;                   // model stride between shots (0 or S)
    int nsrc, nrec, nsf, nrf;
    int sf[5], rf[5];
    const int *src, *rec;           // (B, n, 2) runtime (x, z)
    const float* wavelet;           // (B, nsrc, nt)
    const int* cells;               // band cells of a shot grid, each once
    int ns;
};

struct Fields {
    float* f[5];
};
struct Mems {
    float* m[NMEM];
};

struct Cell {
    int b, z, x, i;                 // shot, coordinates of lane 0, offset in a shot
    bool grid, core;                // inside the grid; some lane is updated by the steps
    __device__ __forceinline__ explicit Cell(const Geo& G)
    {
        const int xb = blockIdx.x % G.nbx;
        b = blockIdx.x / G.nbx;
        x = 4 * (xb * 8 + threadIdx.x);
        z = blockIdx.y * G.rows + threadIdx.y;
        i = z * G.P + x;
        grid = x < G.nx && z < G.nz;
        core = grid && x + 3 >= G.M && x < G.nx - G.M && z >= G.M && z < G.nz - G.M;
    }
    __device__ __forceinline__ bool lane(const Geo& G, int l) const { return x + l >= G.M && x + l < G.nx - G.M; }
};

// ---------------------------------------------- traction-free faces
// Per axis (0 = z, 1 = x) the low surface is the first physical row / column
// and the high surface the last; a free face has no pad, so the surfaces bound
// the core.  Cells past them are air, read by a derivative along the axis as
// the image of the cell mirrored about the surface (about the node for integer
// fields, the half cell next to it for half fields), negated for odd fields;
// the M cells from a surface inwards take a unit-weight 2nd-order difference
// (elastic_free_surface.cuh:200-720), so the full stencil never meets the air.
struct FsAx {
    int lo_on, hi_on, lo, hi, n;
};

template <int AXIS>
__device__ __forceinline__ FsAx fs_axis(const Geo& G)
{
    if (AXIS == 0) return FsAx{G.fs & 1, (G.fs >> 1) & 1, G.z0, G.z1 - 1, G.nz};
    return FsAx{(G.fs >> 2) & 1, (G.fs >> 3) & 1, G.x0, G.x1 - 1, G.nx};
}
template <int M>
__device__ __forceinline__ bool fs_band(const FsAx& x, int j)
{
    return (x.lo_on && j >= x.lo && j < x.lo + M) || (x.hi_on && j > x.hi - M && j <= x.hi);
}
// the cell an air cell j is the image of (j itself in the medium)
__device__ __forceinline__ int fs_image(const FsAx& x, int j, bool half)
{
    if (x.lo_on && j < x.lo) return half ? 2 * x.lo - 1 - j : 2 * x.lo - j;
    if (x.hi_on && j >= (half ? x.hi : x.hi + 1)) return half ? 2 * x.hi - 1 - j : 2 * x.hi - j;
    return j;
}

// derivative along z of the group at p, row iz: FWD the D+ form, else D-
template <int M, bool FS, bool FWD>
__device__ __forceinline__ F4 dz(const Geo& G, const float* p, int iz, bool odd, bool half)
{
    const FsAx x = fs_axis<0>(G);
    if (!FS || !fs_band<M>(x, iz)) return v4::diff_col<M, FWD>(p, G.P, G.c, G.ihz);
    const int j1 = FWD ? iz + 1 : iz, j0 = FWD ? iz : iz - 1;
    const int m1 = fs_image(x, j1, half), m0 = fs_image(x, j0, half);
    const float s1 = odd && m1 != j1 ? -G.ihz : G.ihz, s0 = odd && m0 != j0 ? -G.ihz : G.ihz;
    const F4 a = v4::ldg(p + (m1 - iz) * G.P), b = v4::ldg(p + (m0 - iz) * G.P);
    F4 g;
#pragma unroll
    for (int l = 0; l < 4; ++l) g.v[l] = s1 * a.v[l] - s0 * b.v[l];
    return g;
}
// derivative along x, columns ix .. ix + 3
template <int M, bool FS, bool FWD>
__device__ __forceinline__ F4 dx(const Geo& G, const float* p, int ix, bool odd, bool half)
{
    F4 g = v4::diff_row<M, FWD>(p, G.c, G.ihx);
    if (FS && (G.fs & 12)) {
        const FsAx x = fs_axis<1>(G);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const int j = ix + l;
            if (!fs_band<M>(x, j)) continue;
            const int j1 = FWD ? j + 1 : j, j0 = FWD ? j : j - 1;
            const int m1 = fs_image(x, j1, half), m0 = fs_image(x, j0, half);
            const float s1 = odd && m1 != j1 ? -1.f : 1.f, s0 = odd && m0 != j0 ? -1.f : 1.f;
            g.v[l] = (s1 * __ldg(p + m1 - ix) - s0 * __ldg(p + m0 - ix)) * G.ihx;
        }
    }
    return g;
}

// The adjoint of dd near a free face at index j: the transpose over the output
// cells (weight 1 from a band, else the full weights), plus each free face's
// image of this cell in the air folded back with the field's parity.  add(w,
// m): add w times the value at index m.
template <int M, bool FWD, class Add>
__device__ __forceinline__ void fold(const FsAx& x, const float* c, int j, bool odd, bool half, const Add& add)
{
    auto plain = [&](int m, float s) {
#pragma unroll 1
        for (int k = 1; k <= M; ++k) {
            const int jp = FWD ? m + k - 1 : m + k, jm = FWD ? m - k : m - k + 1;
            if (jp >= 0 && jp < x.n && !fs_band<M>(x, jp)) add(s * c[k], jp);
            if (jm >= 0 && jm < x.n && !fs_band<M>(x, jm)) add(-s * c[k], jm);
        }
        const int p = FWD ? m : m + 1, q = FWD ? m - 1 : m;
        if (fs_band<M>(x, p)) add(s, p);
        if (fs_band<M>(x, q)) add(-s, q);
    };
    plain(j, 1.f);
    const float par = odd ? -1.f : 1.f;
    if (x.lo_on) {
        const int m = half ? 2 * x.lo - 1 - j : 2 * x.lo - j;
        if (m < x.lo) plain(m, par);
    }
    if (x.hi_on) {
        const int m = half ? 2 * x.hi - 1 - j : 2 * x.hi - j;
        if (m >= (half ? x.hi : x.hi + 1)) plain(m, par);
    }
}
// index j is far enough from the free faces for the plain transpose
template <int M>
__device__ __forceinline__ bool fs_far(const FsAx& x, int j)
{
    return (!x.lo_on || j >= x.lo + 2 * M) && (!x.hi_on || j <= x.hi - 2 * M);
}

__device__ __forceinline__ bool fs_zrow(const Geo& G, int iz)
{
    return ((G.fs & 1) && iz == G.z0) || ((G.fs & 2) && iz == G.z1 - 1);
}
__device__ __forceinline__ bool fs_xcol(const Geo& G, int ix)
{
    return ((G.fs & 4) && ix == G.x0) || ((G.fs & 8) && ix == G.x1 - 1);
}
__device__ __forceinline__ bool fs_zero_shear(const Geo& G, int ix, int iz)
{
    return ((G.fs & 2) && iz == G.z1 - 1) || ((G.fs & 8) && ix == G.x1 - 1);
}
__device__ __forceinline__ bool zbox(const Geo& G, int iz) { return iz >= G.z0 && iz < G.z1; }
__device__ __forceinline__ bool xbox(const Geo& G, int ix) { return ix >= G.x0 && ix < G.x1; }
// CPML test of the velocity step and the transposes: outside the physical box
__device__ __forceinline__ bool in_pml(const Geo& G, int ix, int iz) { return !(zbox(G, iz) && xbox(G, ix)); }
// the stress step's: a free surface row / column stays in the CPML branch
__device__ __forceinline__ bool in_pml_stress(const Geo& G, int ix, int iz)
{
    return ix < G.x0 + ((G.fs >> 2) & 1) || ix >= G.x1 - ((G.fs >> 3) & 1) || iz < G.z0 + (G.fs & 1) ||
           iz >= G.z1 - ((G.fs >> 1) & 1);
}
// an axis's profile is zero between these (the half-cell one reaches the box's last cell)
__device__ __forceinline__ bool zband(const Geo& G, int iz) { return iz < G.z0 || iz >= G.z1 - 1; }
__device__ __forceinline__ bool xband(const Geo& G, int ix) { return ix < G.x0 || ix + 3 >= G.x1 - 1; }

// ----------------------------------------------------------------- forward
__device__ __forceinline__ void cpml(float* m, const F4& a, const F4& b, F4& d, const bool (&on)[4])
{
    const F4 old = v4::ld(m);
    F4 t;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        t.v[l] = on[l] ? a.v[l] * old.v[l] + b.v[l] * d.v[l] : 0.f;
        d.v[l] = d.v[l] + t.v[l];
    }
    v4::st(m, t);
}

struct Four {
    F4 xx, xz, zx, zz;              // by field (or row of the tensor) and axis
};

template <int M, bool FS>
__device__ __forceinline__ Four stress_diffs(const Geo& G, const Fields& F, const Cell& q, long long k)
{
    return Four{dx<M, FS, true>(G, F.f[SXX] + k, q.x, true, false), dz<M, FS, false>(G, F.f[SXZ] + k, q.z, true, true),
                dx<M, FS, false>(G, F.f[SXZ] + k, q.x, true, true), dz<M, FS, true>(G, F.f[SZZ] + k, q.z, true, false)};
}
// xx = dvx/dx, xz = dvx/dz, zx = dvz/dx, zz = dvz/dz
template <int M, bool FS>
__device__ __forceinline__ Four velocity_diffs(const Geo& G, const Fields& F, const Cell& q, long long k)
{
    return Four{dx<M, FS, false>(G, F.f[VX] + k, q.x, true, true), dz<M, FS, true>(G, F.f[VX] + k, q.z, false, false),
                dx<M, FS, true>(G, F.f[VZ] + k, q.x, false, false), dz<M, FS, false>(G, F.f[VZ] + k, q.z, true, true)};
}

// velocity step (reference elastic2d/kernels.cuh:48-138)
template <int M, bool FS>
__global__ void __launch_bounds__(kThreads, M <= 4 ? 4 : 3) vel(const Geo G, const Fields F, const Mems W)
{
    const Cell q(G);
    if (!q.core) return;
    const long long k = q.b * G.S + q.i;
    Four d = stress_diffs<M, FS>(G, F, q, k);
    const F4 kv = v4::ldg(G.kv + q.b * G.ms + q.i);
    F4 vx = v4::ld(F.f[VX] + k), vz = v4::ld(F.f[VZ] + k);
    bool on[4];
    bool any = false;
#pragma unroll
    for (int l = 0; l < 4; ++l) any |= on[l] = q.lane(G, l) && in_pml(G, q.x + l, q.z);
    if (any && xband(G, q.x)) {
        cpml(W.m[M_SXXX] + k, v4::ldg(G.axh + q.x), v4::ldg(G.bxh + q.x), d.xx, on);
        cpml(W.m[M_SXZX] + k, v4::ldg(G.ax + q.x), v4::ldg(G.bx + q.x), d.zx, on);
    }
    if (any && zband(G, q.z)) {
        cpml(W.m[M_SZZZ] + k, v4::splat(__ldg(G.azh + q.z)), v4::splat(__ldg(G.bzh + q.z)), d.zz, on);
        cpml(W.m[M_SXZZ] + k, v4::splat(__ldg(G.az + q.z)), v4::splat(__ldg(G.bz + q.z)), d.xz, on);
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (!q.lane(G, l)) continue;
        vx.v[l] = vx.v[l] + kv.v[l] * (d.xx.v[l] + d.xz.v[l]);
        vz.v[l] = vz.v[l] + kv.v[l] * (d.zx.v[l] + d.zz.v[l]);
    }
    v4::st(F.f[VX] + k, vx);
    v4::st(F.f[VZ] + k, vz);
}

// stress step with the free faces' Robertsson corrections, then the zeroing
// (reference elastic2d/kernels.cuh:182-311)
template <int M, bool FS>
__global__ void __launch_bounds__(kThreads, M <= 4 ? 4 : 3) str(const Geo G, const Fields F, const Mems W)
{
    const Cell q(G);
    if (!q.core) return;
    const long long k = q.b * G.S + q.i, mi = q.b * G.ms + q.i;
    Four d = velocity_diffs<M, FS>(G, F, q, k);
    const F4 lam = v4::ldg(G.lam + mi), mu = v4::ldg(G.mu + mi);
    F4 sxx = v4::ld(F.f[SXX] + k), szz = v4::ld(F.f[SZZ] + k), sxz = v4::ld(F.f[SXZ] + k);
    bool on[4];
    bool any = false;
#pragma unroll
    for (int l = 0; l < 4; ++l)
        any |= on[l] = q.lane(G, l) && (FS ? in_pml_stress(G, q.x + l, q.z) : in_pml(G, q.x + l, q.z));
    if (any && xband(G, q.x)) {
        cpml(W.m[M_VXX] + k, v4::ldg(G.ax + q.x), v4::ldg(G.bx + q.x), d.xx, on);
        cpml(W.m[M_VZX] + k, v4::ldg(G.axh + q.x), v4::ldg(G.bxh + q.x), d.zx, on);
    }
    if (any && zband(G, q.z)) {
        cpml(W.m[M_VZZ] + k, v4::splat(__ldg(G.az + q.z)), v4::splat(__ldg(G.bz + q.z)), d.zz, on);
        cpml(W.m[M_VXZ] + k, v4::splat(__ldg(G.azh + q.z)), v4::splat(__ldg(G.bzh + q.z)), d.xz, on);
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (!q.lane(G, l)) continue;
        const float L = lam.v[l], m = mu.v[l], vxx = d.xx.v[l], vzz = d.zz.v[l];
        sxx.v[l] = sxx.v[l] + G.dt * ((L + 2.f * m) * vxx + L * vzz);
        szz.v[l] = szz.v[l] + G.dt * ((L + 2.f * m) * vzz + L * vxx);
        sxz.v[l] = sxz.v[l] + (G.dt * m) * (d.xz.v[l] + d.zx.v[l]);
        if (FS) {
            const bool zs = fs_zrow(G, q.z), xs = fs_xcol(G, q.x + l);
            if (zs) sxx.v[l] = sxx.v[l] + (-G.dt) * L * ((L / (L + 2.f * m)) * vxx + vzz);
            if (xs) szz.v[l] = szz.v[l] + (-G.dt) * L * ((L / (L + 2.f * m)) * vzz + vxx);
            if (zs) szz.v[l] = 0.f;
            if (xs) sxx.v[l] = 0.f;
            if (fs_zero_shear(G, q.x + l, q.z)) sxz.v[l] = 0.f;
        }
    }
    v4::st(F.f[SXX] + k, sxx);
    v4::st(F.f[SZZ] + k, szz);
    v4::st(F.f[SXZ] + k, sxz);
}

// grid offset of location (x, z), or -1 off the grid
__device__ __forceinline__ int loc(const Geo& G, const int* l)
{
    if (l[0] < 0 || l[0] >= G.nx || l[1] < 0 || l[1] >= G.nz) return -1;
    return l[1] * G.P + l[0];
}

// the wavelet of step it, times sign, into every source field
__device__ __forceinline__ void inject_at(const Geo& G, const Fields& F, int e, int it, float sign)
{
    const int c = loc(G, G.src + 2LL * e);
    if (c < 0) return;
    const float w = sign * G.wavelet[(long long)e * G.nt + it];
    for (int k = 0; k < G.nsf; ++k) atomicAdd(F.f[G.sf[k]] + e / G.nsrc * G.S + c, w);
}
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

// ---------------------------------------------------------------- reverse
struct Rev {
    Fields f, a;                    // reconstructed forward fields, adjoint fields
    Mems ai, ao;                    // adjoint CPML memories: read, written
    float* q[3];                    // dt C lambda_s: xx, zz, xz
    float* p[2];                    // kv lambda_v
    float* g[3];                    // per-shot slots (B, S): gl, gm - 2 gl, the rho image (times rho)
    const float* adj;               // (B, nt, nrec, nrf)
    int it;
};

// dt C s of the diagonal; on a surface row (zs) / column (xs) the transposes of
// the corrected updates, with the zeroed stress counting as zero
__device__ __forceinline__ void stiff(float dt, float lam, float mu, float sxx, float szz, bool zs, bool xs, float& qxx,
                                      float& qzz)
{
    if (zs || xs) {
        const float c = 4.f * mu * (lam + mu) / (lam + 2.f * mu);
        qxx = xs ? 0.f : dt * c * sxx;
        qzz = zs ? 0.f : dt * c * szz;
    } else {
        qxx = dt * ((lam + 2.f * mu) * sxx + lam * szz);
        qzz = dt * ((lam + 2.f * mu) * szz + lam * sxx);
    }
}

// signed residuals into the adjoint fields (stress -1, velocity +1) and what
// they add to q; the source of step it out of the forward fields
__global__ void events(const Geo G, const Rev R)
{
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < G.B * G.nsrc) { inject_at(G, R.f, e, R.it, -1.f); return; }
    e -= G.B * G.nsrc;
    if (e >= G.B * G.nrec) return;
    const int b = e / G.nrec, r = e - b * G.nrec;
    const int* l = G.rec + 2LL * e;
    const int c = loc(G, l);
    if (c < 0) return;
    const long long i = b * G.S + c, mi = b * G.ms + c;
    const float* res = R.adj + (((long long)b * G.nt + R.it) * G.nrec + r) * G.nrf;
    for (int k = 0; k < G.nrf; ++k) {
        const int f = G.rf[k];
        const float v = f >= SXX ? -res[k] : res[k];
        atomicAdd(R.a.f[f] + i, v);
        if (f < SXX) continue;
        if (f == SXZ) {
            if (!fs_zero_shear(G, l[0], l[1])) atomicAdd(R.q[2] + i, (G.dt * G.mu[mi]) * v);
            continue;
        }
        float qxx, qzz;
        stiff(G.dt, G.lam[mi], G.mu[mi], f == SXX ? v : 0.f, f == SZZ ? v : 0.f, fs_zrow(G, l[1]), fs_xcol(G, l[0]),
              qxx, qzz);
        if (qxx != 0.f) atomicAdd(R.q[0] + i, qxx);
        if (qzz != 0.f) atomicAdd(R.q[1] + i, qzz);
    }
}

__device__ __forceinline__ void add4(float* p, const F4& a)
{
    F4 t = v4::ld(p);
#pragma unroll
    for (int l = 0; l < 4; ++l) t.v[l] += a.v[l];
    v4::st(p, t);
}

// Stress reconstruction on the reverse box and the image on the physical box:
// with gl, gm the derivatives of the misfit by lambda and mu (up to -dt), grad
// vp = -2 rho vp dt gl, grad vs = -2 rho vs dt (gm - 2 gl), and the stiffness
// part of rho times grad rho, -dt (gl (lam + 2 mu) + (gm - 2 gl) mu)
// (reference kernels.cuh:365-535, 601-663).
template <int M, bool FS>
__device__ __forceinline__ void stress_rev(const Geo& G, const Rev& R, const Cell& q)
{
    if (!q.core || !zbox(G, q.z) || q.x + 3 < G.x0 || q.x >= G.x1) return;
    const long long k = q.b * G.S + q.i, mi = q.b * G.ms + q.i;
    const Four d = velocity_diffs<M, FS>(G, R.f, q, k);
    const F4 lam = v4::ldg(G.lam + mi), mu = v4::ldg(G.mu + mi);
    const F4 bxx = v4::ldg(R.a.f[SXX] + k), bzz = v4::ldg(R.a.f[SZZ] + k), bxz = v4::ldg(R.a.f[SXZ] + k);
    F4 sxx = v4::ld(R.f.f[SXX] + k), szz = v4::ld(R.f.f[SZZ] + k), sxz = v4::ld(R.f.f[SXZ] + k);
    const bool rrow = q.z >= G.rz0 && q.z < G.rz1;
    F4 sl = v4::splat(0.f), sm = sl, sr = sl;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const int x = q.x + l;
        if (!xbox(G, x)) continue;
        const float L = lam.v[l], m = mu.v[l], l2m = L + 2.f * m, vxx = d.xx.v[l], vzz = d.zz.v[l];
        const bool zs = FS && fs_zrow(G, q.z), xs = FS && fs_xcol(G, x);
        float gl, gm;
        if (zs || xs) {
            // the surface's one corrected update (zero in a corner)
            const float r = m / l2m, a = zs && xs ? 0.f : zs ? bxx.v[l] * vxx : bzz.v[l] * vzz;
            gl = a * 4.f * r * r;
            gm = a * 4.f * (1.f - 2.f * r + 2.f * r * r);
        } else {
            gl = (bxx.v[l] + bzz.v[l]) * (vxx + vzz);
            gm = 2.f * (bxx.v[l] * vxx + bzz.v[l] * vzz);
        }
        if (!(FS && fs_zero_shear(G, x, q.z))) gm = gm + bxz.v[l] * (d.xz.v[l] + d.zx.v[l]);
        const float gm2 = gm - 2.f * gl;
        sl.v[l] = gl;
        sm.v[l] = gm2;
        sr.v[l] = -G.dt * (gl * l2m + gm2 * m);
        if (rrow && x >= G.rx0 && x < G.rx1) {
            sxx.v[l] = sxx.v[l] - G.dt * (l2m * vxx + L * vzz);
            szz.v[l] = szz.v[l] - G.dt * (l2m * vzz + L * vxx);
            sxz.v[l] = sxz.v[l] - (G.dt * m) * (d.xz.v[l] + d.zx.v[l]);
        }
    }
    v4::st(R.f.f[SXX] + k, sxx);
    v4::st(R.f.f[SZZ] + k, szz);
    v4::st(R.f.f[SXZ] + k, sxz);
    add4(R.g[0] + k, sl);
    add4(R.g[1] + k, sm);
    add4(R.g[2] + k, sr);
}

// velocity reconstruction on the reverse box with its rho image
template <int M, bool FS>
__device__ __forceinline__ void vel_rev(const Geo& G, const Rev& R, const Cell& q)
{
    if (!q.core || q.z < G.rz0 || q.z >= G.rz1 || q.x + 3 < G.rx0 || q.x >= G.rx1) return;
    const long long k = q.b * G.S + q.i;
    const Four d = stress_diffs<M, FS>(G, R.f, q, k);
    const F4 kv = v4::ldg(G.kv + q.b * G.ms + q.i), lx = v4::ldg(R.a.f[VX] + k), lz = v4::ldg(R.a.f[VZ] + k);
    F4 vx = v4::ld(R.f.f[VX] + k), vz = v4::ld(R.f.f[VZ] + k), sr = v4::splat(0.f);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (q.x + l < G.rx0 || q.x + l >= G.rx1) continue;
        const float ux = kv.v[l] * (d.xx.v[l] + d.xz.v[l]), uz = kv.v[l] * (d.zx.v[l] + d.zz.v[l]);
        vx.v[l] = vx.v[l] - ux;
        vz.v[l] = vz.v[l] - uz;
        sr.v[l] = -(lx.v[l] * ux + lz.v[l] * uz);
    }
    v4::st(R.f.f[VX] + k, vx);
    v4::st(R.f.f[VZ] + k, vz);
    if (R.it > 1) add4(R.g[2] + k, sr);
}

// a transpose's input through its adjoint CPML memory w on the lanes `on`
__device__ __forceinline__ F4 through(const F4& u, const F4& b, const F4& w, const bool (&on)[4])
{
    F4 t;
#pragma unroll
    for (int l = 0; l < 4; ++l) t.v[l] = on[l] ? u.v[l] + b.v[l] * (w.v[l] + u.v[l]) : u.v[l];
    return t;
}

// The negated transpose of a derivative along z / x of the input u (memory w,
// profile prof): FWD the transpose of a D+ form (plain: D-), else of a D- form.
template <int M, bool FS, bool FWD>
__device__ __forceinline__ F4 adj_z(const Geo& G, const Cell& q, const float* u, const float* w, const float* prof,
                                    bool odd, bool half)
{
    const FsAx x = fs_axis<0>(G);
    const bool far = !FS || fs_far<M>(x, q.z);
    if (far && !zband(G, q.z - M) && !zband(G, q.z + M)) return v4::diff_col<M, !FWD>(u, G.P, G.c, G.ihz);
    // within the band's reach every tap takes its memory, one off the band with
    // the profile's zero, so that a thread's loads leave together
    auto row = [&](int j) {             // row q.z + j
        const int z = q.z + j;
        bool on[4];
#pragma unroll
        for (int l = 0; l < 4; ++l) on[l] = in_pml(G, q.x + l, z);
        return through(v4::ldg(u + j * G.P), v4::splat(__ldg(prof + z)), v4::ldg(w + j * G.P), on);
    };
    if (far) return v4::diff<M, !FWD>(row, G.c, G.ihz);
    F4 g = v4::splat(0.f);
    fold<M, FWD>(x, G.c, q.z, odd, half, [&](float c, int j) {
        const F4 t = row(j - q.z);
#pragma unroll
        for (int l = 0; l < 4; ++l) g.v[l] += c * t.v[l];
    });
#pragma unroll
    for (int l = 0; l < 4; ++l) g.v[l] *= G.ihz;
    return g;
}
template <int M, bool FS, bool FWD>
__device__ __forceinline__ F4 adj_x(const Geo& G, const Cell& q, const float* u, const float* w, const float* prof,
                                    bool odd, bool half)
{
    using S = v4::Span<M, !FWD>;
    float v[S::N];
    v4::window<S::LO, S::HI>(u, v);
    if (q.x - 4 * S::LO < G.x0 || q.x + 3 + 4 * S::HI >= G.x1 - 1) {
#pragma unroll
        for (int j = -S::LO; j <= S::HI; ++j) {
            const F4 b = v4::ldg(prof + q.x + 4 * j), t = v4::ldg(w + 4 * j);
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                float& e = v[4 * (j + S::LO) + l];
                if (in_pml(G, q.x + 4 * j + l, q.z)) e = e + b.v[l] * (t.v[l] + e);
            }
        }
    }
    F4 g = v4::diff_x<M, !FWD, S::O>(v, G.c, G.ihx);
    if (FS && (G.fs & 12)) {
        const FsAx ax = fs_axis<1>(G);
#pragma unroll 1
        for (int l = 0; l < 4; ++l) {
            const int j = q.x + l;
            if (fs_far<M>(ax, j) || !q.lane(G, l)) continue;
            float s = 0.f;
            fold<M, FWD>(ax, G.c, j, odd, half, [&](float c, int m) {
                float t = __ldg(u + m - q.x);
                if (in_pml(G, m, q.z)) t = t + __ldg(prof + m) * (__ldg(w + m - q.x) + t);
                s += c * t;
            });
            g.v[l] = s * G.ihx;
        }
    }
    return g;
}

// the next memory a (w + u) of this group in the layers
__device__ __forceinline__ void keep(const float* wi, float* wo, const F4& a, const F4& u, const bool (&on)[4])
{
    const F4 w = v4::ldg(wi);
    F4 t;
#pragma unroll
    for (int l = 0; l < 4; ++l) t.v[l] = on[l] ? a.v[l] * (w.v[l] + u.v[l]) : 0.f;
    v4::st(wo, t);
}

// the stress step's transpose (reference kernels.cuh:664-837): lambda_v on the
// core, then p = kv lambda_v
template <int M, bool FS>
__device__ __forceinline__ void adj_vel(const Geo& G, const Rev& R, const Cell& q)
{
    if (!q.grid) return;
    const long long k = q.b * G.S + q.i;
    const float *qxx = R.q[0] + k, *qzz = R.q[1] + k, *qxz = R.q[2] + k;
    bool on[4];
    bool any = false;
#pragma unroll
    for (int l = 0; l < 4; ++l) any |= on[l] = in_pml(G, q.x + l, q.z);
    if (any && xband(G, q.x)) {
        keep(R.ai.m[M_VXX] + k, R.ao.m[M_VXX] + k, v4::ldg(G.ax + q.x), v4::ldg(qxx), on);
        keep(R.ai.m[M_VZX] + k, R.ao.m[M_VZX] + k, v4::ldg(G.axh + q.x), v4::ldg(qxz), on);
    }
    if (any && zband(G, q.z)) {
        keep(R.ai.m[M_VZZ] + k, R.ao.m[M_VZZ] + k, v4::splat(__ldg(G.az + q.z)), v4::ldg(qzz), on);
        keep(R.ai.m[M_VXZ] + k, R.ao.m[M_VXZ] + k, v4::splat(__ldg(G.azh + q.z)), v4::ldg(qxz), on);
    }
    F4 dvx = v4::splat(0.f), dvz = dvx;
    if (q.core) {
        const F4 a = adj_x<M, FS, false>(G, q, qxx, R.ai.m[M_VXX] + k, G.bx, true, true);
        const F4 b = adj_z<M, FS, true>(G, q, qxz, R.ai.m[M_VXZ] + k, G.bzh, false, false);
        const F4 c = adj_x<M, FS, true>(G, q, qxz, R.ai.m[M_VZX] + k, G.bxh, false, false);
        const F4 d = adj_z<M, FS, false>(G, q, qzz, R.ai.m[M_VZZ] + k, G.bz, true, true);
#pragma unroll
        for (int l = 0; l < 4; ++l)
            if (q.lane(G, l)) { dvx.v[l] = a.v[l] + b.v[l]; dvz.v[l] = c.v[l] + d.v[l]; }
    }
    const F4 kv = v4::ldg(G.kv + q.b * G.ms + q.i);
    F4 vx = v4::ld(R.a.f[VX] + k), vz = v4::ld(R.a.f[VZ] + k), px, pz;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        vx.v[l] = vx.v[l] + dvx.v[l];
        vz.v[l] = vz.v[l] + dvz.v[l];
        px.v[l] = kv.v[l] * vx.v[l];
        pz.v[l] = kv.v[l] * vz.v[l];
    }
    v4::st(R.a.f[VX] + k, vx);
    v4::st(R.a.f[VZ] + k, vz);
    v4::st(R.p[0] + k, px);
    v4::st(R.p[1] + k, pz);
}

// the velocity step's transpose (reference kernels.cuh:873-1019): lambda_s on
// the core, then q = dt C lambda_s
template <int M, bool FS>
__device__ __forceinline__ void adj_str(const Geo& G, const Rev& R, const Cell& q)
{
    if (!q.grid) return;
    const long long k = q.b * G.S + q.i, mi = q.b * G.ms + q.i;
    const float *px = R.p[0] + k, *pz = R.p[1] + k;
    bool on[4];
    bool any = false;
#pragma unroll
    for (int l = 0; l < 4; ++l) any |= on[l] = in_pml(G, q.x + l, q.z);
    if (any && xband(G, q.x)) {
        keep(R.ai.m[M_SXXX] + k, R.ao.m[M_SXXX] + k, v4::ldg(G.axh + q.x), v4::ldg(px), on);
        keep(R.ai.m[M_SXZX] + k, R.ao.m[M_SXZX] + k, v4::ldg(G.ax + q.x), v4::ldg(pz), on);
    }
    if (any && zband(G, q.z)) {
        keep(R.ai.m[M_SXZZ] + k, R.ao.m[M_SXZZ] + k, v4::splat(__ldg(G.az + q.z)), v4::ldg(px), on);
        keep(R.ai.m[M_SZZZ] + k, R.ao.m[M_SZZZ] + k, v4::splat(__ldg(G.azh + q.z)), v4::ldg(pz), on);
    }
    F4 dxx = v4::splat(0.f), dzz = dxx, dxz = dxx;
    if (q.core) {
        const F4 a = adj_x<M, FS, true>(G, q, px, R.ai.m[M_SXXX] + k, G.bxh, true, false);
        const F4 b = adj_z<M, FS, true>(G, q, pz, R.ai.m[M_SZZZ] + k, G.bzh, true, false);
        const F4 c = adj_z<M, FS, false>(G, q, px, R.ai.m[M_SXZZ] + k, G.bz, true, true);
        const F4 d = adj_x<M, FS, false>(G, q, pz, R.ai.m[M_SXZX] + k, G.bx, true, true);
#pragma unroll
        for (int l = 0; l < 4; ++l)
            if (q.lane(G, l)) { dxx.v[l] = a.v[l]; dzz.v[l] = b.v[l]; dxz.v[l] = c.v[l] + d.v[l]; }
    }
    const F4 lam = v4::ldg(G.lam + mi), mu = v4::ldg(G.mu + mi);
    F4 sxx = v4::ld(R.a.f[SXX] + k), szz = v4::ld(R.a.f[SZZ] + k), sxz = v4::ld(R.a.f[SXZ] + k), qxx, qzz, qxz;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const bool zs = FS && fs_zrow(G, q.z), xs = FS && fs_xcol(G, q.x + l);
        const bool sh = FS && fs_zero_shear(G, q.x + l, q.z);
        // what the surfaces zero starts the step at zero (kernels.cuh:592-600)
        sxx.v[l] = (xs ? 0.f : sxx.v[l]) + dxx.v[l];
        szz.v[l] = (zs ? 0.f : szz.v[l]) + dzz.v[l];
        sxz.v[l] = (sh ? 0.f : sxz.v[l]) + dxz.v[l];
        stiff(G.dt, lam.v[l], mu.v[l], sxx.v[l], szz.v[l], zs, xs, qxx.v[l], qzz.v[l]);
        qxz.v[l] = sh ? 0.f : (G.dt * mu.v[l]) * sxz.v[l];
    }
    v4::st(R.a.f[SXX] + k, sxx);
    v4::st(R.a.f[SZZ] + k, szz);
    v4::st(R.a.f[SXZ] + k, sxz);
    v4::st(R.q[0] + k, qxx);
    v4::st(R.q[1] + k, qzz);
    v4::st(R.q[2] + k, qxz);
}

template <int M, bool FS>
__global__ void __launch_bounds__(kThreads, M <= 4 ? 4 : 3) rev_a(const Geo G, const Rev R)
{
    const Cell q(G);
    if (blockIdx.z == 0) adj_vel<M, FS>(G, R, q);
    else stress_rev<M, FS>(G, R, q);
}
template <int M, bool FS>
__global__ void __launch_bounds__(kThreads, M <= 4 ? 4 : 3) rev_b(const Geo G, const Rev R)
{
    const Cell q(G);
    if (blockIdx.z == 0) adj_str<M, FS>(G, R, q);
    else vel_rev<M, FS>(G, R, q);
}

// Fields [f0, f1) of the bands from a step slot.  Velocities add the rho image
// of the box cells outside the reverse box: the difference this makes.
__global__ void restore(const Geo G, const Rev R, const float* __restrict__ slot, int f0, int f1)
{
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)G.B * G.ns) return;
    const int b = (int)(e / G.ns), n = (int)(e - (long long)b * G.ns);
    const int c = __ldg(G.cells + n), z = c / G.P, x = c - z * G.P;
    const long long i = b * G.S + c;
    const bool img = f0 == VX && R.it > 1 && zbox(G, z) && xbox(G, x) &&
                     !(z >= G.rz0 && z < G.rz1 && x >= G.rx0 && x < G.rx1);
    float s = 0.f;
    for (int f = f0; f < f1; ++f) {
        const float v = __ldg(slot + (b * 5LL + f) * G.ns + n);
        if (img) s += R.a.f[f][i] * (v - R.f.f[f][i]);
        R.f.f[f][i] = v;
    }
    if (img) R.g[2][i] += s;
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

// the x profiles, zero past their ends
__global__ void prep_profiles(const float* a, const float* b, const float* ah, const float* bh, int nx, int len,
                              float* out)
{
    const float* in[4] = {a, b, ah, bh};
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 4 * len; e += gridDim.x * blockDim.x) {
        const int f = e / len, c = e - f * len - kGuard;
        out[e] = c >= 0 && c < nx ? in[f][c] : 0.f;
    }
}

// Gradients on the physical box, zero elsewhere, unpitched: (B, cells) for
// per-shot models, else the sum over shots in shot order.
struct Out {
    const float *vp, *vs, *rho;     // the caller's models
    float* g[3];                    // vp, vs, rho
};

__global__ void finalize(const Geo G, const Rev R, const Out o)
{
    const long long cells = (long long)G.nz * G.nx, n = (G.ms ? G.B : 1) * cells;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long b = e / cells;
        const int c = (int)(e - b * cells), z = c / G.nx, x = c - z * G.nx;
        float t[3] = {0.f, 0.f, 0.f};
        if (zbox(G, z) && xbox(G, x)) {
            const long long i = (long long)z * G.P + x;
            for (int j = 0; j < 3; ++j) {
                t[j] = R.g[j][b * G.S + i];
                for (int s = 1; !G.ms && s < G.B; ++s) t[j] += R.g[j][s * G.S + i];
            }
            const float rho = o.rho[e];
            t[0] = -2.f * rho * o.vp[e] * t[0] * G.dt;
            t[1] = -2.f * rho * o.vs[e] * t[1] * G.dt;
            t[2] = t[2] / rho;
        }
        for (int j = 0; j < 3; ++j) o.g[j][e] = t[j];
    }
}

// ------------------------------------------------------------------- host
struct Plan {
    Geo G;
    int nm;                         // model copies
    std::vector<int> cells;
};

// staggered first-derivative weights of half-width M (the closed form
// a_m = (-1)^(m+1) / (2m - 1) prod_{n != m} |(2n-1)^2 / ((2n-1)^2 - (2m-1)^2)|,
// reference operators/staggered.cuh), each rounded from the exact ratio
static void staggered_weights(int M, float* c)
{
    for (int m = 1; m <= M; ++m) {
        long long num = 1, den = 2 * m - 1;
        for (int n = 1; n <= M; ++n) {
            if (n == m) continue;
            const long long a = (long long)(2 * n - 1) * (2 * n - 1), q = (long long)(2 * m - 1) * (2 * m - 1);
            num *= a;
            den *= a > q ? a - q : q - a;
        }
        const double v = (double)num / (double)den;
        c[m] = (float)((m % 2 == 1) ? v : -v);
    }
}

static Plan make_plan(const sweep_elastic_desc* d, int mem_mode)
{
    SWEEP_REQUIRE(d != nullptr, "null descriptor");
    SWEEP_REQUIRE(d->M >= 1 && d->M <= MAXM, "elastic: spatial orders 2 to %d are built (got order %d)", 2 * MAXM,
                  2 * d->M);
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
    G.rz0 = G.z0 + (G.fs & 1 ? 0 : 1); G.rz1 = G.z1 - (G.fs & 2 ? 0 : 1);
    G.rx0 = G.x0 + (G.fs & 4 ? 0 : 1); G.rx1 = G.x1 - (G.fs & 8 ? 0 : 1);
    SWEEP_REQUIRE(G.z1 - G.z0 >= 2 && G.x1 - G.x0 >= 2, "elastic: the physical box must be at least 2 cells per axis");
    G.dt = d->dt; G.ihz = 1.f / d->dz; G.ihx = 1.f / d->dx;
    for (int k = 0; k <= MAXM; ++k) G.c[k] = 0.f;
    staggered_weights(M, G.c);
    G.az = d->az; G.bz = d->bz; G.azh = d->azh; G.bzh = d->bzh;
    const bool per_shot = d->model_stride != 0;
    SWEEP_REQUIRE(!per_shot || d->model_stride == cells, "elastic: model_stride must be 0 or nz * nx");
    G.ms = per_shot ? G.S : 0;
    pl.nm = per_shot ? G.B : 1;
    G.nsrc = d->nsrc; G.nrec = d->nrec; G.nsf = d->nsrc_fields; G.nrf = d->nrec_fields;
    for (int k = 0; k < 5; ++k) { G.sf[k] = d->src_fields[k]; G.rf[k] = d->rec_fields[k]; }
    G.src = d->src_loc; G.rec = d->rec_loc; G.wavelet = d->wavelet;
    // the boundary bands (boundary/strip.cuh:46-123: width M + 1 from M cells
    // outside the box, each band over the box tangentially; a band that would
    // leave the grid slides back inside)
    const int w = M + 1, off = -M;
    auto band_lo = [](int p0, int of, int wd, int n) { int s = p0 + of; if (s + wd > n) s = n - wd; return s < 0 ? 0 : s; };
    auto band_hi = [](int p1, int of, int wd, int n) { int e = p1 - of; if (e - wd < 0) e = wd; return e > n ? n : e; };
    const int ts = band_lo(G.z0, off, w, G.nz), be = band_hi(G.z1, off, w, G.nz);
    const int ls = band_lo(G.x0, off, w, G.nx), re = band_hi(G.x1, off, w, G.nx);
    // (a cell of two bands once: the x bands leave out what the z bands hold)
    auto in_zbands = [&](int z, int x) {
        return x >= G.x0 && x < G.x1 && ((z >= ts && z < ts + w) || (z >= be - w && z < be));
    };
    for (int z = ts; z < ts + w; ++z) for (int x = G.x0; x < G.x1; ++x) pl.cells.push_back(z * G.P + x);
    for (int z = be - w; z < be; ++z) for (int x = G.x0; x < G.x1; ++x) pl.cells.push_back(z * G.P + x);
    for (int z = G.z0; z < G.z1; ++z)
        for (int s : {ls, re - w})
            for (int x = s; x < s + w; ++x)
                if (!in_zbands(z, x)) pl.cells.push_back(z * G.P + x);
    G.ns = (int)pl.cells.size();
    // rows of a block: 32, or 8 where that would leave the GPU with less than
    // two blocks per SM
    G.nbx = (G.nx + 31) / 32;
    G.rows = (long long)G.nbx * G.B * ((G.nz + 31) / 32) >= 2 * 148 ? 32 : 8;
    return pl;
}

struct Ws {
    float *lam, *mu, *kv;
    float* xprof;                   // a, b, a_half, b_half along x, padded
    int* cells;
    float* f[5];
    float* m[2][NMEM];              // forward memories ([0]) / adjoint memories, double-buffered
    float* a[5];
    float* q[3];
    float* p[2];
    float* g[3];
    char *zero0, *zero1;
};

static int xprof_len(const Geo& G) { return G.P + 2 * kGuard; }

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
        for (float*& p : w.m[s]) p = c.take<float>(n);
    if (rev) {
        for (float*& p : w.a) p = c.take<float>(n);
        for (float*& p : w.q) p = c.take<float>(n);
        for (float*& p : w.g) p = c.take<float>(n);
    }
    c.take<char>(0);
    w.zero1 = c.base ? c.base + c.off : nullptr;
    if (rev)
        for (float*& p : w.p) p = c.take<float>(n);
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
    *tape_bytes = ((long long)pl.G.nt * slot_floats(pl) + 5LL * pl.G.B * pl.G.S) * 4;
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
    SWEEP_LAUNCH_CHECK();
    if (G.ns > 0)
        SWEEP_CUDA(cudaMemcpyAsync(w.cells, pl.cells.data(), sizeof(int) * G.ns, cudaMemcpyHostToDevice, st));
    SWEEP_CUDA(cudaMemsetAsync(w.zero0, 0, w.zero1 - w.zero0, st));
}

static dim3 grid_of(const Geo& G, unsigned parts)
{
    return dim3((unsigned)(G.nbx * G.B), (unsigned)((G.nz + G.rows - 1) / G.rows), parts);
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
        // the final state, (5, B, S)
        float* last = tp + (long long)G.nt * slot_floats(pl);
        const long long n = (long long)G.B * G.S;
        for (int f = 0; f < 5; ++f)
            SWEEP_CUDA(cudaMemcpyAsync(last + f * n, w.f[f], sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
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
    const long long n = (long long)G.B * G.S;
    for (int f = 0; f < 5; ++f)
        SWEEP_CUDA(cudaMemcpyAsync(w.f[f], last + f * n, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
    Rev R{};
    for (int k = 0; k < 5; ++k) { R.f.f[k] = w.f[k]; R.a.f[k] = w.a[k]; }
    for (int k = 0; k < 3; ++k) { R.q[k] = w.q[k]; R.g[k] = w.g[k]; }
    for (int k = 0; k < 2; ++k) R.p[k] = w.p[k];
    R.adj = adj;
    const dim3 grid = grid_of(G, 2), block(8, (unsigned)G.rows);
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
        rev_a<M, FS><<<grid, block, 0, s>>>(G, R);
        restore<<<bb, 256, 0, s>>>(G, R, prev, SXX, 5);
        rev_b<M, FS><<<grid, block, 0, s>>>(G, R);
        restore<<<bb, 256, 0, s>>>(G, R, prev, VX, SXX);
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
    case 4: CALL(4); break;           \
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
