// elastic3d_impl.cuh -- the body of the 3-D isotropic elastic path (see
// elastic3d.cu), compiled once per spatial order: the including file defines
// EL3D_M (the stencil half-width, 1..4) and EL3D_NS (the namespace of that
// order's kernels and entry points).  No include guard: one translation unit
// may include it for several orders.
#ifndef EL3D_M
#error "define EL3D_M (the stencil half-width) before including elastic3d_impl.cuh"
#endif
#ifndef EL3D_NS
#error "define EL3D_NS (the namespace of this order) before including elastic3d_impl.cuh"
#endif

#include "bands.cuh"
#include "vec4.cuh"

namespace sweep {
namespace EL3D_NS {

constexpr int M = EL3D_M;
constexpr int kGuard = 16;          // zero floats before and after a packed x profile
constexpr int kMaxGroup = 4;        // shots of an imaging thread, at most

// Staggered first-derivative weight k of order 2M (reference
// operators/staggered.cuh:146-147 order 4, 248-250 order 6, 351-354 order 8;
// order 2: the plain difference)
__host__ __device__ constexpr float wt(int k)
{
    return M == 1   ? 1.f
           : M == 2 ? (k == 1 ? 9.f / 8.f : -1.f / 24.f)
           : M == 3 ? (k == 1 ? 75.f / 64.f : k == 2 ? -25.f / 384.f : 3.f / 640.f)
                    : (k == 1 ? 1225.f / 1024.f : k == 2 ? -245.f / 3072.f : k == 3 ? 49.f / 5120.f : -5.f / 7168.f);
}

enum { VX, VY, VZ, SXX, SYY, SZZ, SXY, SXZ, SYZ, NFLD };
// memories per axis: x {vx, vy, vz, sxx, sxy, sxz}, y {vx, vy, vz, sxy, syy, syz},
// z {vx, vy, vz, sxz, syz, szz} -- the field differenced, the axis of the slab
enum { MX_VX, MX_VY, MX_VZ, MX_SXX, MX_SXY, MX_SXZ };
enum { MY_VX, MY_VY, MY_VZ, MY_SXY, MY_SYY, MY_SYZ };
enum { MZ_VX, MZ_VY, MZ_VZ, MZ_SXZ, MZ_SYZ, MZ_SZZ };

// CPML memories of the band of each axis: x (B, nz, ny, WX), y (B, nz, WY, P),
// z (B, WZ, ny, P); the x slab holds whole groups of four cells.
struct Slabs {
    float *x[6], *y[6], *z[6];
};

// the nine field pointers, passed by value to the point kernels
struct Fields {
    float* f[9];
};

// Boundary-strip storage of the boundary-saving tape.  fp32 and bf16 keep the
// strip set (B, 9, ns), each cell once; fp16 and int8 keep the reference's six
// faces per field -- bands M + 1 wide starting M cells outside the box (z faces
// across the box, y and x faces over its z range, so edge cells sit in two or
// three faces) -- each quantised per field and shot in blocks of kQB cells
// against the block's max |value| (reference boundarysaver.cu:207-460 face
// layout, boundary/strip.cuh:136-175 bands with offset -M and width M + 1,
// boundary/runtime.cuh:313-330 and boundarysaver.cu:925-1095 quantisation).
enum StripFmt { SF_F32 = 0, SF_F16 = 1, SF_BF16 = 2, SF_I8 = 3 };
constexpr int kQB = 256;
constexpr int BW = M + 1;           // face band width

struct StripStore {
    int fmt;                        // StripFmt
    int cells[6], blocks[6];        // per field and shot, per face (top, bottom, front, back, left, right)
    long long pay[6], scl[6];       // byte offsets of each face's codes (9, B, cells) and scales (9, B, blocks)
    long long step;                 // bytes of one step slot
};

struct Geo {
    int B, nz, ny, nx, nt;
    int P, SZ;                      // row pitch (y stride), z stride
    long long S;                    // shot stride
    int nbx, group, nslot;          // x blocks; shots per imaging thread, gradient slots
    int z0, z1, y0, y1, x0, x1;     // physical box
    int XL, XH, SYL, SYH, SZL, SZH;     // slab sides: x below XL or from XH on (multiples of 4); box edge + one cell
    int WX, WY, WZ;
    float dt, idx, idy, idz;
    // profiles a, b at integer and at half positions; the x ones are padded
    // with zeros (kGuard floats before their start and past their end)
    const float *az, *bz, *azh, *bzh, *ay, *by, *ayh, *byh, *ax, *bx, *axh, *bxh;
    int nsrc, nrec, nsf, nrf;
    int sf[9], rf[9];
    const int* src_loc;             // (B, nsrc, 3) runtime (x, y, z)
    const int* rec_loc;             // (B, nrec, 3)
    const float* wavelet;           // (B, nsrc, nt)
    long long ms;                   // model stride between shots (0 or S)
    const int* cells;               // strip cell offsets in a shot grid
    int ns;                         // strip cells
    int fst;                        // traction-free top face: the surface is row z0 (no pad above)
    StripStore st;
};

struct Models {
    const float *lam, *mu, *kv;     // kv = dt * (1 / rho), pitched
};

using v4::F4;

// Rows and planes of a block of 8 x 4 x 4 threads, compiled for eight blocks
// per SM (64 registers).  The gradient of the 2-shot 128^3 survey at order 8:
// 8 x 8 x 4 blocks at 3 / 4 per SM 81.8 / 79.3 ms, 8 x 4 x 4 ones at
// 6 / 8 per SM 79.6 / 78.1 ms.
constexpr int kBY = 4, kBZ = 4;
constexpr int kThreads = 8 * kBY * kBZ, kBlocks = 8;

// the thread's four cells x .. x + 3 of one row
struct Cell {
    int b, z, y, x, i;              // shot (group), coordinates of lane 0, offset in a shot
    bool grid, core;                // inside the grid; some lane is updated by the steps
    __device__ __forceinline__ explicit Cell(const Geo& G)
    {
        const int xb = blockIdx.x % G.nbx;
        b = blockIdx.x / G.nbx;
        x = 4 * (xb * 8 + threadIdx.x);
        y = blockIdx.y * kBY + threadIdx.y;
        z = blockIdx.z * kBZ + threadIdx.z;
        i = z * G.SZ + y * G.P + x;
        grid = x < G.nx && y < G.ny && z < G.nz;
        core = grid && x + 3 >= M && x < G.nx - M && y >= M && y < G.ny - M && z >= M && z < G.nz - M;
    }
    __device__ __forceinline__ bool lane(const Geo& G, int l) const { return x + l >= M && x + l < G.nx - M; }
};

// Staggered differences of the group at p (v4::diff with this order's
// weights): dp to the half cell above, dm to the half cell below.
struct Weights {
    float c[M + 1];
    __device__ __forceinline__ Weights()
    {
        c[0] = 0.f;
#pragma unroll
        for (int k = 1; k <= M; ++k) c[k] = wt(k);
    }
};
__device__ __forceinline__ F4 dp(const float* p, int s, float inv) { return v4::diff_col<M, true>(p, s, Weights().c, inv); }
__device__ __forceinline__ F4 dm(const float* p, int s, float inv) { return v4::diff_col<M, false>(p, s, Weights().c, inv); }
__device__ __forceinline__ F4 dpx(const float* p, float inv) { return v4::diff_row<M, true>(p, Weights().c, inv); }
__device__ __forceinline__ F4 dmx(const float* p, float inv) { return v4::diff_row<M, false>(p, Weights().c, inv); }

// ------------------------------------------------ traction-free top face
// The reference's 3-D image method (common/elastic_free_surface.cuh:723-952,
// elastic3d/kernels.cuh:360-372, 1421-1499): the rows above the surface row z0
// are air, read by a z-derivative as the image of the row mirrored about the
// surface (about z0 for integer fields, z0 - 1/2 for fields half a cell
// below it, negated for odd fields); the full stencil runs over the images.
// Only the M rows from the surface down reach the air; the adjoint is the
// exact transpose, so it differs from the plain one on the M + 1 rows from
// the surface down.  The surface row's sxx and syy take the Robertsson
// correction and its szz is zeroed.
template <bool FS, bool FWD>
__device__ __forceinline__ F4 dz_fs(const Geo& G, const float* p, int iz, bool odd, bool half)
{
    if (!FS || iz >= G.z0 + M) return FWD ? dp(p, G.SZ, G.idz) : dm(p, G.SZ, G.idz);
    auto at = [&](int k) {
        if (k >= G.z0) return v4::ldg(p + (k - iz) * G.SZ);
        const int m = half ? 2 * G.z0 - 1 - k : 2 * G.z0 - k;
        F4 v = v4::ldg(p + (m - iz) * G.SZ);
#pragma unroll
        for (int l = 0; l < 4; ++l) v.v[l] = odd ? -v.v[l] : v.v[l];
        return v;
    };
    return v4::diff<M, FWD>([&](int k) { return at(iz + k); }, Weights().c, G.idz);
}
// negated transpose of dz_fs (the plain one: D- for a D+ forward) of the rows
// row(k), k planes away
template <bool FS, bool FWD, class R>
__device__ __forceinline__ F4 adz_fs(const Geo& G, const R& row, int iz, bool odd, bool half)
{
    if (!FS || iz > G.z0 + M) return v4::diff<M, !FWD>(row, Weights().c, G.idz);
    const int top = G.z0, lo = half ? top - 1 : top;
    const float par = odd ? -1.f : 1.f;
    F4 g = v4::splat(0.f);
    auto add = [&](float w, int j) {
        const F4 r = row(j - iz);
#pragma unroll
        for (int l = 0; l < 4; ++l) g.v[l] += w * r.v[l];
    };
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
        const float w = wt(m + 1);
        const int jp = FWD ? iz + m : iz + m + 1;
        const int jm = FWD ? iz - m - 1 : iz - m;
        const int jg = FWD ? (half ? 2 * top - 1 + m - iz : 2 * top + m - iz)
                           : (half ? 2 * top + m - iz : 2 * top + m + 1 - iz);
        if (jp >= top) add(w, jp);
        if (jm >= top) add(-w, jm);
        if (iz > lo && jg >= top) add(w * par, jg);
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) g.v[l] *= G.idz;
    return g;
}

__device__ __forceinline__ bool in_core(const Geo& G, int ix, int iy, int iz)
{
    return ix >= M && ix < G.nx - M && iy >= M && iy < G.ny - M && iz >= M && iz < G.nz - M;
}
__device__ __forceinline__ bool in_box(const Geo& G, int ix, int iy, int iz)
{
    return ix >= G.x0 && ix < G.x1 && iy >= G.y0 && iy < G.y1 && iz >= G.z0 && iz < G.z1;
}
// slab offsets of a group (-1: no memory along that axis).  A profile is zero
// off its slab, and every cell with a nonzero one lies outside the box shrunk
// by one cell, where the reference's steps run their CPML branch.
__device__ __forceinline__ int xslab(const Geo& G, int x) { return x < G.XL ? x : x >= G.XH ? G.XL + x - G.XH : -1; }
__device__ __forceinline__ int yslab(const Geo& G, int y)
{
    return y < G.SYL ? y : y >= G.ny - G.SYH ? G.SYL + y - (G.ny - G.SYH) : -1;
}
__device__ __forceinline__ int zslab(const Geo& G, int z)
{
    return z < G.SZL ? z : z >= G.nz - G.SZH ? G.SZL + z - (G.nz - G.SZH) : -1;
}
__device__ __forceinline__ long long xsl(const Geo& G, int b, int z, int y, int x)
{
    const int s = xslab(G, x);
    return s < 0 ? -1 : (((long long)b * G.nz + z) * G.ny + y) * G.WX + s;
}
__device__ __forceinline__ long long ysl(const Geo& G, int b, int z, int y, int x)
{
    const int s = yslab(G, y);
    return s < 0 ? -1 : (((long long)b * G.nz + z) * G.WY + s) * G.P + x;
}
__device__ __forceinline__ long long zsl(const Geo& G, int b, int z, int y, int x)
{
    const int s = zslab(G, z);
    return s < 0 ? -1 : (((long long)b * G.WZ + s) * G.ny + y) * G.P + x;
}

// forward CPML memory update of derivative d along an axis: m = a m + b d,
// d += m, on the core's lanes
__device__ __forceinline__ void mem(float* m, const F4& a, const F4& b, F4& d, const bool (&on)[4])
{
    const F4 old = v4::ld(m);
    F4 v;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        v.v[l] = on[l] ? a.v[l] * old.v[l] + b.v[l] * d.v[l] : 0.f;
        d.v[l] += v.v[l];
    }
    v4::st(m, v);
}

// ------------------------------------------------------------------ forward
struct Fwd {
    Geo G;
    Models m;
    float* f[NFLD];
    Slabs mem;
};

// Nine derivatives of a staggered step by field and axis, through their
// memories; U names the field, X / Y / Z the derivative.
struct Nine {
    F4 xx, xy, xz, yx, yy, yz, zx, zy, zz;
};

template <bool FS>
__device__ __forceinline__ Nine stress_diffs(const Geo& G, float* const* f, long long k, int iz)
{
    Nine d;
    d.xx = dpx(f[SXX] + k, G.idx);
    d.xy = dm(f[SXY] + k, G.P, G.idy);
    d.xz = dz_fs<FS, false>(G, f[SXZ] + k, iz, true, true);
    d.yx = dmx(f[SXY] + k, G.idx);
    d.yy = dp(f[SYY] + k, G.P, G.idy);
    d.yz = dz_fs<FS, false>(G, f[SYZ] + k, iz, true, true);
    d.zx = dmx(f[SXZ] + k, G.idx);
    d.zy = dm(f[SYZ] + k, G.P, G.idy);
    d.zz = dz_fs<FS, true>(G, f[SZZ] + k, iz, true, false);
    return d;
}
// d(v_i) / d(j): xx = dvx/dx, xy = dvx/dy, ..., zz = dvz/dz
template <bool FS>
__device__ __forceinline__ Nine velocity_diffs(const Geo& G, float* const* f, long long k, int iz)
{
    Nine d;
    d.xx = dmx(f[VX] + k, G.idx);
    d.xy = dp(f[VX] + k, G.P, G.idy);
    d.xz = dz_fs<FS, true>(G, f[VX] + k, iz, false, false);
    d.yx = dpx(f[VY] + k, G.idx);
    d.yy = dm(f[VY] + k, G.P, G.idy);
    d.yz = dz_fs<FS, true>(G, f[VY] + k, iz, false, false);
    d.zx = dpx(f[VZ] + k, G.idx);
    d.zy = dp(f[VZ] + k, G.P, G.idy);
    d.zz = dz_fs<FS, false>(G, f[VZ] + k, iz, true, true);
    return d;
}

// Velocity and stress steps.  2-shot 128^3 survey at order 8 (9.5 M cells):
// 208 and 245 us, 350 and 428 us with one cell per thread; their field and
// memory traffic takes 100 and 117 us at the copy rate, the rest is the taps'
// L1 and L2 traffic.
template <bool FS>
__global__ void __launch_bounds__(kThreads, kBlocks) vel3(const Fwd A)
{
    const Geo& G = A.G;
    const Cell q(G);
    if (!q.core) return;
    const long long k = q.b * G.S + q.i;
    Nine d = stress_diffs<FS>(G, A.f, k, q.z);
    bool on[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) on[l] = q.lane(G, l);
    if (const long long o = xsl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::ldg(G.ax + q.x), b = v4::ldg(G.bx + q.x);
        mem(A.mem.x[MX_SXX] + o, v4::ldg(G.axh + q.x), v4::ldg(G.bxh + q.x), d.xx, on);
        mem(A.mem.x[MX_SXY] + o, a, b, d.yx, on);
        mem(A.mem.x[MX_SXZ] + o, a, b, d.zx, on);
    }
    if (const long long o = ysl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::splat(__ldg(G.ay + q.y)), b = v4::splat(__ldg(G.by + q.y));
        mem(A.mem.y[MY_SXY] + o, a, b, d.xy, on);
        mem(A.mem.y[MY_SYY] + o, v4::splat(__ldg(G.ayh + q.y)), v4::splat(__ldg(G.byh + q.y)), d.yy, on);
        mem(A.mem.y[MY_SYZ] + o, a, b, d.zy, on);
    }
    if (const long long o = zsl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::splat(__ldg(G.az + q.z)), b = v4::splat(__ldg(G.bz + q.z));
        mem(A.mem.z[MZ_SXZ] + o, a, b, d.xz, on);
        mem(A.mem.z[MZ_SYZ] + o, a, b, d.yz, on);
        mem(A.mem.z[MZ_SZZ] + o, v4::splat(__ldg(G.azh + q.z)), v4::splat(__ldg(G.bzh + q.z)), d.zz, on);
    }
    const F4 kv = v4::ldg(A.m.kv + q.b * G.ms + q.i);
    F4 vx = v4::ld(A.f[VX] + k), vy = v4::ld(A.f[VY] + k), vz = v4::ld(A.f[VZ] + k);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (!on[l]) continue;
        vx.v[l] += kv.v[l] * (d.xx.v[l] + d.xy.v[l] + d.xz.v[l]);
        vy.v[l] += kv.v[l] * (d.yx.v[l] + d.yy.v[l] + d.yz.v[l]);
        vz.v[l] += kv.v[l] * (d.zx.v[l] + d.zy.v[l] + d.zz.v[l]);
    }
    v4::st(A.f[VX] + k, vx);
    v4::st(A.f[VY] + k, vy);
    v4::st(A.f[VZ] + k, vz);
}

// the six stresses of the group at k: s += sgn dt C : d on the lanes `on`
__device__ __forceinline__ void stress_update(const Geo& G, float* const* f, long long k, const Nine& d, const F4& lam,
                                              const F4& mu, float sdt, const bool (&on)[4], bool surf)
{
    auto update = [&](int fl, auto value) {
        F4 s = v4::ld(f[fl] + k);
#pragma unroll
        for (int l = 0; l < 4; ++l)
            if (on[l]) s.v[l] = value(l, s.v[l]);
        v4::st(f[fl] + k, s);
    };
    auto div = [&](int l) { return d.xx.v[l] + d.yy.v[l] + d.zz.v[l]; };
    // surface row: Robertsson sxx / syy (forward only), then szz = 0
    auto rob = [&](int l) {
        return -G.dt * lam.v[l] * (lam.v[l] / (lam.v[l] + 2.f * mu.v[l]) * (d.xx.v[l] + d.yy.v[l]) + d.zz.v[l]);
    };
    update(SXX, [&](int l, float s) {
        s += sdt * (lam.v[l] * div(l) + 2.f * mu.v[l] * d.xx.v[l]);
        return surf ? s + rob(l) : s;
    });
    update(SYY, [&](int l, float s) {
        s += sdt * (lam.v[l] * div(l) + 2.f * mu.v[l] * d.yy.v[l]);
        return surf ? s + rob(l) : s;
    });
    update(SZZ, [&](int l, float s) {
        return surf ? 0.f : s + sdt * (lam.v[l] * div(l) + 2.f * mu.v[l] * d.zz.v[l]);
    });
    update(SXY, [&](int l, float s) { return s + sdt * mu.v[l] * (d.xy.v[l] + d.yx.v[l]); });
    update(SXZ, [&](int l, float s) { return s + sdt * mu.v[l] * (d.xz.v[l] + d.zx.v[l]); });
    update(SYZ, [&](int l, float s) { return s + sdt * mu.v[l] * (d.yz.v[l] + d.zy.v[l]); });
}

template <bool FS>
__global__ void __launch_bounds__(kThreads, kBlocks) str3(const Fwd A)
{
    const Geo& G = A.G;
    const Cell q(G);
    if (!q.core) return;
    const long long k = q.b * G.S + q.i, mi = q.b * G.ms + q.i;
    Nine d = velocity_diffs<FS>(G, A.f, k, q.z);
    bool on[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) on[l] = q.lane(G, l);
    if (const long long o = xsl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::ldg(G.axh + q.x), b = v4::ldg(G.bxh + q.x);
        mem(A.mem.x[MX_VX] + o, v4::ldg(G.ax + q.x), v4::ldg(G.bx + q.x), d.xx, on);
        mem(A.mem.x[MX_VY] + o, a, b, d.yx, on);
        mem(A.mem.x[MX_VZ] + o, a, b, d.zx, on);
    }
    if (const long long o = ysl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::splat(__ldg(G.ayh + q.y)), b = v4::splat(__ldg(G.byh + q.y));
        mem(A.mem.y[MY_VX] + o, a, b, d.xy, on);
        mem(A.mem.y[MY_VY] + o, v4::splat(__ldg(G.ay + q.y)), v4::splat(__ldg(G.by + q.y)), d.yy, on);
        mem(A.mem.y[MY_VZ] + o, a, b, d.zy, on);
    }
    if (const long long o = zsl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::splat(__ldg(G.azh + q.z)), b = v4::splat(__ldg(G.bzh + q.z));
        mem(A.mem.z[MZ_VX] + o, a, b, d.xz, on);
        mem(A.mem.z[MZ_VY] + o, a, b, d.yz, on);
        mem(A.mem.z[MZ_VZ] + o, v4::splat(__ldg(G.az + q.z)), v4::splat(__ldg(G.bz + q.z)), d.zz, on);
    }
    stress_update(G, A.f, k, d, v4::ldg(A.m.lam + mi), v4::ldg(A.m.mu + mi), G.dt, on, FS && q.z == G.z0);
}

// Source injection of step it with sign (+1 forward, -1 taking the forward
// source back out in the reverse) into every source field; one block per shot.
__global__ void src3(const Geo G, const Fields F, int it, float sign)
{
    float* const* f = F.f;
    const int b = blockIdx.x;
    for (int s = threadIdx.x; s < G.nsrc; s += blockDim.x) {
        const int* l = G.src_loc + ((long long)b * G.nsrc + s) * 3;
        if (l[0] < 0 || l[0] >= G.nx || l[1] < 0 || l[1] >= G.ny || l[2] < 0 || l[2] >= G.nz) continue;
        const long long i = b * G.S + (long long)l[2] * G.SZ + l[1] * G.P + l[0];
        const float w = sign * G.wavelet[((long long)b * G.nsrc + s) * G.nt + it];
        for (int k = 0; k < G.nsf; ++k) atomicAdd(f[G.sf[k]] + i, w);
    }
}

// receivers: one thread per (shot, receiver), grid (receiver blocks, shots)
__global__ void rec3(const Geo G, const Fields F, float* record, int it)
{
    float* const* f = F.f;
    const int b = blockIdx.y;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < G.nrec; r += gridDim.x * blockDim.x) {
        const int* l = G.rec_loc + ((long long)b * G.nrec + r) * 3;
        if (l[0] < 0 || l[0] >= G.nx || l[1] < 0 || l[1] >= G.ny || l[2] < 0 || l[2] >= G.nz) continue;
        const long long i = b * G.S + (long long)l[2] * G.SZ + l[1] * G.P + l[0];
        float* out = record + (((long long)b * G.nt + it) * G.nrec + r) * G.nrf;
        for (int k = 0; k < G.nrf; ++k) out[k] = f[G.rf[k]][i];
    }
}

// Face f cell idx (of one field and shot) of the scaled formats -> grid cell:
// z faces (band, box y, box x), y faces (box z, band, box x), x faces (box z,
// box y, band).
__device__ __forceinline__ void face_cell(const Geo& G, int f, int idx, int& iz, int& iy, int& ix)
{
    const int bx = G.x1 - G.x0, by = G.y1 - G.y0;
    if (f < 2) {
        ix = G.x0 + idx % bx; idx /= bx;
        iy = G.y0 + idx % by;
        iz = (f == 0 ? G.z0 - M : G.z1 - 1) + idx / by;
    } else if (f < 4) {
        ix = G.x0 + idx % bx; idx /= bx;
        iy = (f == 2 ? G.y0 - M : G.y1 - 1) + idx % BW;
        iz = G.z0 + idx / BW;
    } else {
        ix = (f == 4 ? G.x0 - M : G.x1 - 1) + idx % BW; idx /= BW;
        iy = G.y0 + idx % by;
        iz = G.z0 + idx / by;
    }
}

// The face a scaled-format restore reads strip cell (iz, iy, ix) from: the
// last of the faces holding it in the reference's write order (top, bottom,
// front, back, left, right), and the cell's index in that face.
__device__ __forceinline__ int face_index(const Geo& G, int iz, int iy, int ix, int& f)
{
    const int bx = G.x1 - G.x0, by = G.y1 - G.y0;
    const bool zin = iz >= G.z0 && iz < G.z1, yin = iy >= G.y0 && iy < G.y1, xin = ix >= G.x0 && ix < G.x1;
    if (zin && yin && ix >= G.x1 - 1 && ix < G.x1 - 1 + BW) { f = 5; return ((iz - G.z0) * by + iy - G.y0) * BW + ix - (G.x1 - 1); }
    if (zin && yin && ix >= G.x0 - M && ix <= G.x0) { f = 4; return ((iz - G.z0) * by + iy - G.y0) * BW + ix - (G.x0 - M); }
    if (zin && xin && iy >= G.y1 - 1 && iy < G.y1 - 1 + BW) { f = 3; return ((iz - G.z0) * BW + iy - (G.y1 - 1)) * bx + ix - G.x0; }
    if (zin && xin && iy >= G.y0 - M && iy <= G.y0) { f = 2; return ((iz - G.z0) * BW + iy - (G.y0 - M)) * bx + ix - G.x0; }
    if (iz >= G.z1 - 1) { f = 1; return ((iz - (G.z1 - 1)) * by + iy - G.y0) * bx + ix - G.x0; }
    f = 0;
    return ((iz - (G.z0 - M)) * by + iy - G.y0) * bx + ix - G.x0;
}

// a[f] of a per-face parameter array without a local-memory copy of the array
template <class T>
__device__ __forceinline__ T pick6(const T (&a)[6], int f)
{
    T v = a[0];
#pragma unroll
    for (int k = 1; k < 6; ++k)
        if (f == k) v = a[k];
    return v;
}

// Saved value of field fl at grid cell c of shot b in a scaled-format slot
// (dequantised as the reference does: fp16 code x scale; int8
// (code - 128) x scale / 127).
__device__ __forceinline__ float face_val(const Geo& G, const void* slot, int fl, int b, int c)
{
    const int ix = c % G.P, r = c / G.P, iy = r % G.ny, iz = r / G.ny;
    int f;
    const int i = face_index(G, iz, iy, ix, f);
    const StripStore& S = G.st;
    const char* base = static_cast<const char*>(slot);
    const long long row = (long long)fl * G.B + b;
    const float scale = reinterpret_cast<const float*>(base + pick6(S.scl, f))[row * pick6(S.blocks, f) + i / kQB];
    const long long q = row * pick6(S.cells, f) + i;
    const char* pay = base + pick6(S.pay, f);
    if (S.fmt == SF_F16) return __half2float(reinterpret_cast<const __half*>(pay)[q]) * scale;
    return ((float)reinterpret_cast<const uint8_t*>(pay)[q] - 128.0f) * (scale * (1.0f / 127.0f));
}

// Strip save (restore = 0) of fields [f0, f1) into / restore out of one step
// slot in format fmt: fp32 / bf16 slots hold the strip set (B, 9, ns); a
// scaled slot (written by quant3) is read from the field's faces.
__global__ void strips3(const Geo G, const Fields F, void* slot, int fmt, int f0, int f1, int restore)
{
    float* const* f = F.f;
    const long long n = (long long)G.B * G.ns;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int b = (int)(e / G.ns), k = (int)(e - (long long)b * G.ns);
        const int c = G.cells[k];
        const long long i = b * G.S + c;
        for (int fl = f0; fl < f1; ++fl) {
            const long long t = ((long long)b * NFLD + fl) * G.ns + k;
            if (fmt == SF_F32) {
                float* p = static_cast<float*>(slot) + t;
                if (restore) f[fl][i] = *p;
                else *p = f[fl][i];
            } else if (fmt == SF_BF16) {
                __nv_bfloat16* p = static_cast<__nv_bfloat16*>(slot) + t;
                if (restore) f[fl][i] = __bfloat162float(*p);
                else *p = __float2bfloat16(f[fl][i]);
            } else if (restore) {
                f[fl][i] = face_val(G, slot, fl, b, c);
            }
        }
    }
}

// One step's nine fields into the scaled faces of a step slot: one CTA per
// (field, shot, face, block of kQB cells) -- the block's max |value| (its
// scale), then the codes (reference boundarysaver.cu:957-990, 1040-1075: int8
// round(v 127 / max) + 128 clamped to [0, 255]; fp16 v (1 / max)).
__global__ void __launch_bounds__(kQB) quant3(const Geo G, const Fields F, void* slot)
{
    const StripStore& S = G.st;
    int per = 0;
#pragma unroll
    for (int f = 0; f < 6; ++f) per += S.blocks[f];
    const int row = blockIdx.x / per;                 // field * B + shot
    const int fl = row / G.B, b = row - fl * G.B;
    int j = blockIdx.x - row * per, f = 0;
#pragma unroll
    for (int k = 0; k < 5; ++k)
        if (f == k && j >= S.blocks[k]) { j -= S.blocks[k]; f = k + 1; }
    const int idx = j * kQB + threadIdx.x;
    const int cells = pick6(S.cells, f), blocks = pick6(S.blocks, f);
    const bool in = idx < cells;
    float v = 0.f;
    if (in) {
        int iz, iy, ix;
        face_cell(G, f, idx, iz, iy, ix);
        v = F.f[fl][b * G.S + (long long)iz * G.SZ + iy * G.P + ix];
    }
    float m = fabsf(v);
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float wmax[kQB / 32];
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
    __syncthreads();
    m = wmax[0];
#pragma unroll
    for (int i = 1; i < kQB / 32; ++i) m = fmaxf(m, wmax[i]);
    char* base = static_cast<char*>(slot);
    if (threadIdx.x == 0) reinterpret_cast<float*>(base + pick6(S.scl, f))[(long long)row * blocks + j] = m;
    if (!in) return;
    const long long q = (long long)row * cells + idx;
    char* pay = base + pick6(S.pay, f);
    if (S.fmt == SF_F16) {
        const float inv = m > 0.0f ? 1.0f / m : 0.0f;
        reinterpret_cast<__half*>(pay)[q] = __float2half(v * inv);
    } else {
        const float qs = m > 0.0f ? 127.0f / m : 0.0f;
        int c = __float2int_rn(v * qs) + 128;
        c = c < 0 ? 0 : (c > 255 ? 255 : c);
        reinterpret_cast<uint8_t*>(pay)[q] = (uint8_t)c;
    }
}

// ------------------------------------------------------------------ reverse
//
// Per step: residuals and source, `stress_rev` (stress reconstruction and the
// vp / vs image), the stress strips, `adj_vel` (the stress step's transpose
// into the adjoint velocities), `adj_str` (the velocity step's transpose into
// the adjoint stresses), `vel_rev` (velocity reconstruction and the rho
// image), the velocity strips.  `adj_str` leaves q = dt C lambda_s beside the
// adjoint stresses it writes (six fields; the reference's nine differ by the
// CPML memory alone), and the adjoint velocities are held as p = kv lambda_v, so
// no pass of its own prepares them and the stencils read one field per tap; a
// band's taps add the adjoint memory, which is therefore double-buffered.
// (q and p formed at every tap from lambda, the stiffness and 1 / rho instead:
// 666 + 556 us a step against 337 + 283 on the 2-shot 128^3 survey at order 8.)
// The rho image of step `it` is lambda_v . (v(it - 1) - v(it)): inside, minus
// kv lambda_v . div s (what the reconstruction takes back), on the box's
// outermost layer the difference of the restored strips (`restore_velocity`).
// The image of the update of step 1 is left out, as by the reference's
// staggered reverse.  All four kernels wait for loads (DRAM at 28 to 45 %); the
// bound of 64 registers makes adj_vel spill 428 bytes, stress_rev 368 and
// vel_rev 160, a quarter to two fifths of their L1 traffic.
struct Rev {
    Geo G;
    Models m;
    float* f[NFLD];      // reconstructed forward fields
    float* a[3];         // adjoint sxx, syy, szz
    float* q[6];         // dt C lambda_s: xx, yy, zz, xy, xz, yz
    float* p[3];         // kv lambda_v
    Slabs ai, ao;        // adjoint memories: read, written
    float* g[3];         // slots of a shot group: gl, dt mu (gm - 2 gl) and the rho image (times rho)
    const float* adj;    // (B, nt, nrec, nrf)
    int it;
};

// dt C s of the diagonal; on a surface row the transposes of the corrected
// updates, with szz counting as zero
__device__ __forceinline__ void stiff(float dt, float lam, float mu, float x, float y, float z, bool surf, float (&q)[3])
{
    const float l2m = lam + 2.f * mu;
    if (surf) {
        const float c1 = 4.f * mu * (lam + mu) / l2m, c2 = 2.f * lam * mu / l2m;
        q[0] = dt * (c1 * x + c2 * y);
        q[1] = dt * (c2 * x + c1 * y);
        q[2] = 0.f;
    } else {
        q[0] = dt * (l2m * x + lam * y + lam * z);
        q[1] = dt * (lam * x + l2m * y + lam * z);
        q[2] = dt * (lam * x + lam * y + l2m * z);
    }
}

__global__ void res3(Rev A)
{
    const Geo& G = A.G;
    const int b = blockIdx.y;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < G.nrec; r += gridDim.x * blockDim.x) {
        const int* l = G.rec_loc + ((long long)b * G.nrec + r) * 3;
        if (l[0] < 0 || l[0] >= G.nx || l[1] < 0 || l[1] >= G.ny || l[2] < 0 || l[2] >= G.nz) continue;
        const long long i = b * G.S + (long long)l[2] * G.SZ + l[1] * G.P + l[0];
        const float* res = A.adj + (((long long)b * G.nt + A.it) * G.nrec + r) * G.nrf;
        for (int k = 0; k < G.nrf; ++k) {
            const int fl = G.rf[k];
            const float v = fl >= SXX ? -res[k] : res[k];
            if (fl < SXX) { atomicAdd(A.p[fl] + i, A.m.kv[b * G.ms + i - b * G.S] * v); continue; }
            const float lam = A.m.lam[b * G.ms + i - b * G.S], mu = A.m.mu[b * G.ms + i - b * G.S];
            if (fl >= SXY) { atomicAdd(A.q[fl - SXX] + i, G.dt * mu * v); continue; }
            atomicAdd(A.a[fl - SXX] + i, v);
            // and what it adds to q
            const float x = fl == SXX ? v : 0.f, y = fl == SYY ? v : 0.f, z = fl == SZZ ? v : 0.f;
            float q3[3];
            stiff(G.dt, lam, mu, x, y, z, G.fst && l[2] == G.z0, q3);
            for (int j = 0; j < 3; ++j)
                if (q3[j] != 0.f) atomicAdd(A.q[j] + i, q3[j]);
        }
    }
}

__device__ __forceinline__ void add4(float* p, const F4& a)
{
    F4 t = v4::ld(p);
#pragma unroll
    for (int l = 0; l < 4; ++l) t.v[l] += a.v[l];
    v4::st(p, t);
}

// Stress reconstruction on the box minus one cell, and on the box the image:
// with gl, gm the derivatives of the misfit by lambda and mu (up to -dt),
// grad vp = -2 rho vp dt gl, grad vs = -2 rho vs dt (gm - 2 gl), and the
// stiffness part of rho times grad rho, -dt (gl (lam + 2 mu) + (gm - 2 gl) mu).
// The shear part of dt mu gm is the shears of q times their strains.
template <bool FS>
__global__ void __launch_bounds__(kThreads, kBlocks) stress_rev(const Rev A)
{
    const Geo& G = A.G;
    const Cell q(G);
    if (!q.core || q.x + 3 < G.x0 || q.x >= G.x1 || q.y < G.y0 || q.y >= G.y1 || q.z < G.z0 || q.z >= G.z1) return;
    const bool inner = q.y > G.y0 && q.y < G.y1 - 1 && q.z > G.z0 && q.z < G.z1 - 1, surf = FS && q.z == G.z0;
    bool box[4], on[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        box[l] = q.x + l >= G.x0 && q.x + l < G.x1;
        on[l] = inner && q.x + l > G.x0 && q.x + l < G.x1 - 1;
    }
    F4 sl = v4::splat(0.f), sm = sl, sr = sl;
    const int b1 = min((q.b + 1) * G.group, G.B);
    for (int b = q.b * G.group; b < b1; ++b) {
        const long long k = b * G.S + q.i, mi = b * G.ms + q.i;
        const Nine d = velocity_diffs<FS>(G, A.f, k, q.z);
        const F4 lam = v4::ldg(A.m.lam + mi), mu = v4::ldg(A.m.mu + mi);
        const F4 bxx = v4::ldg(A.a[0] + k), byy = v4::ldg(A.a[1] + k), bzz = v4::ldg(A.a[2] + k);
        const F4 qxy = v4::ldg(A.q[3] + k), qxz = v4::ldg(A.q[4] + k), qyz = v4::ldg(A.q[5] + k);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            if (!box[l]) continue;
            const float shear = qxz.v[l] * (d.xz.v[l] + d.zx.v[l]) + qxy.v[l] * (d.xy.v[l] + d.yx.v[l]) +
                                qyz.v[l] * (d.yz.v[l] + d.zy.v[l]);
            const float l2m = lam.v[l] + 2.f * mu.v[l];
            float gl, gm;
            if (surf) {
                // the surface row's corrected sxx / syy updates (kernels.cuh:1440-1452)
                const float r = mu.v[l] / l2m, w = lam.v[l] / l2m;
                const float dcl = 4.f * r * r, dcm = 4.f * (1.f - 2.f * r + 2.f * r * r), dc2m = 2.f * w * w;
                gl = dcl * (bxx.v[l] + byy.v[l]) * (d.xx.v[l] + d.yy.v[l]);
                gm = bxx.v[l] * (dcm * d.xx.v[l] + dc2m * d.yy.v[l]) +
                     byy.v[l] * (dc2m * d.xx.v[l] + dcm * d.yy.v[l]);
            } else {
                gl = (bxx.v[l] + byy.v[l] + bzz.v[l]) * (d.xx.v[l] + d.yy.v[l] + d.zz.v[l]);
                gm = 2.f * (bxx.v[l] * d.xx.v[l] + byy.v[l] * d.yy.v[l] + bzz.v[l] * d.zz.v[l]);
            }
            const float gs = (G.dt * mu.v[l]) * (gm - 2.f * gl) + shear;
            sl.v[l] += gl;
            sm.v[l] += gs;
            sr.v[l] -= (G.dt * gl) * l2m + gs;
        }
        if (inner) stress_update(G, A.f, k, d, lam, mu, -G.dt, on, false);
    }
    const long long o = q.b * G.S + q.i;
    add4(A.g[0] + o, sl);
    add4(A.g[1] + o, sm);
    add4(A.g[2] + o, sr);
}

// Velocity reconstruction on the box minus one cell with its rho image.
template <bool FS>
__global__ void __launch_bounds__(kThreads, kBlocks) vel_rev(const Rev A)
{
    const Geo& G = A.G;
    const Cell q(G);
    if (!q.core || q.x + 3 <= G.x0 || q.x >= G.x1 - 1 || q.y <= G.y0 || q.y >= G.y1 - 1 || q.z <= G.z0 || q.z >= G.z1 - 1)
        return;
    F4 sr = v4::splat(0.f);
    const int b1 = min((q.b + 1) * G.group, G.B);
    for (int b = q.b * G.group; b < b1; ++b) {
        const long long k = b * G.S + q.i;
        const Nine d = stress_diffs<FS>(G, A.f, k, q.z);
        const F4 kv = v4::ldg(A.m.kv + b * G.ms + q.i);
        const F4 px = v4::ldg(A.p[VX] + k), py = v4::ldg(A.p[VY] + k), pz = v4::ldg(A.p[VZ] + k);
        F4 vx = v4::ld(A.f[VX] + k), vy = v4::ld(A.f[VY] + k), vz = v4::ld(A.f[VZ] + k);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            if (!(q.x + l > G.x0 && q.x + l < G.x1 - 1)) continue;
            const float gx = d.xx.v[l] + d.xy.v[l] + d.xz.v[l];
            const float gy = d.yx.v[l] + d.yy.v[l] + d.yz.v[l];
            const float gz = d.zx.v[l] + d.zy.v[l] + d.zz.v[l];
            vx.v[l] -= kv.v[l] * gx;
            vy.v[l] -= kv.v[l] * gy;
            vz.v[l] -= kv.v[l] * gz;
            sr.v[l] -= px.v[l] * gx + py.v[l] * gy + pz.v[l] * gz;
        }
        v4::st(A.f[VX] + k, vx);
        v4::st(A.f[VY] + k, vy);
        v4::st(A.f[VZ] + k, vz);
    }
    if (A.it > 1) add4(A.g[2] + q.b * G.S + q.i, sr);
}

// Velocity strips from a step slot; the rho image of the box's outermost
// layer is the difference this makes.  There the thread of a group's first
// shot walks the group's shots, so that the sum does not depend on timing.
__global__ void restore_velocity(const Rev A, const void* slot, int fmt)
{
    const Geo& G = A.G;
    const long long n = (long long)G.B * G.ns;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int b0 = (int)(e / G.ns), k = (int)(e - (long long)b0 * G.ns);
        const int c = G.cells[k];
        const int ix = c % G.P, r = c / G.P;
        const bool img = A.it > 1 && in_box(G, ix, r % G.ny, r / G.ny);
        if (img && b0 % G.group) continue;
        const int b1 = img ? min(b0 + G.group, G.B) : b0 + 1;
        float s = 0.f;
        for (int b = b0; b < b1; ++b) {
            const long long i = b * G.S + c;
            for (int fl = VX; fl <= VZ; ++fl) {
                const long long t = ((long long)b * NFLD + fl) * G.ns + k;
                const float v = fmt == SF_F32    ? static_cast<const float*>(slot)[t]
                                : fmt == SF_BF16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(slot)[t])
                                                 : face_val(G, slot, fl, b, c);
                if (img) s += A.p[fl][i] / A.m.kv[b * G.ms + c] * (v - A.f[fl][i]);
                A.f[fl][i] = v;
            }
        }
        if (img) A.g[2][b0 / G.group * G.S + c] += s;
    }
}

// a q / p entry through its adjoint CPML memory w: bar + b (w + bar); the
// owner's next memory is a (w + bar)
__device__ __forceinline__ F4 through(const F4& bar, const F4& b, const F4& w)
{
    F4 t;
#pragma unroll
    for (int l = 0; l < 4; ++l) t.v[l] = bar.v[l] + b.v[l] * (w.v[l] + bar.v[l]);
    return t;
}
__device__ __forceinline__ void keep(const float* wi, float* wo, const F4& a, const F4& bar)
{
    const F4 w = v4::ldg(wi);
    F4 t;
#pragma unroll
    for (int l = 0; l < 4; ++l) t.v[l] = a.v[l] * (w.v[l] + bar.v[l]);
    v4::st(wo, t);
}
// A transpose's stencil along an axis of field u with the adjoint memory m of
// its taps in the band (profile prof).  Off the band's reach it is the plain
// one; within it every tap takes its memory, those off the slab at a clamped
// place and with the profile's zero, so that a thread's loads leave together
// (a test per tap serialised them: 709 + 438 us a step in the two transposes
// of the 2-shot 128^3 survey at order 8, 377 + 345 us this way).
template <bool PLUS>
__device__ __forceinline__ F4 adj_x(const Geo& G, const Cell& q, const float* u, const float* m, const float* prof)
{
    using S = v4::Span<M, PLUS>;
    float w[S::N];
    v4::window<S::LO, S::HI>(u, w);
    const int lo = q.x - 4 * S::LO, hi = min(q.x + 4 * S::HI, (G.nx - 1) / 4 * 4);
    if (lo < G.XL || hi >= G.XH) {
        const float* row = m + (((long long)q.b * G.nz + q.z) * G.ny + q.y) * G.WX;
#pragma unroll
        for (int j = -S::LO; j <= S::HI; ++j) {
            const int x = min(max(q.x + 4 * j, 0), hi), s = max(xslab(G, x), 0);
            const F4 b = v4::ldg(prof + q.x + 4 * j), t = v4::ldg(row + s);
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                float& e = w[4 * (j + S::LO) + l];
                e = e + b.v[l] * (t.v[l] + e);
            }
        }
    }
    return v4::diff_x<M, PLUS, S::O>(w, Weights().c, G.idx);
}
template <bool PLUS>
__device__ __forceinline__ F4 adj_y(const Geo& G, const Cell& q, const float* u, const float* m, const float* prof)
{
    if (yslab(G, q.y - M) < 0 && yslab(G, q.y + M) < 0) return v4::diff_col<M, PLUS>(u, G.P, Weights().c, G.idy);
    const float* col = m + ((long long)q.b * G.nz + q.z) * G.WY * G.P + q.x;
    return v4::diff<M, PLUS>(
        [&](int j) {
            return through(v4::ldg(u + j * G.P), v4::splat(__ldg(prof + q.y + j)),
                           v4::ldg(col + (long long)max(yslab(G, q.y + j), 0) * G.P));
        },
        Weights().c, G.idy);
}
template <bool FS, bool FWD>
__device__ __forceinline__ F4 adj_z(const Geo& G, const Cell& q, const float* u, const float* m, const float* prof,
                                    bool odd, bool half)
{
    const bool surf = FS && q.z <= G.z0 + M;
    if (!surf && zslab(G, q.z - M) < 0 && zslab(G, q.z + M) < 0)
        return v4::diff_col<M, !FWD>(u, G.SZ, Weights().c, G.idz);
    const float* col = m + ((long long)q.b * G.WZ * G.ny + q.y) * G.P + q.x;
    return adz_fs<FS, FWD>(
        G,
        [&](int j) {
            return through(v4::ldg(u + j * G.SZ), v4::splat(__ldg(prof + q.z + j)),
                           v4::ldg(col + (long long)max(zslab(G, q.z + j), 0) * G.ny * G.P));
        },
        q.z, odd, half);
}

// The stress step's transpose: lambda_v += D(q), held as p, on the core, q
// through the memories of the velocities' derivatives.
template <bool FS>
__global__ void __launch_bounds__(kThreads, kBlocks) adj_vel(const Rev A)
{
    const Geo& G = A.G;
    const Cell q(G);
    if (!q.grid) return;
    const long long k = q.b * G.S + q.i;
    const float *qxx = A.q[0] + k, *qyy = A.q[1] + k, *qzz = A.q[2] + k, *qxy = A.q[3] + k, *qxz = A.q[4] + k,
                *qyz = A.q[5] + k;
    // the next memories of this group
    if (const long long o = xsl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::ldg(G.axh + q.x);
        keep(A.ai.x[MX_VX] + o, A.ao.x[MX_VX] + o, v4::ldg(G.ax + q.x), v4::ldg(qxx));
        keep(A.ai.x[MX_VY] + o, A.ao.x[MX_VY] + o, a, v4::ldg(qxy));
        keep(A.ai.x[MX_VZ] + o, A.ao.x[MX_VZ] + o, a, v4::ldg(qxz));
    }
    if (const long long o = ysl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::splat(__ldg(G.ayh + q.y));
        keep(A.ai.y[MY_VX] + o, A.ao.y[MY_VX] + o, a, v4::ldg(qxy));
        keep(A.ai.y[MY_VY] + o, A.ao.y[MY_VY] + o, v4::splat(__ldg(G.ay + q.y)), v4::ldg(qyy));
        keep(A.ai.y[MY_VZ] + o, A.ao.y[MY_VZ] + o, a, v4::ldg(qyz));
    }
    if (const long long o = zsl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::splat(__ldg(G.azh + q.z));
        keep(A.ai.z[MZ_VX] + o, A.ao.z[MZ_VX] + o, a, v4::ldg(qxz));
        keep(A.ai.z[MZ_VY] + o, A.ao.z[MZ_VY] + o, a, v4::ldg(qyz));
        keep(A.ai.z[MZ_VZ] + o, A.ao.z[MZ_VZ] + o, v4::splat(__ldg(G.az + q.z)), v4::ldg(qzz));
    }
    if (!q.core) return;
    const F4 kv = v4::ldg(A.m.kv + q.b * G.ms + q.i);
    auto put = [&](int fl, const F4& a, const F4& b, const F4& c) {
        F4 p = v4::ld(A.p[fl] + k);
#pragma unroll
        for (int l = 0; l < 4; ++l)
            if (q.lane(G, l)) p.v[l] += kv.v[l] * (a.v[l] + b.v[l] + c.v[l]);
        v4::st(A.p[fl] + k, p);
    };
    put(VX, adj_x<true>(G, q, qxx, A.ai.x[MX_VX], G.bx), adj_y<false>(G, q, qxy, A.ai.y[MY_VX], G.byh),
        adj_z<FS, true>(G, q, qxz, A.ai.z[MZ_VX], G.bzh, false, false));
    put(VY, adj_x<false>(G, q, qxy, A.ai.x[MX_VY], G.bxh), adj_y<true>(G, q, qyy, A.ai.y[MY_VY], G.by),
        adj_z<FS, true>(G, q, qyz, A.ai.z[MZ_VY], G.bzh, false, false));
    put(VZ, adj_x<false>(G, q, qxz, A.ai.x[MX_VZ], G.bxh), adj_y<false>(G, q, qyz, A.ai.y[MY_VZ], G.byh),
        adj_z<FS, false>(G, q, qzz, A.ai.z[MZ_VZ], G.bz, true, true));
}

// The velocity step's transpose: lambda_s += D(p) on the core, p through the
// memories of the stresses' derivatives, and q = dt C lambda_s; of the shears
// q alone is kept (where mu = 0 they reach no result).
template <bool FS>
__global__ void __launch_bounds__(kThreads, kBlocks) adj_str(const Rev A)
{
    const Geo& G = A.G;
    const Cell q(G);
    if (!q.grid) return;
    const long long k = q.b * G.S + q.i, mi = q.b * G.ms + q.i;
    const float *px = A.p[0] + k, *py = A.p[1] + k, *pz = A.p[2] + k;
    if (const long long o = xsl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::ldg(G.ax + q.x);
        keep(A.ai.x[MX_SXX] + o, A.ao.x[MX_SXX] + o, v4::ldg(G.axh + q.x), v4::ldg(px));
        keep(A.ai.x[MX_SXY] + o, A.ao.x[MX_SXY] + o, a, v4::ldg(py));
        keep(A.ai.x[MX_SXZ] + o, A.ao.x[MX_SXZ] + o, a, v4::ldg(pz));
    }
    if (const long long o = ysl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::splat(__ldg(G.ay + q.y));
        keep(A.ai.y[MY_SXY] + o, A.ao.y[MY_SXY] + o, a, v4::ldg(px));
        keep(A.ai.y[MY_SYY] + o, A.ao.y[MY_SYY] + o, v4::splat(__ldg(G.ayh + q.y)), v4::ldg(py));
        keep(A.ai.y[MY_SYZ] + o, A.ao.y[MY_SYZ] + o, a, v4::ldg(pz));
    }
    if (const long long o = zsl(G, q.b, q.z, q.y, q.x); o >= 0) {
        const F4 a = v4::splat(__ldg(G.az + q.z));
        keep(A.ai.z[MZ_SXZ] + o, A.ao.z[MZ_SXZ] + o, a, v4::ldg(px));
        keep(A.ai.z[MZ_SYZ] + o, A.ao.z[MZ_SYZ] + o, a, v4::ldg(py));
        keep(A.ai.z[MZ_SZZ] + o, A.ao.z[MZ_SZZ] + o, v4::splat(__ldg(G.azh + q.z)), v4::ldg(pz));
    }
    const F4 mu = v4::ldg(A.m.mu + mi);
    const F4 zero = v4::splat(0.f);
    auto sum = [](const F4& a, const F4& b) {
        F4 t;
#pragma unroll
        for (int l = 0; l < 4; ++l) t.v[l] = a.v[l] + b.v[l];
        return t;
    };
    const bool c = q.core;
    auto put = [&](int fl, const F4& d, bool clear) {
        F4 v = v4::ld(A.a[fl - SXX] + k);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            if (clear) v.v[l] = 0.f;
            if (c && q.lane(G, l)) v.v[l] += d.v[l];
        }
        v4::st(A.a[fl - SXX] + k, v);
        return v;
    };
    auto shear = [&](int fl, const F4& d) {
        F4 v = v4::ld(A.q[fl - SXX] + k);
#pragma unroll
        for (int l = 0; l < 4; ++l)
            if (c && q.lane(G, l)) v.v[l] += (G.dt * mu.v[l]) * d.v[l];
        v4::st(A.q[fl - SXX] + k, v);
    };
    // (the test before each stencil keeps its loads apart from the next one's:
    // without it the kernel spills 448 bytes instead of 24)
    shear(SXY, c ? sum(adj_y<true>(G, q, px, A.ai.y[MY_SXY], G.by), adj_x<true>(G, q, py, A.ai.x[MX_SXY], G.bx)) : zero);
    shear(SXZ, c ? sum(adj_z<FS, false>(G, q, px, A.ai.z[MZ_SXZ], G.bz, true, true),
                       adj_x<true>(G, q, pz, A.ai.x[MX_SXZ], G.bx)) : zero);
    shear(SYZ, c ? sum(adj_z<FS, false>(G, q, py, A.ai.z[MZ_SYZ], G.bz, true, true),
                       adj_y<true>(G, q, pz, A.ai.y[MY_SYZ], G.by)) : zero);
    const bool surf = FS && q.z == G.z0;
    const F4 sxx = put(SXX, c ? adj_x<false>(G, q, px, A.ai.x[MX_SXX], G.bxh) : zero, false);
    const F4 syy = put(SYY, c ? adj_y<false>(G, q, py, A.ai.y[MY_SYY], G.byh) : zero, false);
    const F4 szz = put(SZZ, c ? adj_z<FS, true>(G, q, pz, A.ai.z[MZ_SZZ], G.bzh, true, false) : zero, surf);
    const F4 lam = v4::ldg(A.m.lam + mi);
    F4 qd[3];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        float t[3];
        stiff(G.dt, lam.v[l], mu.v[l], sxx.v[l], syy.v[l], szz.v[l], surf, t);
#pragma unroll
        for (int j = 0; j < 3; ++j) qd[j].v[l] = t[j];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) v4::st(A.q[j] + k, qd[j]);
}

__global__ void prep3(const float* __restrict__ vp, const float* __restrict__ vs, const float* __restrict__ rho,
                      long long rows, int nx, int P, float dt, float* olam, float* omu, float* okv)
{
    const long long n = rows * P;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long row = k / P;
        const int x = (int)(k - row * P);
        if (x >= nx) { olam[k] = omu[k] = okv[k] = 0.f; continue; }
        const long long i = row * nx + x;
        const float v = vp[i], s = vs[i], r = rho[i];
        omu[k] = __fmul_rn(__fmul_rn(r, s), s);
        olam[k] = __fmul_rn(r, __fsub_rn(__fmul_rn(v, v), __fmul_rn(__fmul_rn(2.0f, s), s)));
        okv[k] = dt * (1.f / r);
    }
}

// the x profiles, zero past their ends
__global__ void prep_profiles3(const float* a, const float* b, const float* ah, const float* bh, int nx, int len,
                               float* out)
{
    const float* in[4] = {a, b, ah, bh};
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 4 * len; e += gridDim.x * blockDim.x) {
        const int f = e / len, c = e - f * len - kGuard;
        out[e] = c >= 0 && c < nx ? in[f][c] : 0.f;
    }
}

// Gradients on the physical box, zero elsewhere, unpitched: per shot for
// per-shot models, else the slots summed in order.
struct Out {
    const float *vp, *vs, *rho;     // the caller's models
    float* g[3];                    // vp, vs, rho
};

__global__ void finalize3(const Rev A, const Out o)
{
    const Geo& G = A.G;
    const long long cells = (long long)G.nz * G.ny * G.nx, n = (G.ms ? G.B : 1) * cells;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long b = e / cells;
        const int c = (int)(e - b * cells);
        const int ix = c % G.nx, r = c / G.nx, iy = r % G.ny, iz = r / G.ny;
        float t[3] = {0.f, 0.f, 0.f};
        if (in_box(G, ix, iy, iz)) {
            const long long i = (long long)iz * G.SZ + iy * G.P + ix;
            for (int j = 0; j < 3; ++j) {
                t[j] = A.g[j][b * G.S + i];
                for (int s = 1; !G.ms && s < G.nslot; ++s) t[j] += A.g[j][s * G.S + i];
            }
            const float rho = o.rho[e];
            t[0] = -2.f * rho * o.vp[e] * t[0] * G.dt;
            t[1] = o.vs[e] != 0.f ? -2.f * t[1] / o.vs[e] : 0.f;     // mu = rho vs^2
            t[2] = t[2] / rho;
        }
        for (int j = 0; j < 3; ++j) o.g[j][e] = t[j];
    }
}

// ------------------------------------------------------------------- host
struct Plan {
    Geo G;
    int nm;                      // model copies
    bool host_tape;              // boundary-saving tape in pinned host memory (SWEEP_MEM_HOST_TAPE)
    bands::Bands bands;          // strip cells
};

static void check_mode(int mem_mode, int ckpt_every)
{
    if (mem_mode & SWEEP_MEM_HOST_TAPE) {
        mem_mode &= ~SWEEP_MEM_HOST_TAPE;
        SWEEP_REQUIRE(mem_mode != SWEEP_MEM_CHECKPOINT && mem_mode != SWEEP_MEM_RECURSIVE,
                      "elastic3d: a host tape goes with boundary saving only");
    }
    SWEEP_REQUIRE(mem_mode == SWEEP_MEM_BOUNDARY || mem_mode == SWEEP_MEM_CHECKPOINT ||
                      mem_mode == SWEEP_MEM_BOUNDARY_FP16 || mem_mode == SWEEP_MEM_BOUNDARY_BF16 ||
                      mem_mode == SWEEP_MEM_BOUNDARY_INT8 || mem_mode == SWEEP_MEM_RECURSIVE,
                  "elastic3d: unknown memory mode %d", mem_mode);
    SWEEP_REQUIRE(mem_mode != SWEEP_MEM_CHECKPOINT || ckpt_every >= 1,
                  "elastic3d: checkpoint interval must be >= 1 (got %d)", ckpt_every);
    SWEEP_REQUIRE(mem_mode != SWEEP_MEM_RECURSIVE || ckpt_every >= 1,
                  "elastic3d: the recursive checkpoint budget must be >= 1 (got %d)", ckpt_every);
}

static Plan make_plan(const sweep_elastic3d_desc* d)
{
    SWEEP_REQUIRE(d != nullptr, "null descriptor");
    SWEEP_REQUIRE(d->M == M, "elastic3d: this build holds order %d (got order %d)", 2 * M, 2 * d->M);
    SWEEP_REQUIRE(d->B >= 1 && d->nt >= 1, "elastic3d: B and nt must be >= 1");
    SWEEP_REQUIRE(d->nsrc >= 0 && d->nrec >= 0, "elastic3d: negative source/receiver count");
    SWEEP_REQUIRE(d->nsrc_fields >= 1 && d->nsrc_fields <= 9, "elastic3d: 1 to 9 source fields (got %d)",
                  d->nsrc_fields);
    for (int k = 0; k < d->nsrc_fields; ++k) {
        SWEEP_REQUIRE(d->src_fields[k] >= 0 && d->src_fields[k] < NFLD, "elastic3d: bad source field %d",
                      d->src_fields[k]);
        for (int j = 0; j < k; ++j)
            SWEEP_REQUIRE(d->src_fields[j] != d->src_fields[k], "elastic3d: source field %d repeated",
                          d->src_fields[k]);
    }
    SWEEP_REQUIRE(d->nrec_fields >= 1 && d->nrec_fields <= 9, "elastic3d: 1 to 9 receiver fields (got %d)",
                  d->nrec_fields);
    for (int k = 0; k < d->nrec_fields; ++k)
        SWEEP_REQUIRE(d->rec_fields[k] >= 0 && d->rec_fields[k] < NFLD, "elastic3d: bad receiver field %d",
                      d->rec_fields[k]);
    if (d->free_surface)
        SWEEP_REQUIRE(d->pad[0] == 0, "elastic3d: a free top face has no PML pad (got %d)", d->pad[0]);
    for (int f = d->free_surface ? 1 : 0; f < 6; ++f)
        SWEEP_REQUIRE(d->pad[f] >= 1, "elastic3d: every absorbing face needs a PML pad >= 1 (face %d has %d)", f,
                      d->pad[f]);
    Plan pl{};
    Geo& G = pl.G;
    G.fst = d->free_surface ? 1 : 0;
    G.B = d->B; G.nz = d->nz; G.ny = d->ny; G.nx = d->nx; G.nt = d->nt;
    const long long cells = (long long)d->nz * d->ny * d->nx;
    G.P = (d->nx + 7) / 8 * 8;
    G.SZ = d->ny * G.P;
    G.S = (long long)d->nz * d->ny * G.P;
    SWEEP_REQUIRE(cells < (1LL << 31) && G.S < (1LL << 31), "elastic3d: one shot's grid must hold < 2^31 cells");
    G.z0 = d->pad[0] + M; G.z1 = d->nz - d->pad[1] - M;
    G.y0 = d->pad[2] + M; G.y1 = d->ny - d->pad[3] - M;
    G.x0 = d->pad[4] + M; G.x1 = d->nx - d->pad[5] - M;
    SWEEP_REQUIRE(G.z1 - G.z0 >= 2 && G.y1 - G.y0 >= 2 && G.x1 - G.x0 >= 2,
                  "elastic3d: the physical box must be at least 2 cells along every axis");
    G.SZL = std::min(G.z0 + 1, d->nz); G.SZH = std::min(d->nz - (G.z1 - 1), d->nz - G.SZL);
    G.SYL = std::min(G.y0 + 1, d->ny); G.SYH = std::min(d->ny - (G.y1 - 1), d->ny - G.SYL);
    G.XL = (G.x0 + 1 + 3) / 4 * 4; G.XH = std::max(G.XL, (G.x1 - 1) / 4 * 4);
    G.WX = G.XL + std::max(0, (d->nx + 3) / 4 * 4 - G.XH); G.WY = G.SYL + G.SYH; G.WZ = G.SZL + G.SZH;
    G.dt = d->dt; G.idx = 1.f / d->dx; G.idy = 1.f / d->dy; G.idz = 1.f / d->dz;
    G.az = d->az; G.bz = d->bz; G.azh = d->azh; G.bzh = d->bzh;
    G.ay = d->ay; G.by = d->by; G.ayh = d->ayh; G.byh = d->byh;
    G.nsrc = d->nsrc; G.nrec = d->nrec;
    G.nsf = d->nsrc_fields; G.nrf = d->nrec_fields;
    for (int k = 0; k < 9; ++k) { G.sf[k] = d->src_fields[k]; G.rf[k] = d->rec_fields[k]; }
    G.src_loc = d->src_loc; G.rec_loc = d->rec_loc; G.wavelet = d->wavelet;
    const bool per_shot = d->model_stride != 0;
    SWEEP_REQUIRE(!per_shot || d->model_stride == cells, "elastic3d: model_stride must be 0 or nz * ny * nx");
    G.ms = per_shot ? G.S : 0;
    pl.nm = per_shot ? d->B : 1;
    G.nbx = (G.nx + 31) / 32;
    // shots per imaging thread: as many as still leave each SM four pairs of
    // blocks along y, which is all it holds; one for per-shot models
    const long long blocks = (long long)G.nbx * ((G.ny + 7) / 8) * ((G.nz + 3) / 4);
    G.group = 1;
    if (!per_shot)
        while (G.group < kMaxGroup && G.group < G.B && blocks * ((G.B + G.group) / (G.group + 1)) >= 4LL * 148) ++G.group;
    G.nslot = (G.B + G.group - 1) / G.group;
    pl.bands = bands::make<3>(M, G.z0, G.z1, G.y0, G.y1, G.x0, G.x1);
    G.ns = pl.bands.count;
    return pl;
}

// Strip storage of a memory mode: the step-slot layout of the boundary-saving
// tape (the checkpoint modes keep their chunk strips as fp32).
static void set_store(Plan& pl, int mem_mode)
{
    pl.host_tape = (mem_mode & SWEEP_MEM_HOST_TAPE) != 0;
    mem_mode &= ~SWEEP_MEM_HOST_TAPE;
    Geo& G = pl.G;
    StripStore& S = G.st;
    S = StripStore{};
    S.fmt = mem_mode == SWEEP_MEM_BOUNDARY_FP16 ? SF_F16
          : mem_mode == SWEEP_MEM_BOUNDARY_BF16 ? SF_BF16
          : mem_mode == SWEEP_MEM_BOUNDARY_INT8 ? SF_I8 : SF_F32;
    auto up = [](long long v, long long a) { return (v + a - 1) / a * a; };
    const long long per = (long long)G.B * NFLD * G.ns;
    if (S.fmt == SF_F32 || S.fmt == SF_BF16) {
        S.step = up(per * (S.fmt == SF_F32 ? 4 : 2), 256);
        return;
    }
    const long long bx = G.x1 - G.x0, by = G.y1 - G.y0, bz = G.z1 - G.z0;
    const long long cells[6] = {BW * by * bx, BW * by * bx, bz * BW * bx, bz * BW * bx, bz * by * BW, bz * by * BW};
    const int esz = S.fmt == SF_F16 ? 2 : 1;
    long long off = 0;
    for (int f = 0; f < 6; ++f) {
        SWEEP_REQUIRE(cells[f] * NFLD * G.B < (1LL << 31), "elastic3d: a strip face holds too many cells");
        S.cells[f] = (int)cells[f];
        S.blocks[f] = (int)((cells[f] + kQB - 1) / kQB);
        S.pay[f] = off;
        off = up(off + (long long)NFLD * G.B * cells[f] * esz, 16);
    }
    for (int f = 0; f < 6; ++f) {
        S.scl[f] = off;
        off = up(off + (long long)NFLD * G.B * S.blocks[f] * 4, 16);
    }
    S.step = up(off, 256);
}

static unsigned quant_blocks(const Geo& G)
{
    long long per = 0;
    for (int f = 0; f < 6; ++f) per += G.st.blocks[f];
    return (unsigned)(per * NFLD * G.B);
}

struct Common {
    float *lam, *mu, *kv;
    float* xprof;                // a, b, a_half, b_half along x, padded
    int* cells;
};

static int xprof_len(const Geo& G) { return G.P + 2 * kGuard; }

static void carve_common(Carve& c, const Plan& pl, Common& w)
{
    const long long mc = (long long)pl.nm * pl.G.S;
    w.lam = c.take<float>(mc); w.mu = c.take<float>(mc); w.kv = c.take<float>(mc);
    w.xprof = c.take<float>(4LL * xprof_len(pl.G));
    w.cells = c.take<int>(std::max(pl.G.ns, 1));
}

static long long slab_count(const Geo& G, int axis)
{
    return axis == 0 ? (long long)G.B * G.nz * G.ny * G.WX
         : axis == 1 ? (long long)G.B * G.nz * G.WY * G.P : (long long)G.B * G.WZ * G.ny * G.P;
}

static void carve_slabs(Carve& c, const Geo& G, Slabs& s)
{
    for (int k = 0; k < 6; ++k) s.x[k] = c.take<float>(slab_count(G, 0));
    for (int k = 0; k < 6; ++k) s.y[k] = c.take<float>(slab_count(G, 1));
    for (int k = 0; k < 6; ++k) s.z[k] = c.take<float>(slab_count(G, 2));
}

static float* slab_ptr(const Slabs& s, int k) { return k < 6 ? s.x[k] : k < 12 ? s.y[k - 6] : s.z[k - 12]; }

struct FwdWs {
    Common cm;
    float* f[NFLD];
    Slabs mem;
    char *zero0, *zero1;
    char* ring;                  // host tape: HostRing::R device strip slots
};

static void carve_fwd(Carve& c, const Plan& pl, FwdWs& w)
{
    carve_common(c, pl, w.cm);
    c.take<char>(0);
    w.zero0 = c.base ? c.base + c.off : nullptr;
    for (int k = 0; k < NFLD; ++k) w.f[k] = c.take<float>((long long)pl.G.B * pl.G.S);
    carve_slabs(c, pl.G, w.mem);
    c.take<char>(0);
    w.zero1 = c.base ? c.base + c.off : nullptr;
    if (pl.host_tape) w.ring = c.take<char>((long long)HostRing::R * pl.G.st.step);
}

struct RevWs {
    Common cm;
    float* f[NFLD];
    float* a[3];
    float* q[6];
    float* p[3];
    Slabs am[2];                 // adjoint memories, double-buffered
    float* g[3];
    char *zero0, *zero1;
    char* ring;                  // host tape: HostRing::R device strip slots
    Slabs fmem;                  // checkpoint modes: forward CPML memories of the replay
    float* chunk;                // checkpoint modes: fp32 strips of one chunk, (k + 1, B, 9, ns)
};

static void carve_rev(Carve& c, const Plan& pl, RevWs& w)
{
    carve_common(c, pl, w.cm);
    const Geo& G = pl.G;
    const long long n = (long long)G.B * G.S;
    c.take<char>(0);
    w.zero0 = c.base ? c.base + c.off : nullptr;
    for (int k = 0; k < NFLD; ++k) w.f[k] = c.take<float>(n);
    for (float*& p : w.a) p = c.take<float>(n);
    for (float*& p : w.q) p = c.take<float>(n);
    for (float*& p : w.p) p = c.take<float>(n);
    for (Slabs& s : w.am) carve_slabs(c, G, s);
    for (float*& p : w.g) p = c.take<float>(G.nslot * G.S);
    c.take<char>(0);
    w.zero1 = c.base ? c.base + c.off : nullptr;
    if (pl.host_tape) w.ring = c.take<char>((long long)HostRing::R * G.st.step);
}

static long long chunk_floats(const Plan& pl) { return (long long)pl.G.B * NFLD * pl.G.ns; }

static void carve_rev_ckpt(Carve& c, const Plan& pl, int k, RevWs& w)
{
    carve_rev(c, pl, w);
    carve_slabs(c, pl.G, w.fmem);
    w.chunk = c.take<float>((long long)(k + 1) * chunk_floats(pl));
}

// rows of a field of every shot
static long long rows_of(const Geo& G) { return (long long)G.B * G.nz * G.ny; }

// Boundary-saving tape: one strip slot per step (G.st.step bytes), then the
// final nine-field state (9, B, nz, ny, nx).
static int64_t tape_bytes_of(const Plan& pl)
{
    return (int64_t)pl.G.nt * pl.G.st.step + (int64_t)NFLD * rows_of(pl.G) * pl.G.nx * 4;
}

static void* tape_slot(const void* tape, const Plan& pl, int it)
{
    return const_cast<char*>(static_cast<const char*>(tape)) + (long long)it * pl.G.st.step;
}

static float* tape_last(const void* tape, const Plan& pl)
{
    return reinterpret_cast<float*>(static_cast<char*>(tape_slot(tape, pl, pl.G.nt)));
}

// Checkpointed boundary saving (SWEEP_MEM_CHECKPOINT, chunk length k): for
// every chunk c >= 1 the tape holds the state after step c k - 1 -- the nine
// fields and the 18 forward CPML memories -- and the fp32 strips of that step;
// the backward replays each chunk from its checkpoint into the strips of that
// chunk and runs the boundary-saving reverse steps over it (the reference's
// staggered driver replays chunks as well, sg_driver.cuh:911-925).  The
// recursive mode (SWEEP_MEM_RECURSIVE) keeps snapshots of the same layout.
static long long slab_floats(const Geo& G) { return 6 * (slab_count(G, 0) + slab_count(G, 1) + slab_count(G, 2)); }

static long long ckpt_stride(const Plan& pl)
{
    Carve c(nullptr);
    c.take<float>((long long)NFLD * pl.G.B * pl.G.S);
    c.take<float>(slab_floats(pl.G));
    c.take<float>(chunk_floats(pl));
    return (c.off + 255) & ~255LL;
}

static int nchunks(const Plan& pl, int k)
{
    SWEEP_REQUIRE(k >= 1, "elastic3d: checkpoint interval must be >= 1 (got %d)", k);
    return (pl.G.nt + k - 1) / k;
}

struct Ckpt {
    float* f[NFLD];
    float* mem;           // the 18 slabs, x then y then z, in carve_slabs order
    float* strips;
};

static Ckpt ckpt_at(void* tape, const Plan& pl, int ch)
{
    Carve c(static_cast<char*>(tape) + (long long)(ch - 1) * ckpt_stride(pl));
    Ckpt k{};
    for (int f = 0; f < NFLD; ++f) k.f[f] = c.take<float>((long long)pl.G.B * pl.G.S);
    k.mem = c.take<float>(slab_floats(pl.G));
    k.strips = c.take<float>(chunk_floats(pl));
    return k;
}

// Copy the 18 slabs between a Slabs set and a packed checkpoint range.
static void slabs_copy(const Slabs& s, float* packed, const Geo& G, bool to_packed, cudaStream_t st)
{
    long long o = 0;
    for (int k = 0; k < 18; ++k) {
        float* p = slab_ptr(s, k);
        const long long cnt = slab_count(G, k / 6);
        if (to_packed) SWEEP_CUDA(cudaMemcpyAsync(packed + o, p, cnt * 4, cudaMemcpyDeviceToDevice, st));
        else SWEEP_CUDA(cudaMemcpyAsync(p, packed + o, cnt * 4, cudaMemcpyDeviceToDevice, st));
        o += cnt;
    }
}

static void slabs_zero(const Slabs& s, const Geo& G, cudaStream_t st)
{
    for (int k = 0; k < 18; ++k) SWEEP_CUDA(cudaMemsetAsync(slab_ptr(s, k), 0, slab_count(G, k / 6) * 4, st));
}

void sizes(const sweep_elastic3d_desc* d, int mem_mode, int ckpt_every, int64_t* ws_bytes, int64_t* tape_bytes)
{
    check_mode(mem_mode, ckpt_every);
    Plan pl = make_plan(d);
    set_store(pl, mem_mode);
    const int mode = mem_mode & ~SWEEP_MEM_HOST_TAPE;
    Carve f(nullptr), r(nullptr);
    FwdWs fw{};
    RevWs rw{};
    carve_fwd(f, pl, fw);
    if (mode == SWEEP_MEM_CHECKPOINT) {
        carve_rev_ckpt(r, pl, ckpt_every, rw);
        *tape_bytes = (int64_t)std::max(nchunks(pl, ckpt_every) - 1, 1) * ckpt_stride(pl);
    } else if (mode == SWEEP_MEM_RECURSIVE) {
        carve_rev_ckpt(r, pl, SWEEP_RECURSIVE_LEAF, rw);
        r.take<char>((long long)ckpt_every * ckpt_stride(pl));          // the snapshot slots
        *tape_bytes = 256;                                               // nothing is kept
    } else {
        carve_rev(r, pl, rw);
        *tape_bytes = tape_bytes_of(pl);
    }
    *ws_bytes = std::max(f.off, r.off);
}

static void setup_common(const sweep_elastic3d_desc* d, Plan& pl, const Common& w, cudaStream_t st)
{
    Geo& G = pl.G;
    G.cells = w.cells;
    prep3<<<1184, 256, 0, st>>>(d->vp, d->vs, d->rho, (long long)pl.nm * G.nz * G.ny, G.nx, G.P, d->dt, w.lam, w.mu,
                                w.kv);
    const int len = xprof_len(G);
    prep_profiles3<<<8, 256, 0, st>>>(d->ax, d->bx, d->axh, d->bxh, G.nx, len, w.xprof);
    G.ax = w.xprof + kGuard; G.bx = G.ax + len; G.axh = G.bx + len; G.bxh = G.axh + len;
    bands::band_table<3><<<592, 256, 0, st>>>(pl.bands, G.P, G.SZ, w.cells);
    SWEEP_LAUNCH_CHECK();
}

static Models models_of(const Common& w) { return Models{w.lam, w.mu, w.kv}; }

static dim3 rec_grid(const Geo& G)
{
    return dim3((unsigned)std::min((G.nrec + 127) / 128, 64), (unsigned)G.B);
}

// n: shots, or shot groups
static dim3 cell_grid(const Geo& G, int n)
{
    return dim3((unsigned)(G.nbx * n), (G.ny + kBY - 1) / kBY, (G.nz + kBZ - 1) / kBZ);
}

static unsigned strip_blocks(const Geo& G)
{
    return (unsigned)std::max<long long>(std::min<long long>(((long long)G.B * G.ns + 255) / 256, 4096), 1);
}

// Forward steps [it0, it1) on the fields / memories of A; strips_of(it) is
// the slot (format fmt) that takes the strips of step it, or null.
template <class StripsOf>
static void forward_steps(const Fwd& A, int it0, int it1, StripsOf strips_of, int fmt, float* record, cudaStream_t st,
                          HostRing* hr = nullptr)
{
    const Geo& G = A.G;
    Fields F{};
    for (int k = 0; k < NFLD; ++k) F.f[k] = A.f[k];
    const dim3 grid = cell_grid(G, G.B), block(8, kBY, kBZ);
    const bool scaled = fmt == SF_F16 || fmt == SF_I8;
    for (int it = it0; it < it1; ++it) {
        if (G.fst) {
            vel3<true><<<grid, block, 0, st>>>(A);
            str3<true><<<grid, block, 0, st>>>(A);
        } else {
            vel3<false><<<grid, block, 0, st>>>(A);
            str3<false><<<grid, block, 0, st>>>(A);
        }
        if (G.nsrc > 0) src3<<<G.B, 128, 0, st>>>(G, F, it, 1.f);
        if (void* slot = strips_of(it)) {
            if (hr) hr->before_write(it);
            if (scaled) quant3<<<quant_blocks(G), kQB, 0, st>>>(G, F, slot);
            else if (G.ns > 0) strips3<<<strip_blocks(G), 256, 0, st>>>(G, F, slot, fmt, 0, NFLD, 0);
            if (hr) hr->after_write(it);
        }
        if (record && G.nrec > 0) rec3<<<rec_grid(G), 128, 0, st>>>(G, F, record, it);
        SWEEP_LAUNCH_CHECK();
    }
}

void forward(const sweep_elastic3d_desc* d, int mem_mode, int ckpt_every, float* record, void* tape, void* ws,
             int64_t ws_bytes, cudaStream_t st)
{
    check_mode(mem_mode, ckpt_every);
    Plan pl = make_plan(d);
    set_store(pl, mem_mode);
    const int mode = mem_mode & ~SWEEP_MEM_HOST_TAPE;
    Carve c(ws);
    FwdWs w{};
    carve_fwd(c, pl, w);
    SWEEP_REQUIRE(ws != nullptr && c.off <= ws_bytes, "elastic3d forward: workspace too small (%lld < %lld bytes)",
                  (long long)ws_bytes, (long long)c.off);
    Geo& G = pl.G;
    setup_common(d, pl, w.cm, st);
    SWEEP_CUDA(cudaMemsetAsync(w.zero0, 0, w.zero1 - w.zero0, st));
    if (record && G.nrec > 0)
        SWEEP_CUDA(cudaMemsetAsync(record, 0, sizeof(float) * (size_t)G.B * G.nt * G.nrec * G.nrf, st));
    Fwd A{};
    A.G = G;
    A.m = models_of(w.cm);
    for (int k = 0; k < NFLD; ++k) A.f[k] = w.f[k];
    A.mem = w.mem;
    const long long n = (long long)G.B * G.S;
    if (mode == SWEEP_MEM_RECURSIVE) tape = nullptr;     // the backward replays from the initial state
    if (mode != SWEEP_MEM_CHECKPOINT) {
        HostRing hr;
        const bool host = tape && pl.host_tape;
        if (host) hr.open(w.ring, tape, G.st.step, st);
        forward_steps(A, 0, G.nt,
                      [&](int it) -> void* { return !tape ? nullptr : host ? hr.slot(it) : tape_slot(tape, pl, it); },
                      G.st.fmt, record, st, host ? &hr : nullptr);
        if (host) hr.close();
        if (tape) {
            float* last = tape_last(tape, pl);
            for (int k = 0; k < NFLD; ++k)
                copy_rows(last + k * rows_of(G) * G.nx, G.nx, w.f[k], G.P, G.nx, rows_of(G), st);
        }
        return;
    }
    const int k = ckpt_every, C = nchunks(pl, k);
    for (int ch = 0; ch < C; ++ch) {
        const int it0 = ch * k, it1 = std::min(G.nt, it0 + k);
        if (tape && ch >= 1) {
            const Ckpt cp = ckpt_at(tape, pl, ch);
            for (int f = 0; f < NFLD; ++f)
                SWEEP_CUDA(cudaMemcpyAsync(cp.f[f], w.f[f], sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
            slabs_copy(w.mem, cp.mem, G, true, st);
        }
        // the last step of a chunk keeps its strips with the next checkpoint
        forward_steps(A, it0, it1,
                      [&](int it) -> void* {
                          return (tape && it == it1 - 1 && ch + 1 < C) ? ckpt_at(tape, pl, ch + 1).strips : nullptr;
                      },
                      SF_F32, record, st);
    }
}

void backward(const sweep_elastic3d_desc* d, int mem_mode, int ckpt_every, const float* adj, const void* tape,
              float* grad_vp, float* grad_vs, float* grad_rho, void* ws, int64_t ws_bytes, cudaStream_t st)
{
    check_mode(mem_mode, ckpt_every);
    Plan pl = make_plan(d);
    set_store(pl, mem_mode);
    const int mode = mem_mode & ~SWEEP_MEM_HOST_TAPE;
    const bool ckpt = mode == SWEEP_MEM_CHECKPOINT, recursive = mode == SWEEP_MEM_RECURSIVE;
    SWEEP_REQUIRE(recursive || tape != nullptr, "elastic3d backward: the forward's tape is required");
    Carve c(ws);
    RevWs w{};
    char* snaps = nullptr;
    if (ckpt) carve_rev_ckpt(c, pl, ckpt_every, w);
    else if (recursive) {
        carve_rev_ckpt(c, pl, SWEEP_RECURSIVE_LEAF, w);
        snaps = c.take<char>((long long)ckpt_every * ckpt_stride(pl));
    } else carve_rev(c, pl, w);
    SWEEP_REQUIRE(ws != nullptr && c.off <= ws_bytes, "elastic3d backward: workspace too small (%lld < %lld bytes)",
                  (long long)ws_bytes, (long long)c.off);
    Geo& G = pl.G;
    setup_common(d, pl, w.cm, st);
    SWEEP_CUDA(cudaMemsetAsync(w.zero0, 0, w.zero1 - w.zero0, st));
    const long long n = (long long)G.B * G.S;
    Rev A{};
    A.G = G;
    A.m = models_of(w.cm);
    for (int k = 0; k < NFLD; ++k) A.f[k] = w.f[k];
    for (int k = 0; k < 6; ++k) A.q[k] = w.q[k];
    for (int k = 0; k < 3; ++k) { A.a[k] = w.a[k]; A.p[k] = w.p[k]; A.g[k] = w.g[k]; }
    A.adj = adj;
    Fields F{};
    for (int k = 0; k < NFLD; ++k) F.f[k] = w.f[k];
    const dim3 grid = cell_grid(G, G.B), ggrid = cell_grid(G, G.nslot), block(8, kBY, kBZ);
    int cur = 0;                 // adjoint memories read by the next reverse step
    HostRing hr;
    const bool host = pl.host_tape && !ckpt && !recursive;
    // Reverse steps it1 - 1 .. max(it0, 1) (the staggered reverse has no
    // it = 0 step) on the reconstruction state after step it1 - 1;
    // strips_of(t) holds the strips (format fmt) of the state after step t.
    auto reverse = [&](int it0, int it1, auto strips_of, int fmt) {
        for (int it = it1 - 1; it >= std::max(it0, 1); --it) {
            A.it = it;
            void* prev = strips_of(it - 1);
            if (host) hr.before_read(it - 1);
            A.ai = w.am[cur];
            A.ao = w.am[cur ^ 1];
            cur ^= 1;
            if (G.nrec > 0) res3<<<rec_grid(G), 128, 0, st>>>(A);
            if (G.nsrc > 0) src3<<<G.B, 128, 0, st>>>(G, F, it, -1.f);
            if (G.fst) stress_rev<true><<<ggrid, block, 0, st>>>(A);
            else stress_rev<false><<<ggrid, block, 0, st>>>(A);
            if (G.ns > 0) strips3<<<strip_blocks(G), 256, 0, st>>>(G, F, prev, fmt, SXX, NFLD, 1);
            if (G.fst) {
                adj_vel<true><<<grid, block, 0, st>>>(A);
                adj_str<true><<<grid, block, 0, st>>>(A);
                vel_rev<true><<<ggrid, block, 0, st>>>(A);
            } else {
                adj_vel<false><<<grid, block, 0, st>>>(A);
                adj_str<false><<<grid, block, 0, st>>>(A);
                vel_rev<false><<<ggrid, block, 0, st>>>(A);
            }
            if (G.ns > 0) restore_velocity<<<strip_blocks(G), 256, 0, st>>>(A, prev, fmt);
            if (host) {
                hr.after_read(it - 1);
                if (it - 1 - HostRing::R >= std::max(it0 - 1, 0)) hr.fetch(it - 1 - HostRing::R, true);
            }
            SWEEP_LAUNCH_CHECK();
        }
    };
    // the replay of the checkpoint modes runs straight into the reconstruction
    // fields, with its own forward CPML memories
    Fwd R{};
    R.G = G;
    R.m = A.m;
    for (int k = 0; k < NFLD; ++k) R.f[k] = w.f[k];
    R.mem = w.fmem;
    const long long cs = chunk_floats(pl);
    auto chunk_slot = [&](int j) -> void* { return w.chunk + (long long)j * cs; };
    if (recursive) {
        // Recursive checkpointing: the bisection of the acoustic drivers; a
        // snapshot slot has the checkpoint layout (nine fields, 18 CPML slabs,
        // strips of the step before), leaves are SWEEP_RECURSIVE_LEAF steps.
        const int L = SWEEP_RECURSIVE_LEAF, count = ckpt_every;
        auto restore = [&](int k) {
            if (k < 0) {
                for (int f = 0; f < NFLD; ++f) SWEEP_CUDA(cudaMemsetAsync(w.f[f], 0, sizeof(float) * n, st));
                slabs_zero(w.fmem, G, st);
            } else {
                const Ckpt cp = ckpt_at(snaps, pl, k + 1);
                for (int f = 0; f < NFLD; ++f)
                    SWEEP_CUDA(cudaMemcpyAsync(w.f[f], cp.f[f], sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
                slabs_copy(w.fmem, cp.mem, G, false, st);
            }
        };
        auto save = [&](int k) {
            const Ckpt cp = ckpt_at(snaps, pl, k + 1);
            for (int f = 0; f < NFLD; ++f)
                SWEEP_CUDA(cudaMemcpyAsync(cp.f[f], w.f[f], sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
            slabs_copy(w.fmem, cp.mem, G, true, st);
        };
        auto strips_from = [&](int k) {        // strips of the step before snapshot k into chunk slot 0
            SWEEP_CUDA(cudaMemcpyAsync(w.chunk, ckpt_at(snaps, pl, k + 1).strips, sizeof(float) * cs,
                                       cudaMemcpyDeviceToDevice, st));
        };
        auto leaf = [&](int a, int e) {
            forward_steps(R, a, e, [&](int it) { return chunk_slot(it - a + 1); }, SF_F32, nullptr, st);
            reverse(a, e, [&](int t) { return chunk_slot(t - (a - 1)); }, SF_F32);
        };
        std::function<void(int, int, int, int)> process = [&](int a, int b, int ka, int free) {
            const int nleaf = (b - a + L - 1) / L;
            if (nleaf <= 1) {
                restore(ka);
                if (a > 0) strips_from(ka);
                leaf(a, b);
                return;
            }
            if (free > 0) {
                const int k = count - free, m = a + L * ((nleaf + 1) / 2);
                restore(ka);
                float* ks = ckpt_at(snaps, pl, k + 1).strips;
                forward_steps(R, a, m, [&](int it) -> void* { return it == m - 1 ? ks : nullptr; }, SF_F32, nullptr,
                              st);
                save(k);
                process(m, b, k, free - 1);
                process(a, m, ka, free);
                return;
            }
            for (int c0 = a + (nleaf - 1) * L; c0 >= a; c0 -= L) {
                restore(ka);
                if (c0 > a)
                    forward_steps(R, a, c0, [&](int it) -> void* { return it == c0 - 1 ? w.chunk : nullptr; },
                                  SF_F32, nullptr, st);
                else if (a > 0)
                    strips_from(ka);
                leaf(c0, std::min(b, c0 + L));
            }
        };
        process(0, G.nt, -1, count);
    } else if (!ckpt) {
        const float* last = tape_last(tape, pl);
        for (int k = 0; k < NFLD; ++k)
            copy_rows(w.f[k], G.P, last + k * rows_of(G) * G.nx, G.nx, G.nx, rows_of(G), st);
        if (host) {
            hr.open(w.ring, const_cast<void*>(tape), G.st.step, st);
            for (int t = G.nt - 2; t >= 0 && t > G.nt - 2 - HostRing::R; --t) hr.fetch(t, false);
            reverse(0, G.nt, [&](int t) { return hr.slot(t); }, G.st.fmt);
            hr.close();
        } else {
            reverse(0, G.nt, [&](int t) { return tape_slot(tape, pl, t); }, G.st.fmt);
        }
    } else {
        const int k = ckpt_every, C = nchunks(pl, k);
        void* tp = const_cast<void*>(tape);
        for (int ch = C - 1; ch >= 0; --ch) {
            const int it0 = ch * k, it1 = std::min(G.nt, it0 + k);
            if (ch == 0) {
                for (int f = 0; f < NFLD; ++f) SWEEP_CUDA(cudaMemsetAsync(w.f[f], 0, sizeof(float) * n, st));
                slabs_zero(w.fmem, G, st);
            } else {
                const Ckpt cp = ckpt_at(tp, pl, ch);
                for (int f = 0; f < NFLD; ++f)
                    SWEEP_CUDA(cudaMemcpyAsync(w.f[f], cp.f[f], sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
                slabs_copy(w.fmem, cp.mem, G, false, st);
                SWEEP_CUDA(cudaMemcpyAsync(w.chunk, cp.strips, sizeof(float) * cs, cudaMemcpyDeviceToDevice, st));
            }
            // replay: chunk slot j holds the strips after step it0 - 1 + j
            forward_steps(R, it0, it1, [&](int it) { return chunk_slot(it - it0 + 1); }, SF_F32, nullptr, st);
            reverse(it0, it1, [&](int t) { return chunk_slot(t - (it0 - 1)); }, SF_F32);
        }
    }
    finalize3<<<1184, 256, 0, st>>>(A, Out{d->vp, d->vs, d->rho, {grad_vp, grad_vs, grad_rho}});
    SWEEP_LAUNCH_CHECK();
}

}  // namespace EL3D_NS
}  // namespace sweep
