// elastic_vec.cuh -- the 2-D elastic steps on four x cells per thread
// (vec4.cuh), for any half-width M: forward velocity and stress step, and the
// reverse step (two kernels around the band restores), with traction-free
// faces (FS) by the image method.  Shared by the orders other than 8
// (elastic_orders.cu) and by the reverse of order 8 (elastic2d.cu).
//
// Measured at order 8 on 16 shots of 400 x 1200: 205 us rev_a, 194 us
// rev_b and 45 us the restores and events, where 32 x 32 tiles of one cell per
// thread and row, with q and p rebuilt in shared memory for tile and halo, took
// 652 us a step.  A reverse kernel moves 68 bytes a cell: 105 us at the copy
// rate; its warps wait for loads (long scoreboard 12 to 13 an issue, DRAM at 42
// and 47 %) at 64 registers a thread, 1024 threads an SM, a bound that spills
// 192 and 80 bytes at order 8, a fifth and a tenth of the L1 traffic.
// The image of up to four shots is summed by a thread (layout): 187 + 170 us
// against 198 + 175 us with a slot per shot, at order 4 on the same grid (both
// with the adjoint velocities beside p, 80 bytes a cell).
#pragma once

#include <algorithm>

#include "common.cuh"
#include "vec4.cuh"

namespace sweep {
namespace evec {

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
    int XL, XH, WX, WZ;             // memory slabs: x below XL or from XH on (multiples of 4), widths
    int nbx, rows;                  // x blocks, rows of a block
    int group, nslot;               // shots per imaging thread, gradient slots
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
// CPML memories of the layers (and the box's last cell, which a half-cell
// profile reaches): along x (B, nz, WX) in whole groups of four cells, along z
// (B, WZ, P).
struct Mems {
    float* m[NMEM];
};
constexpr bool along_x(int k) { return k == M_VXX || k == M_VZX || k == M_SXXX || k == M_SXZX; }

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
// offset of a cell (a group along x) in a memory; a row or group off the slab
// at its first place
__device__ __forceinline__ long long xmem(const Geo& G, int b, int z, int x)
{
    return ((long long)b * G.nz + z) * G.WX + (x < 0 ? 0 : x < G.XL ? x : x >= G.XH ? min(G.XL + x - G.XH, G.WX - 4) : 0);
}
__device__ __forceinline__ long long zmem(const Geo& G, int b, int z, int x)
{
    return ((long long)b * G.WZ + (z < G.z0 ? z : z >= G.z1 - 1 ? G.z0 + z - (G.z1 - 1) : 0)) * G.P + x;
}

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
        const long long mx = xmem(G, q.b, q.z, q.x);
        cpml(W.m[M_SXXX] + mx, v4::ldg(G.axh + q.x), v4::ldg(G.bxh + q.x), d.xx, on);
        cpml(W.m[M_SXZX] + mx, v4::ldg(G.ax + q.x), v4::ldg(G.bx + q.x), d.zx, on);
    }
    if (any && zband(G, q.z)) {
        const long long mz = zmem(G, q.b, q.z, q.x);
        cpml(W.m[M_SZZZ] + mz, v4::splat(__ldg(G.azh + q.z)), v4::splat(__ldg(G.bzh + q.z)), d.zz, on);
        cpml(W.m[M_SXZZ] + mz, v4::splat(__ldg(G.az + q.z)), v4::splat(__ldg(G.bz + q.z)), d.xz, on);
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
        const long long mx = xmem(G, q.b, q.z, q.x);
        cpml(W.m[M_VXX] + mx, v4::ldg(G.ax + q.x), v4::ldg(G.bx + q.x), d.xx, on);
        cpml(W.m[M_VZX] + mx, v4::ldg(G.axh + q.x), v4::ldg(G.bxh + q.x), d.zx, on);
    }
    if (any && zband(G, q.z)) {
        const long long mz = zmem(G, q.b, q.z, q.x);
        cpml(W.m[M_VZZ] + mz, v4::splat(__ldg(G.az + q.z)), v4::splat(__ldg(G.bz + q.z)), d.zz, on);
        cpml(W.m[M_VXZ] + mz, v4::splat(__ldg(G.azh + q.z)), v4::splat(__ldg(G.bzh + q.z)), d.xz, on);
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
// ---------------------------------------------------------------- reverse
// The adjoint velocities are held as p = kv lambda_v and the adjoint shear
// stress as qxz = dt mu lambda_xz alone: the transposes read these, and where
// mu = 0 lambda_xz reaches no result.
struct Rev {
    Fields f;                       // reconstructed forward fields
    float* a[2];                    // adjoint sxx, szz
    float* q[3];                    // dt C lambda_s: xx, zz, xz
    float* p[2];                    // kv lambda_v
    Mems ai, ao;                    // adjoint CPML memories: read, written
    float* g[3];                    // slots of a shot group: gl, dt mu (gm - 2 gl), the rho image (times rho)
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

// signed residuals (stress -1, velocity +1) into the adjoint stresses, q and
// p; the source of step it out of the forward fields
__global__ static void events(const Geo G, const Rev R)
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
        if (f < SXX) { atomicAdd(R.p[f] + i, G.kv[mi] * v); continue; }
        if (f != SXZ) atomicAdd(R.a[f - SXX] + i, v);
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
// (reference kernels.cuh:365-535, 601-663).  The shear part of dt mu gm is
// qxz (dvx/dz + dvz/dx); qxz is zero where a face zeroes the shear.
template <int M, bool FS, bool GRP>
__device__ __forceinline__ void stress_rev(const Geo& G, const Rev& R, const Cell& q)
{
    if (q.b >= G.nslot || !q.core || !zbox(G, q.z) || q.x + 3 < G.x0 || q.x >= G.x1) return;
    const bool rrow = q.z >= G.rz0 && q.z < G.rz1;
    F4 sl = v4::splat(0.f), sm = sl, sr = sl;
    const int b0 = GRP ? q.b * G.group : q.b, b1 = GRP ? min(b0 + G.group, G.B) : b0 + 1;
    for (int b = b0; b < b1; ++b) {
        const long long k = b * G.S + q.i, mi = b * G.ms + q.i;
        const Four d = velocity_diffs<M, FS>(G, R.f, q, k);
        const F4 lam = v4::ldg(G.lam + mi), mu = v4::ldg(G.mu + mi);
        const F4 bxx = v4::ldg(R.a[0] + k), bzz = v4::ldg(R.a[1] + k), qxz = v4::ldg(R.q[2] + k);
        F4 sxx = v4::ld(R.f.f[SXX] + k), szz = v4::ld(R.f.f[SZZ] + k), sxz = v4::ld(R.f.f[SXZ] + k);
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
            const float gs = (G.dt * m) * (gm - 2.f * gl) + qxz.v[l] * (d.xz.v[l] + d.zx.v[l]);
            sl.v[l] += gl;
            sm.v[l] += gs;
            sr.v[l] -= (G.dt * gl) * l2m + gs;
            if (rrow && x >= G.rx0 && x < G.rx1) {
                sxx.v[l] = sxx.v[l] - G.dt * (l2m * vxx + L * vzz);
                szz.v[l] = szz.v[l] - G.dt * (l2m * vzz + L * vxx);
                sxz.v[l] = sxz.v[l] - (G.dt * m) * (d.xz.v[l] + d.zx.v[l]);
            }
        }
        v4::st(R.f.f[SXX] + k, sxx);
        v4::st(R.f.f[SZZ] + k, szz);
        v4::st(R.f.f[SXZ] + k, sxz);
    }
    const long long o = q.b * G.S + q.i;
    add4(R.g[0] + o, sl);
    add4(R.g[1] + o, sm);
    add4(R.g[2] + o, sr);
}

// velocity reconstruction on the reverse box with its rho image
template <int M, bool FS, bool GRP>
__device__ __forceinline__ void vel_rev(const Geo& G, const Rev& R, const Cell& q)
{
    if (q.b >= G.nslot || !q.core || q.z < G.rz0 || q.z >= G.rz1 || q.x + 3 < G.rx0 || q.x >= G.rx1) return;
    F4 sr = v4::splat(0.f);
    const int b0 = GRP ? q.b * G.group : q.b, b1 = GRP ? min(b0 + G.group, G.B) : b0 + 1;
    for (int b = b0; b < b1; ++b) {
        const long long k = b * G.S + q.i;
        const Four d = stress_diffs<M, FS>(G, R.f, q, k);
        const F4 kv = v4::ldg(G.kv + b * G.ms + q.i), px = v4::ldg(R.p[0] + k), pz = v4::ldg(R.p[1] + k);
        F4 vx = v4::ld(R.f.f[VX] + k), vz = v4::ld(R.f.f[VZ] + k);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            if (q.x + l < G.rx0 || q.x + l >= G.rx1) continue;
            const float gx = d.xx.v[l] + d.xz.v[l], gz = d.zx.v[l] + d.zz.v[l];
            vx.v[l] = vx.v[l] - kv.v[l] * gx;
            vz.v[l] = vz.v[l] - kv.v[l] * gz;
            sr.v[l] -= px.v[l] * gx + pz.v[l] * gz;
        }
        v4::st(R.f.f[VX] + k, vx);
        v4::st(R.f.f[VZ] + k, vz);
    }
    if (R.it > 1) add4(R.g[2] + q.b * G.S + q.i, sr);
}

// a transpose's input through its adjoint CPML memory w on the lanes `on`
__device__ __forceinline__ F4 through(const F4& u, const F4& b, const F4& w, const bool (&on)[4])
{
    F4 t;
#pragma unroll
    for (int l = 0; l < 4; ++l) t.v[l] = on[l] ? u.v[l] + b.v[l] * (w.v[l] + u.v[l]) : u.v[l];
    return t;
}

// The negated transpose of a derivative along z / x of the input u (at the
// thread's group; whole memory w, profile prof): FWD the transpose of a D+ form (plain: D-), else of a D- form.
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
        return through(v4::ldg(u + j * G.P), v4::splat(__ldg(prof + z)), v4::ldg(w + zmem(G, q.b, z, q.x)), on);
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
            const F4 b = v4::ldg(prof + q.x + 4 * j), t = v4::ldg(w + xmem(G, q.b, q.z, q.x + 4 * j));
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
                if (in_pml(G, m, q.z) && xband(G, m / 4 * 4)) t = t + __ldg(prof + m) * (__ldg(w + xmem(G, q.b, q.z, m / 4 * 4) + m % 4) + t);
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

// the stress step's transpose (reference kernels.cuh:664-837): lambda_v, as p,
// on the core
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
        const long long mx = xmem(G, q.b, q.z, q.x);
        keep(R.ai.m[M_VXX] + mx, R.ao.m[M_VXX] + mx, v4::ldg(G.ax + q.x), v4::ldg(qxx), on);
        keep(R.ai.m[M_VZX] + mx, R.ao.m[M_VZX] + mx, v4::ldg(G.axh + q.x), v4::ldg(qxz), on);
    }
    if (any && zband(G, q.z)) {
        const long long mz = zmem(G, q.b, q.z, q.x);
        keep(R.ai.m[M_VZZ] + mz, R.ao.m[M_VZZ] + mz, v4::splat(__ldg(G.az + q.z)), v4::ldg(qzz), on);
        keep(R.ai.m[M_VXZ] + mz, R.ao.m[M_VXZ] + mz, v4::splat(__ldg(G.azh + q.z)), v4::ldg(qxz), on);
    }
    if (!q.core) return;
    const F4 a = adj_x<M, FS, false>(G, q, qxx, R.ai.m[M_VXX], G.bx, true, true);
    const F4 b = adj_z<M, FS, true>(G, q, qxz, R.ai.m[M_VXZ], G.bzh, false, false);
    const F4 c = adj_x<M, FS, true>(G, q, qxz, R.ai.m[M_VZX], G.bxh, false, false);
    const F4 d = adj_z<M, FS, false>(G, q, qzz, R.ai.m[M_VZZ], G.bz, true, true);
    const F4 kv = v4::ldg(G.kv + q.b * G.ms + q.i);
    F4 px = v4::ld(R.p[0] + k), pz = v4::ld(R.p[1] + k);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (!q.lane(G, l)) continue;
        px.v[l] = px.v[l] + kv.v[l] * (a.v[l] + b.v[l]);
        pz.v[l] = pz.v[l] + kv.v[l] * (c.v[l] + d.v[l]);
    }
    v4::st(R.p[0] + k, px);
    v4::st(R.p[1] + k, pz);
}

// the velocity step's transpose (reference kernels.cuh:873-1019): lambda_s on
// the core, and q = dt C lambda_s
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
        const long long mx = xmem(G, q.b, q.z, q.x);
        keep(R.ai.m[M_SXXX] + mx, R.ao.m[M_SXXX] + mx, v4::ldg(G.axh + q.x), v4::ldg(px), on);
        keep(R.ai.m[M_SXZX] + mx, R.ao.m[M_SXZX] + mx, v4::ldg(G.ax + q.x), v4::ldg(pz), on);
    }
    if (any && zband(G, q.z)) {
        const long long mz = zmem(G, q.b, q.z, q.x);
        keep(R.ai.m[M_SXZZ] + mz, R.ao.m[M_SXZZ] + mz, v4::splat(__ldg(G.az + q.z)), v4::ldg(px), on);
        keep(R.ai.m[M_SZZZ] + mz, R.ao.m[M_SZZZ] + mz, v4::splat(__ldg(G.azh + q.z)), v4::ldg(pz), on);
    }
    if (!q.core) return;
    const F4 a = adj_x<M, FS, true>(G, q, px, R.ai.m[M_SXXX], G.bxh, true, false);
    const F4 b = adj_z<M, FS, true>(G, q, pz, R.ai.m[M_SZZZ], G.bzh, true, false);
    const F4 c = adj_z<M, FS, false>(G, q, px, R.ai.m[M_SXZZ], G.bz, true, true);
    const F4 d = adj_x<M, FS, false>(G, q, pz, R.ai.m[M_SXZX], G.bx, true, true);
    const F4 lam = v4::ldg(G.lam + mi), mu = v4::ldg(G.mu + mi);
    F4 sxx = v4::ld(R.a[0] + k), szz = v4::ld(R.a[1] + k), qxx, qzz, qxz = v4::ld(R.q[2] + k);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const bool on_core = q.lane(G, l);
        const bool zs = FS && fs_zrow(G, q.z), xs = FS && fs_xcol(G, q.x + l);
        const bool sh = FS && fs_zero_shear(G, q.x + l, q.z);
        // what the surfaces zero starts the step at zero (kernels.cuh:592-600)
        sxx.v[l] = (xs ? 0.f : sxx.v[l]) + (on_core ? a.v[l] : 0.f);
        szz.v[l] = (zs ? 0.f : szz.v[l]) + (on_core ? b.v[l] : 0.f);
        stiff(G.dt, lam.v[l], mu.v[l], sxx.v[l], szz.v[l], zs, xs, qxx.v[l], qzz.v[l]);
        qxz.v[l] = sh ? 0.f : on_core ? qxz.v[l] + (G.dt * mu.v[l]) * (c.v[l] + d.v[l]) : qxz.v[l];
    }
    v4::st(R.a[0] + k, sxx);
    v4::st(R.a[1] + k, szz);
    v4::st(R.q[0] + k, qxx);
    v4::st(R.q[1] + k, qzz);
    v4::st(R.q[2] + k, qxz);
}

template <int M, bool FS, bool GRP>
__global__ void __launch_bounds__(kThreads, M <= 4 ? 4 : 3) rev_a(const Geo G, const Rev R)
{
    const Cell q(G);
    if (blockIdx.z == 0) adj_vel<M, FS>(G, R, q);
    else stress_rev<M, FS, GRP>(G, R, q);
}
template <int M, bool FS, bool GRP>
__global__ void __launch_bounds__(kThreads, M <= 4 ? 4 : 3) rev_b(const Geo G, const Rev R)
{
    const Cell q(G);
    if (blockIdx.z == 0) adj_str<M, FS>(G, R, q);
    else vel_rev<M, FS, GRP>(G, R, q);
}

// the x profiles, zero past their ends
__global__ static void prep_profiles(const float* a, const float* b, const float* ah, const float* bh, int nx, int len,
                              float* out)
{
    const float* in[4] = {a, b, ah, bh};
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 4 * len; e += gridDim.x * blockDim.x) {
        const int f = e / len, c = e - f * len - kGuard;
        out[e] = c >= 0 && c < nx ? in[f][c] : 0.f;
    }
}

// Gradients on the physical box, zero elsewhere, unpitched: (B, cells) for
// per-shot models, else the sum over the slots in order.
struct Out {
    const float *vp, *vs, *rho;     // the caller's models
    float* g[3];                    // vp, vs, rho
};

__global__ static void finalize(const Geo G, const Rev R, const Out o)
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
                for (int s = 1; !G.ms && s < G.nslot; ++s) t[j] += R.g[j][s * G.S + i];
            }
            const float rho = o.rho[e];
            t[0] = -2.f * rho * o.vp[e] * t[0] * G.dt;
            t[1] = o.vs[e] != 0.f ? -2.f * t[1] / o.vs[e] : 0.f;     // mu = rho vs^2
            t[2] = t[2] / rho;
        }
        for (int j = 0; j < 3; ++j) o.g[j][e] = t[j];
    }
}

// Slab and launch geometry from the grid, box and free faces of G; shots of an
// imaging thread: as many as still leave four blocks per SM, at most four, one
// for per-shot models (max_group 1).
inline void layout(Geo& G, int max_group)
{
    G.rz0 = G.z0 + (G.fs & 1 ? 0 : 1); G.rz1 = G.z1 - (G.fs & 2 ? 0 : 1);
    G.rx0 = G.x0 + (G.fs & 4 ? 0 : 1); G.rx1 = G.x1 - (G.fs & 8 ? 0 : 1);
    G.XL = (G.x0 + 3) / 4 * 4; G.XH = std::max(G.XL, (G.x1 - 1) / 4 * 4);
    G.WX = std::max(4, G.XL + std::max(0, (G.nx + 3) / 4 * 4 - G.XH));
    G.WZ = G.z0 + G.nz - (G.z1 - 1);
    // rows of a block: 32, or 8 where that would leave the GPU with less than
    // two blocks per SM
    G.nbx = (G.nx + 31) / 32;
    G.rows = (long long)G.nbx * G.B * ((G.nz + 31) / 32) >= 2 * 148 ? 32 : 8;
    const long long blocks = (long long)G.nbx * ((G.nz + G.rows - 1) / G.rows);
    G.group = 1;
    while (G.group < max_group && G.group < G.B && blocks * ((G.B + G.group) / (G.group + 1)) >= 4LL * 148) ++G.group;
    G.nslot = (G.B + G.group - 1) / G.group;
}
inline void set_group(Geo& G, int shots)
{
    G.group = std::min(shots, G.B);
    G.nslot = (G.B + G.group - 1) / G.group;
}
inline dim3 grid_of(const Geo& G, unsigned parts)
{
    return dim3((unsigned)(G.nbx * G.B), (unsigned)((G.nz + G.rows - 1) / G.rows), parts);
}

inline long long mem_floats(const Geo& G, int k)
{
    return along_x(k) ? (long long)G.B * G.nz * G.WX : (long long)G.B * G.WZ * G.P;
}
inline int xprof_len(const Geo& G) { return G.P + 2 * kGuard; }

// the reverse kernels, for groups of shots (GRP) or a shot per thread
template <int M, bool FS>
inline void launch_a(const Geo& G, const Rev& R, cudaStream_t st)
{
    const dim3 grid = grid_of(G, 2), block(8, (unsigned)G.rows);
    if (G.group > 1) rev_a<M, FS, true><<<grid, block, 0, st>>>(G, R);
    else rev_a<M, FS, false><<<grid, block, 0, st>>>(G, R);
}
template <int M, bool FS>
inline void launch_b(const Geo& G, const Rev& R, cudaStream_t st)
{
    const dim3 grid = grid_of(G, 2), block(8, (unsigned)G.rows);
    if (G.group > 1) rev_b<M, FS, true><<<grid, block, 0, st>>>(G, R);
    else rev_b<M, FS, false><<<grid, block, 0, st>>>(G, R);
}

// Shots whose velocities the restoring thread of shot b and field `part` walks
// on the box's outermost layer: the group's from its first shot's first
// thread, so that the sum of their rho images does not depend on timing.
__device__ __forceinline__ int image_shots(const Geo& G, int b, int part)
{
    return part || b % G.group ? 0 : min(G.group, G.B - b);
}

}  // namespace evec
}  // namespace sweep
