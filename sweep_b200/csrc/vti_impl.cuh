// vti_impl.cuh -- the first-order acoustic VTI path in 2-D and 3-D (ND = 2 /
// 3): kernels templated on the dimension and the half-width M of the stencil
// (orders 2..14), and their host drivers.  vti2d.cu and vti3d.cu hold the C
// entry points' arguments.
//
// Step order (reference src/sweep/csrc/cuda/equations/acoustic_vti_1st_2d/
// and acoustic_vti_1st_3d/ kernels.cuh, forward.cu, backward.cu):
//   forward, per step: velocity step (D+ of sH along x (and y), of sV along
//     z; CPML memories on the half-cell profiles outside the physical box),
//     stress step (D- of the velocities, integer profiles; dh = dvx/dx (+
//     dvy/dy), sH += dt (c11 dh + c13 dvz/dz), sV += dt (c13 dh + c33
//     dvz/dz)), the source into every source field, the fields' boundary
//     bands, receivers;
//   reverse, per step it = nt - 1 .. 1: the residuals (unsigned), the source
//     taken back out, stress reconstruction on the box minus one cell and
//     stress bands, half-step A (p = (ph, ph, pv), ph = c11 lsH + c13 lsV, pv
//     = c13 lsH + c33 lsV, through the stress step's transposed CPML; lambda_v
//     += -dt D+ p), the gradient (forward velocities at the end of the step,
//     stresses at its start), half-step B (q = lambda_v / rho through the
//     velocity step's transposed CPML; lambda_sH += -dt (D-x qx + D-y qy),
//     lambda_sV += -dt D-z qz), velocity reconstruction and bands.
//
// The reverse step is two kernels.  Half-step A needs D- of the forward
// velocities for the reconstruction and for the stiffness gradient and takes
// p at its taps straight from lambda_s; half-step B does the same with the
// stresses, q and the 1 / rho gradient, and lambda_v is held as q = lambda_v /
// rho.  Nothing goes through memory in between (seven kernels and three scratch
// fields before), so the CPML memories of the adjoint are double-buffered: a
// cell's neighbours read them while its owner writes the next ones.  The
// gradient is summed as e = c11 lsH dh + c33 lsV dvz + c13 (lsH dvz + lsV dh),
// lsH dh, lsH dvz + lsV dh and e - lambda_v . grad s / rho (half A leaves a
// step's e for half B: the two parts cancel, so the slot takes their difference,
// not one after the other, which put the density gradient 1.07 and 1.09 times
// as far from 64 bits over 24 seeds of a 90 x 121 grid and 16 of a 40 x 36 x 44
// one); the models' chain rule is applied once, at the end.
// Shots that share a model run in groups inside a thread, which reads the
// stiffness and updates the gradient slots once per group.
//
// Four x cells per thread (vec4.cuh) on pitched rows; a warp covers 32 x 4
// (x, y) cells in 3-D and 32 x 4 (x, z) cells in 2-D.  A memory holds the cells
// where its axis has a damping profile.
//
// 4-shot 128^3 survey at order 4 (17.6 M cells): velocity step 130 us (289 us
// with one cell per thread; 87 us of field traffic at the copy rate), a reverse
// step 604 us and its bands 58 us (1110 us before; 345 us of traffic).  The
// reverse waits for loads (long scoreboard 18 to 21 an issue, DRAM at 40 and 47 %)
// at 64 registers, for which half_a spills 196 bytes, a fifth of its L1 traffic.
#pragma once

#include <algorithm>
#include <vector>

#include "bands.cuh"
#include "common.cuh"
#include "vec4.cuh"

namespace sweep {
namespace vtik {

using v4::F4;

constexpr int MAXM = 7;
constexpr int kGuard = 16;          // zero floats before and after a packed x profile
// Shots of a reverse thread, at most, and blocks per SM the kernels are
// compiled for (64 registers a thread).  Reverse step of the 4-shot 128^3
// survey at order 4: 1 / 2 / 4 shots 852 / 760 / 722 us at three blocks; no bound /
// 3 / 4 / 5 / 6 blocks at four shots 909 / 722 / 635 / 787 / 1053 us.
constexpr int kMaxGroup = 4;
constexpr int kMinBlocks = 4;
constexpr int kBY = 8, kBZ = 4;     // rows and planes of a 3-D block

enum { C11, C33, C13, IRHO };

template <int ND>
struct Lay {                        // field and memory indices
    static constexpr int NF = ND + 2, VX = 0, VZ = ND - 1, SH = ND, SV = ND + 1;
    static constexpr int NMEM = 2 * ND;   // stress-derivative memories (x[, y], z), then the velocities'
};

struct Geo {
    int B, nz, ny, nx, nt, M;       // ny = 1 in 2-D
    int P, SY, SZ;                  // row pitch, y stride (= P), z stride
    long long S;                    // shot stride
    int z0, z1, y0, y1, x0, x1;     // physical box
    int ms0[3], cut[3], wm[3];      // memory slabs by axis: first cell of the high side, cells left out, width
    int nbx;                        // x blocks
    int group, nslot;               // shots per reverse thread, gradient slots
    float dt, ihz, ihy, ihx;
    float c[MAXM + 1];              // staggered weights c[1..M]
    // profiles by axis (0 x, 1 y, 2 z): a, b at integer and at half positions,
    // zero in the stencil halo; the x ones may be read kGuard floats past their ends
    const float *a[3], *b[3], *ah[3], *bh[3];
    const float* cm[4];             // stiffness and 1 / rho, pitched, per model copy
    long long ms;                   // stride between model copies (0: one for every shot)
    int nsrc, nrec, nsf, nrf;
    int sf[5], rf[5];
    const int *src, *rec;           // (B, n, ND) runtime x[, y], z
    const float* wavelet;           // (B, nsrc, nt)
    const int* cells;               // band cells: offset in a shot's field
    int ns;
};

struct Fields {
    float* f[6];
};

// the thread's group of cells
template <int ND>
struct Cell {
    int b, z, y, x, i;              // shot (or shot group), coordinates of lane 0, offset in a shot
    bool core;                      // some lane is updated by the steps
    __device__ __forceinline__ Cell(const Geo& G)
    {
        const int xb = blockIdx.x % G.nbx;
        b = blockIdx.x / G.nbx;
        x = 4 * (xb * 8 + threadIdx.x);
        if (ND == 3) {
            y = blockIdx.y * kBY + threadIdx.y;
            z = blockIdx.z * kBZ + threadIdx.z;
        } else {
            y = 0;
            z = blockIdx.y * 32 + threadIdx.y;
        }
        i = z * G.SZ + y * G.SY + x;
        core = x + 3 >= G.M && x < G.nx - G.M && z >= G.M && z < G.nz - G.M &&
               (ND == 2 || (y >= G.M && y < G.ny - G.M));
    }
    __device__ __forceinline__ bool lane_core(const Geo& G, int l) const
    {
        return x + l >= G.M && x + l < G.nx - G.M;
    }
    // y and z inside the physical box
    __device__ __forceinline__ bool row_in(const Geo& G) const
    {
        return z >= G.z0 && z < G.z1 && (ND == 2 || (y >= G.y0 && y < G.y1));
    }
    __device__ __forceinline__ bool row_rev(const Geo& G) const
    {
        return z > G.z0 && z < G.z1 - 1 && (ND == 2 || (y > G.y0 && y < G.y1 - 1));
    }
};

__device__ __forceinline__ bool x_in(const Geo& G, int x) { return x >= G.x0 && x < G.x1; }

// Forward CPML of one derivative: m = a m + b d, d += m, on the lanes outside
// the physical box (a half-cell profile is nonzero on the box's last cell,
// where the memory runs only if another axis is outside the box).
__device__ __forceinline__ void damp(F4& d, float* m, const F4& a, const F4& b, const bool (&out)[4])
{
    const F4 old = v4::ld(m);
    F4 t;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        t.v[l] = out[l] ? a.v[l] * old.v[l] + b.v[l] * d.v[l] : 0.f;
        d.v[l] = out[l] ? d.v[l] + t.v[l] : d.v[l];
    }
    v4::st(m, t);
}

// the axis at coordinate c has a nonzero profile (half: also the box's last cell)
__device__ __forceinline__ bool band(int c, int c0, int c1, bool half) { return c < c0 || c >= c1 - (half ? 1 : 0); }
__device__ __forceinline__ bool band_x(const Geo& G, int x, bool half)
{
    return x < G.x0 || x + 3 >= G.x1 - (half ? 1 : 0);
}

// Memories: along x (B, nz, ny, wm[0]) in whole groups of four cells, along y
// (B, nz, wm[1], P), along z (B, wm[2], ny, P): the layers of the axis and the
// cells inside them that the taps of a thread near them reach, so that its taps
// lie beside its own place.  Offset of a group near the layers.
template <int ND>
__device__ __forceinline__ long long xmem(const Geo& G, int b, int z, int y, int x)
{
    return (((long long)b * G.nz + z) * (ND == 3 ? G.ny : 1) + y) * G.wm[0] + x - (x >= G.ms0[0] ? G.cut[0] : 0);
}
__device__ __forceinline__ long long ymem(const Geo& G, int b, int z, int y, int x)
{
    return (((long long)b * G.nz + z) * G.wm[1] + y - (y >= G.ms0[1] ? G.cut[1] : 0)) * G.P + x;
}
__device__ __forceinline__ long long zmem(const Geo& G, int b, int z, int y, int x)
{
    return ((long long)b * G.wm[2] + z - (z >= G.ms0[2] ? G.cut[2] : 0)) * G.SZ + y * G.SY + x;
}

// the CPML memories of the ND derivatives d[0..ND) (x[, y], z) of a forward
// step, memories w[m0 ..], profiles at half or integer positions
template <int ND, bool HALF>
__device__ __forceinline__ void damp_all(const Geo& G, const Cell<ND>& q, F4 (&d)[ND], const Fields& W, int m0)
{
    const bool rin = q.row_in(G);
    if (rin && q.x >= G.x0 && q.x + 3 < G.x1) return;
    bool out[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) out[l] = q.lane_core(G, l) && !(rin && x_in(G, q.x + l));
    if (band_x(G, q.x, HALF))
        damp(d[0], W.f[m0] + xmem<ND>(G, q.b, q.z, q.y, q.x), v4::ldg((HALF ? G.ah[0] : G.a[0]) + q.x),
             v4::ldg((HALF ? G.bh[0] : G.b[0]) + q.x), out);
    if (ND == 3 && band(q.y, G.y0, G.y1, HALF))
        damp(d[1], W.f[m0 + 1] + ymem(G, q.b, q.z, q.y, q.x), v4::splat(__ldg((HALF ? G.ah[1] : G.a[1]) + q.y)),
             v4::splat(__ldg((HALF ? G.bh[1] : G.b[1]) + q.y)), out);
    if (band(q.z, G.z0, G.z1, HALF))
        damp(d[ND - 1], W.f[m0 + ND - 1] + zmem(G, q.b, q.z, q.y, q.x),
             v4::splat(__ldg((HALF ? G.ah[2] : G.a[2]) + q.z)), v4::splat(__ldg((HALF ? G.bh[2] : G.b[2]) + q.z)), out);
}

constexpr int kThreads = 256;

// velocity step
template <int M, int ND>
__global__ void __launch_bounds__(kThreads, kMinBlocks) vel(const Geo G, const Fields F, const Fields W)
{
    using L = Lay<ND>;
    const Cell<ND> q(G);
    if (!q.core) return;
    const long long k = q.b * G.S + q.i;
    F4 d[ND];
    d[0] = v4::diff_row<M, true>(F.f[L::SH] + k, G.c, G.ihx);
    if (ND == 3) d[1] = v4::diff_col<M, true>(F.f[L::SH] + k, G.SY, G.c, G.ihy);
    d[ND - 1] = v4::diff_col<M, true>(F.f[L::SV] + k, G.SZ, G.c, G.ihz);
    const F4 ir = v4::ldg(G.cm[IRHO] + q.b * G.ms + q.i);
    F4 v[ND];
#pragma unroll
    for (int a = 0; a < ND; ++a) v[a] = v4::ld(F.f[a] + k);
    damp_all<ND, true>(G, q, d, W, 0);
#pragma unroll
    for (int a = 0; a < ND; ++a) {
#pragma unroll
        for (int l = 0; l < 4; ++l)
            if (q.lane_core(G, l)) v[a].v[l] = v[a].v[l] + (G.dt * ir.v[l]) * d[a].v[l];
        v4::st(F.f[a] + k, v[a]);
    }
}

// stress step
template <int M, int ND>
__global__ void __launch_bounds__(kThreads, kMinBlocks) str(const Geo G, const Fields F, const Fields W)
{
    using L = Lay<ND>;
    const Cell<ND> q(G);
    if (!q.core) return;
    const long long k = q.b * G.S + q.i, mi = q.b * G.ms + q.i;
    F4 d[ND];
    d[0] = v4::diff_row<M, false>(F.f[L::VX] + k, G.c, G.ihx);
    if (ND == 3) d[1] = v4::diff_col<M, false>(F.f[1] + k, G.SY, G.c, G.ihy);
    d[ND - 1] = v4::diff_col<M, false>(F.f[L::VZ] + k, G.SZ, G.c, G.ihz);
    const F4 c11 = v4::ldg(G.cm[C11] + mi), c33 = v4::ldg(G.cm[C33] + mi), c13 = v4::ldg(G.cm[C13] + mi);
    F4 sh = v4::ld(F.f[L::SH] + k), sv = v4::ld(F.f[L::SV] + k);
    damp_all<ND, false>(G, q, d, W, ND);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        if (!q.lane_core(G, l)) continue;
        const float dh = ND == 3 ? d[0].v[l] + d[1].v[l] : d[0].v[l], dz = d[ND - 1].v[l];
        sh.v[l] = sh.v[l] + G.dt * (c11.v[l] * dh + c13.v[l] * dz);
        sv.v[l] = sv.v[l] + G.dt * (c13.v[l] * dh + c33.v[l] * dz);
    }
    v4::st(F.f[L::SH] + k, sh);
    v4::st(F.f[L::SV] + k, sv);
}

struct Slots {
    float* g[4];                    // sums over time and a shot group: e, lsH dh, lsH dvz + lsV dh, e - lv . grad s / rho
    float* e;                       // e of the step at hand
};

__device__ __forceinline__ void add(float* p, const F4& a)
{
    F4 t = v4::ld(p);
#pragma unroll
    for (int l = 0; l < 4; ++l) t.v[l] += a.v[l];
    v4::st(p, t);
}

// Transposed CPML of one axis at a tap: p + b (w + p), and the owner's next
// memory a (w + p).
__device__ __forceinline__ float up(float p, float b, float w) { return p + b * (w + p); }

// Reverse half-step A: stress reconstruction (box minus one cell), the
// stiffness products of the gradient (box), lambda_v += -dt D+ p, held as q =
// lambda_v / rho (core).
// Wi / Wo: the adjoint memories of the stress step, read / written.
template <int M, int ND>
__global__ void __launch_bounds__(kThreads, kMinBlocks) half_a(const Geo G, const Fields F, const Fields A, const Fields Wi,
                                                   const Fields Wo, const Slots g)
{
    using L = Lay<ND>;
    using S = v4::Span<M, true>;
    const Cell<ND> q(G);
    if (!q.core) return;
    const bool rin = q.row_in(G), rrev = q.row_rev(G);
    const bool img = rin && q.x + 3 >= G.x0 && q.x < G.x1;
    // some tap along x reaches the x band; the rows' own band tests are per tap
    const bool bx = q.x - (M - 1) < G.x0 || q.x + 3 + M >= G.x1;
    const int b0 = q.b * G.group, b1 = min(b0 + G.group, G.B);
    F4 ge = v4::splat(0.f), g11 = ge, g13 = ge;
    for (int b = b0; b < b1; ++b) {
        const long long k = b * G.S + q.i;
        const float *c11 = G.cm[C11] + b * G.ms + q.i, *c13 = G.cm[C13] + b * G.ms + q.i,
                    *c33 = G.cm[C33] + b * G.ms + q.i;
        const float *lsh = A.f[L::SH] + k, *lsv = A.f[L::SV] + k;
        const F4 m11 = v4::ldg(c11), m13 = v4::ldg(c13), m33 = v4::ldg(c33), h0 = v4::ldg(lsh), v0 = v4::ldg(lsv);
        if (img) {
            F4 d[ND];
            d[0] = v4::diff_row<M, false>(F.f[L::VX] + k, G.c, G.ihx);
            if (ND == 3) d[1] = v4::diff_col<M, false>(F.f[1] + k, G.SY, G.c, G.ihy);
            d[ND - 1] = v4::diff_col<M, false>(F.f[L::VZ] + k, G.SZ, G.c, G.ihz);
            F4 sh = v4::ld(F.f[L::SH] + k), sv = v4::ld(F.f[L::SV] + k);
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const float dh = ND == 3 ? d[0].v[l] + d[1].v[l] : d[0].v[l], dz = d[ND - 1].v[l];
                if (x_in(G, q.x + l)) {
                    const float p11 = h0.v[l] * dh, p13 = h0.v[l] * dz + v0.v[l] * dh;
                    ge.v[l] += m11.v[l] * p11 + m33.v[l] * (v0.v[l] * dz) + m13.v[l] * p13;
                    g11.v[l] += p11;
                    g13.v[l] += p13;
                }
                if (rrev && q.x + l > G.x0 && q.x + l < G.x1 - 1) {
                    sh.v[l] = sh.v[l] - G.dt * (m11.v[l] * dh + m13.v[l] * dz);
                    sv.v[l] = sv.v[l] - G.dt * (m13.v[l] * dh + m33.v[l] * dz);
                }
            }
            if (rrev) {
                v4::st(F.f[L::SH] + k, sh);
                v4::st(F.f[L::SV] + k, sv);
            }
        }
        F4 d[ND], ph0, pv0;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            ph0.v[l] = m11.v[l] * h0.v[l] + m13.v[l] * v0.v[l];
            pv0.v[l] = m13.v[l] * h0.v[l] + m33.v[l] * v0.v[l];
        }
        {
            float p[S::N];
            const long long m = xmem<ND>(G, b, q.z, q.y, q.x);
#pragma unroll
            for (int j = -S::LO; j <= S::HI; ++j) {
                F4 t = ph0;
                if (j != 0) {
                    const F4 e = v4::ldg(c11 + 4 * j), f = v4::ldg(c13 + 4 * j), h = v4::ldg(lsh + 4 * j),
                             v = v4::ldg(lsv + 4 * j);
#pragma unroll
                    for (int l = 0; l < 4; ++l) t.v[l] = e.v[l] * h.v[l] + f.v[l] * v.v[l];
                }
                if (bx) {
                    const F4 pb = v4::ldg(G.b[0] + q.x + 4 * j), w = v4::ldg(Wi.f[ND] + m + 4 * j);
                    if (j == 0) {
                        const F4 pa = v4::ldg(G.a[0] + q.x);
                        F4 nw;
#pragma unroll
                        for (int l = 0; l < 4; ++l) nw.v[l] = pa.v[l] * (w.v[l] + t.v[l]);
                        if (band_x(G, q.x, false)) v4::st(Wo.f[ND] + m, nw);
                    }
#pragma unroll
                    for (int l = 0; l < 4; ++l)
                        t.v[l] = up(t.v[l], pb.v[l], w.v[l]);
                }
#pragma unroll
                for (int l = 0; l < 4; ++l) p[4 * (j + S::LO) + l] = t.v[l];
            }
            d[0] = v4::diff_x<M, true, S::O>(p, G.c, G.ihx);
        }
        // a row tap along an axis: p there, and within the band's reach (`near`)
        // through its memory -- a tap off the band with the profile's zero, so
        // that a thread's loads leave together
        auto tap = [&](int off, int c, const float* prof, const float* mem, const float* ca, const float* cb, F4 own,
                       bool centre, bool near) {
            F4 t = own;
            if (!centre) {
                const F4 e = v4::ldg(ca + off), f = v4::ldg(cb + off), h = v4::ldg(lsh + off), v = v4::ldg(lsv + off);
#pragma unroll
                for (int l = 0; l < 4; ++l) t.v[l] = e.v[l] * h.v[l] + f.v[l] * v.v[l];
            }
            if (near) {
                const float pb = __ldg(prof + c);
                const F4 w = v4::ldg(mem);
#pragma unroll
                for (int l = 0; l < 4; ++l) t.v[l] = up(t.v[l], pb, w.v[l]);
            }
            return t;
        };
        auto rows = [&](int stride, int c, const float* prof, auto place, const float* ca, const float* cb, const F4& own,
                        bool near, float inv) {
            if (near) {
                const float* mem = place();
                return v4::diff<M, true>(
                    [&](int j) { return tap(j * stride, c + j, prof, mem + j * stride, ca, cb, own, j == 0, true); }, G.c,
                    inv);
            }
            return v4::diff<M, true>(
                [&](int j) { return tap(j * stride, c + j, prof, nullptr, ca, cb, own, j == 0, false); }, G.c, inv);
        };
        if (ND == 3) {
            d[1] = rows(G.SY, q.y, G.b[1], [&] { return Wi.f[ND + 1] + ymem(G, b, q.z, q.y, q.x); }, c11, c13, ph0,
                        band(q.y - (M - 1), G.y0, G.y1, false) || band(q.y + M, G.y0, G.y1, false), G.ihy);
            if (band(q.y, G.y0, G.y1, false)) {
                const float pa = __ldg(G.a[1] + q.y);
                const long long o = ymem(G, b, q.z, q.y, q.x);
                F4 w = v4::ldg(Wi.f[ND + 1] + o);
#pragma unroll
                for (int l = 0; l < 4; ++l) w.v[l] = q.lane_core(G, l) ? pa * (w.v[l] + ph0.v[l]) : 0.f;
                v4::st(Wo.f[ND + 1] + o, w);
            }
        }
        d[ND - 1] = rows(G.SZ, q.z, G.b[2], [&] { return Wi.f[2 * ND - 1] + zmem(G, b, q.z, q.y, q.x); }, c13, c33, pv0,
                         band(q.z - (M - 1), G.z0, G.z1, false) || band(q.z + M, G.z0, G.z1, false), G.ihz);
        if (band(q.z, G.z0, G.z1, false)) {
            const float pa = __ldg(G.a[2] + q.z);
            const long long o = zmem(G, b, q.z, q.y, q.x);
            F4 w = v4::ldg(Wi.f[2 * ND - 1] + o);
#pragma unroll
            for (int l = 0; l < 4; ++l) w.v[l] = q.lane_core(G, l) ? pa * (w.v[l] + pv0.v[l]) : 0.f;
            v4::st(Wo.f[2 * ND - 1] + o, w);
        }
        const F4 ir = v4::ldg(G.cm[IRHO] + b * G.ms + q.i);
#pragma unroll
        for (int a = 0; a < ND; ++a) {
            F4 v = v4::ld(A.f[a] + k);
#pragma unroll
            for (int l = 0; l < 4; ++l)
                if (q.lane_core(G, l)) v.v[l] += (-G.dt * ir.v[l]) * d[a].v[l];
            v4::st(A.f[a] + k, v);
        }
    }
    if (img) {
        const long long s = q.b * G.S + q.i;
        add(g.g[0] + s, ge);
        add(g.g[1] + s, g11);
        add(g.g[2] + s, g13);
        v4::st(g.e + s, ge);
    }
}

// Reverse half-step B: velocity reconstruction (box minus one cell), the
// 1 / rho product of the gradient (box), lambda_s += -dt D- q (core).
template <int M, int ND>
__global__ void __launch_bounds__(kThreads, kMinBlocks) half_b(const Geo G, const Fields F, const Fields A, const Fields Wi,
                                                   const Fields Wo, const Slots g)
{
    using L = Lay<ND>;
    using S = v4::Span<M, false>;
    const Cell<ND> q(G);
    if (!q.core) return;
    const bool rin = q.row_in(G), rrev = q.row_rev(G);
    const bool img = rin && q.x + 3 >= G.x0 && q.x < G.x1;
    const bool zin = q.z >= G.z0 && q.z < G.z1, yin = ND == 2 || (q.y >= G.y0 && q.y < G.y1);
    const bool bx = q.x - M < G.x0 || q.x + 3 + M - 1 >= G.x1 - 1;
    const int b0 = q.b * G.group, b1 = min(b0 + G.group, G.B);
    F4 gr = v4::splat(0.f);
    for (int b = b0; b < b1; ++b) {
        const long long k = b * G.S + q.i;
        F4 q0[ND];
#pragma unroll
        for (int a = 0; a < ND; ++a) q0[a] = v4::ldg(A.f[a] + k);
        if (img) {
            F4 d[ND];
            d[0] = v4::diff_row<M, true>(F.f[L::SH] + k, G.c, G.ihx);
            if (ND == 3) d[1] = v4::diff_col<M, true>(F.f[L::SH] + k, G.SY, G.c, G.ihy);
            d[ND - 1] = v4::diff_col<M, true>(F.f[L::SV] + k, G.SZ, G.c, G.ihz);
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (!x_in(G, q.x + l)) continue;
                float s = q0[0].v[l] * d[0].v[l];
#pragma unroll
                for (int a = 1; a < ND; ++a) s += q0[a].v[l] * d[a].v[l];
                gr.v[l] -= s;
            }
            if (rrev) {
                const F4 r0 = v4::ldg(G.cm[IRHO] + b * G.ms + q.i);
#pragma unroll
                for (int a = 0; a < ND; ++a) {
                    F4 v = v4::ld(F.f[a] + k);
#pragma unroll
                    for (int l = 0; l < 4; ++l)
                        if (q.x + l > G.x0 && q.x + l < G.x1 - 1) v.v[l] = v.v[l] - (G.dt * r0.v[l]) * d[a].v[l];
                    v4::st(F.f[a] + k, v);
                }
            }
        }
        F4 d[ND];
        {
            float p[S::N];
            const long long m = xmem<ND>(G, b, q.z, q.y, q.x);
#pragma unroll
            for (int j = -S::LO; j <= S::HI; ++j) {
                F4 t = j == 0 ? q0[0] : v4::ldg(A.f[0] + k + 4 * j);
                if (bx) {
                    const F4 pb = v4::ldg(G.bh[0] + q.x + 4 * j), w = v4::ldg(Wi.f[0] + m + 4 * j);
                    if (j == 0 && band_x(G, q.x, true)) {
                        const F4 pa = v4::ldg(G.ah[0] + q.x);
                        F4 nw;
#pragma unroll
                        for (int l = 0; l < 4; ++l)
                            nw.v[l] = rin && x_in(G, q.x + l) ? 0.f : pa.v[l] * (w.v[l] + t.v[l]);
                        v4::st(Wo.f[0] + m, nw);
                    }
#pragma unroll
                    for (int l = 0; l < 4; ++l)
                        t.v[l] = up(t.v[l], rin && x_in(G, q.x + 4 * j + l) ? 0.f : pb.v[l], w.v[l]);
                }
#pragma unroll
                for (int l = 0; l < 4; ++l) p[4 * (j + S::LO) + l] = t.v[l];
            }
            d[0] = v4::diff_x<M, false, S::O>(p, G.c, G.ihx);
        }
        // a row tap along y or z (see half_a); in: the row at c + j and the other
        // of y and z lie in the box, where the memory runs outside it along x only
        auto rows = [&](int stride, int c, int c0, int c1, bool oin, const float* prof, auto place, const float* lam,
                        const F4& own, float inv) {
            auto value = [&](int j) { return j == 0 ? own : v4::ldg(lam + j * stride); };
            if (!band(c - M, c0, c1, true) && !band(c + M - 1, c0, c1, true)) return v4::diff<M, false>(value, G.c, inv);
            const float* mem = place();
            return v4::diff<M, false>(
                [&](int j) {
                    F4 t = value(j);
                    const bool in = oin && c + j >= c0 && c + j < c1;
                    const float pb = __ldg(prof + c + j);
                    const F4 w = v4::ldg(mem + j * stride);
#pragma unroll
                    for (int l = 0; l < 4; ++l) t.v[l] = up(t.v[l], in && x_in(G, q.x + l) ? 0.f : pb, w.v[l]);
                    return t;
                },
                G.c, inv);
        };
        auto keep = [&](int mem, long long o, float pa, const F4& own) {
            F4 w = v4::ldg(Wi.f[mem] + o);
#pragma unroll
            for (int l = 0; l < 4; ++l)
                w.v[l] = q.lane_core(G, l) && !(rin && x_in(G, q.x + l)) ? pa * (w.v[l] + own.v[l]) : 0.f;
            v4::st(Wo.f[mem] + o, w);
        };
        if (ND == 3) {
            d[1] = rows(G.SY, q.y, G.y0, G.y1, zin, G.bh[1], [&] { return Wi.f[1] + ymem(G, b, q.z, q.y, q.x); },
                        A.f[1] + k, q0[1], G.ihy);
            if (band(q.y, G.y0, G.y1, true)) keep(1, ymem(G, b, q.z, q.y, q.x), __ldg(G.ah[1] + q.y), q0[1]);
        }
        d[ND - 1] = rows(G.SZ, q.z, G.z0, G.z1, yin, G.bh[2],
                         [&] { return Wi.f[ND - 1] + zmem(G, b, q.z, q.y, q.x); }, A.f[L::VZ] + k, q0[ND - 1], G.ihz);
        if (band(q.z, G.z0, G.z1, true)) keep(ND - 1, zmem(G, b, q.z, q.y, q.x), __ldg(G.ah[2] + q.z), q0[ND - 1]);
        F4 sh = v4::ld(A.f[L::SH] + k), sv = v4::ld(A.f[L::SV] + k);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            if (!q.lane_core(G, l)) continue;
            sh.v[l] += -G.dt * (ND == 3 ? d[0].v[l] + d[1].v[l] : d[0].v[l]);
            sv.v[l] += -G.dt * d[ND - 1].v[l];
        }
        v4::st(A.f[L::SH] + k, sh);
        v4::st(A.f[L::SV] + k, sv);
    }
    if (img) {
        const long long s = q.b * G.S + q.i;
        const F4 e = v4::ld(g.e + s);
#pragma unroll
        for (int l = 0; l < 4; ++l) gr.v[l] += e.v[l];
        add(g.g[3] + s, gr);
    }
}

// ------------------------------------------------ sources, receivers, bands
// offset of location l (x[, y], z) in a shot's field, or -1 off the grid
template <int ND>
__device__ __forceinline__ int loc(const Geo& G, const int* l)
{
    const int x = l[0], y = ND == 3 ? l[1] : 0, z = l[ND - 1];
    if (x < 0 || x >= G.nx || y < 0 || y >= G.ny || z < 0 || z >= G.nz) return -1;
    return z * G.SZ + y * G.SY + x;
}

// the wavelet of step it, times sign, into every source field
template <int ND>
__device__ __forceinline__ void inject_at(const Geo& G, const Fields& F, int e, int it, float sign)
{
    const int c = loc<ND>(G, G.src + (long long)ND * e);
    if (c < 0) return;
    const float w = sign * G.wavelet[(long long)e * G.nt + it];
    for (int k = 0; k < G.nsf; ++k) atomicAdd(F.f[G.sf[k]] + e / G.nsrc * G.S + c, w);
}

template <int ND>
__global__ void inject(const Geo G, const Fields F, int it)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < G.B * G.nsrc) inject_at<ND>(G, F, e, it, 1.f);
}

// reverse: the source of step it taken out of F, the residuals (unsigned)
// into the adjoint fields (the velocities' as q)
template <int ND>
__global__ void events(const Geo G, const Fields F, const Fields A, const float* __restrict__ adj, int it)
{
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < G.B * G.nsrc) { inject_at<ND>(G, F, e, it, -1.f); return; }
    e -= G.B * G.nsrc;
    if (e >= G.B * G.nrec) return;
    const int b = e / G.nrec, r = e - b * G.nrec;
    const int c = loc<ND>(G, G.rec + (long long)ND * e);
    if (c < 0) return;
    const float* res = adj + (((long long)b * G.nt + it) * G.nrec + r) * G.nrf;
    for (int k = 0; k < G.nrf; ++k) {
        const int f = G.rf[k];
        atomicAdd(A.f[f] + b * G.S + c, f < Lay<ND>::SH ? G.cm[IRHO][b * G.ms + c] * res[k] : res[k]);
    }
}

// forward: record[b, it, r, k] = field rf[k] at receiver r (slot and record
// optional), and every field's bands into one step slot (B, NF, ns)
template <int ND>
__global__ void save(const Geo G, const Fields F, float* record, float* slot, int it)
{
    constexpr int NF = Lay<ND>::NF;
    long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nr = record ? (long long)G.B * G.nrec : 0;
    if (e < nr) {
        const int b = (int)(e / G.nrec), r = (int)(e - (long long)b * G.nrec);
        const int c = loc<ND>(G, G.rec + ND * e);
        if (c < 0) return;
        float* out = record + (((long long)b * G.nt + it) * G.nrec + r) * G.nrf;
        for (int k = 0; k < G.nrf; ++k) out[k] = F.f[G.rf[k]][b * G.S + c];
        return;
    }
    e -= nr;
    if (!slot || e >= (long long)G.B * G.ns) return;
    const int b = (int)(e / G.ns), n = (int)(e - (long long)b * G.ns);
    const long long k = b * G.S + __ldg(G.cells + n);
#pragma unroll
    for (int f = 0; f < NF; ++f) slot[(long long)(b * NF + f) * G.ns + n] = F.f[f][k];
}

// fields [f0, f1) of the bands from a step slot
template <int ND>
__global__ void restore(const Geo G, const Fields F, const float* __restrict__ slot, int f0, int f1)
{
    constexpr int NF = Lay<ND>::NF;
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)G.B * G.ns) return;
    const int b = (int)(e / G.ns), n = (int)(e - (long long)b * G.ns);
    const long long k = b * G.S + __ldg(G.cells + n);
    for (int f = f0; f < f1; ++f) F.f[f][k] = __ldg(slot + (long long)(b * NF + f) * G.ns + n);
}

// -------------------------------------------------------------- per call
// stiffness per model copy, pitched, each operation rounded once (reference
// derived_models.cu:40-53)
__global__ static void prep(const float* __restrict__ vp, const float* __restrict__ eps, const float* __restrict__ dlt,
                     const float* __restrict__ rho, long long rows, int nx, int P, float* c11, float* c33, float* c13,
                     float* irho)
{
    const long long n = rows * P;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long row = k / P;
        const int x = (int)(k - row * P);
        if (x >= nx) { c11[k] = c33[k] = c13[k] = irho[k] = 0.f; continue; }
        const long long i = row * nx + x;
        const float v = vp[i], r = rho[i];
        const float rv2 = __fmul_rn(r, __fmul_rn(v, v));
        c33[k] = rv2;
        c11[k] = __fmul_rn(rv2, __fadd_rn(1.0f, __fmul_rn(2.0f, eps[i])));
        c13[k] = __fmul_rn(rv2, __fsqrt_rn(__fadd_rn(1.0f, __fmul_rn(2.0f, dlt[i]))));
        irho[k] = __fdiv_rn(1.0f, r);
    }
}

// one axis's four profiles on the cells the steps update, zero elsewhere
__global__ static void prep_profiles(const float* a, const float* b, const float* ah, const float* bh, int n, int M, int lead,
                              int len, float* out)
{
    const float* in[4] = {a, b, ah, bh};
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 4 * len; e += gridDim.x * blockDim.x) {
        const int f = e / len, c = e - f * len - lead;
        out[e] = c >= M && c < n - M ? in[f][c] : 0.f;
    }
}

// Gradients on the physical box, zero elsewhere, from the summed products
// (reference kernels.cuh:822-912 chain rule): (B, cells) for per-shot models,
// else the sum over the slots in order.
struct Models {
    const float *vp, *eps, *dlt, *rho;
};
struct Grads {
    float* g[4];                    // vp, epsilon, delta, rho
};

template <int ND>
__global__ void finalize(const Geo G, const Slots s, const Models m, const Grads out)
{
    const long long cells = (long long)G.nz * G.ny * G.nx;
    const long long n = (G.ms ? G.B : 1) * cells;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long b = e / cells;
        const int c = (int)(e - b * cells);
        const int x = c % G.nx, r = c / G.nx, y = r % G.ny, z = r / G.ny;
        float gv = 0.f, ge = 0.f, gd = 0.f, gp = 0.f;
        if (x_in(G, x) && z >= G.z0 && z < G.z1 && (ND == 2 || (y >= G.y0 && y < G.y1))) {
            const int i = z * G.SZ + y * G.SY + x;
            float t[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (G.ms) {
                    t[j] = s.g[j][b * G.S + i];
                } else {
                    t[j] = s.g[j][i];
                    for (int k = 1; k < G.nslot; ++k) t[j] += s.g[j][k * G.S + i];
                }
                t[j] *= G.dt;
            }
            // c11 = c33 (1 + 2 eps), c13 = c33 sqrt(1 + 2 delta), c33 = rho v^2;
            // in vacuum (v = 0) every stiffness is zero, so t[0] is
            const float v = m.vp[e], rho = m.rho[e], rv2 = rho * (v * v);
            gv = v != 0.f ? 2.f * t[0] / v : 0.f;
            ge = 2.f * t[1] * rv2;
            gd = t[2] * rv2 / fmaxf(sqrtf(1.f + 2.f * m.dlt[e]), 1e-12f);
            gp = t[3] / rho;
        }
        out.g[0][e] = gv;
        out.g[1][e] = ge;
        out.g[2][e] = gd;
        out.g[3][e] = gp;
    }
}

// ------------------------------------------------------------------- host
// What the C descriptors of the 2-D and the 3-D equation hold.
struct Desc {
    int B, nz, ny, nx, nt, M;
    int pad[6];                     // z_lo, z_hi, y_lo, y_hi, x_lo, x_hi
    float dt, dz, dy, dx;
    const float* prof[3][4];        // by axis (x, y, z): a, b, a_half, b_half
    Models m;
    int64_t model_stride;
    int nsrc, nrec, nsf, nrf;
    const int32_t *sf, *rf;
    const int *src, *rec;
    const float* wavelet;
};

struct Plan {
    Geo G;
    bands::Bands bands;
    int nm;                         // model copies
    const char* name;
};

template <int ND>
Plan make_plan(const Desc& d, int mem_mode, const char* name)
{
    constexpr int NF = Lay<ND>::NF;
    SWEEP_REQUIRE(d.M >= 1 && d.M <= MAXM, "%s: spatial orders 2 to %d are built (got order %d)", name, 2 * MAXM,
                  2 * d.M);
    SWEEP_REQUIRE(mem_mode == SWEEP_MEM_BOUNDARY,
                  "%s: boundary saving with fp32 strips in device memory is built (mem_mode %d)", name, mem_mode);
    SWEEP_REQUIRE(d.nsrc >= 0 && d.nrec >= 0, "%s: negative source/receiver count", name);
    SWEEP_REQUIRE(d.nsf >= 1 && d.nsf <= NF, "%s: 1 to %d source fields", name, NF);
    SWEEP_REQUIRE(d.nrf >= 1 && d.nrf <= NF, "%s: 1 to %d receiver fields", name, NF);
    for (int k = 0; k < d.nsf; ++k) {
        SWEEP_REQUIRE(d.sf[k] >= 0 && d.sf[k] < NF, "%s: bad source field %d", name, d.sf[k]);
        for (int j = 0; j < k; ++j) SWEEP_REQUIRE(d.sf[j] != d.sf[k], "%s: source field %d repeated", name, d.sf[k]);
    }
    for (int k = 0; k < d.nrf; ++k)
        SWEEP_REQUIRE(d.rf[k] >= 0 && d.rf[k] < NF, "%s: bad receiver field %d", name, d.rf[k]);
    for (int f = 0; f < 6; ++f)
        if (ND == 3 || f < 2 || f > 3)
            SWEEP_REQUIRE(d.pad[f] >= 1, "%s: every face needs a PML pad >= 1 (face %d has %d)", name,
                          ND == 2 && f > 3 ? f - 2 : f, d.pad[f]);
    Plan pl{};
    pl.name = name;
    Geo& G = pl.G;
    const int M = d.M;
    G.B = d.B; G.nz = d.nz; G.ny = d.ny; G.nx = d.nx; G.nt = d.nt; G.M = M;
    const long long cells = (long long)d.nz * d.ny * d.nx;
    G.P = (d.nx + 7) / 8 * 8;
    G.S = (long long)d.nz * d.ny * G.P;
    SWEEP_REQUIRE(cells < (1LL << 31) && G.S < (1LL << 31), "%s: one shot's grid must hold < 2^31 cells", name);
    G.SY = G.P; G.SZ = d.ny * G.P;
    G.z0 = d.pad[0] + M; G.z1 = G.nz - d.pad[1] - M;
    G.y0 = ND == 3 ? d.pad[2] + M : 0; G.y1 = ND == 3 ? G.ny - d.pad[3] - M : 1;
    G.x0 = d.pad[4] + M; G.x1 = G.nx - d.pad[5] - M;
    SWEEP_REQUIRE(G.z1 - G.z0 >= 2 && (ND == 2 || G.y1 - G.y0 >= 2) && G.x1 - G.x0 >= 2,
                  "%s: the physical box must be at least 2 cells per axis", name);
    G.dt = d.dt; G.ihz = 1.f / d.dz; G.ihy = 1.f / d.dy; G.ihx = 1.f / d.dx;
    v4::staggered_weights(M, G.c);
    const bool per_shot = d.model_stride != 0;
    SWEEP_REQUIRE(!per_shot || d.model_stride == cells, "%s: model_stride must be 0 or the cells of a shot", name);
    G.ms = per_shot ? G.S : 0;
    pl.nm = per_shot ? G.B : 1;
    G.nsrc = d.nsrc; G.nrec = d.nrec; G.nsf = d.nsf; G.nrf = d.nrf;
    for (int k = 0; k < NF; ++k) { G.sf[k] = d.sf[k]; G.rf[k] = d.rf[k]; }
    G.src = d.src; G.rec = d.rec; G.wavelet = d.wavelet;
    // a thread within M cells of the layers reads memories up to M cells (along
    // x: the groups of those) further in
    auto slab = [&](int a, int c0, int c1, int n, int reach, int unit) {
        const int low = (c0 + reach + unit - 1) / unit * unit, high = std::max(0, c1 - 1 - reach) / unit * unit;
        G.ms0[a] = high;
        G.cut[a] = std::max(0, high - low);
        G.wm[a] = (n + unit - 1) / unit * unit - G.cut[a];
    };
    slab(0, G.x0, G.x1, G.nx, M + 4 * v4::groups(M) + 4, 4);
    slab(1, G.y0, G.y1, G.ny, 2 * M, 1);
    slab(2, G.z0, G.z1, G.nz, 2 * M, 1);
    G.nbx = (G.nx + 31) / 32;
    // shots per reverse thread: as many as still leave four blocks per SM;
    // one for per-shot models
    const long long blocks = (long long)G.nbx * (ND == 3 ? (long long)((G.ny + 7) / 8) * ((G.nz + 3) / 4) : (G.nz + 31) / 32);
    G.group = 1;
    if (!per_shot)
        while (G.group < kMaxGroup && G.group < G.B && blocks * ((G.B + G.group) / (G.group + 1)) >= 4LL * 148) ++G.group;
    G.nslot = (G.B + G.group - 1) / G.group;
    pl.bands = bands::make<ND>(M, G.z0, G.z1, G.y0, G.y1, G.x0, G.x1);
    G.ns = pl.bands.count;
    return pl;
}

struct Ws {
    float* cm[4];
    float* prof[3];
    int* cells;
    float* f[5];
    float* m[2][6];                 // forward: [0]; reverse: the adjoint's, double-buffered
    float* a[5];
    float* g[4];
    float* e;
    char *zero0, *zero1;
};

// memory k: x[, y], z of the stress derivatives, then of the velocities'
template <int ND>
long long mem_floats(const Geo& G, int k)
{
    const int a = k % ND;
    return a == 0        ? (long long)G.B * G.nz * G.ny * G.wm[0]
           : a == ND - 1 ? (long long)G.B * G.wm[2] * G.SZ
                         : (long long)G.B * G.nz * G.wm[1] * G.P;
}

template <int ND>
void carve(Carve& c, const Plan& pl, bool rev, Ws& w)
{
    using L = Lay<ND>;
    const Geo& G = pl.G;
    const long long n = (long long)G.B * G.S;
    w = Ws{};
    for (float*& p : w.cm) p = c.take<float>(pl.nm * G.S);
    const int len[3] = {G.P + 2 * kGuard, G.ny, G.nz};
    for (int a = 0; a < 3; ++a) w.prof[a] = c.take<float>(4LL * len[a]);
    w.cells = c.take<int>(std::max(G.ns, 1));
    c.take<char>(0);
    w.zero0 = c.base ? c.base + c.off : nullptr;
    for (int k = 0; k < L::NF; ++k) w.f[k] = c.take<float>(n);
    for (int s = 0; s < (rev ? 2 : 1); ++s)
        for (int k = 0; k < L::NMEM; ++k) w.m[s][k] = c.take<float>(mem_floats<ND>(G, k));
    if (rev) {
        for (int k = 0; k < L::NF; ++k) w.a[k] = c.take<float>(n);
        for (float*& p : w.g) p = c.take<float>(G.nslot * G.S);
    }
    c.take<char>(0);
    w.zero1 = c.base ? c.base + c.off : nullptr;
    if (rev) w.e = c.take<float>(G.nslot * G.S);
}

template <int ND>
long long slot_floats(const Plan& pl) { return (long long)pl.G.B * Lay<ND>::NF * pl.G.ns; }

// rows of a field of every shot
inline long long rows_of(const Geo& G) { return (long long)G.B * G.nz * G.ny; }

template <int ND>
void sizes(const Plan& pl, int64_t* ws_bytes, int64_t* tape_bytes)
{
    Carve f(nullptr), r(nullptr);
    Ws w;
    carve<ND>(f, pl, false, w);
    carve<ND>(r, pl, true, w);
    *ws_bytes = std::max(f.off, r.off);
    *tape_bytes = ((long long)pl.G.nt * slot_floats<ND>(pl) + Lay<ND>::NF * rows_of(pl.G) * pl.G.nx) * 4;
}

inline unsigned blocks(long long n) { return (unsigned)std::max<long long>((n + 255) / 256, 1); }

template <int ND>
void setup(const Desc& d, Plan& pl, const Ws& w, cudaStream_t st)
{
    Geo& G = pl.G;
    for (int k = 0; k < 4; ++k) G.cm[k] = w.cm[k];
    G.cells = w.cells;
    const long long rows = (long long)pl.nm * G.nz * G.ny;
    prep<<<std::min(blocks(rows * G.P), 4096u), 256, 0, st>>>(d.m.vp, d.m.eps, d.m.dlt, d.m.rho, rows, G.nx, G.P,
                                                              w.cm[C11], w.cm[C33], w.cm[C13], w.cm[IRHO]);
    const int n[3] = {G.nx, G.ny, G.nz};
    for (int a = 0; a < 3; ++a) {
        if (ND == 2 && a == 1) continue;
        const int lead = a == 0 ? kGuard : 0, len = a == 0 ? G.P + 2 * kGuard : n[a];
        prep_profiles<<<std::min(blocks(4LL * len), 64u), 256, 0, st>>>(d.prof[a][0], d.prof[a][1], d.prof[a][2],
                                                                        d.prof[a][3], n[a], G.M, lead, len, w.prof[a]);
        G.a[a] = w.prof[a] + lead; G.b[a] = G.a[a] + len;
        G.ah[a] = G.b[a] + len; G.bh[a] = G.ah[a] + len;
    }
    bands::band_table<ND><<<std::min(blocks(G.ns), 1024u), 256, 0, st>>>(pl.bands, G.SY, G.SZ, w.cells);
    SWEEP_LAUNCH_CHECK();
    SWEEP_CUDA(cudaMemsetAsync(w.zero0, 0, w.zero1 - w.zero0, st));
}

template <int ND>
dim3 grid_of(const Geo& G, int nb)
{
    if (ND == 3) return dim3((unsigned)(G.nbx * nb), (G.ny + kBY - 1) / kBY, (G.nz + kBZ - 1) / kBZ);
    return dim3((unsigned)(G.nbx * nb), (G.nz + 31) / 32);
}

template <int ND>
dim3 block_of() { return ND == 3 ? dim3(8, kBY, kBZ) : dim3(8, 32); }

template <int M, int ND>
void forward(const Desc& d, Plan& pl, float* record, void* tape, void* ws, int64_t ws_bytes, cudaStream_t st)
{
    using L = Lay<ND>;
    Carve c(ws);
    Ws w;
    carve<ND>(c, pl, false, w);
    SWEEP_REQUIRE(ws != nullptr && c.off <= ws_bytes, "%s forward: workspace too small (%lld < %lld bytes)", pl.name,
                  (long long)ws_bytes, (long long)c.off);
    setup<ND>(d, pl, w, st);
    const Geo& G = pl.G;
    if (G.nrec == 0) record = nullptr;
    if (record) SWEEP_CUDA(cudaMemsetAsync(record, 0, sizeof(float) * (size_t)G.B * G.nt * G.nrec * G.nrf, st));
    Fields F{}, W{};
    for (int k = 0; k < L::NF; ++k) F.f[k] = w.f[k];
    for (int k = 0; k < L::NMEM; ++k) W.f[k] = w.m[0][k];
    float* tp = static_cast<float*>(tape);
    const dim3 grid = grid_of<ND>(G, G.B), block = block_of<ND>();
    const long long nsave = (record ? (long long)G.B * G.nrec : 0) + (tp ? (long long)G.B * G.ns : 0);
    StepGraphs sg(st, resolve_graph_steps(-1));
    for (int it = 0; it < G.nt; ++it) {
        cudaStream_t s = sg.stream();
        vel<M, ND><<<grid, block, 0, s>>>(G, F, W);
        str<M, ND><<<grid, block, 0, s>>>(G, F, W);
        if (G.nsrc > 0) inject<ND><<<(G.B * G.nsrc + 127) / 128, 128, 0, s>>>(G, F, it);
        if (nsave > 0)
            save<ND><<<blocks(nsave), 256, 0, s>>>(G, F, record, tp ? tp + it * slot_floats<ND>(pl) : nullptr, it);
        SWEEP_LAUNCH_CHECK();
        sg.step_done();
    }
    sg.flush();
    if (tp) {
        float* last = tp + (long long)G.nt * slot_floats<ND>(pl);
        for (int f = 0; f < L::NF; ++f) copy_rows(last + f * rows_of(G) * G.nx, G.nx, w.f[f], G.P, G.nx, rows_of(G), st);
    }
}

template <int M, int ND>
void backward(const Desc& d, Plan& pl, const float* adj, const void* tape, const Grads& out, void* ws,
              int64_t ws_bytes, cudaStream_t st)
{
    using L = Lay<ND>;
    SWEEP_REQUIRE(tape != nullptr, "%s backward: the forward's tape is required", pl.name);
    Carve c(ws);
    Ws w;
    carve<ND>(c, pl, true, w);
    SWEEP_REQUIRE(ws != nullptr && c.off <= ws_bytes, "%s backward: workspace too small (%lld < %lld bytes)", pl.name,
                  (long long)ws_bytes, (long long)c.off);
    setup<ND>(d, pl, w, st);
    const Geo& G = pl.G;
    const float* tp = static_cast<const float*>(tape);
    const float* last = tp + (long long)G.nt * slot_floats<ND>(pl);
    for (int f = 0; f < L::NF; ++f) copy_rows(w.f[f], G.P, last + f * rows_of(G) * G.nx, G.nx, G.nx, rows_of(G), st);
    Fields F{}, A{}, W[2]{};
    for (int k = 0; k < L::NF; ++k) { F.f[k] = w.f[k]; A.f[k] = w.a[k]; }
    for (int k = 0; k < L::NMEM; ++k) { W[0].f[k] = w.m[0][k]; W[1].f[k] = w.m[1][k]; }
    const Slots g{{w.g[0], w.g[1], w.g[2], w.g[3]}, w.e};
    const dim3 grid = grid_of<ND>(G, G.nslot), block = block_of<ND>();
    const long long ne = (long long)G.B * G.nsrc + (long long)G.B * G.nrec;
    const unsigned bb = blocks((long long)G.B * G.ns);
    int cur = 0;
    StepGraphs sg(st, resolve_graph_steps(-1));
    for (int it = G.nt - 1; it >= 1; --it) {
        cudaStream_t s = sg.stream();
        const float* prev = tp + (long long)(it - 1) * slot_floats<ND>(pl);
        if (ne > 0) events<ND><<<(unsigned)((ne + 127) / 128), 128, 0, s>>>(G, F, A, adj, it);
        half_a<M, ND><<<grid, block, 0, s>>>(G, F, A, W[cur], W[cur ^ 1], g);
        restore<ND><<<bb, 256, 0, s>>>(G, F, prev, L::SH, L::NF);
        half_b<M, ND><<<grid, block, 0, s>>>(G, F, A, W[cur], W[cur ^ 1], g);
        restore<ND><<<bb, 256, 0, s>>>(G, F, prev, 0, L::SH);
        SWEEP_LAUNCH_CHECK();
        cur ^= 1;
        sg.step_done();
    }
    sg.flush();
    const long long cells = (long long)pl.nm * G.nz * G.ny * G.nx;
    finalize<ND><<<std::min(blocks(cells), 8192u), 256, 0, st>>>(G, g, d.m, out);
    SWEEP_LAUNCH_CHECK();
}

#define SWEEP_VTI_DISPATCH(M_, CALL) \
    switch (M_) {                    \
    case 1: CALL(1); break;          \
    case 2: CALL(2); break;          \
    case 3: CALL(3); break;          \
    case 4: CALL(4); break;          \
    case 5: CALL(5); break;          \
    case 6: CALL(6); break;          \
    default: CALL(7); break;         \
    }

}  // namespace vtik
}  // namespace sweep
