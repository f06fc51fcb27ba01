// acoustic_vec.cuh -- the acoustic steps on four x cells per thread (vec4.cuh),
// for any half-width M and in 2-D (ND = 2) and 3-D (ND = 3): the forward step,
// the adjoint step and the reconstruction of one group of cells, with the CPML
// of an axis only where its profile reaches.  Shared by the kernels of the
// orders other than 8 (acoustic_orders.cu) and by the 2-D order-8 kernels of
// small grids (acoustic2d.cu).
#pragma once

#include "common.cuh"
#include "vec4.cuh"

namespace sweep {
namespace avec {

using v4::F4;

constexpr int MAXM = 7;
constexpr int kGuard = 16;          // zero floats before and after a packed x profile
constexpr int kBY = 8, kBZ = 4;     // rows and planes of a 3-D block

struct Geo {
    int nd, B, nz, ny, nx, nt, M;   // ny = 1 in 2-D
    int P, SY, SZ;                  // row pitch, y stride (= P), z stride
    long long S;                    // shot stride
    int lo[3], hi[3];               // physical box by axis (0 x, 1 y, 2 z)
    int rlo[3], rhi[3];             // reconstruction box (physical box minus the strips)
    int wl[3], wh[3];               // strip widths
    int n_top, n_bot, nring, ns;    // strip cells: z faces, a ring between them, all of a shot
    int nbx;                        // x blocks
    float dt, ih2[3], ih[3];        // 1 / h^2, 1 / h by axis
    float lc[MAXM + 1], gc[MAXM + 1];
    // profiles by axis: a, b, d b, d a (centred difference of a), packed; the x
    // ones may be read kGuard floats past their ends
    const float *a[3], *b[3], *db[3], *da[3];
    const float *cf, *ca;           // ((v v) dt) dt and (v v) (dt dt), pitched, per model copy
    const float* vp;                // the caller's models
    long long ms;                   // stride between model copies (0: one for every shot)
    int nsrc, nrec;
    const int *src, *rec;           // (B, n, nd): x[, y], z
    const float* wavelet;           // (B, nsrc, nt)
};

template <int ND>
struct Cell {
    int b, c[3], i;                 // shot, coordinates of lane 0 by axis, offset in a shot
    bool core;                      // some lane is updated by the steps
    __device__ __forceinline__ explicit Cell(const Geo& G)
    {
        const int xb = blockIdx.x / G.B;
        b = blockIdx.x - xb * G.B;
        c[0] = 4 * (xb * 8 + threadIdx.x);
        if (ND == 3) {
            c[1] = blockIdx.y * kBY + threadIdx.y;
            c[2] = blockIdx.z * kBZ + threadIdx.z;
        } else {
            c[1] = 0;
            c[2] = blockIdx.y * blockDim.y + threadIdx.y;
        }
        finish(G);
    }
    Cell() = default;
    __device__ __forceinline__ void finish(const Geo& G)
    {
        i = c[2] * G.SZ + c[1] * G.SY + c[0];
        core = c[0] + 3 >= G.M && c[0] < G.nx - G.M && c[2] >= G.M && c[2] < G.nz - G.M &&
               (ND == 2 || (c[1] >= G.M && c[1] < G.ny - G.M));
    }
    __device__ __forceinline__ bool lane_core(const Geo& G, int l) const
    {
        return c[0] + l >= G.M && c[0] + l < G.nx - G.M;
    }
};

template <int AXIS>
__device__ __forceinline__ int stride_of(const Geo& G) { return AXIS == 0 ? 1 : AXIS == 1 ? G.SY : G.SZ; }

// some lane lies within n cells of the outside of the physical box
template <int AXIS>
__device__ __forceinline__ bool near(const Geo& G, const int (&c)[3], int n)
{
    return c[AXIS] < G.lo[AXIS] + n || c[AXIS] + (AXIS == 0 ? 3 : 0) >= G.hi[AXIS] - n;
}

__device__ __forceinline__ float tap(float uk, float u0) { return __fsub_rn(uk, u0); }

// Values of a field (times `mul` when given) at the 2M + 1 cells along an axis
// around each lane: along x a window of neighbouring groups, along y and z one
// group per tap.  at(k, l): lane l, k cells away.
template <int M, int AXIS>
struct Line {
    static constexpr int W = v4::groups(M);
    static constexpr int N = AXIS == 0 ? 4 * (2 * W + 1) : 4 * (2 * M + 1);
    float w[N];
    __device__ __forceinline__ void load(const float* p, int stride)
    {
        if (AXIS == 0) {
#pragma unroll
            for (int j = 0; j < 2 * W + 1; ++j) put(j, v4::ldg(p + 4 * (j - W)));
        } else {
#pragma unroll
            for (int j = 0; j < 2 * M + 1; ++j) put(j, v4::ldg(p + (j - M) * stride));
        }
    }
    __device__ __forceinline__ void load_product(const float* p, const float* q, int stride)
    {
        constexpr int R = AXIS == 0 ? W : M;
#pragma unroll
        for (int j = 0; j < 2 * R + 1; ++j) {
            const int o = AXIS == 0 ? 4 * (j - R) : (j - R) * stride;
            const F4 x = v4::ldg(p + o), y = v4::ldg(q + o);
            F4 t;
#pragma unroll
            for (int l = 0; l < 4; ++l) t.v[l] = x.v[l] * y.v[l];
            put(j, t);
        }
    }
    __device__ __forceinline__ void put(int j, const F4& t)
    {
#pragma unroll
        for (int l = 0; l < 4; ++l) w[4 * j + l] = t.v[l];
    }
    static constexpr __device__ __forceinline__ int index(int k, int l)
    {
        return AXIS == 0 ? 4 * W + k + l : 4 * (M + k) + l;
    }
    __device__ __forceinline__ float at(int k, int l) const { return w[index(k, l)]; }
};

// a profile at the same cells: per lane along x, one value per tap along y and z
template <int M, int AXIS>
struct Prof {
    static constexpr int W = v4::groups(M);
    static constexpr int N = AXIS == 0 ? 4 * (2 * W + 1) : 2 * M + 1;
    float w[N];
    __device__ __forceinline__ void load(const float* p)
    {
        if (AXIS == 0) {
#pragma unroll
            for (int j = 0; j < 2 * W + 1; ++j) {
                const F4 t = v4::ldg(p + 4 * (j - W));
#pragma unroll
                for (int l = 0; l < 4; ++l) w[4 * j + l] = t.v[l];
            }
        } else {
#pragma unroll
            for (int j = 0; j < 2 * M + 1; ++j) w[j] = __ldg(p + j - M);
        }
    }
    __device__ __forceinline__ float at(int k, int l) const { return w[AXIS == 0 ? 4 * W + k + l : M + k]; }
};

// one value of a profile per lane
template <int AXIS>
__device__ __forceinline__ F4 prof_at(const float* p)
{
    return AXIS == 0 ? v4::ldg(p) : v4::splat(__ldg(p));
}

// forward / reconstruction Laplacian along one axis
template <int M, int AXIS>
__device__ __forceinline__ F4 lap(const Line<M, AXIS>& u, const Geo& G)
{
    F4 r;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const float u0 = u.at(0, l);
        float acc;
        if (M == 2) {
            acc = (G.lc[1] * (u.at(-1, l) + u.at(1, l)) + G.lc[2] * (u.at(-2, l) + u.at(2, l))) - 2.5f * u0;
        } else {
            acc = G.lc[1] * (tap(u.at(-1, l), u0) + tap(u.at(1, l), u0));
#pragma unroll
            for (int k = 2; k <= M; ++k) acc = acc + G.lc[k] * (tap(u.at(-k, l), u0) + tap(u.at(k, l), u0));
        }
        r.v[l] = acc * G.ih2[AXIS];
    }
    return r;
}

// ----------------------------------------------------------- forward step
struct Step {
    const float *un, *up;
    float* unx;
    const float* ps[3];             // CPML psi per axis, read
    float* psn[3];                  // written
    float* zt[3];                   // zeta per axis, in place
    float* slot;                    // this step's strips, or null
};

// One axis of the forward: the Laplacian, through the CPML where the axis's
// band reaches.  2-D: tmp = ((1 + b) lap + db du) + d(a psi); 3-D: tmp =
// (((1 + b) lap + db du) + a d(psi)) + d(a) psi; then w = (1 + b) tmp + a
// zeta, psi' = b du + a psi, zeta' = b tmp + a zeta (reference
// acoustic2d/forward_split.cu:86-168, acoustic3d/forward_split.cu:120-215).
template <int M, int ND, int AXIS>
__device__ __forceinline__ F4 axis_fwd(const Geo& G, const Cell<ND>& q, const Step& A, long long k)
{
    Line<M, AXIS> u;
    u.load(A.un + k, stride_of<AXIS>(G));
    F4 w = lap<M, AXIS>(u, G);
    const int c = q.c[AXIS];
    if (!near<AXIS>(G, q.c, ND == 2 ? M : 1)) return w;
    const F4 a = prof_at<AXIS>(G.a[AXIS] + c), b = prof_at<AXIS>(G.b[AXIS] + c), db = prof_at<AXIS>(G.db[AXIS] + c);
    Line<M, AXIS> ps;
    ps.load(A.ps[AXIS] + k, stride_of<AXIS>(G));
    Prof<M, AXIS> pa;
    F4 da;
    if (ND == 2) pa.load(G.a[AXIS] + c);
    else da = prof_at<AXIS>(G.da[AXIS] + c);
    const bool out = near<AXIS>(G, q.c, 0);
    const F4 z = out ? v4::ld(A.zt[AXIS] + k) : v4::splat(0.f);
    F4 pn, zn;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        float du = G.gc[1] * (u.at(1, l) - u.at(-1, l)), dp;
        if (ND == 2) dp = G.gc[1] * (pa.at(1, l) * ps.at(1, l) - pa.at(-1, l) * ps.at(-1, l));
        else dp = G.gc[1] * (ps.at(1, l) - ps.at(-1, l));
#pragma unroll
        for (int j = 2; j <= M; ++j) {
            du = du + G.gc[j] * (u.at(j, l) - u.at(-j, l));
            if (ND == 2) dp = dp + G.gc[j] * (pa.at(j, l) * ps.at(j, l) - pa.at(-j, l) * ps.at(-j, l));
            else dp = dp + G.gc[j] * (ps.at(j, l) - ps.at(-j, l));
        }
        du *= G.ih[AXIS];
        dp *= G.ih[AXIS];
        const float p0 = ps.at(0, l), bb = 1.f + b.v[l];
        const float tmp = ND == 2 ? (bb * w.v[l] + db.v[l] * du) + dp
                                  : ((bb * w.v[l] + db.v[l] * du) + a.v[l] * dp) + da.v[l] * p0;
        w.v[l] = bb * tmp + a.v[l] * z.v[l];
        const bool in = q.lane_core(G, l);
        pn.v[l] = in ? b.v[l] * du + a.v[l] * p0 : 0.f;
        zn.v[l] = in ? b.v[l] * tmp + a.v[l] * z.v[l] : 0.f;
    }
    // both are zero inside the box, where a = b = 0
    if (out) {
        v4::st(A.psn[AXIS] + k, pn);
        v4::st(A.zt[AXIS] + k, zn);
    }
    return w;
}

// index of a strip cell in a shot's strip set: z faces over the whole box,
// then per plane between them the y faces and the x faces (z, y, x in the box
// and not all in the reconstruction box)
template <int ND>
__device__ __forceinline__ int strip_index(const Geo& G, int z, int y, int x)
{
    const int bx = G.hi[0] - G.lo[0], by = ND == 3 ? G.hi[1] - G.lo[1] : 1;
    const int rz = z - G.lo[2], ry = ND == 3 ? y - G.lo[1] : 0, rx = x - G.lo[0];
    if (rz < G.wl[2]) return (rz * by + ry) * bx + rx;
    if (z >= G.hi[2] - G.wh[2]) return G.n_top + ((z - (G.hi[2] - G.wh[2])) * by + ry) * bx + rx;
    int s = G.n_top + G.n_bot + (rz - G.wl[2]) * G.nring;
    if (ND == 3) {
        if (ry < G.wl[1]) return s + ry * bx + rx;
        s += G.wl[1] * bx;
        if (y >= G.hi[1] - G.wh[1]) return s + (y - (G.hi[1] - G.wh[1])) * bx + rx;
        s += G.wh[1] * bx + (ry - G.wl[1]) * (G.wl[0] + G.wh[0]);
    }
    return s + (rx < G.wl[0] ? rx : G.wl[0] + x - (G.hi[0] - G.wh[0]));
}

template <int ND>
__device__ __forceinline__ bool in_box(const int* lo, const int* hi, int z, int y, int x)
{
    return x >= lo[0] && x < hi[0] && z >= lo[2] && z < hi[2] && (ND == 2 || (y >= lo[1] && y < hi[1]));
}

// Which lanes of a group lie in the physical box, and which of those in the
// reconstruction box.
template <int ND>
__device__ __forceinline__ void lanes(const Geo& G, const Cell<ND>& q, bool (&phys)[4], bool (&rec)[4], bool& any)
{
    any = false;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        phys[l] = in_box<ND>(G.lo, G.hi, q.c[2], q.c[1], q.c[0] + l);
        rec[l] = phys[l] && in_box<ND>(G.rlo, G.rhi, q.c[2], q.c[1], q.c[0] + l);
        any |= phys[l];
    }
}

// u_next = (2 u - u_prev) + v^2 dt^2 w of a group on the core
template <int M, int ND>
__device__ __forceinline__ F4 step_cells(const Geo& G, const Cell<ND>& q, const Step& A, long long k, F4& u0)
{
    u0 = v4::ldg(A.un + k);
    const F4 up = v4::ldg(A.up + k), cf = v4::ldg(G.cf + q.b * G.ms + q.i);
    // one axis after the other: with every axis's taps loaded first the 2-D
    // survey's step at order 4 takes 28.6 instead of 24.1 us, the 3-D one's 87
    // instead of 70 us (fewer warps, or spills)
    F4 w = axis_fwd<M, ND, 0>(G, q, A, k);
    if constexpr (ND == 3) {
        const F4 t = axis_fwd<M, ND, 1>(G, q, A, k);
#pragma unroll
        for (int l = 0; l < 4; ++l) w.v[l] += t.v[l];
    }
    const F4 t = axis_fwd<M, ND, 2>(G, q, A, k);
    F4 un;
#pragma unroll
    for (int l = 0; l < 4; ++l) un.v[l] = (2.f * u0.v[l] - up.v[l]) + cf.v[l] * (w.v[l] + t.v[l]);
    return un;
}

// a group stored on the core's lanes
template <int ND>
__device__ __forceinline__ void store_core(const Geo& G, const Cell<ND>& q, float* p, const F4& v)
{
    if (q.c[0] >= G.M && q.c[0] + 3 < G.nx - G.M) {
        v4::st(p, v);
        return;
    }
#pragma unroll
    for (int l = 0; l < 4; ++l)
        if (q.lane_core(G, l)) p[l] = v.v[l];
}

// ----------------------------------------------------------- reverse step
struct Rev {
    const float *ln, *lp;           // lambda(it + 1), lambda(it + 2)
    float* lx;                      // lambda(it); may be lp's buffer, which a thread reads at its own cells alone
    const float *ps[3], *zt[3];     // adjoint CPML memories (read)
    float *pso[3], *zto[3];         // (written)
    const float *rn, *rp;           // u(it), u(it + 1)
    float* rx;                      // u(it - 1); null at it = 0 (no reconstruction)
    const float* slot;              // strips of u(it - 1)
    float* g;                       // image, per shot: sum of (u(it-1) - 2 u(it) + u(it+1)) lambda(it)
};

// One axis of the adjoint: the difference-form Laplacian of gw = ca lambda,
// through the transposed CPML where the axis's band reaches: with t = b zeta +
// (1 + b) gw at every tap, lap((1 + b) t) - d(b psi + db t); psi' = a (psi -
// d t) in 2-D, a psi + da t - d(a t) in 3-D; zeta' = a (zeta + gw) (reference
// acoustic2d/adjoint_split.cu:27-196, acoustic3d/adjoint_split.cu:14-320).
template <int M, int ND, int AXIS>
__device__ __forceinline__ F4 axis_adj(const Geo& G, const Cell<ND>& q, const Rev& A, long long k, long long mi)
{
    Line<M, AXIS> g;
    g.load_product(G.ca + mi, A.ln + k, stride_of<AXIS>(G));
    F4 r;
    const int c = q.c[AXIS];
    if (!near<AXIS>(G, q.c, M + 1)) {
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            float acc = 0.f;
#pragma unroll
            for (int j = 1; j <= M; ++j)
                acc = acc + G.lc[j] * (tap(g.at(j, l), g.at(0, l)) + tap(g.at(-j, l), g.at(0, l)));
            r.v[l] = acc * G.ih2[AXIS];
        }
        return r;
    }
    Prof<M, AXIS> b, db, a;
    b.load(G.b[AXIS] + c);
    db.load(G.db[AXIS] + c);
    Line<M, AXIS> h, z;
    z.load(A.zt[AXIS] + k, stride_of<AXIS>(G));
    h.load(A.ps[AXIS] + k, stride_of<AXIS>(G));
    F4 p0, z0, g0;
#pragma unroll
    for (int l = 0; l < 4; ++l) { p0.v[l] = h.at(0, l); z0.v[l] = z.at(0, l); g0.v[l] = g.at(0, l); }
    // in place: z <- t, h <- b psi + db t, g <- (1 + b) t
#pragma unroll
    for (int e = 0; e < Line<M, AXIS>::N; ++e) {
        const int pe = AXIS == 0 ? e : e / 4;
        const float t = b.w[pe] * z.w[e] + (1.f + b.w[pe]) * g.w[e];
        z.w[e] = t;
        h.w[e] = b.w[pe] * h.w[e] + db.w[pe] * t;
        g.w[e] = (1.f + b.w[pe]) * t;
    }
    const bool out = near<AXIS>(G, q.c, 0);
    if (ND == 3 && out) a.load(G.a[AXIS] + c);
    F4 dq;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        float L = 0.f, D = 0.f, Q = 0.f;
#pragma unroll
        for (int j = 1; j <= M; ++j) {
            L = L + G.lc[j] * (tap(g.at(j, l), g.at(0, l)) + tap(g.at(-j, l), g.at(0, l)));
            D = D + G.gc[j] * (h.at(j, l) - h.at(-j, l));
            if (out) {
                if (ND == 2) Q = Q + G.gc[j] * (z.at(j, l) - z.at(-j, l));
                else Q = Q + G.gc[j] * (a.at(j, l) * z.at(j, l) - a.at(-j, l) * z.at(-j, l));
            }
        }
        r.v[l] = L * G.ih2[AXIS] - D * G.ih[AXIS];
        dq.v[l] = Q * G.ih[AXIS];
    }
    // inside the box the memories only meet a = b = 0
    if (out) {
        const F4 a0 = prof_at<AXIS>(G.a[AXIS] + c);
        F4 pn, zn;
        F4 da;
        if (ND == 3) da = prof_at<AXIS>(G.da[AXIS] + c);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const bool in = q.lane_core(G, l) &&
                            (AXIS != 0 || q.c[0] + l < G.lo[0] || q.c[0] + l >= G.hi[0]);
            const float p = ND == 2 ? a0.v[l] * (p0.v[l] - dq.v[l])
                                    : (a0.v[l] * p0.v[l] + da.v[l] * z.at(0, l)) - dq.v[l];
            pn.v[l] = in ? p : 0.f;
            zn.v[l] = in ? a0.v[l] * (z0.v[l] + g0.v[l]) : 0.f;
        }
        v4::st(A.pso[AXIS] + k, pn);
        v4::st(A.zto[AXIS] + k, zn);
    }
    return r;
}

// lambda(it) of a group on the core
template <int M, int ND>
__device__ __forceinline__ F4 adj_cells(const Geo& G, const Cell<ND>& q, const Rev& A, long long k, long long mi)
{
    const F4 l0 = v4::ldg(A.ln + k), lp = v4::ld(A.lp + k);
    F4 w = axis_adj<M, ND, 0>(G, q, A, k, mi);
    if constexpr (ND == 3) {
        const F4 t = axis_adj<M, ND, 1>(G, q, A, k, mi);
#pragma unroll
        for (int l = 0; l < 4; ++l) w.v[l] += t.v[l];
    }
    const F4 t = axis_adj<M, ND, 2>(G, q, A, k, mi);
    F4 lx;
#pragma unroll
    for (int l = 0; l < 4; ++l) lx.v[l] = (2.f * l0.v[l] - lp.v[l]) + (w.v[l] + t.v[l]);
    return lx;
}

// the forward's coefficient of a group from the caller's models, which are not
// pitched (a reverse that keeps one pitched model field keeps the adjoint's)
template <int ND>
__device__ __forceinline__ F4 coef(const Geo& G, const Cell<ND>& q)
{
    const long long row = ((G.ms ? (long long)q.b * G.nz : 0) + q.c[2]) * G.ny + q.c[1];
    F4 c;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const float v = __ldg(G.vp + row * G.nx + min(q.c[0] + l, G.nx - 1));
        c.v[l] = ((v * v) * G.dt) * G.dt;
    }
    return c;
}

// (2 u(it) - u(it+1)) + cf Lap u(it) of a group
template <int M, int ND>
__device__ __forceinline__ F4 recon_cells(const Geo& G, const float* rn, long long k, const F4& cf, const F4& u0,
                                          const F4& up)
{
    Line<M, 0> x;
    Line<M, 2> z;
    x.load(rn + k, 1);
    z.load(rn + k, G.SZ);
    F4 w = lap<M, 0>(x, G);
    if constexpr (ND == 3) {
        Line<M, 1> y;
        y.load(rn + k, G.SY);
        const F4 t = lap<M, 1>(y, G);
#pragma unroll
        for (int l = 0; l < 4; ++l) w.v[l] += t.v[l];
    }
    const F4 t = lap<M, 2>(z, G);
    F4 un;
#pragma unroll
    for (int l = 0; l < 4; ++l) un.v[l] = (2.f * u0.v[l] - up.v[l]) + cf.v[l] * (w.v[l] + t.v[l]);
    return un;
}

// one axis's profiles a, b, d b, d a (da: centred difference on [M, n - M), 0
// outside), zero past their ends
__global__ static void prep_profiles(const float* a, const float* b, const float* db, int n, const Geo G, float ih, int lead,
                              int len, float* out)
{
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < len; e += gridDim.x * blockDim.x) {
        const int c = e - lead;
        const bool in = c >= 0 && c < n;
        float da = 0.f;
        if (c >= G.M && c < n - G.M)
            for (int k = 1; k <= G.M; ++k) da = da + G.gc[k] * (a[c + k] - a[c - k]);
        out[e] = in ? a[c] : 0.f;
        out[len + e] = in ? b[c] : 0.f;
        out[2 * len + e] = in ? db[c] : 0.f;
        out[3 * len + e] = da * ih;
    }
}

}  // namespace avec
}  // namespace sweep
