// conv_bf16.cu -- BF16 3x3 convolutions (stride 1, zero padding 1) as
// implicit GEMMs on the tensor cores with FP32 accumulation, for the U-Net
// preconditioner of the FWI update.  No counterpart in the reference (it has
// no learned preconditioner); checked against PyTorch's float64 conv2d.
//
// Layout: activations NHWC bf16 with C a multiple of 8 (16-byte channel
// groups); weights (Co, 3, 3, C) bf16.  Tap t = (dy + 1) * 3 + (dx + 1).
//
//   forward  y[p, co]  = sum_{t, c} x[p + off(t), c] w[co, t, c]          (M = pixels, N = Co, K = 9 C)
//   data     dx[p, c]  = sum_{t, co} dy[p - off(t), co] w[co, t, c]       (M = pixels, N = C,  K = 9 Co)
//   weight   dw[co, t, c] = sum_p dy[p, co] x[p + off(t), c]              (M = Co, N = 9 C, K = pixels)
//
// All three run on the 5th-generation tensor cores from the same shared-memory
// image of the activations: a tile of 8 x 16 (w, h) pixels with its one-pixel
// halo, stored as planes of 8 channels -- plane[c / 8][row][column], 16 bytes a
// pixel, zeros outside the image -- by 16-byte asynchronous copies.  Eight
// pixels of a row are then 128 consecutive bytes, one core matrix of the
// no-swizzle operand layouts, at any column: a tap is the same planes from
// another start address, so a tile is loaded once for all nine taps (the
// gather of a tile per tap and K step took 9x the loads and shared-memory
// writes and bound the kernels: 148 us a pass on 16 x 64 x 192 pixels, 64 -> 64
// channels, 208 us the weight gradient; 46 and 38 us the forward and the data
// pass and 44 us the weight gradient now.  No unit is near its limit: the
// copies, MMAs and epilogue of one CTA an SM overlap in part).
//   conv_pass  (forward, data): A = tile, K-major (M = 128 pixels, K = channels),
//              B = the weights of the CTA's 64 outputs, all nine taps resident;
//              a CTA walks its tiles, the loads of the next one and the
//              epilogue of the last one beside the MMAs of this one.
//   conv_wgrad (weights): A = tile, MN-major (M = 64 channels of tap dx and
//              the same 64 of tap dx + 1, which is a second copy of the planes
//              one pixel on; K = pixels), B = dy of the tile, MN-major; the
//              nine taps accumulate in tensor memory over all tiles of the
//              CTA, which adds them to dw once.
// MMAs are issued by one thread (M 128, N 64, K 16); tcgen05.commit on an
// mbarrier per buffer releases a tile's buffer.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "tma.cuh"

namespace sweep {
namespace conv {

constexpr int BM = 128, BN = 64;
// threads of the tensor-core kernels: the copies and the epilogue are bound by
// their instructions, at one CTA per SM (256 threads: 49, 40 and 49 us)
constexpr int NT = 512;
constexpr int COLS = BN / (NT / 128);        // accumulator columns of a thread
constexpr int NTC = 256;                     // threads of the cotangent's pass

// ------------------------------------------------------------ tcgen05 path
namespace umma {

constexpr int BW = 8, BH = 16;               // pixels of a tile
constexpr int PW = BW + 2, PN = PW * (BH + 2);   // row and size of a plane with its halo
// plane strides in bytes: odd multiples of 16, so that the eight planes of a
// pixel are stored without bank conflicts
constexpr int PS = (PN + 1) * 16;            // tile with halo
constexpr int DS = (BM + 1) * 16;            // tile without
constexpr int BS = BN * 16;                  // weights
constexpr int CK = 64;                       // channels per step
constexpr int B_TAP = CK / 8 * BS;           // weights of one tap
constexpr int A_BYTES = (CK / 8 * PS + 127) / 128 * 128;
constexpr int A2_BYTES = (2 * CK / 8 * PS + 127) / 128 * 128;
constexpr int D_BYTES = (CK / 8 * DS + 127) / 128 * 128;

enum ErrCode { ERR_MMA_WAIT = 11 };

constexpr int NB = 3;                        // tile buffers
struct Head {
    uint64_t done[NB];                       // MMAs of a buffer finished (tcgen05.commit)
    uint32_t tmem;                           // accumulator base address from tcgen05.alloc
};
constexpr int HEAD = 128;

// Shared-memory matrix descriptor: start address, leading / stride byte
// offsets (16-byte units), descriptor version 1, no swizzle.  K-major: leading
// = next 8 of K, stride = next 8 rows; MN-major: leading = next 8 of K, stride
// = next 8 of M or N.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::f16: D F32, A and B BF16, N 64, M 128; both
// operands K-major, or both MN-major (bits 15 and 16).
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
constexpr uint32_t kIdescMN = kIdesc | (1u << 15) | (1u << 16);

__device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        :
        : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)accumulate), "r"(0), "r"(0), "r"(0), "r"(0));
}

__device__ __forceinline__ void commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     tma::smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void ld8(uint32_t taddr, float (&v)[8])
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 bytes of global to shared memory, zeros if !in
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool in)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void close_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// wait for this thread's copies, those of its `newest` last groups excepted
template <int newest>
__device__ __forceinline__ void wait_copies()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(newest) : "memory");
}

__device__ __forceinline__ void alloc(Head& h, uint32_t cols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tma::smem_u32(&h.tmem)),
                 "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void dealloc(uint32_t tmem, uint32_t cols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}

__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

}  // namespace umma

struct Shape {
    int N, H, W;        // images, height, width
    int C;              // channels of the gathered tensor (multiple of 8)
    int Nout;           // output channels (multiple of 8)
    int ntx, nty;       // tiles of an image
    int tiles;          // tiles in all
};

struct Tile {
    int img, h0, w0;
    __device__ __forceinline__ Tile(const Shape& S, int t)
    {
        const int r = t / S.ntx;
        w0 = (t - r * S.ntx) * umma::BW;
        img = r / S.nty;
        h0 = (r - img * S.nty) * umma::BH;
    }
};

// A thread's share of a tile with its halo: one group of 8 channels of every
// ROWS-th pixel.
struct Halo {
    static constexpr int ROWS = NT / 8, N = (umma::PN + ROWS - 1) / ROWS;
    int kc, at[N];                           // row << 8 | column, or -1
    __device__ __forceinline__ Halo()
    {
        kc = threadIdx.x & 7;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int q = (threadIdx.x >> 3) + ROWS * u, r = q / umma::PW;
            at[u] = q < umma::PN ? r << 8 | (q - r * umma::PW) : -1;
        }
    }
    // channels [c0, c0 + 64) of tile t, `shift` pixels to the right, into the planes at dst
    __device__ __forceinline__ void load(const Shape& S, const __nv_bfloat16* __restrict__ act, const Tile& T, int c0,
                                         int shift, uint32_t dst) const
    {
        const int c = c0 + 8 * kc, hb = T.h0 - 1, wb = T.w0 - 1 + shift;
        const __nv_bfloat16* base = act + (((long long)T.img * S.H + hb) * S.W + wb) * S.C + c;
        const uint32_t d = dst + kc * umma::PS + (threadIdx.x >> 3) * 16;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            if (at[u] < 0) continue;
            const int r = at[u] >> 8, w = at[u] & 255;
            const bool in = (unsigned)(hb + r) < (unsigned)S.H && (unsigned)(wb + w) < (unsigned)S.W && c < S.C;
            umma::copy16(d + u * ROWS * 16, in ? base + ((long long)r * S.W + w) * S.C : act, in);
        }
    }
};

__device__ __forceinline__ void put8(float* o, const float (&v)[8])
{
    *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8])
{
    uint4 r;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    return r;
}
__device__ __forceinline__ void put8(__nv_bfloat16* o, const float (&v)[8]) { *reinterpret_cast<uint4*>(o) = pack8(v); }

// out[p, n] = sum_{t, c} act[p + off(t), c] B[n, t, c] (+ bias[n]), p - off(t)
// if flip.  One CTA: outputs [64 blockIdx.y, + 64) of `per` tiles from per *
// blockIdx.x on.  With one step of channels (C <= 64) the accumulators of
// consecutive tiles alternate between two; else every tile keeps its own (per
// <= 8) while the CTA walks its tiles once per 64 channels, the next weights
// arriving in parts beside the tiles.
template <class Out>
__global__ void __launch_bounds__(NT) conv_pass(const __nv_bfloat16* __restrict__ act,
                                                const __nv_bfloat16* __restrict__ Bt, const float* __restrict__ bias,
                                                Out* __restrict__ out, const Shape S, int per, int cols, bool flip,
                                                int* err)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    umma::Head& hd = *reinterpret_cast<umma::Head*>(smem);
    const uint32_t sa = tma::smem_u32(smem) + umma::HEAD, sb = sa + umma::NB * umma::A_BYTES;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.y * BN, t0 = blockIdx.x * per, nt = min(per, S.tiles - t0);
    const int nch = (S.C + umma::CK - 1) / umma::CK, steps = nch * nt;
    if (warp == 0) umma::alloc(hd, (uint32_t)cols);
    if (tid == 0) {
        for (uint64_t& d : hd.done) tma::mbar_init(&d, 1);
        tma::fence_barrier_init();
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = hd.tmem;

    // weights of taps [a, b) of channel step ch
    auto load_weights = [&](int ch, int a, int b) {
        const int c0 = ch * umma::CK;
        const uint32_t dst = sb + (ch & 1) * 9 * umma::B_TAP;
        for (int id = a * 512 + tid; id < b * 512; id += NT) {
            const int t = id >> 9, kc = (id >> 5 & 3) * 2 + (id & 1), n = (id >> 7 & 3) * 16 + (id >> 1 & 15);
            const int c = c0 + 8 * kc;
            const bool in = n0 + n < S.Nout && c < S.C;
            umma::copy16(dst + t * umma::B_TAP + kc * umma::BS + n * 16,
                         in ? Bt + ((long long)(n0 + n) * 9 + t) * S.C + c : Bt, in);
        }
    };
    // this thread's columns of the outputs and their bias
    const int col = COLS * (warp >> 2), n1 = n0 + col;
    float bv[COLS];
#pragma unroll
    for (int e = 0; e < COLS; ++e) bv[e] = bias && n1 + e < S.Nout ? __ldg(bias + n1 + e) : 0.f;
    auto epilogue = [&](int i) {
        const Tile T(S, t0 + i);
        const int m = 32 * (warp & 3) + lane, h = T.h0 + (m >> 3), w = T.w0 + (m & 7);
        const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (nch == 1 ? (i & 1) : i) * BN + col;
        float v[COLS / 8][8];
#pragma unroll
        for (int j = 0; j < COLS / 8; ++j) umma::ld8(ta + 8 * j, v[j]);
        umma::wait_ld();
        if (h >= S.H || w >= S.W) return;
        Out* o = out + (((long long)T.img * S.H + h) * S.W + w) * S.Nout + n1;
#pragma unroll
        for (int j = 0; j < COLS / 8; ++j) {
            if (n1 + 8 * j >= S.Nout) break;
#pragma unroll
            for (int e = 0; e < 8; ++e) v[j][e] += bv[8 * j + e];
            put8(o + 8 * j, v[j]);
        }
    };

    const Halo halo;
    auto load = [&](int s) {                             // the tile and channels of step s
        const int ch = s / nt;
        halo.load(S, act, Tile(S, t0 + s - ch * nt), ch * umma::CK, 0, sa + s % umma::NB * umma::A_BYTES);
    };
    load_weights(0, 0, 9);
    load(0);
    umma::close_group();
    if (steps > 1) load(1);
    umma::close_group();
    bool ok = true;
    int buf = 0, prev = 0;                               // buffers of this step and of the one before
    uint32_t phase = 0, pphase = 0;
    for (int s = 0; s < steps; ++s) {
        const int ch = s / nt, i = s - ch * nt;
        // the tile of this step; at a new channel step its last weights too
        if (i == 0 && ch > 0) umma::wait_copies<0>();
        else umma::wait_copies<1>();
        umma::fence_async_smem();                        // copied operands -> tensor-core reads
        umma::fence_before();
        __syncthreads();
        if (tid == 0) {
            umma::fence_after();
            const uint32_t d = tmem + (nch == 1 ? (i & 1) : i) * BN;
            const int nk = (min(umma::CK, S.C - ch * umma::CK) + 15) / 16;
            // the taps in the order of their places in the halo
            const uint64_t da = umma::smem_desc(sa + buf * umma::A_BYTES, umma::PS, umma::PW * 16);
            uint64_t db = umma::smem_desc(sb + ((ch & 1) * 9 + (flip ? 8 : 0)) * umma::B_TAP, umma::BS, 128);
            const uint64_t step = flip ? 0 - (uint64_t)(umma::B_TAP >> 4) : (uint64_t)(umma::B_TAP >> 4);
#pragma unroll
            for (int u = 0; u < 9; ++u) {
#pragma unroll
                for (int k = 0; k < umma::CK / 16; ++k)
                    if (k < nk)
                        umma::mma(d, da + (uint64_t)((u / 3) * umma::PW + u % 3 + 2 * k * umma::PS / 16),
                                  db + (uint64_t)(2 * k * umma::BS / 16), umma::kIdesc, ch > 0 || u > 0 || k > 0);
                db += step;
            }
            umma::commit(&hd.done[buf]);
        }
        // the MMAs of the step before are done: its buffer takes the tile after the next
        if (s > 0) ok = ok && tma::mbar_wait(&hd.done[prev], pphase, err, umma::ERR_MMA_WAIT);
        if (s + 2 < steps) load(s + 2);
        if (ch + 1 < nch) load_weights(ch + 1, 9 * i / nt, 9 * (i + 1) / nt);
        umma::close_group();
        if (ch == nch - 1 && i > 0) {
            umma::fence_after();
            if (ok) epilogue(i - 1);
        }
        prev = buf;
        pphase = phase;
        if (++buf == umma::NB) { buf = 0; phase ^= 1; }
    }
    ok = ok && tma::mbar_wait(&hd.done[prev], pphase, err, umma::ERR_MMA_WAIT);
    umma::fence_after();
    if (ok) epilogue(nt - 1);
    umma::wait_copies<0>();
    umma::fence_before();
    __syncthreads();
    if (warp == 0) umma::dealloc(tmem, (uint32_t)cols);
}

// The sum of a CTA's products of one weight over the pixels inside the image.
__device__ __noinline__ float inside_sum(const Shape& S, const __nv_bfloat16* __restrict__ x,
                                         const __nv_bfloat16* __restrict__ dy, int t0, int nt, int tap, int c, int n)
{
    float sum = 0.f;
    for (int t = t0; t < t0 + nt; ++t) {
        const Tile T(S, t);
        for (int q = 0; q < BM; ++q) {
            const int h = T.h0 + (q >> 3), w = T.w0 + (q & 7), hx = h + tap / 3 - 1, wx = w + tap % 3 - 1;
            if (h >= S.H || w >= S.W || hx < 0 || hx >= S.H || wx < 0 || wx >= S.W) continue;
            const long long img = (long long)T.img * S.H;
            sum += __bfloat162float(dy[((img + h) * S.W + w) * S.Nout + n]) *
                   __bfloat162float(x[((img + hx) * S.W + wx) * S.C + c]);
        }
    }
    return sum;
}

// dw[co, t, c] += the sum over this CTA's tiles: c in [64 blockIdx.x, + 64), co
// in [64 blockIdx.y, + 64), tiles [per blockIdx.z, + per).  Accumulator 2 dy holds
// taps (dy, -1) and (dy, 0), rows 0..63 and 64..127; 2 dy + 1 tap (dy, 1) and
// 64 rows that are not used.
__global__ void __launch_bounds__(NT) conv_wgrad(const __nv_bfloat16* __restrict__ x,
                                                 const __nv_bfloat16* __restrict__ dy, float* __restrict__ dw,
                                                 const Shape S, int per, int* err)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    umma::Head& hd = *reinterpret_cast<umma::Head*>(smem);
    const uint32_t sa = tma::smem_u32(smem) + umma::HEAD, sd = sa + umma::NB * umma::A2_BYTES;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.x * umma::CK, n0 = blockIdx.y * BN, t0 = blockIdx.z * per, nt = min(per, S.tiles - t0);
    constexpr uint32_t cols = 512;
    if (warp == 0) umma::alloc(hd, cols);
    if (tid == 0) {
        for (uint64_t& d : hd.done) tma::mbar_init(&d, 1);
        tma::fence_barrier_init();
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = hd.tmem;

    const Halo halo;
    auto load = [&](int s) {
        const Tile T(S, t0 + s);
        const uint32_t a = sa + s % umma::NB * umma::A2_BYTES, d = sd + s % umma::NB * umma::D_BYTES;
        halo.load(S, x, T, c0, 0, a);
        halo.load(S, x, T, c0, 1, a + 8 * umma::PS);
        const int n = n0 + 8 * halo.kc;
#pragma unroll
        for (int u = 0; u < BM / Halo::ROWS; ++u) {
            const int q = (tid >> 3) + Halo::ROWS * u, h = T.h0 + (q >> 3), w = T.w0 + (q & 7);
            const bool in = h < S.H && w < S.W && n < S.Nout;
            umma::copy16(d + halo.kc * umma::DS + q * 16,
                         in ? dy + (((long long)T.img * S.H + h) * S.W + w) * S.Nout + n : dy, in);
        }
    };
    load(0);
    umma::close_group();
    if (nt > 1) load(1);
    umma::close_group();
    bool ok = true;
    int buf = 0, prev = 0;
    uint32_t phase = 0, pphase = 0;
    for (int s = 0; s < nt; ++s) {
        umma::wait_copies<1>();
        umma::fence_async_smem();                        // copied operands -> tensor-core reads
        __syncthreads();
        if (tid == 0) {
            umma::fence_after();
            const uint64_t da = umma::smem_desc(sa + buf * umma::A2_BYTES, umma::PW * 16, umma::PS);
            const uint64_t db = umma::smem_desc(sd + buf * umma::D_BYTES, 128, umma::DS);
#pragma unroll
            for (int k = 0; k < umma::BH / 2; ++k)       // two rows of 8 pixels
#pragma unroll
                for (int j = 0; j < 6; ++j)
                    umma::mma(tmem + j * BN, da + (uint64_t)((2 * k + j / 2) * umma::PW + (j & 1) * 2),
                              db + (uint64_t)(16 * k), umma::kIdescMN, s > 0 || k > 0);
            umma::commit(&hd.done[buf]);
        }
        if (s > 0) ok = ok && tma::mbar_wait(&hd.done[prev], pphase, err, umma::ERR_MMA_WAIT);
        if (s + 2 < nt) load(s + 2);
        umma::close_group();
        prev = buf;
        pphase = phase;
        if (++buf == umma::NB) { buf = 0; phase ^= 1; }
    }
    ok = ok && tma::mbar_wait(&hd.done[prev], pphase, err, umma::ERR_MMA_WAIT);
    umma::fence_after();
    const int m = 32 * (warp & 3) + lane, c = c0 + (m & 63), col = COLS * (warp >> 2), n = n0 + col;
    const bool over = S.H % umma::BH != 0 || S.W % umma::BW != 0;
#pragma unroll 1
    for (int j = 0; j < 6; ++j) {
        const int tap = (j / 2) * 3 + (j & 1 ? 2 : m >> 6);
        const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + j * BN + col;
        float v[COLS / 8][8];
#pragma unroll
        for (int i = 0; i < COLS / 8; ++i) umma::ld8(ta + 8 * i, v[i]);
        umma::wait_ld();
        if (!ok || c >= S.C || ((j & 1) && m >= 64)) continue;
#pragma unroll
        for (int i = 0; i < COLS / 8; ++i)
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int co = n + 8 * i + e;
                if (co >= S.Nout) continue;
                // the zero dy of a tile's pixels outside the image makes a NaN of
                // an infinite x that only such a pixel's tap reads
                const float s = over && v[i][e] != v[i][e] ? inside_sum(S, x, dy, t0, nt, tap, c, co) : v[i][e];
                atomicAdd(dw + ((long long)co * 9 + tap) * S.C + c, s);
            }
    }
    umma::wait_copies<0>();
    umma::fence_before();
    __syncthreads();
    if (warp == 0) umma::dealloc(tmem, cols);
}

// HBM-bound: 75 MB in 14.5 us at 196608 x 64 (a cast and a sum took 12 + 73 us).
// The output gradient (rows, co) in bf16 and, if part, the sums of its columns
// over each block's rows: part (gridDim.x, co).  A thread holds 8 channels.
__global__ void __launch_bounds__(NTC) cotangent(const float* __restrict__ g, __nv_bfloat16* __restrict__ out,
                                                float* __restrict__ part, long long rows, int co)
{
    extern __shared__ float sums[];
    const int cg = co / 8, lanes = NTC / cg > 0 ? NTC / cg : 1;
    for (int c8 = threadIdx.x % cg; c8 < cg; c8 += NTC) {
        const int r0 = cg > NTC ? 0 : threadIdx.x / cg;
        float acc[8] = {};
        if (r0 < lanes) {
            for (long long r = (long long)blockIdx.x * lanes + r0; r < rows; r += (long long)gridDim.x * lanes) {
                const float4* p = reinterpret_cast<const float4*>(g + r * co + 8 * c8);
                const float4 a = __ldcs(p), b = __ldcs(p + 1);
                const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                *reinterpret_cast<uint4*>(out + r * co + 8 * c8) = pack8(v);
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] += v[e];
            }
            float* s = lanes > 1 ? sums + r0 * co : part + (long long)blockIdx.x * co;
            if (part)
#pragma unroll
                for (int e = 0; e < 8; ++e) s[8 * c8 + e] = acc[e];
        }
        if (cg <= NTC) break;
    }
    if (!part || lanes == 1) return;
    __syncthreads();
    for (int c = threadIdx.x; c < co; c += NTC) {
        float s = 0.f;
        for (int r = 0; r < lanes; ++r) s += sums[r * co + c];
        part[(long long)blockIdx.x * co + c] = s;
    }
}

// The weights transposed per tap: wt[c][t][o] = w[o][t][c]
__global__ void transpose_weights(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wt, int co, int c)
{
    const long long n = 9LL * co * c;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int o = (int)(e % co);
        const long long r = e / co;                      // c * 9 + t
        wt[e] = w[((long long)o * 9 + r % 9) * c + r / 9];
    }
}

// db[c] = sum over n rows of part
__global__ void bias_sum(const float* __restrict__ part, int n, int co, float* __restrict__ db)
{
    __shared__ float s[8][32];
    const int c = blockIdx.x * 32 + threadIdx.x;
    float a = 0.f;
    if (c < co)
        for (int r = threadIdx.y; r < n; r += 8) a += part[(long long)r * co + c];
    s[threadIdx.y][threadIdx.x] = a;
    __syncthreads();
    if (threadIdx.y || c >= co) return;
#pragma unroll
    for (int r = 1; r < 8; ++r) a += s[r][threadIdx.x];
    db[c] = a;
}

// Device error flag of the convolution kernels (one per process; zeroed
// when made and by every status call).
int* error_flag()
{
    static int* flag = nullptr;
    if (!flag) {
        SWEEP_CUDA(cudaMalloc(&flag, sizeof(int)));
        SWEEP_CUDA(cudaMemset(flag, 0, sizeof(int)));
    }
    return flag;
}

}  // namespace conv
}  // namespace sweep

using namespace sweep;

namespace sweep {
namespace conv {

static Shape shape_of(int n, int h, int w, int c, int nout)
{
    Shape S{n, h, w, c, nout, (w + umma::BW - 1) / umma::BW, (h + umma::BH - 1) / umma::BH, 0};
    const long long t = (long long)n * S.ntx * S.nty;
    SWEEP_REQUIRE(t < (1LL << 31), "conv3x3: the image holds 2^31 tiles or more");
    S.tiles = (int)t;
    return S;
}

template <class Out>
static void pass(const void* act, const void* bt, const float* bias, Out* out, int n, int h, int w, int c, int nout,
                 int sign, cudaStream_t st)
{
    SWEEP_REQUIRE(act && bt && out, "conv3x3: null pointer");
    SWEEP_REQUIRE(n >= 1 && h >= 1 && w >= 1 && nout >= 1, "conv3x3: empty shape");
    SWEEP_REQUIRE(c >= 8 && c % 8 == 0, "conv3x3: channels must be a positive multiple of 8 (got %d)", c);
    SWEEP_REQUIRE(sign == 1 || sign == -1, "conv3x3: sign must be +1 or -1");
    SWEEP_REQUIRE(((uintptr_t)act & 15) == 0 && ((uintptr_t)bt & 15) == 0, "conv3x3: operands must be 16-byte aligned");
    SWEEP_REQUIRE(nout % 8 == 0, "conv3x3: output channels must be a multiple of 8 (got %d)", nout);
    SWEEP_REQUIRE(((uintptr_t)out & 15) == 0, "conv3x3: output must be 16-byte aligned");
    const Shape S = shape_of(n, h, w, c, nout);
    const int gx = (nout + BN - 1) / BN, nch = (c + umma::CK - 1) / umma::CK;
    // one CTA per SM (its shared memory); tiles per CTA: an even share, within
    // the eight accumulators when the channels take more than one step
    long long per = ((long long)S.tiles * gx + 147) / 148;
    if (nch > 1) per = std::min(per, 8LL);
    const int acc = nch == 1 ? 2 : (int)per;
    const int cols = acc <= 2 ? 128 : acc <= 4 ? 256 : 512;
    const int smem = umma::HEAD + umma::NB * umma::A_BYTES + std::min(nch, 2) * 9 * umma::B_TAP;
    SWEEP_CUDA(cudaFuncSetAttribute(conv_pass<Out>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    conv_pass<Out><<<dim3((unsigned)((S.tiles + per - 1) / per), (unsigned)gx), NT, smem, st>>>(
        static_cast<const __nv_bfloat16*>(act), static_cast<const __nv_bfloat16*>(bt), bias, out, S, (int)per, cols,
        sign < 0, error_flag());
    SWEEP_LAUNCH_CHECK();
}

static void wgrad(const void* x, const void* dy, float* dw, int n, int h, int w, int c, int co, cudaStream_t st)
{
    SWEEP_REQUIRE(x && dy && dw, "conv3x3 wgrad: null pointer");
    SWEEP_REQUIRE(c >= 8 && c % 8 == 0 && co >= 8 && co % 8 == 0,
                  "conv3x3 wgrad: channel counts must be positive multiples of 8 (got %d, %d)", c, co);
    SWEEP_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)dy & 15) == 0, "conv3x3 wgrad: operands must be 16-byte aligned");
    SWEEP_CUDA(cudaMemsetAsync(dw, 0, sizeof(float) * (size_t)co * 9 * c, st));
    if (n < 1 || h < 1 || w < 1) return;
    const Shape S = shape_of(n, h, w, c, co);
    // one CTA per SM; the tiles split evenly over the CTAs that the channel
    // blocks leave room for
    const unsigned gx = (unsigned)((c + umma::CK - 1) / umma::CK), gy = (unsigned)((co + BN - 1) / BN);
    const long long splits = std::max(1LL, 148LL / ((long long)gx * gy));
    const int per = (int)((S.tiles + splits - 1) / splits);
    const dim3 grid(gx, gy, (unsigned)((S.tiles + per - 1) / per));
    constexpr int smem = umma::HEAD + umma::NB * (umma::A2_BYTES + umma::D_BYTES);
    SWEEP_CUDA(cudaFuncSetAttribute(conv_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    conv_wgrad<<<grid, NT, smem, st>>>(static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(dy), dw, S,
                                       per, error_flag());
    SWEEP_LAUNCH_CHECK();
}

// Scratch of the backward: dy in bf16, the transposed weights, the column sums
// of each block.
struct BackwardWs {
    __nv_bfloat16 *dy, *wt;
    float* part;
};
constexpr int kParts = 592;
static void carve(Carve& k, long long px, int c, int co, BackwardWs& w)
{
    w.dy = k.take<__nv_bfloat16>(px * co);
    w.wt = k.take<__nv_bfloat16>(9LL * co * c);
    w.part = k.take<float>((long long)kParts * co);
}

}  // namespace conv
}  // namespace sweep

extern "C" int sweep_b200_conv3x3_gemm(const void* act, const void* bt, const float* bias, float* out,
                                                      int32_t n, int32_t h, int32_t w, int32_t c, int32_t nout,
                                                      int32_t sign, void* stream, char* err, int32_t err_cap)
{
    return guarded(err, err_cap, [&] {
        conv::pass(act, bt, bias, out, n, h, w, c, nout, sign, static_cast<cudaStream_t>(stream));
    });
}

extern "C" int sweep_b200_conv3x3_wgrad(const void* x, const void* dy, float* dw, int32_t n, int32_t h,
                                                       int32_t w, int32_t c, int32_t co, void* stream, char* err,
                                                       int32_t err_cap)
{
    return guarded(err, err_cap, [&] { conv::wgrad(x, dy, dw, n, h, w, c, co, static_cast<cudaStream_t>(stream)); });
}

extern "C" int64_t sweep_b200_conv3x3_backward_bytes(int32_t n, int32_t h, int32_t w, int32_t c, int32_t co)
{
    Carve k(nullptr);
    conv::BackwardWs ws;
    conv::carve(k, (long long)n * h * w, c, co, ws);
    return k.off;
}

extern "C" int sweep_b200_conv3x3_backward(const float* gout, const void* x, const void* wb, void* dx, float* dw, float* db,
                                           void* scratch, int64_t scratch_bytes, int32_t n, int32_t h, int32_t w, int32_t c,
                                           int32_t co, void* stream, char* err, int32_t err_cap)
{
    return guarded(err, err_cap, [&] {
        SWEEP_REQUIRE(gout && scratch && (!dx || wb) && (!dw || x), "conv3x3 backward: null pointer");
        SWEEP_REQUIRE(n >= 1 && h >= 1 && w >= 1, "conv3x3 backward: empty shape");
        SWEEP_REQUIRE(c >= 8 && c % 8 == 0 && co >= 8 && co % 8 == 0,
                      "conv3x3 backward: channel counts must be positive multiples of 8 (got %d, %d)", c, co);
        SWEEP_REQUIRE(((uintptr_t)gout & 15) == 0 && ((uintptr_t)scratch & 255) == 0,
                      "conv3x3 backward: operands must be 16-byte and the scratch 256-byte aligned");
        const long long px = (long long)n * h * w;
        Carve k(scratch);
        conv::BackwardWs ws;
        conv::carve(k, px, c, co, ws);
        SWEEP_REQUIRE(k.off <= scratch_bytes, "conv3x3 backward: scratch too small (%lld < %lld bytes)",
                      (long long)scratch_bytes, (long long)k.off);
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        const int lanes = std::max(1, conv::NTC / (co / 8));
        const int blocks = (int)std::min<long long>((px + lanes - 1) / lanes, conv::kParts);
        const size_t smem = lanes > 1 ? (size_t)lanes * co * 4 : 0;      // 8 KB at most
        conv::cotangent<<<blocks, conv::NTC, smem, st>>>(gout, ws.dy, db ? ws.part : nullptr, px, co);
        if (db) conv::bias_sum<<<(co + 31) / 32, dim3(32, 8), 0, st>>>(ws.part, blocks, co, db);
        SWEEP_LAUNCH_CHECK();
        if (dx) {
            conv::transpose_weights<<<(unsigned)std::min<long long>((9LL * co * c + 255) / 256, 592), 256, 0, st>>>(
                static_cast<const __nv_bfloat16*>(wb), ws.wt, co, c);
            SWEEP_LAUNCH_CHECK();
            conv::pass(ws.dy, ws.wt, nullptr, static_cast<__nv_bfloat16*>(dx), n, h, w, co, c, -1, st);
        }
        if (dw) conv::wgrad(x, ws.dy, dw, n, h, w, c, co, st);
    });
}

extern "C" int sweep_b200_conv3x3_status(void* stream, char* err, int32_t err_cap)
{
    return guarded(err, err_cap, [&] {
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        int* flag = conv::error_flag();
        int h_flag = 0;
        SWEEP_CUDA(cudaMemcpyAsync(&h_flag, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
        SWEEP_CUDA(cudaStreamSynchronize(st));
        if (h_flag) SWEEP_CUDA(cudaMemset(flag, 0, sizeof(int)));
        SWEEP_REQUIRE(h_flag == 0, "conv3x3: a tensor-core wait did not complete in time (code %d); "
                                   "outputs since the last status call are invalid", h_flag);
    });
}
