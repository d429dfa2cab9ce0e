// Learned dispersion corrector (include/ouc_corrector.h): a 4-layer 5x5 CNN
// whose convolutions run as implicit GEMMs on the sm_100a tensor cores.
//
// A convolution's GEMM M is 128 consecutive pixels of one image row, N the
// output channels (32 or 16) of up to four rows, K 25 taps x input channels.
// A work item is kCB consecutive rows of 128 pixels; its (kCB + 4)-row x
// 132-column input patch (zeros outside the image) lies in shared memory in
// the no-swizzle K-major "core matrix" layout -- [row][channel chunk of 8]
// [column][8 channels], 16 bytes per (column, chunk) -- so that the A operand
// of tap (dx, dz) is simply the patch shifted by (dx, dz): a shared-memory
// matrix descriptor whose start address moves by 16 * (dx * chunks * 132 + dz)
// bytes, with the leading-dimension offset = one chunk plane (132 * 16 B)
// and the stride offset = 8 pixels (128 B).  No im2col copy is made.  The
// weights of all taps sit in shared memory for the whole (persistent) CTA in
// the same kind of layout, [dz][chunk][dx, descending][out channel][8].  The
// roles are split over warps and the items pipelined two deep: eight warps
// copy (16-byte asynchronous copies; tensor copies of this layout, whose
// innermost extent is 16 bytes, were no faster), one thread issues the
// tcgen05.mma instructions (kind::f16, BF16 x BF16 -> FP32 in tensor memory),
// and four warps read the finished 128 x N accumulators back with tcgen05.ld
// (warp w owns lanes 32w..32w+31, i.e. pixels 32w..32w+31) for the epilogue:
// bias + ReLU -> BF16 activations, bias -> FP32 outputs, or (input-gradient
// pass) the ReLU mask of the forward activation.
//
// Every wait is bounded: an mbarrier that does not complete within ~2 s
// sets the network's error flag; the CTA then waits for the multiplications
// it has committed (also bounded, run_items) and releases its tensor memory.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <random>
#include <vector>

#include "../../include/ouc.h"
#include "../../include/ouc_corrector.h"
#include "pipeline.h"

namespace ouc {
namespace cnn {

using bf16 = __nv_bfloat16;

constexpr int kTile = 128;            // GEMM M: pixels per tile
constexpr int kPC = kTile + 4;        // patch columns (2 + 2 halo)
constexpr int kTaps = 25;
constexpr int kMaxPairs = 32 * 32;     // (cin, cout) pairs of the widest layer
constexpr int kRB = 2;                 // image rows of a weight-gradient work item
constexpr int kCB = 4;                 // image rows of a convolution work item
constexpr int kWgradCtas = 148;        // CTAs (partial-sum slots) of k_wgrad_tc
constexpr int kBgradBlocks = 592;      // blocks of k_bgrad
constexpr int kCopyThreads = 256;      // copy warps 5-12
constexpr int kThreadsConv = 160 + kCopyThreads;   // epilogue warps 0-3, MMA warp 4, copy warps

struct LayerDims {
    int cin, cout, cin_pad, cout_pad;
};
constexpr LayerDims kL[4] = {{OUC_CNN_IN, OUC_CNN_WIDTH, 16, 32},
                             {OUC_CNN_WIDTH, OUC_CNN_WIDTH, 32, 32},
                             {OUC_CNN_WIDTH, OUC_CNN_WIDTH, 32, 32},
                             {OUC_CNN_WIDTH, OUC_CNN_OUT, 32, 16}};

constexpr int w_count(int l) { return kL[l].cout * kL[l].cin * kTaps; }
constexpr int p_offset(int l) { return l == 0 ? 0 : p_offset(l - 1) + w_count(l - 1) + kL[l - 1].cout; }
constexpr int kNParams = p_offset(3) + w_count(3) + kL[3].cout;

// ---- PTX helpers (tcgen05, mbarrier) ---------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor, no swizzle, K-major canonical layout:
// start address, leading-dimension byte offset (between the two 8-element K
// chunks), stride byte offset (between 8-row groups), all >> 4; version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :
        : "r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One hardware-suspended try: the thread sleeps until the phase completes or
// a time limit of about 0.1 ms passes (no busy polling beside the copies).
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity), "r"(100000u)
        : "memory");
    return done != 0;
}

// Bounded wait: false after 2^14 suspended tries (over a second).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < (1 << 14); ++i)
        if (mbar_try(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 16-byte asynchronous copy, zero-filled when !in (src is then not read).
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// The wait takes the loaded registers as operands, so that no use of them can
// be scheduled before it.
#define OUC_R16(r, o)                                                                                               \
    "+r"(r[o + 0]), "+r"(r[o + 1]), "+r"(r[o + 2]), "+r"(r[o + 3]), "+r"(r[o + 4]), "+r"(r[o + 5]), "+r"(r[o + 6]), \
        "+r"(r[o + 7]), "+r"(r[o + 8]), "+r"(r[o + 9]), "+r"(r[o + 10]), "+r"(r[o + 11]), "+r"(r[o + 12]),          \
        "+r"(r[o + 13]), "+r"(r[o + 14]), "+r"(r[o + 15])

template <int NC>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[NC]) {
    static_assert(NC == 16 || NC == 32, "16 or 32 columns");
    uint32_t q0[16], q1[16];
    tmem_ld16(taddr, q0);
    if (NC == 32) tmem_ld16(taddr + 16, q1);
    asm volatile("tcgen05.wait::ld.sync.aligned;" : OUC_R16(q0, 0)::"memory");
    if (NC == 32) asm volatile("" : OUC_R16(q1, 0));
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        r[k] = q0[k];
        if (NC == 32) r[16 + k] = q1[k];
    }
}

// ---- convolution kernel ----------------------------------------------------

enum Epi : int { kHidden = 0, kOut = 1, kDgrad = 2 };

struct ConvArgs {
    int n, H, W;
    const bf16* x;        // [n][H][W][CIN]
    const bf16* w;        // packed [tap][CIN / 8][COUT][8]
    const float* bias;    // [COUT] or null
    const bf16* mask;     // kDgrad: forward activation [n][H][W][COUT]
    void* y;              // bf16 [n][H][W][COUT] (kHidden, kDgrad) or float [n][H][W][cout_real] (kOut)
    int cout_real;
    int* err;
};

// Work items of RB rows x 128 pixels.
template <int RB>
struct Items {
    int tiles_w, row_blocks, count;
    __host__ __device__ Items(int n, int H, int W)
        : tiles_w((W + kTile - 1) / kTile), row_blocks((H + RB - 1) / RB), count(n * row_blocks * tiles_w) {}
    __device__ __forceinline__ void at(int item, int& img, int& h, int& z0) const {
        const int tw = item % tiles_w, rest = item / tiles_w;
        img = rest / row_blocks;
        h = (rest - img * row_blocks) * RB;
        z0 = tw * kTile;
    }
    // items of this CTA: blockIdx.x, then every gridDim.x-th
    __device__ __forceinline__ int of_cta() const {
        return count > (int)blockIdx.x ? (count - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    }
};

// This thread's copies have landed: make them visible to the tensor core's
// proxy and count the thread in.
__device__ __forceinline__ void hand_over(uint64_t* full) {
    cp_wait<0>();
    fence_proxy_async();
    mbar_arrive(full);
}

// Copy threads (t = 0 .. kCopyThreads-1): rows h .. h+ROWS-1, columns
// z .. z+COLS-1 of one NHWC image with C channels into shared memory as
// [row][chunk of 8][column][8 channels], zeros outside the image.  A thread
// keeps its chunk and column and walks down the rows.
template <int C, int ROWS, int COLS>
__device__ __forceinline__ void copy_patch(uint32_t dst, const bf16* x, int img, int h, int z, int H, int W, int t) {
    constexpr int NQ = C / 8, CPP = kCopyThreads / NQ;   // columns per pass
    const int q = t % NQ, c0 = t / NQ;
    const ptrdiff_t row = (ptrdiff_t)W * C;
#pragma unroll
    for (int p = 0; p < (COLS + CPP - 1) / CPP; ++p) {
        const int c = c0 + p * CPP, gz = z + c;
        if (c >= COLS) break;
        const bool col = gz >= 0 && gz < W;
        const bf16* src = x + (((ptrdiff_t)img * H + h) * W + gz) * C + q * 8;
        const uint32_t d = dst + (q * COLS + c) * 16;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const bool in = col && (unsigned)(h + r) < (unsigned)H;
            cp16(d + r * NQ * COLS * 16, in ? src + r * row : x, in);
        }
    }
}

template <int CIN, int COUT>
struct ConvGeo {
    static constexpr int NQ = CIN / 8;
    static constexpr int w_bytes = kTaps * CIN * COUT * 2;
    static constexpr int row_bytes = NQ * kPC * 16;
    static constexpr int p_bytes = (kCB + 4) * row_bytes;     // one stage
    static constexpr int bytes = w_bytes + 2 * p_bytes;
    static constexpr int acc_cols = 2 * kCB * COUT;
    static constexpr int tmem_cols = acc_cols <= 128 ? 128 : 256;
    static_assert(acc_cols <= 256, "two accumulator stages fit tensor memory");
};

// An input row i of an item (row h - 2 + i of the image) feeds the output rows
// o = i - dx, dx = 0 .. 4, with one A operand per column shift dz and channel
// chunk pair.  The accumulators of the item's rows lie side by side in tensor
// memory and the weights of the five dx side by side, in descending dx, in
// shared memory, so one MMA serves all of them (N up to 4 x COUT): 83 MMAs per
// item instead of 200.  Input rows run upwards, so that every output row
// still sums its taps in the order dx, dz, channel.
//
// Bound: the MMAs, about 85 cycles each nearly whatever their N (the same
// with the copies left out).  A 32 -> 32 layer on 4 images of 290 x 158:
// 72 us at first (128 threads staged the patch of one row, then waited for its
// MMAs), 33 us pipelined with an MMA per tap, 24 us with one for five.
template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(kThreadsConv, 1) k_conv5(const ConvArgs a) {
    using G = ConvGeo<CIN, COUT>;
    constexpr int NQ = G::NQ;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* s_w = smem;
    uint8_t* s_p = smem + G::w_bytes;
    __shared__ __align__(8) uint64_t full[2], done[2], drained[2];   // copied; multiplied; accumulators read
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const Items<kCB> items(a.n, a.H, a.W);
    const int mine = items.of_cta();

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full[s], kCopyThreads);
            mbar_init(&done[s], 1);
            mbar_init(&drained[s], 128);
        }
    }
    // weights [tap = dx 5 + dz][chunk][out channel][8] -> [dz][chunk][4 - dx][out channel][8]
    for (int i = tid; i < G::w_bytes / 16; i += kThreadsConv) {
        const int co = i % COUT, q = i / COUT % NQ, tap = i / (COUT * NQ), dx = tap / 5, dz = tap - 5 * dx;
        cp16(smem_u32(s_w) + (((dz * NQ + q) * 5 + 4 - dx) * COUT + co) * 16, a.w + (size_t)i * 8, true);
    }
    cp_commit();
    cp_wait<0>();
    fence_proxy_async();
    __syncwarp();   // .sync.aligned tcgen05 instructions need a converged warp
    if (warp == 0) tmem_alloc(&tmem_base, G::tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    bool ok = true;
    if (warp >= 5) {   // copies: a stage is free once the MMAs of the item two before are done
        int k = 0;
        for (int it = blockIdx.x; it < items.count; it += gridDim.x, ++k) {
            const int s = k & 1;
            if (k > 0) hand_over(&full[s ^ 1]);
            if (k >= 2 && !(ok = mbar_wait(&done[s], (uint32_t)((k >> 1) - 1) & 1u))) break;
            int img, h, z0;
            items.at(it, img, h, z0);
            copy_patch<CIN, kCB + 4, kPC>(smem_u32(s_p) + s * G::p_bytes, a.x, img, h - 2, z0 - 2, a.H, a.W, tid - 160);
            cp_commit();
        }
        if (k > 0 && ok) hand_over(&full[(k - 1) & 1]);
    } else if (tid == 128) {   // MMAs
        const uint64_t bd0 = umma_desc(smem_u32(s_w), 5 * COUT * 16, 128);
        const auto ready = [&](int k) {
            const uint32_t ph = (uint32_t)(k >> 1) & 1u;
            return (k < 2 || mbar_wait(&drained[k & 1], ph ^ 1u)) && mbar_wait(&full[k & 1], ph);
        };
        const auto issue = [&](int k) {
            const int s = k & 1;
            tc_fence_after();
            // descriptors: the start address (in 16-byte units) is the low
            // field, so a tap or chunk is one addition
            const uint64_t ad0 = umma_desc(smem_u32(s_p) + s * G::p_bytes, kPC * 16, 128);
            const uint32_t d0 = tmem + (uint32_t)(s * kCB * COUT);
#pragma unroll
            for (int i = 0; i < kCB + 4; ++i) {
                const int o0 = i > 4 ? i - 4 : 0, o1 = i < kCB ? i : kCB - 1;   // output rows o0 .. o1
                const int b0 = 4 - (i - o0);                                    // block of dx = i - o0
#pragma unroll
                for (int dz = 0; dz < 5; ++dz) {
#pragma unroll
                    for (int ks = 0; ks < NQ / 2; ++ks) {
                        const uint64_t ad = ad0 + (uint32_t)((i * NQ + 2 * ks) * kPC + dz);
                        const uint64_t bd = bd0 + (uint32_t)(((dz * NQ + 2 * ks) * 5 + b0) * COUT);
                        const bool first = i < kCB && dz == 0 && ks == 0;       // row i's first product overwrites
                        const int n = o1 - o0 + (first ? 0 : 1);
                        if (n > 0) umma_bf16(d0 + (uint32_t)(o0 * COUT), ad, bd, idesc_bf16(kTile, n * COUT), 1u);
                        if (first) umma_bf16(d0 + (uint32_t)(i * COUT), ad, bd + (uint32_t)((i - o0) * COUT), idesc_bf16(kTile, COUT), 0u);
                    }
                }
            }
            umma_commit(&done[s]);
        };
        ok = run_items(mine, ready, issue, [&](int s, uint32_t parity) { return mbar_wait(&done[s], parity); });
    } else if (warp < 4) {   // epilogue
        int k = 0;
        for (int it = blockIdx.x; it < items.count; it += gridDim.x, ++k) {
            const int s = k & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(&done[s], (uint32_t)(k >> 1) & 1u));
            if (!ok) break;
            tc_fence_after();
            int img, h, z0;
            items.at(it, img, h, z0);
            const int gz = z0 + warp * 32 + lane;
#pragma unroll 1
            for (int q = 0; q < kCB; ++q) {
                uint32_t r[COUT];
                __syncwarp();
                tmem_ld<COUT>(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((s * kCB + q) * COUT), r);
                if (q == kCB - 1) {
                    tc_fence_before();
                    mbar_arrive(&drained[s]);
                }
                if (gz >= a.W || h + q >= a.H) continue;
                const size_t p = ((size_t)img * a.H + h + q) * a.W + gz;
                if (EPI == kOut) {
                    float* y = static_cast<float*>(a.y) + p * a.cout_real;
#pragma unroll
                    for (int c = 0; c < COUT; ++c)
                        if (c < a.cout_real) y[c] = __uint_as_float(r[c]) + a.bias[c];   // the caller's buffer: float-aligned
                } else {
                    uint4* y = reinterpret_cast<uint4*>(static_cast<bf16*>(a.y) + p * COUT);
                    const uint4* mk = EPI == kDgrad ? reinterpret_cast<const uint4*>(a.mask + p * COUT) : nullptr;
#pragma unroll
                    for (int c8 = 0; c8 < COUT / 8; ++c8) {
                        __align__(16) bf16 o[8];
                        __align__(16) bf16 mv[8];
                        if (EPI == kDgrad) *reinterpret_cast<uint4*>(mv) = mk[c8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int c = 8 * c8 + e;
                            float v = __uint_as_float(r[c]);
                            if (EPI == kHidden) v = fmaxf(v + a.bias[c], 0.f);
                            else v = __bfloat162float(mv[e]) > 0.f ? v : 0.f;
                            o[e] = __float2bfloat16_rn(v);
                        }
                        y[c8] = *reinterpret_cast<const uint4*>(o);
                    }
                }
            }
        }
    }
    if (!ok) atomicExch(a.err, 1);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    __syncwarp();
    if (warp == 0) tmem_dealloc(tmem, G::tmem_cols);
}

template <int CIN, int COUT, int EPI>
cudaError_t launch_conv(const ConvArgs& a, int sms, cudaStream_t s) {
    constexpr int bytes = ConvGeo<CIN, COUT>::bytes;
    // the shared-memory opt-in is a per-device setting: set on the current
    // device at every launch (a host-side call; a few launches per step);
    // if it is refused nothing is launched and the caller reports it
    const cudaError_t e =
        cudaFuncSetAttribute(k_conv5<CIN, COUT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    const int count = Items<kCB>(a.n, a.H, a.W).count;
    k_conv5<CIN, COUT, EPI><<<count < sms ? count : sms, kThreadsConv, bytes, s>>>(a);
    return cudaSuccess;
}

// ---- weight gradients on the tensor cores ------------------------------------
//
// dW[tap][co][ci] = sum_p X[p + s(tap)][ci] G[p][co] over all pixels p, with
// s(dx, dz) = (dx - 2, dz - 2).  The pixels are the GEMM's K dimension, so
// the operand that carries the tap shift must move along K by whole 16-byte
// rows: both operands use the no-swizzle MN-major layout, in which K
// advances 16 bytes per pixel.  Per work item (kRB rows of 128 pixels) the
// copy warps bring
//   * the input patch, rows h-2..h+kRB+1 and columns z0-2..z0+129, as [row]
//     [channel chunk of 8][column][8 channels] -- the layout of k_conv5 -- so
//     that M = 128 consecutive 8-channel groups are (row, chunk) pairs at one
//     uniform stride: 4 rows x 32 channels (or 8 x 16), and the tap shift dz
//     is a start offset of 16 dz bytes.  The last row group of a pixel row
//     reads up to three rows beyond the five taps (whatever the buffer holds
//     there); their accumulator rows are never read;
//   * the output gradient of the tile, [row][chunk of 8 output channels]
//     [pixel][8 channels] with zeros beyond the row's end, the N operand;
// and one thread issues, for each row, 16 pixels, dz and row group, an MMA
// (kind::f16, BF16 inputs, FP32 accumulation in tensor memory):
// D[(dx, ci)][co], accumulated over all of the CTA's items.  Copies and MMAs
// of consecutive items overlap (two stages).  At the end each warp reads its
// 32 accumulator lanes (rows (dx, ci)) and writes the CTA's partial sums,
// which k_grad_sum adds in CTA order: the result does not depend on
// scheduling, so training repeats bit for bit.
//
// Bound: the MMAs, as above (3 of 8 rows are spent on the padding above).
// 32 -> 32, 4 images of 290 x 158: 370 -> 50 us
// (first form: 64 CTAs that staged and multiplied in turn).
template <int CIN, int COUT>
struct WgradGeo {
    static constexpr int NQ = CIN / 8;                  // input-channel chunks
    static constexpr int RPG = 128 / CIN;               // patch rows per M = 128 row group
    static constexpr int NRG = (5 + RPG - 1) / RPG;     // row groups covering dx = 0..4
    static constexpr int row_bytes = NQ * kPC * 16;
    static constexpr int p_bytes = (kRB + 4) * row_bytes;          // one stage
    static constexpr int slack = (NRG * RPG - 5) * row_bytes;      // rows read beyond the last stage's patch
    static constexpr int g_bytes = kRB * (COUT / 8) * kTile * 16;  // one stage
    static constexpr int oG = 2 * p_bytes + slack;
    static constexpr int bytes = oG + 2 * g_bytes;
    static_assert(row_bytes % 128 == 0 && oG % 128 == 0, "operand rows start on 128-byte boundaries");
    static constexpr int ncols = 5 * NRG * COUT;        // accumulator columns
    static constexpr int tmem_cols = ncols <= 32 ? 32 : ncols <= 64 ? 64 : ncols <= 128 ? 128 : ncols <= 256 ? 256 : 512;
    static_assert(ncols <= 512, "accumulators fit tensor memory");
};

// Instruction descriptor as idesc_bf16 with both operands MN-major
// (bit 15: A, bit 16: B).
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int M, int N) { return idesc_bf16(M, N) | (1u << 15) | (1u << 16); }

// No-swizzle MN-major descriptor: 8 K rows of 16 bytes per core matrix, K
// groups of 8 rows at `kgroup` bytes, M/N groups of 8 elements at `mgroup`
// bytes (leading-dimension offset = K-group stride, stride offset = M/N
// group stride for this layout).
__device__ __forceinline__ uint64_t umma_desc_mn(uint32_t saddr, uint32_t kgroup, uint32_t mgroup) {
    return umma_desc(saddr, kgroup, mgroup);
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(kThreadsConv, 1) k_wgrad_tc(int n, int H, int W, const bf16* x, const bf16* g,
                                                           int cin_real, int cout_real, float* part, int* err) {
    using G = WgradGeo<CIN, COUT>;
    constexpr int NQ = G::NQ, NRG = G::NRG, QO = COUT / 8;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* s_p = smem;
    uint8_t* s_g = smem + G::oG;
    __shared__ __align__(8) uint64_t full[2], done[2];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const Items<kRB> items(n, H, W);
    const int mine = items.of_cta();

    if (tid == 0)
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full[s], kCopyThreads);
            mbar_init(&done[s], 1);
        }
    __syncwarp();
    if (warp == 0) tmem_alloc(&tmem_base, G::tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    bool ok = true;
    if (warp >= 5) {   // copies, as in k_conv5
        int k = 0;
        for (; k < mine; ++k) {
            const int s = k & 1;
            if (k > 0) hand_over(&full[s ^ 1]);
            if (k >= 2 && !(ok = mbar_wait(&done[s], (uint32_t)((k >> 1) - 1) & 1u))) break;
            int img, h, z0;
            items.at(blockIdx.x + k * gridDim.x, img, h, z0);
            copy_patch<CIN, kRB + 4, kPC>(smem_u32(s_p) + s * G::p_bytes, x, img, h - 2, z0 - 2, H, W, tid - 160);
            copy_patch<COUT, kRB, kTile>(smem_u32(s_g) + s * G::g_bytes, g, img, h, z0, H, W, tid - 160);
            cp_commit();
        }
        if (k > 0 && ok) hand_over(&full[(k - 1) & 1]);
    } else if (tid == 128) {   // MMAs
        constexpr uint32_t idesc = idesc_bf16_mn(128, COUT);
        uint32_t acc = 0;
        const auto ready = [&](int k) { return mbar_wait(&full[k & 1], (uint32_t)(k >> 1) & 1u); };
        const auto issue = [&](int k) {
            const int s = k & 1;
            tc_fence_after();
            int img, h, z0;
            items.at(blockIdx.x + k * gridDim.x, img, h, z0);
            const int ksn = min(kTile, W - z0 + 15) / 16;   // 16-pixel steps that hold pixels of the row
            const uint64_t ad0 = umma_desc_mn(smem_u32(s_p) + s * G::p_bytes, 128, kPC * 16);
            const uint64_t bd0 = umma_desc_mn(smem_u32(s_g) + s * G::g_bytes, 128, kTile * 16);
#pragma unroll 1
            for (int r = 0; r < kRB && h + r < H; ++r) {
                const uint64_t adr = ad0 + (uint32_t)(r * NQ * kPC), bdr = bd0 + (uint32_t)(r * QO * kTile);
                // consecutive MMAs go to different accumulators
#pragma unroll 1
                for (int ks = 0; ks < ksn; ++ks) {
#pragma unroll
                    for (int dz = 0; dz < 5; ++dz) {
#pragma unroll
                        for (int rg = 0; rg < NRG; ++rg)
                            umma_bf16(tmem + (uint32_t)((dz * NRG + rg) * COUT), adr + (uint32_t)(rg * G::RPG * NQ * kPC + dz + 16 * ks),
                                      bdr + (uint32_t)(16 * ks), idesc, acc);
                    }
                    acc = 1;
                }
            }
            umma_commit(&done[s]);
        };
        ok = run_items(mine, ready, issue, [&](int s, uint32_t parity) { return mbar_wait(&done[s], parity); });
    }
    if (!ok) atomicExch(err, 1);
    tc_fence_before();
    ok = __syncthreads_and(ok);
    tc_fence_after();
    // accumulator row m = 32 warp + lane: 8-channel group j = m / 8 = (row in
    // group, chunk), channel e = m % 8; column (dz, rg) * COUT + co
    if (ok && mine > 0 && warp < 4) {
        const int m = warp * 32 + lane, j = m >> 3, e = m & 7;
        const int ci = (j % NQ) * 8 + e;
#pragma unroll 1
        for (int dz = 0; dz < 5; ++dz) {
#pragma unroll 1
            for (int rg = 0; rg < NRG; ++rg) {
                uint32_t r[COUT];
                __syncwarp();
                tmem_ld<COUT>(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((dz * NRG + rg) * COUT), r);
                const int dx = rg * G::RPG + j / NQ;
                if (dx < 5 && ci < cin_real) {
                    const int tap = dx * 5 + dz;
                    float* out = part + ((size_t)blockIdx.x * kTaps + tap) * kMaxPairs;
#pragma unroll
                    for (int co = 0; co < COUT; ++co)
                        if (co < cout_real) out[co * cin_real + ci] = __uint_as_float(r[co]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    __syncwarp();
    if (warp == 0) tmem_dealloc(tmem, G::tmem_cols);
}

template <int CIN, int COUT>
cudaError_t launch_wgrad(int n, int H, int W, const bf16* x, const bf16* g, int cin_real, int cout_real, float* part,
                         int* err, int* nblocks, cudaStream_t s) {
    constexpr int bytes = WgradGeo<CIN, COUT>::bytes;
    const cudaError_t e = cudaFuncSetAttribute(k_wgrad_tc<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    // a fixed grid (at most kWgradCtas partial-sum slots), independent of the device
    const int count = Items<kRB>(n, H, W).count, grid = count < kWgradCtas ? count : kWgradCtas;
    k_wgrad_tc<CIN, COUT><<<grid, kThreadsConv, bytes, s>>>(n, H, W, x, g, cin_real, cout_real, part, err);
    *nblocks = grid;
    return cudaSuccess;
}

// ---- gradient sums, bias gradients, packing, Adam ---------------------------

// Per-block sums of the output gradient's channels: a thread adds one chunk
// of 8 channels over its pixels, then the block adds its threads in a fixed
// order.  part[block][32].
template <int COUT>
__global__ void __launch_bounds__(256) k_bgrad(size_t npix, const bf16* g, float* part) {
    constexpr int QO = COUT / 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const uint4* g4 = reinterpret_cast<const uint4*>(g);
    const size_t n4 = npix * QO;   // the stride is a multiple of QO: a thread keeps its chunk
    for (size_t i = threadIdx.x + (size_t)blockIdx.x * 256; i < n4; i += (size_t)256 * gridDim.x) {
        const uint4 u = g4[i];
        __align__(16) bf16 v[8];
        *reinterpret_cast<uint4*>(v) = u;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += __bfloat162float(v[e]);
    }
    __shared__ float red[8][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
#pragma unroll
        for (int o = 16; o >= QO; o >>= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
        if (lane < QO) red[w][lane * 8 + e] = acc[e];
    }
    __syncthreads();
    if (threadIdx.x < COUT) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) s += red[k][threadIdx.x];
        part[(size_t)blockIdx.x * 32 + threadIdx.x] = s;
    }
}

// dw[co][ci][tap] += the CTAs' partial sums in a fixed order: eight threads
// each add an eighth of the CTAs in order, then the eight; the last four blocks
// add the bias sums, a warp per channel, lanes striding the blocks and a
// fixed tree over the lanes.
__global__ void __launch_bounds__(256) k_grad_sum(int nblocks, int cin_real, int cout_real, const float* part, float* dw,
                                                  int nbias, const float* bpart, float* db) {
    if (blockIdx.x >= gridDim.x - 4) {
        const int lane = threadIdx.x & 31, c = 8 * (int)(blockIdx.x - (gridDim.x - 4)) + (threadIdx.x >> 5);
        if (c >= cout_real) return;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < (kBgradBlocks + 31) / 32; ++k) {
            const int b = lane + 32 * k;
            if (b < nbias) s += bpart[(size_t)b * 32 + c];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) db[c] += s;
        return;
    }
    __shared__ float red[8][32];
    const int npairs = cin_real * cout_real, grp = threadIdx.x >> 5, t = threadIdx.x & 31;
    const int i = blockIdx.x * 32 + t;
    const bool in = i < kTaps * npairs;
    const int tap = in ? i / npairs : 0, pr = in ? i - tap * npairs : 0;
    const float* p = part + (size_t)tap * kMaxPairs + pr;
    const int b0 = nblocks * grp / 8, b1 = nblocks * (grp + 1) / 8;
    float s = 0.f;
#pragma unroll 8
    for (int b = b0; b < b1; ++b) s += p[(size_t)b * kTaps * kMaxPairs];
    red[grp][t] = s;
    __syncthreads();
    if (grp == 0 && in) {
        const int ci = pr % cin_real, co = pr / cin_real;
        float v = red[0][t];
#pragma unroll
        for (int k = 1; k < 8; ++k) v += red[k][t];
        dw[((size_t)co * cin_real + ci) * kTaps + tap] += v;
    }
}

// float [P][CREAL] -> bf16 [P][16], zero-padded channels; a thread per pixel.
template <int CREAL>
__global__ void __launch_bounds__(256) k_to_bf16(size_t npix, const float* in, bf16* out) {
    static_assert(CREAL <= 16, "padded to 16 channels");
    for (size_t p = threadIdx.x + (size_t)blockIdx.x * 256; p < npix; p += (size_t)256 * gridDim.x) {
        __align__(16) bf16 o[16];
        const float* f = in + p * CREAL;
#pragma unroll
        for (int c = 0; c < 16; ++c) o[c] = __float2bfloat16_rn(c < CREAL ? f[c] : 0.f);   // only float alignment is known
        uint4* y = reinterpret_cast<uint4*>(out + p * 16);
        y[0] = reinterpret_cast<const uint4*>(o)[0];
        y[1] = reinterpret_cast<const uint4*>(o)[1];
    }
}

// Pack W[cout][cin][5][5] (FP32) into the B-operand layout [tap][cin_pad/8][cout_pad][8]
// (forward), or, transposed and flipped, into the input-gradient weights
// W'[tap'][cout_pad/8][cin_pad][8] with W'[ci][co][tap'] = W[co][ci][24 - tap'].
__global__ void k_pack(const float* w, int cin, int cout, int cin_pad, int cout_pad, bool dgrad, bf16* out) {
    const int kin = dgrad ? cout_pad : cin_pad, kout = dgrad ? cin_pad : cout_pad;
    const int total = kTaps * kin * kout;
    for (int i = threadIdx.x + blockIdx.x * blockDim.x; i < total; i += blockDim.x * gridDim.x) {
        const int e = i % 8, rest = i / 8, o = rest % kout, rest2 = rest / kout, q = rest2 % (kin / 8),
                  tap = rest2 / (kin / 8);
        const int k = q * 8 + e;   // input channel of this (possibly transposed) convolution
        float v = 0.f;
        if (!dgrad) {
            if (k < cin && o < cout) v = w[((size_t)o * cin + k) * kTaps + tap];
        } else {
            if (k < cout && o < cin) v = w[((size_t)k * cin + o) * kTaps + (kTaps - 1 - tap)];
        }
        out[i] = __float2bfloat16_rn(v);
    }
}

__global__ void k_adam(int n, float* p, const float* g, float* m, float* v, float lr_t, float b1, float b2, float eps) {
    for (int i = threadIdx.x + blockIdx.x * blockDim.x; i < n; i += blockDim.x * gridDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr_t * mi / (sqrtf(vi) + eps);
    }
}

// Masked mean squared error of n images [n][H][W][8] against targets:
// g = 2 (y - t) / count on the rectangle [i0, i1) x [j0, j1) of every image
// and 0 elsewhere; loss += sum (y - t)^2 / count.
__global__ void k_mse(int n, int H, int W, int i0, int i1, int j0, int j1, float inv_count, const float* y,
                      const float* t, float* g, double* loss) {
    double acc = 0.0;
    const size_t P = (size_t)n * H * W;
    for (size_t p = threadIdx.x + (size_t)blockIdx.x * blockDim.x; p < P; p += (size_t)blockDim.x * gridDim.x) {
        const int j = (int)(p % W), i = (int)((p / W) % H);
        const bool in = i >= i0 && i < i1 && j >= j0 && j < j1;
#pragma unroll
        for (int c = 0; c < OUC_CNN_OUT; ++c) {
            const float d = in ? y[p * OUC_CNN_OUT + c] - t[p * OUC_CNN_OUT + c] : 0.f;
            g[p * OUC_CNN_OUT + c] = 2.f * d * inv_count;
            acc += (double)d * d;
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, acc * inv_count);
}

}  // namespace cnn
}  // namespace ouc

using namespace ouc::cnn;

struct ouc_cnn {
    int device = 0;
    int sms = 148;
    float* params = nullptr;     // FP32 master [kNParams]
    float* grads = nullptr;
    float* adam_m = nullptr;
    float* adam_v = nullptr;
    long long adam_t = 0;
    bf16* wf[4] = {};            // packed forward weights
    bf16* wd[4] = {};            // packed input-gradient weights (layers 1..3)
    int* err = nullptr;
    float* part = nullptr;       // gradient partial sums, reduced in a fixed order (kWgradCtas x 25 x kMaxPairs)
    float* bpart = nullptr;      // bias partial sums (kBgradBlocks x 32)
    // activations of the last forward
    int n = 0, H = 0, W = 0;
    size_t cap = 0;              // pixels the buffers hold
    bf16* x0 = nullptr;          // [P][16]
    bf16* y[3] = {};             // [P][32]
    bf16* g16 = nullptr;         // [P][16]  output-layer gradient
    bf16* g[2] = {};             // [P][32]
};

namespace {

int repack(ouc_cnn* net, cudaStream_t s) {
    for (int l = 0; l < 4; ++l) {
        const LayerDims d = kL[l];
        const float* w = net->params + p_offset(l);
        k_pack<<<64, 256, 0, s>>>(w, d.cin, d.cout, d.cin_pad, d.cout_pad, false, net->wf[l]);
        if (l > 0) k_pack<<<64, 256, 0, s>>>(w, d.cin, d.cout, d.cin_pad, d.cout_pad, true, net->wd[l]);
    }
    return cudaGetLastError() == cudaSuccess ? OUC_OK : OUC_ECUDA;
}

int ensure_acts(ouc_cnn* net, size_t P) {
    if (P <= net->cap) return OUC_OK;
    cudaFree(net->x0); cudaFree(net->g16);
    for (auto& p : net->y) cudaFree(p);
    for (auto& p : net->g) cudaFree(p);
    net->cap = 0;
    bool ok = cudaMalloc(&net->x0, P * 16 * 2) == cudaSuccess && cudaMalloc(&net->g16, P * 16 * 2) == cudaSuccess;
    for (auto& p : net->y) ok = ok && cudaMalloc(&p, P * 32 * 2) == cudaSuccess;
    for (auto& p : net->g) ok = ok && cudaMalloc(&p, P * 32 * 2) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        return OUC_ENOMEM;
    }
    net->cap = P;
    return OUC_OK;
}

}  // namespace

extern "C" {

int ouc_cnn_nparams(void) { return kNParams; }

int ouc_cnn_create(int device, ouc_cnn** out) {
    if (!out) return OUC_EINVAL;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return OUC_ENODEV;
    }
    cudaDeviceProp prop;
    if (cudaSetDevice(device) != cudaSuccess || cudaGetDeviceProperties(&prop, device) != cudaSuccess ||
        prop.major != 10)
        return OUC_ENODEV;
    ouc_cnn* net = new (std::nothrow) ouc_cnn();
    if (!net) return OUC_ENOMEM;
    net->device = device;
    net->sms = prop.multiProcessorCount;
    const size_t pb = (size_t)kNParams * 4;
    bool ok = cudaMalloc(&net->params, pb) == cudaSuccess && cudaMalloc(&net->grads, pb) == cudaSuccess &&
              cudaMalloc(&net->adam_m, pb) == cudaSuccess && cudaMalloc(&net->adam_v, pb) == cudaSuccess &&
              cudaMalloc(&net->err, sizeof(int)) == cudaSuccess &&
              cudaMalloc(&net->part, (size_t)kWgradCtas * kTaps * kMaxPairs * sizeof(float)) == cudaSuccess &&
              cudaMalloc(&net->bpart, (size_t)kBgradBlocks * 32 * sizeof(float)) == cudaSuccess;
    for (int l = 0; l < 4 && ok; ++l) {
        ok = cudaMalloc(&net->wf[l], (size_t)kTaps * kL[l].cin_pad * kL[l].cout_pad * 2) == cudaSuccess;
        if (ok && l > 0) ok = cudaMalloc(&net->wd[l], (size_t)kTaps * kL[l].cin_pad * kL[l].cout_pad * 2) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();
        ouc_cnn_destroy(net);
        return OUC_ENOMEM;
    }
    cudaMemset(net->params, 0, pb);
    cudaMemset(net->grads, 0, pb);
    cudaMemset(net->adam_m, 0, pb);
    cudaMemset(net->adam_v, 0, pb);
    cudaMemset(net->err, 0, sizeof(int));
    if (repack(net, nullptr) || cudaDeviceSynchronize() != cudaSuccess) {
        ouc_cnn_destroy(net);
        return OUC_ECUDA;
    }
    *out = net;
    return OUC_OK;
}

int ouc_cnn_destroy(ouc_cnn* net) {
    if (!net) return OUC_OK;
    cudaSetDevice(net->device);
    cudaDeviceSynchronize();
    cudaFree(net->params); cudaFree(net->grads); cudaFree(net->adam_m); cudaFree(net->adam_v); cudaFree(net->err); cudaFree(net->part); cudaFree(net->bpart);
    for (auto* p : net->wf) cudaFree(p);
    for (auto* p : net->wd) cudaFree(p);
    cudaFree(net->x0); cudaFree(net->g16);
    for (auto* p : net->y) cudaFree(p);
    for (auto* p : net->g) cudaFree(p);
    delete net;
    return OUC_OK;
}

int ouc_cnn_set_params(ouc_cnn* net, const float* params) {
    if (!net || !params) return OUC_EINVAL;
    cudaSetDevice(net->device);
    if (cudaMemcpy(net->params, params, (size_t)kNParams * 4, cudaMemcpyHostToDevice) != cudaSuccess) return OUC_ECUDA;
    if (repack(net, nullptr)) return OUC_ECUDA;
    return cudaDeviceSynchronize() == cudaSuccess ? OUC_OK : OUC_ECUDA;
}

int ouc_cnn_get_params(const ouc_cnn* net, float* params) {
    if (!net || !params) return OUC_EINVAL;
    cudaSetDevice(net->device);
    return cudaMemcpy(params, net->params, (size_t)kNParams * 4, cudaMemcpyDeviceToHost) == cudaSuccess ? OUC_OK
                                                                                                      : OUC_ECUDA;
}

int ouc_cnn_forward_dev(ouc_cnn* net, int n, int H, int W, const float* d_in, float* d_out, void* stream) {
    if (!net || !d_in || !d_out || n < 1 || H < 1 || W < 1) return OUC_EINVAL;
    cudaSetDevice(net->device);
    cudaStream_t s = (cudaStream_t)stream;
    const size_t P = (size_t)n * H * W;
    if (ensure_acts(net, P)) return OUC_ENOMEM;
    net->n = n; net->H = H; net->W = W;
    k_to_bf16<OUC_CNN_IN><<<1184, 256, 0, s>>>(P, d_in, net->x0);
    ConvArgs a{};
    a.n = n; a.H = H; a.W = W; a.err = net->err;
    a.x = net->x0; a.w = net->wf[0]; a.bias = net->params + p_offset(0) + w_count(0); a.y = net->y[0];
    if (launch_conv<16, 32, kHidden>(a, net->sms, s) != cudaSuccess) return OUC_ECUDA;
    for (int l = 1; l < 3; ++l) {
        a.x = net->y[l - 1]; a.w = net->wf[l]; a.bias = net->params + p_offset(l) + w_count(l); a.y = net->y[l];
        if (launch_conv<32, 32, kHidden>(a, net->sms, s) != cudaSuccess) return OUC_ECUDA;
    }
    a.x = net->y[2]; a.w = net->wf[3]; a.bias = net->params + p_offset(3) + w_count(3); a.y = d_out;
    a.cout_real = OUC_CNN_OUT;
    if (launch_conv<32, 16, kOut>(a, net->sms, s) != cudaSuccess) return OUC_ECUDA;
    return cudaGetLastError() == cudaSuccess ? OUC_OK : OUC_ECUDA;
}

int ouc_cnn_backward_dev(ouc_cnn* net, const float* d_gout, void* stream) {
    if (!net || !d_gout) return OUC_EINVAL;
    if (net->n == 0) return OUC_ESTATE;
    cudaSetDevice(net->device);
    cudaStream_t s = (cudaStream_t)stream;
    const int n = net->n, H = net->H, W = net->W;
    const size_t P = (size_t)n * H * W;
    int nb = 0;   // CTAs of the weight-gradient launch: partial-sum slots to add
    k_to_bf16<OUC_CNN_OUT><<<1184, 256, 0, s>>>(P, d_gout, net->g16);
    // layer 4: weights and bias, then the gradient into layer 3's output
    float* gp = net->grads;
    if (launch_wgrad<32, 16>(n, H, W, net->y[2], net->g16, kL[3].cin, kL[3].cout, net->part, net->err, &nb, s) !=
        cudaSuccess)
        return OUC_ECUDA;
    k_bgrad<16><<<kBgradBlocks, 256, 0, s>>>(P, net->g16, net->bpart);
    k_grad_sum<<<kTaps * kMaxPairs / 32 + 4, 256, 0, s>>>(nb, kL[3].cin, kL[3].cout, net->part, gp + p_offset(3), kBgradBlocks, net->bpart,
                                   gp + p_offset(3) + w_count(3));
    ConvArgs a{};
    a.n = n; a.H = H; a.W = W; a.err = net->err;
    a.x = net->g16; a.w = net->wd[3]; a.mask = net->y[2]; a.y = net->g[0];
    if (launch_conv<16, 32, kDgrad>(a, net->sms, s) != cudaSuccess) return OUC_ECUDA;
    // layers 3 and 2
    for (int l = 2; l >= 1; --l) {
        const bf16* gl = net->g[(2 - l) & 1];
        if (launch_wgrad<32, 32>(n, H, W, net->y[l - 1], gl, kL[l].cin, kL[l].cout, net->part, net->err, &nb, s) !=
            cudaSuccess)
            return OUC_ECUDA;
        k_bgrad<32><<<kBgradBlocks, 256, 0, s>>>(P, gl, net->bpart);
        k_grad_sum<<<kTaps * kMaxPairs / 32 + 4, 256, 0, s>>>(nb, kL[l].cin, kL[l].cout, net->part, gp + p_offset(l), kBgradBlocks, net->bpart,
                                   gp + p_offset(l) + w_count(l));
        a.x = gl; a.w = net->wd[l]; a.mask = net->y[l - 1]; a.y = net->g[(3 - l) & 1];
        if (launch_conv<32, 32, kDgrad>(a, net->sms, s) != cudaSuccess) return OUC_ECUDA;
    }
    // layer 1
    const bf16* g1 = net->g[0];
    if (launch_wgrad<16, 32>(n, H, W, net->x0, g1, kL[0].cin, kL[0].cout, net->part, net->err, &nb, s) != cudaSuccess)
        return OUC_ECUDA;
    k_bgrad<32><<<kBgradBlocks, 256, 0, s>>>(P, g1, net->bpart);
    k_grad_sum<<<kTaps * kMaxPairs / 32 + 4, 256, 0, s>>>(nb, kL[0].cin, kL[0].cout, net->part, gp + p_offset(0), kBgradBlocks, net->bpart,
                                   gp + p_offset(0) + w_count(0));
    return cudaGetLastError() == cudaSuccess ? OUC_OK : OUC_ECUDA;
}

int ouc_cnn_zero_grad(ouc_cnn* net, void* stream) {
    if (!net) return OUC_EINVAL;
    cudaSetDevice(net->device);
    return cudaMemsetAsync(net->grads, 0, (size_t)kNParams * 4, (cudaStream_t)stream) == cudaSuccess ? OUC_OK
                                                                                                      : OUC_ECUDA;
}

int ouc_cnn_get_grads(const ouc_cnn* net, float* grads) {
    if (!net || !grads) return OUC_EINVAL;
    cudaSetDevice(net->device);
    return cudaMemcpy(grads, net->grads, (size_t)kNParams * 4, cudaMemcpyDeviceToHost) == cudaSuccess ? OUC_OK
                                                                                                    : OUC_ECUDA;
}

int ouc_cnn_adam_step(ouc_cnn* net, float lr, float beta1, float beta2, float eps, void* stream) {
    if (!net || !(lr > 0) || !(beta1 >= 0 && beta1 < 1) || !(beta2 >= 0 && beta2 < 1) || !(eps > 0)) return OUC_EINVAL;
    cudaSetDevice(net->device);
    cudaStream_t s = (cudaStream_t)stream;
    ++net->adam_t;
    const double c1 = 1.0 - std::pow((double)beta1, (double)net->adam_t);
    const double c2 = 1.0 - std::pow((double)beta2, (double)net->adam_t);
    const float lr_t = (float)(lr * std::sqrt(c2) / c1);
    k_adam<<<64, 256, 0, s>>>(kNParams, net->params, net->grads, net->adam_m, net->adam_v, lr_t, beta1, beta2, eps);
    return repack(net, s);
}

int ouc_cnn_train(ouc_cnn* net, const float* d_in, const float* d_tgt, int npairs, int H, int W, int i0, int i1, int j0,
                  int j1, int batch, int epochs, float lr, unsigned seed, float* epoch_loss, void* stream) {
    if (!net || !d_in || !d_tgt || npairs < 1 || H < 1 || W < 1 || batch < 1 || epochs < 1 || !(lr > 0)) return OUC_EINVAL;
    if (!(0 <= i0 && i0 < i1 && i1 <= H && 0 <= j0 && j0 < j1 && j1 <= W)) return OUC_EINVAL;
    cudaSetDevice(net->device);
    cudaStream_t s = (cudaStream_t)stream;
    batch = std::min(batch, npairs);
    const size_t img = (size_t)H * W;
    float *bin = nullptr, *btg = nullptr, *by = nullptr, *bg = nullptr;
    double* dloss = nullptr;
    bool ok = cudaMalloc(&bin, batch * img * OUC_CNN_IN * 4) == cudaSuccess &&
              cudaMalloc(&btg, batch * img * OUC_CNN_OUT * 4) == cudaSuccess &&
              cudaMalloc(&by, batch * img * OUC_CNN_OUT * 4) == cudaSuccess &&
              cudaMalloc(&bg, batch * img * OUC_CNN_OUT * 4) == cudaSuccess &&
              cudaMalloc(&dloss, sizeof(double)) == cudaSuccess;
    int rc = ok ? OUC_OK : OUC_ENOMEM;
    std::vector<int> order(npairs);
    for (int k = 0; k < npairs; ++k) order[k] = k;
    std::mt19937 rng(seed);
    const int nb = (npairs + batch - 1) / batch;
    for (int e = 0; e < epochs && rc == OUC_OK; ++e) {
        std::shuffle(order.begin(), order.end(), rng);
        cudaMemsetAsync(dloss, 0, sizeof(double), s);
        for (int b = 0; b < nb && rc == OUC_OK; ++b) {
            const int n = std::min(batch, npairs - b * batch);
            for (int k = 0; k < n; ++k) {
                const size_t q = order[b * batch + k];
                cudaMemcpyAsync(bin + k * img * OUC_CNN_IN, d_in + q * img * OUC_CNN_IN, img * OUC_CNN_IN * 4,
                                cudaMemcpyDeviceToDevice, s);
                cudaMemcpyAsync(btg + k * img * OUC_CNN_OUT, d_tgt + q * img * OUC_CNN_OUT, img * OUC_CNN_OUT * 4,
                                cudaMemcpyDeviceToDevice, s);
            }
            if ((rc = ouc_cnn_forward_dev(net, n, H, W, bin, by, s))) break;
            const float inv = 1.f / ((float)n * (i1 - i0) * (j1 - j0) * OUC_CNN_OUT);
            k_mse<<<592, 256, 0, s>>>(n, H, W, i0, i1, j0, j1, inv, by, btg, bg, dloss);
            if ((rc = ouc_cnn_zero_grad(net, s)) || (rc = ouc_cnn_backward_dev(net, bg, s))) break;
            // bias-free network: a zero input gives a zero output
            for (int l = 0; l < 4; ++l)
                cudaMemsetAsync(net->grads + p_offset(l) + w_count(l), 0, kL[l].cout * sizeof(float), s);
            if ((rc = ouc_cnn_adam_step(net, lr, 0.9f, 0.999f, 1e-8f, s))) break;
        }
        double l = 0;
        if (rc == OUC_OK && cudaMemcpyAsync(&l, dloss, sizeof(double), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
            cudaStreamSynchronize(s) == cudaSuccess) {
            if (epoch_loss) epoch_loss[e] = (float)(l / nb);
        } else if (rc == OUC_OK) {
            rc = OUC_ECUDA;
        }
    }
    cudaStreamSynchronize(s);
    cudaFree(bin); cudaFree(btg); cudaFree(by); cudaFree(bg); cudaFree(dloss);
    if (rc == OUC_OK && cudaGetLastError() != cudaSuccess) rc = OUC_ECUDA;
    return rc;
}

int ouc_cnn_error(ouc_cnn* net) {
    if (!net) return OUC_EINVAL;
    cudaSetDevice(net->device);
    int e = 0;
    cudaMemcpy(&e, net->err, sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemset(net->err, 0, sizeof(int));
    return e;
}

}  // extern "C"
