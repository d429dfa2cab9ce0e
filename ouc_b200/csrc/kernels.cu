// Kernel instantiations and the small per-shot kernels (mute, imaging of
// the last level, image normalisation + Laplacian + FP64 stack, gather
// transposes, field packing).
#include <cuda_runtime.h>

#include <algorithm>

#include "fd_march.cuh"
#include "fd_small.cuh"
#include "fd_step.cuh"
#include "ouc_internal.h"

namespace ouc {

template <class K>
static cudaError_t configure_kernel(K kernel, int bytes) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return e;
}

template <int N, int MODE>
static cudaError_t configure_one() {
    cudaError_t e = configure_kernel(k_step<N, MODE>, TileGeo<N>::bytes);
    if (e == cudaSuccess) e = configure_kernel(k_step<N, MODE, MidGeo<N>>, MidGeo<N>::bytes);
    if (e == cudaSuccess) e = configure_kernel(k_small<N, MODE, 16, 1>, SmallGeo<N, 16>::bytes);
    if (e == cudaSuccess) e = configure_kernel(k_small<N, MODE, 16, 2>, SmallGeo<N, 16>::bytes);
    if (e == cudaSuccess) e = configure_kernel(k_small<N, MODE, 24, 1>, SmallGeo<N, 24>::bytes);
    if (e == cudaSuccess) e = configure_kernel(k_step_q<N, MODE>, TileGeo<N>::bytes);
    if (e == cudaSuccess) e = configure_kernel(k_march<N, MODE>, MarchGeo<N>::bytes);
    return e;
}

template <int N>
static cudaError_t configure_modes() {
    cudaError_t e = configure_kernel(k_small_back<N, 16, 1>, SmallGeo<N, 16>::bytes);
    if (e == cudaSuccess) e = configure_kernel(k_small_back<N, 16, 2>, SmallGeo<N, 16>::bytes);
    if (e == cudaSuccess) e = configure_kernel(k_small_back<N, 24, 1>, SmallGeo<N, 24>::bytes);
    if (e == cudaSuccess) e = configure_one<N, kFwd>();
    if (e == cudaSuccess) e = configure_one<N, kRcv>();
    if (e == cudaSuccess) e = configure_one<N, kRec>();
    return e;
}

// Shared-memory attributes of the step kernels of half-order N on the current
// device (a per-device setting): ouc_create sets them for its device, the
// no-allocation entry point at its set-up on each device.
cudaError_t configure_step_kernels(int N) {
    if (N == 2) return configure_modes<2>();
    if (N == 5) return configure_modes<5>();
    if (N == 6) return configure_modes<6>();
    return cudaErrorInvalidValue;
}

int march_segments(Mode mode, const StepArgs& a) {
    constexpr int RB = 16;
    const int row0 = mode == kRec ? (a.L / RB) * RB : 0;
    const int row_end = mode == kRec ? a.X - a.L : (a.X + RB - 1) / RB * RB;
    return (row_end - row0 + a.seg_rows - 1) / a.seg_rows;
}

struct Grid {
    int tiles_z, tiles;
};
static Grid grid_of(Mode mode, const StepArgs& a, int TX, int TZ) {
    const int rows = mode == kRec ? a.X - 2 * a.L : a.X, cols = mode == kRec ? a.Z - a.L - a.tile_z0 : a.Z;
    Grid g;
    g.tiles_z = (cols + TZ - 1) / TZ;
    g.tiles = (rows + TX - 1) / TX * g.tiles_z;
    return g;
}
// 24-row tiles may end beyond the rows the field allocation keeps for 32-row ones.
bool fits24(Mode mode, const StepArgs& a, int N) {
    const int rows = mode == kRec ? a.X - 2 * a.L : a.X, x0 = mode == kRec ? a.tile_x0 : 0;
    return x0 + (rows + 23) / 24 * 24 + N <= (int)(a.fstride / a.pitch) - kGX;
}
// Tile shape of a launch, or of two that run beside each other.  A launch
// lasts as long as its waves of CTAs, so what decides is how many tiles there
// are for the SMs.  us per forward step without strips / per back-step, one
// shot unless stated, B200, half-order 5 (6 where marked):
//     grid (padded)      small 16x1   small 24   small 16x2   mid    large
//     160 x 120 (6)        6.7          9.0         9.9       10.9    19.3
//     296 x 296           11.6          8.3         9.9       12.9    23.4
//     397 x 301 (6)       12.9         15.9        11.5       13.5    24.2
//     560 x 310 back      26.6         24.2        22.1       19.0    29.3
//     1060 x 560          44.0          -          35.1       24.1    28.9
//     1060 x 560, 2 shots 95.7         87.7        71.7       43.0    46.5
//     1060 x 560, 4 shots  -            -            -        84.5    82.3
// Small tiles in one wave: one CTA of 576 threads per SM (16 rows) or of 768
// (24 rows); two of 576 with fewer registers each up to two per SM and a
// third of a wave more (306 tiles, half-order 2: 10.9 against 11.9 us on 16 x
// 64 tiles; 334, a back-step of 296 x 296: 15.4 against 18.3; 350: 17.4
// against 14.9).  Beyond that 16 x 64 tiles, whose last wave is half as long as a 32 x 64 one, until
// the launch has about five waves of them; then the 32 x 64 tiles, which
// recompute less halo.
Tier pick_tier(int N, const StepArgs* rec, const StepArgs* other, Mode other_mode, int nshots) {
    int t16 = 0, t24 = 0, mid = 0;
    bool ok24 = true;
    auto add = [&](Mode mode, const StepArgs& a) {
        t16 += grid_of(mode, a, 16, 32).tiles * nshots;
        t24 += grid_of(mode, a, 24, 32).tiles * nshots;
        mid += grid_of(mode, a, 16, 64).tiles * nshots;
        ok24 = ok24 && fits24(mode, a, N);
    };
    if (rec) add(kRec, *rec);
    if (other) add(other_mode, *other);
    const int set = (other ? other : rec)->nsm, nsm = set > 0 ? set : 148;
    if (t16 <= nsm) return kSmall16;
    if (t24 <= nsm && ok24) return kSmall24;
    if (t16 <= 2 * nsm + nsm / 3) return kSmall16x2;
    return mid <= 10 * nsm ? kMid : kLarge;
}

template <int N, int MODE>
static void launch_one(const StepArgs& a, int tiles_x, int nshots, cudaStream_t s) {
    if (a.seg_rows > 0) {
        const int nseg = march_segments((Mode)MODE, a);
        k_march<N, MODE><<<dim3(nseg * a.tiles_z, nshots), kThreads, MarchGeo<N>::bytes, s>>>(a);
        return;
    }
    if (a.seg_rows < 0 && a.queue && a.order[MODE == kRec ? 1 : 0]) {
        const int ntiles = tiles_x * a.tiles_z;
        const int items = ntiles * nshots, grid = items < 2 * a.nsm ? items : 2 * a.nsm;
        k_step_q<N, MODE><<<grid, kThreads, TileGeo<N>::bytes, s>>>(a, nshots, ntiles);
        return;
    }
    const Mode mode = (Mode)MODE;
    const Tier tier = a.tier != kAuto ? (Tier)a.tier : pick_tier(N, nullptr, &a, mode, nshots);
    if (tier == kLarge) {
        launch_pdl(k_step<N, MODE>, dim3(tiles_x * a.tiles_z, nshots), kThreads, TileGeo<N>::bytes, s, a.ordinary, a);
        return;
    }
    StepArgs b = a;
    if (tier == kMid) {
        const Grid g = grid_of(mode, a, 16, 64);
        launch_pdl(k_step<N, MODE, MidGeo<N>>, dim3(g.tiles, nshots), kThreads, MidGeo<N>::bytes, s, a.ordinary, b);
        return;
    }
    const Grid g = grid_of(mode, a, tier == kSmall24 ? 24 : 16, 32);
    const dim3 grid(g.tiles, nshots);
    b.tiles_z = g.tiles_z;
    if (tier == kSmall24) launch_pdl(k_small<N, MODE, 24, 1>, grid, SmallGeo<N, 24>::NT, SmallGeo<N, 24>::bytes, s, a.ordinary, b);
    else if (tier == kSmall16) launch_pdl(k_small<N, MODE, 16, 1>, grid, SmallGeo<N, 16>::NT, SmallGeo<N, 16>::bytes, s, a.ordinary, b);
    else launch_pdl(k_small<N, MODE, 16, 2>, grid, SmallGeo<N, 16>::NT, SmallGeo<N, 16>::bytes, s, a.ordinary, b);
}

template <int N>
static int launch_back_n(const StepArgs& rec, const StepArgs& rcv, Tier tier, int nshots, cudaStream_t s) {
    const int tx = tier == kSmall24 ? 24 : 16;
    const Grid g0 = grid_of(kRec, rec, tx, 32), g1 = grid_of(kRcv, rcv, tx, 32);
    StepArgs a0 = rec, a1 = rcv;
    a0.tiles_z = g0.tiles_z;
    a1.tiles_z = g1.tiles_z;
    const dim3 grid(g0.tiles + g1.tiles, nshots);
    if (tier == kSmall24) launch_pdl(k_small_back<N, 24, 1>, grid, SmallGeo<N, 24>::NT, SmallGeo<N, 24>::bytes, s, rec.ordinary, a0, a1, g0.tiles);
    else if (tier == kSmall16) launch_pdl(k_small_back<N, 16, 1>, grid, SmallGeo<N, 16>::NT, SmallGeo<N, 16>::bytes, s, rec.ordinary, a0, a1, g0.tiles);
    else if (tier == kSmall16x2) launch_pdl(k_small_back<N, 16, 2>, grid, SmallGeo<N, 16>::NT, SmallGeo<N, 16>::bytes, s, rec.ordinary, a0, a1, g0.tiles);
    else return 1;
    return 0;
}

template <int N>
static int launch_mode(Mode m, const StepArgs& a, int tiles_x, int nshots, cudaStream_t s) {
    switch (m) {
        case kFwd: launch_one<N, kFwd>(a, tiles_x, nshots, s); return 0;
        case kRcv: launch_one<N, kRcv>(a, tiles_x, nshots, s); return 0;
        case kRec: launch_one<N, kRec>(a, tiles_x, nshots, s); return 0;
    }
    return 1;
}

// Refuses (returns 1) a launch whose state map is missing or whose now[]
// pointers are not fields of the mapped block, so that no step kernel runs
// a tensor copy with coordinates the map does not describe.
static int resolve_fields(const StepArgs& a, StepArgs& b) {
    if (!a.state0 || a.fstride == 0 || a.nfields <= 0) return 1;
    b = a;
    const float* f0 = a.state0 + (size_t)kGX * a.pitch + kZOFF;   // field 0 of slot 0, cell (0, 0)
    auto field_of = [&](const float* q) -> int {
        if (!q || q < f0) return -1;
        const size_t d = (size_t)(q - f0);
        return d % a.fstride == 0 && d / a.fstride < (size_t)a.nfields ? (int)(d / a.fstride) : -1;
    };
    for (int q = 0; q < 4; ++q) {
        b.now_field[q] = field_of(a.now[q]);
        if (b.now_field[q] < 0) return 1;
        b.past_field[q] = field_of(a.past[q]);
        b.rcv_field[q] = field_of(a.rcv[q]);
        if (q < 3) b.acc_field[q] = field_of(a.acc[q]);
        b.fold_field[q] = field_of(a.f_old[q]);
    }
    for (int q = 0; q < 8; ++q) b.o_field[q] = field_of(a.o[q]);
    return 0;
}

int launch_step(int N, Mode mode, const StepArgs& a, int tiles_x, int nshots, cudaStream_t s) {
    StepArgs b;
    if (resolve_fields(a, b)) return 1;
    switch (N) {
        case 2: return launch_mode<2>(mode, b, tiles_x, nshots, s);
        case 5: return launch_mode<5>(mode, b, tiles_x, nshots, s);
        case 6: return launch_mode<6>(mode, b, tiles_x, nshots, s);
    }
    return 1;
}

// The reconstruction + imaging of one back-step and the receiver step after
// it as one launch of small tiles.  Refuses as launch_step does, and any
// other tile shape.
int launch_back(int N, const StepArgs& rec, const StepArgs& rcv, int nshots, cudaStream_t s) {
    StepArgs b0, b1;
    if (resolve_fields(rec, b0) || resolve_fields(rcv, b1)) return 1;
    switch (N) {
        case 2: return launch_back_n<2>(b0, b1, (Tier)rcv.tier, nshots, s);
        case 5: return launch_back_n<5>(b0, b1, (Tier)rcv.tier, nshots, s);
        case 6: return launch_back_n<6>(b0, b1, (Tier)rcv.tier, nshots, s);
    }
    return 1;
}

TensorMapEncode tensor_map_encoder() {
    static TensorMapEncode fn = []() -> TensorMapEncode {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<TensorMapEncode>(p);
    }();
    return fn;
}

namespace {
template <int N>
cudaError_t encode_for(StepArgs& a, const float* state0, int pitch, int rows, int nfields, int nslots, size_t fstride) {
    using G = TileGeo<N>;
    TensorMapEncode enc = tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    // dimensions innermost first: columns, rows, fields, slots; strides in bytes
    const cuuint64_t dims[4] = {(cuuint64_t)pitch, (cuuint64_t)rows, (cuuint64_t)nfields, (cuuint64_t)nslots};
    const cuuint64_t strides[3] = {(cuuint64_t)pitch * 4, (cuuint64_t)fstride * 4, (cuuint64_t)fstride * nfields * 4};
    const cuuint32_t box[4] = {(cuuint32_t)G::UC, (cuuint32_t)G::UR, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    static_assert((G::UC * 4) % 16 == 0, "the box's rows are whole 16-byte units");
    if (reinterpret_cast<uintptr_t>(state0) % 16 != 0 || (pitch * 4) % 16 != 0 || (fstride * 4) % 16 != 0)
        return cudaErrorInvalidValue;
    const CUresult r = enc(&a.box_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(state0), dims, strides,
                           box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    const cuuint32_t own[4] = {(cuuint32_t)G::TZ, (cuuint32_t)G::TX, 1, 1};
    const CUresult r2 = enc(&a.own_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(state0), dims, strides,
                            own, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r2 != CUDA_SUCCESS) return cudaErrorInvalidValue;
    const cuuint32_t sbox[4] = {(cuuint32_t)G::SC, (cuuint32_t)G::SR, 1, 1};
    const CUresult r3 = enc(&a.s_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(state0), dims, strides,
                            sbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r3 != CUDA_SUCCESS) return cudaErrorInvalidValue;
    auto u_box = [&](CUtensorMap* m, int uc, int ur) {
        const cuuint32_t ubox[4] = {(cuuint32_t)uc, (cuuint32_t)ur, 1, 1};
        return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(state0), dims, strides, ubox, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!u_box(&a.mid_map, MidGeo<N>::UC, MidGeo<N>::UR) ||
        !u_box(&a.small_map[0], SmallGeo<N, 16>::UC, SmallGeo<N, 16>::UR) ||
        !u_box(&a.small_map[1], SmallGeo<N, 24>::UC, SmallGeo<N, 24>::UR))
        return cudaErrorInvalidValue;
    a.state0 = state0;
    a.fstride = fstride;
    a.nfields = nfields;
    return cudaSuccess;
}
}  // namespace

cudaError_t encode_box_map(StepArgs& a, const float* state0, int pitch, int rows, int nfields, int nslots,
                           size_t fstride, int N) {
    a.state0 = nullptr;
    if (N == 2) return encode_for<2>(a, state0, pitch, rows, nfields, nslots, fstride);
    if (N == 5) return encode_for<5>(a, state0, pitch, rows, nfields, nslots, fstride);
    if (N == 6) return encode_for<6>(a, state0, pitch, rows, nfields, nslots, fstride);
    return cudaErrorInvalidValue;
}

int step_smem_bytes(int N) {
    switch (N) {
        case 2: return TileGeo<2>::bytes;
        case 5: return TileGeo<5>::bytes;
        case 6: return TileGeo<6>::bytes;
    }
    return 0;
}

// Imaging at the last time level, where the reference correlates without a
// reconstruction step (corr_v at t = NT-1, PS:2361 after PS:2319-2324).
// Source P is the forward's final level; the receiver fields are the ones
// after the receiver's first back-step.
__global__ void k_image_only(const StepArgs p) {
    const int i = blockIdx.y + p.L;
    const size_t off = (size_t)blockIdx.z * p.shot_stride;
    for (int j = p.L + threadIdx.x + blockIdx.x * blockDim.x; j < p.Z - p.L; j += blockDim.x * gridDim.x) {
        const ptrdiff_t g = (ptrdiff_t)i * p.pitch + j + off;
        const float sx = p.now[0][g], sz = p.now[1][g];
        p.acc[0][g] += sx * p.rcv[0][g] + sz * p.rcv[1][g];
        p.acc[2][g] += sx * sx + sz * sz;
        p.acc[1][g] += sx * p.rcv[2][g] + sz * p.rcv[3][g];
    }
}

void launch_image_only(const StepArgs& a, int nshots, cudaStream_t s) {
    const int nx = a.X - 2 * a.L;
    dim3 grid((a.Z - 2 * a.L + 255) / 256, nx, nshots);
    k_image_only<<<grid, 256, 0, s>>>(a);
}

// image = num / illumination (image_fun, PS:1441-1455), then the 5-point
// Laplacian scaled by 1/dh^2 on [L+2, X-L-2) x [L+2, Z-L-2) (Laplace,
// PS:1457-1469), zero on the two-cell rim of the interior; written dense
// nx x nz and added into the FP64 stack.
__device__ __forceinline__ float img_at(const float* num, const float* den, ptrdiff_t g) { return num[g] / den[g]; }

// The same from compensated sums: value = acc - c, the quotient formed in
// double and rounded once.
__device__ __forceinline__ float img_at_comp(const float* num, const float* cn, const float* den, const float* cd,
                                             ptrdiff_t g) {
    return (float)(((double)num[g] - (double)cn[g]) / ((double)den[g] - (double)cd[g]));
}

__global__ void k_finalize(const FinalizeArgs f) {
    const int nx = f.X - 2 * f.L, nz = f.Z - 2 * f.L;
    const int ii = blockIdx.y;
    const int i = ii + f.L;
    for (int jj = threadIdx.x + blockIdx.x * blockDim.x; jj < nz; jj += blockDim.x * gridDim.x) {
        const int j = jj + f.L;
        const size_t o = (size_t)ii * nz + jj;
        double spp = 0.0, sps = 0.0, sil = 0.0;
        for (int b = 0; b < f.nshots; ++b) {   // shots in order: the FP64 stack is deterministic
            const ptrdiff_t g = (ptrdiff_t)i * f.pitch + j + (ptrdiff_t)(b * f.shot_stride);
            float lpp = 0.f, lps = 0.f;
            if (i >= f.L + 2 && i < f.X - f.L - 2 && j >= f.L + 2 && j < f.Z - f.L - 2) {
                const float* npp = f.acc[0];
                const float* nps = f.acc[1];
                const float* den = f.acc[2];
                const ptrdiff_t P = f.pitch;
                const float c = 1 / f.dh / f.dh;
                if (!f.comp[0]) {
                    lpp = c * (img_at(npp, den, g + P) + img_at(npp, den, g - P) - 2 * img_at(npp, den, g) +
                               img_at(npp, den, g + 1) + img_at(npp, den, g - 1) - 2 * img_at(npp, den, g));
                    lps = c * (img_at(nps, den, g + P) + img_at(nps, den, g - P) - 2 * img_at(nps, den, g) +
                               img_at(nps, den, g + 1) + img_at(nps, den, g - 1) - 2 * img_at(nps, den, g));
                } else {
                    const float *cpp = f.comp[0], *cps = f.comp[1], *cd = f.comp[2];
                    auto ip = [&](ptrdiff_t q) { return img_at_comp(npp, cpp, den, cd, q); };
                    auto is = [&](ptrdiff_t q) { return img_at_comp(nps, cps, den, cd, q); };
                    lpp = c * (ip(g + P) + ip(g - P) - 2 * ip(g) + ip(g + 1) + ip(g - 1) - 2 * ip(g));
                    lps = c * (is(g + P) + is(g - P) - 2 * is(g) + is(g + 1) + is(g - 1) - 2 * is(g));
                }
            }
            if (f.img) {
                f.img[((size_t)b * 2 + 0) * nx * nz + o] = lpp;
                f.img[((size_t)b * 2 + 1) * nx * nz + o] = lps;
            }
            spp += (double)lpp;
            sps += (double)lps;
            sil += f.illum_scale * (f.comp[2] ? (double)f.acc[2][g] - (double)f.comp[2][g] : (double)f.acc[2][g]);
        }
        if (f.stack[0] && !(f.status && *f.status)) {   // a failed batch leaves the stack as it was
            f.stack[0][o] += spp;
            f.stack[1][o] += sps;
            f.stack[2][o] += sil;
        }
    }
}

// Conversion of one f16 strip slot from the staging ring once its field
// maxima are complete (the forward step converts slot t-1 itself; this
// converts the last slot).  blockIdx.y = shot; a shot's fields follow each
// other at its own ring's length, shorter than the context's on a sub-grid.
__global__ void k_strip_pack(const ShotDesc* shots, int slot) {
    const ShotDesc& d = shots[blockIdx.y];
    const size_t ring = d.ring.R, n = kStripFields * ring;
    const float* src = d.stage + (size_t)(slot & 1) * d.strip_slot;
    __half* dst = reinterpret_cast<__half*>(d.strips) + (size_t)slot * d.strip_slot;
    const unsigned* am = d.amax + (size_t)slot * kStripFields;
    for (size_t e = threadIdx.x + (size_t)blockIdx.x * blockDim.x; e < n; e += (size_t)blockDim.x * gridDim.x)
        dst[e] = __float2half_rn(scale2(src[e], f16_exp(am[e / ring])));
}

void launch_strip_pack(const ShotDesc* shots, int nshots, int slot, size_t strip_slot, cudaStream_t s) {
    const int blocks = (int)std::min<size_t>((strip_slot + 255) / 256, 1184);   // of the widest possible shot
    k_strip_pack<<<dim3(blocks, nshots), 256, 0, s>>>(shots, slot);
}

// ---- source-wavefield snapshots ---------------------------------------------

__device__ __forceinline__ size_t snap_index(const SnapArgs& a, int b, int comp, int ii, int jj) {
    return (size_t)b * a.shot_elems + ((size_t)a.slot * 2 + comp) * a.nx * a.nz + (size_t)ii * a.nz + jj;
}

// Largest |Px|, |Pz| of each shot's interior (f16 snapshots): block maxima,
// then one atomic per block and component.  grid (z blocks, nx, shots).
__global__ void k_snap_amax(const SnapArgs a) {
    const int ii = blockIdx.y, b = blockIdx.z;
    const size_t off = (size_t)b * a.shot_stride;
    float m0 = 0.f, m1 = 0.f;
    for (int jj = threadIdx.x + blockIdx.x * blockDim.x; jj < a.nz; jj += blockDim.x * gridDim.x) {
        const ptrdiff_t g = (ptrdiff_t)(ii + a.L) * a.pitch + (jj + a.L) + off;
        m0 = fmaxf(m0, fabsf(a.px[g]));
        m1 = fmaxf(m1, fabsf(a.pz[g]));
    }
    __shared__ float red[2][32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
        m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    }
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) { red[0][w] = m0; red[1][w] = m1; }
    __syncthreads();
    if (threadIdx.x < 2) {
        float m = 0.f;
        for (int q = 0; q < nw; ++q) m = fmaxf(m, red[threadIdx.x][q]);
        if (m > 0.f) atomicMax(a.amax + ((size_t)b * a.nslots + a.slot) * 2 + threadIdx.x, __float_as_uint(m));
    }
}

// Store the interior Px, Pz as snapshot `slot` in the snapshot type.
__global__ void k_snap_store(const SnapArgs a) {
    const int ii = blockIdx.y, b = blockIdx.z;
    const size_t off = (size_t)b * a.shot_stride;
    int k0 = 0, k1 = 0;
    if (a.prec == kStripF16) {
        const unsigned* am = a.amax + ((size_t)b * a.nslots + a.slot) * 2;
        k0 = f16_exp(am[0]);
        k1 = f16_exp(am[1]);
    }
    for (int jj = threadIdx.x + blockIdx.x * blockDim.x; jj < a.nz; jj += blockDim.x * gridDim.x) {
        const ptrdiff_t g = (ptrdiff_t)(ii + a.L) * a.pitch + (jj + a.L) + off;
        const float v0 = a.px[g], v1 = a.pz[g];
        const size_t e0 = snap_index(a, b, 0, ii, jj), e1 = snap_index(a, b, 1, ii, jj);
        if (a.prec == kStripF32) {
            static_cast<float*>(a.snaps)[e0] = v0;
            static_cast<float*>(a.snaps)[e1] = v1;
        } else if (a.prec == kStripBF16) {
            static_cast<__nv_bfloat16*>(a.snaps)[e0] = __float2bfloat16_rn(v0);
            static_cast<__nv_bfloat16*>(a.snaps)[e1] = __float2bfloat16_rn(v1);
        } else {
            static_cast<__half*>(a.snaps)[e0] = __float2half_rn(scale2(v0, k0));
            static_cast<__half*>(a.snaps)[e1] = __float2half_rn(scale2(v1, k1));
        }
    }
}

void launch_snap_store(const SnapArgs& a, int nshots, cudaStream_t s) {
    const dim3 grid((a.nz + 255) / 256, a.nx, nshots);
    if (a.prec == kStripF16) k_snap_amax<<<grid, 256, 0, s>>>(a);
    k_snap_store<<<grid, 256, 0, s>>>(a);
}

__device__ __forceinline__ float snap_get(const SnapArgs& a, size_t e, int k) {
    if (a.prec == kStripF32) return static_cast<const float*>(a.snaps)[e];
    if (a.prec == kStripBF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(a.snaps)[e]);
    return scale2(__half2float(static_cast<const __half*>(a.snaps)[e]), -k);
}

__device__ __forceinline__ void kahan_add(float* acc, float* c, float term) {
    const float y = __fsub_rn(term, *c);
    const float t = __fadd_rn(*acc, y);
    *c = __fsub_rn(__fsub_rn(t, *acc), y);
    *acc = t;
}

// Zero-lag imaging at a snapshot level: the stored source P against the
// receiver wavefield after its back-step, with the rounding of corr_v
// (acc + fma(p, q, u v), PS:1434-1436).  grid (z blocks, nx, shots).
__global__ void k_image_snap(const SnapArgs a) {
    const int ii = blockIdx.y, b = blockIdx.z;
    const size_t off = (size_t)b * a.shot_stride;
    int k0 = 0, k1 = 0;
    if (a.prec == kStripF16) {
        const unsigned* am = a.amax + ((size_t)b * a.nslots + a.slot) * 2;
        k0 = f16_exp(am[0]);
        k1 = f16_exp(am[1]);
    }
    for (int jj = threadIdx.x + blockIdx.x * blockDim.x; jj < a.nz; jj += blockDim.x * gridDim.x) {
        const ptrdiff_t g = (ptrdiff_t)(ii + a.L) * a.pitch + (jj + a.L) + off;
        const float sx = snap_get(a, snap_index(a, b, 0, ii, jj), k0);
        const float sz = snap_get(a, snap_index(a, b, 1, ii, jj), k1);
        const float rpx = a.rcv[0][g], rpz = a.rcv[1][g], rsx = a.rcv[2][g], rsz = a.rcv[3][g];
        const float tpp = __fmaf_rn(sx, rpx, __fmul_rn(sz, rpz));
        const float tps = __fmaf_rn(sx, rsx, __fmul_rn(sz, rsz));
        const float til = __fmaf_rn(sx, sx, __fmul_rn(sz, sz));
        if (!a.comp_image) {
            a.acc[0][g] = __fadd_rn(a.acc[0][g], tpp);
            a.acc[1][g] = __fadd_rn(a.acc[1][g], tps);
            a.acc[2][g] = __fadd_rn(a.acc[2][g], til);
        } else {
            kahan_add(a.acc[0] + g, a.comp[0] + g, tpp);
            kahan_add(a.acc[1] + g, a.comp[1] + g, tps);
            kahan_add(a.acc[2] + g, a.comp[2] + g, til);
        }
    }
}

void launch_image_snap(const SnapArgs& a, int nshots, cudaStream_t s) {
    k_image_snap<<<dim3((a.nz + 255) / 256, a.nx, nshots), 256, 0, s>>>(a);
}

void launch_finalize(const FinalizeArgs& f, cudaStream_t s) {
    const int nx = f.X - 2 * f.L, nz = f.Z - 2 * f.L;
    dim3 grid((nz + 255) / 256, nx);
    k_finalize<<<grid, 256, 0, s>>>(f);
}

// Direct-wave mute (remove, PS:1634-1657) on a time-major gather [nt][X]:
// zero sample t of receiver i when t < 2 t0 + dist(i) * dh / (dt * v), with
// the reference's mix of float and double arithmetic.
__global__ void k_mute(float* gx, float* gz, int X, int nt, int sx, int sz, int rz, int t0, float dt, float dh,
                       float v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= X) return;
    const int dxi = abs(sx - i), dzi = abs(rz - sz);
    const float dist = sqrtf(float(dxi * dxi + dzi * dzi));
    const double thr = 2 * t0 + (double)(dist * dh) * 1.0 / (double)(dt * v);
    for (int t = blockIdx.y; t < nt; t += gridDim.y) {
        if (t < thr) {
            gx[(size_t)t * X + i] = 0.f;
            gz[(size_t)t * X + i] = 0.f;
        }
    }
}

void launch_mute(float* gx, float* gz, int X, int nt, int sx, int sz, int rz, int t0, float dt, float dh, float v,
                 cudaStream_t s) {
    dim3 grid((X + 127) / 128, nt < 1024 ? nt : 1024);
    k_mute<<<grid, 128, 0, s>>>(gx, gz, X, nt, sx, sz, rz, t0, dt, dh, v);
}

// Non-finite detector: bit 1 of *status when any of the n floats at p is
// NaN or infinite (an unstable or overflowing run).  One vote per warp, one
// atomic per warp that saw one; the data is only read.
__global__ void k_finite(const float* __restrict__ p, size_t n, int* status) {
    bool bad = false;
    const size_t n4 = n / 4;
    const float4* p4 = reinterpret_cast<const float4*>(p);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        const float4 v = p4[i];
        bad |= !isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z) || !isfinite(v.w);
    }
    for (size_t i = 4 * n4 + blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        bad |= !isfinite(p[i]);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, 2);
}

void launch_finite_check(const float* p, size_t n, int* status, cudaStream_t s) {
    k_finite<<<1184, 256, 0, s>>>(p, n, status);   // 8 CTAs of 256 per SM, grid-stride
}

// out[c][r] = in[r][c] through a 32x33 shared tile.
__global__ void k_transpose(const float* __restrict__ in, float* __restrict__ out, int rows, int cols) {
    __shared__ float tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int r = r0 + k, c = c0 + threadIdx.x;
        if (r < rows && c < cols) tile[k][threadIdx.x] = in[(size_t)r * cols + c];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int c = c0 + k, r = r0 + threadIdx.x;
        if (r < rows && c < cols) out[(size_t)c * rows + r] = tile[threadIdx.x][k];
    }
}

void launch_transpose(const float* in, float* out, int rows, int cols, cudaStream_t s) {
    dim3 grid((cols + 31) / 32, (rows + 31) / 32);
    k_transpose<<<grid, dim3(32, 8), 0, s>>>(in, out, rows, cols);
}

// Gather nf pitched fields into a dense [nf][X][Z] buffer.
// FWI gradient of one back-step (the formula of the reference's unused
// gradfun, PS:1518-1575), for every shot of the launch (blockIdx.y):
//   G_vp -= 2 rho Vp (dUx/dx + dUz/dz) theta_r
//   G_vs -= 2 rho Vs (omega_r (dUx/dz - dUz/dx) + Qzx_r dUz/dx + Qzz_r dUz/dz + Qxz_r dUx/dz + Qxx_r dUx/dx)
//   S    += Ux_s^2 + Uz_s^2
// with U_s = P + S of the source at the imaged level, its staggered
// derivatives (dUx/dx = D-x, dUz/dz = D-z, dUz/dx = D+x, dUx/dz = D+z), and
// the receiver's stress fields from U_r = P + S after the back-step
// (PS:373-378 without damping memories), on [L+N, X-L-N) x [L+N, Z-L-N):
// every stencil reads interior cells only.  A CTA stages the four U fields
// of a 16 x 64 tile with an N-row and 8-column halo in shared memory.
//
// Derivative sums run as acc = fma(a_k, d_k, acc) from 0, k = 1 .. N, then one
// correctly rounded division.  Bound: shared-memory loads and issue; float4
// windows, packed x derivatives and the corrected-reciprocal division in place
// of scalar loads and IEEE divisions, and no work in tiles outside the
// gradient's cells: 6 shots of 280 x 190, 29.7 -> 9.6 us.
template <int N, bool PLUS>
__device__ __forceinline__ float4 grad_dx(const float* col, int st, const float* a, const Div& dv) {
    float2 l = dup2(0.f), h = dup2(0.f);
#pragma unroll
    for (int k = 1; k <= N; ++k) {
        const float4 hi = ld4(col + (PLUS ? k : k - 1) * st), lo = ld4(col + (PLUS ? 1 - k : -k) * st);
        l = fma2(dup2(a[k - 1]), sub2(lo2(hi), lo2(lo)), l);
        h = fma2(dup2(a[k - 1]), sub2(hi2(hi), hi2(lo)), h);
    }
    return div4(cat4(l, h), dv);
}
template <int N, bool PLUS>
__device__ __forceinline__ float4 grad_dz(const float* row, const float* a, const Div& dv) {
    constexpr int NB = (N + 3) / 4;
    float w[4 * (2 * NB + 1)];
#pragma unroll
    for (int b = 0; b < 2 * NB + 1; ++b) {
        const float4 v = ld4(row + 4 * (b - NB));
        w[4 * b + 0] = v.x; w[4 * b + 1] = v.y; w[4 * b + 2] = v.z; w[4 * b + 3] = v.w;
    }
    float o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = 4 * NB + q;
        float acc = 0.f;
#pragma unroll
        for (int k = 1; k <= N; ++k)
            acc = PLUS ? __fmaf_rn(a[k - 1], __fsub_rn(w[c + k], w[c - k + 1]), acc)
                       : __fmaf_rn(a[k - 1], __fsub_rn(w[c + k - 1], w[c - k]), acc);
        o[q] = acc;
    }
    return div4(make_float4(o[0], o[1], o[2], o[3]), dv);
}

template <int N>
__global__ void __launch_bounds__(256) k_grad(const GradArgs a) {
    constexpr int TR = 16, TC = 64, HC = 8, BR = TR + 2 * N, BC = TC + 2 * HC;
    __shared__ float4 sbox4[4 * BR * BC / 4];
    float* box = reinterpret_cast<float*>(sbox4);
    const int b = blockIdx.y;
    const int tiles_c = (a.Z + TC - 1) / TC;
    const int x0 = (blockIdx.x / tiles_c) * TR, z0 = (blockIdx.x % tiles_c) * TC;
    // tiles without a gradient cell
    if (x0 + TR <= a.L + N || z0 + TC <= a.L + N || z0 >= a.Z - a.L - N) return;
    const size_t off = (size_t)b * a.shot_stride;
    for (int k = threadIdx.x; k < BR * (BC / 4); k += blockDim.x) {
        const int r = k / (BC / 4), c4 = k - r * (BC / 4);
        const ptrdiff_t g = (ptrdiff_t)(x0 - N + r) * a.pitch + (z0 - HC + 4 * c4);
        float4 v[8];
#pragma unroll
        for (int f = 0; f < 4; ++f) { v[f] = ldg4(a.src[f] + off + g); v[4 + f] = ldg4(a.rcv[f] + off + g); }
        float4* o = sbox4 + r * (BC / 4) + c4;
        o[0 * BR * BC / 4] = add4(v[0], v[2]);   // P + S: source Ux, Uz, receiver Ux, Uz
        o[1 * BR * BC / 4] = add4(v[1], v[3]);
        o[2 * BR * BC / 4] = add4(v[4], v[6]);
        o[3 * BR * BC / 4] = add4(v[5], v[7]);
    }
    __syncthreads();
    float w[N];
#pragma unroll
    for (int k = 0; k < N; ++k) w[k] = a.a[k];
    const Div dvx = make_div(a.dx, a.rdx), dvz = make_div(a.dz, a.rdz);
    const int r = threadIdx.x / (TC / 4), c0 = 4 * (threadIdx.x % (TC / 4));
    const int i = x0 + r;
    if (i < a.L + N || i >= a.X - a.L - N || z0 + c0 + 4 <= a.L + N || z0 + c0 >= a.Z - a.L - N) return;
    const int at = (r + N) * BC + (c0 + HC);
    const float* usx = box + at;
    const float* usz = box + BR * BC + at;
    const float* urx = box + 2 * BR * BC + at;
    const float* urz = box + 3 * BR * BC + at;
    const ptrdiff_t g = (ptrdiff_t)i * a.pitch + z0 + c0;
    const size_t og = (size_t)b * a.grad_stride + g;
    const float4 vpv = ldg4(a.vp + g), vsv = ldg4(a.vs + g);
    float4 rhov = make_float4(1.f, 1.f, 1.f, 1.f);
    if (a.rho) rhov = ldg4(a.rho + g);
    float4 g0 = ldg4(a.g[0] + og), g1 = ldg4(a.g[1] + og), g2 = ldg4(a.g[2] + og);
    const float4 sxx4 = grad_dx<N, false>(usx, BC, w, dvx), szx4 = grad_dx<N, true>(usz, BC, w, dvx);
    const float4 rxx4 = grad_dx<N, false>(urx, BC, w, dvx), rzx4 = grad_dx<N, true>(urz, BC, w, dvx);
    const float4 szz4 = grad_dz<N, false>(usz, w, dvz), sxz4 = grad_dz<N, true>(usx, w, dvz);
    const float4 rzz4 = grad_dz<N, false>(urz, w, dvz), rxz4 = grad_dz<N, true>(urx, w, dvz);
    const float4 ux4 = ld4(usx), uz4 = ld4(usz);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int j = z0 + c0 + q;
        if (j < a.L + N || j >= a.Z - a.L - N) continue;
        const float sxx = comp(sxx4, q), szz = comp(szz4, q), szx = comp(szx4, q), sxz = comp(sxz4, q);
        const float rxx = comp(rxx4, q), rzz = comp(rzz4, q), rzx = comp(rzx4, q), rxz = comp(rxz4, q);
        const float vp = comp(vpv, q), vs = comp(vsv, q), vp2 = vp * vp, vs2 = vs * vs;
        const float rho = comp(rhov, q);
        const float th = vp2 * (rxx + rzz), om = vs2 * (rxz - rzx);
        // om (sxz - szx) + vs2 rzx szx + vs2 rzz szz + vs2 rxz sxz + vs2 rxx sxx
        float s_vs = __fmaf_rn(om, __fsub_rn(sxz, szx), __fmul_rn(__fmul_rn(vs2, rzx), szx));
        s_vs = __fmaf_rn(__fmul_rn(vs2, rzz), szz, s_vs);
        s_vs = __fmaf_rn(__fmul_rn(vs2, rxz), sxz, s_vs);
        s_vs = __fmaf_rn(__fmul_rn(vs2, rxx), sxx, s_vs);
        set_comp(g0, q, comp(g0, q) - 2.f * rho * vp * ((sxx + szz) * th));
        set_comp(g1, q, comp(g1, q) - 2.f * rho * vs * s_vs);
        const float ux = comp(ux4, q), uz = comp(uz4, q);
        set_comp(g2, q, comp(g2, q) + (ux * ux + uz * uz));
    }
    stg4(a.g[0] + og, g0);
    stg4(a.g[1] + og, g1);
    stg4(a.g[2] + og, g2);
}

void launch_grad(const GradArgs& a, cudaStream_t s) {
    // tile rows only up to the last gradient row X-L-N-1: the staged rows then
    // end below X-L+14, inside the fields' 16 guard rows
    const int tiles = ((a.X - a.L - a.N + 15) / 16) * ((a.Z + 63) / 64);
    const dim3 grid(tiles, a.nshots);
    if (a.N == 2) k_grad<2><<<grid, 256, 0, s>>>(a);
    else if (a.N == 5) k_grad<5><<<grid, 256, 0, s>>>(a);
    else k_grad<6><<<grid, 256, 0, s>>>(a);
}

// FP64 stack of the shots' gradients over the interior, shots in order.
__global__ void k_grad_stack(const GradStackArgs a) {
    const int nz = a.Z - 2 * a.L;
    const int ii = blockIdx.y, i = ii + a.L;
    for (int jj = threadIdx.x + blockIdx.x * blockDim.x; jj < nz; jj += blockDim.x * gridDim.x) {
        const ptrdiff_t g = (ptrdiff_t)i * a.pitch + jj + a.L;
        double s[3] = {0.0, 0.0, 0.0};
        for (int b = 0; b < a.nshots; ++b)
            for (int k = 0; k < 3; ++k) s[k] += (double)a.g[k][(size_t)b * a.grad_stride + g];
        for (int k = 0; k < 3; ++k) a.stack[k][(size_t)ii * nz + jj] += s[k];
    }
}

void launch_grad_stack(const GradStackArgs& a, cudaStream_t s) {
    const int nz = a.Z - 2 * a.L, nx = a.X - 2 * a.L;
    k_grad_stack<<<dim3((nz + 255) / 256, nx), 256, 0, s>>>(a);
}

struct PackArgs {
    const float* f[12];
    const float* g[12];      // second addend of a sum, or null
    int nf, X, Z, pitch;
    float* out;
};
__global__ void k_pack(const PackArgs a) {
    const int i = blockIdx.y, k = blockIdx.z;
    for (int j = threadIdx.x + blockIdx.x * blockDim.x; j < a.Z; j += blockDim.x * gridDim.x) {
        const ptrdiff_t c = (ptrdiff_t)i * a.pitch + j;
        float v = a.f[k][c];
        if (a.g[k]) v += a.g[k][c];
        a.out[((size_t)k * a.X + i) * a.Z + j] = v;
    }
}

void launch_pack_fields(const float* const* f, int nf, int X, int Z, int pitch, float* out, cudaStream_t s,
                        const float* const* g) {
    PackArgs a;
    for (int k = 0; k < 12; ++k) { a.f[k] = k < nf ? f[k] : nullptr; a.g[k] = g && k < nf ? g[k] : nullptr; }
    a.nf = nf; a.X = X; a.Z = Z; a.pitch = pitch; a.out = out;
    dim3 grid((Z + 255) / 256, X, nf);
    k_pack<<<grid, 256, 0, s>>>(a);
}

}  // namespace ouc
