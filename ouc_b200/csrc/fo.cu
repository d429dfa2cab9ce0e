// First-order velocity-stress forward modeling (ouc_forward_fo): the scheme
// of the reference's stress (PS:487-560) and velocity (PS:390-486) kernels,
// which its main() never calls, as one fused sm_100a launch per time step.
//
// State: the P/S velocity parts (Vpx, Vpz, Vsx, Vsz) and eight split stresses
// (theta_x, theta_z, omega_x, omega_z and the four Q fields), each
// ping-ponged so that the halo reads of one step never meet its writes.  One
// tile per CTA (32 x 64, 16 x 64 or the small tiles of fd_small.cuh, chosen
// as for the second-order step), in three phases like that kernel:
//   1. U = P + S velocity over the tile and a 2N halo into shared memory;
//   2. the stress update over the tile and an N halo (four staggered velocity
//      derivatives, the split-field damping (1 - dt a/2)/(1 + dt a/2), the
//      source on theta), own cells written out, theta/omega/Q kept on chip;
//   3. the velocity update of the own cells from eight stress derivatives,
//      U = P + S, the receiver row recorded after the update.
// Derivatives use the rounding-exact helpers of fd_step.cuh; the damping
// factors and updates are the reference's expressions verbatim (double
// literals, so double arithmetic rounded once to float), powf(v, 2) as
// there, so that the compiler contracts them as it does the reference's.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "../../include/ouc.h"
#include "ctx.h"
#include "fd_small.cuh"
#include "fd_step.cuh"

namespace ouc {
namespace fo {

struct FoArgs {
    alignas(64) CUtensorMap map;     // U box of the launch's tile over the state block
    int vfield[4];                   // fields of vold[] in the block
    int* err;                        // device status word (bit 0: a copy wait ran out)
    int X, Z, pitch, tiles_z, t, nt;
    int sx, sz, rz;                  // padded source cell and receiver row
    float a[6];
    float dx, dz, dt, rdx, rdz;
    const float* vold[4];            // Vpx Vpz Vsx Vsz at the old half level
    float* vnew[4];
    const float* sold[8];            // theta_x theta_z omega_x omega_z Qxx Qxz Qzx Qzz
    float* snew[8];
    const float* vp2;                // powf(Vp, 2), powf(Vs, 2) (k_squares), damping x, z
    const float* vs2;
    const float* ax;
    const float* az;
    const float* wavelet;            // source samples, or null (back-propagation)
    float* rec_x;                    // gather row t (time-major), or null
    float* rec_z;
    const float* inj_x;              // records injected into U at the receiver
    const float* inj_z;              // row on [L, X-L) (row t), or null
    int L;
    unsigned copy_tx_extra;          // test hook, as StepArgs::copy_tx_extra
};

// split-field stress update, the reference's expression (PS:547-556)
__device__ __forceinline__ float stress_upd(float damp, float dt, float term, float old) {
    return (1.0 / (1.0 + 0.5 * dt * damp)) * (term + (1.0 - 0.5 * dt * damp) * old);
}
// velocity update, the reference's expression (PS:471-474)
__device__ __forceinline__ float vel_upd(float damp, float dt, float old, float sum) {
    return (1.0 / (1.0 + 0.5 * dt * damp)) * ((1 - 0.5 * dt * damp) * old + dt * sum);
}
// Both updates where the damping is 0 (the interior): the factors are exactly
// 1, and the double sum of two floats rounded to float is their float sum
// (53 >= 2*24 + 2: the double rounding is innocuous), so the result is one
// float addition -- bit-identical, without the double arithmetic.
__device__ __forceinline__ bool undamped4(const float4& ax, const float4& az) {
    return ax.x == 0.f && ax.y == 0.f && ax.z == 0.f && ax.w == 0.f && az.x == 0.f && az.y == 0.f && az.z == 0.f &&
           az.w == 0.f;
}

// powf(v, 2) of the model once per call, as the kernels evaluate it per cell
// (PS:547); guard cells hold 0.
__global__ void k_squares(const float* __restrict__ vp, const float* __restrict__ vs, float* vp2, float* vs2,
                          size_t n) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        vp2[k] = powf(vp[k], 2);
        vs2[k] = powf(vs[k], 2);
    }
}

// Wait for the tile's copies, form U = P + S (and at the receiver row the
// injected records).  False, with bit 0 of *p.err set, when they did not land.
template <class G>
__device__ __forceinline__ bool fo_u_box(const FoArgs& p, float* sm, int x0, int z0, uint64_t* bar) {
    constexpr int UC = G::UC, NT = G::NT;
    float* sUx = sm + G::oUx;
    float* sUz = sm + G::oUz;
    const float* stS = sm + G::oTh;
    const int tid = threadIdx.x;
    const int err_word = *(volatile const int*)p.err;
    const bool landed = mbar_wait(bar, 0u);
    if (!__syncthreads_and(landed && !(err_word & 1))) {
        if (tid == 0) {
            if (!landed) mbar_wait(bar, 0u);   // copies in flight land before the CTA ends
            atomicOr(p.err, 1);
        }
        __syncthreads();
        return false;
    }
    for (int idx = tid; idx < G::UR * (UC / 4); idx += NT) {
        st4(sUx + 4 * idx, add4(ld4(sUx + 4 * idx), ld4(stS + 4 * idx)));                // Vx = Vpx + Vsx
        st4(sUz + 4 * idx, add4(ld4(sUz + 4 * idx), ld4(stS + G::UR * UC + 4 * idx)));
    }
    const int ux_i0 = x0 - G::SHX - G::N, col = p.rz - (z0 - G::HU);
    if (p.inj_x && col >= 0 && col < UC) {
        // load_record (PS:1472-1481): U at the receiver row replaced by the
        // records before the stress update reads it
        __syncthreads();
        for (int r = tid; r < G::UR; r += NT) {
            const int gi = ux_i0 + r;
            if (gi >= p.L && gi < p.X - p.L) {
                sUx[r * UC + col] = p.inj_x[gi];
                sUz[r * UC + col] = p.inj_z[gi];
            }
        }
    }
    __syncthreads();
    return true;
}

// Whether the tile's S region meets the x or z damping layers (elsewhere the
// damping is exactly 0 and its profiles are not read).
template <class G>
__device__ __forceinline__ bool fo_damped(const FoArgs& p, int x0, int z0) {
    return x0 - G::SHX < p.L || x0 + G::TX + G::SHX - 1 >= p.X - p.L || z0 - G::HS < p.L ||
           z0 + G::TZ + G::HS - 1 >= p.Z - p.L;
}

// live[k]: cell k of the quad is updated by the reference
__device__ __forceinline__ unsigned fo_live(const FoArgs& p, int N, int gi, int gj) {
    unsigned m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) m |= (gi >= N && gi < p.X - N && gj + k >= N && gj + k < p.Z - N) ? (1u << k) : 0u;
    return m;
}
__device__ __forceinline__ float4 fo_mask(float4 v, unsigned live) {
    return make_float4(live & 1u ? v.x : 0.f, live & 2u ? v.y : 0.f, live & 4u ? v.z : 0.f, live & 8u ? v.w : 0.f);
}
// Products that an addition follows: scalar, since the compiler contracts a
// packed multiplication with the packed addition after it.
__device__ __forceinline__ float4 prod4(float4 a, float4 b) {
    return make_float4(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z), __fmul_rn(a.w, b.w));
}
// term + old, or the damped update, of one quad (dd: its damping, 0 where flat)
__device__ __forceinline__ float4 fo_stress4(bool flat, float4 dd, float dt, float4 term, float4 old) {
    if (flat) return add4(term, old);
    return make_float4(stress_upd(dd.x, dt, term.x, old.x), stress_upd(dd.y, dt, term.y, old.y),
                       stress_upd(dd.z, dt, term.z, old.z), stress_upd(dd.w, dt, term.w, old.w));
}
__device__ __forceinline__ float4 fo_vel4(bool flat, float4 dd, float dt, float4 old, float4 sum) {
    if (flat) return add4(old, prod4(sum, make_float4(dt, dt, dt, dt)));
    return make_float4(vel_upd(dd.x, dt, old.x, sum.x), vel_upd(dd.y, dt, old.y, sum.y), vel_upd(dd.z, dt, old.z, sum.z),
                       vel_upd(dd.w, dt, old.w, sum.w));
}
__device__ __forceinline__ float4 neg4(float4 v) { return make_float4(-v.x, -v.y, -v.z, -v.w); }

// Bound: latency and issue, as the second-order step.  1060 x 560, per step:
// 32 x 64 tiles with plain loads 52 us; 16 x 64 tiles, tensor copies and
// operands ahead of the derivatives 33 us (40 us before inside a time loop).
template <int N, class G>
__global__ void __launch_bounds__(kThreads, 2) k_fo(const __grid_constant__ FoArgs p) {
    constexpr int TX = G::TX, TZ = G::TZ, SHX = G::SHX, HS = G::HS, HU = G::HU, UC = G::UC, SC = G::SC;
    extern __shared__ __align__(128) float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    float* sUx = sm + G::oUx;
    float* sUz = sm + G::oUz;
    float* sTh = sm + G::oTh;
    float* sOm = sm + G::oOm;
    float* sQxz = sm + G::oQxz;
    float* sQzz = sm + G::oQzz;
    float* sQxx = sm + G::oQxx;
    float* sQzx = sm + G::oQzx;
    __shared__ uint64_t bar;
    const int tid = threadIdx.x;
    const int P = p.pitch;
    const int tz = blockIdx.x % p.tiles_z, tx = blockIdx.x / p.tiles_z;
    const int x0 = tx * TX, z0 = tz * TZ;
    pdl_launch_dependents();
    if (tid == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_map(&p.map);
        pdl_wait();
        issue_box<G>(&p.map, p.vfield, p.copy_tx_extra, sm, x0, z0, 0, &bar);
    }
    float a[N];
#pragma unroll
    for (int k = 0; k < N; ++k) a[k] = p.a[k];
    const Div dvx = make_div(p.dx, p.rdx), dvz = make_div(p.dz, p.rdz);
    const float dt = p.dt;
    const bool damped = fo_damped<G>(p, x0, z0);
    __syncthreads();   // the mbarrier is initialised
    pdl_wait();

    // ---- phase 1: U = P + S velocity over the tile and a 2N halo ----------
    if (!fo_u_box<G>(p, sm, x0, z0, &bar)) return;

    // ---- phase 2: stresses on the tile plus an N halo ----------------------
    if (tid < G::itemsA + G::itemsB) {
        int r0, c;
        const bool groupA = tid < G::itemsA;
        if (groupA) {
            r0 = -SHX + G::RS * (tid / (TZ / 4));
            c = 4 * (tid % (TZ / 4));
        } else {
            const int k = tid - G::itemsA;
            r0 = G::RS * (k / (2 * HS / 4));
            const int cc = k % (2 * HS / 4);
            c = cc < HS / 4 ? -HS + 4 * cc : TZ + 4 * (cc - HS / 4);
        }
        const float* ux0 = sUx + (r0 + SHX + N) * UC + (c + HU);
        const float* uz0 = sUz + (r0 + SHX + N) * UC + (c + HU);
        const bool ownc = c >= 0 && c < TZ;
#pragma unroll 1
        for (int q0 = 0; q0 < G::RS; q0 += 2) {
        float4 exx[2], ezx[2];
        dx4<N, 2, false>(ux0 + q0 * UC, UC, a, dvx, exx);   // dvxdx = D-x Vx
        dx4<N, 2, true>(uz0 + q0 * UC, UC, a, dvx, ezx);    // dvzdx = D+x Vz
#pragma unroll
        for (int qq = 0; qq < 2; ++qq) {
            const int q = q0 + qq, r = r0 + q, gi = x0 + r, gjb = z0 + c;
            const int g = gi * P + gjb;
            // operands first: their latency runs under the z derivatives
            const float4 vp2v = ldg4(p.vp2 + g), vs2v = ldg4(p.vs2 + g);
            float4 so[8];
#pragma unroll
            for (int f = 0; f < 8; ++f) so[f] = ldg4(p.sold[f] + g);
            float4 axv = zero4(), azv = zero4();
            if (damped) { axv = ldg4(p.ax + g); azv = ldg4(p.az + g); }
            const float4 exz = dz4<N, true>(ux0 + q * UC, a, dvz);    // dvxdz = D+z Vx
            const float4 ezz = dz4<N, false>(uz0 + q * UC, a, dvz);   // dvzdz = D-z Vz
            const bool flat = !damped || undamped4(axv, azv);
            // dt Vp^2 d, dt Vs^2 d and -dt Vs^2 d, each rounded as the reference's float products
            const float4 cp = mul4s(vp2v, dt), cs = mul4s(vs2v, dt), cm = neg4(cs);
            const unsigned live = fo_live(p, N, gi, gjb);
            float4 sn[8];
            sn[0] = fo_stress4(flat, axv, dt, prod4(cp, exx[qq]), so[0]);   // theta_x
            sn[1] = fo_stress4(flat, azv, dt, prod4(cp, ezz), so[1]);       // theta_z
            sn[2] = fo_stress4(flat, axv, dt, prod4(cm, ezx[qq]), so[2]);   // omega_x
            sn[3] = fo_stress4(flat, azv, dt, prod4(cs, exz), so[3]);       // omega_z
            sn[4] = fo_stress4(flat, axv, dt, prod4(cs, exx[qq]), so[4]);   // Qxx (duxdx)
            sn[5] = fo_stress4(flat, azv, dt, prod4(cs, exz), so[5]);       // Qxz (duxdz)
            sn[6] = fo_stress4(flat, axv, dt, prod4(cs, ezx[qq]), so[6]);   // Qzx (duzdx)
            sn[7] = fo_stress4(flat, azv, dt, prod4(cs, ezz), so[7]);       // Qzz (duzdz)
            if (live != 0xfu) {
#pragma unroll
                for (int f = 0; f < 8; ++f) sn[f] = fo_mask(sn[f], live);   // the reference never updates these cells
            }
            float4 th = add4(sn[0], sn[1]);
            const float4 om = add4(sn[2], sn[3]);
            // theta_x + theta_z + s with s = 0 off the source (PS:557): the
            // second addition turns -0 into +0
            float4 sv = zero4();
            if (p.wavelet && gi == p.sx && p.sz >= gjb && p.sz < gjb + 4 && (live >> (p.sz - gjb) & 1u))
                set_comp(sv, p.sz - gjb, p.wavelet[p.t]);
            th = add4(th, sv);
            if (ownc && r >= 0 && r < TX) {
#pragma unroll
                for (int f = 0; f < 8; ++f) stg4(p.snew[f] + g, sn[f]);
            }
            const int sr = r + SHX, scol = c + HS;
            st4(sTh + sr * SC + scol, th);
            st4(sOm + sr * SC + scol, om);
            if (groupA) {
                st4(sQxz + sr * TZ + c, sn[5]);
                st4(sQzz + sr * TZ + c, sn[7]);
            }
            if (r >= 0 && r < TX) {
                st4(sQxx + r * SC + scol, sn[4]);
                st4(sQzx + r * SC + scol, sn[6]);
            }
        }
        }
    }
    __syncthreads();

    // ---- phase 3: velocities of the own cells --------------------------------
    {
        const int rr = G::RU * (tid / (TZ / 4));
        const int c = 4 * (tid % (TZ / 4));
        const int scol = c + HS;
#pragma unroll 1
        for (int q = 0; q < G::RU; ++q) {
            const int r = rr + q, gi = x0 + r;
            const int g = gi * P + (z0 + c);
            const float4 opx = ldg4(p.vold[0] + g), opz = ldg4(p.vold[1] + g);
            const float4 osx = ldg4(p.vold[2] + g), osz = ldg4(p.vold[3] + g);
            float4 axv = zero4(), azv = zero4();
            if (damped) { axv = ldg4(p.ax + g); azv = ldg4(p.az + g); }
            float4 txv[1], wxv[1], dB[1], dE[1];
            dx4<N, 1, true>(sTh + (r + SHX) * SC + scol, SC, a, dvx, txv);    // dthetadx = D+x theta
            dx4<N, 1, false>(sOm + (r + SHX) * SC + scol, SC, a, dvx, wxv);   // domegadx = D-x omega
            dx4<N, 1, false>(sQxz + (r + SHX) * TZ + c, TZ, a, dvx, dB);      // dux_zdx = D-x Qxz
            dx4<N, 1, true>(sQzz + (r + SHX) * TZ + c, TZ, a, dvx, dE);       // duz_zdx = D+x Qzz
            const float4 tzv = dz4<N, true>(sTh + (r + SHX) * SC + scol, a, dvz);   // dthetadz
            const float4 wzv = dz4<N, false>(sOm + (r + SHX) * SC + scol, a, dvz);  // domegadz
            const float4 dA = dz4<N, true>(sQxx + r * SC + scol, a, dvz);           // dux_xdz = D+z Qxx
            const float4 dC = dz4<N, false>(sQzx + r * SC + scol, a, dvz);          // duz_xdz = D-z Qzx
            const bool flat = !damped || undamped4(axv, azv);
            const unsigned live = fo_live(p, N, gi, z0 + c);
            float4 npx = fo_vel4(flat, axv, dt, opx, sub4(add4(txv[0], dC), dE[0]));
            float4 npz = fo_vel4(flat, azv, dt, opz, sub4(add4(tzv, dB[0]), dA));
            float4 nsx = fo_vel4(flat, axv, dt, osx, sub4(add4(wzv, dC), dE[0]));
            float4 nsz = fo_vel4(flat, azv, dt, osz, sub4(add4(neg4(wxv[0]), dB[0]), dA));
            if (live != 0xfu) { npx = fo_mask(npx, live); npz = fo_mask(npz, live); nsx = fo_mask(nsx, live); nsz = fo_mask(nsz, live); }
            stg4(p.vnew[0] + g, npx); stg4(p.vnew[1] + g, npz);
            stg4(p.vnew[2] + g, nsx); stg4(p.vnew[3] + g, nsz);
            if (p.rec_x && p.rz >= z0 + c && p.rz < z0 + c + 4 && gi < p.X) {
                const int k = p.rz - z0 - c;   // post-update value at the receiver row
                p.rec_x[gi] = comp(npx, k) + comp(nsx, k);
                p.rec_z[gi] = comp(npz, k) + comp(nsz, k);
            }
        }
    }
}

// The same step on small tiles, its work cut across threads as in
// fd_small.cuh: the x-damped stresses (theta_x, omega_x, Qxx, Qzx) need only
// the two x derivatives and the z-damped ones only the two z derivatives, so
// an item's x and z threads meet only in theta and omega; four threads per U
// item take two stress derivatives each and finish one velocity component.
template <int N, int TXr, int CTAS>
__global__ void __launch_bounds__(SmallGeo<N, TXr>::NT, CTAS) k_fo_small(const __grid_constant__ FoArgs p) {
    using G = SmallGeo<N, TXr>;
    constexpr int TX = G::TX, TZ = G::TZ, SHX = G::SHX, HS = G::HS, HU = G::HU, UC = G::UC, SC = G::SC, NT = G::NT;
    extern __shared__ __align__(128) float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    float* sUx = sm + G::oUx;
    float* sUz = sm + G::oUz;
    float* sTh = sm + G::oTh;
    float* sOm = sm + G::oOm;
    float* sQxz = sm + G::oQxz;
    float* sQzz = sm + G::oQzz;
    float* sQxx = sm + G::oQxx;
    float* sQzx = sm + G::oQzx;
    float4* const sE = reinterpret_cast<float4*>(sm + G::oE);       // [2][itemsS]: theta_z, omega_z
    float4* const sD = reinterpret_cast<float4*>(sm);               // [8][itemsU]: derivatives
    float4* const sN = reinterpret_cast<float4*>(sm + G::oNew);     // [4][itemsU]: new velocities
    __shared__ uint64_t bar;
    const int tid = threadIdx.x;
    const int P = p.pitch;
    const int tz = blockIdx.x % p.tiles_z, tx = blockIdx.x / p.tiles_z;
    const int x0 = tx * TX, z0 = tz * TZ;
    pdl_launch_dependents();
    if (tid == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_map(&p.map);
    }
    float a[N];
#pragma unroll
    for (int k = 0; k < N; ++k) a[k] = p.a[k];
    const Div dvx = make_div(p.dx, p.rdx), dvz = make_div(p.dz, p.rdz);
    const float dt = p.dt;
    const bool damped = fo_damped<G>(p, x0, z0);
    const bool xt = tid < NT / 2;   // x thread of an S item, or z thread
    const int item = xt ? tid : tid - NT / 2;
    const bool has_s = item < G::itemsS;
    int r = 0, c = 0;
    if (has_s) {
        if (item < G::itemsA) {
            r = -SHX + item / (TZ / 4);
            c = 4 * (item % (TZ / 4));
        } else {
            const int k = item - G::itemsA, cc = k % (2 * HS / 4);
            r = k / (2 * HS / 4);
            c = cc < HS / 4 ? -HS + 4 * cc : TZ + 4 * (cc - HS / 4);
        }
    }
    const int gs = (x0 + r) * P + (z0 + c);
    const int task = tid / G::itemsU, ui = tid % G::itemsU;   // theta omega | Qxz Qzz along x, theta omega | Qxx Qzx along z
    const bool has_u = task < 4;
    const int ur = ui / (TZ / 4), uc = 4 * (ui % (TZ / 4));
    const int gi = x0 + ur, gu = gi * P + (z0 + uc);
    float4 vp2v = zero4(), vs2v = zero4(), axs = zero4(), azs = zero4(), so[4];
    if (has_s) {
        vp2v = ldg4(p.vp2 + gs);
        vs2v = ldg4(p.vs2 + gs);
        if (damped) { axs = ldg4(p.ax + gs); azs = ldg4(p.az + gs); }
    }
    __syncthreads();   // the mbarrier is initialised
    pdl_wait();
    if (tid == 0) issue_box<G>(&p.map, p.vfield, p.copy_tx_extra, sm, x0, z0, 0, &bar);
    if (has_s) {
        // theta_x omega_x Qxx Qzx | theta_z omega_z Qxz Qzz
#pragma unroll
        for (int f = 0; f < 4; ++f) so[f] = ldg4((xt ? p.sold[2 * f] : p.sold[2 * f + 1]) + gs);
    }
    if (!fo_u_box<G>(p, sm, x0, z0, &bar)) return;

    // ---- stresses ------------------------------------------------------------
    const float* ux0 = sUx + (r + SHX + N) * UC + (c + HU);
    const float* uz0 = sUz + (r + SHX + N) * UC + (c + HU);
    const int sr = r + SHX, scol = c + HS;
    float4 v0 = zero4(), v1 = zero4();   // theta_x, omega_x of an x thread
    unsigned slive = 0;
    if (has_s) {
        const bool flat = !damped || undamped4(axs, azs);
        const float4 cp = mul4s(vp2v, dt), cs = mul4s(vs2v, dt);
        slive = fo_live(p, N, x0 + r, z0 + c);
        float4 d1, d2;   // exx, ezx | ezz, exz
        if (xt) {
            float4 e1[1], e2[1];
            dx4<N, 1, false>(ux0, UC, a, dvx, e1);   // dvxdx = D-x Vx
            dx4<N, 1, true>(uz0, UC, a, dvx, e2);    // dvzdx = D+x Vz
            d1 = e1[0];
            d2 = e2[0];
        } else {
            d2 = dz4<N, true>(ux0, a, dvz);    // dvxdz = D+z Vx
            d1 = dz4<N, false>(uz0, a, dvz);   // dvzdz = D-z Vz
        }
        const float4 dd = xt ? axs : azs;
        v0 = fo_stress4(flat, dd, dt, prod4(cp, d1), so[0]);                     // theta_x | theta_z
        v1 = fo_stress4(flat, dd, dt, prod4(xt ? neg4(cs) : cs, d2), so[1]);     // omega_x | omega_z
        float4 v2 = fo_stress4(flat, dd, dt, prod4(cs, xt ? d1 : d2), so[2]);    // Qxx | Qxz
        float4 v3 = fo_stress4(flat, dd, dt, prod4(cs, xt ? d2 : d1), so[3]);    // Qzx | Qzz
        if (slive != 0xfu) { v0 = fo_mask(v0, slive); v1 = fo_mask(v1, slive); v2 = fo_mask(v2, slive); v3 = fo_mask(v3, slive); }
        if (r >= 0 && r < TX && c >= 0 && c < TZ) {
            const float4 v[4] = {v0, v1, v2, v3};
#pragma unroll
            for (int f = 0; f < 4; ++f) stg4((xt ? p.snew[2 * f] : p.snew[2 * f + 1]) + gs, v[f]);
        }
        if (xt) {
            if (r >= 0 && r < TX) {
                st4(sQxx + r * SC + scol, v2);
                st4(sQzx + r * SC + scol, v3);
            }
        } else {
            sE[item] = v0;
            sE[G::itemsS + item] = v1;
            if (item < G::itemsA) {
                st4(sQxz + sr * TZ + c, v2);
                st4(sQzz + sr * TZ + c, v3);
            }
        }
    }
    float4 old = zero4(), dd = zero4(), ax2 = zero4(), az2 = zero4();   // U operands
    if (has_u) {
        old = ldg4((task == 0 ? p.vold[0] : task == 1 ? p.vold[1] : task == 2 ? p.vold[2] : p.vold[3]) + gu);
        if (damped) { ax2 = ldg4(p.ax + gu); az2 = ldg4(p.az + gu); }
    }
    __syncthreads();
    if (has_s && xt) {
        float4 sv = zero4();
        const int k = p.sz - z0 - c;
        if (p.wavelet && x0 + r == p.sx && k >= 0 && k < 4 && (slive >> k & 1u)) set_comp(sv, k, p.wavelet[p.t]);
        st4(sTh + sr * SC + scol, add4(add4(v0, sE[item]), sv));   // PS:557
        st4(sOm + sr * SC + scol, add4(v1, sE[G::itemsS + item]));
    }
    __syncthreads();

    // ---- velocities ------------------------------------------------------------
    if (has_u) {
        float4 d1, d2;
        if (task < 2) {
            float4 e1[1], e2[1];
            if (task == 0) {
                dx4<N, 1, true>(sTh + (ur + SHX) * SC + (uc + HS), SC, a, dvx, e1);    // dthetadx
                dx4<N, 1, false>(sOm + (ur + SHX) * SC + (uc + HS), SC, a, dvx, e2);   // domegadx
            } else {
                dx4<N, 1, false>(sQxz + (ur + SHX) * TZ + uc, TZ, a, dvx, e1);         // dux_zdx = B
                dx4<N, 1, true>(sQzz + (ur + SHX) * TZ + uc, TZ, a, dvx, e2);          // duz_zdx = E
            }
            d1 = e1[0];
            d2 = e2[0];
        } else {
            const float* f1 = task == 2 ? sTh + (ur + SHX) * SC + (uc + HS) : sQxx + ur * SC + (uc + HS);
            const float* f2 = task == 2 ? sOm + (ur + SHX) * SC + (uc + HS) : sQzx + ur * SC + (uc + HS);
            d1 = dz4<N, true>(f1, a, dvz);    // dthetadz | dux_xdz = A
            d2 = dz4<N, false>(f2, a, dvz);   // domegadz | duz_xdz = C
        }
        sD[(2 * task) * G::itemsU + ui] = d1;
        sD[(2 * task + 1) * G::itemsU + ui] = d2;
    }
    __syncthreads();
    if (has_u) {
        auto D = [&](int k) { return sD[k * G::itemsU + ui]; };   // tx wx B E tz wz A C
        const bool xc = task == 0 || task == 2;
        float4 e0 = D(task == 0 ? 0 : task == 1 ? 4 : task == 2 ? 5 : 1);
        if (task == 3) e0 = neg4(e0);
        const float4 sum = sub4(add4(e0, xc ? D(7) : D(2)), xc ? D(3) : D(6));
        const bool flat = !damped || undamped4(ax2, az2);
        dd = xc ? ax2 : az2;
        float4 nv = fo_vel4(flat, dd, dt, old, sum);
        const unsigned live = fo_live(p, N, gi, z0 + uc);
        if (live != 0xfu) nv = fo_mask(nv, live);
        stg4((task == 0 ? p.vnew[0] : task == 1 ? p.vnew[1] : task == 2 ? p.vnew[2] : p.vnew[3]) + gu, nv);
        sN[task * G::itemsU + ui] = nv;
    }
    if (p.rec_x && p.rz >= z0 && p.rz < z0 + TZ) {
        __syncthreads();
        if (tid < TX && x0 + tid < p.X) {
            const float* n0 = sm + G::oNew;
            const int o = tid * TZ + (p.rz - z0);
            p.rec_x[x0 + tid] = n0[o] + n0[2 * TX * TZ + o];   // post-update value at the receiver row
            p.rec_z[x0 + tid] = n0[TX * TZ + o] + n0[3 * TX * TZ + o];
        }
    }
}

// The shared-memory opt-in is a per-device attribute: set on the current
// device before every loop (fo_run), not once per process.
template <int N>
cudaError_t configure() {
    auto set = [](auto kernel, int bytes) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    cudaError_t e = set(k_fo<N, TileGeo<N>>, TileGeo<N>::bytes);
    if (e == cudaSuccess) e = set(k_fo<N, MidGeo<N>>, MidGeo<N>::bytes);
    if (e == cudaSuccess) e = set(k_fo_small<N, 16, 1>, SmallGeo<N, 16>::bytes);
    if (e == cudaSuccess) e = set(k_fo_small<N, 16, 2>, SmallGeo<N, 16>::bytes);
    if (e == cudaSuccess) e = set(k_fo_small<N, 24, 1>, SmallGeo<N, 24>::bytes);
    return e;
}

// One step on the tiles of `tier` (pick_tier: the same shapes pay at the same
// sizes as for the second-order step).
template <int N>
void launch(FoArgs& a, Tier tier, cudaStream_t s) {
    const int tx = tier == kLarge ? 32 : tier == kSmall24 ? 24 : 16, tz = tier == kLarge || tier == kMid ? 64 : 32;
    a.tiles_z = (a.Z + tz - 1) / tz;
    const dim3 grid((a.X + tx - 1) / tx * a.tiles_z);
    if (tier == kLarge) launch_pdl(k_fo<N, TileGeo<N>>, grid, kThreads, TileGeo<N>::bytes, s, false, a);
    else if (tier == kMid) launch_pdl(k_fo<N, MidGeo<N>>, grid, kThreads, MidGeo<N>::bytes, s, false, a);
    else if (tier == kSmall24) launch_pdl(k_fo_small<N, 24, 1>, grid, SmallGeo<N, 24>::NT, SmallGeo<N, 24>::bytes, s, false, a);
    else if (tier == kSmall16) launch_pdl(k_fo_small<N, 16, 1>, grid, SmallGeo<N, 16>::NT, SmallGeo<N, 16>::bytes, s, false, a);
    else launch_pdl(k_fo_small<N, 16, 2>, grid, SmallGeo<N, 16>::NT, SmallGeo<N, 16>::bytes, s, false, a);
}

// Five-digit weights of the reference's first-order kernels (PS:405,
// PS:501): double literals converted to float, as a float array initialised
// from them; other half-orders use the context's weights.
constexpr float kFoWeights6[6] = {(float)1.2213e+0, (float)-9.6931e-2, (float)1.7448e-2,
                                  (float)-2.9673e-3, (float)3.5901e-4, (float)-2.1848e-5};

}  // namespace fo
}  // namespace ouc

using namespace ouc;
using namespace ouc::host;

namespace {

int fo_check(ouc_ctx* ctx, const ouc_shot* shot) {
    if (!ctx) return OUC_EINVAL;
    int rc = check_shot(ctx, shot);
    if (rc) return rc;
    if (shot->src_type != OUC_SRC_THETA) return fail(ctx, OUC_EINVAL, "the first-order scheme has the theta source only");
    if (ctx->cfg.density) return fail(ctx, OUC_EINVAL, "the first-order scheme is density-normalised");
    return OUC_OK;
}

// The first-order time loop on the source side's 24 fields (velocities
// now[4] / past[4], stresses fo[4] + o[0..3] / fn[4] + o[4..7], ping-ponged
// by step).  Forward: t = 0 .. nt-1 with the source and the record into the
// context's gathers.  Backward: t = nt-1 .. 0 injecting the context's
// gathers (row t) at the receiver row.  fields (host, 16*X*Z, or null): the
// final state; `theta_src` is the source sample theta carries at the source
// cell in the last step (0 backward).
int fo_run(ouc_ctx* ctx, const ouc_shot* shot, bool backward, float theta_src, float* fields) {
    int rc;
    const size_t C = (size_t)ctx->X * ctx->Z;
    if (!ctx->fo_sq) {
        if (cudaMalloc(&ctx->fo_sq, 2 * ctx->fstride * sizeof(float)) != cudaSuccess) {
            cudaGetLastError();
            ctx->fo_sq = nullptr;
            return fail(ctx, OUC_ENOMEM, "cannot allocate the first-order model squares");
        }
        ctx->bytes += 2 * ctx->fstride * sizeof(float);
    }
    // raw field bases (guards included) of Vp, Vs (model fields 6, 7) and the squares
    fo::k_squares<<<4 * 148, 256, 0, ctx->stream>>>(ctx->model + 6 * ctx->fstride, ctx->model + 7 * ctx->fstride,
                                                    ctx->fo_sq, ctx->fo_sq + ctx->fstride, ctx->fstride);
    ctx->timing.kernel_launches += 1;
    const cudaError_t ce = ctx->N == 2 ? fo::configure<2>() : ctx->N == 5 ? fo::configure<5>() : fo::configure<6>();
    if (ce != cudaSuccess) return cuda_fail(ctx, ce, "first-order kernel configuration");
    if ((rc = zero_side(ctx, 1, 0, false))) return rc;
    const Side& s = ctx->src0;
    const float* vA[4] = {s.now[0], s.now[1], s.now[2], s.now[3]};
    float* vB[4] = {s.past[0], s.past[1], s.past[2], s.past[3]};
    float* sA[8] = {s.fo[0], s.fo[1], s.fo[2], s.fo[3], s.o[0], s.o[1], s.o[2], s.o[3]};
    float* sB[8] = {s.fn[0], s.fn[1], s.fn[2], s.fn[3], s.o[4], s.o[5], s.o[6], s.o[7]};
    fo::FoArgs a;
    memset(&a, 0, sizeof(a));
    a.X = ctx->X; a.Z = ctx->Z; a.pitch = ctx->pitch; a.tiles_z = ctx->tiles_z; a.nt = ctx->nt; a.L = ctx->L;
    a.sx = shot->sx + ctx->L; a.sz = shot->sz + ctx->L; a.rz = shot->rz + ctx->L;
    for (int k = 0; k < 6; ++k) a.a[k] = ctx->N == 6 ? fo::kFoWeights6[k] : ctx->a[k];
    a.dx = ctx->cfg.dx; a.dz = ctx->cfg.dz; a.dt = ctx->cfg.dt;
    a.rdx = 1.0f / ctx->cfg.dx; a.rdz = 1.0f / ctx->cfg.dz;
    a.vp2 = ctx->field(ctx->fo_sq, 0); a.vs2 = ctx->field(ctx->fo_sq, 1); a.ax = ctx->ax; a.az = ctx->az;
    a.wavelet = backward ? nullptr : ctx->d_wavelet;
    a.err = ctx->d_status;
    const StepArgs b = base_args(ctx);
    a.copy_tx_extra = b.copy_tx_extra;
    const Tier tier = b.tier != kAuto ? (Tier)b.tier : pick_tier(ctx->N, nullptr, &b, kFwd, 1);
    a.map = tier == kLarge ? b.box_map : tier == kMid ? b.mid_map : b.small_map[tier == kSmall24 ? 1 : 0];
    auto field_of = [&](const float* f) { return (int)((f - ctx->field(ctx->state, 0)) / (ptrdiff_t)ctx->fstride); };
    float* gx = ctx->gather(0, 0);
    float* gz = ctx->gather(0, 1);
    cudaEventRecord(ctx->ev[1], ctx->stream);
    for (int n = 0; n < ctx->nt; ++n) {
        const int t = backward ? ctx->nt - 1 - n : n;
        const bool even = (n & 1) == 0;
        for (int k = 0; k < 4; ++k) { a.vold[k] = even ? vA[k] : vB[k]; a.vnew[k] = even ? vB[k] : (float*)vA[k]; a.vfield[k] = field_of(a.vold[k]); }
        for (int k = 0; k < 8; ++k) { a.sold[k] = even ? sA[k] : sB[k]; a.snew[k] = even ? sB[k] : sA[k]; }
        a.t = t;
        if (backward) {
            a.inj_x = gx + (size_t)t * ctx->X;
            a.inj_z = gz + (size_t)t * ctx->X;
        } else {
            a.rec_x = gx + (size_t)t * ctx->X;
            a.rec_z = gz + (size_t)t * ctx->X;
        }
        if (ctx->N == 2) fo::launch<2>(a, tier, ctx->stream);
        else if (ctx->N == 5) fo::launch<5>(a, tier, ctx->stream);
        else fo::launch<6>(a, tier, ctx->stream);
        ctx->timing.kernel_launches += 1;
    }
    cudaEventRecord(ctx->ev[2], ctx->stream);
    const cudaError_t le = cudaGetLastError();   // launch-configuration errors are not reported by the sync
    if (le != cudaSuccess) return cuda_fail(ctx, le, "first-order step launch");
    if (fields) {
        const bool touched = touch_pages({{fields, nullptr, 16 * C * 4}});   // while the time loop runs
        // the newest level: written by the last step
        const bool last_even = ((ctx->nt - 1) & 1) == 0;
        const float* v[4];
        const float* st[8];
        for (int k = 0; k < 4; ++k) v[k] = last_even ? vB[k] : vA[k];
        for (int k = 0; k < 8; ++k) st[k] = last_even ? sB[k] : sA[k];
        // 16 host fields: Vx Vz Vpx Vpz Vsx Vsz theta omega Qzx Qzz Qxx Qxz theta_x theta_z omega_x omega_z
        const float* order[12] = {v[0], v[1], v[2], v[3], st[6], st[7], st[4], st[5], st[0], st[1], st[2], st[3]};
        const int dst[12] = {2, 3, 4, 5, 8, 9, 10, 11, 12, 13, 14, 15};
        for (int k = 0; k < 12; k += 4) {
            launch_pack_fields(order + k, 4, ctx->X, ctx->Z, ctx->pitch, ctx->staging, ctx->stream);
            if ((rc = to_host(ctx, fields + (size_t)dst[k] * C, ctx->staging, 4 * C * 4, touched))) return rc;   // 4 fields in a row
        }
        // totals as the kernels form them: U = P + S, theta = theta_x +
        // theta_z + s, omega = omega_x + omega_z (the source term below)
        const float* f[4] = {v[0], v[1], st[0], st[2]};
        const float* g[4] = {v[2], v[3], st[1], st[3]};
        launch_pack_fields(f, 4, ctx->X, ctx->Z, ctx->pitch, ctx->staging, ctx->stream, g);
        if ((rc = to_host(ctx, fields, ctx->staging, 2 * C * 4, touched))) return rc;
        if ((rc = to_host(ctx, fields + 6 * C, ctx->staging + 2 * C, 2 * C * 4, touched))) return rc;
    }
    const cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "first-order time loop");
    if ((rc = check_status(ctx))) return rc;
    if (fields) fields[6 * C + (size_t)(shot->sx + ctx->L) * ctx->Z + (shot->sz + ctx->L)] += theta_src;
    (backward ? ctx->timing.backward_ms : ctx->timing.forward_ms) = elapsed(ctx->ev[1], ctx->ev[2]);
    return OUC_OK;
}

}  // namespace

extern "C" {

int ouc_forward_fo(ouc_ctx* ctx, const ouc_shot* shot, const float* wavelet, float* gather_vx, float* gather_vz,
                   float* fields) {
    int rc = fo_check(ctx, shot);
    if (rc) return rc;
    if (!wavelet) return fail(ctx, OUC_EINVAL, "wavelet is NULL");
    cudaSetDevice(ctx->device);
    ctx->step_phase = ouc_ctx::kIdle;
    ctx->timing = ouc_timing{};
    if (cudaMemcpyAsync(ctx->d_wavelet, wavelet, (size_t)ctx->nt * 4, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess)
        return fail(ctx, OUC_ECUDA, "wavelet upload failed");
    if ((rc = fo_run(ctx, shot, false, wavelet[ctx->nt - 1], fields))) return rc;
    if (gather_vx && (rc = gather_out(ctx, ctx->gather(0, 0), gather_vx, true))) return rc;
    if (gather_vz && (rc = gather_out(ctx, ctx->gather(0, 1), gather_vz, true))) return rc;
    const cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "gather download");
    return OUC_OK;
}

int ouc_backward_fo(ouc_ctx* ctx, const ouc_shot* shot, const float* rec_vx, const float* rec_vz, float* fields) {
    int rc = fo_check(ctx, shot);
    if (rc) return rc;
    if (!rec_vx || !rec_vz) return fail(ctx, OUC_EINVAL, "records are NULL");
    cudaSetDevice(ctx->device);
    ctx->step_phase = ouc_ctx::kIdle;
    ctx->timing = ouc_timing{};
    if ((rc = records_in(ctx, {{rec_vx, ctx->gather(0, 0), ctx->X}, {rec_vz, ctx->gather(0, 1), ctx->X}}, true))) return rc;
    return fo_run(ctx, shot, true, 0.0f, fields);
}

}  // extern "C"
