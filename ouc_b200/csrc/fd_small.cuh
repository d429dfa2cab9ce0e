// The fused time step of fd_step.cuh on small tiles, for launches that do
// not fill the GPU with 32 x 64 tiles (one shot on a small or mid-size grid).
//
// Such a launch lasts as long as one tile: at 256 x 256 a 32 x 64 tile grid is
// 50 CTAs on 148 SMs, and each takes 30,000-46,000 cycles because a thread
// works through eight derivatives of two rows and the operand latencies of
// both stages one after the other.  Here a tile is 16 x 32 cells and its work
// is cut across 576 threads so that every dependent chain is short:
//   * S-stage: one thread takes the two x derivatives of a (row, four columns)
//     item and another the two z derivatives; the z results (and their damping
//     memories) pass through shared memory to the x thread, which forms theta
//     and omega;
//   * U-stage: the eight derivatives of an item go to four threads, two each
//     (with their damping memories), and after one exchange each of those
//     threads finishes one component (Px, Pz, Sx, Sz), so that its leapfrog
//     operands are two loads issued long before.
// Every operand load is issued ahead of the wait it would otherwise add to:
// the model before the tile's tensor copies land, the damping memories and
// the leapfrog levels before the S-stage; what is constant through a time
// loop before the previous launch has even finished (pdl_wait).  Arithmetic,
// rounding order and outputs are those of step_tile, bit for bit.
//
// Bound: latency (a 160 x 120 step is 40 CTAs).  After pdl_wait a CTA takes
// about 2,200 cycles until its copies have landed, 500 for the sum, 2,300 and
// 600 in the two parts of the S-stage, 1,800 and 800 in those of the U-stage;
// the next launch's wait returns 1.4 us after the last CTA's stores.  Per
// forward step, 32 x 64 tiles -> these: 160 x 120 grid 20.0 -> 6.7 us,
// 296 x 296 23.9 -> 8.3 us (24-row tiles), 397 x 301 24.4 -> 11.5 us.
#pragma once
#include "fd_step.cuh"

namespace ouc {

template <int N_, int TX_>
struct SmallGeo {
    static constexpr int N = N_;
    static constexpr bool small = true, mid = false;
    static constexpr int TX = TX_, TZ = 32;        // tile rows (x) and columns (z)
    static constexpr int NT = TX == 16 ? 576 : 768;   // threads
    static constexpr int SHX = N;                  // S-stage row halo
    static constexpr int HS = (N + 3) & ~3;        // S-stage column halo (float4 aligned)
    static constexpr int HU = (HS + N + 3) & ~3;   // U column halo
    static constexpr int UR = TX + 2 * (SHX + N);  // U rows held
    static constexpr int UC = TZ + 2 * HU;         // U columns held
    static constexpr int SR = TX + 2 * SHX;        // rows of theta/omega/Qxz/Qzz
    static constexpr int SC = TZ + 2 * HS;         // columns of theta/omega/Qxx/Qzx
    static constexpr int itemsA = SR * (TZ / 4);         // S items over all rows, own columns
    static constexpr int itemsB = TX * (2 * HS / 4);     // S items over own rows, halo columns
    static constexpr int itemsS = itemsA + itemsB;
    static constexpr int itemsU = TX * (TZ / 4);
    // U box, then the S-stage exchange; both free in the U-stage, whose
    // exchange (16 float4 per item) overlays them
    static constexpr int oUx = 0;
    static constexpr int oUz = UR * UC;
    static constexpr int oE = 2 * UR * UC;
    static constexpr int endE = oE + 16 * itemsS;
    static constexpr int oTh = endE > 64 * itemsU ? endE : 64 * itemsU;
    static constexpr int oOm = oTh + SR * SC;
    static constexpr int oQxz = oOm + SR * SC;     // SR x TZ (x-derivative only)
    static constexpr int oQzz = oQxz + SR * TZ;
    static constexpr int oQxx = oQzz + SR * TZ;    // TX x SC (z-derivative only)
    static constexpr int oQzx = oQxx + TX * SC;
    static constexpr int endS = oQzx + TX * SC;
    static constexpr int oNew = endS > oTh + 2 * UR * UC ? endS : oTh + 2 * UR * UC;   // new level, 4 components
    static constexpr int floats = oNew + 16 * itemsU;
    static constexpr int bytes = floats * 4;
    static_assert(2 * itemsS <= NT && NT / 2 % 32 == 0, "an x and a z thread per S item, in different warps");
    static_assert(4 * itemsU <= NT && itemsU % 32 == 0, "four threads per U item, in different warps");
    static_assert(oTh % 32 == 0, "tensor-copy destinations are 128-byte aligned");
};

template <class G, int MODE, int CTAS>
__device__ __forceinline__ bool small_tile(const StepArgs& p, const Geo& gm, const ShotView& sv, float* sm, int x0, int z0,
                                           const TileFlags& f, uint64_t* bar) {
    constexpr int N = G::N, NT = G::NT;
    constexpr int TX = G::TX, TZ = G::TZ, SHX = G::SHX, HS = G::HS, HU = G::HU, UC = G::UC, SC = G::SC;
    const int tid = threadIdx.x;
    const int P = p.pitch;
    const size_t R = gm.ring.R;
    float* sUx = sm + G::oUx;
    float* sUz = sm + G::oUz;
    float* sTh = sm + G::oTh;
    float* sOm = sm + G::oOm;
    float* sQxz = sm + G::oQxz;
    float* sQzz = sm + G::oQzz;
    float* sQxx = sm + G::oQxx;
    float* sQzx = sm + G::oQzx;
    float4* const sE = reinterpret_cast<float4*>(sm + G::oE);       // [4][itemsS]: ezz, exz, fzz, fxz
    float4* const sD = reinterpret_cast<float4*>(sm);               // [16][itemsU]: derivatives, memories
    float4* const sN = reinterpret_cast<float4*>(sm + G::oNew);     // [4][itemsU]
    float a[N];
#pragma unroll
    for (int k = 0; k < N; ++k) a[k] = p.a[k];
    const Div dvx = make_div(p.dx, p.rdx), dvz = make_div(p.dz, p.rdz);
    const size_t off = sv.off;
    const float dt = p.dt;
    const int ux_i0 = x0 - SHX - N, ux_j0 = z0 - HU;   // global origin of the U box

    // S item of this thread: x threads in the lower half of the CTA, z threads in the upper
    const bool sx_thread = tid < NT / 2;
    const int item = sx_thread ? tid : tid - NT / 2;
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
    const bool s_own = has_s && r >= 0 && r < TX && c >= 0 && c < TZ;
    const int gs = (x0 + r) * P + (z0 + c);
    // U item: task 0 (theta, omega along x), 1 (Qxz, Qzz along x), 2 (theta,
    // omega along z), 3 (Qxx, Qzx along z); afterwards component 0 .. 3 (Px Pz Sx Sz)
    const int task = tid / G::itemsU, ui = tid % G::itemsU;
    const bool has_u = task < 4;
    const int ur = ui / (TZ / 4), uc = 4 * (ui % (TZ / 4));
    const int gi = x0 + ur;
    const int gu = gi * P + (z0 + uc);

    // ---- operands: issued here, used after the copies and in the two stages --
    float4 m1 = zero4(), m2 = zero4(), vp2 = zero4(), vs2 = zero4(), dS = zero4();   // S-stage
    const bool s_damp = MODE != kRec && has_s && (sx_thread ? f.px : f.pz);
    if (has_s) {
        if (sx_thread) vp2 = ldg4(gm.vp2 + gs);
        vs2 = ldg4(gm.vs2 + gs);
    }
    if (s_damp) dS = ldg4((sx_thread ? gm.ax : gm.az) + gs);
    float4 o1 = zero4(), o2 = zero4(), dU = zero4(), now4 = zero4(), past4 = zero4();   // U-stage
    const bool u_damp = MODE != kRec && has_u && (task < 2 ? f.px : f.pz);
    pdl_wait();   // everything above is constant through a time loop
    if (tid == 0) issue_u_box<G>(p, sm, x0, z0, sv.b, bar);
    if (s_damp) {
        m1 = ldg4((sx_thread ? p.f_old[0] : p.f_old[1]) + off + gs);   // xx | zz
        m2 = ldg4((sx_thread ? p.f_old[3] : p.f_old[2]) + off + gs);   // zx | xz
    }
    float* const op1 = task == 0 ? p.o[4] : task == 1 ? p.o[2] : task == 2 ? p.o[5] : p.o[3];   // Tx B Tz A
    float* const op2 = task == 0 ? p.o[7] : task == 1 ? p.o[1] : task == 2 ? p.o[6] : p.o[0];   // Wx E Wz C
    const float* const nowp = task == 0 ? p.now[0] : task == 1 ? p.now[1] : task == 2 ? p.now[2] : p.now[3];
    float* const pastp = task == 0 ? p.past[0] : task == 1 ? p.past[1] : task == 2 ? p.past[2] : p.past[3];
    auto load_u = [&]() {
        if (u_damp) {
            dU = ldg4((task < 2 ? gm.ax : gm.az) + gu);
            o1 = ldg4(op1 + off + gu);
            o2 = ldg4(op2 + off + gu);
        }
        if (has_u) {
            now4 = ldg4(nowp + off + gu);
            past4 = ldg4(pastp + off + gu);
        }
    };
    if constexpr (CTAS == 1) load_u();

    // ---- phase 1: U = P + S over the tile and a 2N halo ---------------------
    float* stS = sm + G::oTh;   // Sx then Sz staging, UR x UC each
    const int err_word = p.err ? *(volatile const int*)p.err : 0;   // consumed after the wait
    const bool landed = mbar_wait(bar, 0u);
    if (!__syncthreads_and(landed && !(err_word & 1))) {
        // as in step_tile: let copies in flight land, then report
        if (tid == 0) {
            if (!landed) mbar_wait(bar, 0u);
            if (p.err) atomicOr(p.err, 1);
        }
        __syncthreads();
        return false;
    }
    for (int idx = tid; idx < G::UR * (UC / 4); idx += NT) {
        st4(sUx + 4 * idx, add4(ld4(sUx + 4 * idx), ld4(stS + 4 * idx)));                  // Ux = Px + Sx (PS:302)
        st4(sUz + 4 * idx, add4(ld4(sUz + 4 * idx), ld4(stS + G::UR * UC + 4 * idx)));     // Uz = Pz + Sz
    }
    if (MODE == kRcv && f.inj) {
        __syncthreads();
        // load_record (PS:1471-1483), as in step_tile
        const int col = sv.rz - ux_j0;
        for (int q = tid; q < G::UR; q += NT) {
            const int i = ux_i0 + q;
            if (i >= p.L && i < gm.X - p.L) {
                sUx[q * UC + col] = sv.inj_x[i];
                sUz[q * UC + col] = sv.inj_z[i];
            }
        }
    }
    if (MODE == kRec && f.ring) {
        __syncthreads();
        // read_wavefiled1 (PS:1344-1376), as in step_tile
        const ShotDesc& d = p.shots[sv.b];
        const void* su = strip_slot_ptr(p, d, p.slot_u);
        const unsigned* am = d.amax ? d.amax + (size_t)p.slot_u * kStripFields : nullptr;
        for_ring<NT>(gm.ring, ux_i0, ux_i0 + G::UR, ux_j0, ux_j0 + UC, [&](int i, int j, int ri) {
            const int o = (i - ux_i0) * UC + (j - ux_j0);
            const float ux = strip_get(p, su, am, kSUx, kSUx * R + ri);
            const float uz = strip_get(p, su, am, kSUz, kSUz * R + ri);
            sUx[o] = ux;
            sUz[o] = uz;
        });
    }
    __syncthreads();

    // ---- phase 2: S-stage on the tile plus an N halo -------------------------
    const bool s_border = MODE != kRec && f.border;
    unsigned s_live = 0xfu;
    if (s_border) {   // cells outside [N, X-N) x [N, Z-N) are never updated and stay zero
        const bool row_live = x0 + r >= N && x0 + r < gm.X - N;
        s_live = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) s_live |= (row_live && z0 + c + k >= N && z0 + c + k < p.Z - N) ? (1u << k) : 0u;
    }
    auto mask4 = [](float4& v, unsigned live) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (!(live & (1u << k))) set_comp(v, k, 0.f);
    };
    const float* ux0 = sUx + (r + SHX + N) * UC + (c + HU);
    const float* uz0 = sUz + (r + SHX + N) * UC + (c + HU);
    const int sr = r + SHX, scol = c + HS;
    float4 exx[1], ezx[1];
    if (has_s && sx_thread) {
        dx4<N, 1, false>(ux0, UC, a, dvx, exx);   // dvxdx = D-x Ux
        dx4<N, 1, true>(uz0, UC, a, dvx, ezx);    // dvzdx = D+x Uz
        if (s_damp) {
            m1 = cpml4(m1, dS, exx[0], dt);   // Fxx
            m2 = cpml4(m2, dS, ezx[0], dt);   // Fzx
        }
        float4 qzx = mul4(vs2, sub4(ezx[0], m2)), qxx = mul4(vs2, sub4(exx[0], m1));
        if (s_border) { mask4(qzx, s_live); mask4(qxx, s_live); }
        if (r >= 0 && r < TX) {
            st4(sQxx + r * SC + scol, qxx);
            st4(sQzx + r * SC + scol, qzx);
        }
    } else if (has_s) {
        const float4 exz = dz4<N, true>(ux0, a, dvz);    // dvxdz = D+z Ux
        const float4 ezz = dz4<N, false>(uz0, a, dvz);   // dvzdz = D-z Uz
        if (s_damp) {
            m1 = cpml4(m1, dS, ezz, dt);      // Fzz
            m2 = cpml4(m2, dS, exz, dt);      // Fxz
            sE[2 * G::itemsS + item] = m1;
            sE[3 * G::itemsS + item] = m2;
        }
        sE[item] = ezz;
        sE[G::itemsS + item] = exz;
        float4 qzz = mul4(vs2, sub4(ezz, m1)), qxz = mul4(vs2, sub4(exz, m2));
        if (s_border) { mask4(qzz, s_live); mask4(qxz, s_live); }
        if (item < G::itemsA) {
            st4(sQxz + sr * TZ + c, qxz);
            st4(sQzz + sr * TZ + c, qzz);
        }
    }
    __syncthreads();
    if (has_s && sx_thread) {
        // theta = Vp^2 (exx + ezz - Fxx - Fzz), omega = Vs^2 (exz - ezx - Fxz + Fzx) (PS:373-378)
        const float4 ezz = sE[item], exz = sE[G::itemsS + item];
        float4 fzz = zero4(), fxz = zero4();
        if (MODE != kRec && f.pz) { fzz = sE[2 * G::itemsS + item]; fxz = sE[3 * G::itemsS + item]; }
        float4 th = mul4(vp2, sub4(sub4(add4(exx[0], ezz), m1), fzz));
        float4 om = mul4(vs2, add4(sub4(sub4(exz, ezx[0]), fxz), m2));
        if (s_border) { mask4(th, s_live); mask4(om, s_live); }
        if (f.src && MODE != kRcv && !(MODE == kFwd && sv.src_type == 1) && x0 + r == sv.sx) {
            // source term on theta after the Q fields (PS:380)
            const int k = sv.sz - z0 - c;
            if (k >= 0 && k < 4) set_comp(th, k, comp(th, k) + sv.wavelet[MODE == kRec ? p.t + 1 : p.t]);
        }
        st4(sTh + sr * SC + scol, th);
        st4(sOm + sr * SC + scol, om);
    }
    if (s_damp && s_own) {
        if (s_border) { mask4(m1, s_live); mask4(m2, s_live); }
        stg4((sx_thread ? p.f_new[0] : p.f_new[1]) + off + gs, m1);
        stg4((sx_thread ? p.f_new[3] : p.f_new[2]) + off + gs, m2);
    }
    if (f.ring) {
        __syncthreads();
        const ShotDesc& d = p.shots[sv.b];
        if (MODE == kRec) {
            // read_wavefiled2 (PS:1377-1424), as in step_tile
            const void* ss = strip_slot_ptr(p, d, p.slot_s);
            const unsigned* am = d.amax ? d.amax + (size_t)p.slot_s * kStripFields : nullptr;
            for_ring<NT>(gm.ring, x0 - SHX, x0 + TX + SHX, z0 - HS, z0 + TZ + HS, [&](int i, int j, int ri) {
                const int q = i - x0, w = j - z0;
                const bool rin = q >= 0 && q < TX, cin = w >= 0 && w < TZ;
                float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (rin || cin) {
                    v[0] = strip_get(p, ss, am, kSTh, kSTh * R + ri);
                    v[1] = strip_get(p, ss, am, kSOm, kSOm * R + ri);
                }
                if (cin) {
                    v[2] = strip_get(p, ss, am, kSQxz, kSQxz * R + ri);
                    v[3] = strip_get(p, ss, am, kSQzz, kSQzz * R + ri);
                }
                if (rin) {
                    v[4] = strip_get(p, ss, am, kSQxx, kSQxx * R + ri);
                    v[5] = strip_get(p, ss, am, kSQzx, kSQzx * R + ri);
                }
                if (rin || cin) {
                    const int o = (q + SHX) * SC + (w + HS);
                    sTh[o] = v[0];
                    sOm[o] = v[1];
                }
                if (cin) {
                    sQxz[(q + SHX) * TZ + w] = v[2];
                    sQzz[(q + SHX) * TZ + w] = v[3];
                }
                if (rin) {
                    sQxx[q * SC + (w + HS)] = v[4];
                    sQzx[q * SC + (w + HS)] = v[5];
                }
            });
        }
        if (MODE == kFwd) {
            // save_wavefiled (PS:1230-1287), as in step_tile
            void* s = strip_save_ptr(p, d);
            float m[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for_ring<NT>(gm.ring, x0, x0 + TX, z0, z0 + TZ, [&](int i, int j, int ri) {
                const int q = i - x0, w = j - z0;
                const int o = (q + SHX) * SC + (w + HS);
                const float v[6] = {sTh[o], sOm[o], sQzx[q * SC + (w + HS)], sQzz[(q + SHX) * TZ + w],
                                    sQxx[q * SC + (w + HS)], sQxz[(q + SHX) * TZ + w]};
#pragma unroll
                for (int e = 0; e < 6; ++e) {
                    strip_put(p, s, (kSTh + e) * R + ri, v[e]);
                    m[e] = fmaxf(m[e], fabsf(v[e]));
                }
            });
            if (p.strip_prec == kStripF16) amax_commit<6>(d.amax + (size_t)p.t * kStripFields, kSTh, m);
        }
    }
    __syncthreads();

    // ---- phase 3: U-stage on the tile's own cells ----------------------------
    if constexpr (CTAS == 2) load_u();
    unsigned live = 0xfu;
    if (f.border) {
        live = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) live |= u_live<N, MODE>(p, gm, gi, z0 + uc + k) ? (1u << k) : 0u;
    }
    if (has_u) {
        float4 d1, d2;
        if (task < 2) {
            float4 e1[1], e2[1];
            if (task == 0) {
                dx4<N, 1, true>(sTh + (ur + SHX) * SC + (uc + HS), SC, a, dvx, e1);    // dthetadx = D+x theta
                dx4<N, 1, false>(sOm + (ur + SHX) * SC + (uc + HS), SC, a, dvx, e2);   // domegadx = D-x omega
            } else {
                dx4<N, 1, false>(sQxz + (ur + SHX) * TZ + uc, TZ, a, dvx, e1);         // dux_zdx = D-x Qxz
                dx4<N, 1, true>(sQzz + (ur + SHX) * TZ + uc, TZ, a, dvx, e2);          // duz_zdx = D+x Qzz
            }
            d1 = e1[0];
            d2 = e2[0];
        } else {
            // theta, omega | Qxx, Qzx: D+z of the first, D-z of the second
            const float* f1 = task == 2 ? sTh + (ur + SHX) * SC + (uc + HS) : sQxx + ur * SC + (uc + HS);
            const float* f2 = task == 2 ? sOm + (ur + SHX) * SC + (uc + HS) : sQzx + ur * SC + (uc + HS);
            d1 = dz4<N, true>(f1, a, dvz);
            d2 = dz4<N, false>(f2, a, dvz);
        }
        sD[(2 * task) * G::itemsU + ui] = d1;
        sD[(2 * task + 1) * G::itemsU + ui] = d2;
        if (u_damp) {
            o1 = cpml4(o1, dU, d1, dt);
            o2 = cpml4(o2, dU, d2, dt);
            sD[(8 + 2 * task) * G::itemsU + ui] = o1;
            sD[(9 + 2 * task) * G::itemsU + ui] = o2;
            if (f.border) { mask4(o1, live); mask4(o2, live); }
            stg4(op1 + off + gu, o1);
            stg4(op2 + off + gu, o2);
        }
    }
    // imaging operands of this thread's accumulator (0 PP, 1 PS, 2
    // illumination): read before the barrier, as the levels are overwritten
    // after it
    float4 isx = zero4(), isz = zero4(), ra = zero4(), rb = zero4(), acc = zero4(), cmp = zero4();
    if (MODE == kRec && has_u && task < 3) {
        const float* const* lv = p.img_past ? (const float* const*)p.past : p.now;
        isx = ldg4(lv[0] + off + gu);
        isz = ldg4(lv[1] + off + gu);
        if (task < 2) {
            ra = ldg4((task == 0 ? p.rcv[0] : p.rcv[2]) + off + gu);
            rb = ldg4((task == 0 ? p.rcv[1] : p.rcv[3]) + off + gu);
        } else {
            ra = isx;
            rb = isz;
        }
        acc = ldg4((task == 0 ? p.acc[0] : task == 1 ? p.acc[1] : p.acc[2]) + off + gu);
        if (p.comp_image) cmp = ldg4((task == 0 ? p.comp[0] : task == 1 ? p.comp[1] : p.comp[2]) + off + gu);
    }
    __syncthreads();
    if (has_u) {
        auto D = [&](int k) { return sD[k * G::itemsU + ui]; };   // tx wx B E tz wz A C, then their memories
        // leapfrog brackets in the reference's order (PS:291-294), as in step_tile
        const bool xcomp = task == 0 || task == 2;   // Px, Sx: C, E; Pz, Sz: B, A
        const int k0 = task == 0 ? 0 : task == 1 ? 4 : task == 2 ? 5 : 1;   // tx tz wz wx
        const bool k0x = task == 0 || task == 3;     // an x derivative
        float4 e0 = D(k0), e1 = xcomp ? D(7) : D(2), e2 = xcomp ? D(3) : D(6);
        float4 q0 = zero4(), q1 = zero4(), q2 = zero4();   // memories of e0, e1 (C | B), e2 (E | A)
        if (MODE != kRec && (k0x ? f.px : f.pz)) q0 = D(8 + k0);
        if (MODE != kRec && f.pz) { if (xcomp) q1 = D(15); else q2 = D(14); }   // C | A
        if (MODE != kRec && f.px) { if (xcomp) q2 = D(11); else q1 = D(10); }   // E | B
        float4 sum;
        if (task == 3) sum = add4(make_float4(-e0.x, -e0.y, -e0.z, -e0.w), q0);
        else sum = sub4(e0, q0);
        sum = add4(sub4(sub4(add4(sum, e1), e2), q1), q2);
        if (p.density) sum = mul4(sum, ldg4((xcomp ? gm.bx : gm.bz) + gu));
        const float2 two = dup2(2.f), dt2 = dup2(p.dt2), neg = dup2(-1.f);
        float4 nv = cat4(fma2(dt2, lo2(sum), fma2(two, lo2(now4), mul2(lo2(past4), neg))),
                         fma2(dt2, hi2(sum), fma2(two, hi2(now4), mul2(hi2(past4), neg))));
        if (MODE == kFwd && task == 1 && f.src && sv.src_type == 1 && gi == sv.sx && sv.sz >= z0 + uc && sv.sz < z0 + uc + 4)
            set_comp(nv, sv.sz - z0 - uc, comp(nv, sv.sz - z0 - uc) + p.dt2 * sv.wavelet[p.t]);
        if (f.border) mask4(nv, live);
        stg4(pastp + off + gu, nv);
        if (MODE == kFwd) sN[task * G::itemsU + ui] = nv;   // for the record and the strips
        if (MODE == kRec && task < 3) {
            // zero-lag imaging condition (corr_v, PS:1426-1439) on the interior, as in step_tile
            auto corr = [&](float4 v) {
                return cat4(add2(lo2(v), fma2(lo2(isx), lo2(ra), mul2(lo2(isz), lo2(rb)))),
                            add2(hi2(v), fma2(hi2(isx), hi2(ra), mul2(hi2(isz), hi2(rb)))));
            };
            float* accp = (task == 0 ? p.acc[0] : task == 1 ? p.acc[1] : p.acc[2]) + off + gu;
            if (!p.comp_image) {
                const float4 v = corr(acc);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (live & (1u << k)) set_comp(acc, k, comp(v, k));
                stg4(accp, acc);
            } else {
                const float4 term = corr(zero4());
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (!(live & (1u << k))) continue;
                    const float y = __fsub_rn(comp(term, k), comp(cmp, k));
                    const float t = __fadd_rn(comp(acc, k), y);
                    set_comp(cmp, k, __fsub_rn(__fsub_rn(t, comp(acc, k)), y));
                    set_comp(acc, k, t);
                }
                stg4(accp, acc);
                stg4((task == 0 ? p.comp[0] : task == 1 ? p.comp[1] : p.comp[2]) + off + gu, cmp);
            }
        }
    }
    if (MODE == kFwd) {
        const bool rec = sv.rec_x && sv.rz >= z0 && sv.rz < z0 + TZ;
        if (rec || f.ring) {
            __syncthreads();
            const float* n0 = sm + G::oNew;
            if (rec && tid < TX && x0 + tid < gm.X) {
                const int o = tid * TZ + (sv.rz - z0);
                sv.rec_x[x0 + tid] = __fadd_rn(n0[o], n0[2 * TX * TZ + o]);            // post-update value (PS:307-311)
                sv.rec_z[x0 + tid] = __fadd_rn(n0[TX * TZ + o], n0[3 * TX * TZ + o]);
            }
            if (f.ring) {
                // save_wavefiled (PS:1230-1287): the new displacement of the tile's ring cells
                const ShotDesc& d = p.shots[sv.b];
                void* s = strip_save_ptr(p, d);
                float m[2] = {0.f, 0.f};
                for_ring<NT>(gm.ring, x0, x0 + TX, z0, z0 + TZ, [&](int i, int j, int ri) {
                    const int o = (i - x0) * TZ + (j - z0);
                    const float ux = __fadd_rn(n0[o], n0[2 * TX * TZ + o]);
                    const float uz = __fadd_rn(n0[TX * TZ + o], n0[3 * TX * TZ + o]);
                    strip_put(p, s, kSUx * R + ri, ux);
                    strip_put(p, s, kSUz * R + ri, uz);
                    m[0] = fmaxf(m[0], fabsf(ux));
                    m[1] = fmaxf(m[1], fabsf(uz));
                });
                if (p.strip_prec == kStripF16) {
                    amax_commit<2>(d.amax + (size_t)p.t * kStripFields, kSUx, m);
                    if (p.t > 0) {
                        // slot t-1 is complete: convert this tile's cells, as in step_tile
                        const float* src = d.stage + (size_t)((p.t - 1) & 1) * d.strip_slot;
                        __half* dst = reinterpret_cast<__half*>(static_cast<char*>(d.strips) + (size_t)(p.t - 1) * slot_bytes(p, d));
                        const unsigned* am = d.amax + (size_t)(p.t - 1) * kStripFields;
                        int k[kStripFields];
#pragma unroll
                        for (int q = 0; q < kStripFields; ++q) k[q] = f16_exp(am[q]);
                        for_ring<NT>(gm.ring, x0, x0 + TX, z0, z0 + TZ, [&](int, int, int ri) {
                            float v[kStripFields];   // all loads before the stores
#pragma unroll
                            for (int q = 0; q < kStripFields; ++q) v[q] = src[q * R + ri];
#pragma unroll
                            for (int q = 0; q < kStripFields; ++q) dst[q * R + ri] = __float2half_rn(scale2(v[q], k[q]));
                        });
                    }
                }
            }
        }
    }
    return true;
}

template <class G, int MODE, int CTAS>
__device__ __forceinline__ void small_cta(const StepArgs& p, int tile, float* sm) {
    const int tz = tile % p.tiles_z, tx = tile / p.tiles_z;
    const int x0 = p.tile_x0 + tx * G::TX, z0 = p.tile_z0 + tz * G::TZ;
    __shared__ uint64_t bar;
    pdl_launch_dependents();
    const ShotDesc& d = p.shots[blockIdx.y];
    if (tx * G::TX >= (MODE == kRec ? d.X - 2 * p.L : d.X)) return;   // beyond this shot's width
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_map(u_map<G>(p));
    }
    const Geo gm = geo_of(d);
    const ShotView sv = shot_view(p, blockIdx.y);
    const TileFlags f = tile_flags<G, MODE>(p, gm, sv, x0, z0);
    if (MODE == kRec && f.ring) prefetch_ring<G>(p, gm, d, x0, z0);
    __syncthreads();   // the mbarrier is initialised
    small_tile<G, MODE, CTAS>(p, gm, sv, sm, x0, z0, f, &bar);
}

template <int N, int MODE, int TX, int CTAS>
__global__ void __launch_bounds__(SmallGeo<N, TX>::NT, CTAS) k_small(const __grid_constant__ StepArgs p) {
    extern __shared__ __align__(128) float4 smem4[];
    small_cta<SmallGeo<N, TX>, MODE, CTAS>(p, blockIdx.x, reinterpret_cast<float*>(smem4));
}

// A whole back-step in one launch: the reconstruction + imaging of step t+1
// (tiles 0 .. nrec-1) beside the receiver step t.  The two are independent:
// both read the receiver level that step t+1 wrote, and the receiver step
// writes the older one.
template <int N, int TX, int CTAS>
__global__ void __launch_bounds__(SmallGeo<N, TX>::NT, CTAS) k_small_back(const __grid_constant__ StepArgs rec,
                                                                          const __grid_constant__ StepArgs rcv, int nrec) {
    extern __shared__ __align__(128) float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    if ((int)blockIdx.x < nrec) small_cta<SmallGeo<N, TX>, kRec, CTAS>(rec, blockIdx.x, sm);
    else small_cta<SmallGeo<N, TX>, kRcv, CTAS>(rcv, blockIdx.x - nrec, sm);
}

}  // namespace ouc
