// Pair-walk backward (sm_100a), one state per channel; the decomposition is described in cs2d_pair.cuh, the adjoint
// recurrence at the top of cs2d_blk_bwd.cu.
//
// Bands are walked bottom-up, each from right to left in groups of 8 columns.  For a group the thread recomputes h, q, delta
// and the derivative of softplus from the column on the left and the row above, which the forward left, and keeps them in
// TENSOR MEMORY (8 of its 256 columns per pixel: nothing is computed twice and nothing of it goes through shared memory);
// then it walks back with the adjoint.  (m, a) of a band's first row go to the band above through a scratch row.
// dB and dC are summed over the warp's 64 channels through shared memory, 8 pixels at a time, and added to global memory:
// one reduction per 32 elements of the scan.
#include "cs2d_pair.cuh"

namespace cs2d {

struct PwBwd {   // a warp's shared memory
    static constexpr int PP = 34;                            // pitch of a pixel's partial sums
    static constexpr int delta = 0, u = PW_IN, g = 2 * PW_IN, bc = 3 * PW_IN;
    static constexpr int part = bc + 64 * 8;                 // float2 [8 pixels][PP] (dB, dC) of every lane
    static constexpr int total = part + 8 * PP * 8;
};

__device__ __forceinline__ void tm_st8(uint32_t a, float2 x, float2 y, float2 z, float2 w) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(a), "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(z.x), "f"(z.y), "f"(w.x), "f"(w.y) : "memory");
}
__device__ __forceinline__ void tm_ld8(uint32_t a, float2 (&x)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(x[0].x), "=f"(x[0].y), "=f"(x[1].x), "=f"(x[1].y), "=f"(x[2].x), "=f"(x[2].y), "=f"(x[3].x), "=f"(x[3].y) : "r"(a) : "memory");
}
// the loaded values pass through the wait, so that nothing uses them before it
__device__ __forceinline__ void tm_wait_ld8(float2 (&x)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(x[0].x), "+f"(x[0].y), "+f"(x[1].x), "+f"(x[1].y), "+f"(x[2].x), "+f"(x[2].y), "+f"(x[3].x), "+f"(x[3].y)::"memory");
}

// DIRS: flips, shared channels or the merge.  G32: 16-bit inputs with an fp32 gradient (read without staging).
template <int DT, bool DIRS, bool EL, bool G32, bool CK>
__global__ void __launch_bounds__(PW_WARPS * 32, 2) pair_bwd_kernel(const __grid_constant__ Pw P) {
    using S = PwBwd;
    constexpr int ES = pw_io<DT>::ES, FS = pw_io<DT>::FS;
    extern __shared__ __align__(128) unsigned char smem_[];
    __shared__ uint32_t tm_base;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t sm = smem_addr(smem_) + warp * S::total;
    float2 *sBC = reinterpret_cast<float2 *>(smem_ + warp * S::total + S::bc), *sPart = reinterpret_cast<float2 *>(smem_ + warp * S::total + S::part);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tm_base)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tm = __shfl_sync(0xffffffffu, tm_base, 0) + ((uint32_t)warp << 21);   // this warp's lane quadrant; 8 columns per pixel: h left of it, q, delta, sigmoid

    const int rw = 1 << P.rwl, w = warp & (rw - 1), nsub = PW_WARPS >> P.rwl, stride = gridDim.x * nsub;
    const int first = blockIdx.x * nsub, lmax = (P.items - first + stride - 1) / stride * P.npass * P.period;
    const int steps = lmax + rw - 1;

    PwPos pos;
    pos.item = first + (warp >> P.rwl); pos.pass = pos.strip = 0;
    pos.decode(P);
    auto blk_of = [&](const PwPos &q) { return P.nblk - 1 - (q.pass * rw + w); };     // bands from the bottom up, blocks from the right
    auto live = [&](const PwPos &q, int L) { return L >= 0 && L < lmax && q.item < P.items && q.strip < P.nstrip && q.pass * rw + w < P.nblk; };
    const int lp = min(lane, P.nl - 1);   // this lane's place in the checkpoints
    PwLane PL;
    if constexpr (CK) PL.at(P, sm);
    PwBC<DT> bcr;
    auto blocks = [&](const PwPos &q, auto &&f) {   // f(delta's block, u's, dout's) of a position
        const int r0 = blk_of(q) * PW_R, c0 = (P.nstrip - 1 - q.strip) * P.fs, ch0 = q.tile * PW_CH, cg = q.g * P.dpg + ch0, b = q.bg / P.G, nch = P.dpg - ch0;
        const bool fh = DIRS && ((P.flip_h >> q.g) & 1u), fw = DIRS && ((P.flip_w >> q.g) & 1u);
        f(pw_block<DT>(P.delta, (int64_t)b * P.dl_bs + (int64_t)cg * P.dl_ds, P.dl_ds, P.dl_hs, nch, r0, c0, P, fh, fw),
          pw_block<DT>(P.u, (int64_t)b * P.u_bs + (int64_t)(DIRS && (P.shared & 1) ? ch0 : cg) * P.u_ds, P.u_ds, P.u_hs, nch, r0, c0, P, fh, fw),
          pw_block<DT>(P.out, (int64_t)b * P.o_bs + (int64_t)(DIRS && (P.shared & 2) ? ch0 : cg) * P.o_ds, P.o_ds, P.o_hs, nch, r0, c0, P, fh, fw));
    };
    auto start = [&](const PwPos &q) {   // fetch a block
        blocks(q, [&](const PwBlock &d, const PwBlock &u, const PwBlock &g) {
            if constexpr (CK) {
                pw_fetch_ck(sm + S::delta, d, P, P.delta); pw_fetch_ck(sm + S::u, u, P, P.u);
                if constexpr (!G32) pw_fetch_ck(sm + S::g, g, P, P.out);
                return;
            }
            if (!EL && P.vin == 8) {
                pw_fetch<8, false>(sm + S::delta, d, P, P.delta); pw_fetch<8, false>(sm + S::u, u, P, P.u);
                if constexpr (!G32) pw_fetch<8, false>(sm + S::g, g, P, P.out);
            } else {
                pw_fetch<4, EL>(sm + S::delta, d, P, P.delta); pw_fetch<4, EL>(sm + S::u, u, P, P.u);
                if constexpr (!G32) pw_fetch<4, EL>(sm + S::g, g, P, P.out);
            }
        });
        bk_commit();
        bcr.load(P, q, blk_of(q) * PW_R, (P.nstrip - 1 - q.strip) * P.fs, DIRS && ((P.flip_h >> q.g) & 1u), DIRS && ((P.flip_w >> q.g) & 1u));
    };
    float2 A1 = bc(0.f), A2 = bc(0.f), D2 = bc(0.f), bias2 = bc(0.f), mw2 = bc(1.f);
    float2 dA = bc(0.f), dD = bc(0.f), dbias = bc(0.f), dwa = bc(0.f), mcorner = bc(0.f);
    float2 e[PW_R], t[PW_R], ar[PW_R], mr[PW_R];               // column on the right
#pragma unroll
    for (int r = 0; r < PW_R; ++r) e[r] = t[r] = ar[r] = mr[r] = bc(0.f);
    if (w == 0 && live(pos, 0)) start(pos);
    for (int gs = 0; gs < steps; ++gs) {
        const int L = gs - w;
        PwPos nxt = pos;
        if (L >= 0) nxt.next(P, stride);
        const bool non = live(nxt, L + 1);
        if (!live(pos, L)) {   // before the worker's first block, past its last band, or past its items
            if (non) start(nxt);
            if (rw > 1) __syncthreads();
            pos = nxt;
            continue;
        }
        const int blk = blk_of(pos), r0 = blk * PW_R, c0 = (P.nstrip - 1 - pos.strip) * P.fs, ch0 = pos.tile * PW_CH, cg = pos.g * P.dpg + ch0, nch = P.dpg - ch0, b = pos.bg / P.G;
        const bool fh = DIRS && ((P.flip_h >> pos.g) & 1u), fw = DIRS && ((P.flip_w >> pos.g) & 1u);
        const int nc = min(P.fs, P.W - c0);
        const int nl = P.nl;
        const float4 *above = P.row + (((int64_t)pos.item * (P.nblk - 1) + blk - 1) * P.wp + c0) * nl + lp;
        float4 *arow = P.adj + ((int64_t)(first + (warp >> P.rwl)) * P.wp + c0) * 32 + lane;
        if (pos.strip == 0) {
            if (pos.pass == 0) {   // a new item
                const int k0 = min(2 * lane, nch - 1), k1 = min(2 * lane + 1, nch - 1);
                A1 = f2(__ldg(P.A + (int64_t)(cg + k0) * P.A_ds), __ldg(P.A + (int64_t)(cg + k1) * P.A_ds));
                A2 = mul2(A1, bc(LOG2E));
                D2 = P.D ? f2(__ldg(P.D + cg + k0), __ldg(P.D + cg + k1)) : bc(0.f);
                bias2 = P.bias ? f2(__ldg(P.bias + cg + k0), __ldg(P.bias + cg + k1)) : bc(0.f);
                if (DIRS && P.mw) mw2 = f2(__ldg(P.mw + cg + k0), __ldg(P.mw + cg + k1));
            }
            mcorner = bc(0.f);
#pragma unroll
            for (int r = 0; r < PW_R; ++r) e[r] = t[r] = ar[r] = mr[r] = bc(0.f);
        }
        // What two columns need from global memory is loaded two columns ahead: the row above, for the recomputation the column on
        // the left of a group too, for the way back the adjoint row below.
        float4 up[2], colq[PW_R], dn[2];
        float2 cola[PW_R], cnr = bc(0.f), hup[2];
        auto load_up = [&](int c) {
            up[0] = bk_ld16<true>(above + c * nl, blk > 0);
            up[1] = bk_ld16<true>(above + (c + 1) * nl, blk > 0);
        };
        auto load_group = [&](int c) {
            const bool left = c0 + c > 0;
            const int64_t o = ((((int64_t)pos.item * P.nblk + blk) * (P.nsub - 1) + ((c0 + c) >> 3) - 1) * 4) * nl + lp;
#pragma unroll
            for (int r = 0; r < PW_R; ++r) {
                colq[r] = bk_ld16<true>(P.colq + o + r * nl, left);
                cola[r] = pw_ld8(P.cola + o + r * nl, left);
            }
            cnr = pw_ld8(above + (c - 1) * nl, left && blk > 0);
            load_up(c);
        };
        auto load_back = [&](int c) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                dn[i] = bk_ld16<false>(arow + (c + i) * 32, blk + 1 < P.nblk);
                hup[i] = pw_ld8(above + (c + i) * nl, blk > 0);
            }
        };
        load_group((nc - 1) & ~7);
        PwView<DT, EL> vd, vu, vg;
        PwViewCk<DT, S::delta> cd;
        PwViewCk<DT, S::u> cu;
        PwViewCk<DT, S::g> cg_;
        blocks(pos, [&](const PwBlock &d, const PwBlock &u, const PwBlock &g) {
            if constexpr (CK) {
                cd.at(P, d); cu.at(P, u);
                if constexpr (!G32) cg_.at(P, g);
                return;
            }
            const int pit = P.vin == 8 ? 136 : 132;
            vd.at(sm + S::delta, d, pit); vu.at(sm + S::u, u, pit);
            if constexpr (!G32) vg.at(sm + S::g, g, pit);
        });
        bcr.put(sBC);
        bk_wait<0>();
        __syncwarp();
        if constexpr (CK && G32) pw_clear<ES>(P, PL, r0, fh, fw, cd, cu);
        else if constexpr (CK) pw_clear<ES>(P, PL, r0, fh, fw, cd, cu, cg_);
        const int64_t HW = (int64_t)P.H * P.W;
        const bool merge = DIRS && P.mw;
#pragma unroll 1
        for (int c1 = (nc - 1) & ~7; c1 >= 0; c1 -= 8) {   // groups of 8 columns
            const int c2 = min(c1 + 8, (nc + 1) & ~1);
            float2 hcur[PW_R];                             // h of the current column on the way back
            // ---- recompute ----
            {
                float2 hl[PW_R], al[PW_R], ql[PW_R], sl[PW_R], hcorner = cnr;
#pragma unroll
                for (int r = 0; r < PW_R; ++r) {
                    ql[r] = f2(colq[r].x, colq[r].y); sl[r] = f2(colq[r].z, colq[r].w);
                    al[r] = cola[r];
                    hl[r] = add2(ql[r], sl[r]);
                }
#pragma unroll 1
                for (int c = c1; c < c2; c += 2) {
                    const float2 hu2[2] = {f2(up[0].x, up[0].y), f2(up[1].x, up[1].y)}, au2[2] = {f2(up[0].z, up[0].w), f2(up[1].z, up[1].w)};
                    if (c + 2 < c2) load_up(c + 2);
                    else load_back(c);
                    const bool on1 = c + 1 < nc;
                    int o[PW_R], o1[PW_R];
                    pw_offsets<ES, EL, CK>(P, c, fh, fw, o, o1);
                    float xd[PW_R][2][2], xu[PW_R][2][2];   // row, channel, column
#pragma unroll
                    for (int r = 0; r < PW_R; ++r)
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            if constexpr (CK) { cd.load(PL, r, k, o1[r], fw, xd[r][k]); cu.load(PL, r, k, o1[r], fw, xu[r][k]); continue; }
                            vd.load(r, k, o[r], o1[r], fw, r0 + r < P.H, on1, xd[r][k]); vu.load(r, k, o[r], o1[r], fw, r0 + r < P.H, on1, xu[r][k]);
                        }
                    const uint32_t tt = tm + (c - c1) * 32;
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        float2 hd = hcorner, hu = hu2[cc], au = au2[cc];
                        hcorner = hu;
#pragma unroll
                        for (int r = 0; r < PW_R; ++r) {
                            const float2 u = f2(xu[r][0][cc], xu[r][1][cc]), x = add2(f2(xd[r][0][cc], xd[r][1][cc]), bias2);
                            const float B = sBC[r * FS + c + cc].x;
                            float2 sg;
                            const float2 dl = pw_softplus2<true>(x, &sg);
                            const float2 a = ex2_2(mul2(dl, A2)), p = mul2(bc(B), mul2(dl, u));
                            const float2 z = add2(ql[r], fma2(mul2(add2(au, al[r]), hd), bc(-0.5f), hu));
                            const float2 s = fma2(a, sl[r], p);
                            const float2 q = mul2(a, z), h = fma2(a, z, s);
                            tm_st8(tt + 8 * (cc * 4 + r), hl[r], q, dl, sg);
                            hd = hl[r]; hu = h; au = a;
                            hl[r] = h; al[r] = a; ql[r] = q; sl[r] = s;
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < PW_R; ++r) hcur[r] = hl[r];
            }
            tm_wait_st();
            // ---- walk back with the adjoint ----
#pragma unroll 1
            for (int c = c2 - 2; c >= c1; c -= 2) {
                const float2 m2[2] = {f2(dn[0].x, dn[0].y), f2(dn[1].x, dn[1].y)}, a2[2] = {f2(dn[0].z, dn[0].w), f2(dn[1].z, dn[1].w)}, h2[2] = {hup[0], hup[1]};
                if (c > c1) load_back(c - 2);
                else if (c1 > 0) load_group(c1 - 8);
                int o[PW_R], o1[PW_R];
                pw_offsets<ES, EL, CK>(P, c, fh, fw, o, o1);
                const bool on1 = c + 1 < nc;
                float xg[PW_R][2][2], xu[PW_R][2][2];   // row, channel, column
#pragma unroll
                for (int r = 0; r < PW_R; ++r)
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        if constexpr (G32) {
                            const uint32_t *src = reinterpret_cast<const uint32_t *>(P.out) + (int64_t)b * P.o_bs + (int64_t)((P.shared & 2 ? ch0 : cg) + 2 * lane + k) * P.o_ds + (int64_t)(fh ? P.H - 1 - r0 - r : r0 + r) * P.o_hs;
                            const int fc = fw ? P.W - 1 - c0 - c : c0 + c;
                            const bool on = r0 + r < P.H && 2 * lane + k < nch;
                            xg[r][k][0] = __uint_as_float(bk_ldp<CS2D_F32>(src + fc, on)); xg[r][k][1] = __uint_as_float(bk_ldp<CS2D_F32>(src + (fw ? fc - 1 : fc + 1), on && on1));
                        } else {
                            if constexpr (CK) cg_.load(PL, r, k, o1[r], fw, xg[r][k]);
                            else vg.load(r, k, o[r], o1[r], fw, r0 + r < P.H, on1, xg[r][k]);
                        }
                        if constexpr (CK) cu.load(PL, r, k, o1[r], fw, xu[r][k]);
                        else vu.load(r, k, o[r], o1[r], fw, r0 + r < P.H, on1, xu[r][k]);
                    }
                const uint32_t tt = tm + (c - c1) * 32;
                float2 rv[2][4];
                tm_ld8(tt + 8 * 7, rv[1]);
                float2 du[PW_R][2], dd[PW_R][2];
#pragma unroll
                for (int cc = 1; cc >= 0; --cc) {
                    float2 md = m2[cc], ad = a2[cc], mdd = mcorner;
                    mcorner = md;
#pragma unroll
                    for (int r = PW_R - 1; r >= 0; --r) {
                        const int j = cc * 4 + r, s = j & 1;
                        tm_wait_ld8(rv[s]);
                        const float2 hlf = rv[s][0], q = rv[s][1], dl = rv[s][2], sg = rv[s][3];
                        if (j > 0) tm_ld8(tt + 8 * (j - 1), rv[s ^ 1]);
                        const float2 u = f2(xu[r][0][cc], xu[r][1][cc]), gr = f2(xg[r][0][cc], xg[r][1][cc]), gv = DIRS ? mul2(gr, mw2) : gr;
                        const float2 BC = sBC[r * FS + c + cc], B = bc(BC.x), C = bc(BC.y);
                        const float2 a = ex2_2(mul2(dl, A2)), dlu = mul2(dl, u), p = mul2(B, dlu), gC = mul2(C, gv);
                        const float2 h = hcur[r], ha = r ? hcur[r ? r - 1 : 0] : h2[cc];
                        const float2 w1 = mul2(add2(ar[r], ad), mdd);
                        const float2 ev = fma2(ar[r], e[r], fma2(w1, bc(-0.5f), md));
                        const float2 tv = fma2(ar[r], t[r], gC);
                        const float2 m = mul2(a, add2(ev, tv));
                        const float2 X = fma2(md, hlf, mul2(mr[r], ha));
                        const float2 hp = fma2(p, bc(-1.f), h);
                        const float2 G = fma2(mul2(a, X), bc(-0.5f), fma2(ev, hp, mul2(tv, q)));
                        const float2 eps = fma2(gC, bc(0.25f), ev), yq = fma2(p, bc(0.25f), q);
                        const float2 S1 = mul2(B, eps), dBv = mul2(dlu, eps), dCv = mul2(gv, yq);
                        dA = fma2(dl, G, dA);
                        if constexpr (DIRS) dwa = fma2(mul2(C, yq), gr, dwa);
                        dD = fma2(gr, u, dD);
                        du[r][cc] = fma2(D2, gv, mul2(dl, S1));
                        dd[r][cc] = mul2(fma2(u, S1, mul2(A1, G)), sg);
                        dbias = add2(dbias, dd[r][cc]);
                        sPart[(cc * 4 + r) * S::PP + lane] = f2(dBv.x + dBv.y, dCv.x + dCv.y);
                        mdd = mr[r]; md = m; ad = a;
                        e[r] = ev; t[r] = tv; ar[r] = a; mr[r] = m;
                        if (r == 0 && blk > 0) arow[(c + cc) * 32] = make_float4(m.x, m.y, a.x, a.y);
                        hcur[r] = hlf;
                    }
                }
                // du takes the place of u, ddelta that of delta
                if (merge) {
                    const int fc = fw ? P.W - 1 - c0 - c : c0 + c;
#pragma unroll
                    for (int r = 0; r < PW_R; ++r) {
                        float *p = reinterpret_cast<float *>(P.du) + ((int64_t)b * P.dpg + ch0 + 2 * lane) * HW + (int64_t)(fh ? P.H - 1 - r0 - r : r0 + r) * P.W;
                        pw_put32(p, fc, du[r][0].x, du[r][1].x, fw, r0 + r < P.H && 2 * lane < nch, on1, P.v32, true);
                        pw_put32(p + HW, fc, du[r][0].y, du[r][1].y, fw, r0 + r < P.H && 2 * lane + 1 < nch, on1, P.v32, true);
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < PW_R; ++r) {
                        if constexpr (CK) { cu.store(PL, r, 0, o1[r], fw, du[r][0].x, du[r][1].x); cu.store(PL, r, 1, o1[r], fw, du[r][0].y, du[r][1].y); continue; }
                        vu.store(r, 0, o[r], o1[r], fw, du[r][0].x, du[r][1].x, on1); vu.store(r, 1, o[r], o1[r], fw, du[r][0].y, du[r][1].y, on1);
                    }
                }
#pragma unroll
                for (int r = 0; r < PW_R; ++r) {
                        if constexpr (CK) { cd.store(PL, r, 0, o1[r], fw, dd[r][0].x, dd[r][1].x); cd.store(PL, r, 1, o1[r], fw, dd[r][0].y, dd[r][1].y); continue; }
                        vd.store(r, 0, o[r], o1[r], fw, dd[r][0].x, dd[r][1].x, on1); vd.store(r, 1, o[r], o1[r], fw, dd[r][0].y, dd[r][1].y, on1);
                    }
                // dB, dC of the two columns: a lane sums a quarter of a pixel's 32 pairs
                __syncwarp();
                const float4 *src = reinterpret_cast<const float4 *>(sPart + (lane & 7) * S::PP + (lane >> 3) * 8);
                float2 x = bc(0.f), y = bc(0.f);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 v = src[i];
                    x = add2(x, f2(v.x, v.y)); y = add2(y, f2(v.z, v.w));
                }
                x = add2(x, y);
                const bool hi = lane & 8;      // this lane keeps dC, else dB
                float v = hi ? x.y : x.x;
                v += __shfl_xor_sync(0xffffffffu, hi ? x.x : x.y, 8);
                v += __shfl_xor_sync(0xffffffffu, v, 16);
                const int rr = r0 + (lane & 3), fc = c0 + c + ((lane >> 2) & 1);
                float *dst = (hi ? P.dC : P.dB) + (int64_t)pos.bg * HW + (int64_t)(fh ? P.H - 1 - rr : rr) * P.W + (fw ? P.W - 1 - fc : fc);
                bk_st<CS2D_F32, true>(dst, 0, v, lane < 16 && rr < P.H && fc < P.W);
                __syncwarp();
            }
        }
        __syncwarp();
        {
            const int64_t o = ((int64_t)b * P.dpg * P.G + cg) * HW;
            blocks(pos, [&](const PwBlock &d, const PwBlock &u, const PwBlock &) {
                if constexpr (CK) {
                    if (!merge) pw_store_ck(sm + S::u, pw_block<DT>(P.du, o, HW, P.W, nch, r0, c0, P, fh, fw), u, P);
                    pw_store_ck(sm + S::delta, pw_block<DT>(P.ddelta, o, HW, P.W, nch, r0, c0, P, fh, fw), d, P);
                    return;
                }
                if (!merge) pw_store(sm + S::u, pw_block<DT>(P.du, o, HW, P.W, nch, r0, c0, P, fh, fw), u, P);
                pw_store(sm + S::delta, pw_block<DT>(P.ddelta, o, HW, P.W, nch, r0, c0, P, fh, fw), d, P);
            });
        }
        __syncwarp();
        if (non) start(nxt);
        if (pos.strip == P.nstrip - 1 && blk - rw < 0) {   // the worker leaves the item: parameter gradients of its share
            const int k = cg + 2 * lane;
            const bool o0 = 2 * lane < nch, o1 = 2 * lane + 1 < nch;
            bk_st<CS2D_F32, true>(P.dA, k, dA.x, o0); bk_st<CS2D_F32, true>(P.dA, k + 1, dA.y, o1);
            if (P.dbias) { bk_st<CS2D_F32, true>(P.dbias, k, dbias.x, o0); bk_st<CS2D_F32, true>(P.dbias, k + 1, dbias.y, o1); }
            if (P.dD) { bk_st<CS2D_F32, true>(P.dD, k, dD.x * mw2.x, o0); bk_st<CS2D_F32, true>(P.dD, k + 1, dD.y * mw2.y, o1); }
            if (DIRS && P.dw) {
                const float2 v = fma2(D2, dD, dwa);
                bk_st<CS2D_F32, true>(P.dw, k, v.x, o0); bk_st<CS2D_F32, true>(P.dw, k + 1, v.y, o1);
            }
            dA = dbias = dD = dwa = bc(0.f);
        }
        if (rw > 1) __syncthreads();   // the adjoint row written in this step is there for the other workers
        pos = nxt;
    }
    bk_wait<0>();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(256));
}

template <int DT, bool DIRS, bool EL, bool G32, bool CK>
static cudaError_t launch(const Pw &P, cudaStream_t st) {
    auto kernel = pair_bwd_kernel<DT, DIRS, EL, G32, CK>;
    constexpr int smem = PwBwd::total * PW_WARPS;
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    kernel<<<P.grid, PW_WARPS * 32, smem, st>>>(P);
    return cudaGetLastError();
}
template <int DT>
static cudaError_t launch_dt(const Pw &P, cudaStream_t st) {
    if constexpr (DT != CS2D_F32) {
        if (P.f32) return P.ck ? launch<DT, true, false, true, true>(P, st) : P.el ? launch<DT, true, true, true, false>(P, st) : launch<DT, true, false, true, false>(P, st);
    }
    const bool dirs = P.flip_h || P.flip_w || P.shared || P.mw;
    if (P.ck) return dirs ? launch<DT, true, false, false, true>(P, st) : launch<DT, false, false, false, true>(P, st);
    if (dirs) return P.el ? launch<DT, true, true, false, false>(P, st) : launch<DT, true, false, false, false>(P, st);
    return P.el ? launch<DT, false, true, false, false>(P, st) : launch<DT, false, false, false, false>(P, st);
}
cudaError_t launch_pair_bwd(const Pw &P, cudaStream_t st) {
    switch (P.io_dt) {
        case CS2D_F32: return launch_dt<CS2D_F32>(P, st);
        case CS2D_F16: return launch_dt<CS2D_F16>(P, st);
        default: return launch_dt<CS2D_BF16>(P, st);
    }
}

}  // namespace cs2d
