// Pair-walk forward (sm_100a), one state per channel; the decomposition is described in cs2d_pair.cuh, the recurrence
// (carried as q = h - s) at the top of cs2d_blk_fwd.cu.
#include "cs2d_pair.cuh"

namespace cs2d {

struct PwFwd {   // a warp's shared memory
    static constexpr int delta = 0, u = PW_IN, bc = 2 * PW_IN, total = bc + 64 * 8;
};

// KEEP: a backward follows.  DIRS: flips, shared channels, the merge, or fp32 results of 16-bit inputs.
template <int DT, bool KEEP, bool DIRS, bool EL, bool CK>
__global__ void __launch_bounds__(PW_WARPS * 32, 3) pair_fwd_kernel(const __grid_constant__ Pw P) {
    constexpr int ES = pw_io<DT>::ES, FS = pw_io<DT>::FS;
    extern __shared__ __align__(128) unsigned char smem_[];
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t sm = smem_addr(smem_) + warp * PwFwd::total;
    float2 *sBC = reinterpret_cast<float2 *>(smem_ + warp * PwFwd::total + PwFwd::bc);
    const int rw = 1 << P.rwl, w = warp & (rw - 1), nsub = PW_WARPS >> P.rwl, stride = gridDim.x * nsub;
    const int first = blockIdx.x * nsub, lmax = (P.items - first + stride - 1) / stride * P.npass * P.period;
    const int steps = lmax + rw - 1;

    PwPos pos;
    pos.item = first + (warp >> P.rwl); pos.pass = pos.strip = 0;
    pos.decode(P);
    auto live = [&](const PwPos &q, int L) { return L >= 0 && L < lmax && q.item < P.items && q.strip < P.nstrip && q.pass * rw + w < P.nblk; };
    const int lp = min(lane, P.nl - 1);   // this lane's place in the checkpoints
    PwLane PL;
    if constexpr (CK) PL.at(P, sm);
    PwBC<DT> bcr;
    auto blocks = [&](const PwPos &q, auto &&f) {   // f(delta's block, u's block) of a position
        const int r0 = (q.pass * rw + w) * PW_R, c0 = q.strip * P.fs, ch0 = q.tile * PW_CH, cg = q.g * P.dpg + ch0, b = q.bg / P.G, nch = P.dpg - ch0;
        const bool fh = DIRS && ((P.flip_h >> q.g) & 1u), fw = DIRS && ((P.flip_w >> q.g) & 1u);
        f(pw_block<DT>(P.delta, (int64_t)b * P.dl_bs + (int64_t)cg * P.dl_ds, P.dl_ds, P.dl_hs, nch, r0, c0, P, fh, fw),
          pw_block<DT>(P.u, (int64_t)b * P.u_bs + (int64_t)(DIRS && (P.shared & 1) ? ch0 : cg) * P.u_ds, P.u_ds, P.u_hs, nch, r0, c0, P, fh, fw));
    };
    auto start = [&](const PwPos &q) {   // fetch a block
        blocks(q, [&](const PwBlock &d, const PwBlock &u) {
            if constexpr (CK) { pw_fetch_ck(sm + PwFwd::delta, d, P, P.delta); pw_fetch_ck(sm + PwFwd::u, u, P, P.u); return; }
            if (!EL && P.vin == 8) { pw_fetch<8, false>(sm + PwFwd::delta, d, P, P.delta); pw_fetch<8, false>(sm + PwFwd::u, u, P, P.u); }
            else { pw_fetch<4, EL>(sm + PwFwd::delta, d, P, P.delta); pw_fetch<4, EL>(sm + PwFwd::u, u, P, P.u); }
        });
        bk_commit();
        bcr.load(P, q, (q.pass * rw + w) * PW_R, q.strip * P.fs, DIRS && ((P.flip_h >> q.g) & 1u), DIRS && ((P.flip_w >> q.g) & 1u));
    };
    float2 A2 = bc(0.f), D2 = bc(0.f), bias2 = bc(0.f), mw2 = bc(1.f);
    float2 hl[PW_R], al[PW_R], ql[PW_R], sl[PW_R], hcorner = bc(0.f);   // the column on the left; h of the row above it
#pragma unroll
    for (int r = 0; r < PW_R; ++r) hl[r] = al[r] = ql[r] = sl[r] = bc(0.f);
    if (w == 0 && live(pos, 0)) start(pos);
    for (int g = 0; g < steps; ++g) {
        const int L = g - w;
        PwPos nxt = pos;
        if (L >= 0) nxt.next(P, stride);
        const bool non = live(nxt, L + 1);
        if (!live(pos, L)) {   // before the worker's first block, past its last band, or past its items
            if (non) start(nxt);
            if (rw > 1) __syncthreads();
            pos = nxt;
            continue;
        }
        const int blk = pos.pass * rw + w, r0 = blk * PW_R, c0 = pos.strip * P.fs, ch0 = pos.tile * PW_CH, cg = pos.g * P.dpg + ch0, nch = P.dpg - ch0, b = pos.bg / P.G;
        const bool fh = DIRS && ((P.flip_h >> pos.g) & 1u), fw = DIRS && ((P.flip_w >> pos.g) & 1u);
        const int nc = min(P.fs, P.W - c0);
        // row of the band above (rolling: the same row), row of this band (rolling: the team's)
        const int nl = KEEP ? P.nl : 32;
        float4 *row = P.row + ((KEEP ? (int64_t)pos.item * (P.nblk - 1) + blk : (int64_t)(first + (warp >> P.rwl))) * P.wp + c0) * nl + (KEEP ? lp : lane);
        const float4 *above = KEEP ? row - (int64_t)P.wp * nl : row;
        float4 up[2];
        auto fetch_up = [&](int c) {
            up[0] = bk_ld16<false>(above + c * nl, blk > 0);
            up[1] = bk_ld16<false>(above + (c + 1) * nl, blk > 0);
        };
        fetch_up(0);
        if (pos.strip == 0) {
            if (pos.pass == 0) {   // a new item
                const int k0 = min(2 * lane, nch - 1), k1 = min(2 * lane + 1, nch - 1);
                A2 = f2(__ldg(P.A + (int64_t)(cg + k0) * P.A_ds) * LOG2E, __ldg(P.A + (int64_t)(cg + k1) * P.A_ds) * LOG2E);
                D2 = P.D ? f2(__ldg(P.D + cg + k0), __ldg(P.D + cg + k1)) : bc(0.f);
                bias2 = P.bias ? f2(__ldg(P.bias + cg + k0), __ldg(P.bias + cg + k1)) : bc(0.f);
                if (DIRS && P.mw) mw2 = f2(__ldg(P.mw + cg + k0), __ldg(P.mw + cg + k1));
            }
#pragma unroll
            for (int r = 0; r < PW_R; ++r) hl[r] = al[r] = ql[r] = sl[r] = bc(0.f);
            hcorner = bc(0.f);
        }
        PwView<DT, EL> vd, vu;
        PwViewCk<DT, PwFwd::delta> cd;
        PwViewCk<DT, PwFwd::u> cu;
        blocks(pos, [&](const PwBlock &d, const PwBlock &u) {
            if constexpr (CK) { cd.at(P, d); cu.at(P, u); }
            else { vd.at(sm + PwFwd::delta, d, P.vin == 8 ? 136 : 132); vu.at(sm + PwFwd::u, u, P.vin == 8 ? 136 : 132); }
        });
        bcr.put(sBC);
        bk_wait<0>();
        __syncwarp();
        if constexpr (CK) pw_clear<ES>(P, PL, r0, fh, fw, cd, cu);
#pragma unroll 1
        for (int c = 0; c < nc; c += 2) {
            if (KEEP && c0 + c > 0 && ((c0 + c) & 7) == 0) {   // the column left of a group of 8
                const int64_t o = ((((int64_t)pos.item * P.nblk + blk) * (P.nsub - 1) + ((c0 + c) >> 3) - 1) * 4) * nl + lp;
#pragma unroll
                for (int r = 0; r < PW_R; ++r) {
                    P.colq[o + r * nl] = make_float4(ql[r].x, ql[r].y, sl[r].x, sl[r].y);
                    P.cola[o + r * nl] = al[r];
                }
            }
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
            const float2 hu2[2] = {f2(up[0].x, up[0].y), f2(up[1].x, up[1].y)}, au2[2] = {f2(up[0].z, up[0].w), f2(up[1].z, up[1].w)};
            if (c + 2 < nc) fetch_up(c + 2);
            float2 y[PW_R][2];
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                float2 hd = hcorner, hu = hu2[cc], au = au2[cc];
                hcorner = hu;
#pragma unroll
                for (int r = 0; r < PW_R; ++r) {
                    const float2 u = f2(xu[r][0][cc], xu[r][1][cc]), x = add2(f2(xd[r][0][cc], xd[r][1][cc]), bias2);
                    const float2 BC = sBC[r * FS + c + cc];
                    const float2 dl = pw_softplus2<false>(x, nullptr);
                    const float2 a = ex2_2(mul2(dl, A2)), p = mul2(bc(BC.x), mul2(dl, u));
                    const float2 z = add2(ql[r], fma2(mul2(add2(au, al[r]), hd), bc(-0.5f), hu));
                    const float2 s = fma2(a, sl[r], p);
                    const float2 q = mul2(a, z), h = fma2(a, z, s);
                    y[r][cc] = fma2(bc(BC.y), fma2(p, bc(0.25f), q), mul2(D2, u));
                    hd = hl[r]; hu = h; au = a;
                    hl[r] = h; al[r] = a; ql[r] = q; sl[r] = s;
                }
                bk_st16(row + (c + cc) * nl, make_float4(hl[PW_R - 1].x, hl[PW_R - 1].y, al[PW_R - 1].x, al[PW_R - 1].y), blk + 1 < P.nblk);
            }
            if (DIRS && (P.mw || P.f32)) {   // straight to the fp32 results (merge: onto the image)
                const int fc = fw ? P.W - 1 - c0 - c : c0 + c;
#pragma unroll
                for (int r = 0; r < PW_R; ++r) {
                    float *p = reinterpret_cast<float *>(P.out) + (int64_t)b * P.o_bs + (int64_t)((P.mw ? ch0 : cg) + 2 * lane) * P.o_ds + (int64_t)(fh ? P.H - 1 - r0 - r : r0 + r) * P.o_hs;
                    const float2 y0 = mul2(y[r][0], mw2), y1 = mul2(y[r][1], mw2);
                    pw_put32(p, fc, y0.x, y1.x, fw, r0 + r < P.H && 2 * lane < nch, on1, P.v32, P.mw);
                    pw_put32(p + P.o_ds, fc, y0.y, y1.y, fw, r0 + r < P.H && 2 * lane + 1 < nch, on1, P.v32, P.mw);
                }
            } else {
#pragma unroll
                for (int r = 0; r < PW_R; ++r) {
                    if constexpr (CK) { cu.store(PL, r, 0, o1[r], fw, y[r][0].x, y[r][1].x); cu.store(PL, r, 1, o1[r], fw, y[r][0].y, y[r][1].y); continue; }
                    vu.store(r, 0, o[r], o1[r], fw, y[r][0].x, y[r][1].x, on1); vu.store(r, 1, o[r], o1[r], fw, y[r][0].y, y[r][1].y, on1);
                }
            }
        }
        __syncwarp();
        if (!DIRS || !(P.mw || P.f32)) {
            blocks(pos, [&](const PwBlock &, const PwBlock &u) {
                const PwBlock y = pw_block<DT>(P.out, (int64_t)b * P.o_bs + (int64_t)cg * P.o_ds, P.o_ds, P.o_hs, nch, r0, c0, P, fh, fw);
                if constexpr (CK) pw_store_ck(sm + PwFwd::u, y, u, P);
                else pw_store(sm + PwFwd::u, y, u, P);
            });
            __syncwarp();
        }
        if (non) start(nxt);
        if (rw > 1) __syncthreads();   // the row written in this step is there for the other workers
        pos = nxt;
    }
    bk_wait<0>();
}

template <int DT, bool KEEP, bool DIRS, bool EL, bool CK>
static cudaError_t launch(const Pw &P, cudaStream_t st) {
    auto kernel = pair_fwd_kernel<DT, KEEP, DIRS, EL, CK>;
    constexpr int smem = PwFwd::total * PW_WARPS;
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
template <int DT, bool KEEP>
static cudaError_t launch_el(const Pw &P, cudaStream_t st) {
    const bool dirs = P.flip_h || P.flip_w || P.shared || P.mw || P.f32;
    if (P.ck) return dirs ? launch<DT, KEEP, true, false, true>(P, st) : launch<DT, KEEP, false, false, true>(P, st);
    if (dirs) return P.el ? launch<DT, KEEP, true, true, false>(P, st) : launch<DT, KEEP, true, false, false>(P, st);
    return P.el ? launch<DT, KEEP, false, true, false>(P, st) : launch<DT, KEEP, false, false, false>(P, st);
}
template <int DT>
static cudaError_t launch_dt(const Pw &P, bool keep, cudaStream_t st) { return keep ? launch_el<DT, true>(P, st) : launch_el<DT, false>(P, st); }
cudaError_t launch_pair_fwd(const Pw &P, bool keep, cudaStream_t st) {
    switch (P.io_dt) {
        case CS2D_F32: return launch_dt<CS2D_F32>(P, keep, st);
        case CS2D_F16: return launch_dt<CS2D_F16>(P, keep, st);
        default: return launch_dt<CS2D_BF16>(P, keep, st);
    }
}

}  // namespace cs2d
