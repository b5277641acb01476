// Block-walk forward (sm_100a); the decomposition is described in cs2d_blk.cuh.
//   q(r,c) = a*(q(r,c-1) + T),  T = h(r-1,c) - 0.5*(a(r-1,c) + a(r,c-1))*h(r-1,c-1)
//   s(r,c) = a*s(r,c-1) + p,    h = q + s,    y = D*u + sum_n C*(q + p/4)
// which is the reference's recurrence (include/cusoflex/selective_scan_fwd_kernel_oflex.cuh:214-338: h, the row scan
// s, y = C*(h - s + p/4)) carried as q = h - s, so that the difference y needs is never formed by subtraction.
#include "cs2d_blk.cuh"

namespace cs2d {

// B and C in the order the walk consumes them: [batch*G][nblk][nstrip][32 pixels, column by column][NG] (B, C), fp32, in
// scan coordinates; pixels outside the image and states past dstate are zero.  One 16-byte asynchronous copy per lane then
// fetches what two states of a pixel need, without address arithmetic or conversions in the walk.
template <int DT>
__global__ void blk_bc_kernel(const __grid_constant__ Blk P, int NG) {
    using T = typename bk_type<DT>::t;
    const int nt = P.nblk * P.nstrip, tile = blockIdx.x % nt, bg = blockIdx.x / nt, g = bg % P.G, b = bg / P.G;
    const int strip = tile % P.nstrip, blk = tile / P.nstrip;
    const bool fh = (P.flip_h >> g) & 1u, fw = (P.flip_w >> g) & 1u;
    const T *B = reinterpret_cast<const T *>(P.B) + (int64_t)b * P.B_bs + (int64_t)g * P.B_gs;
    const T *C = reinterpret_cast<const T *>(P.C) + (int64_t)b * P.C_bs + (int64_t)g * P.C_gs;
    float2 *dst = P.bc + ((int64_t)bg * P.nblk * P.nstrip + tile) * BK_PX * NG;
    __shared__ float2 sm[16][BK_PX + 1];
    for (int e = threadIdx.x; e < BK_PX * NG; e += blockDim.x) {   // read along rows
        const int px = e % BK_PX, n = e / BK_PX, r = blk * BK_R + px / BK_S, c = strip * BK_S + px % BK_S;
        const bool on = n < P.N && r < P.H && c < P.W;
        const int64_t o = (int64_t)(fw ? P.W - 1 - c : c);
        const int fr = fh ? P.H - 1 - r : r;
        const uint32_t bv = bk_ldp<DT>(B + (int64_t)n * P.B_ns + (int64_t)fr * P.B_hs + o, on), cv = bk_ldp<DT>(C + (int64_t)n * P.C_ns + (int64_t)fr * P.C_hs + o, on);
        sm[n][px] = f2(bk_cvt<DT>(bv), bk_cvt<DT>(cv));
    }
    __syncthreads();
    for (int e = threadIdx.x; e < BK_PX * NG; e += blockDim.x) {   // write in walk order
        const int n = e % NG, i = e / NG;
        dst[e] = sm[NG == 16 ? (n >> 1) + (n & 1) * 8 : n][(i % BK_R) * BK_S + i / BK_R];   // (states n and n + 8 side by side)
    }
}

template <int NG>
struct BkFwd {   // a warp's shared memory
    static constexpr int SPW = 32 / NG, YP = 34;                  // slots per warp; pitch of a pixel's sums
    static constexpr int in = 0;                                  // float4 [SPW][33] (dl, dl', dlu, dlu') of the two channels, row by row
    static constexpr int par = in + SPW * 33 * 16;                // float4 [SPW] (delta_bias, delta_bias', D, D')
    static constexpr int y = par + SPW * 16;                      // float2 [16][YP] half a block's C*(q + p/4) of every lane
    static constexpr int bc = y + 16 * YP * 8;                    // float2 [4][8][NG] B, C: ring of quarter blocks
    static constexpr int y0 = bc + 4 * 8 * NG * 8;                // float2 [SPW][33] D*u
    static constexpr int top = y0 + SPW * 33 * 8;                 // float2 [SPW][9]  dl of the row above
    static constexpr int total = (top + SPW * 9 * 8 + 15) & ~15;
};

template <int NG, int DT, bool KEEP>
__global__ void __launch_bounds__(BK_MAXRW * 32, 2) blk_fwd_kernel(const __grid_constant__ Blk P) {
    using S = BkFwd<NG>;
    using T = typename bk_type<DT>::t;
    constexpr int SPW = S::SPW, YP = S::YP, NCP = NG / 8;   // NCP: 16-byte copies per lane and quarter block
    extern __shared__ __align__(16) unsigned char smem_[];
    __shared__ int sCount[BK_MAXRW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char *sm = smem_ + warp * S::total;
    float4 *sIn = reinterpret_cast<float4 *>(sm + S::in), *sPar = reinterpret_cast<float4 *>(sm + S::par);
    float2 *sY = reinterpret_cast<float2 *>(sm + S::y), *sBC = reinterpret_cast<float2 *>(sm + S::bc);
    float2 *sY0 = reinterpret_cast<float2 *>(sm + S::y0), *sTop = reinterpret_cast<float2 *>(sm + S::top);
    const int rw = 1 << P.rwl, w = warp & (rw - 1), nsub = P.warps >> P.rwl, stride = gridDim.x * nsub;
    const int n = lane % NG, sl_ = lane / NG;              // this thread's state and slot of the warp
    const int lr = lane >> 3, lc = lane & 7;               // its pixel when staging
    const int first = blockIdx.x * nsub + (warp >> P.rwl);   // this team's first item
    const bool softplus = P.softplus != 0, drep1 = P.drep == 1;
    const float2 lgd = bc(P.decay ? log2f(__ldg(P.decay)) : 0.f);

    BkPos pos;
    pos.start(P, SPW, first, w);
    RowSeq rs;
    rs.init(sCount, warp, rw, P.nstrip);
    if (rw > 1) __syncthreads();

    // ---- loads of the next block: raw delta and u of the lane's pixel for every channel of the warp, delta of the row above ----
    uint32_t vd[2 * SPW], vu[2 * SPW], vt[SPW / 2];
    const T *pd = nullptr, *pu = nullptr, *pt = nullptr;   // at the first block of the row of blocks
    auto load_raw = [&](const BkPos &q) {
        const int r0 = q.row * BK_R, ch0 = q.slot * 2, cg = q.g * P.dpg + ch0;
        const bool fw = (P.flip_w >> q.g) & 1u;
        if (q.strip == 0) {
            const bool fh = (P.flip_h >> q.g) & 1u;
            const int b = q.bg / P.G, fr = fh ? P.H - 1 - (r0 + lr) : r0 + lr, fc = fw ? P.W - 1 - lc : lc;
            const T *db = reinterpret_cast<const T *>(P.delta) + (int64_t)b * P.dl_bs + fc;
            pd = db + (int64_t)fr * P.dl_hs + (int64_t)(cg / P.drep) * P.dl_ds;
            pt = db + (int64_t)(fh ? P.H - r0 : r0 - 1) * P.dl_hs + (drep1 ? (int64_t)(cg + lr) * P.dl_ds : 0);
            pu = reinterpret_cast<const T *>(P.u) + (int64_t)b * P.u_bs + (int64_t)((P.shared & 1) ? ch0 : cg) * P.u_ds + (int64_t)fr * P.u_hs + fc;
        }
        const int64_t cs = fw ? -q.strip * BK_S : q.strip * BK_S;
        const bool okc = q.strip * BK_S + lc < P.W, pix = okc && r0 + lr < P.H;
        const int nch = P.dpg - ch0;
        const T *qd = pd + cs, *qu = pu + cs;
        if (drep1) {
#pragma unroll
            for (int k = 0; k < 2 * SPW; ++k) {
                vd[k] = bk_ldp<DT>(qd, pix && k < nch);
                vu[k] = bk_ldp<DT>(qu, pix && k < nch);
                qd += P.dl_ds; qu += P.u_ds;
            }
#pragma unroll
            for (int i = 0; i < SPW / 2; ++i) vt[i] = bk_ldp<DT>(pt + cs + 4 * i * P.dl_ds, okc && r0 > 0 && lr + 4 * i < nch);
        } else {
#pragma unroll
            for (int k = 0; k < 2 * SPW; ++k) {
                vd[k] = bk_ldp<DT>(qd + (int64_t)((cg + k) / P.drep - cg / P.drep) * P.dl_ds, pix && k < nch);
                vu[k] = bk_ldp<DT>(qu, pix && k < nch);
                qu += P.u_ds;
            }
#pragma unroll
            for (int i = 0; i < SPW / 2; ++i)
                vt[i] = bk_ldp<DT>(pt + cs + (int64_t)((cg + lr + 4 * i) / P.drep) * P.dl_ds, okc && r0 > 0 && lr + 4 * i < nch);
        }
    };
    // quarter qt (two columns) of B and C of a block into its place in the ring
    auto copy_bc = [&](const unsigned char *src, int qt, bool on) {
        unsigned char *dst = reinterpret_cast<unsigned char *>(sBC + qt * 8 * NG) + lane * 16;
        src += qt * 64 * NG + lane * 16;
        if (on) {
#pragma unroll
            for (int i = 0; i < NCP; ++i) bk_cp16(dst + 512 * i, src + 512 * i);
        }
        bk_commit();
    };

    float2 A2 = bc(0.f), hcorner = bc(0.f);
    float2 hl[BK_R], al[BK_R], ql[BK_R], sl[BK_R];         // column left of the block
    float4 up0, up1;                                       // the row of h above: of the next quarter block and the one after it; hcorner: left of the current column
    up0 = up1 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < BK_R; ++r) { hl[r] = al[r] = ql[r] = sl[r] = bc(0.f); }
    int64_t oo = 0;
    // places of the block after the current one: B and C, the row of h it writes, the row of h above it, the column left of it
    const unsigned char *nbc = nullptr;
    float4 *nrow = nullptr, *ncol = nullptr;
    auto RL = [&]() -> int64_t { return KEEP ? P.NL : 32; };      // between the four parts of a block's row of h
    const int64_t up = KEEP ? (int64_t)P.nstrip * 4 * P.NL : 0;   // from a block's row of h back to the one above it
    auto place = [&](const BkPos &q) {   // at the start of a row of blocks
        const int blk = q.row;
        const int64_t lin = ((int64_t)q.bg * P.nsl + min(q.slot + sl_, P.nsl - 1)) * P.NS + min(n, P.NS - 1);
        nbc = reinterpret_cast<const unsigned char *>(P.bc + ((int64_t)q.bg * P.nblk + blk) * P.nstrip * BK_PX * NG);
        if constexpr (KEEP) nrow = P.row + (int64_t)blk * P.nstrip * 4 * P.NL + lin;
        else nrow = P.row + (int64_t)first * P.nstrip * 4 * 32 + lane;   // (an item's first row of blocks reads nothing)
        ncol = P.col + ((int64_t)blk * (P.nstrip - 1) - 1) * 4 * P.NL + lin;
    };
    auto above = [&](const float4 *row, int qt, bool there) { return bk_ld16<false>(row - up + qt * RL(), there); };   // a quarter of the row above the one at `row`
    // the first half of the row above of a row of blocks' first block; false: the wait for it ran out
    auto enter_row = [&](const BkPos &q) {
        if (rw > 1 && !rs.wait(q.seq)) return false;
        up0 = above(nrow, 0, q.row > 0); up1 = above(nrow, 1, q.row > 0);
        return true;
    };
    bool fresh = true, ok = true;   // the block is the first of its item; no wait has run out
    if (pos.item < P.items) {
        place(pos);
        load_raw(pos);
        copy_bc(nbc, 0, true); copy_bc(nbc, 1, true); copy_bc(nbc, 2, true);
        ok = enter_row(pos);
    }
    while (ok && pos.item < P.items) {
        BkPos nxt = pos;
        const bool leave = nxt.next(P, SPW, rw, stride), non = nxt.item < P.items;
        const int blk = pos.row, G0 = pos.g;
        const unsigned char *tbc = nbc;
        float4 *trow = nrow, *tcol = ncol;
        if (nxt.strip == 0) { if (non) place(nxt); }
        else { nbc += BK_PX * NG * 8; nrow += 4 * RL(); ncol += 4 * P.NL; }
        const bool mine = !KEEP || pos.slot + sl_ < P.nsl;   // (rolling: every lane has a place)
        {
            const int ch0 = pos.slot * 2, cg = G0 * P.dpg + ch0, nch = P.dpg - ch0, r0 = blk * BK_R;
            const bool pix = r0 + lr < P.H && pos.strip * BK_S + lc < P.W;
            if (pos.strip == 0) {
                const bool fh = (P.flip_h >> G0) & 1u, fw = (P.flip_w >> G0) & 1u;
                const int r = r0 + ((lane >> 2) & 3), c = lane & 3;
                oo = (int64_t)(pos.bg / P.G) * P.o_bs + (int64_t)((P.mw ? ch0 : cg) + 2 * (lane >> 4)) * P.o_ds +
                     (int64_t)(fh ? P.H - 1 - r : r) * P.o_hs + (fw ? P.W - 1 - c : c);
                if (fresh) {   // a new item
                    const int c0 = min(2 * sl_, nch - 1), c1 = min(2 * sl_ + 1, nch - 1);
                    const float *a = P.A + (int64_t)cg * P.A_ds + n * P.A_ns;
                    A2 = n < P.N ? f2(__ldg(a + c0 * P.A_ds) * LOG2E, __ldg(a + c1 * P.A_ds) * LOG2E) : bc(0.f);
                    if (lane < SPW) {
                        const int k = 2 * lane;
                        sPar[lane] = make_float4(P.bias && k < nch ? __ldg(P.bias + (cg + k) / P.drep) : 0.f, P.bias && k + 1 < nch ? __ldg(P.bias + (cg + k + 1) / P.drep) : 0.f,
                                                 P.D && k < nch ? __ldg(P.D + cg + k) : 0.f, P.D && k + 1 < nch ? __ldg(P.D + cg + k + 1) : 0.f);
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int r = 0; r < BK_R; ++r) { hl[r] = al[r] = ql[r] = sl[r] = bc(0.f); }
                hcorner = bc(0.f);
            } else if (KEEP) {   // q, s of the column left of the block
#pragma unroll
                for (int r = 0; r < BK_R; ++r) bk_st16(tcol + r * P.NL, make_float4(ql[r].x, ql[r].y, sl[r].x, sl[r].y), mine);
            }
            // ---- stage: pixels and channels outside the image get dl = 0 (a = 1 or the decay, p = 0) ----
#pragma unroll
            for (int i = 0; i < SPW; ++i) {
                const float4 par = sPar[i];
                const float2 uv = f2(bk_cvt<DT>(vu[2 * i]), bk_cvt<DT>(vu[2 * i + 1]));
                float2 dl = f2(bk_cvt<DT>(vd[2 * i]) + par.x, bk_cvt<DT>(vd[2 * i + 1]) + par.y);
                if (softplus) dl = bk_softplus2<false>(dl, nullptr);
                dl = f2(pix && 2 * i < nch ? dl.x : 0.f, pix && 2 * i + 1 < nch ? dl.y : 0.f);
                const float2 dlu = mul2(dl, uv);
                sIn[i * 33 + lane] = make_float4(dl.x, dl.y, dlu.x, dlu.y);
                sY0[i * 33 + lane] = mul2(uv, f2(par.z, par.w));
            }
#pragma unroll
            for (int i = 0; i < SPW / 2; ++i) {
                const int k = lr + 4 * i;
                const float4 par = sPar[k >> 1];
                float2 dl = bc(bk_cvt<DT>(vt[i]) + ((k & 1) ? par.y : par.x));
                if (softplus) dl = bk_softplus2<false>(dl, nullptr);
                reinterpret_cast<float *>(sTop)[((k >> 1) * 9 + lc) * 2 + (k & 1)] = dl.x;   // (columns outside the image meet h = 0)
            }
        }
        __syncwarp();
        if (non) load_raw(nxt);
        // Two columns - a quarter block - at a time; quarters that the image does not have are left out.  Software pipeline over
        // their pixels (column by column): the shared-memory loads of a pixel are issued two pixels ahead.  Only two quarters of the
        // row of h above are held (the whole of it, and instances that left out the right half of a row's last block, spilled 36
        // to 352 bytes): 32x4x192x16x56x56 fp32 forward 1355 -> 1218 us, 128x4x384x16x28x28 bf16 3057 -> 2480, and without a backward
        // 64x4x768x16x10x10 bf16 550 -> 446, 4x4x192x16x56x56 bf16 210 -> 192.  Not unrolled it is the slower one (1500 us; by halves
        // 1298), and so is a test per column (1394).
        const float4 *tIn = sIn + sl_ * 33;
        const float2 *tTop = sTop + sl_ * 9;
        const bool ahead = non && (rw == 1 || nxt.strip > 0);   // (with row workers the first block of a row is waited for when this one is done)
#pragma unroll
        for (int qt = 0; qt < 4; ++qt) {
            bk_wait<2>();
            __syncwarp();   // this quarter's B and C are here, the quarter before it has been read by all lanes
            copy_bc(qt == 0 ? tbc : nbc, (qt + 3) & 3, qt == 0 || non);
            // The row of h above travels two quarters ahead.  What a load reads was written two quarters ago by this thread, or by a worker
            // that has been waited for.
            if (qt == 2 && rw > 1 && ahead) ok = rs.wait(nxt.seq);
            const float4 hup = up0;
            up0 = up1;
            up1 = qt < 2 ? above(trow, qt + 2, blk > 0) : above(nrow, qt - 2, ahead && nxt.row > 0);
            if (pos.strip * BK_S + 2 * qt < P.W) {
                const float4 *qIn = tIn + qt * 2;
                const float2 *tBC = sBC + qt * 8 * NG + (NG == 16 ? (n & 7) * 2 + (n >> 3) : n);
                float2 *qY = sY + (qt & 1) * 2 * YP + lane;
                float4 rin[2];
                float2 rbc[2], hb[2];
                float2 hd, hu, au;
#pragma unroll
                for (int x = 0; x < 2; ++x) { rin[x] = qIn[x * BK_S]; rbc[x] = tBC[x * NG]; }
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const int c = x / 4, r = x % 4;
                    const float4 in = rin[x & 1];
                    const float2 b = rbc[x & 1];
                    if (x + 2 < 8) { rin[x & 1] = qIn[((x + 2) % 4) * BK_S + (x + 2) / 4]; rbc[x & 1] = tBC[(x + 2) * NG]; }
                    if (r == 0) { hd = hcorner; hu = hcorner = c ? f2(hup.z, hup.w) : f2(hup.x, hup.y); au = blk > 0 ? ex2_2(fma2(tTop[qt * 2 + c], A2, lgd)) : bc(0.f); }
                    const float2 a = ex2_2(fma2(f2(in.x, in.y), A2, lgd));
                    const float2 p = mul2(bc(b.x), f2(in.z, in.w));
                    const float2 t = mul2(add2(au, al[r]), hd);
                    const float2 z = add2(ql[r], fma2(t, bc(-0.5f), hu));
                    const float2 s = fma2(a, sl[r], p);
                    const float2 q = mul2(a, z), h = fma2(a, z, s);
                    qY[(r * 4 + c) * YP] = mul2(bc(b.y), fma2(p, bc(0.25f), q));
                    hd = hl[r]; hu = h; au = a;
                    hl[r] = h; al[r] = a; ql[r] = q; sl[r] = s;
                    if (r == BK_R - 1) hb[c] = h;
                }
                bk_st16(trow + qt * RL(), make_float4(hb[0].x, hb[0].y, hb[1].x, hb[1].y), mine && blk + 1 < P.nblk);   // the block's last row of h
            }   // (a pair that the image does not have leaves no row of h: the backward copies its place, whatever it holds, and does not use it)
            if (!(qt & 1)) continue;
            const int k = qt >> 1, c0 = pos.strip * BK_S + k * 4;
            if (c0 >= P.W) continue;
            __syncwarp();
            {   // sums over the states of half a block: a lane takes one pixel of every second slot
                const bool fw = (P.flip_w >> G0) & 1u;
                const int px = lane & 15, nch = P.dpg - pos.slot * 2 - 2 * (lane >> 4);
                const bool okp = blk * BK_R + (px >> 2) < P.H && c0 + (px & 3) < P.W;
                const int64_t o = oo + (fw ? -c0 : c0);
#pragma unroll
                for (int i = 0; i < SPW / 2; ++i) {
                    const int s2 = (lane >> 4) + 2 * i;
                    const float4 *yp = reinterpret_cast<const float4 *>(sY + px * YP + s2 * NG);
                    float2 v = sY0[s2 * 33 + (px >> 2) * BK_S + k * 4 + (px & 3)], v2 = bc(0.f);
#pragma unroll
                    for (int m = 0; m < NG / 2; ++m) {
                        const float4 t = yp[m];
                        v = add2(v, f2(t.x, t.y)); v2 = add2(v2, f2(t.z, t.w));
                    }
                    v = add2(v, v2);
                    const int64_t oi = o + (int64_t)(4 * i) * P.o_ds;
                    const bool ok0 = okp && 4 * i < nch, ok1 = okp && 4 * i + 1 < nch;
                    if (P.mw) {
                        const float *m = P.mw + G0 * P.dpg + pos.slot * 2 + 2 * s2;
                        bk_st<CS2D_F32, true>(P.out, oi, ok0 ? v.x * __ldg(m) : 0.f, ok0);
                        bk_st<CS2D_F32, true>(P.out, oi + P.o_ds, ok1 ? v.y * __ldg(m + 1) : 0.f, ok1);
                    } else if (P.out_dt == CS2D_F32) {
                        bk_st<CS2D_F32, false>(P.out, oi, v.x, ok0);
                        bk_st<CS2D_F32, false>(P.out, oi + P.o_ds, v.y, ok1);
                    } else {
                        bk_st<DT, false>(P.out, oi, v.x, ok0);
                        bk_st<DT, false>(P.out, oi + P.o_ds, v.y, ok1);
                    }
                }
            }
            __syncwarp();
        }
        if (rw > 1) {
            rs.done(pos.seq);
            if (non && nxt.strip == 0) ok = enter_row(nxt);
        }
        pos = nxt;
        fresh = leave;
    }
    if (!ok) rs.abandon(P.status);
    bk_wait<0>();
}

template <int NG, int DT, bool KEEP>
static cudaError_t launch(const Blk &P, cudaStream_t st) {
    auto kernel = blk_fwd_kernel<NG, DT, KEEP>;
    constexpr int smem = BkFwd<NG>::total * BK_MAXRW;
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    blk_bc_kernel<DT><<<P.nblk * P.nstrip * (P.items / P.ntile), 128, 0, st>>>(P, NG);
    kernel<<<P.grid, P.warps * 32, BkFwd<NG>::total * P.warps, st>>>(P);
    return cudaGetLastError();
}
template <int NG, int DT>
static cudaError_t launch_keep(const Blk &P, cudaStream_t st) { return P.roll ? launch<NG, DT, false>(P, st) : launch<NG, DT, true>(P, st); }
template <int NG>
static cudaError_t launch_dt(const Blk &P, cudaStream_t st) {
    switch (P.io_dt) {
        case CS2D_F32: return launch_keep<NG, CS2D_F32>(P, st);
        case CS2D_F16: return launch_keep<NG, CS2D_F16>(P, st);
        default: return launch_keep<NG, CS2D_BF16>(P, st);
    }
}

cudaError_t launch_blk_fwd(const Blk &P, int NG, cudaStream_t st) {
    switch (NG) {
        case 16: return launch_dt<16>(P, st);
        case 8: return launch_dt<8>(P, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace cs2d
