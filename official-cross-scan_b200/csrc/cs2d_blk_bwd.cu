// Block-walk backward (sm_100a); the decomposition is described in cs2d_blk.cuh, the gradients at the top of cs2d_bwd.cu.
// With q = h - s (see the forward), e = dh + ds and t = -ds the adjoint of the reference's recurrences
// (include/cusoflex/selective_scan_bwd_kernel_oflex.cuh:383-476, :689-724) reads
//   e(r,c) = m(r+1,c) + a(r,c+1)*e(r,c+1) - 0.5*(a(r,c+1) + a(r+1,c))*m(r+1,c+1)
//   t(r,c) = a(r,c+1)*t(r,c+1) + g*C,     m = a*(e + t)
//   G      = e*(h - p) + t*q - 0.5*a*(m(r+1,c)*h(r,c-1) + m(r,c+1)*h(r-1,c))      [= a * dLoss/da]
// so that neither difference (h - s, dh + ds) is formed by subtraction.
//
// A thread owns two channels (packed) and one state.  Blocks are walked bottom-up and right to left.  For each block the
// thread recomputes h and q from the column left of the block and the row above it, both written by the forward, keeps
// them in TENSOR MEMORY - 4 columns of its warp's lane quadrant per pixel: 256 KB per SM that nothing else uses here, with
// a path of its own beside the shared-memory unit that bounds the kernel (measured: 1.3 to 1.6 cycles of an SM per
// 512-byte access of a warp, 4 through shared memory, each way) - and walks back over them with the adjoint.
// What crosses a block to the left stays in registers; m of the block's first row goes to the row of blocks above through
// a scratch buffer, like the forward's h.
// Sums over the states (du, ddelta) and over the warp's channels (dB, dC) go through shared memory column by column; dB and dC
// are then added to global memory with reductions, half a block at a time.
#include "cs2d_blk.cuh"

namespace cs2d {

// Tensor memory as this thread's own: pairs of floats at column `a`.
__device__ __forceinline__ void tm_st(uint32_t a, float2 x) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(a), "f"(x.x), "f"(x.y) : "memory");
}
__device__ __forceinline__ void tm_ld(uint32_t a, float2 (&x)[2]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=f"(x[0].x), "=f"(x[0].y), "=f"(x[1].x), "=f"(x[1].y) : "r"(a) : "memory");
}
// the loaded values pass through the wait, so that nothing uses them before it
__device__ __forceinline__ void tm_wait_ld(float2 (&x)[2]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(x[0].x), "+f"(x[0].y), "+f"(x[1].x), "+f"(x[1].y)::"memory");
}

template <int NG>
struct BkBwd {   // a warp's shared memory
    static constexpr int SPW = 32 / NG, NP = 33;                  // slots per warp; pitch of a slot's pixels
    static constexpr int CTAS = NG == 16 ? 3 : 2;                 // CTAs per SM
    static constexpr int in = 0;                                  // float4 [SPW][NP] (dl, dl', dlu, dlu')
    static constexpr int us = in + SPW * NP * 16;                 // float4 [SPW][NP] (u, u', sigmoid, sigmoid')
    static constexpr int sum = us + SPW * NP * 16;                // float4 [SPW][4][10] sums over the states (S1, S1', S2, S2')
    static constexpr int par = sum + SPW * 40 * 16;               // float4 [SPW] (delta_bias, delta_bias', D, D')
    static constexpr int part = par + SPW * 16;                   // float4 [4][NP] a column's (S1, S1', S2, S2') of every lane
    static constexpr int partd = part + 4 * NP * 16;              // float2 [4][40] a column's (dB, dC) of every lane, summed over its channels
    static constexpr int bc = partd + 4 * 40 * 8;                 // float2 [32][NG] B, C of the block (see blk_bc_kernel)
    static constexpr int dbc = bc + BK_PX * NG * 8;               // float [4 rows][NG][2][4 columns] half a block's dB, dC; a row's pitch is DR
    static constexpr int DR = NG * 8 + 4;
    static constexpr int g = dbc + 4 * DR * 4;  // float2 [SPW][NP] dout
    static constexpr int halo = g + SPW * NP * 8;                 // float2 [SPW][3][9] dl of the row above, the row below, the column left
    static constexpr int mw = halo + SPW * 27 * 8;                // float2 [SPW] merge weights
    static constexpr int total = (mw + SPW * 8 + 15) & ~15;
};

// EXTRA: the direction merge's dw, or dA_decay, is wanted.  HALF: the last block of a row has its left half only, whose right
// half is left out (a 28-wide map: an eighth of the work; kept out of the other instances, which have no register to spare).
template <int NG, int DT, bool EXTRA, bool HALF>
__global__ void __launch_bounds__(BK_WARPS * 32, BkBwd<NG>::CTAS) blk_bwd_kernel(const __grid_constant__ Blk P) {
    using S = BkBwd<NG>;
    using T = typename bk_type<DT>::t;
    constexpr int SPW = S::SPW, NP = S::NP;
    extern __shared__ __align__(16) unsigned char smem_[];
    __shared__ uint32_t tm_base;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (known to be the same in the whole warp)
    unsigned char *sm = smem_ + warp * S::total;
    float4 *sIn = reinterpret_cast<float4 *>(sm + S::in), *sUS = reinterpret_cast<float4 *>(sm + S::us), *sS = reinterpret_cast<float4 *>(sm + S::sum);
    float4 *sPar = reinterpret_cast<float4 *>(sm + S::par), *sPart = reinterpret_cast<float4 *>(sm + S::part);
    float2 *sPartD = reinterpret_cast<float2 *>(sm + S::partd), *sBC = reinterpret_cast<float2 *>(sm + S::bc);
    float2 *sMw = reinterpret_cast<float2 *>(sm + S::mw), *sHalo = reinterpret_cast<float2 *>(sm + S::halo);
    float *sD = reinterpret_cast<float *>(sm + S::dbc);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tm_base)), "r"(128) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tm = __shfl_sync(0xffffffffu, tm_base, 0) + ((uint32_t)warp << 21);   // this warp's lane quadrant; columns 4i..4i+3: h of the pixel left of pixel i, q of pixel i

    const int rw = 1 << P.rwl, w = warp & (rw - 1), nsub = BK_WARPS >> P.rwl, stride = gridDim.x * nsub;
    const int n = lane % NG, sl_ = lane / NG;              // this thread's state and slot of the warp
    const int lr = lane >> 3, lc = lane & 7;               // its pixel when staging and writing
    const int first = blockIdx.x * nsub, lmax = (P.items - first + stride - 1) / stride * P.npass * P.period;
    const int steps = lmax + BK_LAG * (rw - 1);
    const bool softplus = P.softplus != 0, drep1 = P.drep == 1;
    const float2 lgd = bc(P.decay ? log2f(__ldg(P.decay)) : 0.f);

    BkPos pos;
    pos.item = first + (warp >> P.rwl); pos.pass = pos.strip = 0;
    pos.decode(P, SPW);
    auto blk_of = [&](const BkPos &q) { return P.nblk - 1 - (q.pass * rw + w); };     // rows of blocks from the bottom up
    auto live = [&](const BkPos &q, int L) { return L >= 0 && L < lmax && q.item < P.items && q.strip < P.nstrip && q.pass * rw + w < P.nblk; };

    // B and C of four columns of a block: the places are free as soon as the walk back has left those columns of the block before
    auto copy_bc = [&](const BkPos &q, int k) {
        const unsigned char *src = reinterpret_cast<const unsigned char *>(P.bc + (((int64_t)q.bg * P.nblk + blk_of(q)) * P.nstrip + (P.nstrip - 1 - q.strip)) * BK_PX * NG) + k * NG * 128 + lane * 16;
        unsigned char *dst = reinterpret_cast<unsigned char *>(sBC) + k * NG * 128 + lane * 16;
#pragma unroll
        for (int i = 0; i < NG / 4; ++i) bk_cp16(dst + 512 * i, src + 512 * i);
    };

    float2 A2 = bc(0.f), dA = bc(0.f), mcorner = bc(0.f), mwv = bc(1.f), dwa = bc(0.f), dec = bc(0.f);
    float2 e[BK_R], t[BK_R], ar[BK_R], mr[BK_R];               // column right of the block
    float2 accD[SPW], accB[SPW];                               // sums of dout*u and ddelta over the lane's pixels
#pragma unroll
    for (int i = 0; i < SPW; ++i) accD[i] = accB[i] = bc(0.f);
#pragma unroll
    for (int r = 0; r < BK_R; ++r) e[r] = t[r] = ar[r] = mr[r] = bc(0.f);
    // ---- raw delta, u, dout of the lane's pixel for the warp's channels; delta of the rows above and below (column lc, channels
    // lr, lr + 4, ..) and of the column on the left (row lane & 3, channel lane >> 2) ----
    constexpr int NC = 2 * SPW, NH = NC / 4;
    uint32_t vd[NC], vu[NC], vg[NC], vt[NH], vb[NH], vl;
    const bool g32 = DT != CS2D_F32 && P.out_dt == CS2D_F32;   // 16-bit inputs with an fp32 gradient
    const T *pd = nullptr, *pu = nullptr, *pt = nullptr, *pb = nullptr, *pl = nullptr;   // of column 0 of a row of blocks (pl: column -1)
    int64_t pg = 0;
    int nchq = 0;
    auto load_raw = [&](const BkPos &q) {
        const int r0 = blk_of(q) * BK_R, c0 = (P.nstrip - 1 - q.strip) * BK_S, cg = q.g * P.dpg + q.slot * 2;
        const bool fw = (P.flip_w >> q.g) & 1u;
        const int kl = lane >> 2, rl = r0 + (lane & 3);
        if (q.strip == 0) {   // a new row of blocks
            const int ch0 = q.slot * 2, b = q.bg / P.G;
            const bool fh = (P.flip_h >> q.g) & 1u;
            const int fr = fh ? P.H - 1 - (r0 + lr) : r0 + lr, fc = fw ? P.W - 1 - lc : lc;
            nchq = P.dpg - ch0;
            const T *db = reinterpret_cast<const T *>(P.delta) + (int64_t)b * P.dl_bs;
            pd = db + (int64_t)fr * P.dl_hs + fc + (int64_t)(drep1 ? cg : 0) * P.dl_ds;
            pt = db + (int64_t)(fh ? P.H - r0 : r0 - 1) * P.dl_hs + fc + (int64_t)(drep1 ? cg + lr : 0) * P.dl_ds;
            pb = db + (int64_t)(fh ? P.H - 1 - BK_R - r0 : r0 + BK_R) * P.dl_hs + fc + (int64_t)(drep1 ? cg + lr : 0) * P.dl_ds;
            pl = db + (int64_t)(fh ? P.H - 1 - rl : rl) * P.dl_hs + (fw ? P.W : -1) + (int64_t)((cg + kl) / P.drep) * P.dl_ds;
            pu = reinterpret_cast<const T *>(P.u) + (int64_t)b * P.u_bs + (int64_t)((P.shared & 1) ? ch0 : cg) * P.u_ds + (int64_t)fr * P.u_hs + fc;
            pg = (int64_t)b * P.o_bs + (int64_t)((P.shared & 2) ? ch0 : cg) * P.o_ds + (int64_t)fr * P.o_hs + fc;
        }
        const bool okc = c0 + lc < P.W, pix = okc && r0 + lr < P.H;
        const bool tok = okc && r0 > 0, bok = okc && r0 + BK_R < P.H, lok = c0 > 0 && rl < P.H;
        const int64_t cs = fw ? -c0 : c0;
        if (g32) {
            const uint32_t *p = reinterpret_cast<const uint32_t *>(P.out) + pg + cs;
#pragma unroll
            for (int k = 0; k < NC; ++k) { vg[k] = bk_ldp<CS2D_F32>(p, pix && k < nchq); p += P.o_ds; }
        } else {
            const T *p = reinterpret_cast<const T *>(P.out) + pg + cs;
#pragma unroll
            for (int k = 0; k < NC; ++k) { vg[k] = bk_ldp<DT>(p, pix && k < nchq); p += P.o_ds; }
        }
        const T *qu = pu + cs, *qd = pd + cs;
#pragma unroll
        for (int k = 0; k < NC; ++k) { vu[k] = bk_ldp<DT>(qu, pix && k < nchq); qu += P.u_ds; }
        if (drep1) {
#pragma unroll
            for (int k = 0; k < NC; ++k) { vd[k] = bk_ldp<DT>(qd, pix && k < nchq); qd += P.dl_ds; }
#pragma unroll
            for (int i = 0; i < NH; ++i) {
                vt[i] = bk_ldp<DT>(pt + cs + 4 * i * P.dl_ds, tok && lr + 4 * i < nchq);
                vb[i] = bk_ldp<DT>(pb + cs + 4 * i * P.dl_ds, bok && lr + 4 * i < nchq);
            }
        } else {
#pragma unroll
            for (int k = 0; k < NC; ++k) vd[k] = bk_ldp<DT>(qd + (int64_t)((cg + k) / P.drep) * P.dl_ds, pix && k < nchq);
#pragma unroll
            for (int i = 0; i < NH; ++i) {
                const int64_t o = (int64_t)((cg + lr + 4 * i) / P.drep) * P.dl_ds + cs;
                vt[i] = bk_ldp<DT>(pt + o, tok && lr + 4 * i < nchq);
                vb[i] = bk_ldp<DT>(pb + o, bok && lr + 4 * i < nchq);
            }
        }
        vl = bk_ldp<DT>(pl + cs, lok && kl < NC && kl < nchq);
    };
    // what the forward left for a block: the row of h above (half a block at a time), q and s of the column on the left
    const float4 *row = nullptr, *col = nullptr;
    float4 *arow = nullptr;                // m of the row below the block, two columns per float4
    bool row_on = false;
    float4 rowv[2], colv[BK_R], cnr;
    auto fetch_row = [&](int k) {   // of half k of the block
        rowv[0] = bk_ld16<true>(row + 2 * k * P.NL, row_on);
        rowv[1] = bk_ld16<true>(row + (2 * k + 1) * P.NL, row_on);
    };
    auto adj_at = [&](int strip) { return P.adj + ((int64_t)(first + (warp >> P.rwl)) * P.nstrip + strip) * 4 * 32 + lane; };
    auto fetch = [&](const BkPos &q) {
        const int blk = blk_of(q), strip = P.nstrip - 1 - q.strip;
        if (q.strip == 0) {
            const int64_t lin = ((int64_t)q.bg * P.nsl + min(q.slot + sl_, P.nsl - 1)) * P.NS + min(n, P.NS - 1);
            row = P.row + ((int64_t)((blk - 1) * P.nstrip + strip) * 4) * P.NL + lin;
            col = P.col + ((int64_t)blk * (P.nstrip - 1) + strip - 1) * 4 * P.NL + lin;
            if (NG == 8) arow = adj_at(strip);
        } else {
            row -= 4 * P.NL; col -= 4 * P.NL;
            if (NG == 8) arow -= 4 * 32;
        }
        row_on = blk > 0;
        fetch_row(0);
        cnr = bk_ld16<true>(row - P.NL, row_on && strip > 0);
#pragma unroll
        for (int r = 0; r < BK_R; ++r) colv[r] = bk_ld16<true>(col + r * P.NL, strip > 0);
    };
    auto enter = [&](const BkPos &q) {   // the first block after a pause
        copy_bc(q, 0); copy_bc(q, 1);
        load_raw(q);
    };
    if (w == 0 && live(pos, 0)) enter(pos);
    for (int g = 0; g < steps; ++g) {
        const int L = g - BK_LAG * w;
        BkPos nxt = pos;
        if (L >= 0) nxt.next(P, SPW, stride);
        const bool non = live(nxt, L + 1);
        if (!live(pos, L)) {   // before the worker's first block, past its last row of blocks, or past its items
            if (non) enter(nxt);
            if (rw > 1) __syncthreads();
            pos = nxt;
            continue;
        }
        const int blk = blk_of(pos), strip = P.nstrip - 1 - pos.strip, r0 = blk * BK_R, c0 = strip * BK_S, G0 = pos.g;
        const int ch0 = pos.slot * 2, cg = G0 * P.dpg + ch0, nch = P.dpg - ch0, b = pos.bg / P.G;
        const bool fh = (P.flip_h >> G0) & 1u, fw = (P.flip_w >> G0) & 1u;
        const bool mine = pos.slot + sl_ < P.nsl;
        const int nhalf = !HALF || c0 + 4 < P.W ? 2 : 1;   // halves of the block that the image has
        if (pos.pass == 0 && pos.strip == 0) {   // a new item
            const int k0 = min(2 * sl_, nch - 1), k1 = min(2 * sl_ + 1, nch - 1);
            const float *a = P.A + (int64_t)cg * P.A_ds + n * P.A_ns;
            A2 = n < P.N ? f2(__ldg(a + k0 * P.A_ds) * LOG2E, __ldg(a + k1 * P.A_ds) * LOG2E) : bc(0.f);
            dA = bc(0.f);
            dwa = dec = bc(0.f);
            mwv = P.mw ? f2(__ldg(P.mw + cg + k0), __ldg(P.mw + cg + k1)) : bc(1.f);
            for (int i = lane; i < SPW; i += 32) {
                const int k = 2 * i;
                const bool o0 = k < nch, o1 = k + 1 < nch;
                sPar[i] = make_float4(P.bias && o0 ? __ldg(P.bias + (cg + k) / P.drep) : 0.f, P.bias && o1 ? __ldg(P.bias + (cg + k + 1) / P.drep) : 0.f,
                                      P.D && o0 ? __ldg(P.D + cg + k) : 0.f, P.D && o1 ? __ldg(P.D + cg + k + 1) : 0.f);
                sMw[i] = f2(o0 && P.mw ? __ldg(P.mw + cg + k) : 1.f, o1 && P.mw ? __ldg(P.mw + cg + k + 1) : 1.f);
            }
            __syncwarp();
        }
        if (pos.strip == 0) {
            mcorner = bc(0.f);
#pragma unroll
            for (int r = 0; r < BK_R; ++r) e[r] = t[r] = ar[r] = mr[r] = bc(0.f);
        }
        fetch(pos);
        const bool pix = c0 + lc < P.W && r0 + lr < P.H;
        const int fr = fh ? P.H - 1 - (r0 + lr) : r0 + lr, fc = fw ? P.W - 1 - (c0 + lc) : c0 + lc;
        float2 hcur[BK_R];                 // h of the current column on the way back
        // ---- transform and stage: pixels and channels outside the image get zeros (a = 1 or the decay, p = 0, no adjoint) ----
#pragma unroll
        for (int i = 0; i < SPW; ++i) {
            const int s = i;
            const float4 par = sPar[s];
            const float2 uv = f2(bk_cvt<DT>(vu[2 * i]), bk_cvt<DT>(vu[2 * i + 1]));
            float2 dl = f2(bk_cvt<DT>(vd[2 * i]) + par.x, bk_cvt<DT>(vd[2 * i + 1]) + par.y), sg = bc(1.f);
            if (softplus) dl = bk_softplus2<true>(dl, &sg);
            const bool k0 = pix && 2 * s < nch, k1 = pix && 2 * s + 1 < nch;
            dl = f2(k0 ? dl.x : 0.f, k1 ? dl.y : 0.f);
            const float2 dlu = mul2(dl, uv);
            const float2 gv = f2(g32 ? __uint_as_float(vg[2 * i]) : bk_cvt<DT>(vg[2 * i]), g32 ? __uint_as_float(vg[2 * i + 1]) : bk_cvt<DT>(vg[2 * i + 1]));
            sIn[s * NP + lane] = make_float4(dl.x, dl.y, dlu.x, dlu.y);
            sUS[s * NP + lane] = make_float4(uv.x, uv.y, sg.x, sg.y);
            reinterpret_cast<float2 *>(sm + S::g)[s * NP + lane] = gv;
        }
        float *hf = reinterpret_cast<float *>(sHalo);
#pragma unroll
        for (int i = 0; i < NH; ++i) {
            const int k = lr + 4 * i;
            const float4 par = sPar[k >> 1];
            const float bv = (k & 1) ? par.y : par.x;
            float2 x = f2(bk_cvt<DT>(vt[i]) + bv, bk_cvt<DT>(vb[i]) + bv);
            if (softplus) x = bk_softplus2<false>(x, nullptr);
            hf[((k >> 1) * 27 + lc) * 2 + (k & 1)] = x.x;
            hf[((k >> 1) * 27 + 9 + lc) * 2 + (k & 1)] = x.y;
        }
        if (NC == 8 || lane < 4 * NC) {
            const int k = lane >> 2;
            const float4 par = sPar[k >> 1];
            float2 x = bc(bk_cvt<DT>(vl) + ((k & 1) ? par.y : par.x));
            if (softplus) x = bk_softplus2<false>(x, nullptr);
            hf[((k >> 1) * 27 + 18 + (lane & 3)) * 2 + (k & 1)] = x.x;
        }
        bk_commit();
        bk_wait<0>();      // this block's B and C
        __syncwarp();
        const float4 *tIn = sIn + sl_ * NP;
        const float2 *tBC = sBC + (NG == 16 ? (n & 7) * 2 + (n >> 3) : n);
        const float2 *tH = sHalo + sl_ * 27;
        // ---- recompute h and q of the block, half a block per iteration ----
        {
            float2 hl[BK_R], al[BK_R], ql[BK_R], sl[BK_R], hc = f2(cnr.z, cnr.w);
#pragma unroll
            for (int r = 0; r < BK_R; ++r) {
                ql[r] = f2(colv[r].x, colv[r].y); sl[r] = f2(colv[r].z, colv[r].w);
                hl[r] = add2(ql[r], sl[r]);
                al[r] = ex2_2(fma2(tH[18 + r], A2, lgd));   // (meets h = 0 at the image's edge)
                tm_st(tm + 4 * r, hl[r]);
            }
            float4 rin[2];           // two pixels ahead (past the block's last pixel: read, not used)
            float2 rb[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) { rin[i] = tIn[i * BK_S]; rb[i] = tBC[i * NG]; }
#pragma unroll 1
            for (int k = 0; k < nhalf; ++k) {
                const float2 up[4] = {f2(rowv[0].x, rowv[0].y), f2(rowv[0].z, rowv[0].w), f2(rowv[1].x, rowv[1].y), f2(rowv[1].z, rowv[1].w)};
                if (nhalf == 2) fetch_row(1);
                const float4 *kIn = tIn + 4 * k;
                const float2 *kBC = tBC + 16 * k * NG;
                const uint32_t tk = tm + 64 * k;
                float2 hd, hu, au;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int r = j & 3;
                    const float4 in = rin[j & 1];
                    const float b = rb[j & 1].x;
                    rin[j & 1] = kIn[((j + 2) & 3) * BK_S + (j + 2) / 4]; rb[j & 1] = kBC[(j + 2) * NG];
                    if (r == 0) { hd = hc; hu = hc = up[j / 4]; au = ex2_2(fma2(tH[4 * k + j / 4], A2, lgd)); }
                    const float2 a = ex2_2(fma2(f2(in.x, in.y), A2, lgd));
                    const float2 p = mul2(bc(b), f2(in.z, in.w));
                    const float2 z = add2(ql[r], fma2(mul2(add2(au, al[r]), hd), bc(-0.5f), hu));
                    const float2 s = fma2(a, sl[r], p);
                    const float2 q = mul2(a, z), h = fma2(a, z, s);
                    hd = hl[r]; hu = h; au = a;
                    hl[r] = h; al[r] = a; ql[r] = q; sl[r] = s;
                    if (j < 12 || k == 0) tm_st(tk + 4 * (j + BK_R), h);   // (the last column stays in registers)
                    tm_st(tk + 4 * j + 2, q);
                }
            }
#pragma unroll
            for (int r = 0; r < BK_R; ++r) hcur[r] = hl[r];
        }
        tm_wait_st();
        // ---- walk back with the adjoint, half a block per iteration ----
        if (NG == 16) arow = adj_at(strip);   // (three CTAs per SM have no register to keep it; 32x4x192x16x56x56 fp32 3850 -> 3760 us)
        float4 adjv[2];
        auto fetch_adj = [&](int k) {
            const bool there = blk + 1 < P.nblk;
            adjv[0] = bk_ld16<false>(arow + 2 * k * 32, there);
            adjv[1] = bk_ld16<false>(arow + (2 * k + 1) * 32, there);
        };
        fetch_adj(nhalf - 1);
        if (non && nhalf == 1) copy_bc(nxt, 1);
        const float2 *tG = reinterpret_cast<const float2 *>(sm + S::g) + sl_ * NP;
        float2 dAt = bc(0.f);
        const int64_t HW = (int64_t)P.H * P.W;
        float *dbc_row = (((lane >> 2) & 1) ? P.dC : P.dB) + ((int64_t)pos.bg * P.N + (lane >> 3)) * HW + (int64_t)(fh ? P.H - 1 - (r0 + (lane & 3)) : r0 + (lane & 3)) * P.W;
        float4 rin[2];
        float2 rb[2], rg[2], rhq[2][2];
        // what pixel 16k + j (j may be -1: the half on the left) needs, into set j & 1
        auto load = [&](int k, int j) {
            const int o = j & 1, r = j & 3, cc = j < 0 ? -1 : j / 4;
            rin[o] = tIn[r * BK_S + 4 * k + cc];
            rb[o] = tBC[(16 * k + j) * NG];
            rg[o] = tG[r * BK_S + 4 * k + cc];
            tm_ld(tm + 64 * k + 4 * j, rhq[o]);
        };
        load(nhalf - 1, 15);
#pragma unroll 1
        for (int k = nhalf - 1; k >= 0; --k) {
            const float2 up[4] = {f2(rowv[0].x, rowv[0].y), f2(rowv[0].z, rowv[0].w), f2(rowv[1].x, rowv[1].y), f2(rowv[1].z, rowv[1].w)};
            const float2 dn[4] = {f2(adjv[0].x, adjv[0].y), f2(adjv[0].z, adjv[0].w), f2(adjv[1].x, adjv[1].y), f2(adjv[1].z, adjv[1].w)};
            if (k) { fetch_row(0); fetch_adj(0); }
            float2 mb[4];
#pragma unroll
            for (int cc = 3; cc >= 0; --cc) {
                float2 md = dn[cc], mdd = mcorner, ad = ex2_2(fma2(tH[9 + 4 * k + cc], A2, lgd));
                mcorner = md;
#pragma unroll
                for (int r = BK_R - 1; r >= 0; --r) {
                    const int j = cc * 4 + r, o = j & 1;
                    tm_wait_ld(rhq[o]);
                    const float4 in = rin[o];
                    const float2 B = bc(rb[o].x), C = bc(rb[o].y), gr = rg[o], gv = EXTRA ? mul2(gr, mwv) : gr;   // dout, times the merge weight
                    const float2 hlf = rhq[o][0], q = rhq[o][1];
                    if (j > 0 || k > 0) load(k, j - 1);
                    const float2 dl = f2(in.x, in.y), dlu = f2(in.z, in.w);
                    const float2 a = ex2_2(fma2(dl, A2, lgd));
                    const float2 p = mul2(B, dlu), gC = mul2(C, gv);
                    const float2 h = hcur[r], hup = r ? hcur[r ? r - 1 : 0] : up[cc];
                    const float2 w1 = mul2(add2(ar[r], ad), mdd);
                    const float2 ev = fma2(ar[r], e[r], fma2(w1, bc(-0.5f), md));
                    const float2 tv = fma2(ar[r], t[r], gC);
                    const float2 m = mul2(a, add2(ev, tv));
                    const float2 X = fma2(md, hlf, mul2(mr[r], hup));
                    const float2 hp = fma2(p, bc(-1.f), h);
                    const float2 G = fma2(mul2(a, X), bc(-0.5f), fma2(ev, hp, mul2(tv, q)));
                    const float2 eps = fma2(gC, bc(0.25f), ev), yq = fma2(p, bc(0.25f), q);
                    const float2 S1 = mul2(B, eps), S2 = mul2(A2, G), dBv = mul2(dlu, eps), dCv = mul2(gv, yq);
                    dAt = fma2(dl, G, dAt);
                    if constexpr (EXTRA) {
                        dwa = fma2(mul2(C, yq), gr, dwa);
                        dec = add2(dec, fma2(tv, fma2(q, bc(-1.f), hp), G));
                    }
                    sPart[r * NP + lane] = make_float4(S1.x, S1.y, S2.x, S2.y);
                    sPartD[r * 40 + lane] = f2(dBv.x + dBv.y, dCv.x + dCv.y);
                    mdd = mr[r]; md = m; ad = a;
                    e[r] = ev; t[r] = tv; ar[r] = a; mr[r] = m;
                    if (r == 0) mb[cc] = m;
                    hcur[r] = hlf;
                }
                __syncwarp();
                // sums over the states: four lanes share a slot's row r, and are left with one of its four sums each
#pragma unroll
                for (int s0 = 0; s0 < SPW; s0 += 2) {
                    const int r = lane & 3, s = s0 + ((lane >> 3) & 1), part = ((lane >> 2) & 1) + 2 * (lane >> 4);   // a quarter of the slot's states
                    float2 x = bc(0.f), y = bc(0.f);
#pragma unroll
                    for (int i = 0; i < NG / 4; ++i) {
                        const float4 v = sPart[r * NP + s * NG + part * (NG / 4) + i];
                        x = add2(x, f2(v.x, v.y)); y = add2(y, f2(v.z, v.w));
                    }
                    const bool hi = lane & 16, hi2 = lane & 4;
                    float2 kk = hi ? y : x, ss = hi ? x : y;
                    kk.x += __shfl_xor_sync(0xffffffffu, ss.x, 16); kk.y += __shfl_xor_sync(0xffffffffu, ss.y, 16);
                    float v = hi2 ? kk.y : kk.x;
                    v += __shfl_xor_sync(0xffffffffu, hi2 ? kk.x : kk.y, 4);
                    reinterpret_cast<float *>(sS)[(s * 40 + r * 10 + 4 * k + cc) * 4 + (hi ? 2 : 0) + (hi2 ? 1 : 0)] = v;
                }
                // sums over the slots: rows and states over the lanes
#pragma unroll
                for (int i = 0; i < NG / 8; ++i) {
                    const int r = lane >> 3, st = (lane & 7) + 8 * i;
                    float2 x = sPartD[r * 40 + st];
#pragma unroll
                    for (int s = 1; s < SPW; ++s) x = add2(x, sPartD[r * 40 + s * NG + st]);
                    sD[r * S::DR + st * 8 + cc] = x.x; sD[r * S::DR + st * 8 + 4 + cc] = x.y;
                }
                __syncwarp();
            }
            if (blk > 0) {   // m of the block's first row (lanes past the last slot write the zeros that they read above)
                arow[2 * k * 32] = make_float4(mb[0].x, mb[0].y, mb[1].x, mb[1].y);
                arow[(2 * k + 1) * 32] = make_float4(mb[2].x, mb[2].y, mb[3].x, mb[3].y);
            }
            if (non) copy_bc(nxt, k);
            // half a block's dB and dC onto the results: four columns at a time where the rows allow it, else one
            if (P.vec_dbc) {
                const int frow = r0 + (lane & 3), kind = (lane >> 2) & 1;
                const bool okd = frow < P.H && c0 + 4 * k < P.W;
                float *dst = dbc_row + (fw ? P.W - 4 - (c0 + 4 * k) : c0 + 4 * k);
#pragma unroll
                for (int i = 0; i < NG / 4; ++i) {
                    const int st = (lane >> 3) + 4 * i;
                    float4 v = *reinterpret_cast<const float4 *>(sD + (lane & 3) * S::DR + st * 8 + kind * 4);
                    if (fw) v = make_float4(v.w, v.z, v.y, v.x);
                    bk_red16(dst + (int64_t)(4 * i) * HW, v, okd && st < P.N);
                }
            } else {
                const int fcol = c0 + 4 * k + (lane & 3), frow = r0 + ((lane >> 2) & 3), kind = lane >> 4;
                float *dst = (kind ? P.dC : P.dB) + (int64_t)pos.bg * P.N * HW + (int64_t)(fh ? P.H - 1 - frow : frow) * P.W + (fw ? P.W - 1 - fcol : fcol);
                const float *src = sD + ((lane >> 2) & 3) * S::DR + kind * 4 + (lane & 3);
#pragma unroll 4
                for (int i = 0; i < P.N; ++i) { bk_st<CS2D_F32, true>(dst, 0, src[i * 8], frow < P.H && fcol < P.W); dst += HW; }
            }
            __syncwarp();
        }
        // ---- the block is done; the next one's data travels while its results are written ----
        if (non) load_raw(nxt);
        dA = add2(dA, dAt);
        {   // du, ddelta: one pixel per lane, slot by slot
            const int64_t pixo = (int64_t)fr * P.W + fc;
            const int64_t odu = ((int64_t)b * (P.mw ? P.dpg : P.dpg * P.G) + (P.mw ? ch0 : cg)) * HW + pixo, odd = ((int64_t)b * P.dpg * P.G + cg) * HW + pixo;
#pragma unroll
            for (int s = 0; s < SPW; ++s) {
                const float4 S = sS[s * 40 + lr * 10 + lc], us = sUS[s * NP + lane], in = sIn[s * NP + lane], par = sPar[s];
                const float2 gr = reinterpret_cast<const float2 *>(sm + S::g)[s * NP + lane], gv = EXTRA ? mul2(gr, sMw[s]) : gr;
                const float2 u2 = f2(us.x, us.y), S1 = f2(S.x, S.y);
                const float2 du = fma2(f2(par.z, par.w), gv, mul2(f2(in.x, in.y), S1));
                const float2 dd = mul2(fma2(u2, S1, mul2(f2(S.z, S.w), bc(0.6931471805599453f))), f2(us.z, us.w));
                const bool k0 = pix && 2 * s < nch, k1 = pix && 2 * s + 1 < nch;
                accD[s] = fma2(gr, u2, accD[s]); accB[s] = add2(accB[s], HALF ? f2(pix ? dd.x : 0.f, pix ? dd.y : 0.f) : dd);   // (no sums where a half was left out)
                const int64_t ch = (int64_t)(2 * s) * HW;
                if (P.mw) {
                    bk_st<CS2D_F32, true>(P.du, odu + ch, du.x, k0);
                    bk_st<CS2D_F32, true>(P.du, odu + ch + HW, du.y, k1);
                } else {
                    bk_st<DT, false>(P.du, odu + ch, du.x, k0);
                    bk_st<DT, false>(P.du, odu + ch + HW, du.y, k1);
                }
                bk_st<DT, false>(P.ddelta, odd + ch, dd.x, k0);
                bk_st<DT, false>(P.ddelta, odd + ch + HW, dd.y, k1);
            }
        }
        __syncwarp();
        if (pos.strip == P.nstrip - 1 && blk - rw < 0) {   // the worker leaves the item: parameter gradients of its share
            const int k0 = 2 * sl_;
            const bool o0 = mine && k0 < nch, o1 = mine && k0 + 1 < nch;
            float *q = P.dA + (int64_t)(cg + k0) * P.N + n;
            bk_st<CS2D_F32, true>(q, 0, dA.x, o0 && n < P.N);
            bk_st<CS2D_F32, true>(q, P.N, dA.y, o1 && n < P.N);
            dA = bc(0.f);
            float2 dws = dwa;
            if constexpr (EXTRA) {
                float dv = dec.x * (o0 ? 1.f : 0.f) + dec.y * (o1 ? 1.f : 0.f);
#pragma unroll
                for (int off = 16; off; off >>= 1) dv += __shfl_xor_sync(0xffffffffu, dv, off);
                if (P.ddecay && lane == 0) atomicAdd(P.ddecay, dv / __ldg(P.decay));
#pragma unroll
                for (int off = NG / 2; off; off >>= 1) dws = add2(dws, shfl_xor2<32>(dws, off));
                dwa = dec = bc(0.f);
                if (P.dw && n == 0) {
                    bk_st<CS2D_F32, true>(P.dw + cg + k0, 0, dws.x, o0);
                    bk_st<CS2D_F32, true>(P.dw + cg + k0 + 1, 0, dws.y, o1);
                }
            }
            
#pragma unroll
            for (int s = 0; s < SPW; ++s) {   // dD, ddelta_bias
                float4 v = make_float4(accD[s].x, accD[s].y, accB[s].x, accB[s].y);
                accD[s] = accB[s] = bc(0.f);
#pragma unroll
                for (int off = 16; off; off >>= 1) {
                    v.x += __shfl_xor_sync(0xffffffffu, v.x, off); v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
                    v.z += __shfl_xor_sync(0xffffffffu, v.z, off); v.w += __shfl_xor_sync(0xffffffffu, v.w, off);
                }
                const int x = lane & 1, k = 2 * s + x;
                if (lane < 2 && k < nch) {
                    const float gu = x ? v.y : v.x;      // sum of dout*u
                    if (P.dD) atomicAdd(P.dD + cg + k, gu * (x ? sMw[s].y : sMw[s].x));
                    if (EXTRA && P.dw) atomicAdd(P.dw + cg + k, gu * (x ? sPar[s].w : sPar[s].z));
                    if (P.dbias) atomicAdd(P.dbias + cg + k, x ? v.w : v.z);
                }
            }
        }
        if (rw > 1) __syncthreads();   // the rows of m written in this step are there for the other workers
        pos = nxt;
    }
    bk_commit();
    bk_wait<0>();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(128));
}

template <int NG, int DT, bool EXTRA, bool HALF>
static cudaError_t launch(const Blk &P, cudaStream_t st) {
    auto kernel = blk_bwd_kernel<NG, DT, EXTRA, HALF>;
    constexpr int smem = BkBwd<NG>::total * BK_WARPS;
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    kernel<<<P.grid, BK_WARPS * 32, smem, st>>>(P);
    return cudaGetLastError();
}
template <int NG, int DT>
static cudaError_t launch_ex(const Blk &P, cudaStream_t st) {
    const bool half = ((P.W - 1) & 7) < 4;   // columns in the last block: at most 4
    if (P.mw || P.ddecay) return half ? launch<NG, DT, true, true>(P, st) : launch<NG, DT, true, false>(P, st);
    return half ? launch<NG, DT, false, true>(P, st) : launch<NG, DT, false, false>(P, st);
}
template <int NG>
static cudaError_t launch_dt(const Blk &P, cudaStream_t st) {
    switch (P.io_dt) {
        case CS2D_F32: return launch_ex<NG, CS2D_F32>(P, st);
        case CS2D_F16: return launch_ex<NG, CS2D_F16>(P, st);
        default: return launch_ex<NG, CS2D_BF16>(P, st);
    }
}
cudaError_t launch_blk_bwd(const Blk &P, int NG, cudaStream_t st) { return NG == 16 ? launch_dt<16>(P, st) : launch_dt<8>(P, st); }

}  // namespace cs2d
