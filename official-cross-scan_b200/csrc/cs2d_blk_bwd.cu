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
// a path of its own beside the shared-memory unit (measured: 1.3 to 1.6 cycles of an SM per 512-byte access of a warp, 4 through
// shared memory, each way) - and walks back over them with the adjoint.  What crosses a block to the left stays in registers; m of
// the block's first row goes to the row of blocks above through a scratch buffer, like the forward's h.
// Sums over the states (du, ddelta) are formed through tensor memory as well: a pixel's place takes its four sums' terms once h and
// q have been read from it, and a column's sixteen terms come back with the lanes (states) transposed against the columns of
// the memory; the sums over the warp's channels (dB, dC) are shuffles, added to global memory half a block at a time.
// All that a block reads from global memory travels while the block before it is walked: its inputs as they lie in memory (a row of
// eight columns per lane, asynchronously), B and C and the row of h above likewise, the column on its left into registers.
//
// What bounds it: instruction issue and fetch.  A block is some 4000 instructions per warp (128 per pixel, 37 of them packed fp32);
// measured on B200, straight-line code runs at one instruction per 1, 3 and 5.7 cycles of a scheduler where a loop takes up to 8, 32 and more KB
// of code, whatever the other warps do.  So the walks take two columns per iteration (a column: registers are copied to their places
// at the end of each, 19 instructions per pixel; four: 17 KB of code; 32x4x192x16x56x56 fp32 4150 / 3790 / 3970 us), everything else
// that can be is a loop over slots, and addresses that the compiler would make again for every use are held (bk_keep: 3790 -> 3640).
// With two states per thread in place of one the instructions fall to 99 but the body takes 16 KB (5400 us; a column per iteration: 4080).
// Before (sums through shared memory, inputs loaded into registers at the end of a block, 4 columns per iteration, a CTA barrier per
// block) and now: 3770 -> 3660; 128x4x384x16x28x28 bf16 8530 -> 7540, 2x4x192x16x200x336 bf16 6150 -> 5820, 32x4x192x4x56x56 bf16 2760 -> 2200,
// 3x4x51x7x45x61 fp16 228 -> 156.  What is asked of tensor memory is waited for in the same iteration, not across its end (no difference in time).
#include "cs2d_blk.cuh"

namespace cs2d {

// Tensor memory as this thread's own: floats at column `a`.
__device__ __forceinline__ void tm_st4(uint32_t a, float2 x, float2 y) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
}
// h left of, and q of, two pixels of a column
__device__ __forceinline__ void tm_ld8(uint32_t a, float2 (&x)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(x[0].x), "=f"(x[0].y), "=f"(x[1].x), "=f"(x[1].y), "=f"(x[2].x), "=f"(x[2].y), "=f"(x[3].x), "=f"(x[3].y) : "r"(a));
}
// 16 lanes by 16 columns: lane t gets, of columns 2(t%4), 2(t%4)+1 and of those eight further on, what lanes t/4 and t/4 + 8 of the 16 hold:
// x[0], x[1] of the first eight columns, x[2], x[3] of the others
__device__ __forceinline__ void tm_ld_t(uint32_t a, float2 (&x)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(x[0].x), "=f"(x[0].y), "=f"(x[1].x), "=f"(x[1].y), "=f"(x[2].x), "=f"(x[2].y), "=f"(x[3].x), "=f"(x[3].y) : "r"(a));
}
// the loaded values pass through the wait, so that nothing uses them before it
__device__ __forceinline__ void tm_wait_ld(float2 (&x)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(x[0].x), "+f"(x[0].y), "+f"(x[1].x), "+f"(x[1].y), "+f"(x[2].x), "+f"(x[2].y), "+f"(x[3].x), "+f"(x[3].y));
}
__device__ __forceinline__ void tm_wait_ld(float2 (&x)[4], float2 (&y)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(x[0].x), "+f"(x[0].y), "+f"(x[1].x), "+f"(x[1].y), "+f"(x[2].x), "+f"(x[2].y), "+f"(x[3].x), "+f"(x[3].y),
                   "+f"(y[0].x), "+f"(y[0].y), "+f"(y[1].x), "+f"(y[1].y), "+f"(y[2].x), "+f"(y[2].y), "+f"(y[3].x), "+f"(y[3].y));
}
__device__ __forceinline__ void tm_wait_ld(float2 (&h)[4], float2 (&x)[4], float2 (&y)[4]) {
    tm_wait_ld(x, y);
    asm volatile("" : "+f"(h[0].x), "+f"(h[0].y), "+f"(h[1].x), "+f"(h[1].y), "+f"(h[2].x), "+f"(h[2].y), "+f"(h[3].x), "+f"(h[3].y));
}
__device__ __forceinline__ float2 sel2(bool c, float2 a, float2 b) { return f2(c ? a.x : b.x, c ? a.y : b.y); }
// keep one of two values and add to it what the lane `off` away sends of its own
__device__ __forceinline__ float2 fold2(bool hi, float2 lo_v, float2 hi_v, int off) {
    const float2 k = sel2(hi, hi_v, lo_v), s = sel2(hi, lo_v, hi_v);
    return add2(k, f2(__shfl_xor_sync(0xffffffffu, s.x, off), __shfl_xor_sync(0xffffffffu, s.y, off)));
}
__device__ __forceinline__ float fold1(bool hi, float lo_v, float hi_v, int off) {
    return (hi ? hi_v : lo_v) + __shfl_xor_sync(0xffffffffu, hi ? lo_v : hi_v, off);
}

// a value that is to be held in a register, and not made again from its parts
__device__ __forceinline__ int bk_keep(int x) {
    asm volatile("" : "+r"(x));
    return x;
}

template <int NG>
struct BkBwd {   // a warp's shared memory
    static constexpr int SPW = 32 / NG, NP = 33;                  // slots per warp; pitch of a slot's pixels
    static constexpr int WARPS = NG == 16 ? 12 : 8;               // warps that share the registers of an SM, in CTAs of 4 or 8
    static constexpr int in = 0;                                  // float4 [SPW][NP] (dl, dl', dlu, dlu')
    static constexpr int us = in + SPW * NP * 16;                 // float4 [SPW][NP] (u, u', sigmoid, sigmoid')
    static constexpr int g = us + SPW * NP * 16;                  // float2 [SPW][NP] dout
    static constexpr int halo = g + SPW * NP * 8;                 // float2 [SPW][3][9] dl of the row above, the row below, the column left
    static constexpr int par = (halo + SPW * 27 * 8 + 15) & ~15;  // float4 [SPW] (delta_bias, delta_bias', D, D')
    static constexpr int mw = par + SPW * 16;                     // float2 [SPW] merge weights
    static constexpr int SP = 41;
    static constexpr int sum = mw + SPW * 8;                  // float4 [SPW][SP]: [4][10] sums over the states (S1, S1', S2, S2')
    static constexpr int bc = sum + SPW * SP * 16;                // float2 [32][NG] B, C of the block (see blk_bc_kernel)
    static constexpr int row = bc + BK_PX * NG * 8;               // float4 [4][32] the row of h above the block
    static constexpr int dbc = row + 4 * 32 * 16;                 // float [4 columns][DN][32] dB and dC of half a block (DN: rows, or pairs of them)
    static constexpr int DN = NG / 4;
    static constexpr int acc = dbc + 4 * DN * 32 * 4;             // float4 [SPW][32] sums of dout*u and ddelta over the lane's pixels
    // the next block's inputs as they lie in memory: rows of eight columns, of NC channels each: 4 of u, of delta, of dout, 2 (above and
    // below) of delta; and the words with delta of the column on the left
    static constexpr int NC = 2 * SPW;
    static constexpr int raw = acc + SPW * 32 * 16, ru = raw, rd = ru + NC * 128, rg = rd + NC * 128, rh = rg + NC * 128, rl = rh + NC * 64;
    static constexpr int total = rl + NC * 16;
    static constexpr int UC = 2;                                  // columns per iteration of the walks
    static constexpr int TM = BK_PX * 4;                          // columns of tensor memory
};

template <int V>
__device__ __forceinline__ void bk_cp(void *dst, const void *src, bool on) {
    if constexpr (V == 16)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(smem_addr(dst)), "l"(src), "r"((int)on) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p cp.async.ca.shared.global [%0], [%1], %3;\n\t}" ::"r"(smem_addr(dst)), "l"(src), "r"((int)on), "n"(V) : "memory");
}
__device__ __forceinline__ float2 bk_ld8(const float2 *p, bool on) {
    float2 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t@p ld.global.v2.f32 {%0,%1}, [%2];\n\t}"
                 : "=f"(v.x), "=f"(v.y) : "l"(p), "r"((int)on) : "memory");
    return v;
}
// EXTRA: the direction merge's dw, or dA_decay, is wanted.
template <int NG, int DT, bool EXTRA>
__global__ void __launch_bounds__(BkBwd<NG>::WARPS * 32, 1) blk_bwd_kernel(const __grid_constant__ Blk P) {
    using S = BkBwd<NG>;
    using T = typename bk_type<DT>::t;
    constexpr int SPW = S::SPW, NP = S::NP;
    extern __shared__ __align__(16) unsigned char smem_[];
    __shared__ uint32_t tm_base;
    __shared__ int sCount[BK_MAXRW];
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = bk_keep(threadIdx.x & 31);   // (known to be the same in the whole warp)
    unsigned char *sm = smem_ + bk_keep(warp * S::total);
    float4 *sS = reinterpret_cast<float4 *>(sm + S::sum);
    float2 *sBC = reinterpret_cast<float2 *>(sm + S::bc);
    float4 *sRow = reinterpret_cast<float4 *>(sm + S::row) + lane;
    float4 *sAcc = reinterpret_cast<float4 *>(sm + S::acc) + lane;
    float *sDBC = reinterpret_cast<float *>(sm + S::dbc) + lane;
    const int rw = 1 << P.rwl, w = warp & (rw - 1), nsub = P.warps >> P.rwl, stride = gridDim.x * nsub;
    RowSeq rs;
    rs.init(sCount, warp, rw, P.nstrip);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tm_base)), "r"(P.warps / 4 * S::TM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // this warp's columns of its lane quadrant: four per pixel, column by column: h of the pixel left of it, q; then the terms of the
    // sums over the states; then, in the first pixel's place, the column's dB and dC
    const uint32_t tm = __shfl_sync(0xffffffffu, tm_base, 0) + ((uint32_t)(warp & 3) << 21) + (warp >> 2) * S::TM;

    const int n = lane % NG, sl_ = lane / NG;              // this thread's state and slot of the warp
    const int lr = lane >> 3, lc = lane & 7;               // its pixel when staging and writing
    const int first = blockIdx.x * nsub + (warp >> P.rwl);   // this team's first item
    const bool softplus = P.softplus != 0, drep1 = P.drep == 1;
    const float2 lgd = bc(P.decay ? log2f(__ldg(P.decay)) : 0.f);
    const int64_t HW = (int64_t)P.H * P.W;
    auto blk_of = [&](const BkPos &q) { return P.nblk - 1 - q.row; };     // rows of blocks from the bottom up
    auto strip_of = [&](const BkPos &q) { return P.nstrip - 1 - q.strip; };   // and their blocks from the right

    // where this lane's share of the sums over the states goes: slot, row, which of the sums (of column 0)
    float *sSw = reinterpret_cast<float *>(sS) + bk_keep(NG == 16 ? ((lane >> 4) * S::SP + (((lane >> 2) & 2) + ((lane >> 1) & 1)) * 10) * 4 + 2 * (lane & 1) + ((lane >> 2) & 1)
                                                           : ((lane >> 3) * S::SP + (((lane >> 1) & 2) + ((lane >> 1) & 1)) * 10) * 4 + 2 * (lane & 1));
    constexpr int ES = DT == CS2D_F32 ? 4 : 2;
    const bool g32 = DT != CS2D_F32 && P.out_dt == CS2D_F32;   // 16-bit inputs with an fp32 gradient
    const int rp = DT != CS2D_F32 && P.vin == 2 ? 20 : 8 * ES;  // bytes between rows of the copied inputs
    // ---- asynchronous copies of a block's inputs, P.vin bytes at a time.  16-bit rows that start in the middle of a word (vin = 2) are
    // copied from that word on and keep their offset, of which there is a bit per row (a word that holds an element can be read) ----
    unsigned ou = 0, od = 0, og = 0, oh = 0, ol = 0;
    auto copy_raw = [&](const BkPos &q) {
        const int r0 = blk_of(q) * BK_R, c0 = strip_of(q) * BK_S, ch0 = q.slot * 2, cg = q.g * P.dpg + ch0, nch = P.dpg - ch0;
        const bool fw = (P.flip_w >> q.g) & 1u, fh = (P.flip_h >> q.g) & 1u;
        const int fc = fw ? P.W - BK_S - c0 : c0, lo = max(-fc, 0), hi = min(BK_S, P.W - fc);   // first column of the block in memory; those that exist
        auto image_row = [&](int r) { return fh ? P.H - 1 - r : r; };
        auto dch = [&](int k) { return (int64_t)(drep1 ? cg + k : (cg + k) / P.drep); };
        auto rows = [&](int dst, const char *p, int es, int v, bool on) {   // one row per lane; returns which of them start in the middle of a word
            unsigned odd = 0;
            if (v == 2) {
                const int o = (int)(reinterpret_cast<uintptr_t>(p) & 2);
                odd = __ballot_sync(0xffffffffu, o != 0);
#pragma unroll
                for (int i = 0; i < 5; ++i) bk_cp<4>(sm + dst + 4 * i, p - o + 4 * i, on && 4 * i + 4 > lo * 2 + o && 4 * i < hi * 2 + o);
            } else if (v == 4) {
#pragma unroll 4
                for (int i = 0; i < 8 * es; i += 4) bk_cp<4>(sm + dst + i, p + i, on && i >= lo * es && i < hi * es);
            } else if (v == 8) {
#pragma unroll
                for (int i = 0; i < 4; ++i) { if (8 * i < 8 * es) bk_cp<8>(sm + dst + 8 * i, p + 8 * i, on && 8 * i >= lo * es && 8 * i < hi * es); }
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i) { if (16 * i < 8 * es) bk_cp<16>(sm + dst + 16 * i, p + 16 * i, on && 16 * i >= lo * es && 16 * i < hi * es); }
            }
            return odd;
        };
        const int64_t ub = (int64_t)q.b * P.u_bs + (int64_t)((P.shared & 1) ? ch0 : cg) * P.u_ds + fc, gb = (int64_t)q.b * P.o_bs + (int64_t)((P.shared & 2) ? ch0 : cg) * P.o_ds + fc;
        const char *D = reinterpret_cast<const char *>(P.delta) + ((int64_t)q.b * P.dl_bs + fc) * ES, *U = reinterpret_cast<const char *>(P.u) + ub * ES;
        const char *Gp = reinterpret_cast<const char *>(P.out) + gb * (g32 ? 4 : ES);
        const int k = (lane >> 2) & (S::NC - 1), r = lane & 3, fr = image_row(r0 + r);
        const bool on = k < nch && r0 + r < P.H;
        const char *d = D + (dch(k) * P.dl_ds + (int64_t)fr * P.dl_hs) * ES, *u = U + ((int64_t)k * P.u_ds + (int64_t)fr * P.u_hs) * ES, *g = Gp + ((int64_t)k * P.o_ds + (int64_t)fr * P.o_hs) * (g32 ? 4 : ES);
        const int kh = (lane >> 1) & (S::NC - 1), rh = (lane & 1) ? r0 + BK_R : r0 - 1;   // the rows above and below
        const char *h = D + (dch(kh) * P.dl_ds + (int64_t)image_row(rh) * P.dl_hs) * ES;
        const bool onh = kh < nch && rh >= 0 && rh < P.H;
        if (S::NC == 8) {   // a row per lane
            od = rows(S::rd + lane * rp, d, ES, P.vin, on);
            ou = rows(S::ru + lane * rp, u, ES, P.vin, on);
            if (g32) rows(S::rg + lane * 32, g, 4, max(P.vin, 4), on);
            else og = rows(S::rg + lane * rp, g, ES, P.vin, on);
            oh = rows(S::rh + (lane & 15) * rp, h, ES, P.vin, onh && lane < 16);
        } else {            // half the lanes each
            const bool hi = lane & 16;
            const unsigned o = rows((hi ? S::rd : S::ru) + (lane & 15) * rp, hi ? d : u, ES, P.vin, on);
            ou = o & 0xffffu; od = o >> 16;
            if (g32) rows(S::rg + (lane & 15) * 32, g, 4, max(P.vin, 4), on && !hi);
            const unsigned o2 = rows(hi ? S::rh + (lane & 7) * rp : S::rg + (g32 ? 0 : (lane & 15) * rp), hi ? h : g, ES, P.vin, hi ? onh && !(lane & 8) : on && !g32);
            og = o2 & 0xffffu; oh = (o2 >> 16) & 0xffu;
        }
        // the column on the left: its word
        const uintptr_t l = reinterpret_cast<uintptr_t>(d + (fw ? BK_S : -1) * ES);
        ol = (unsigned)(l & 2);
        bk_cp<4>(sm + S::rl + (lane & (4 * S::NC - 1)) * 4, reinterpret_cast<const char *>(l & ~(uintptr_t)3), on && c0 > 0 && lane < 4 * S::NC);
    };
    // ---- transform and stage them: pixels and channels outside the image get zeros (a = 1 or the decay, p = 0, no adjoint) ----
    auto stage = [&](const BkPos &q) {
        const int nch = P.dpg - q.slot * 2, r0 = blk_of(q) * BK_R, c0 = strip_of(q) * BK_S;
        const bool fw = (P.flip_w >> q.g) & 1u;
        const bool pix = c0 + lc < P.W && r0 + lr < P.H;
        const int mc = (fw ? 7 - lc : lc);
        const float4 *sPar = reinterpret_cast<const float4 *>(sm + S::par);
        auto elem = [&](int base, int row, unsigned odd, bool on) {   // this lane's column of a row
            const unsigned char *p = sm + base + row * rp + mc * ES + (DT != CS2D_F32 ? ((odd >> row) & 1u) * 2 : 0);
            if constexpr (DT == CS2D_F32) return on ? *reinterpret_cast<const float *>(p) : 0.f;
            else return on ? bk_cvt<DT>(*reinterpret_cast<const uint16_t *>(p)) : 0.f;
        };
#pragma unroll 1
        for (int s = 0; s < SPW; ++s) {
            const float4 par = sPar[s];
            const bool k0 = pix && 2 * s < nch, k1 = pix && 2 * s + 1 < nch;
            const int row = 8 * s + lr;
            const float2 uv = f2(elem(S::ru, row, ou, k0), elem(S::ru, row + 4, ou, k1));
            float2 dl = f2(elem(S::rd, row, od, k0) + par.x, elem(S::rd, row + 4, od, k1) + par.y), sg = bc(1.f), gv;
            if (g32) {
                const float *p = reinterpret_cast<const float *>(sm + S::rg + row * 32) + mc;
                gv = f2(k0 ? p[0] : 0.f, k1 ? p[32] : 0.f);
            } else {
                gv = f2(elem(S::rg, row, og, k0), elem(S::rg, row + 4, og, k1));
            }
            if (softplus) dl = bk_softplus2<true>(dl, &sg);
            dl = f2(k0 ? dl.x : 0.f, k1 ? dl.y : 0.f);
            const float2 dlu = mul2(dl, uv);
            reinterpret_cast<float4 *>(sm + S::in)[s * NP + lane] = make_float4(dl.x, dl.y, dlu.x, dlu.y);
            reinterpret_cast<float4 *>(sm + S::us)[s * NP + lane] = make_float4(uv.x, uv.y, sg.x, sg.y);
            reinterpret_cast<float2 *>(sm + S::g)[s * NP + lane] = gv;
        }
        float *hf = reinterpret_cast<float *>(sm + S::halo);
#pragma unroll 1
        for (int i = 0; i <= S::NC / 4; ++i) {   // (rows and columns outside the image meet h = 0 or m = 0: any finite value will do)
            const bool left = i == S::NC / 4;
            const int k = left ? (lane >> 2) & (S::NC - 1) : lr + 4 * i;
            const float4 par = sPar[k >> 1];
            const float bv = (k & 1) ? par.y : par.x;
            float2 x;
            if (!left) {
                const bool okc = c0 + lc < P.W && k < nch;
                x = f2(elem(S::rh, 2 * k, oh, okc && r0 > 0), elem(S::rh, 2 * k + 1, oh, okc && r0 + BK_R < P.H));
            } else {
                const uint32_t v = *reinterpret_cast<const uint32_t *>(sm + S::rl + (lane & (4 * S::NC - 1)) * 4);
                const bool okl = c0 > 0 && k < nch && r0 + (lane & 3) < P.H;
                x = bc(okl ? bk_cvt<DT>(DT == CS2D_F32 ? v : ol ? v >> 16 : v & 0xffffu) : 0.f);
            }
            x = add2(x, bc(bv));
            if (softplus) x = bk_softplus2<false>(x, nullptr);
            float *h = hf + (k >> 1) * 54 + (k & 1);
            if (!left) { h[2 * lc] = x.x; h[18 + 2 * lc] = x.y; }
            else h[36 + 2 * (lane & 3)] = x.x;
        }
    };
    // ---- asynchronous copies for a block: B and C of four columns, and the row of h above them.  The places are free as soon as the walk
    // back has left those columns of the block before ----
    auto lane_of = [&](const BkPos &q) { return (uint32_t)(min(q.slot + sl_, P.nsl - 1) * P.NS + min(n, P.NS - 1)); };   // its place in the group's share of a checkpoint
    auto copy_half = [&](const BkPos &q, int k) {
        const int blk = blk_of(q);
        const unsigned char *src = reinterpret_cast<const unsigned char *>(P.bc + (((int64_t)q.bg * P.nblk + blk) * P.nstrip + strip_of(q)) * BK_PX * NG) + k * NG * 128 + lane * 16;
        unsigned char *dst = reinterpret_cast<unsigned char *>(sBC) + k * NG * 128 + lane * 16;
#pragma unroll
        for (int i = 0; i < NG / 4; ++i) bk_cp<16>(dst + 512 * i, src + 512 * i, true);
        if (blk > 0) {
            const float4 *row = P.row + (((int64_t)((blk - 1) * P.nstrip + strip_of(q)) * 4 + 2 * k) * P.NL + (int64_t)q.bg * P.nsl * P.NS) + lane_of(q);
            bk_cp<16>(sRow + 2 * k * 32, row, true); bk_cp<16>(sRow + (2 * k + 1) * 32, row + P.NL, true);
        } else {
            sRow[2 * k * 32] = sRow[(2 * k + 1) * 32] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    // what the forward left of the column on the left: q and s, and h of the row above it
    float4 colv[BK_R];
    float2 cnr;
    auto load_col = [&](const BkPos &q) {
        const bool left = strip_of(q) > 0, corner = left && blk_of(q) > 0;
        const int64_t lin = (int64_t)q.bg * P.nsl * P.NS + lane_of(q);
        const float4 *col = P.col + ((int64_t)blk_of(q) * (P.nstrip - 1) + strip_of(q) - 1) * 4 * P.NL + lin;
#pragma unroll
        for (int r = 0; r < BK_R; ++r) { colv[r] = bk_ld16<true>(col, left); col += P.NL; }
        cnr = bk_ld8(reinterpret_cast<const float2 *>(P.row + ((int64_t)((blk_of(q) - 1) * P.nstrip + strip_of(q)) * 4 - 1) * P.NL + lin) + 1, corner);
    };

    float2 A2 = bc(0.f), dA = bc(0.f), mcorner = bc(0.f), mwv = bc(1.f), dwa = bc(0.f), dec = bc(0.f);
    float2 e[BK_R], t[BK_R], ar[BK_R], mr[BK_R];               // column right of the block
#pragma unroll
    for (int s = 0; s < SPW; ++s) sAcc[s * 32] = make_float4(0.f, 0.f, 0.f, 0.f);

    BkPos pos;
    pos.start(P, SPW, first, w);
    if (pos.item < P.items) {
        copy_raw(pos); copy_half(pos, 0); copy_half(pos, 1);
        bk_commit();
        load_col(pos);
    }
    int item = -1;   // of the block before
    const float4 *tIn = reinterpret_cast<const float4 *>(sm + S::in) + sl_ * NP;
    const float2 *tBC = sBC + bk_keep(NG == 16 ? (n & 7) * 2 + (n >> 3) : n);
    const float2 *tH = reinterpret_cast<const float2 *>(sm + S::halo) + sl_ * 27;
    const float2 *tG = reinterpret_cast<const float2 *>(sm + S::g) + sl_ * NP;
#pragma unroll 1
    while (pos.item < P.items) {
        BkPos nxt = pos;
        const bool leave = nxt.next(P, SPW, rw, stride), non = nxt.item < P.items;   // leave: the worker is done with its item after this block
        const int blk = blk_of(pos), strip = strip_of(pos), r0 = blk * BK_R, c0 = strip * BK_S, G0 = pos.g, ngrp = (min(BK_S, P.W - c0) + S::UC - 1) / S::UC;   // ngrp: groups of columns that the image has
        const int ch0 = pos.slot * 2, cg = G0 * P.dpg + ch0, nch = P.dpg - ch0;
        if (pos.item != item) {
            item = pos.item;
            const int k0 = min(2 * sl_, nch - 1), k1 = min(2 * sl_ + 1, nch - 1);
            const float *a = P.A + (int64_t)cg * P.A_ds + n * P.A_ns;
            A2 = n < P.N ? f2(__ldg(a + k0 * P.A_ds) * LOG2E, __ldg(a + k1 * P.A_ds) * LOG2E) : bc(0.f);
            dA = bc(0.f);
            dwa = dec = bc(0.f);
            if (EXTRA) mwv = P.mw ? f2(__ldg(P.mw + cg + k0), __ldg(P.mw + cg + k1)) : bc(1.f);
            __syncwarp();   // the item before has left its parameters: two lanes read them last, for its sums
            if (lane < SPW) {
                const int k = 2 * lane;
                const bool o0 = k < nch, o1 = k + 1 < nch;
                reinterpret_cast<float4 *>(sm + S::par)[lane] = make_float4(P.bias && o0 ? __ldg(P.bias + (cg + k) / P.drep) : 0.f, P.bias && o1 ? __ldg(P.bias + (cg + k + 1) / P.drep) : 0.f,
                                                                            P.D && o0 ? __ldg(P.D + cg + k) : 0.f, P.D && o1 ? __ldg(P.D + cg + k + 1) : 0.f);
                reinterpret_cast<float2 *>(sm + S::mw)[lane] = f2(o0 && P.mw ? __ldg(P.mw + cg + k) : 1.f, o1 && P.mw ? __ldg(P.mw + cg + k + 1) : 1.f);
            }
        }
        bk_wait<0>();      // this block's copies
        __syncwarp();
        stage(pos);
        __syncwarp();
        if (non) { copy_raw(nxt); bk_commit(); }
        float2 hcur[BK_R];                 // h of the current column on the way back
        {
            // ---- recompute h and q of the block, a group of columns per iteration ----
            float2 hl[BK_R], al[BK_R], ql[BK_R], sl[BK_R], hc = cnr;
#pragma unroll
            for (int r = 0; r < BK_R; ++r) {
                ql[r] = f2(colv[r].x, colv[r].y); sl[r] = f2(colv[r].z, colv[r].w);
                hl[r] = add2(ql[r], sl[r]);
                al[r] = ex2_2(fma2(tH[18 + r], A2, lgd));   // (meets h = 0 at the image's edge)
            }
            float4 rin[2];           // two pixels ahead (past the block's last pixel: read, not used)
            float rb[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) { rin[i] = tIn[i * BK_S]; rb[i] = tBC[i * NG].x; }
#pragma unroll 1
            for (int k = 0; k < ngrp; ++k) {
                const float4 *kIn = tIn + S::UC * k;
                const float2 *kBC = tBC + 4 * S::UC * k * NG;
                const uint32_t tk = tm + 16 * S::UC * k;
                float4 up;
                float2 hd, hu, au;
#pragma unroll
                for (int j = 0; j < 4 * S::UC; ++j) {
                    const int r = j & 3;
                    const float4 in = rin[j & 1];
                    const float b = rb[j & 1];
                    rin[j & 1] = kIn[((j + 2) & 3) * BK_S + (j + 2) / 4]; rb[j & 1] = kBC[(j + 2) * NG].x;
                    if (j % 8 == 0) up = sRow[(S::UC / 2 * k + j / 8) * 32];
                    if (r == 0) { hd = hc; hu = hc = j & 4 ? f2(up.z, up.w) : f2(up.x, up.y); au = ex2_2(fma2(tH[S::UC * k + j / 4], A2, lgd)); }
                    const float2 a = ex2_2(fma2(f2(in.x, in.y), A2, lgd));
                    const float2 p = mul2(bc(b), f2(in.z, in.w));
                    const float2 z = add2(ql[r], fma2(mul2(add2(au, al[r]), hd), bc(-0.5f), hu));
                    const float2 s = fma2(a, sl[r], p);
                    const float2 q = mul2(a, z), h = fma2(a, z, s);
                    tm_st4(tk + 4 * j, hl[r], q);
                    hd = hl[r]; hu = h; au = a;
                    hl[r] = h; al[r] = a; ql[r] = q; sl[r] = s;
                }
            }
#pragma unroll
            for (int r = 0; r < BK_R; ++r) hcur[r] = hl[r];
        }
        if (non && ngrp * S::UC <= 4) { copy_half(nxt, 1); bk_commit(); }
        {
            const bool fh = (P.flip_h >> G0) & 1u, fw = (P.flip_w >> G0) & 1u;
            if (pos.strip == 0) {
                mcorner = bc(0.f);
#pragma unroll
                for (int r = 0; r < BK_R; ++r) e[r] = t[r] = ar[r] = mr[r] = bc(0.f);
            }
            tm_wait_st();
            // ---- walk back with the adjoint, a group of columns per iteration ----
            if (rw > 1 && !rs.wait(pos.seq)) { rs.abandon(P.status); break; }
            float4 *arow = P.adj + ((int64_t)first * P.nstrip + strip) * 4 * 32 + lane;   // m of the row below the block, two columns per float4
            constexpr int PR = S::UC / 2;   // pairs of columns
            float4 dnv[PR];
#pragma unroll
            for (int i = 0; i < PR; ++i) dnv[i] = bk_ld16<false>(arow + ((ngrp - 1) * PR + i) * 32, blk + 1 < P.nblk);
            float4 rin[BK_R];
            float2 rb[BK_R], rg[BK_R], hq[2][4];   // of two pixels each: hq[1] of rows 3 and 2
            // what two pixels of a column need
            auto load2 = [&](int c, int r) {
#pragma unroll
                for (int i = r; i > r - 2; --i) { rin[i] = tIn[i * BK_S + c]; rb[i] = tBC[(4 * c + i) * NG]; rg[i] = tG[i * BK_S + c]; }
                tm_ld8(tm + 16 * c + 4 * (r - 1), hq[r >> 1]);
            };
            // sums over the states of a column, from what tensor memory holds of it
            float2 x[4], y[4];
            auto ask_states = [&](int c) { tm_wait_st(); tm_ld_t(tm + 16 * c, x); tm_ld_t(tm + (16u << 16) + 16 * c, y); };
            auto sum_states = [&](int c) {
                const bool b2 = lane & 4, b3 = lane & 8, b4 = lane & 16;
                if constexpr (NG == 16) {   // x: slot 0, y: slot 1
                    const float2 v0 = fold2(b4, add2(x[0], x[1]), add2(y[0], y[1]), 16), v1 = fold2(b4, add2(x[2], x[3]), add2(y[2], y[3]), 16);
                    const float2 v = fold2(b3, v0, v1, 8);
                    sSw[c * 4] = fold1(b2, v.x, v.y, 4);
                } else {                    // x: slots 0 and 1, y: 2 and 3
                    const float2 v0 = fold2(b4, x[0], y[0], 16), v1 = fold2(b4, x[1], y[1], 16), v2 = fold2(b4, x[2], y[2], 16), v3 = fold2(b4, x[3], y[3], 16);
                    const float2 w0 = fold2(b3, v0, v1, 8), w1 = fold2(b3, v2, v3, 8);
                    *reinterpret_cast<float2 *>(sSw + c * 4) = fold2(b2, w0, w1, 4);
                }
            };
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = y[i] = bc(0.f);
            // dB (lower half of the lanes) or dC of the lane's state, of the first row that it writes
            const int frow = r0 + (NG == 16 ? 0 : (lane >> 3) & 1), rstep = fh ? -P.W : P.W;
            float *dbc = ((lane >> 4) ? P.dC : P.dB) + ((int64_t)pos.bg * P.N + n) * HW + (int64_t)(fh ? P.H - 1 - frow : frow) * P.W;
            float2 dAt = bc(0.f);   // of this block: sums of sums
            load2(S::UC * ngrp - 1, 3);
            tm_wait_ld(hq[1]);
#pragma unroll 1
            for (int k = ngrp - 1; k >= 0; --k) {
                float4 dn[PR], mb[PR], up;
#pragma unroll
                for (int i = 0; i < PR; ++i) dn[i] = dnv[i];
                if (k) {
#pragma unroll
                    for (int i = 0; i < PR; ++i) dnv[i] = bk_ld16<false>(arow + ((k - 1) * PR + i) * 32, blk + 1 < P.nblk);
                }
#pragma unroll
                for (int cc = S::UC - 1; cc >= 0; --cc) {
                    const int c = S::UC * k + cc;
                    if (cc & 1) up = sRow[(PR * k + cc / 2) * 32];
                    float2 md = cc & 1 ? f2(dn[cc / 2].z, dn[cc / 2].w) : f2(dn[cc / 2].x, dn[cc / 2].y), mdd = mcorner, ad = ex2_2(fma2(tH[9 + c], A2, lgd));
                    mcorner = md;
                    float dv[BK_R];
#pragma unroll
                    for (int r = BK_R - 1; r >= 0; --r) {
                        if (r == 3) {   // of the column two columns on: its terms have been asked for a column ago (at first: nothing, not used)
                            if (cc < S::UC - 1) tm_wait_ld(hq[1], x, y);
                            load2(c, 1);
                            sum_states(c + 2);
                        } else if (r == 1) {
                            tm_wait_ld(hq[0]);
                            load2(cc ? c - 1 : max(c - 1, 0), 3);   // (column 0 once more: not used)
                            ask_states(min(c + 1, 7));
                        }
                        const float4 in = rin[r];
                        const float2 B = bc(rb[r].x), C = bc(rb[r].y), gr = rg[r], gv = EXTRA ? mul2(gr, mwv) : gr;   // dout, times the merge weight
                        const float2 hlf = hq[r >> 1][2 * (r & 1)], q = hq[r >> 1][2 * (r & 1) + 1];
                        const float2 dl = f2(in.x, in.y), dlu = f2(in.z, in.w);
                        const float2 a = ex2_2(fma2(dl, A2, lgd));
                        const float2 p = mul2(B, dlu), gC = mul2(C, gv);
                        const float2 h = hcur[r], hup = r ? hcur[r ? r - 1 : 0] : (cc & 1 ? f2(up.z, up.w) : f2(up.x, up.y));
                        const float2 ev = fma2(ar[r], e[r], fma2(mul2(add2(ar[r], ad), mdd), bc(-0.5f), md));
                        const float2 tv = fma2(ar[r], t[r], gC);
                        const float2 m = mul2(a, add2(ev, tv));
                        const float2 X = fma2(md, hlf, mul2(mr[r], hup));
                        const float2 hp = fma2(p, bc(-1.f), h);
                        const float2 G = fma2(mul2(a, X), bc(-0.5f), fma2(ev, hp, mul2(tv, q)));
                        const float2 eps = fma2(gC, bc(0.25f), ev), yq = fma2(p, bc(0.25f), q);
                        const float2 dBv = mul2(dlu, eps), dCv = mul2(gv, yq);
                        dAt = fma2(dl, G, dAt);
                        if constexpr (EXTRA) {
                            dwa = fma2(mul2(C, yq), gr, dwa);
                            dec = add2(dec, fma2(tv, fma2(q, bc(-1.f), hp), G));
                        }
                        tm_st4(tm + 16 * c + 4 * r, mul2(B, eps), mul2(A2, G));
                        dv[r] = fold1(lane & 16, dBv.x + dBv.y, dCv.x + dCv.y, 16);   // dB in the lower half of the lanes, dC in the upper one
                        mdd = mr[r]; md = m; ad = a;
                        e[r] = ev; t[r] = tv; ar[r] = a; mr[r] = m;
                        hcur[r] = hlf;
                    }
                    if (cc & 1) { mb[cc / 2].z = md.x; mb[cc / 2].w = md.y; }
                    else { mb[cc / 2].x = md.x; mb[cc / 2].y = md.y; }
                    float *d = sDBC + (c & 3) * S::DN * 32;   // [column][row, or pair of rows with bit 3 of the lane the row of the pair]
                    if constexpr (NG == 16) {
#pragma unroll
                        for (int r = 0; r < BK_R; ++r) d[r * 32] = dv[r];
                    } else {
                        const bool b3 = lane & 8;
                        d[0] = fold1(b3, dv[0], dv[1], 8); d[32] = fold1(b3, dv[2], dv[3], 8);
                    }
                }
                tm_wait_ld(hq[1], x, y);   // nothing that has been asked for crosses a branch: its registers may be copied there
                if (blk > 0) {   // m of the block's first row
#pragma unroll
                    for (int i = 0; i < PR; ++i) arow[(k * PR + i) * 32] = mb[i];
                }
                if (S::UC * k & 3) continue;
                // half a block's dB and dC onto the results: four columns at a time where the rows allow it, else one
                const int cf = c0 + S::UC * k;
                if (P.vec_dbc) {
                    float *dst = dbc + (fw ? P.W - 4 - cf : cf);
                    const float *d = fw ? sDBC + 3 * S::DN * 32 : sDBC;
                    const int ds = fw ? -S::DN * 32 : S::DN * 32;
#pragma unroll
                    for (int i = 0; i < S::DN; ++i) {
                        bk_red16(dst, make_float4(d[i * 32], d[i * 32 + ds], d[i * 32 + 2 * ds], d[i * 32 + 3 * ds]), n < P.N && r0 + (NG == 16 ? i : 2 * i + ((lane >> 3) & 1)) < P.H);
                        dst += NG == 16 ? rstep : 2 * rstep;
                    }
                } else {
                    __syncwarp();
                    const int fcol = cf + (lane & 3);
#pragma unroll 1
                    for (int j = 0; j < 4; ++j) {   // eight lanes' sums at a time, a column per lane
                        const int l = 8 * j + (lane >> 2), st = l % NG, fr = r0 + (NG == 16 ? 0 : j & 1);
                        const float *d = reinterpret_cast<const float *>(sm + S::dbc) + (lane & 3) * S::DN * 32 + l;
                        float *dst = ((j >> 1) ? P.dC : P.dB) + ((int64_t)pos.bg * P.N + st) * HW + (int64_t)(fh ? P.H - 1 - fr : fr) * P.W + (fw ? P.W - 1 - fcol : fcol);
#pragma unroll
                        for (int i = 0; i < S::DN; ++i) {
                            bk_st<CS2D_F32, true>(dst, 0, d[i * 32], fr + (NG == 16 ? i : 2 * i) < P.H && st < P.N && fcol < P.W);
                            dst += NG == 16 ? rstep : 2 * rstep;
                        }
                    }
                }
                __syncwarp();
                if (non) { copy_half(nxt, S::UC * k >> 2); bk_commit(); }
            }
            dA = add2(dA, dAt);
            if (non) load_col(nxt);
            sum_states(1);
            ask_states(0);
            tm_wait_ld(x, y);
            sum_states(0);
            if (rw > 1) rs.done(pos.seq);
            __syncwarp();
            {   // du, ddelta: one pixel per lane, slot by slot
                const bool pix = c0 + lc < P.W && r0 + lr < P.H;
                const int fr = fh ? P.H - 1 - (r0 + lr) : r0 + lr, fc = fw ? P.W - 1 - (c0 + lc) : c0 + lc, b = pos.b;
                const int64_t pixo = (int64_t)fr * P.W + fc;
                const int64_t odu = ((int64_t)b * (P.mw ? P.dpg : P.dpg * P.G) + (P.mw ? ch0 : cg)) * HW + pixo, odd = ((int64_t)b * P.dpg * P.G + cg) * HW + pixo;
#pragma unroll 1
                for (int s = 0; s < SPW; ++s) {
                    const float4 S4 = sS[s * S::SP + lr * 10 + lc], us = reinterpret_cast<const float4 *>(sm + S::us)[s * NP + lane], in = reinterpret_cast<const float4 *>(sm + S::in)[s * NP + lane];
                    const float4 pr = reinterpret_cast<const float4 *>(sm + S::par)[s];
                    const float2 gr = reinterpret_cast<const float2 *>(sm + S::g)[s * NP + lane], gv = EXTRA ? mul2(gr, reinterpret_cast<const float2 *>(sm + S::mw)[s]) : gr;
                    const float2 u2 = f2(us.x, us.y), S1 = f2(S4.x, S4.y);
                    const float2 du = fma2(f2(pr.z, pr.w), gv, mul2(f2(in.x, in.y), S1));
                    const float2 dd = mul2(fma2(u2, S1, mul2(f2(S4.z, S4.w), bc(0.6931471805599453f))), f2(us.z, us.w));
                    const bool k0 = pix && 2 * s < nch, k1 = pix && 2 * s + 1 < nch;
                    const float4 ac = sAcc[s * 32];
                    const float2 sd = fma2(gr, u2, f2(ac.x, ac.y)), sb = add2(f2(ac.z, ac.w), f2(pix ? dd.x : 0.f, pix ? dd.y : 0.f));   // (no sums where columns were left out)
                    sAcc[s * 32] = make_float4(sd.x, sd.y, sb.x, sb.y);
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
            if (leave) {   // parameter gradients of the worker's share of the item
                const int k0 = 2 * sl_;
                const bool mine = pos.slot + sl_ < P.nsl, o0 = mine && k0 < nch, o1 = mine && k0 + 1 < nch;
                float *q = P.dA + (int64_t)(cg + k0) * P.N + n;
                bk_st<CS2D_F32, true>(q, 0, dA.x, o0 && n < P.N);
                bk_st<CS2D_F32, true>(q, P.N, dA.y, o1 && n < P.N);
                float2 dws = dwa;
                if constexpr (EXTRA) {
                    float dv = dec.x * (o0 ? 1.f : 0.f) + dec.y * (o1 ? 1.f : 0.f);
#pragma unroll
                    for (int off = 16; off; off >>= 1) dv += __shfl_xor_sync(0xffffffffu, dv, off);
                    if (P.ddecay && lane == 0) atomicAdd(P.ddecay, dv / __ldg(P.decay));
#pragma unroll
                    for (int off = NG / 2; off; off >>= 1) dws = add2(dws, shfl_xor2<32>(dws, off));
                    if (P.dw && n == 0) {
                        bk_st<CS2D_F32, true>(P.dw + cg + k0, 0, dws.x, o0);
                        bk_st<CS2D_F32, true>(P.dw + cg + k0 + 1, 0, dws.y, o1);
                    }
                }
#pragma unroll
                for (int s = 0; s < SPW; ++s) {   // dD, ddelta_bias
                    float4 v = sAcc[s * 32];
                    sAcc[s * 32] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int off = 16; off; off >>= 1) {
                        v.x += __shfl_xor_sync(0xffffffffu, v.x, off); v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
                        v.z += __shfl_xor_sync(0xffffffffu, v.z, off); v.w += __shfl_xor_sync(0xffffffffu, v.w, off);
                    }
                    const int x = lane & 1, k = 2 * s + x;
                    const float4 pr = reinterpret_cast<const float4 *>(sm + S::par)[s];
                    const float2 mw = reinterpret_cast<const float2 *>(sm + S::mw)[s];
                    if (lane < 2 && k < nch) {
                        const float gu = x ? v.y : v.x;      // sum of dout*u
                        if (P.dD) atomicAdd(P.dD + cg + k, gu * (x ? mw.y : mw.x));
                        if (EXTRA && P.dw) atomicAdd(P.dw + cg + k, gu * (x ? pr.w : pr.z));
                        if (P.dbias) atomicAdd(P.dbias + cg + k, x ? v.w : v.z);
                    }
                }
            }
        }
        pos = nxt;
    }
    bk_commit();
    bk_wait<0>();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(P.warps / 4 * S::TM));
}

template <int NG, int DT, bool EXTRA>
static cudaError_t launch(const Blk &P, cudaStream_t st) {
    auto kernel = blk_bwd_kernel<NG, DT, EXTRA>;
    constexpr int smem = BkBwd<NG>::total * BK_MAXRW;
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    kernel<<<P.grid, P.warps * 32, BkBwd<NG>::total * P.warps, st>>>(P);
    return cudaGetLastError();
}
template <int NG, int DT>
static cudaError_t launch_ex(const Blk &P, cudaStream_t st) {
    return P.mw || P.ddecay ? launch<NG, DT, true>(P, st) : launch<NG, DT, false>(P, st);
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
