// Block-walk kernels (sm_100a): what the forward (cs2d_blk_fwd.cu) and the backward (cs2d_blk_bwd.cu) share.
//
// A thread owns the recurrences of two channels - the halves of packed fp32x2 registers - for one state, and walks
// the image in blocks of 4 rows by 8 columns: along a block column by column, the four rows of a column one after the
// other, then on to the next block of the row of blocks, then to the next row of blocks.  Nothing is exchanged
// between threads to solve the recurrence: no scan over lanes, no second pass, no skew to fill and drain.  What
// crosses a block goes through registers (along the row: h, q, s, a of the last column) or through one row of h per
// row of blocks (down: written as float4, 512 consecutive bytes per warp, read back by the block below).
//
// A warp is self-contained: its lanes are the NG states of 32/NG slots (a slot is a channel pair), it loads, transforms
// (softplus) and stages delta and u of its own slots in shared memory, sums over the states (forward: through shared memory,
// backward: through tensor memory) and writes the results.  Neighbouring lanes share delta and u (measured on B200: a
// 128-bit shared load takes 2 cycles of the SM's load unit when neighbouring lanes share their address, 4 otherwise, whatever
// else is broadcast).  That unit bounds the forward, with 16 warps per SM; the backward, with 8 to 12, is bound by the issue
// and fetch of instructions.  The walks have no CTA barriers.
//
// Images with few recurrences run with 2, 4 or 8 row WORKERS (warps of one CTA): the rows of blocks of a team's items are one
// sequence, and worker w takes every RW-th of them.  A block needs the row of h (backward: of m) that the row before it in the
// sequence left for the same columns, so a worker follows its predecessor a block behind: every worker counts its finished
// blocks in shared memory, and waits for the count of the worker before it (RowSeq).
#pragma once

#include "cs2d_common.cuh"

namespace cs2d {

constexpr int BK_R = 4, BK_S = 8, BK_PX = BK_R * BK_S;   // a block: rows, columns, pixels
constexpr int BK_WARPS = 4;                               // warps per CTA (8 with 8 row workers)
constexpr int BK_MAXRW = 8;                               // row workers per CTA
static_assert(BK_R == RB, "row blocks and checkpoint cadence agree with the other kernels");

struct Blk {
    int H, W, N, G, dpg, drep, io_dt, out_dt, softplus;
    int nblk, nstrip;       // rows of blocks, blocks per row
    int rwl;                // log2 of the row workers per CTA
    int nsl;                // slots per group
    int ntile, items;       // warps' worth of slots per group; work items = batch * G * ntile
    int grid, warps;        // CTAs, warps of a CTA
    int *status;            // device status word (see ERR_*)
    unsigned flip_h, flip_w;
    int shared;             // bit 0: u has dpg channels shared by the groups, bit 1: dout
    int roll;               // forward: one rolling row of h instead of the checkpoints
    int NS;                 // places of a slot in the checkpoints (see below)
    int64_t NL;             // batch * G * nsl * NS
    const void *u, *delta, *B, *C;
    const float *A, *D, *bias, *decay;
    int64_t u_bs, u_ds, u_hs, dl_bs, dl_ds, dl_hs, A_ds, A_ns;
    int64_t B_bs, B_gs, B_ns, B_hs, C_bs, C_gs, C_ns, C_hs;
    void *out; int64_t o_bs, o_ds, o_hs;    // forward: out; backward: dout
    const float *mw; float *dw;             // direction merge (see Dev)
    // Checkpoints, threads innermost so that a warp moves whole lines.  A slot has NS places: of up to four states one each
    // and one for all lanes past them, which hold the same values (B = C = 0); 8 or 16 otherwise.  Lane n uses place min(n, NS - 1).
    //   row [nblk-1][nstrip][4][NL] float4 = h of the block's last row, two columns per float4
    //       (rolling: [teams][nstrip][4][32], one row per warp, or per team of row workers, that is on the GPU at a time)
    //   col [nblk][nstrip-1][4][NL] float4 = (q, s) of the column left of block strip+1, one row per float4
    float4 *row, *col;
    float2 *bc;                             // B and C in walk order (blk_bc_kernel)
    // backward
    float4 *adj;                            // [teams][nstrip][4][32]: the adjoint row m between rows of blocks
    void *du, *ddelta;
    float *dA, *dB, *dC, *dD, *dbias, *ddecay;
    int vin;                                // bytes of u, delta and dout that are copied at once: 16, 8, 4 or 2
    int vec_dbc;                            // dB, dC: rows of whole aligned groups of four columns
};

// stores to tensor memory have been made
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 16-byte asynchronous copies to shared memory, in groups
__device__ __forceinline__ void bk_cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void bk_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bk_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Position in a worker's stream of blocks: the rows of blocks of its team's items, blocks of a row.
struct BkPos {
    int item, row, strip, bg, b, g, slot;    // row of blocks in walking order; batch * G + group, batch, group, first slot of the item inside its group
    int seq;                              // blocks of the team's sequence before this one
    __device__ __forceinline__ void decode(const Blk &P, int spw) {
        bg = item / P.ntile;
        b = bg / P.G;
        g = bg - b * P.G;
        slot = (item - bg * P.ntile) * spw;
    }
    __device__ __forceinline__ void start(const Blk &P, int spw, int first, int w) {
        item = first; row = w; strip = 0; seq = w * P.nstrip;   // (there are no more workers than rows)
        decode(P, spw);
    }
    // returns whether the next block is of another item
    __device__ __forceinline__ bool next(const Blk &P, int spw, int rw, int stride) {
        ++seq;
        if (++strip < P.nstrip) return false;
        strip = 0;
        seq += (rw - 1) * P.nstrip;
        row += rw;
        if (row < P.nblk) return false;
        row -= P.nblk;
        item += stride;
        decode(P, spw);
        return true;
    }
};

// How many blocks of the sequence the workers of a CTA have left behind, and the wait of a worker for the one before it.
struct RowSeq {
    uint32_t mine, before;   // shared-memory addresses of the two counts
    int nstrip;
    __device__ __forceinline__ void init(int *count, int warp, int rw, int nstrip_) {   // all threads of the CTA, before a CTA barrier
        nstrip = nstrip_;
        const int w = warp & (rw - 1);
        mine = smem_addr(count + warp); before = smem_addr(count + warp - w + ((w - 1) & (rw - 1)));
        if ((threadIdx.x & 31) == 0) count[warp] = 0;
    }
    // what the warp's threads have written is there for whoever sees the count
    __device__ __forceinline__ void done(int seq) const {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(mine), "r"(seq + 1) : "memory");
    }
    // until the block above (in walking order) block `seq` is done.  Bounded by the number of polls
    // (between two of them a thread sleeps 0 to 40 ns; a block takes some 10 us), then false.
    __device__ __forceinline__ bool wait(int seq, int polls = 1 << 22) const {
        const int need = seq + 1 - nstrip;   // (of the first row of a sequence: 0 or less)
#pragma unroll 1
        for (int i = 0; i < polls; ++i) {
            int have;
            asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(have) : "r"(before) : "memory");
            if (__all_sync(0xffffffffu, have >= need)) return true;
            __nanosleep(20);
        }
        return false;
    }
    // gives up: flags the error and lets the other workers run to their ends
    __device__ __forceinline__ void abandon(int *status) const {
        if ((threadIdx.x & 31) == 0) {
            atomicOr(status, ERR_WORKER_TIMEOUT);
            asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(mine), "r"(0x7fffffff) : "memory");
        }
    }
};

__device__ __forceinline__ float rcp(float x) {   // of a value in [1, 4]: no range to guard
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// softplus(x) = max(x, 0) + log(1 + t), t = exp(-|x|) in (0, 1]; log(1 + t) = 2 atanh(s) with s = t / (2 + t) <= 1/3
// from its power series (terms up to s^13: remainder below 1e-8 of the sum), two values at a time.  x above 20
// passes through: the logarithm is then below half a unit in the last place.  SIG: `sig` = 1 / (1 + exp(-x)).
// About 3e-7 relative.
template <bool SIG>
__device__ __forceinline__ float2 bk_softplus2(float2 x, float2 *sig) {
    const float2 t = f2(ex2(-fabsf(x.x) * LOG2E), ex2(-fabsf(x.y) * LOG2E)), d = add2(t, bc(2.f));
    const float2 s = mul2(t, f2(rcp(d.x), rcp(d.y))), z = mul2(s, s);
    float2 q = fma2(z, bc(1.f / 13.f), bc(1.f / 11.f));
    q = fma2(q, z, bc(1.f / 9.f)); q = fma2(q, z, bc(1.f / 7.f)); q = fma2(q, z, bc(0.2f)); q = fma2(q, z, bc(1.f / 3.f));
    const float2 h = fma2(mul2(s, z), q, s);
    if constexpr (SIG) {
        const float2 e = add2(t, bc(1.f)), r = f2(rcp(e.x), rcp(e.y)), tr = mul2(t, r);
        *sig = f2(x.x >= 0.f ? r.x : tr.x, x.y >= 0.f ? r.y : tr.y);
    }
    return fma2(h, bc(2.f), f2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f)));
}

// Elements of the input type.  bk_ldp: loaded only when `on` (else 0), as raw bits: the guard is a predicate on the
// load, and nothing depends on the register until the value is used.
template <int DT> struct bk_type { using t = uint16_t; };
template <> struct bk_type<CS2D_F32> { using t = uint32_t; };
template <int DT>
__device__ __forceinline__ uint32_t bk_ldp(const typename bk_type<DT>::t *p, bool on) {
    if constexpr (DT == CS2D_F32) {
        uint32_t v;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.nc.b32 %0, [%1];\n\t}" : "=r"(v) : "l"(p), "r"((int)on));
        return v;
    } else {
        uint32_t v;   // (a 32-bit register: nothing converts the value, and so waits for it, before it is used)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.nc.u16 %0, [%1];\n\t}" : "=r"(v) : "l"(p), "r"((int)on));
        return v;
    }
}
// 16 bytes: zeros unless `on`.  NC: through the read-only path (nothing in this kernel writes them).
template <bool NC>
__device__ __forceinline__ float4 bk_ld16(const float4 *p, bool on) {
    float4 v;
    if constexpr (NC)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t@p ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];\n\t}"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p), "r"((int)on));
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t@p ld.global.v4.f32 {%0,%1,%2,%3}, [%4];\n\t}"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p), "r"((int)on) : "memory");
    return v;
}
__device__ __forceinline__ void bk_red16(float *p, float4 v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p red.global.add.v4.f32 [%0], {%1,%2,%3,%4};\n\t}" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"((int)on) : "memory");
}
__device__ __forceinline__ void bk_st16(float4 *p, float4 v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p st.global.v4.f32 [%0], {%1,%2,%3,%4};\n\t}" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"((int)on) : "memory");
}
template <int DT>
__device__ __forceinline__ float bk_cvt(uint32_t raw) {
    if constexpr (DT == CS2D_F32) return __uint_as_float(raw);
    else if constexpr (DT == CS2D_BF16) return __uint_as_float(raw << 16);
    else return __half2float(__ushort_as_half((unsigned short)raw));
}
// Results: fp32, the input type, or (merge) added onto an fp32 image.
template <int DT, bool MERGE>
__device__ __forceinline__ void bk_st(void *base, int64_t i, float v, bool on) {
    if constexpr (MERGE) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p red.global.add.f32 [%0], %1;\n\t}" ::"l"(reinterpret_cast<float *>(base) + i), "f"(v), "r"((int)on) : "memory");
    } else if constexpr (DT == CS2D_F32) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(reinterpret_cast<float *>(base) + i), "f"(v), "r"((int)on) : "memory");
    } else {
        const unsigned short h = DT == CS2D_BF16 ? __bfloat16_as_ushort(__float2bfloat16(v)) : __half_as_ushort(__float2half(v));
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.b16 [%0], %1;\n\t}" ::"l"(reinterpret_cast<uint16_t *>(base) + i), "h"(h), "r"((int)on) : "memory");
    }
}
}  // namespace cs2d
