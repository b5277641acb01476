// Pair-walk kernels (sm_100a), one state per channel: what the forward (cs2d_pair_fwd.cu) and the backward
// (cs2d_pair_bwd.cu) share.
//
// A thread owns two channels (the halves of packed fp32x2 registers) and walks their image alone: in bands of 4 rows, along
// a band two columns at a time.  No scan over lanes, no skew, no sum over states, and the 64 channels of a warp share each
// pixel's B and C and one sum of its dB and dC.  All lanes are at the same pixel, so columns that a map does not have are
// skipped by the whole warp.  The unrolled body is 8 pixels: with twice that the two loops of the backward overflowed the
// instruction cache (a fifth of the stalls on 14x14 maps).
//
// The planes of 64 channels are far apart in memory, so a warp fetches blocks of them into shared memory, asynchronously, and
// every thread picks its own channels from there.  Results take the place of the inputs they came from and leave the same
// way.  A channel's block is
//   the whole band, one contiguous piece of its plane, where it fits 128 bytes and rows are contiguous ("linear"), else
//   4 rows of 32 bytes (16-bit inputs that are not aligned to words: 16 bytes).
// Blocks are moved in pieces of 8 or 4 bytes.  16-bit rows or planes of an odd number of elements start in the middle of a
// word for every other channel or row: the block is then fetched from the word its first element lies in (a word that holds
// an element of the tensor can be read), keeps that offset in shared memory, and is read and written element by element
// ("EL"; so are fp32 blocks that only allow 4-byte pieces).  A channel's pitch in shared memory is 132 or 136 bytes, an odd
// number of pieces.
//
// Where rows are whole pairs and a linear block's chunks fit 128 bytes, or rows are whole 16-byte chunks ("CK"), the 16-byte chunks of memory that
// a block touches are copied instead (a chunk that holds an element of the tensor can be read): copies of 16 bytes pass the L1 cache
// by - measured, 64 channels of 112 bytes: 570 cycles of a warp, in pieces of 8 or 4 bytes 3660, as 64 bulk copies 3800.  A channel then has
// 128 bytes, a linear block's byte the place that it has in its chunks, a row's one of 32 that the low bits of its address say, chunks
// swizzled over the lanes; an address takes an instruction more, and four lanes share a bank.  So blocks read element by element stay as they
// are (13x13 fp32 forward and backward 150 + 322 -> 168 + 369 us, 7x7 bf16 166 + 330 -> 188 + 401), and in the backward those
// that are not whole chunks (128x3072x14x14 bf16 607 -> 620).  us, pieces / chunks: 128x3072x14x14 bf16 forward 283 / 235,
// 64x1536x16x16 fp32 129 + 277 / 103 + 264, four corners 8x384x112x112 bf16 655 + 1199 / 501 + 1064.
//
// What crosses a band or 8 columns goes through global memory, threads innermost (512 bytes per warp and access):
//   row  [item][band][column][nl] float4 (h, h', a, a') of a band's last row (rolling: [team][column][32], one row
//        per warp, or team of row workers, that is on the GPU at a time)
//   colq [item][band][column / 8 - 1][4 rows][nl] float4 (q, q', s, s') of the column left of a group of 8
//   cola the same, float2 (a, a')
// (q = h - s; an item is a warp's 64 channels of one image and group.  nl: 32, or in groups of less than 63 channels their
// pairs and one place for all lanes past them, which hold the same values: lane i uses place min(i, nl - 1).)
//
// Few items run with 2 or 4 row WORKERS per CTA of four warps: worker w takes every RW-th band, one step behind worker
// w - 1; the CTA's warps then meet on its barrier once per step.
#pragma once

#include "cs2d_blk.cuh"

namespace cs2d {

constexpr int PW_R = 4, PW_CH = 64, PW_WARPS = 4;
constexpr int PW_HALF = 32 * 136, PW_IN = 2 * PW_HALF;    // bytes of one input's block: the even channels, the odd ones

struct Pw {
    int H, W, G, dpg, io_dt;
    int nblk, nstrip, nsub, wp;   // bands; fetched blocks per band; groups of 8 columns; columns, even
    int period, rwl, npass;       // steps per band, log2 of the row workers, bands per worker
    int ntile, items, grid;       // warps' worth of channels per group; batch * G * ntile
    int nl;                       // places of an item (see above)
    unsigned flip_h, flip_w;
    int shared;                   // bit 0: u has dpg channels shared by the groups, bit 1: dout
    int fs, lin, el;              // columns of a fetched block; whole bands; element by element
    int ck, al;                   // chunks; what the addresses of blocks (linear) or rows are multiples of, 16 at most
    int vin, vout;                // bytes of a piece of the inputs (8 or 4) and of the results (16, 8, 4 or 2)
    int lpin, lpout;              // lanes (a power of two) that move a channel's block
    int v32;                      // fp32 results of 16-bit inputs (merge: images) take two elements at once
    int f32;                      // 16-bit inputs with an fp32 result (forward) or gradient (backward)
    const void *u, *delta, *B, *C;
    const float *A, *D, *bias;
    int64_t u_bs, u_ds, u_hs, dl_bs, dl_ds, dl_hs, A_ds;
    int64_t B_bs, B_gs, B_hs, C_bs, C_gs, C_hs;
    void *out; int64_t o_bs, o_ds, o_hs;    // forward: out; backward: dout
    const float *mw; float *dw;             // direction merge (see Dev)
    float4 *row, *colq; float2 *cola;
    float4 *adj;                            // backward, [team][column][32]: (m, m', a, a') of the row below a band
    void *du, *ddelta;
    float *dA, *dB, *dC, *dD, *dbias;
};

template <int DT> struct pw_io {
    static constexpr int ES = DT == CS2D_F32 ? 4 : 2, FS = 32 / ES;   // FS: most columns of a fetched block
};

// 8 bytes that nothing in the kernel writes: zeros unless `on`
__device__ __forceinline__ float2 pw_ld8(const void *p, bool on) {
    float2 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t@p ld.global.nc.v2.f32 {%0,%1}, [%2];\n\t}" : "=f"(v.x), "=f"(v.y) : "l"(p), "r"((int)on));
    return v;
}

// bk_ldp through a 16-bit register (through a 32-bit one, whose value nothing waits for, the backward is 1 to 2 % slower)
template <int DT>
__device__ __forceinline__ uint32_t pw_ldp(const typename bk_type<DT>::t *p, bool on) {
    if constexpr (DT == CS2D_F32) return bk_ldp<DT>(p, on);
    unsigned short v = 0;
    if constexpr (DT != CS2D_F32)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b16 %0, 0;\n\t@p ld.global.nc.b16 %0, [%1];\n\t}" : "=h"(v) : "l"(p), "r"((int)on));
    return v;
}

struct PwPos {   // position in a warp's stream of blocks
    int item, pass, strip, bg, g, tile;
    __device__ __forceinline__ void decode(const Pw &P) {
        bg = item / P.ntile;
        g = bg % P.G;
        tile = item % P.ntile;
    }
    __device__ __forceinline__ void next(const Pw &P, int stride) {
        if (++strip < P.period) return;
        strip = 0;
        if (++pass < P.npass) return;
        pass = 0;
        item += stride;
        decode(P);
    }
};

// A block of one tensor, in memory order: `nseg` segments (rows, or one band) per channel
struct PwBlock {
    const char *p;        // first element of segment 0 of channel 0; it may lie outside the image
    int64_t ds, hs;       // bytes between channels; between segments (scan rows)
    int nch, nseg;        // channels and segments that exist
    int lo, hi;           // bytes of a segment that exist
    // offset in shared memory of the first element of segment r of channels of parity k (16-bit elements in the middle of a word)
    __device__ __forceinline__ int odd(int k, int r) const { return (int)(reinterpret_cast<uintptr_t>(p) + k * ds + r * hs) & 2; }
};

template <int DT>
__device__ __forceinline__ PwBlock pw_block(const void *base, int64_t off, int64_t ds, int64_t hs, int nch, int r0, int c0, const Pw &P, bool fh, bool fw) {
    constexpr int ES = pw_io<DT>::ES;
    PwBlock b;
    b.ds = ds * ES;
    b.nch = nch;
    if (P.lin) {
        const int fr = fh ? P.H - PW_R - r0 : r0;
        b.p = reinterpret_cast<const char *>(base) + (off + (int64_t)fr * P.W) * ES;
        b.hs = 0; b.nseg = 1;
        b.lo = fr < 0 ? -fr * P.W * ES : 0;
        b.hi = fh ? PW_R * P.W * ES : min(PW_R, P.H - r0) * P.W * ES;
    } else {
        const int fr = fh ? P.H - 1 - r0 : r0, fc = fw ? P.W - c0 - P.fs : c0;
        b.p = reinterpret_cast<const char *>(base) + (off + (int64_t)fr * hs + fc) * ES;
        b.hs = (fh ? -hs : hs) * ES; b.nseg = min(PW_R, P.H - r0);
        b.lo = fc < 0 ? -fc * ES : 0;
        b.hi = (fw ? P.fs : min(P.fs, P.W - c0)) * ES;
    }
    return b;
}

// What copies of nothing name as their source: it has to be a multiple of the copy's size even so, which a tensor's own address need not be
__device__ __forceinline__ const char *pw_nothing(const void *tensor) { return reinterpret_cast<const char *>(reinterpret_cast<uintptr_t>(tensor) & ~(uintptr_t)15); }
// Fetch a block, V bytes at a time; pieces without anything that exists become zero.  EL: from the word of the first element.
template <int V, bool EL>
__device__ __forceinline__ void pw_fetch(uint32_t dst, const PwBlock &b, const Pw &P, const void *tensor) {
    const int lane = threadIdx.x & 31, x = lane & (P.lpin - 1), seg = P.lin ? 0 : x / (P.lpin / 4), o = (P.lin ? x : x % (P.lpin / 4)) * V;
    const int step = 32 / P.lpin, pit = V == 8 ? 136 : 132;
    const char *src = b.p + (lane / P.lpin) * b.ds + seg * b.hs;
    const int64_t add = step * b.ds;
    const char *nothing = pw_nothing(tensor);
    dst += seg * 32 + o;
#pragma unroll 8
    for (int ch = lane / P.lpin; ch < PW_CH; ch += step) {
        const int od = EL ? (int)(reinterpret_cast<uintptr_t>(src) & 3) : 0;
        const bool on = ch < b.nch && seg < b.nseg && o + V > b.lo + od && o < b.hi + od;
        const char *s = src - od + o;
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst + (ch & 1) * PW_HALF + (ch >> 1) * pit), "l"(on ? s : nothing), "n"(V), "r"(on ? V : 0) : "memory");
        src += add;
    }
}
// The way back; `in`: the block whose place the results took (its offsets in shared memory)
template <int V>
__device__ __forceinline__ void pw_store_v(uint32_t from, const PwBlock &b, const PwBlock &in, const Pw &P) {
    const int lane = threadIdx.x & 31, step = P.lpout > 32 ? 1 : 32 / P.lpout, pit = P.vin == 8 ? 136 : 132;
#pragma unroll 1
    for (int x = lane & (P.lpout - 1); x < P.lpout; x += 32) {
        const int seg = P.lin ? 0 : x / (P.lpout / 4), o = (P.lin ? x : x % (P.lpout / 4)) * V;
        const bool ok = seg < b.nseg && o >= b.lo && o < b.hi;
        char *dst = const_cast<char *>(b.p) + (lane / P.lpout) * b.ds + seg * b.hs + o;
        const int64_t add = step * b.ds;
        const uint32_t f0 = from + seg * 32 + o + (V == 2 ? in.odd(0, seg) : 0), f1 = from + PW_HALF + seg * 32 + o + (V == 2 ? in.odd(1, seg) : 0);
#pragma unroll 8
        for (int ch = lane / P.lpout; ch < PW_CH; ch += step) {
            const uint32_t a = ((ch & 1) ? f1 : f0) + (ch >> 1) * pit;
            const int on = ok && ch < b.nch;
            if constexpr (V == 8)
                asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 x, y;\n\tsetp.ne.b32 p, %2, 0;\n\tld.shared.v2.b32 {x,y}, [%1];\n\t@p st.global.v2.b32 [%0], {x,y};\n\t}" ::"l"(dst), "r"(a), "r"(on) : "memory");
            else if constexpr (V == 4)
                asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 x;\n\tsetp.ne.b32 p, %2, 0;\n\tld.shared.b32 x, [%1];\n\t@p st.global.b32 [%0], x;\n\t}" ::"l"(dst), "r"(a), "r"(on) : "memory");
            else
                asm volatile("{\n\t.reg .pred p;\n\t.reg .b16 x;\n\tsetp.ne.b32 p, %2, 0;\n\tld.shared.b16 x, [%1];\n\t@p st.global.b16 [%0], x;\n\t}" ::"l"(dst), "r"(a), "r"(on) : "memory");
            dst += add;
        }
    }
}
__device__ __forceinline__ void pw_store(uint32_t from, const PwBlock &b, const PwBlock &in, const Pw &P) {
    if (P.vout == 8) pw_store_v<8>(from, b, in, P);
    else if (P.vout == 4) pw_store_v<4>(from, b, in, P);
    else pw_store_v<2>(from, b, in, P);
}

// CK: place of the byte whose address has the low bits x (linear blocks: x bytes from the block's first chunk) of segment seg of channel ch
__device__ __forceinline__ uint32_t pw_place(const Pw &P, int ch, int seg, uint32_t x) {
    return (ch & 1) * PW_HALF + (ch >> 1) * 128 + ((P.lin ? x : seg * 32 + (x & 31)) ^ (((ch >> 1) & 7) << 4));
}
__device__ __forceinline__ void pw_fetch_ck(uint32_t dst, const PwBlock &b, const Pw &P, const void *tensor) {
    const int lane = threadIdx.x & 31, x = lane & 7, seg = P.lin ? 0 : x >> 1, o = P.lin ? x * 16 : (x & 1) * 16;
    const char *src = b.p + (lane >> 3) * b.ds + seg * b.hs;
    const int64_t add = 4 * b.ds;
    const char *nothing = pw_nothing(tensor);
#pragma unroll 4
    for (int ch = lane >> 3; ch < PW_CH; ch += 4) {
        const int od = (int)(reinterpret_cast<uintptr_t>(src) & 15);
        const char *s = src + (o - od);
        const bool on = ch < b.nch && seg < b.nseg && o + 16 > b.lo + od && o < b.hi + od;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + pw_place(P, ch, seg, P.lin ? o : (uint32_t)reinterpret_cast<uintptr_t>(s))), "l"(on ? s : nothing), "r"(on ? 16 : 0) : "memory");
        src += add;
    }
}
// The way back: pieces of P.vout bytes
template <int V>
__device__ __forceinline__ void pw_store_ckv(uint32_t from, const PwBlock &b, const PwBlock &in, const Pw &P) {
    const int lane = threadIdx.x & 31, step = 32 / P.lpout, x = lane & (P.lpout - 1);   // (a channel is 32 pieces at most)
    const int seg = P.lin ? 0 : x / (P.lpout / 4), o = (P.lin ? x : x % (P.lpout / 4)) * V;
    const bool ok = seg < b.nseg && o >= b.lo && o < b.hi;
    char *dst = const_cast<char *>(b.p) + (lane / P.lpout) * b.ds + seg * b.hs + o;
    const int64_t add = step * b.ds;
    uint32_t at = (uint32_t)reinterpret_cast<uintptr_t>(in.p) + (lane / P.lpout) * (uint32_t)in.ds + seg * (uint32_t)in.hs;
    const uint32_t iadd = step * (uint32_t)in.ds;
#pragma unroll 8
    for (int ch = lane / P.lpout; ch < PW_CH; ch += step) {
        const uint32_t a = from + pw_place(P, ch, seg, (P.lin ? at & 15 : at) + o);
        const int on = ok && ch < b.nch;
        if constexpr (V == 16)
            asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 x, y, z, w;\n\tsetp.ne.b32 p, %2, 0;\n\tld.shared.v4.b32 {x,y,z,w}, [%1];\n\t@p st.global.v4.b32 [%0], {x,y,z,w};\n\t}" ::"l"(dst), "r"(a), "r"(on) : "memory");
        else if constexpr (V == 8)
            asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 x, y;\n\tsetp.ne.b32 p, %2, 0;\n\tld.shared.v2.b32 {x,y}, [%1];\n\t@p st.global.v2.b32 [%0], {x,y};\n\t}" ::"l"(dst), "r"(a), "r"(on) : "memory");
        else
            asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 x;\n\tsetp.ne.b32 p, %2, 0;\n\tld.shared.b32 x, [%1];\n\t@p st.global.b32 [%0], x;\n\t}" ::"l"(dst), "r"(a), "r"(on) : "memory");
        dst += add; at += iadd;
    }
}
__device__ __forceinline__ void pw_store_ck(uint32_t from, const PwBlock &b, const PwBlock &in, const Pw &P) {
    if (P.vout == 16) pw_store_ckv<16>(from, b, in, P);
    else if (P.vout == 8) pw_store_ckv<8>(from, b, in, P);
    else pw_store_ckv<4>(from, b, in, P);
}

// This lane's view of an input's block: elements of two neighbouring columns
template <int DT, bool EL>
struct PwView {
    static constexpr int ES = pw_io<DT>::ES;
    uint32_t a[2][2];   // [parity of the row][channel]; not EL: [0][0]
    __device__ __forceinline__ void at(uint32_t base, const PwBlock &b, int pit) {
        const uint32_t x = base + (threadIdx.x & 31) * pit;
        if constexpr (EL) {
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i >> 1][i & 1] = x + (i & 1) * PW_HALF + (ES == 2 ? b.odd(i & 1, i >> 1) : 0);
        } else {
            a[0][0] = x;
        }
    }
    // x[0], x[1]: scan columns c, c + 1 of scan row r; `o` is the offset of column c, `o1` that of column c + 1 (EL) or of the
    // lower of the two in memory.  What is not there (on, on1: row r, column c + 1 exist) is zero; EL: in its place there are other
    // elements, which share words or rows with the block.
    __device__ __forceinline__ void load(int r, int k, int o, int o1, bool rev, bool on, bool on1, float (&x)[2]) const {
        if constexpr (EL) {
            const uint32_t p = a[r & 1][k];
            x[0] = elem(p + o, on); x[1] = elem(p + o1, on && on1);
        } else {
            const uint32_t p = a[0][0] + k * PW_HALF + o1;
            uint32_t lo, hi;
            if constexpr (ES == 4) {
                asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(p) : "memory");
            } else {
                uint32_t w;
                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(p) : "memory");
                lo = w & 0xffffu; hi = w >> 16;
                if constexpr (DT == CS2D_BF16) { x[0] = __uint_as_float(rev ? w & 0xffff0000u : w << 16); x[1] = __uint_as_float(rev ? w << 16 : w & 0xffff0000u); return; }
            }
            const uint32_t f = rev ? hi : lo, s = rev ? lo : hi;
            x[0] = bk_cvt<DT>(f); x[1] = bk_cvt<DT>(s);
        }
    }
    __device__ __forceinline__ void store(int r, int k, int o, int o1, bool rev, float x0, float x1, bool on1) const {   // on1: column c + 1 exists
        if constexpr (EL) {
            const uint32_t p = a[r & 1][k];
            put(p + o, x0, true); put(p + o1, x1, on1);
        } else {
            const uint32_t p = a[0][0] + k * PW_HALF + o1;
            const float lo = rev ? x1 : x0, hi = rev ? x0 : x1;
            if constexpr (ES == 4) {
                asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(p), "f"(lo), "f"(hi) : "memory");
            } else {
                uint32_t w;
                if constexpr (DT == CS2D_BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(hi), "f"(lo));
                else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(hi), "f"(lo));
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(p), "r"(w) : "memory");
            }
        }
    }
    static __device__ __forceinline__ float elem(uint32_t p, bool on) {
        if constexpr (ES == 4) {
            uint32_t v;
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.shared.b32 %0, [%1];\n\t}" : "=r"(v) : "r"(p), "r"((int)on) : "memory");
            return __uint_as_float(v);
        } else {
            unsigned short v;
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b16 %0, 0;\n\t@p ld.shared.b16 %0, [%1];\n\t}" : "=h"(v) : "r"(p), "r"((int)on) : "memory");
            return bk_cvt<DT>(v);
        }
    }
    static __device__ __forceinline__ void put(uint32_t p, float x, bool on) {
        if constexpr (ES == 4) {
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.f32 [%0], %1;\n\t}" ::"r"(p), "f"(x), "r"((int)on) : "memory");
        } else {
            const unsigned short v = DT == CS2D_BF16 ? __bfloat16_as_ushort(__float2bfloat16(x)) : __half_as_ushort(__float2half(x));
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.b16 [%0], %1;\n\t}" ::"r"(p), "h"(v), "r"((int)on) : "memory");
        }
    }
};
// The same for chunks
struct PwLane {   // what the views of a lane share: where its channels' rows lie, the bits of an address that count
    uint32_t base[PW_R], mask;
    __device__ __forceinline__ void at(const Pw &P, uint32_t sm) {
        const int lane = threadIdx.x & 31;
        mask = P.lin ? 127 : 31;
#pragma unroll
        for (int r = 0; r < PW_R; ++r) base[r] = sm + lane * 128 + (((lane & 7) << 4) ^ (P.lin ? 0 : r * 32));   // (sm is a multiple of 128)
    }
};
template <int DT, int AT>   // AT: where the input's block lies in the warp's shared memory
struct PwViewCk {
    static constexpr int ES = pw_io<DT>::ES;
    uint32_t a[2], hs;   // low bits of the channels' addresses, or their offsets in the first chunk of linear blocks; of the step to the next segment
    __device__ __forceinline__ void at(const Pw &P, const PwBlock &b) {
        const uint32_t ds = (uint32_t)b.ds, m = P.lin ? 15 : ~0u, p = (uint32_t)reinterpret_cast<uintptr_t>(b.p) + 2 * (threadIdx.x & 31) * ds;
        a[0] = p & m; a[1] = (p + ds) & m;
        hs = (uint32_t)b.hs;
    }
    __device__ __forceinline__ uint32_t pair(const PwLane &L, int r, int k, int o) const { return (L.base[r] ^ ((a[k] + (r * hs + o)) & L.mask)) + (AT + k * PW_HALF); }
    __device__ __forceinline__ void load(const PwLane &L, int r, int k, int o1, bool rev, float (&x)[2]) const {
        const uint32_t p = pair(L, r, k, o1);
        if constexpr (ES == 4) {
            float lo, hi;
            asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(lo), "=f"(hi) : "r"(p) : "memory");
            x[0] = rev ? hi : lo; x[1] = rev ? lo : hi;
        } else {
            uint32_t w;
            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(p) : "memory");
            if constexpr (DT == CS2D_BF16) {
                x[0] = __uint_as_float(rev ? w & 0xffff0000u : w << 16); x[1] = __uint_as_float(rev ? w << 16 : w & 0xffff0000u);
            } else {
                x[0] = bk_cvt<DT>(rev ? w >> 16 : w & 0xffffu); x[1] = bk_cvt<DT>(rev ? w & 0xffffu : w >> 16);
            }
        }
    }
    __device__ __forceinline__ void store(const PwLane &L, int r, int k, int o1, bool rev, float x0, float x1) const {
        const uint32_t p = pair(L, r, k, o1);
        const float lo = rev ? x1 : x0, hi = rev ? x0 : x1;
        if constexpr (ES == 4) {
            asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(p), "f"(lo), "f"(hi) : "memory");
        } else {
            uint32_t w;
            if constexpr (DT == CS2D_BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(hi), "f"(lo));
            else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(hi), "f"(lo));
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(p), "r"(w) : "memory");
        }
    }
};
// Offsets of the columns c, c + 1 (c counts from the block's first) in a block's rows: o[r], and o1[r] for PwView
template <int ES, bool EL, bool CK = false>
__device__ __forceinline__ void pw_offsets(const Pw &P, int c, bool fh, bool fw, int (&o)[PW_R], int (&o1)[PW_R]) {
    const int width = P.lin ? P.W : P.fs, mc = fw ? width - 1 - c : c, mc1 = EL ? (fw ? mc - 1 : mc + 1) : (fw ? mc - 1 : mc);
#pragma unroll
    for (int r = 0; r < PW_R; ++r) {
        const int row = P.lin ? (fh ? PW_R - 1 - r : r) * P.W * ES : CK ? 0 : r * 32;   // (CK: the views count the rows)
        o[r] = row + mc * ES;
        o1[r] = row + mc1 * ES;
    }
}

// CK: rows of a linear block that the image does not have share chunks with others: zeros in their place
template <int ES, typename... Views>
__device__ __forceinline__ void pw_clear(const Pw &P, const PwLane &L, int r0, bool fh, bool fw, const Views &...v) {
    if (!P.lin || r0 + PW_R <= P.H) return;
#pragma unroll 1
    for (int c = 0; c < P.W; c += 2) {
        int o[PW_R], o1[PW_R];
        pw_offsets<ES, false, true>(P, c, fh, fw, o, o1);
#pragma unroll
        for (int r = 1; r < PW_R; ++r)
            if (r0 + r >= P.H) { (v.store(L, r, 0, o1[r], false, 0.f, 0.f), ...); (v.store(L, r, 1, o1[r], false, 0.f, 0.f), ...); }
    }
}

// B and C of a block as (B, C) pairs in scan order: raw values of this lane's pixels, one block ahead
template <int DT> struct PwBC {
    static constexpr int FS = pw_io<DT>::FS, PX = 4 * FS / 32;   // pixels per lane
    uint32_t b[PX], c[PX];
    __device__ __forceinline__ void load(const Pw &P, const PwPos &q, int r0, int c0, bool fh, bool fw) {
        using T = typename bk_type<DT>::t;
        const int lane = threadIdx.x & 31, bi = q.bg / P.G;
        const T *B = reinterpret_cast<const T *>(P.B) + (int64_t)bi * P.B_bs + (int64_t)q.g * P.B_gs;
        const T *C = reinterpret_cast<const T *>(P.C) + (int64_t)bi * P.C_bs + (int64_t)q.g * P.C_gs;
#pragma unroll
        for (int i = 0; i < PX; ++i) {
            const int px = i * 32 + lane, r = r0 + px / FS, cc = c0 + px % FS;   // (more columns than a narrow block has: not used)
            const bool on = r < P.H && cc < P.W;
            const int fr = fh ? P.H - 1 - r : r, fc = fw ? P.W - 1 - cc : cc;
            b[i] = pw_ldp<DT>(B + (int64_t)fr * P.B_hs + fc, on);
            c[i] = pw_ldp<DT>(C + (int64_t)fr * P.C_hs + fc, on);
        }
    }
    __device__ __forceinline__ void put(float2 *s) const {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int i = 0; i < PX; ++i) s[i * 32 + lane] = f2(bk_cvt<DT>(b[i]), bk_cvt<DT>(c[i]));
    }
};

// softplus, and (SIG) its derivative
template <bool SIG>
__device__ __forceinline__ float2 pw_softplus2(float2 x, float2 *sig) {
    const float2 t = f2(ex2(-fabsf(x.x) * LOG2E), ex2(-fabsf(x.y) * LOG2E));
    if constexpr (SIG) {
        const float2 e = add2(t, bc(1.f)), r = f2(rcp(e.x), rcp(e.y)), tr = mul2(t, r);
        *sig = f2(x.x >= 0.f ? r.x : tr.x, x.y >= 0.f ? r.y : tr.y);
    }
    return fma2(log1p_over(t), t, f2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f)));
}

// Writes the scan columns c, c + 1 of a row of fp32 results (image column fc, and the one on its right, or left when rev), or adds them
__device__ __forceinline__ void pw_put32(float *row, int fc, float x0, float x1, bool rev, bool on, bool on1, bool vec, bool add) {
    if (vec) {   // even width and alignment: both exist
        float *p = row + (rev ? fc - 1 : fc);
        const float lo = rev ? x1 : x0, hi = rev ? x0 : x1;
        if (add) asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p red.global.add.v2.f32 [%0], {%1,%2};\n\t}" ::"l"(p), "f"(lo), "f"(hi), "r"((int)on) : "memory");
        else asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p st.global.v2.f32 [%0], {%1,%2};\n\t}" ::"l"(p), "f"(lo), "f"(hi), "r"((int)on) : "memory");
    } else if (add) {
        bk_st<CS2D_F32, true>(row, fc, x0, on); bk_st<CS2D_F32, true>(row, rev ? fc - 1 : fc + 1, x1, on && on1);
    } else {
        bk_st<CS2D_F32, false>(row, fc, x0, on); bk_st<CS2D_F32, false>(row, rev ? fc - 1 : fc + 1, x1, on && on1);
    }
}
}  // namespace cs2d
