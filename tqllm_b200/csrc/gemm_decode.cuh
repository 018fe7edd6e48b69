// Weight decoders of the tensor-core grouped GEMM: one 64-column step of one 16-row bank tile -> fp16 A operand in registers.
// A 256-column chunk has four steps (two units of two); a warp decodes all of every other chunk: prep once, then for J = 0 .. 3 load<J> (what the
// step needs from shared memory; the caller asks for it a step ahead) and step<J>.
//
// A warp owns a row tile; lane L = 4 g + t holds, in the bank's lane-major layout, the code words of rows g and g + 8
// (formats.cuh). Every code word (or pair of IQ3_S grid entries) decodes to eight fp16 values, so a step leaves sixteen
// registers per lane: exactly the fragment that tcgen05.st.16x256b.x4 puts into tensor memory as the A operand of four
// K = 16 products (register 4 i + 2 r + c of the lane: row g + 8 r, columns 16 i + 4 t + 2 c .. + 1 of the step). Which
// columns a word covers depends on the format (a Q4_K byte holds column c of two different sub-blocks, an IQ4 byte columns
// c and c + 16, ...): rather than shuffling values between lanes, the GEMM permutes the 64 columns of a step: colmap<T>(pos)
// is the column stored at operand position pos, and the activation rows are written in the same order (the sum over K does
// not care).
//
// Values: the formula of the format's host decoder (dequantize_host, src/formats/weight/dequant.cpp:80-99,137-150,
// 177-192,352-360,397-409) in fp16 arithmetic on two weights per instruction, arranged so that every intermediate but the
// last is exact: IQ3_S (odd magnitude x (1 + 2 s)) exact, then x d; the 4-bit IQ3_S codes the same; IQ4_NL kvalue x d;
// NVFP4 e2m1 x e4m3 exact (the fp32 row scale is applied to the accumulator in the epilogue): one rounding each. Q4_K:
// sc q exact, x d - the leading fp16 term of dmin m (one rounding), + the rest of dmin m (a second rounding, which removes
// the error the 32 weights of a sub-block would otherwise share). IQ4_XS multiplies the kvalue by
// fp16(d (ls - 32)): that factor's rounding (relative 2^-12, the same for the 32 weights of a sub-block) comes on top.
#pragma once
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "formats.cuh"

namespace b2 {
namespace gdec {

// column (0..63, inside the step) held at operand position pos (0..63)
template <uint32_t T> __host__ __device__ inline int colmap(int pos) {
    const int i = pos >> 4, t = (pos >> 2) & 3;                        // K = 16 product, lane of the row's four
    const int w = t + 4 * (i >> 1), q = 4 * (i & 1) + (pos & 3);       // code word of the step, value inside the word as the decoder emits it
    // word w: low nibbles = sub-block 0, high nibbles = sub-block 1; inside each the decoder emits bytes 0, 2, 1, 3 (nibble pairs 16 bits apart)
    if (T == T_Q4_K || T == T_IQ3S4) return (q < 4 ? 0 : 32) + 4 * w + ((q & 1) << 1) + ((q >> 1) & 1);
    if (T == T_IQ4_XS || T == T_IQ4_NL) return 32 * (w >> 2) + 4 * (w & 3) + (q >> 1) + 16 * (q & 1);   // byte i: columns i, i + 16
    return 8 * w + q;                                                  // IQ3_S, NVFP4G: eight consecutive columns per word
}

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
// the eight values of word b (0: word t, 1: word t + 4) of row g + 8 r into the lane's fragment
__device__ __forceinline__ void put(uint32_t (&f)[16], int r, int b, const uint4 & o) {
    f[8 * b + 2 * r] = o.x; f[8 * b + 2 * r + 1] = o.y;
    f[8 * b + 4 + 2 * r] = o.z; f[8 * b + 4 + 2 * r + 1] = o.w;
}
// the four words of plane j of a 256-column tile of nibble planes: {row g: word t, word t + 4; row g + 8: the same}
__device__ __forceinline__ uint4 plane(const uint8_t * chunk, int j, int lane) { return *reinterpret_cast<const uint4 *>(chunk + 512 * j + 16 * lane); }

// (v & mask) | bits in one instruction: it takes one constant as an immediate, so `bits` has to be in a register and look like a
// variable (with two constants the compiler writes two instructions: 16 more per step of the formats below)
__device__ __forceinline__ uint32_t in_register(uint32_t v) {
    uint32_t r;
    asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t and_or(uint32_t v, uint32_t mask, uint32_t bits) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(mask), "r"(bits));
    return r;
}

template <uint32_t T> struct Dec;
// the constants of sub-block t of a unit, rows g and g + 8, in the warp's scratch
__device__ __forceinline__ void put_constants(const uint2 (&c)[2], int lane, uint8_t * scratch) {
    uint2 * to = reinterpret_cast<uint2 *>(scratch) + lane;
    to[0] = c[0];
    to[32] = c[1];
}

// ---------------------------------------------------------------------------------------------------------------
template <> struct Dec<T_Q4_K> {
    static constexpr int TAB_BYTES = 0;
    __device__ static void init(void *, int, int) {}
    // Two weights per instruction. A nibble under the exponent of 1024 is 1024 + q (low nibbles) or 1024 + 16 q (high nibbles):
    // one logic operation for two weights. t = (1024 + q) S - 1024 S = sc q (an integer below 1024: exact, and 1024 sc <= 64512
    // is an fp16 number), with S = sc for the low and sc / 16 for the high nibbles; then t d + MH (exact product, one rounding
    // of the weight) and + ML, where MH + ML = -dmin m split into two fp16 terms. Rounding the sub-block's d sc or dmin m to
    // one fp16 constant would be cheaper, but that error is shared by the 32 weights of the sub-block and adds up along a
    // row, and rounding t d before the subtraction loses the bits that cancel (both measured: 2.5 to 3 times the output error).
    __device__ __forceinline__ static uint32_t two(uint32_t n1024, __half2 S, __half2 NS, __half2 MH, __half2 ML, __half2 D) {
        return h2_bits(__hadd2(__hfma2(__hfma2(bits_h2(n1024), S, NS), D, MH), ML));
    }
    // Once per chunk: lane t of a row's four lanes turns the headers of its two rows into the constants of sub-blocks t and 4 + t
    // and leaves them in the warp's scratch, two in a word (the arithmetic takes either half of a register twice at no
    // cost; spread there, they took twice the registers and loads): [row][sub-block]((S, -1024 S), (MH, ML)). The scratch holds a unit; the second one's words wait in registers (Pre::late)
    // until the first one's are read. With scratch for both, items of 128 and 256 tokens had a raw slot less (294 to 805 experts: 3 instead of 4):
    // a layer on 512 experts, 50 tokens each 527 us, with it 514; 128 each 980, 964; on 384, 125 each 711, 699.
    // The scales and mins are exact as fp16, MH = fp16(-dmin m), ML = the exact rest. (Constants of two rows in one register,
    // fetched with shuffles and spread with byte permutes, took 45 more instructions a step, 36 of them in the integer pipe.)
    static constexpr int SCRATCH = 16 * 4 * 8;
    struct Pre { uint32_t D[2], magic; uint2 late[2]; };
    __device__ __forceinline__ static Pre prep(const uint8_t * chunk, int lane, uint8_t * scratch) {
        const int g = lane >> 2, t = lane & 3;
        const uint4 h0 = *reinterpret_cast<const uint4 *>(chunk + 2048 + 16 * g), h1 = *reinterpret_cast<const uint4 *>(chunk + 2048 + 16 * (g + 8));    // d, dmin | s[12]
        const __half2 dm = bits_h2(__byte_perm(h0.x, h1.x, 0x7632) ^ 0x80008000u);       // -dmin of the two rows
        const uint32_t sel = uint32_t(t) * 0x0101u + 0x0400u;               // selector nibbles 0 and 2: byte t of the first, of the second word
        auto pick = [&](uint32_t x, uint32_t y) {                            // byte t of either word, 16 bits apart, as fp16: 1024 + byte, then - 1024
            const uint32_t v = __byte_perm(x, y, sel);
            return __hadd2(bits_h2((v & 0x003F003Fu) | 0x64006400u), __float2half2_rn(-1024.f));
        };
        Pre p{{__byte_perm(h0.x, 0u, 0x1010), __byte_perm(h1.x, 0u, 0x1010)}, in_register(0x64006400u)};
        auto unit = [&](uint2 * to, uint32_t sc0, uint32_t mn0, uint32_t sc1, uint32_t mn1) {      // a unit's four scales and four mins as bytes -> (row g, row g + 8)
            __half2 sc = pick(sc0, sc1);
            const __half2 mn = pick(mn0, mn1);
            if (t & 1) sc = __hmul2(sc, __float2half2_rn(0.0625f));
            const __half2 ns = __hmul2(sc, __float2half2_rn(-1024.f)), mh = __hmul2(dm, mn), ml = __hfma2(dm, mn, __hneg2(mh));
            to[0] = make_uint2(h2_bits(__lows2half2(sc, ns)), h2_bits(__lows2half2(mh, ml)));
            to[1] = make_uint2(h2_bits(__highs2half2(sc, ns)), h2_bits(__highs2half2(mh, ml)));
        };
        uint2 now[2];
        unit(now, h0.y, h0.z, h1.y, h1.z);                                     // (src/formats/weight/dequant.cpp:56-64)
        unit(p.late, (h0.w & 0x0F0F0F0Fu) | ((h0.y >> 2) & 0x30303030u), ((h0.w >> 4) & 0x0F0F0F0Fu) | ((h0.z >> 2) & 0x30303030u),
             (h1.w & 0x0F0F0F0Fu) | ((h1.y >> 2) & 0x30303030u), ((h1.w >> 4) & 0x0F0F0F0Fu) | ((h1.z >> 2) & 0x30303030u));
        put_constants(now, lane, scratch);
        return p;
    }
    __device__ __forceinline__ static void second_unit(const Pre & p, int lane, uint8_t * scratch) { put_constants(p.late, lane, scratch); }
    struct Raw { uint4 w, c[2]; };                                           // code words; constants of both sub-blocks of row g, of row g + 8
    template <int J> __device__ __forceinline__ static Raw load(const uint8_t * chunk, int lane, const uint8_t * scratch) {
        const uint4 * c = reinterpret_cast<const uint4 *>(scratch) + 2 * (lane >> 2) + (J & 1);
        return Raw{plane(chunk, J, lane), {c[0], c[16]}};
    }
    template <int J> __device__ __forceinline__ static void step(const Raw & raw, int, const void *, const Pre & p, uint32_t (&f)[16]) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint4 cc = raw.c[r];
            const __half2 D = bits_h2(p.D[r]);
            auto lo = [&](uint32_t w) { return two(and_or(w, 0x000F000Fu, p.magic), __low2half2(bits_h2(cc.x)), __high2half2(bits_h2(cc.x)), __low2half2(bits_h2(cc.y)), __high2half2(bits_h2(cc.y)), D); };
            auto hi = [&](uint32_t w) { return two(and_or(w, 0x00F000F0u, p.magic), __low2half2(bits_h2(cc.z)), __high2half2(bits_h2(cc.z)), __low2half2(bits_h2(cc.w)), __high2half2(bits_h2(cc.w)), D); };
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const uint32_t v = r ? (b ? raw.w.w : raw.w.z) : (b ? raw.w.y : raw.w.x), v8 = v >> 8;
                // bytes 0 and 2, bytes 1 and 3: low nibbles, then high nibbles
                put(f, r, b, make_uint4(lo(v), lo(v8), hi(v), hi(v8)));
            }
        }
    }
};

// IQ3_S held as 4-bit codes (formats.cuh, Fmt<T_IQ3S4>): the tile has the Q4_K shape and a weight is d (1 + 2 s) (2 n - 15):
// t = (1 + n / 16) (32 (1 + 2 s)) - 47 (1 + 2 s) = (1 + 2 s) (2 n - 15), an integer below 512 from exact constants, then t d
// (one rounding). The nibble has to sit in the top four mantissa bits here: 1024 + n would need the constant 2063 (1 + 2 s),
// which is no fp16 number.
template <> struct Dec<T_IQ3S4> {
    static constexpr int TAB_BYTES = 0;
    __device__ static void init(void *, int, int) {}
    // the nibbles at bits POS and POS + 16 of w as the half2 (1 + n / 16, 1 + n' / 16)
    template <int POS> __device__ __forceinline__ static __half2 pair(uint32_t w, uint32_t one) {
        return bits_h2(and_or(POS <= 6 ? w << (6 - POS) : w >> (POS - 6), 0x03C003C0u, one));
    }
    // The constants of (row, sub-block) in the warp's scratch, as for Q4_K but of both units: (32 (1 + 2 s), -47 (1 + 2 s)) in a word. Spread over two they took twice the scratch, and a raw slot
    // from items of 128 and 256 tokens (614 to 1125 experts: 3 instead of 4); a unit's at a time took longer. Layers on 512 experts, us, spread / a unit at a time / this:
    // 2000 tokens 473 / 478 / 466, 4210 686 / 686 / 675, 8192 1202 / 1204 / 1199
    static constexpr int SCRATCH = 2 * 16 * 4 * 4;
    __device__ __forceinline__ static void constants(const uint8_t * chunk, int lane, uint8_t * scratch) {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t sc = *reinterpret_cast<const uint32_t *>(chunk + 2048 + 4 * (g + 8 * r)) >> (4 * t);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const __half2 s = bits_h2((((sc >> (16 * u)) & 15u) * 0x00400040u) | 0x3C003C00u);        // the 4-bit scale under the exponent of 1: 1 + s / 16
                reinterpret_cast<uint32_t *>(scratch)[64 * u + lane + 32 * r] = h2_bits(__hfma2(s, __floats2half2_rn(1024.f, -1504.f), __floats2half2_rn(-992.f, 1457.f)));
            }
        }
    }
    struct Pre { uint32_t D[2], one; };
    __device__ __forceinline__ static Pre prep(const uint8_t * chunk, int lane, uint8_t * scratch) {
        constants(chunk, lane, scratch);
        auto d = [&](int row) { return uint32_t(*reinterpret_cast<const unsigned short *>(chunk + 2112 + 2 * row)) * 0x10001u; };
        return Pre{{d(lane >> 2), d((lane >> 2) + 8)}, in_register(0x3C003C00u)};
    }
    struct Raw { uint4 w; uint2 c[2]; };
    template <int J> __device__ __forceinline__ static Raw load(const uint8_t * chunk, int lane, const uint8_t * scratch) {
        const uint2 * c = reinterpret_cast<const uint2 *>(scratch) + 32 * (J >> 1) + 2 * (lane >> 2) + (J & 1);       // both sub-blocks of the step
        return Raw{plane(chunk, J, lane), {c[0], c[16]}};
    }
    template <int J> __device__ __forceinline__ static void step(const Raw & raw, int, const void *, const Pre & p, uint32_t (&f)[16]) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint2 k = raw.c[r];
            const __half2 D = bits_h2(p.D[r]), S0 = __low2half2(bits_h2(k.x)), C0 = __high2half2(bits_h2(k.x)), S1 = __low2half2(bits_h2(k.y)), C1 = __high2half2(bits_h2(k.y));
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const uint32_t v = r ? (b ? raw.w.w : raw.w.z) : (b ? raw.w.y : raw.w.x);
                put(f, r, b, make_uint4(h2_bits(__hmul2(__hfma2(pair<0>(v, p.one), S0, C0), D)), h2_bits(__hmul2(__hfma2(pair<8>(v, p.one), S0, C0), D)),
                                        h2_bits(__hmul2(__hfma2(pair<4>(v, p.one), S1, C1), D)), h2_bits(__hmul2(__hfma2(pair<12>(v, p.one), S1, C1), D))));
            }
        }
    }
};

// ---------------------------------------------------------------------------------------------------------------
// The same tiles without a rounding, for the GEMM that scales its sums itself once per 256 columns: the operand is the integer
// sc q (Q4_K, at most 945) or (1 + 2 s)(2 n - 15) (IQ3_S codes, at most 465), exact in fp16, one logic operation and one
// multiply-add for two weights. consts: what a row's sums of the chunk are multiplied with, fp32 (d, and for Q4_K -32 dmin
// for the sums over the mins: the activation sums that these meet come divided by 32); mins: the fragment of the eight mins of
// a row (16x256b.x1: lane 4 g + t holds positions 4 t .. 4 t + 3 of rows g, g + 8), twice: for the leading and the low halves of the
// activation sums.
template <uint32_t T> struct Exact;
template <> struct Exact<T_Q4_K> {
    static constexpr bool MINS = true;
    static constexpr int SCRATCH = 2 * 16 * 4 * 4;
    struct Pre { uint32_t magic; };
    __device__ __forceinline__ static Pre prep(const uint8_t * chunk, int lane, uint8_t * scratch) {
        const int g = lane >> 2, t = lane & 3;
        const uint32_t * h0 = reinterpret_cast<const uint32_t *>(chunk + 2048 + 16 * g), * h1 = h0 + 32;       // d, dmin | s[12]
        const uint32_t s0 = h0[1], s1 = h1[1], l0 = h0[3], l1 = h1[3], sel = uint32_t(t) * 0x0101u + 0x0400u;
        uint32_t * to = reinterpret_cast<uint32_t *>(scratch) + lane;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t sc0 = u ? (l0 & 0x0F0F0F0Fu) | ((s0 >> 2) & 0x30303030u) : s0, sc1 = u ? (l1 & 0x0F0F0F0Fu) | ((s1 >> 2) & 0x30303030u) : s1;
            const uint32_t v = __byte_perm(sc0, sc1, sel);                  // byte t of either row's word, 16 bits apart
            __half2 sc = __hadd2(bits_h2((v & 0x003F003Fu) | 0x64006400u), __float2half2_rn(-1024.f));
            if (t & 1) sc = __hmul2(sc, __float2half2_rn(0.0625f));
            const __half2 ns = __hmul2(sc, __float2half2_rn(-1024.f));
            to[64 * u] = h2_bits(__lows2half2(sc, ns));
            to[64 * u + 32] = h2_bits(__highs2half2(sc, ns));
        }
        return Pre{in_register(0x64006400u)};
    }
    struct Raw { uint4 w; uint2 c[2]; };
    template <int J> __device__ __forceinline__ static Raw load(const uint8_t * chunk, int lane, const uint8_t * scratch) {
        const uint2 * c = reinterpret_cast<const uint2 *>(scratch) + 32 * (J >> 1) + 2 * (lane >> 2) + (J & 1);
        return Raw{plane(chunk, J, lane), {c[0], c[16]}};
    }
    template <int J> __device__ __forceinline__ static void step(const Raw & raw, int, const void *, const Pre & p, uint32_t (&f)[16]) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint2 k = raw.c[r];
            const __half2 S0 = __low2half2(bits_h2(k.x)), N0 = __high2half2(bits_h2(k.x)), S1 = __low2half2(bits_h2(k.y)), N1 = __high2half2(bits_h2(k.y));
            auto lo = [&](uint32_t w) { return h2_bits(__hfma2(bits_h2(and_or(w, 0x000F000Fu, p.magic)), S0, N0)); };
            auto hi = [&](uint32_t w) { return h2_bits(__hfma2(bits_h2(and_or(w, 0x00F000F0u, p.magic)), S1, N1)); };
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const uint32_t v = r ? (b ? raw.w.w : raw.w.z) : (b ? raw.w.y : raw.w.x), v8 = v >> 8;
                put(f, r, b, make_uint4(lo(v), lo(v8), hi(v), hi(v8)));
            }
        }
    }
    __device__ __forceinline__ static float2 consts(const uint8_t * chunk, int row) {
        const __half2 h = *reinterpret_cast<const __half2 *>(chunk + 2048 + 16 * row);
        return make_float2(__low2float(h), -32.f * __high2float(h));
    }
    __device__ __forceinline__ static void mins(const uint8_t * chunk, int lane, uint32_t (&f)[4]) {
        const int g = lane >> 2;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint4 h = *reinterpret_cast<const uint4 *>(chunk + 2048 + 16 * (g + 8 * r));
            // mins of sub-blocks 0 .. 3 (lanes t = 0, 2) or 4 .. 7 as bytes (src/formats/weight/dequant.cpp:56-64)
            const uint32_t m = lane & 1 ? ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3F3F3F3Fu;
            f[2 * r] = h2_bits(__hadd2(bits_h2(__byte_perm(m, 0x64646464u, 0x4140)), __float2half2_rn(-1024.f)));
            f[2 * r + 1] = h2_bits(__hadd2(bits_h2(__byte_perm(m, 0x64646464u, 0x4342)), __float2half2_rn(-1024.f)));
        }
    }
};
template <> struct Exact<T_IQ3S4> {
    using D = Dec<T_IQ3S4>;
    static constexpr bool MINS = false;
    static constexpr int SCRATCH = D::SCRATCH;
    struct Pre { uint32_t one; };
    __device__ __forceinline__ static Pre prep(const uint8_t * chunk, int lane, uint8_t * scratch) {
        D::constants(chunk, lane, scratch);
        return Pre{in_register(0x3C003C00u)};
    }
    using Raw = D::Raw;
    template <int J> __device__ __forceinline__ static Raw load(const uint8_t * chunk, int lane, const uint8_t * scratch) { return D::load<J>(chunk, lane, scratch); }
    template <int J> __device__ __forceinline__ static void step(const Raw & raw, int, const void *, const Pre & p, uint32_t (&f)[16]) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint2 k = raw.c[r];
            const __half2 S0 = __low2half2(bits_h2(k.x)), C0 = __high2half2(bits_h2(k.x)), S1 = __low2half2(bits_h2(k.y)), C1 = __high2half2(bits_h2(k.y));
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const uint32_t v = r ? (b ? raw.w.w : raw.w.z) : (b ? raw.w.y : raw.w.x);
                put(f, r, b, make_uint4(h2_bits(__hfma2(D::pair<0>(v, p.one), S0, C0)), h2_bits(__hfma2(D::pair<8>(v, p.one), S0, C0)),
                                        h2_bits(__hfma2(D::pair<4>(v, p.one), S1, C1)), h2_bits(__hfma2(D::pair<12>(v, p.one), S1, C1))));
            }
        }
    }
    __device__ __forceinline__ static float2 consts(const uint8_t * chunk, int row) {
        return make_float2(__half2float(*reinterpret_cast<const __half *>(chunk + 2112 + 2 * row)), 0.f);
    }
    __device__ __forceinline__ static void mins(const uint8_t *, int, uint32_t (&)[4]) {}
};

// ---------------------------------------------------------------------------------------------------------------
// The eight 4-bit codes of a word -> their kvalues (exact) times `scale`, in nibble order, through a 256-entry table byte ->
// half2 in shared memory with a copy per lane (no bank conflicts: entry b of lane l at word 32 b + l). Per code byte: a dot product
// of the word's four bytes with 128 at that byte's place and 0 elsewhere makes the address (extraction, scaling and base in one instruction), one load, one product by
// the scale. With a byte permute and a multiply-add for the address: c5, 24 tokens 277 -> 263.5 us a layer; with shift, mask and add gate/up was bound by the integer pipe (332 us, 0.69 of it), byte
// permutes over a codebook in registers take 23 instructions a word, fifteen of them there (370 us).
constexpr int LUT_BYTES = 256 * 32 * 4;
__device__ inline void build_lut(void * tab, int tid, int nthreads) {
    uint32_t * lut = static_cast<uint32_t *>(tab);
    for (int i = tid; i < 256 * 32; i += nthreads) lut[i] = pack_h2(float(c_kvalues_iq4nl[(i >> 5) & 15]), float(c_kvalues_iq4nl[i >> 9]));
}
// the lane's copy: its shared-memory address
__device__ __forceinline__ uint32_t lut_of(const void * tab, int lane) { return uint32_t(__cvta_generic_to_shared(tab)) + 4u * uint32_t(lane); }
__device__ __forceinline__ uint4 lut_word(uint32_t base, uint32_t w, __half2 scale) {
    auto val = [&](uint32_t entry_bytes) {                             // 128, the bytes of an entry, at the code byte's place
        uint32_t v;
        asm("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(__dp4a(w, entry_bytes, base)));
        return h2_bits(__hmul2(bits_h2(v), scale));
    };
    return make_uint4(val(0x00000080u), val(0x00008000u), val(0x00800000u), val(0x80000000u));
}

template <> struct Dec<T_IQ4_XS> {
    static constexpr int SCRATCH = 0;
    static constexpr int TAB_BYTES = LUT_BYTES;
    __device__ static void init(void * tab, int tid, int n) { build_lut(tab, tid, n); }
    // once per chunk: lane t holds fp16(d (ls - 32)) of sub-blocks t and 4 + t, for its two rows
    struct Pre { uint32_t dl[2]; };
    __device__ __forceinline__ static Pre prep(const uint8_t * chunk, int lane, uint8_t *) {
        const int g = lane >> 2, t = lane & 3;
        float dl[2][2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint2 h = *reinterpret_cast<const uint2 *>(chunk + 2048 + 8 * (g + 8 * r));       // d, scales_h | scales_l[4]
            const float d = __half2float(__ushort_as_half((unsigned short)(h.x & 0xffffu)));
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int ib = 4 * u + t, ls = int((h.y >> (4 * ib)) & 15u) | int(((h.x >> (16 + 2 * ib)) & 3u) << 4);
                dl[u][r] = d * float(ls - 32);
            }
        }
        return Pre{{pack_h2(dl[0][0], dl[0][1]), pack_h2(dl[1][0], dl[1][1])}};
    }
    struct Raw { uint4 w; };
    template <int J> __device__ __forceinline__ static Raw load(const uint8_t * chunk, int lane, const uint8_t *) { return Raw{plane(chunk, J, lane)}; }
    template <int J> __device__ __forceinline__ static void step(const Raw & raw, int lane, const void * tab, const Pre & p, uint32_t (&f)[16]) {
        const uint32_t lut = lut_of(tab, lane);
        const int src = (lane & ~3) | (2 * (J & 1));
        const __half2 d0 = bits_h2(__shfl_sync(0xffffffffu, p.dl[J >> 1], src)), d1 = bits_h2(__shfl_sync(0xffffffffu, p.dl[J >> 1], src + 1));
        put(f, 0, 0, lut_word(lut, raw.w.x, __low2half2(d0)));
        put(f, 0, 1, lut_word(lut, raw.w.y, __low2half2(d1)));
        put(f, 1, 0, lut_word(lut, raw.w.z, __high2half2(d0)));
        put(f, 1, 1, lut_word(lut, raw.w.w, __high2half2(d1)));
    }
};

template <> struct Dec<T_IQ4_NL> {
    static constexpr int SCRATCH = 0;
    struct Pre {};
    __device__ __forceinline__ static Pre prep(const uint8_t *, int, uint8_t *) { return Pre{}; }
    static constexpr int TAB_BYTES = LUT_BYTES;
    __device__ static void init(void * tab, int tid, int n) { build_lut(tab, tid, n); }
    struct Raw { uint2 w[2]; __half d[2][2]; };
    template <int J> __device__ __forceinline__ static Raw load(const uint8_t * chunk, int lane, const uint8_t *) {
        const int g = lane >> 2;
        Raw raw;
#pragma unroll
        for (int b = 0; b < 2; ++b) {                                   // the step's two 32-column tiles: the rows' code words and fp16 scales
            const uint8_t * tile = chunk + (2 * J + b) * Fmt<T_IQ4_NL>::TILE;
            raw.w[b] = *reinterpret_cast<const uint2 *>(tile + 8 * lane);
            raw.d[b][0] = *reinterpret_cast<const __half *>(tile + 256 + 2 * g);
            raw.d[b][1] = *reinterpret_cast<const __half *>(tile + 256 + 2 * (g + 8));
        }
        return raw;
    }
    template <int J> __device__ __forceinline__ static void step(const Raw & raw, int lane, const void * tab, const Pre &, uint32_t (&f)[16]) {
        const uint32_t lut = lut_of(tab, lane);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            put(f, 0, b, lut_word(lut, raw.w[b].x, __half2half2(raw.d[b][0])));
            put(f, 1, b, lut_word(lut, raw.w[b].y, __half2half2(raw.d[b][1])));
        }
    }
};

// ---------------------------------------------------------------------------------------------------------------
template <> struct Dec<T_NVFP4G> {
    static constexpr int SCRATCH = 0;
    struct Pre {};
    __device__ __forceinline__ static Pre prep(const uint8_t *, int, uint8_t *) { return Pre{}; }
    static constexpr int TAB_BYTES = 0;
    __device__ static void init(void *, int, int) {}
    // the eight e2m1 codes of a word -> eight fp16 values (the hardware conversion, two codes per instruction: low nibble
    // first) times `scale`; every product of an e2m1 and an e4m3 value is exact in fp16
    __device__ __forceinline__ static uint4 word(uint32_t w, __half2 scale) {
        uint32_t v0, v1, v2, v3;
        asm("{\n .reg .b8 b0, b1, b2, b3;\n mov.b32 {b0, b1, b2, b3}, %4;\n cvt.rn.f16x2.e2m1x2 %0, b0;\n cvt.rn.f16x2.e2m1x2 %1, b1;\n"
            " cvt.rn.f16x2.e2m1x2 %2, b2;\n cvt.rn.f16x2.e2m1x2 %3, b3;\n}" : "=r"(v0), "=r"(v1), "=r"(v2), "=r"(v3) : "r"(w));
        return make_uint4(h2_bits(__hmul2(bits_h2(v0), scale)), h2_bits(__hmul2(bits_h2(v1), scale)), h2_bits(__hmul2(bits_h2(v2), scale)),
                          h2_bits(__hmul2(bits_h2(v3), scale)));
    }
    struct Raw { uint4 w; uint32_t sc[2]; };
    template <int J> __device__ __forceinline__ static Raw load(const uint8_t * chunk, int lane, const uint8_t *) {
        const uint8_t * tile = chunk + (J >> 1) * Fmt<T_NVFP4G>::TILE;      // a unit is one 128-column tile; plane P = sub-blocks 2 P, 2 P + 1 of it
        constexpr int P = J & 1;
        const uint8_t * sc = tile + 1024 + 8 * (lane >> 2) + 4 * P;
        return Raw{plane(tile, P, lane), {*reinterpret_cast<const uint32_t *>(sc), *reinterpret_cast<const uint32_t *>(sc + 64)}};
    }
    template <int J> __device__ __forceinline__ static void step(const Raw & raw, int lane, const void *, const Pre &, uint32_t (&f)[16]) {
        const uint32_t sel = (lane & 3) < 2 ? 0x4420u : 0x4431u;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            // E4M3 scales of sub-blocks 2 P (bytes 0, 1) and 2 P + 1 (bytes 2, 3); the 16-weight group of word t is t / 2
            const uint32_t two = __byte_perm(raw.sc[r], 0u, sel);
            const __half2 s = __half2(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)two, __NV_E4M3));
            put(f, r, 0, word(r ? raw.w.z : raw.w.x, __low2half2(s)));
            put(f, r, 1, word(r ? raw.w.w : raw.w.y, __high2half2(s)));
        }
    }
};

// ---------------------------------------------------------------------------------------------------------------
template <> struct Dec<T_IQ3_S> {
    static constexpr int SCRATCH = 0;
    struct Pre {};
    __device__ __forceinline__ static Pre prep(const uint8_t *, int, uint8_t *) { return Pre{}; }
    // table: grid entry -> its four odd magnitudes as fp16 (8 bytes)
    static constexpr int TAB_BYTES = 512 * 8;
    __device__ static void init(void * tab, int tid, int n) {
        uint2 * t2 = static_cast<uint2 *>(tab);
        for (int i = tid; i < 512; i += n) {
            const uint32_t m = c_iq3s_grid[i];
            t2[i] = make_uint2(pack_h2(float(m & 255u), float((m >> 8) & 255u)), pack_h2(float((m >> 16) & 255u), float(m >> 24)));
        }
    }
    struct Raw { const uint8_t * chunk; };                               // (a step's words would take thirteen registers)
    template <int J> __device__ __forceinline__ static Raw load(const uint8_t * chunk, int, const uint8_t *) { return Raw{chunk}; }
    template <int J> __device__ __forceinline__ static void step(const Raw & raw, int lane, const void * tab, const Pre &, uint32_t (&f)[16]) {
        const uint8_t * chunk = raw.chunk;
        const int g = lane >> 2;
        const uint2 * mags = static_cast<const uint2 *>(tab);
        uint32_t w[13];
        {
            const uint4 p0 = reinterpret_cast<const uint4 *>(chunk)[lane], p1 = reinterpret_cast<const uint4 *>(chunk + 512)[lane],
                        p2 = reinterpret_cast<const uint4 *>(chunk + 1024)[lane];
            w[0] = p0.x; w[1] = p0.y; w[2] = p0.z; w[3] = p0.w; w[4] = p1.x; w[5] = p1.y; w[6] = p1.z; w[7] = p1.w;
            w[8] = p2.x; w[9] = p2.y; w[10] = p2.z; w[11] = p2.w;
            w[12] = reinterpret_cast<const uint32_t *>(chunk + 1536)[lane];
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int row = g + 8 * r;
            const uint32_t scales = *reinterpret_cast<const uint32_t *>(chunk + 1664 + 4 * row);
            const __half2 d2 = __half2half2(__ushort_as_half(*reinterpret_cast<const unsigned short *>(chunk + 1728 + 2 * row)));
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int ib = 2 * J + b;
                const __half2 s2 = __float2half2_rn(float(1 + 2 * int((scales >> (4 * ib)) & 15u)));      // 1 + 2 s: exact
                const uint32_t sg = r ? w[11 + (ib >> 2)] : w[9 + (ib >> 2)];
                uint32_t o[4];
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) {
                    // entry n = 16 r + 2 ib + jj of the lane's 9-bit stream; r = 1 starts at bit 144 = word 4, bit 16
                    const int n0 = 2 * ib + jj;
                    const int bitA = 9 * n0, bitB = 9 * (16 + n0);
                    const uint32_t ia = (((bitA & 31) > 23 ? __funnelshift_r(w[bitA >> 5], w[(bitA >> 5) + 1], bitA & 31) : w[bitA >> 5] >> (bitA & 31))) & 511u;
                    const uint32_t ibx = (((bitB & 31) > 23 ? __funnelshift_r(w[bitB >> 5], w[(bitB >> 5) + 1 > 8 ? 8 : (bitB >> 5) + 1], bitB & 31) : w[bitB >> 5] >> (bitB & 31))) & 511u;
                    const uint32_t idx = r ? ibx : ia;
                    const uint2 m = mags[idx];
                    const int R = 2 * (ib & 3) + jj;
                    // (mag x (1 + 2 s)) exact (<= 465), x d: one rounding; then the sign bits of the pairs (0, 1) and (2, 3)
                    o[2 * jj] = h2_bits(__hmul2(__hmul2(bits_h2(m.x), s2), d2)) ^ ((sg << (15 - R)) & 0x80008000u);
                    o[2 * jj + 1] = h2_bits(__hmul2(__hmul2(bits_h2(m.y), s2), d2)) ^ ((R <= 7 ? sg << (7 - R) : sg >> (R - 7)) & 0x80008000u);
                }
                put(f, r, b, make_uint4(o[0], o[1], o[2], o[3]));
            }
        }
    }
};

}  // namespace gdec
}  // namespace b2
