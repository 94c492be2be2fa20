// Device-side pieces of the blockwise quantiser and of the bf16 rotary embedding, shared by the quantiser / cache-write
// kernels (quant.cu) and by the decode kernel that writes a step's new token itself (decode_tc.cu).  One definition, so
// that every writer produces the same codes and scales bit for bit.
#pragma once
#include <cuda_bf16.h>

#include "hs_common.cuh"

namespace hs {

__device__ __forceinline__ float code8(int i) { return __fdiv_rn(static_cast<float>(i) - 127.0f, 127.0f); }
__device__ __forceinline__ float mid8(int j) { return __fmul_rn(0.5f, __fadd_rn(code8(j), code8(j + 1))); }

// Index of y in the 8-bit linear codebook.  The candidate round(y*127)+127 is exact unless y*127 sits
// within 1e-3 of a half-integer; only then are the true f32 midpoints consulted (smid: the 255 midpoints in shared
// memory, so the rare path costs two loads and not four divisions for every lane of the warp).
// (rounding by the magic-number add: t + 1.5 * 2^23 is round-to-nearest-even of t in the low mantissa bits for |t| < 2^22 -
// the same integer rintf gives - at full rate, where rintf and the float -> int conversion run on the quarter-rate pipe)
__device__ __forceinline__ int index_int8(float y, const float *smid) {
    float t = __fmul_rn(y, 127.0f);
    const float tm = __fadd_rn(t, 12582912.0f);
    const float r = __fadd_rn(tm, -12582912.0f);
    int c = max(0, min(255, __float_as_int(tm) - 0x4B400000 + 127));
    if (fabsf(t - r) > 0.499f) {  // within 1e-3 of a half-integer
        if (c > 0 && !(y > smid[c - 1])) c--;
        else if (c < 255 && y > smid[c]) c++;
    }
    return c;
}

// The same index with the midpoints worked out on the spot (two IEEE divisions, on the rare tie path only): for a caller
// that has no table in shared memory.  mid8 is the function the table is filled from, so the results are identical.
__device__ __forceinline__ int index_int8_direct(float y) {
    float t = __fmul_rn(y, 127.0f);
    const float tm = __fadd_rn(t, 12582912.0f);
    const float r = __fadd_rn(tm, -12582912.0f);
    int c = max(0, min(255, __float_as_int(tm) - 0x4B400000 + 127));
    if (fabsf(t - r) > 0.499f) {
        if (c > 0 && !(y > mid8(c - 1))) c--;
        else if (c < 255 && y > mid8(c)) c++;
    }
    return c;
}

// ---- index of y in a 16-entry ascending codebook: the number of its 15 midpoints strictly below y ----
// [-1, 1] is cut into buckets of 1/16 whose edges lie at (i + 1/8) / 16: at least 0.07 / 16 away from every midpoint of either
// codebook, so the rounding of the bucket arithmetic cannot move y across an edge that matters, and a bucket holds at most one
// midpoint.  Index = midpoints below the bucket + (y > the bucket's own midpoint).  Values outside [-1, 1] clamp to the first or
// last bucket, whose comparison gives 0 or 15; a NaN goes to the first one and compares false: 0, as counting gives.
constexpr int kIndexBuckets = 33;
struct IndexEntry { float mid; int below; };
struct IndexBuckets { IndexEntry e[kIndexBuckets]; };
constexpr IndexBuckets make_index_buckets(bool nf4) {
    const float t[16] = {nf4 ? -1.0f : 0.0f, nf4 ? -0.6961928009986877f : 0.0625f, nf4 ? -0.5250730514526367f : 0.125f,
                         nf4 ? -0.39491748809814453f : 0.1875f, nf4 ? -0.28444138169288635f : 0.25f, nf4 ? -0.18477343022823334f : 0.3125f,
                         nf4 ? -0.09105003625154495f : 0.375f, nf4 ? 0.0f : 0.4375f, nf4 ? 0.07958029955625534f : 0.5f,
                         nf4 ? 0.16093020141124725f : 0.5625f, nf4 ? 0.24611230945587158f : 0.625f, nf4 ? 0.33791524171829224f : 0.6875f,
                         nf4 ? 0.44070982933044434f : 0.75f, nf4 ? 0.5626170039176941f : 0.8125f, nf4 ? 0.7229568362236023f : 0.875f, 1.0f};
    IndexBuckets b{};
    for (int i = 0; i < kIndexBuckets; ++i) {  // bucket i: 16 y in [i - 16.875, i - 15.875)
        b.e[i].mid = __builtin_huge_valf();
        b.e[i].below = 0;
        for (int j = 0; j < 15; ++j) {
            const float m = 0.5f * (t[j] + t[j + 1]);
            if (16.0f * m < i - 16.875f) b.e[i].below++;
            else if (16.0f * m < i - 15.875f) b.e[i].mid = m;
        }
    }
    return b;
}
static __device__ __constant__ IndexBuckets c_index_nf4 = make_index_buckets(true);
static __device__ __constant__ IndexBuckets c_index_fp4 = make_index_buckets(false);

// What index lookups need in shared memory; fill() by all threads of a block of at least 255, then a block barrier.
// 4-bit: every lane has a column of its own (no bank conflicts whatever the values); a lookup is a multiply-add to the bucket, a
// multiply-add to the address, an 8-byte load and one comparison, where counting took 15 loads and comparisons.
template <int KIND>
struct IndexTable {
    IndexEntry e[kIndexBuckets][32];
    __device__ __forceinline__ void fill() {
        const IndexBuckets &src = KIND == HS_KV_NF4 ? c_index_nf4 : c_index_fp4;
        for (int i = threadIdx.x; i < kIndexBuckets * 32; i += blockDim.x) e[i >> 5][i & 31] = src.e[i >> 5];
    }
    __device__ __forceinline__ int operator()(float y) const {
        const float t = fmaf(fminf(fmaxf(y, -1.0f), 1.0f), 16.0f, 16.375f) + 12582912.0f;  // nearest integer, in the low mantissa bits
        const IndexEntry v = e[__float_as_int(t) - 0x4B400000][threadIdx.x & 31];
        return v.below + (y > v.mid ? 1 : 0);
    }
};
template <>
struct IndexTable<HS_KV_INT8> {
    float mid[256];
    __device__ __forceinline__ void fill() {
        if (threadIdx.x < 255) mid[threadIdx.x] = mid8(threadIdx.x);
    }
    __device__ __forceinline__ int operator()(float y) const { return index_int8(y, mid); }
};
template <>
struct IndexTable<HS_KV_BF16> {  // nothing to look up
    __device__ __forceinline__ void fill() {}
    __device__ __forceinline__ int operator()(float) const { return 0; }
};
struct IndexDirect {  // u8 codes without a table
    __device__ __forceinline__ int operator()(float y) const { return index_int8_direct(y); }
};

// Codebook values of 8 consecutive codes; fill() by all threads, then a block barrier.
template <int KIND>
struct ValueTable {
    float v[16][32];  // a column per lane
    __device__ __forceinline__ void fill() {
        for (int i = threadIdx.x; i < 16 * 32; i += blockDim.x) v[i >> 5][i & 31] = KIND == HS_KV_NF4 ? c_nf4[i >> 5] : c_fp4[i >> 5];
    }
    __device__ __forceinline__ float value(int c) const { return v[c][threadIdx.x & 31]; }
    __device__ __forceinline__ void values8(uint2 w, float (&x)[8]) const {
        const char *col = reinterpret_cast<const char *>(&v[0][threadIdx.x & 31]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {  // the even element sits in the high nibble; entries are 128 bytes apart
            const int at = 8 * (i >> 1) + (i & 1 ? 0 : 4);  // bit position of the nibble
            const uint32_t off = (at >= 7 ? w.x >> (at - 7) : w.x << (7 - at)) & (15u << 7);
            x[i] = *reinterpret_cast<const float *>(col + off);
        }
    }
};
template <>
struct ValueTable<HS_KV_BF16> {  // nothing to look up
    __device__ __forceinline__ void fill() {}
};
template <>
struct ValueTable<HS_KV_INT8> {
    float v[256];
    __device__ __forceinline__ void fill() {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) v[i] = code8(i);
    }
    __device__ __forceinline__ float value(int c) const { return v[c]; }
    __device__ __forceinline__ void values8(uint2 w, float (&x)[8]) const {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = v[((i < 4 ? w.x : w.y) >> (8 * (i & 3))) & 0xffu];
    }
};

__device__ __forceinline__ float f16_sat_round(float a) {
    // nearest-even to f16, saturating: anything that would round past 65504 stays 65504
    return a >= 65520.0f ? 65504.0f : __half2float(__float2half_rn(a));
}

// two fp32 values as one operand of the packed fp32 instructions (each half is rounded as the scalar instruction rounds it)
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// code words of N elements: 4 u8 codes a word, or 8 4-bit codes a word (the even element in the high nibble of its byte)
template <int KIND, int N>
struct CodeWords {
    static constexpr int kCount = KIND == HS_KV_INT8 ? N / 4 : N / 8;
    uint32_t w[kCount];
    __device__ __forceinline__ int code(int i) const {
        return KIND == HS_KV_INT8 ? (w[i >> 2] >> (8 * (i & 3))) & 0xff : (w[i >> 3] >> (8 * ((i >> 1) & 3) + (i & 1 ? 0 : 4))) & 0xf;
    }
};

// ---- quantise the N values of a thread; `tpb` consecutive lanes (a power of two <= 32) share a block ----
// Returns the stored scale (already rounded in f16 mode); `cw` receives N indices.
//
// u8 codes, two values per instruction: t = x (127 / absmax), and t + (1.5 * 2^23 + 127) holds the candidate code in its low byte
// (a NaN's low byte is 255, the index the scalar form gives it).  Only where a candidate's t lies within 1e-4 of a half-integer
// (the roundings are off by less than 4e-5) are the true midpoints consulted, value by value; so is a block whose values leave
// [-1, 1].  That path is a call: inlined 16 times it made the write kernel miss the instruction cache.
template <typename Index>
__device__ __noinline__ uint32_t index_int8_word(float x0, float x1, float x2, float x3, float inv, const Index &index) {
    return static_cast<uint32_t>(index(__fmul_rn(x0, inv))) | static_cast<uint32_t>(index(__fmul_rn(x1, inv))) << 8 |
           static_cast<uint32_t>(index(__fmul_rn(x2, inv))) << 16 | static_cast<uint32_t>(index(__fmul_rn(x3, inv))) << 24;
}

// The codes of the N values of this thread, given the largest magnitude of their block (over all its lanes).
template <int KIND, int N, typename Index>
__device__ __forceinline__ float quantize_given_max(const float (&x)[N], float amax, int scale_dtype, const Index &index, CodeWords<KIND, N> &cw) {
    const float a = scale_dtype == HS_SCALE_F16 ? f16_sat_round(amax) : amax;
    if (a == 0.0f) {
        const uint32_t zw = KIND == HS_KV_INT8 ? 0x7f7f7f7fu : (KIND == HS_KV_NF4 ? 0x77777777u : 0u);
#pragma unroll
        for (int i = 0; i < CodeWords<KIND, N>::kCount; ++i) cw.w[i] = zw;
        return a;
    }
    const float inv = __fdiv_rn(1.0f, a);
    if constexpr (KIND == HS_KV_INT8) {
        const float inv127 = __fmul_rn(inv, 127.0f);
        const uint64_t scale = f2_pack(inv127, inv127), magic = f2_pack(12583039.0f, 12583039.0f), unmagic = f2_pack(-12583039.0f, -12583039.0f),
                       minus1 = f2_pack(-1.0f, -1.0f);
        // a scale that f16 cut short, or a reciprocal that overflows, lets t leave the range in which the low byte is the code
        const float wide = __fmul_rn(amax, inv127) > 127.3f ? 1.0f : 0.0f;
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const uint64_t t0 = f2_mul(f2_pack(x[i], x[i + 1]), scale), t1 = f2_mul(f2_pack(x[i + 2], x[i + 3]), scale);
            const uint64_t m0 = f2_add(t0, magic), m1 = f2_add(t1, magic);
            float b[4], d[4];
            f2_unpack(m0, b[0], b[1]);
            f2_unpack(m1, b[2], b[3]);
            f2_unpack(f2_fma(f2_add(m0, unmagic), minus1, t0), d[0], d[1]);
            f2_unpack(f2_fma(f2_add(m1, unmagic), minus1, t1), d[2], d[3]);
            const uint32_t lo = __byte_perm(__float_as_uint(b[0]), __float_as_uint(b[1]), 0x0040), hi = __byte_perm(__float_as_uint(b[2]), __float_as_uint(b[3]), 0x0040);
            cw.w[i / 4] = __byte_perm(lo, hi, 0x5410);
            const float off = fmaxf(fmaxf(fmaxf(wide, fabsf(d[0])), fabsf(d[1])), fmaxf(fabsf(d[2]), fabsf(d[3])));
            if (off > 0.4999f) cw.w[i / 4] = index_int8_word(x[i], x[i + 1], x[i + 2], x[i + 3], inv, index);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 8) {
            uint32_t w = 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) w += static_cast<uint32_t>(index(__fmul_rn(x[i + e], inv))) << (8 * (e >> 1) + (e & 1 ? 0 : 4));
            cw.w[i / 8] = w;
        }
    }
    return a;
}
template <int KIND, int N, typename Index>
__device__ __forceinline__ float quantize_n(const float (&x)[N], int tpb, int scale_dtype, const Index &index, CodeWords<KIND, N> &cw) {
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) amax = fmaxf(amax, fabsf(x[i]));
    for (int o = 1; o < tpb; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    return quantize_given_max<KIND, N>(x, amax, scale_dtype, index, cw);
}
// largest magnitude of 8 bf16 values (a NaN is passed over, as fmaxf passes over it)
__device__ __forceinline__ float absmax8_bf16(const uint4 &w) {
    const uint32_t ww[4] = {w.x & 0x7fff7fffu, w.y & 0x7fff7fffu, w.z & 0x7fff7fffu, w.w & 0x7fff7fffu};
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(ww);
    const __nv_bfloat162 m = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    return fmaxf(fmaxf(__low2float(m), __high2float(m)), 0.0f);
}

__device__ __forceinline__ void store_scale(void *p, int64_t idx, int scale_dtype, float a) {
    if (scale_dtype == HS_SCALE_F16) reinterpret_cast<__half *>(p)[idx] = __float2half_rn(a);
    else reinterpret_cast<float *>(p)[idx] = a;
}

__device__ __forceinline__ float load_elem(const void *src, int dtype, int64_t i) {
    if (dtype == HS_DTYPE_BF16) return bf16_bits_to_f32(reinterpret_cast<const uint16_t *>(src)[i]);
    if (dtype == HS_DTYPE_F16) return __half2float(reinterpret_cast<const __half *>(src)[i]);
    return reinterpret_cast<const float *>(src)[i];
}

__device__ __forceinline__ void unpack8_bf16(const uint4 &w, float (&x)[8]) {
    x[0] = bf16lo(w.x); x[1] = bf16hi(w.x); x[2] = bf16lo(w.y); x[3] = bf16hi(w.y);
    x[4] = bf16lo(w.z); x[5] = bf16hi(w.z); x[6] = bf16lo(w.w); x[7] = bf16hi(w.w);
}

template <int KIND>
__device__ __forceinline__ void store_codes8(uint8_t *codes, int64_t e0, int64_t n, const CodeWords<KIND, 8> &c, bool full) {
    if (KIND == HS_KV_INT8) {
        if (full) *reinterpret_cast<uint2 *>(codes + e0) = make_uint2(c.w[0], c.w[CodeWords<KIND, 8>::kCount - 1]);
        else for (int i = 0; i < 8 && e0 + i < n; ++i) codes[e0 + i] = static_cast<uint8_t>(c.code(i));
    } else {
        if (full) *reinterpret_cast<uint32_t *>(codes + (e0 >> 1)) = c.w[0];
        else
            for (int i = 0; i < 8 && e0 + i < n; i += 2)
                codes[(e0 + i) >> 1] = static_cast<uint8_t>((c.code(i) << 4) | (e0 + i + 1 < n ? c.code(i + 1) : 0));
    }
}

// ---- RoPE ------------------------------------------------------------------------------------------
// Every product, difference and sum is rounded to bf16 (rope.rs:243-244).
// The rotation on packed bf16 pairs: a product of two bf16 values is exact in fp32, so mul.rn.bf16x2 rounds it once exactly as
// "multiply in fp32, round to bf16" does, and the difference / sum of two bf16 values rounds to the same bf16 either way - three
// instructions per pair instead of an unpack, three roundings and two multiplies per element.
__device__ __forceinline__ uint32_t rope_pair(uint32_t own, uint32_t partner, uint32_t s, uint32_t c, bool first_half) {
    const __nv_bfloat162 o = *reinterpret_cast<const __nv_bfloat162 *>(&own), p = *reinterpret_cast<const __nv_bfloat162 *>(&partner);
    const __nv_bfloat162 s2 = *reinterpret_cast<const __nv_bfloat162 *>(&s), c2 = *reinterpret_cast<const __nv_bfloat162 *>(&c);
    const __nv_bfloat162 oc = __hmul2_rn(o, c2), ps = __hmul2_rn(p, s2);  // (_rn: never fused with the sum, which would skip a rounding)
    const __nv_bfloat162 r = first_half ? __hsub2_rn(oc, ps) : __hadd2_rn(ps, oc);  // x1*cos - x2*sin | x1*sin + x2*cos
    return *reinterpret_cast<const uint32_t *>(&r);
}
// 8 consecutive values of a sin and a cos row (any alignment of the tables)
__device__ __forceinline__ void load_sincos8(const uint16_t *srow, const uint16_t *crow, uint32_t (&sw)[4], uint32_t (&cw)[4]) {
    if (((reinterpret_cast<uintptr_t>(srow) | reinterpret_cast<uintptr_t>(crow)) & 15u) == 0) {
        const uint4 s4 = *reinterpret_cast<const uint4 *>(srow), c4 = *reinterpret_cast<const uint4 *>(crow);
        sw[0] = s4.x; sw[1] = s4.y; sw[2] = s4.z; sw[3] = s4.w;
        cw[0] = c4.x; cw[1] = c4.y; cw[2] = c4.z; cw[3] = c4.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            sw[i] = static_cast<uint32_t>(srow[2 * i]) | (static_cast<uint32_t>(srow[2 * i + 1]) << 16);
            cw[i] = static_cast<uint32_t>(crow[2 * i]) | (static_cast<uint32_t>(crow[2 * i + 1]) << 16);
        }
    }
}

// The 8 bf16 elements [d0, d0+8) of a row, rotated when sin != NULL.
__device__ __forceinline__ uint4 row8_rope(const uint16_t *row, int d0, const uint16_t *sin, const uint16_t *cos, int pos, int rotary_dim) {
    uint4 ow = *reinterpret_cast<const uint4 *>(row + d0);
    if (sin != nullptr && d0 < rotary_dim) {
        const int half = rotary_dim >> 1;
        const bool first = d0 < half;
        const uint4 pw = *reinterpret_cast<const uint4 *>(row + (first ? d0 + half : d0 - half));
        const int j0 = first ? d0 : d0 - half;
        uint32_t sw[4], cw[4];
        load_sincos8(sin + static_cast<int64_t>(pos) * half + j0, cos + static_cast<int64_t>(pos) * half + j0, sw, cw);
        ow.x = rope_pair(ow.x, pw.x, sw[0], cw[0], first); ow.y = rope_pair(ow.y, pw.y, sw[1], cw[1], first);
        ow.z = rope_pair(ow.z, pw.z, sw[2], cw[2], first); ow.w = rope_pair(ow.w, pw.w, sw[3], cw[3], first);
    }
    return ow;
}
__device__ __forceinline__ void load_row8_rope(const uint16_t *row, int d0, const uint16_t *sin, const uint16_t *cos,
                                               int pos, int rotary_dim, float (&x)[8]) {
    unpack8_bf16(row8_rope(row, d0, sin, cos, pos, rotary_dim), x);
}

}  // namespace hs
