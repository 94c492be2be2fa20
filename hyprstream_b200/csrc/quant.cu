// Blockwise KV quantiser for sm_100a: flat quantise / dequantise, RoPE, quantise-on-write into a
// (paged) cache view, and the gather-dequantise compatibility read.
//
// Arithmetic contract (bit-exact with the CPU specification used by the parity tests):
//   absmax = max|x| over the block in f32; in f16-scale mode it is rounded to f16 (nearest even,
//   saturating at 65504) before use;  y = x * (1/absmax), one IEEE rounding each;
//   index = number of f32 codeword midpoints 0.5*(c[j]+c[j+1]) strictly below y;
//   an all-zero block stores absmax 0 and the index of the codeword 0;
//   4-bit codes pack the even element into the high nibble.
// Codebooks and block geometry follow bitsandbytes-sys/src/lib.rs:104-181 and
// crates/hyprstream/src/runtime/kv_cache.rs:704,741-957.
//
// All kernels here are HBM-streaming: a thread owns chunks of 8 (16) consecutive elements with 16-byte loads and stores,
// a block's absmax is reduced with warp shuffles, nothing is staged.
#include "hs_common.cuh"
#include "quant_dev.cuh"

namespace hs {

constexpr int kQThreads = 256;
constexpr int kWriteElems = 64;  // elements per thread of the quantise-on-write kernel (as 8- or 16-element chunks)

// ---- flat quantise ----------------------------------------------------------------------------
// HBM streaming by design.  A thread takes kFlatChunks chunks of 8 elements, all of them loaded before the first is worked on
// (one chunk per thread left too few bytes in flight), 16-byte loads for every dtype, and a 4-bit index is one lookup instead
// of 15 comparisons (quant_dev.cuh): 20 M bf16 elements to NF4 47.7 -> 25.2 us (50 MB, 7.7 us at the copy rate).
constexpr int kFlatChunks = 4;

template <int DTYPE>
__device__ __forceinline__ void load_chunk8(const void *src, int64_t e0, int64_t n, bool vec, float (&x)[8]) {
    if (vec && e0 + 8 <= n) {
        if constexpr (DTYPE == HS_DTYPE_F32) {
            const float4 *p = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(src) + e0);
            const float4 a = p[0], b = p[1];
            x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
        } else {
            const uint4 w = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(src) + e0);
            if constexpr (DTYPE == HS_DTYPE_BF16) {
                unpack8_bf16(w, x);
            } else {
                const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&ww[i]));
                    x[2 * i] = f.x; x[2 * i + 1] = f.y;
                }
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = (e0 + i < n) ? load_elem(src, DTYPE, e0 + i) : 0.0f;
    }
}

template <int KIND, int DTYPE>
__global__ void __launch_bounds__(kQThreads) quantize_flat_kernel(const void *__restrict__ src, int64_t n,
                                                                  int block, int scale_dtype, uint8_t *__restrict__ codes,
                                                                  void *__restrict__ absmax, int vec_ok) {
    __shared__ IndexTable<KIND> tab;
    tab.fill();
    __syncthreads();
    const int64_t chunk0 = static_cast<int64_t>(blockIdx.x) * (kQThreads * kFlatChunks) + threadIdx.x;
    const int tpb = block / 8, block_shift = __ffs(block) - 1;
    float x[kFlatChunks][8];
#pragma unroll
    for (int u = 0; u < kFlatChunks; ++u) load_chunk8<DTYPE>(src, (chunk0 + u * kQThreads) * 8, n, vec_ok != 0, x[u]);
#pragma unroll
    for (int u = 0; u < kFlatChunks; ++u) {
        const int64_t chunk = chunk0 + u * kQThreads, e0 = chunk * 8;
        CodeWords<KIND, 8> c;
        const float a = quantize_n<KIND, 8>(x[u], tpb, scale_dtype, tab, c);
        if (e0 < n) {
            if ((threadIdx.x & (tpb - 1)) == 0) store_scale(absmax, e0 >> block_shift, scale_dtype, a);
            store_codes8<KIND>(codes, e0, n, c, e0 + 8 <= n);
        }
    }
}

// ---- flat dequantise ----------------------------------------------------------------------------
__device__ __forceinline__ void store_elem(void *out, int dtype, int64_t i, float v) {
    if (dtype == HS_DTYPE_BF16) reinterpret_cast<uint16_t *>(out)[i] = f32_to_bf16_bits(v);
    else if (dtype == HS_DTYPE_F16) reinterpret_cast<__half *>(out)[i] = __float2half_rn(v);
    else reinterpret_cast<float *>(out)[i] = v;
}

// A thread takes kFlatChunks chunks of 8 elements: whole-word loads of the codes, 16-byte stores (element-wise only at the end
// of the tensor and for buffers that are not aligned for it).  The 8-bit codebook is worked out ((code - 127) / 127, one IEEE
// division: a 256-entry table in shared memory), the 4-bit ones are looked up in a table that every lane has a column of.
// 20 M NF4 elements to bf16 53.9 -> 13.6 us (single 2-byte stores before).
template <int KIND, int DTYPE>
__global__ void __launch_bounds__(kQThreads) dequantize_flat_kernel(const uint8_t *__restrict__ codes,
                                                                    const void *__restrict__ absmax, int64_t n, int block,
                                                                    int scale_dtype, void *__restrict__ out, int vec_ok) {
    __shared__ ValueTable<KIND> tab;
    tab.fill();
    __syncthreads();
    const int64_t chunk0 = static_cast<int64_t>(blockIdx.x) * (kQThreads * kFlatChunks) + threadIdx.x;
    const bool pow2 = (block & (block - 1)) == 0;
    const int block_shift = __ffs(block) - 1;
    uint2 w[kFlatChunks];
    float a[kFlatChunks];
#pragma unroll
    for (int u = 0; u < kFlatChunks; ++u) {
        const int64_t e0 = (chunk0 + u * kQThreads) * 8;
        w[u] = make_uint2(0u, 0u);
        a[u] = 0.0f;
        if (e0 < n) {
            a[u] = load_scale(absmax, pow2 ? e0 >> block_shift : e0 / block, scale_dtype);
            if (vec_ok && e0 + 8 <= n) {
                if constexpr (KIND == HS_KV_INT8) w[u] = *reinterpret_cast<const uint2 *>(codes + e0);
                else w[u].x = *reinterpret_cast<const uint32_t *>(codes + (e0 >> 1));
            }
        }
    }
#pragma unroll
    for (int u = 0; u < kFlatChunks; ++u) {
        const int64_t e0 = (chunk0 + u * kQThreads) * 8;
        if (e0 >= n) return;
        if (vec_ok && e0 + 8 <= n) {
            float v[8];
            tab.values8(w[u], v);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(v[i], a[u]);
            if constexpr (DTYPE == HS_DTYPE_F32) {
                float4 *p = reinterpret_cast<float4 *>(reinterpret_cast<float *>(out) + e0);
                p[0] = make_float4(v[0], v[1], v[2], v[3]);
                p[1] = make_float4(v[4], v[5], v[6], v[7]);
            } else {
                uint32_t o[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if constexpr (DTYPE == HS_DTYPE_BF16) {
                        o[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
                    } else {
                        const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
                        o[i] = *reinterpret_cast<const uint32_t *>(&h);
                    }
                }
                *reinterpret_cast<uint4 *>(reinterpret_cast<uint16_t *>(out) + e0) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        } else {
            for (int i = 0; i < 8 && e0 + i < n; ++i) {
                const int64_t e = e0 + i;
                const int c = KIND == HS_KV_INT8 ? codes[e] : ((e & 1) ? (codes[e >> 1] & 0xf) : (codes[e >> 1] >> 4));
                store_elem(out, DTYPE, e, __fmul_rn(tab.value(c), a[u]));
            }
        }
    }
}

// ---- RoPE (device helpers in quant_dev.cuh) ------------------------------------------------------------
// A thread takes the 8 elements at j of a head's first rotated half together with their partners in the second half - both are
// read and written once, and one pair of sin / cos loads serves both - or 8 elements that pass through unrotated.  HBM bound: a
// block covers whole rows (one position each) with 32-bit arithmetic; the 64-bit divisions per 8 elements of the earlier form
// were most of its instructions: 65,536 rows of 32 x 128 248 -> 157 us = 6.8 TB/s.
__global__ void __launch_bounds__(kQThreads) rope_kernel(const uint16_t *__restrict__ x, uint16_t *__restrict__ out,
                                                         const uint16_t *__restrict__ sin, const uint16_t *__restrict__ cos,
                                                         const int32_t *__restrict__ positions, int64_t n_rows, int n_heads,
                                                         int head_dim, int rotary_dim, int n_positions, int rows_per_block, int *__restrict__ err) {
    const int half = rotary_dim >> 1;
    const unsigned rot = static_cast<unsigned>(half) / 8u;                               // rotated pairs of chunks per head
    const unsigned upr = rot + static_cast<unsigned>(head_dim - rotary_dim) / 8u;        // work units per head
    const unsigned units = upr * static_cast<unsigned>(n_heads);                         // ... and per row
    const int64_t row0 = static_cast<int64_t>(blockIdx.x) * rows_per_block;
    const unsigned rows = static_cast<unsigned>(min(static_cast<int64_t>(rows_per_block), n_rows - row0));
#pragma unroll 2
    for (unsigned i = threadIdx.x; i < rows * units; i += kQThreads) {
        const unsigned rr = i / units, u = i - rr * units, h = u / upr, c = u - h * upr;
        const int64_t r = row0 + rr;
        const int64_t base = (r * n_heads + h) * head_dim;
        const int pos = positions[r];
        const bool in_table = pos >= 0 && pos < n_positions;
        if (!in_table) atomicOr(err, HS_DEVERR_ROPE_RANGE);  // recorded; the row is copied unrotated
        if (c >= rot) {
            const int64_t at = base + rotary_dim + (c - rot) * 8u;
            *reinterpret_cast<uint4 *>(out + at) = *reinterpret_cast<const uint4 *>(x + at);
            continue;
        }
        const uint4 w1 = *reinterpret_cast<const uint4 *>(x + base + c * 8u), w2 = *reinterpret_cast<const uint4 *>(x + base + half + c * 8u);
        uint32_t o1[4] = {w1.x, w1.y, w1.z, w1.w}, o2[4] = {w2.x, w2.y, w2.z, w2.w};
        if (in_table) {
            uint32_t sw[4], cw[4];
            load_sincos8(sin + static_cast<int64_t>(pos) * half + c * 8u, cos + static_cast<int64_t>(pos) * half + c * 8u, sw, cw);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t a = o1[k], b = o2[k];
                o1[k] = rope_pair(a, b, sw[k], cw[k], true);
                o2[k] = rope_pair(b, a, sw[k], cw[k], false);
            }
        }
        *reinterpret_cast<uint4 *>(out + base + c * 8u) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
        *reinterpret_cast<uint4 *>(out + base + half + c * 8u) = make_uint4(o2[0], o2[1], o2[2], o2[3]);
    }
}

// Optional per-head RMS norm of K fused into quantise-on-write (weight == NULL: off).
struct KNormArgs {
    const float *weight;  // f32 [head_dim]
    float eps;
    int plus_one;         // multiply by (1 + w) instead of w
    uint16_t *k_out;      // optional bf16 [n_seqs, n_tokens, n_kv_heads, head_dim]: the normed, rotated keys
    int pos_bias;         // added to dst_pos[s] (or 0): -1 when the caller hands the attended lengths instead of positions
};

// 8 norm weights, `add` (0 or 1) added to each
__device__ __forceinline__ void load_weight8(const float *w, float add, float (&out)[8]) {
    const float4 a = *reinterpret_cast<const float4 *>(w), b = *reinterpret_cast<const float4 *>(w + 4);
    out[0] = a.x + add; out[1] = a.y + add; out[2] = a.z + add; out[3] = a.w + add;
    out[4] = b.x + add; out[5] = b.y + add; out[6] = b.z + add; out[7] = b.w + add;
}

// ---- quantise-on-write into a cache view ----------------------------------------------------------------
// E = elements per thread: 16 for long writes (prefill: bound by instruction issue, so the per-chunk costs are paid
// half as often), 8 for short ones (a decode step's single token per sequence: latency matters, not throughput).
//
// Issue bound, not HBM bound, as first written (523 warp instructions per 16-element chunk, a fifth of the stalls for
// instruction fetch).  Where a block's rows lie in one page and need no rotation or norm (V always; K that arrives finished) the
// source and the cache have the same layout: one linear copy-and-quantise with all of a thread's loads in flight and no
// (token, head) split; the norm is an instantiation of its own.  3 x 8,192 tokens of 8 x 128 into int8: 77.7 -> 54.9 us.
template <int KIND, int E, bool NORM>
__global__ void __launch_bounds__(kQThreads) kv_write_kernel(ViewDev view, const uint16_t *__restrict__ k_new,
                                                             const uint16_t *__restrict__ v_new, int n_seqs, int n_tokens,
                                                             const int32_t *__restrict__ dst_pos,
                                                             const uint16_t *__restrict__ sin, const uint16_t *__restrict__ cos,
                                                             int rotary_dim, int n_positions, int *__restrict__ err, KNormArgs kn) {
    // a decode launch that follows as a programmatic dependent may start now (it waits for this grid's completion before
    // it reads the cache); a no-op for every other successor
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    EndOfGridWait order;  // (it may itself run beside the QK norm of the same layer)
    __shared__ IndexTable<KIND> tab;
    tab.fill();
    __syncthreads();
    // grid: x = groups of kUnroll * 256 E-element chunks of one sequence's new rows, y = 2 * sequence + (0: K, 1: V).
    // A thread owns E consecutive elements of a (token, head) row (16-byte loads; at E = 16 one 16-byte store of int8
    // codes): the index split, the page division, the pointer loads, the IEEE division of the scale and the shuffles
    // are paid once per chunk.  head_dim and the block are powers of two (64, 128, 256), the number of kv heads usually
    // is: shifts instead of divisions.
    const bool is_v = (blockIdx.y & 1) != 0;
    const int s = static_cast<int>(blockIdx.y >> 1);
    const int D = view.head_dim, H = view.n_kv_heads;
    constexpr int kUnroll = kWriteElems / E;
    const uint32_t cpr = static_cast<uint32_t>(D) / static_cast<uint32_t>(E);
    const uint32_t total = static_cast<uint32_t>(n_tokens) * static_cast<uint32_t>(H) * cpr;
    const int base_pos = (dst_pos ? dst_pos[s] : 0) + kn.pos_bias;
    void *const *data_pages = is_v ? view.v_pages : view.k_pages;
    void *const *scale_pages = is_v ? view.v_scale_pages : view.k_scale_pages;
    const int tpb = view.block / E;
    const int bpr = D / view.block;  // blocks per (token, head) row
    const int cpr_shift = __ffs(static_cast<int>(cpr)) - 1, block_shift = __ffs(view.block) - 1;
    const bool h_pow2 = (H & (H - 1)) == 0, page_pow2 = (view.page_tokens & (view.page_tokens - 1)) == 0;
    const int h_shift = __ffs(H) - 1, page_shift = __ffs(view.page_tokens) - 1;
    if constexpr (E == 16) {
        const uint32_t c0 = blockIdx.x * static_cast<uint32_t>(kUnroll * kQThreads), c1 = min(c0 + static_cast<uint32_t>(kUnroll * kQThreads), total);
        const uint32_t hc = static_cast<uint32_t>(H) * cpr;                 // chunks per token
        const int pos0 = base_pos + static_cast<int>(c0 / hc), pos1 = base_pos + static_cast<int>((c1 - 1u) / hc);
        const int page = pos0 / view.page_tokens;
        if (c0 >= total) return;
        if ((is_v || (!NORM && sin == nullptr)) && base_pos >= 0 && pos1 / view.page_tokens == page && page < view.pages_per_seq) {
            const int64_t pidx = static_cast<int64_t>(s) * view.pages_per_seq + page;
            // element offset between the source rows of this sequence and their place in the page
            const int64_t shift = (static_cast<int64_t>(base_pos) - static_cast<int64_t>(page) * view.page_tokens) * H * D;
            const uint4 *src = reinterpret_cast<const uint4 *>((is_v ? v_new : k_new) + static_cast<int64_t>(s) * n_tokens * H * D);
            uint4 w[kUnroll][2];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const uint32_t chunk = c0 + u * kQThreads + threadIdx.x;
                w[u][0] = w[u][1] = make_uint4(0, 0, 0, 0);
                if (chunk < total) {
                    w[u][0] = src[2 * static_cast<int64_t>(chunk)];
                    w[u][1] = src[2 * static_cast<int64_t>(chunk) + 1];
                }
            }
            uint8_t *data = reinterpret_cast<uint8_t *>(data_pages[pidx]);
            void *scales = KIND == HS_KV_BF16 ? nullptr : scale_pages[pidx];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const uint32_t chunk = c0 + u * kQThreads + threadIdx.x;
                const int64_t e0 = shift + static_cast<int64_t>(chunk) * 16;
                if constexpr (KIND == HS_KV_BF16) {
                    if (chunk < total) {
                        reinterpret_cast<uint4 *>(data + 2 * e0)[0] = w[u][0];
                        reinterpret_cast<uint4 *>(data + 2 * e0)[1] = w[u][1];
                    }
                } else {
                    float amax = fmaxf(absmax8_bf16(w[u][0]), absmax8_bf16(w[u][1]));
                    for (int o = 1; o < tpb; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                    if (chunk >= total) continue;
                    float x[16];
                    unpack8_bf16(w[u][0], *reinterpret_cast<float(*)[8]>(&x[0]));
                    unpack8_bf16(w[u][1], *reinterpret_cast<float(*)[8]>(&x[8]));
                    CodeWords<KIND, 16> c;
                    const float a = quantize_given_max<KIND, 16>(x, amax, view.scale_dtype, tab, c);
                    if ((threadIdx.x & (tpb - 1)) == 0) store_scale(scales, e0 >> block_shift, view.scale_dtype, a);
                    if constexpr (KIND == HS_KV_INT8) *reinterpret_cast<uint4 *>(data + e0) = make_uint4(c.w[0], c.w[1], c.w[2], c.w[3]);
                    else *reinterpret_cast<uint2 *>(data + (e0 >> 1)) = make_uint2(c.w[0], c.w[1]);
                }
            }
            return;
        }
    }
#pragma unroll 1
    for (int u = 0; u < kUnroll; ++u) {
        const uint32_t chunk = (blockIdx.x * static_cast<uint32_t>(kUnroll) + u) * static_cast<uint32_t>(kQThreads) + threadIdx.x;
        if (chunk - threadIdx.x >= total) break;  // (uniform over the block)
        const bool live = chunk < total;
        const uint32_t cc = live ? chunk : 0u;  // dead lanes still take part in the shuffles
        const uint32_t row_in_seq = cc >> cpr_shift;   // (token, head)
        const int d0 = static_cast<int>(cc & (cpr - 1u)) * E;
        const int t = static_cast<int>(h_pow2 ? row_in_seq >> h_shift : row_in_seq / static_cast<uint32_t>(H));
        const int h = static_cast<int>(row_in_seq - static_cast<uint32_t>(t) * static_cast<uint32_t>(H));
        const int64_t row = static_cast<int64_t>(s) * n_tokens * H + row_in_seq;  // (seq, token, head)
        const int pos = base_pos + t;
        const int page = page_pow2 ? pos >> page_shift : pos / view.page_tokens;
        bool ok = live && pos >= 0 && page < view.pages_per_seq;
        if (!is_v && sin != nullptr && (pos < 0 || pos >= n_positions)) ok = false;
        if (live && !ok) atomicOr(err, HS_DEVERR_KV_WRITE_RANGE);  // recorded, access skipped
        const uint16_t *src = (is_v ? v_new : k_new) + row * D;
        float x[E];
        if (NORM && !is_v) {
            // ---- K with its per-head RMS norm fused in (qwen3_5.rs:1077-1091; llama.rs:929-992): the row's sum of squares is
            // formed exactly as hs_qk_norm_rope forms it (an 8-element chain per 16-byte chunk, then pairwise over the chunks
            // of the row), so the normed, rotated values - and with them the stored codes - equal the two-kernel route bit
            // for bit.  Dead and refused lanes carry zeros and still take part in the shuffles.
            float ssq[E / 8];
#pragma unroll
            for (int part = 0; part < E / 8; ++part) {
                float p8[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                if (ok) unpack8_bf16(*reinterpret_cast<const uint4 *>(src + d0 + 8 * part), p8);
                float ss = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) { x[8 * part + i] = p8[i]; ss = fmaf(p8[i], p8[i], ss); }
                ssq[part] = ss;
            }
            float ss = ssq[0];
            if constexpr (E == 16) ss += ssq[1];
            for (uint32_t off = 1; off < cpr; off <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
            const float rrms = rsqrtf(ss * (1.0f / static_cast<float>(D)) + kn.eps);
            const float add = kn.plus_one ? 1.0f : 0.0f;
            const bool rope = sin != nullptr && ok;
            const int half = rotary_dim >> 1;
#pragma unroll
            for (int part = 0; part < E / 8; ++part) {
                const int dd = d0 + 8 * part;
                // the normed chunk as bf16 pairs (one packed conversion per pair = the one rounding to the model dtype), rotated in
                // packed bf16 arithmetic like load_row8_rope: the same values as the scalar form, bit for bit
                float wt[8];
                load_weight8(kn.weight + dd, add, wt);
                uint32_t ow[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) ow[i] = pack_bf16(x[8 * part + 2 * i] * rrms * wt[2 * i], x[8 * part + 2 * i + 1] * rrms * wt[2 * i + 1]);
                if (rope && dd < rotary_dim) {
                    const bool first = dd < half;
                    const int pd = first ? dd + half : dd - half;  // the rotation partner's chunk, normed the same way
                    float p8[8];
                    unpack8_bf16(*reinterpret_cast<const uint4 *>(src + pd), p8);
                    load_weight8(kn.weight + pd, add, wt);
                    const int j0 = first ? dd : dd - half;
                    uint32_t sw[4], cw[4];
                    load_sincos8(sin + static_cast<int64_t>(pos) * half + j0, cos + static_cast<int64_t>(pos) * half + j0, sw, cw);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        ow[i] = rope_pair(ow[i], pack_bf16(p8[2 * i] * rrms * wt[2 * i], p8[2 * i + 1] * rrms * wt[2 * i + 1]), sw[i], cw[i], first);
                }
                if (kn.k_out != nullptr && ok)  // the normed, rotated keys in bf16, for a prompt's own attention
                    *reinterpret_cast<uint4 *>(kn.k_out + row * D + dd) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
#pragma unroll
                for (int i = 0; i < 4; ++i) { x[8 * part + 2 * i] = bf16lo(ow[i]); x[8 * part + 2 * i + 1] = bf16hi(ow[i]); }
            }
        } else {
#pragma unroll
            for (int part = 0; part < E / 8; ++part) {
                float p8[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                if (ok) load_row8_rope(src, d0 + 8 * part, is_v ? nullptr : sin, cos, pos, rotary_dim, p8);
#pragma unroll
                for (int i = 0; i < 8; ++i) x[8 * part + i] = p8[i];
            }
        }
        const int64_t in_page = static_cast<int64_t>(pos - page * view.page_tokens) * H + h;  // (token, head) row inside the page
        const int64_t pidx = static_cast<int64_t>(s) * view.pages_per_seq + page;
        if (KIND == HS_KV_BF16) {
            if (ok) {
                uint16_t *dst = reinterpret_cast<uint16_t *>(data_pages[pidx]) + in_page * D + d0;
#pragma unroll
                for (int part = 0; part < E / 8; ++part) {
                    uint4 w;
                    w.x = pack_bf16(x[8 * part], x[8 * part + 1]); w.y = pack_bf16(x[8 * part + 2], x[8 * part + 3]);
                    w.z = pack_bf16(x[8 * part + 4], x[8 * part + 5]); w.w = pack_bf16(x[8 * part + 6], x[8 * part + 7]);
                    reinterpret_cast<uint4 *>(dst)[part] = w;
                }
            }
            continue;
        }
        constexpr int QK = KIND == HS_KV_BF16 ? HS_KV_INT8 : KIND;
        CodeWords<QK, E> c;
        float a = quantize_n<QK, E>(x, tpb, view.scale_dtype, tab, c);
        if (!ok) continue;
        uint8_t *codes = reinterpret_cast<uint8_t *>(data_pages[pidx]);
        void *scales = scale_pages[pidx];
        if ((d0 & (view.block - 1)) == 0) store_scale(scales, in_page * bpr + (d0 >> block_shift), view.scale_dtype, a);
        const int64_t e0 = in_page * D + d0;
        if constexpr (E == 8) {
            store_codes8<QK>(codes, e0, e0 + 8, c, true);
        } else if constexpr (QK == HS_KV_INT8) {
            *reinterpret_cast<uint4 *>(codes + e0) = make_uint4(c.w[0], c.w[1], c.w[2], c.w[3]);
        } else {
            *reinterpret_cast<uint2 *>(codes + (e0 >> 1)) = make_uint2(c.w[0], c.w[1]);
        }
    }
}

// ---- gather-dequantise (LayerKVCache::get compatibility read) ------------------------------------------------
// grid: x = groups of kGatherChunks * 256 chunks of 8 elements of one sequence's rows, y = 2 * sequence + (0: K, 1: V).  A thread
// has kGatherChunks loads in flight; shifts and 32-bit arithmetic in place of the 64-bit divisions per 8 elements it had: 4,333
// int8 tokens of 8 x 128 21.0 -> 11.0 us.
constexpr int kGatherChunks = 4;
template <int KIND>
__global__ void __launch_bounds__(kQThreads) kv_gather_kernel(ViewDev view, const int32_t *__restrict__ seq_lens, int out_tokens,
                                                              uint16_t *__restrict__ k_out, uint16_t *__restrict__ v_out) {
    __shared__ ValueTable<KIND> tab;
    tab.fill();
    __syncthreads();
    const bool is_v = (blockIdx.y & 1u) != 0;
    const int s = static_cast<int>(blockIdx.y >> 1);
    const int D = view.head_dim, H = view.n_kv_heads;
    const int cpr_shift = __ffs(D) - 4;   // head_dim is a power of two: 8-element chunks per (token, head) row
    const int block_shift = __ffs(view.block) - 1, bpr = D / view.block;
    const bool page_pow2 = (view.page_tokens & (view.page_tokens - 1)) == 0, h_pow2 = (H & (H - 1)) == 0;
    const int page_shift = __ffs(view.page_tokens) - 1, h_shift = __ffs(H) - 1;
    const int64_t total = (static_cast<int64_t>(out_tokens) * H) << cpr_shift;
    const int64_t chunk0 = static_cast<int64_t>(blockIdx.x) * (kGatherChunks * kQThreads) + threadIdx.x;
    const int len = seq_lens ? min(seq_lens[s], out_tokens) : out_tokens;
    void *const *data_pages = (is_v ? view.v_pages : view.k_pages) + static_cast<int64_t>(s) * view.pages_per_seq;
    void *const *scale_pages = KIND == HS_KV_BF16 ? nullptr : (is_v ? view.v_scale_pages : view.k_scale_pages) + static_cast<int64_t>(s) * view.pages_per_seq;
    uint4 w[kGatherChunks];
    float a[kGatherChunks];
    bool live[kGatherChunks];
#pragma unroll
    for (int u = 0; u < kGatherChunks; ++u) {
        const int64_t chunk = chunk0 + u * kQThreads;
        w[u] = make_uint4(0, 0, 0, 0);
        a[u] = 0.0f;
        live[u] = false;
        if (chunk >= total) continue;
        const int d0 = static_cast<int>(chunk & ((1 << cpr_shift) - 1)) * 8;
        const int64_t row = chunk >> cpr_shift;
        const int t = static_cast<int>(h_pow2 ? row >> h_shift : row / H);
        const int h = static_cast<int>(row - static_cast<int64_t>(t) * H);
        const int page = page_pow2 ? t >> page_shift : t / view.page_tokens;
        live[u] = t < len && page < view.pages_per_seq;
        if (!live[u]) continue;
        const int64_t in_page = static_cast<int64_t>(t - page * view.page_tokens) * H + h;
        const unsigned char *data = reinterpret_cast<const unsigned char *>(data_pages[page]);
        if constexpr (KIND == HS_KV_BF16) {
            w[u] = *reinterpret_cast<const uint4 *>(data + (in_page * D + d0) * 2);
        } else {
            a[u] = load_scale(scale_pages[page], in_page * bpr + (d0 >> block_shift), view.scale_dtype);
            if constexpr (KIND == HS_KV_INT8) {
                const uint2 c = *reinterpret_cast<const uint2 *>(data + in_page * D + d0);
                w[u].x = c.x; w[u].y = c.y;
            } else {
                w[u].x = *reinterpret_cast<const uint32_t *>(data + ((in_page * D + d0) >> 1));
            }
        }
    }
#pragma unroll
    for (int u = 0; u < kGatherChunks; ++u) {
        const int64_t chunk = chunk0 + u * kQThreads;
        if (chunk >= total) return;
        if constexpr (KIND != HS_KV_BF16) {
            float v[8];
            tab.values8(make_uint2(w[u].x, w[u].y), v);
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = live[u] ? pack_bf16(__fmul_rn(v[2 * i], a[u]), __fmul_rn(v[2 * i + 1], a[u])) : 0u;
            w[u] = make_uint4(o[0], o[1], o[2], o[3]);
        }
        *reinterpret_cast<uint4 *>((is_v ? v_out : k_out) + ((static_cast<int64_t>(s) * total + chunk) << 3)) = w[u];
    }
}

}  // namespace hs

using namespace hs;

extern "C" {

int32_t hs_quantize_blockwise(int32_t kind, const void *src, int32_t dtype, int64_t n, int32_t block, int32_t scale_dtype,
                              uint8_t *codes, void *absmax, hs_stream_t stream) {
    if (int32_t st = check_device()) return st;
    if (kind < HS_KV_INT8 || kind > HS_KV_FP4) return fail(HS_ERR_ARG, "hs_quantize_blockwise: unknown kind %d", kind);
    if (dtype < HS_DTYPE_BF16 || dtype > HS_DTYPE_F32) return fail(HS_ERR_ARG, "hs_quantize_blockwise: unknown dtype %d", dtype);
    if (block != 64 && block != 128 && block != 256) return fail(HS_ERR_UNSUPPORTED, "hs_quantize_blockwise: block %d (supported: 64, 128, 256)", block);
    if (scale_dtype != HS_SCALE_F32 && scale_dtype != HS_SCALE_F16) return fail(HS_ERR_ARG, "hs_quantize_blockwise: unknown scale dtype %d", scale_dtype);
    if (n < 0) return fail(HS_ERR_ARG, "hs_quantize_blockwise: negative n");
    if (n == 0) return HS_OK;
    if (!src || !codes || !absmax) return fail(HS_ERR_ARG, "hs_quantize_blockwise: NULL pointer");
    const size_t esz = dtype == HS_DTYPE_F32 ? 4 : 2;
    if (!aligned(src, esz) || !aligned(absmax, scale_dtype == HS_SCALE_F16 ? 2 : 4))
        return fail(HS_ERR_ARG, "hs_quantize_blockwise: misaligned pointer");
    if (!aligned(codes, kind == HS_KV_INT8 ? 8 : 4)) return fail(HS_ERR_ARG, "hs_quantize_blockwise: codes must be 8-byte aligned");
    const int vec_ok = aligned(src, 16) ? 1 : 0;
    const int64_t chunks = (n + 7) / 8;
    // whole quantisation blocks per warp: 32 * 8 elements are a multiple of every supported block
    const unsigned grid = static_cast<unsigned>((chunks + kQThreads * kFlatChunks - 1) / (kQThreads * kFlatChunks));
    cudaStream_t s = as_stream(stream);
#define HS_QUANT(K, T) quantize_flat_kernel<K, T><<<grid, kQThreads, 0, s>>>(src, n, block, scale_dtype, codes, absmax, vec_ok)
#define HS_QUANT_T(K) do { if (dtype == HS_DTYPE_BF16) HS_QUANT(K, HS_DTYPE_BF16); else if (dtype == HS_DTYPE_F16) HS_QUANT(K, HS_DTYPE_F16); \
                           else HS_QUANT(K, HS_DTYPE_F32); } while (0)
    if (kind == HS_KV_INT8) HS_QUANT_T(HS_KV_INT8);
    else if (kind == HS_KV_NF4) HS_QUANT_T(HS_KV_NF4);
    else HS_QUANT_T(HS_KV_FP4);
#undef HS_QUANT_T
#undef HS_QUANT
    return check_launch("hs_quantize_blockwise");
}

int32_t hs_dequantize_blockwise(int32_t kind, const uint8_t *codes, const void *absmax, int64_t n, int32_t block,
                                int32_t scale_dtype, void *out, int32_t dtype, hs_stream_t stream) {
    if (int32_t st = check_device()) return st;
    if (kind < HS_KV_INT8 || kind > HS_KV_FP4) return fail(HS_ERR_ARG, "hs_dequantize_blockwise: unknown kind %d", kind);
    if (dtype < HS_DTYPE_BF16 || dtype > HS_DTYPE_F32) return fail(HS_ERR_ARG, "hs_dequantize_blockwise: unknown dtype %d", dtype);
    if (block <= 0) return fail(HS_ERR_ARG, "hs_dequantize_blockwise: block must be positive");
    if (scale_dtype != HS_SCALE_F32 && scale_dtype != HS_SCALE_F16) return fail(HS_ERR_ARG, "hs_dequantize_blockwise: unknown scale dtype %d", scale_dtype);
    if (n < 0) return fail(HS_ERR_ARG, "hs_dequantize_blockwise: negative n");
    if (n == 0) return HS_OK;
    if (!codes || !absmax || !out) return fail(HS_ERR_ARG, "hs_dequantize_blockwise: NULL pointer");
    if (block % 8 != 0) return fail(HS_ERR_UNSUPPORTED, "hs_dequantize_blockwise: block must be a multiple of 8");
    if (!aligned(out, dtype == HS_DTYPE_F32 ? 4 : 2) || !aligned(absmax, scale_dtype == HS_SCALE_F16 ? 2 : 4))
        return fail(HS_ERR_ARG, "hs_dequantize_blockwise: misaligned pointer");
    const int64_t chunks = (n + 7) / 8;
    const unsigned grid = static_cast<unsigned>((chunks + kQThreads * kFlatChunks - 1) / (kQThreads * kFlatChunks));
    const int vec_ok = aligned(codes, kind == HS_KV_INT8 ? 8 : 4) && aligned(out, 16) ? 1 : 0;
    cudaStream_t s = as_stream(stream);
#define HS_DEQUANT(K, T) dequantize_flat_kernel<K, T><<<grid, kQThreads, 0, s>>>(codes, absmax, n, block, scale_dtype, out, vec_ok)
#define HS_DEQUANT_T(K) do { if (dtype == HS_DTYPE_BF16) HS_DEQUANT(K, HS_DTYPE_BF16); else if (dtype == HS_DTYPE_F16) HS_DEQUANT(K, HS_DTYPE_F16); \
                             else HS_DEQUANT(K, HS_DTYPE_F32); } while (0)
    if (kind == HS_KV_INT8) HS_DEQUANT_T(HS_KV_INT8);
    else if (kind == HS_KV_NF4) HS_DEQUANT_T(HS_KV_NF4);
    else HS_DEQUANT_T(HS_KV_FP4);
#undef HS_DEQUANT_T
#undef HS_DEQUANT
    return check_launch("hs_dequantize_blockwise");
}

int32_t hs_rope_apply(const void *x, void *out, const void *sin, const void *cos, const int32_t *positions, int64_t n_rows,
                      int32_t n_heads, int32_t head_dim, int32_t rotary_dim, int32_t n_positions, hs_stream_t stream) {
    if (int32_t st = check_device()) return st;
    if (n_rows < 0 || n_heads <= 0 || head_dim <= 0 || n_positions <= 0) return fail(HS_ERR_ARG, "hs_rope_apply: bad sizes");
    if (head_dim % 8 != 0 || rotary_dim % 16 != 0 || rotary_dim < 0 || rotary_dim > head_dim)
        return fail(HS_ERR_UNSUPPORTED, "hs_rope_apply: head_dim %% 8 and rotary_dim %% 16 must be 0, rotary_dim <= head_dim");
    if (n_rows == 0) return HS_OK;
    if (!x || !out || !sin || !cos || !positions) return fail(HS_ERR_ARG, "hs_rope_apply: NULL pointer");
    if (!aligned(x, 16) || !aligned(out, 16) || !aligned(sin, 2) || !aligned(cos, 2) || !aligned(positions, 4))
        return fail(HS_ERR_ARG, "hs_rope_apply: x and out must be 16-byte aligned");
    if (x == out && rotary_dim > 0) return fail(HS_ERR_ARG, "hs_rope_apply: in-place rotation is not supported (a lane reads its partner half)");
    int *err = device_error_word();
    if (!err) return fail(HS_ERR_DEVICE, "hs_rope_apply: device error word unavailable");
    const int units = (rotary_dim / 16 + (head_dim - rotary_dim) / 8) * n_heads;  // work units of a row
    // about four units per thread; never more than the grid can be addressed with
    int64_t rows_per_block = max(1, min(1 << 16, 4 * kQThreads / max(1, units)));
    if ((n_rows + rows_per_block - 1) / rows_per_block < 2 * sm_count()) rows_per_block = max(1, kQThreads / max(1, units));  // few rows: spread them
    const unsigned grid = static_cast<unsigned>((n_rows + rows_per_block - 1) / rows_per_block);
    rope_kernel<<<grid, kQThreads, 0, as_stream(stream)>>>(
        reinterpret_cast<const uint16_t *>(x), reinterpret_cast<uint16_t *>(out), reinterpret_cast<const uint16_t *>(sin),
        reinterpret_cast<const uint16_t *>(cos), positions, n_rows, n_heads, head_dim, rotary_dim, n_positions, static_cast<int>(rows_per_block), err);
    return check_launch("hs_rope_apply");
}

static int32_t kv_write_impl(const char *who, const hs_kv_view *view, const void *k_new, const void *v_new, int32_t n_seqs, int32_t n_tokens,
                             const int32_t *dst_pos, const void *sin, const void *cos, int32_t rotary_dim, int32_t n_positions, hs::KNormArgs kn,
                             hs_stream_t stream, bool overlap = false) {
    if (int32_t st = check_device()) return st;
    if (int32_t st = validate_view(view)) return st;
    if (n_seqs < 0 || n_tokens < 0) return fail(HS_ERR_ARG, "%s: negative sizes", who);
    if (n_seqs == 0 || n_tokens == 0) return HS_OK;
    if (!k_new || !v_new) return fail(HS_ERR_ARG, "%s: NULL input", who);
    if (!aligned(k_new, 16) || !aligned(v_new, 16)) return fail(HS_ERR_ARG, "%s: inputs must be 16-byte aligned", who);
    if (sin != nullptr) {
        if (!cos) return fail(HS_ERR_ARG, "%s: sin given without cos", who);
        if (rotary_dim <= 0 || rotary_dim % 16 != 0 || rotary_dim > view->head_dim || n_positions <= 0)
            return fail(HS_ERR_UNSUPPORTED, "%s: rotary_dim must be a positive multiple of 16 <= head_dim", who);
    }
    if (kn.weight != nullptr && (!aligned(kn.weight, 16) || (kn.k_out && !aligned(kn.k_out, 16))))
        return fail(HS_ERR_ARG, "%s: the norm weight and the key output must be 16-byte aligned", who);
    ViewDev d = to_dev(view);
    const int64_t elems = static_cast<int64_t>(n_tokens) * d.n_kv_heads * d.head_dim;  // per sequence and per K / V
    if (elems / 8 > 0x7fffffffLL || n_seqs > 32767) return fail(HS_ERR_UNSUPPORTED, "%s: more than 2^31 chunks per sequence or 32767 sequences in one call", who);
    const bool wide = elems >= (1 << 16);  // long writes: 16 elements per thread
    dim3 grid(static_cast<unsigned>((elems + static_cast<int64_t>(kQThreads) * kWriteElems - 1) / (static_cast<int64_t>(kQThreads) * kWriteElems)), 2u * static_cast<unsigned>(n_seqs));
    cudaStream_t s = as_stream(stream);
    int *err = device_error_word();
    if (!err) return fail(HS_ERR_DEVICE, "%s: device error word unavailable", who);
    const uint16_t *k = reinterpret_cast<const uint16_t *>(k_new), *v = reinterpret_cast<const uint16_t *>(v_new);
    const uint16_t *sn = reinterpret_cast<const uint16_t *>(sin), *cs = reinterpret_cast<const uint16_t *>(cos);
#define HS_KV_WRITE_N(K, N) do { if (wide) launch_maybe_overlapped(kv_write_kernel<K, 16, N>, grid, kQThreads, s, overlap, d, k, v, n_seqs, n_tokens, dst_pos, sn, cs, rotary_dim, n_positions, err, kn); \
                                 else launch_maybe_overlapped(kv_write_kernel<K, 8, N>, grid, kQThreads, s, overlap, d, k, v, n_seqs, n_tokens, dst_pos, sn, cs, rotary_dim, n_positions, err, kn); } while (0)
#define HS_KV_WRITE(K) do { if (kn.weight != nullptr) HS_KV_WRITE_N(K, true); else HS_KV_WRITE_N(K, false); } while (0)
    switch (view->kind) {
        case HS_KV_BF16: HS_KV_WRITE(HS_KV_BF16); break;
        case HS_KV_INT8: HS_KV_WRITE(HS_KV_INT8); break;
        case HS_KV_NF4: HS_KV_WRITE(HS_KV_NF4); break;
        default: HS_KV_WRITE(HS_KV_FP4); break;
    }
#undef HS_KV_WRITE
#undef HS_KV_WRITE_N
    return check_launch(who);
}

int32_t hs_kv_quantize_write(const hs_kv_view *view, const void *k_new, const void *v_new, int32_t n_seqs, int32_t n_tokens,
                             const int32_t *dst_pos, const void *sin, const void *cos, int32_t rotary_dim,
                             int32_t n_positions, hs_stream_t stream) {
    return kv_write_impl("hs_kv_quantize_write", view, k_new, v_new, n_seqs, n_tokens, dst_pos, sin, cos, rotary_dim, n_positions,
                         hs::KNormArgs{nullptr, 0.0f, 0, nullptr, 0}, stream);
}

}  // extern "C"

int32_t hs::kv_write_at(const hs_kv_view *view, const void *k_new, const void *v_new, int32_t n_tokens, int32_t start_pos, const void *sin,
                        const void *cos, int32_t rotary_dim, int32_t n_positions, hs_stream_t stream) {
    return kv_write_impl("hs_cache_update", view, k_new, v_new, 1, n_tokens, nullptr, sin, cos, rotary_dim, n_positions,
                         hs::KNormArgs{nullptr, 0.0f, 0, nullptr, start_pos}, stream);
}

// hs_kv_quantize_write of one new token per sequence at position seq_lens[s] - 1 (used by hs_attn_decode_append when the
// caller gives no positions and the attention kernel does not take the write itself)
int32_t hs::kv_write_at_end(const hs_kv_view *view, const void *k_new, const void *v_new, int32_t n_seqs, const int32_t *seq_lens, const void *sin,
                            const void *cos, int32_t rotary_dim, int32_t n_positions, hs_stream_t stream) {
    return kv_write_impl("hs_attn_decode_append", view, k_new, v_new, n_seqs, 1, seq_lens, sin, cos, rotary_dim, n_positions,
                         hs::KNormArgs{nullptr, 0.0f, 0, nullptr, -1}, stream);
}

int32_t hs::kv_norm_rope_write_impl(const hs_kv_view *view, const void *k_proj, const void *v_new, int32_t n_seqs, int32_t n_tokens,
                                    const int32_t *dst_pos, const float *k_norm_weight, float eps, int32_t weight_plus_one, const void *sin,
                                    const void *cos, int32_t rotary_dim, int32_t n_positions, void *k_out, bool overlap, hs_stream_t stream) {
    if (!k_norm_weight) return fail(HS_ERR_ARG, "hs_kv_norm_rope_quantize_write: NULL norm weight (use hs_kv_quantize_write)");
    return kv_write_impl("hs_kv_norm_rope_quantize_write", view, k_proj, v_new, n_seqs, n_tokens, dst_pos, sin, cos, rotary_dim, n_positions,
                         hs::KNormArgs{k_norm_weight, eps, weight_plus_one, reinterpret_cast<uint16_t *>(k_out), 0}, stream, overlap);
}

extern "C" {

int32_t hs_kv_norm_rope_quantize_write(const hs_kv_view *view, const void *k_proj, const void *v_new, int32_t n_seqs, int32_t n_tokens,
                                       const int32_t *dst_pos, const float *k_norm_weight, float eps, int32_t weight_plus_one, const void *sin,
                                       const void *cos, int32_t rotary_dim, int32_t n_positions, void *k_out, hs_stream_t stream) {
    return kv_norm_rope_write_impl(view, k_proj, v_new, n_seqs, n_tokens, dst_pos, k_norm_weight, eps, weight_plus_one, sin, cos, rotary_dim, n_positions,
                                   k_out, false, stream);
}

static int32_t gather_launch(const hs_kv_view *view, const int32_t *seq_lens, int32_t n_seqs, int32_t out_tokens, void *k_out, void *v_out,
                             hs_stream_t stream) {
    ViewDev d = to_dev(view);
    const int64_t chunks = static_cast<int64_t>(out_tokens) * d.n_kv_heads * (d.head_dim / 8);
    dim3 grid(static_cast<unsigned>((chunks + kGatherChunks * kQThreads - 1) / (kGatherChunks * kQThreads)), 2u * static_cast<unsigned>(n_seqs));
    cudaStream_t s = as_stream(stream);
    uint16_t *ko = reinterpret_cast<uint16_t *>(k_out), *vo = reinterpret_cast<uint16_t *>(v_out);
    switch (view->kind) {
        case HS_KV_BF16: kv_gather_kernel<HS_KV_BF16><<<grid, kQThreads, 0, s>>>(d, seq_lens, out_tokens, ko, vo); break;
        case HS_KV_INT8: kv_gather_kernel<HS_KV_INT8><<<grid, kQThreads, 0, s>>>(d, seq_lens, out_tokens, ko, vo); break;
        case HS_KV_NF4: kv_gather_kernel<HS_KV_NF4><<<grid, kQThreads, 0, s>>>(d, seq_lens, out_tokens, ko, vo); break;
        default: kv_gather_kernel<HS_KV_FP4><<<grid, kQThreads, 0, s>>>(d, seq_lens, out_tokens, ko, vo); break;
    }
    return check_launch("hs_kv_gather_dequantize");
}

int32_t hs_kv_gather_dequantize(const hs_kv_view *view, const int32_t *seq_lens, int32_t n_seqs, int32_t out_tokens,
                                void *k_out, void *v_out, hs_stream_t stream) {
    if (int32_t st = check_device()) return st;
    if (int32_t st = validate_view(view)) return st;
    if (n_seqs < 0 || out_tokens < 0) return fail(HS_ERR_ARG, "hs_kv_gather_dequantize: negative sizes");
    if (n_seqs == 0 || out_tokens == 0) return HS_OK;
    if (!seq_lens || !k_out || !v_out) return fail(HS_ERR_ARG, "hs_kv_gather_dequantize: NULL pointer");
    if (!aligned(k_out, 16) || !aligned(v_out, 16)) return fail(HS_ERR_ARG, "hs_kv_gather_dequantize: outputs must be 16-byte aligned");
    if (n_seqs > 32767) {  // the grid's second dimension holds 2 * 32767 rows: the rest in calls of their own
        const int64_t step = static_cast<int64_t>(32767) * out_tokens * view->n_kv_heads * view->head_dim * 2;
        hs_kv_view rest = *view;
        const int64_t pages = static_cast<int64_t>(32767) * view->pages_per_seq;
        rest.k_pages += pages;
        rest.v_pages += pages;
        if (rest.k_scale_pages) rest.k_scale_pages += pages;
        if (rest.v_scale_pages) rest.v_scale_pages += pages;
        if (int32_t st = hs_kv_gather_dequantize(view, seq_lens, 32767, out_tokens, k_out, v_out, stream)) return st;
        return hs_kv_gather_dequantize(&rest, seq_lens + 32767, n_seqs - 32767, out_tokens, static_cast<char *>(k_out) + step,
                                       static_cast<char *>(v_out) + step, stream);
    }
    return gather_launch(view, seq_lens, n_seqs, out_tokens, k_out, v_out, stream);
}

}  // extern "C"

int32_t hs::kv_gather_len(const hs_kv_view *view, int32_t len, void *k_out, void *v_out, hs_stream_t stream) {
    if (int32_t st = check_device()) return st;
    if (int32_t st = validate_view(view)) return st;
    if (!aligned(k_out, 16) || !aligned(v_out, 16)) return fail(HS_ERR_ARG, "hs_cache_get: outputs must be 16-byte aligned");
    return gather_launch(view, nullptr, 1, len, k_out, v_out, stream);
}
