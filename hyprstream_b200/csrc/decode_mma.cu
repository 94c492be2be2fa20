// Decode attention over a bf16, int8 or 4-bit cache, any head_dim in {64, 128, 256} and 1 / 2 / 4 / 8 query heads per kv head, on the
// tensor cores.  (The int8 / 4-bit caches of the two served models' shapes go to decode_tc.cu, whose tiles span all kv heads.)
//
// HBM bound: a cached token of one kv head is read once.  What a CUDA-core form spent its time on instead: two tokens in flight
// per lane group (latency), and 2 * G fp32 FMAs plus the unpacking per element (issue).  Here
//   * a warp works by itself: 16 tokens of one kv head are one tile, its K and V rows come into the warp's own ring of shared
//     memory with 16-byte cp.async (rows XOR-swizzled, so that reads are free of bank conflicts), its block scales through
//     registers; no block barrier inside a sequence, any page size, rows past the end of a sequence filled with zeros;
//   * S = q.K^T on mma.sync m16n8k16 with the query heads as rows and O^T += V^T.P^T with head_dim as rows, so that P's accumulator
//     registers are the B operand as they are; bf16 operands, fp32 sums.  bf16 rows go in as stored, u8 codes as the exact
//     integers code - 127, 4-bit codes as two bf16 terms of the table values
//     (one lookup per code byte; V's nibbles of two neighbouring tokens are mixed into bytes first);
//   * P (times V's block scale) keeps 16 bits of mantissa: p = hi + lo, both bf16.  With up to 4 query heads the second half of the
//     MMA's 8 columns is free and carries lo (one MMA for both); with 8 heads lo takes an MMA and an accumulator of its own.  A bf16
//     output is as near to 64 bits as with fp32 P (1.4e-3 to 1.8e-3: its own rounding).  fp32 results are not (1.6e-6 to 4.6e-6 in
//     place of 3e-7), so a caller who takes them (EXACT: a shard's output and log-sum-exp) gets a third term of P and of the NF4
//     values, all their products above 2^-24, and a tile's sum added to the accumulator by fp32 additions: 2.3e-7 to 3.9e-7.  32
//     sequences of 4,096 to 8,192 tokens, EXACT against two terms (and the CUDA-core form): bf16 32 / 8 x 128 140 / 136 (416) us, int8
//     8 / 8 x 128 125 / 119 (240), NF4 16 / 2 x 256 171 / 117 (555), NF4 8 / 8 x 128 230 / 152 (172: the third lookup);
//   * the warps of a CTA merge their sums at the end of a sequence and write one partial per (CTA, sequence).
// Measured against the CUDA-core form (a cold launch by itself), bf16, 32 / 8 heads x 128: 16 paged sequences of 100 to 6,000 tokens
// (247 MB) 150 -> 44.0 us = 5.6 TB/s; one sequence of 4,096 tokens 23.3 -> 9.3 us.  Whole steps of 32 sequences of 4,096 to 8,192
// tokens: NF4 16 / 2 x 256 617 -> 121 us, NF4 32 / 8 x 64 321 -> 101, NF4 8 / 8 x 128 208 -> 158, int8 32 / 8 x 64 289 -> 97, int8
// 8 / 8 x 128 251 -> 127 us (floors 16 to 65 us: the warps' instruction chain bounds the codes, not HBM).
#include "hs_common.cuh"
#include "quant_dev.cuh"

namespace hs {

constexpr int kMmWarps = 4;
constexpr int kMmThreads = kMmWarps * 32;
constexpr int kMmTile = 16;  // tokens per tile of the flat partition = one warp step

// KIND: HS_KV_BF16, HS_KV_INT8, or HS_KV_NF4 for both 4-bit kinds (the table is chosen at run time).
template <int KIND, int D, int G, bool EXACT>
struct MmLayout {
    static constexpr bool kQuant = KIND != HS_KV_BF16;
    static constexpr int kRow = KIND == HS_KV_BF16 ? D * 2 : (KIND == HS_KV_INT8 ? D : D / 2);  // bytes of one (token, head) row
    static constexpr int kChunks = kRow / 16;
    static constexpr int kScaleOff = 2 * kMmTile * kRow;                                       // float [K, V][scale block][token]
    static constexpr int kTileBytes = kScaleOff + (kQuant ? 2 * kMmTile * (D / 64) * 4 : 0);
    // bytes in flight: 6.5 TB/s / 148 SMs at ~1 us is ~44 KB per SM; the rings of an SM hold 100-190 KB (32-64 KB for the small
    // rows of head_dim 64).  At least three stages: a tile's scales are parked one fetch after its rows.
    static constexpr int kStages = kTileBytes >= 4096 ? 3 : 5;
    static constexpr int kORow = D + 4;                 // floats between the heads of a warp's merge rows (bank spread)
    static constexpr int kMergeOff = kMmWarps * kStages * kTileBytes;
    static constexpr int kMlOff = kMergeOff + kMmWarps * G * kORow * 4;
    // 4-bit kinds: uint2 [256][kLutCols], code byte -> both values as bf16 pairs (upper terms, lower terms).  8 columns, two
    // lanes of a half warp each (16 would be free of bank conflicts and cost a CTA per SM).  FP4 needs the upper terms only; the rule
    // does not tell it from NF4 (8 / 8 x 128, 32 sequences of 4,096 to 8,192 tokens: 150 us, the CUDA-core form 173)
    static constexpr int kLutCols = 8;
    static constexpr int kLutOff = (kMlOff + kMmWarps * G * 2 * 4 + 127) / 128 * 128;
    static constexpr int kLut2Cols = 8;  // EXACT: uint32_t [256][kLut2Cols], the pairs' third terms
    static constexpr int kLut2Off = kLutOff + (kQuant && KIND != HS_KV_INT8 ? 256 * kLutCols * 8 : 0);
    static constexpr int kTotal = kLut2Off + (EXACT && kQuant && KIND != HS_KV_INT8 ? 256 * kLut2Cols * 4 : 0);
    // codes take several times the instructions per byte that bf16 rows take: as many warps as the registers allow (a warp's chain
    // of lookups, MMAs and shuffles is latency, not throughput)
    static constexpr int kWant = !kQuant || D == 256 || G == 8 ? 2 : (D == 128 ? 3 : 4);
    static constexpr int kCtasPerSm = kWant * (kTotal + 1024) <= 228 * 1024 ? kWant : (2 * (kTotal + 1024) <= 228 * 1024 ? 2 : 1);
    static_assert(kTotal + 1024 <= 228 * 1024, "a CTA must fit its SM's shared memory");
    // 16-byte chunk c of token row t sits at chunk c ^ swz(t).  bf16: ldmatrix reads 8 rows at one chunk.  u8 and 4-bit codes: a
    // K read takes 4 (2) chunks of neighbouring rows, a V read 2 (1) chunks of every other row.
    static __device__ __forceinline__ int swz(int t) {
        if constexpr (!kQuant) return t & 7;
        else if constexpr (kChunks >= 8) return (((t >> 1) & 3) << 1) ^ ((t & 1) << 2);
        else if constexpr (kChunks == 4) return ((t >> 1) & 1) << 1;
        else return 0;
    }
};

__device__ __forceinline__ void mm_cp16(uint32_t dst, const void *src, int bytes) {  // bytes = 16, or 0: sixteen zero bytes, src not read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mm_cp4(uint32_t dst, const void *src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
constexpr int kLog2(int x) { return x <= 1 ? 0 : 1 + kLog2(x / 2); }
__device__ __forceinline__ void mm_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void mm_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// four u8 codes of a word as (code - 127) in bf16, two words of pairs: 2^23 + byte by a byte permute, an exact subtraction, and
// the upper halves (an integer of at most 8 bits is exact in bf16)
__device__ __forceinline__ void codes4_bf16(uint32_t w, uint32_t &lo, uint32_t &hi) {
    float f[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 + i)) - 8388735.0f;
    lo = __byte_perm(__float_as_uint(f[0]), __float_as_uint(f[1]), 0x7632);
    hi = __byte_perm(__float_as_uint(f[2]), __float_as_uint(f[3]), 0x7632);
}
// the next bf16 term of a table value: `rest` = what the terms before it leave.  Where they leave nothing of a value other than zero, the
// smallest number of its sign: a block scale may be infinite, and infinity x 0 would spoil the value's own infinity (as a term of
// a finite sum it is 2^-126 of the scale)
__device__ __forceinline__ float next_term(float rest, float value) {
    const float t = bf16_round(rest);
    return t == 0.0f && value != 0.0f ? copysignf(1.17549435e-38f, value) : t;
}
// the values of code byte `k` (0..3) of w, high nibble first, as two bf16 pairs: upper terms in .x, lower terms (the rest, rounded to
// bf16) in .y; `lut` = address of this lane's column, entries `stride` bytes apart
template <int STRIDE>
__device__ __forceinline__ uint2 lut_pairs(uint32_t lut, uint32_t w, uint32_t k) {
    const uint32_t byte = __byte_perm(w, 0u, 0x4440u | k);
    uint2 v;
    asm("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(byte * STRIDE + lut));
    return v;
}

template <int STRIDE>
__device__ __forceinline__ uint32_t lut_third(uint32_t lut2, uint32_t w, uint32_t k) {
    const uint32_t byte = __byte_perm(w, 0u, 0x4440u | k);
    uint32_t v;
    asm("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(byte * STRIDE + lut2));
    return v;
}

template <int KIND, int D, int G, bool EXACT>
__global__ void __launch_bounds__(kMmThreads, MmLayout<KIND, D, G, EXACT>::kCtasPerSm)
decode_mma_kernel(ViewDev view, const uint16_t *__restrict__ q, const int32_t *__restrict__ seq_lens, int n_seqs, int n_q_heads,
                  float scale_log2, float *__restrict__ o_part, float *__restrict__ lse_part, int *__restrict__ err, AppendArgs ap) {
    using LT = MmLayout<KIND, D, G, EXACT>;
    constexpr bool kQuant = LT::kQuant, kFour = kQuant && KIND != HS_KV_INT8;
    constexpr int kChunks = LT::kChunks;           // 16-byte chunks of a row
    constexpr int kStages = LT::kStages;
    extern __shared__ __align__(128) unsigned char mm_smem[];
    // the merge kernel that follows as a programmatic dependent may start; it waits for this grid before it reads anything
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    EndOfGridWait order;  // (also blocks without work: the merge waits for this grid alone, and the write in front of it may still run)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kvh = blockIdx.y, H = view.n_kv_heads;
    const int64_t cta = blockIdx.x;
    const int cap = view.page_tokens * view.pages_per_seq;  // lengths beyond the view's pages are cut (and recorded)
    auto tiles_of = [&](int L) { return (min(max(L, 0), cap) + kMmTile - 1) / kMmTile; };

    // ---- the CTA's range of the concatenated tile list (every warp for itself, 32 lengths per load) ----
    int64_t total = 0;
    bool over = false, unwritable = false;
    for (int base = 0; base < n_seqs; base += 32) {
        const int L = base + lane < n_seqs ? seq_lens[base + lane] : 0;
        over |= L > cap;
        unwritable |= base + lane < n_seqs && (L > cap || L <= 0);  // no place for a new token at L - 1
        total += __reduce_add_sync(0xffffffffu, static_cast<unsigned>(tiles_of(L)));
    }
    if (over && warp == 0 && cta == 0 && kvh == 0) atomicOr(err, HS_DEVERR_DECODE_RANGE);
    if (!kQuant && ap.k_new != nullptr && unwritable && warp == 0 && cta == 0 && kvh == 0) atomicOr(err, HS_DEVERR_KV_WRITE_RANGE);
    // never more working CTAs than tiles (the merge uses the same rule)
    const int64_t n_ctas = total < static_cast<int64_t>(gridDim.x) ? (total > 0 ? total : 1) : static_cast<int64_t>(gridDim.x);
    if (cta >= n_ctas) return;
    const int64_t t_begin = part_begin(cta, total, n_ctas), t_end = part_begin(cta + 1, total, n_ctas);
    if (t_begin >= t_end) return;
    // first sequence of the range and the tile count in front of it
    int r_first = 0;
    int64_t before_first = 0;
    for (int base = 0, done = 0; base < n_seqs && !done; base += 32) {
        int inc = base + lane < n_seqs ? tiles_of(seq_lens[base + lane]) : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += t;
        }
        const unsigned past = __ballot_sync(0xffffffffu, before_first + inc > t_begin);  // sequences that end behind t_begin
        const int at = past ? __ffs(past) - 1 : 32;
        r_first = base + at;
        if (at > 0) before_first += __shfl_sync(0xffffffffu, inc, at - 1);
        done = past != 0;
    }
    constexpr uint32_t kLutStride = LT::kLutCols * 8, kLut2Stride = LT::kLut2Cols * 4;
    uint32_t lut = 0, lut2 = 0;
    const bool two_terms = view.kind == HS_KV_NF4;  // (FP4 values are exact in bf16)
    if constexpr (kFour) {
        uint2 *tab = reinterpret_cast<uint2 *>(mm_smem + LT::kLutOff);
        const float *book = view.kind == HS_KV_NF4 ? c_nf4 : c_fp4;
        for (int e = warp * 64 + (lane & 1); e < warp * 64 + 64; e += 2) {  // a warp's quarter of the bytes, two at a time, 16 lanes a byte
            const float v0 = book[e >> 4], v1 = book[e & 15], u0 = bf16_round(v0), u1 = bf16_round(v1);
            if ((lane >> 1) < LT::kLutCols) tab[e * LT::kLutCols + (lane >> 1)] = make_uint2(pack_bf16(u0, u1), pack_bf16(next_term(v0 - u0, v0), next_term(v1 - u1, v1)));
            if constexpr (EXACT) {
                if ((lane >> 1) < LT::kLut2Cols)
                    reinterpret_cast<uint32_t *>(mm_smem + LT::kLut2Off)[e * LT::kLut2Cols + (lane >> 1)] =
                        pack_bf16(next_term(v0 - u0 - bf16_round(v0 - u0), v0), next_term(v1 - u1 - bf16_round(v1 - u1), v1));
            }
        }
        lut2 = static_cast<uint32_t>(__cvta_generic_to_shared(mm_smem + LT::kLut2Off)) + 4u * (lane & (LT::kLut2Cols - 1));
        lut = static_cast<uint32_t>(__cvta_generic_to_shared(tab)) + 8u * (lane & (LT::kLutCols - 1));
        __syncthreads();
    }

    // ---- feeding the ring: this warp's tiles are t_begin + warp, + kMmWarps, ... ----
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(mm_smem)) + warp * (kStages * LT::kTileBytes);
    unsigned char *ring_ptr = mm_smem + warp * (kStages * LT::kTileBytes);
    int64_t f_tile = t_begin + warp, f_before = before_first;  // next tile to fetch; tiles in front of sequence f_r
    int f_r = r_first, f_len = min(max(seq_lens[r_first], 0), cap), f_stage = 0;
    const bool whole_pages = view.pages_per_seq == 1 || view.page_tokens % kMmTile == 0;  // a tile lies in one page
    constexpr int kMaxBpr = D / 64;
    const int bpr = kQuant ? D / view.block : 1, bpr_shift = __ffs(bpr) - 1;
    float f_scale[kMaxBpr];  // scales of the tile fetched last: lanes 0-15 K of token `lane`, lanes 16-31 V
    auto park_scales = [&](int stage) {  // ... into its ring stage, one fetch later: their load has had a tile's time
        if constexpr (kQuant) {
            float *dst = reinterpret_cast<float *>(ring_ptr + stage * LT::kTileBytes + LT::kScaleOff) + (lane >> 4) * (kMaxBpr * kMmTile) + (lane & 15);
#pragma unroll
            for (int i = 0; i < kMaxBpr; ++i)
                if (i < bpr) dst[i * kMmTile] = f_scale[i] * (KIND == HS_KV_INT8 ? 1.0f / 127.0f : 1.0f);
        }
    };
#pragma unroll
    for (int i = 0; i < kMaxBpr; ++i) f_scale[i] = 0.0f;
    auto fetch = [&]() {
        park_scales(f_stage == 0 ? kStages - 1 : f_stage - 1);
        if (f_tile < t_end) {
            int nt = (f_len + kMmTile - 1) / kMmTile;
            while (f_tile >= f_before + nt) {
                f_before += nt;
                f_len = min(max(seq_lens[++f_r], 0), cap);
                nt = (f_len + kMmTile - 1) / kMmTile;
            }
            const int t0 = static_cast<int>(f_tile - f_before) * kMmTile;
            const int64_t pages = static_cast<int64_t>(f_r) * view.pages_per_seq;
            void *const *kp = view.k_pages + pages;
            void *const *vp = view.v_pages + pages;
            const uint32_t sK = ring + f_stage * LT::kTileBytes;
            const int page0 = view.pages_per_seq == 1 ? 0 : t0 / view.page_tokens;
            const unsigned char *k0 = reinterpret_cast<const unsigned char *>(kp[page0]), *v0 = reinterpret_cast<const unsigned char *>(vp[page0]);
            constexpr int kPer = kMmTile * kChunks / 32, kRows = 32 / kChunks;  // copies per lane and operand; rows the warp covers per copy
            const int row0 = lane / kChunks, c = lane % kChunks;
            // The step's new token (bf16 cache of one sequence, whose tokens nobody else looks at; LayerKVCache::update in the same
            // launch, kv_cache.rs:1275-1496): the warp that fetches the last tile takes the token's K (rotated) and V row of its kv head
            // from the inputs, writes them to the cache - the bits the write kernel writes - and puts them into the ring in place of
            // a copy.  A position past the rotation table is recorded and its K row left as it is, as the write kernel does.
            int k_row = -1, v_row = -1;  // rows of this tile that do not come from the cache
            if constexpr (!kQuant) {
                const int pos = f_len - 1;
                if (ap.k_new != nullptr && pos - t0 < kMmTile && seq_lens[f_r] <= cap) {
                    v_row = pos - t0;
                    const bool in_table = ap.sin == nullptr || pos < ap.n_positions;
                    if (in_table) k_row = v_row;
                    else if (lane == 0) atomicOr(err, HS_DEVERR_KV_WRITE_RANGE);
                    const int page = view.pages_per_seq == 1 ? 0 : pos / view.page_tokens;
                    const int64_t at = (static_cast<int64_t>(pos - page * view.page_tokens) * H + kvh) * LT::kRow;
                    const int64_t src = (static_cast<int64_t>(f_r) * H + kvh) * D;
                    for (int i = lane; i < 2 * kChunks; i += 32) {
                        const bool is_v = i >= kChunks;
                        const int ch = is_v ? i - kChunks : i;
                        if (!is_v && !in_table) continue;
                        const uint4 w = row8_rope((is_v ? ap.v_new : ap.k_new) + src, ch * 8, is_v ? nullptr : ap.sin, ap.cos, pos, ap.rotary_dim);
                        *reinterpret_cast<uint4 *>(static_cast<unsigned char *>((is_v ? vp : kp)[page]) + at + ch * 16) = w;
                        *reinterpret_cast<uint4 *>(ring_ptr + f_stage * LT::kTileBytes + (is_v ? kMmTile * LT::kRow : 0) + v_row * LT::kRow +
                                                   ((ch ^ LT::swz(v_row)) << 4)) = w;
                    }
                }
            }
            const bool fast = whole_pages && (!kQuant || ((reinterpret_cast<uintptr_t>(k0) | reinterpret_cast<uintptr_t>(v0)) & 15u) == 0);
            if (fast) {
                const int64_t off = (static_cast<int64_t>(t0 - page0 * view.page_tokens + row0) * H + kvh) * LT::kRow + c * 16;
                const int64_t step = static_cast<int64_t>(kRows) * H * LT::kRow;
                const unsigned char *ka = k0 + off, *va = v0 + off;
#pragma unroll 4
                for (int i = 0; i < kPer; ++i, ka += step, va += step) {
                    const int row = i * kRows + row0;
                    const bool live = t0 + row < f_len;
                    const uint32_t dst = sK + row * LT::kRow + ((c ^ LT::swz(row)) << 4);
                    if (kQuant || row != k_row) mm_cp16(dst, live ? ka : k0, live ? 16 : 0);
                    if (kQuant || row != v_row) mm_cp16(dst + kMmTile * LT::kRow, live ? va : v0, live ? 16 : 0);
                }
            } else {
#pragma unroll 1
                for (int i = 0; i < kPer; ++i) {
                    const int row = i * kRows + row0, t = t0 + row;
                    const bool live = t < f_len;
                    const int page = live ? t / view.page_tokens : page0;
                    const int64_t off = live ? (static_cast<int64_t>(t - page * view.page_tokens) * H + kvh) * LT::kRow + c * 16 : 0;
                    const uint32_t dst = sK + row * LT::kRow + ((c ^ LT::swz(row)) << 4);
                    const unsigned char *ka = reinterpret_cast<const unsigned char *>(kp[page]) + off, *va = reinterpret_cast<const unsigned char *>(vp[page]) + off;
                    if (!kQuant || ((reinterpret_cast<uintptr_t>(ka) | reinterpret_cast<uintptr_t>(va)) & 15u) == 0) {
                        if (kQuant || row != k_row) mm_cp16(dst, ka, live ? 16 : 0);
                        if (kQuant || row != v_row) mm_cp16(dst + kMmTile * LT::kRow, va, live ? 16 : 0);
                    } else {  // pages of codes that are aligned to words only
                        for (int b = 0; b < 16; b += 4) {
                            mm_cp4(dst + b, ka + b, live ? 4 : 0);
                            mm_cp4(dst + kMmTile * LT::kRow + b, va + b, live ? 4 : 0);
                        }
                    }
                }
            }
            if constexpr (kQuant) {
                const int t = t0 + (lane & 15);
#pragma unroll
                for (int i = 0; i < kMaxBpr; ++i) f_scale[i] = 0.0f;
                if (t < f_len) {
                    const int page = whole_pages ? page0 : t / view.page_tokens;
                    const void *sp = ((lane & 16) ? view.v_scale_pages : view.k_scale_pages)[pages + page];
                    const int64_t at = (static_cast<int64_t>(t - page * view.page_tokens) * H + kvh) * bpr;
#pragma unroll
                    for (int i = 0; i < kMaxBpr; ++i)
                        if (i < bpr) f_scale[i] = load_scale(sp, at + i, view.scale_dtype);
                }
            }
            f_tile += kMmWarps;
        }
        mm_commit();  // (an empty group when there is nothing left: the wait below counts groups)
        f_stage = f_stage + 1 == kStages ? 0 : f_stage + 1;
    };
    // a launch behind the write kernel of the same step (programmatic dependent) may get here before that kernel is done
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) fetch();

    const int g = lane >> 2, j = lane & 3;
    const int head = G == 8 ? g : (g & 3) % G;       // query head of this lane's score row; rows 4..7 repeat rows 0..3 for G <= 4
    const bool low_half = G < 8 && g >= 4;           // ... and carry the low parts of P
    int64_t tile = t_begin + warp;
    int stage = 0;
    int64_t before = before_first;
    float *m_o = reinterpret_cast<float *>(mm_smem + LT::kMergeOff);  // [warp][G][kORow]
    float *m_ml = reinterpret_cast<float *>(mm_smem + LT::kMlOff);    // [warp][G][2]: running maximum, sum
    for (int r = r_first; r < n_seqs && before < t_end; ++r) {
        const int L = min(max(seq_lens[r], 0), cap);
        const int nt_seq = (L + kMmTile - 1) / kMmTile;
        if (nt_seq == 0) continue;
        const int64_t hi = min(t_end, before + nt_seq);
        // query fragments.  bf16 cache: k-step s holds d = 16 s .. 16 s + 15 in order (ldmatrix).  Codes: k-step s of 64-wide block b
        // holds, for lane column j, d = 64 b + 16 j + 4 s .. + 3, so that one 16-byte (8-byte) read of codes feeds four k-steps.
        uint32_t qa[D / 16][2];
        const uint16_t *qp = q + (static_cast<int64_t>(r) * n_q_heads + kvh * G + head) * D;
#pragma unroll
        for (int s = 0; s < D / 16; ++s) {
            if constexpr (!kQuant) {
                qa[s][0] = *reinterpret_cast<const uint32_t *>(qp + 2 * j + 16 * s);
                qa[s][1] = *reinterpret_cast<const uint32_t *>(qp + 2 * j + 16 * s + 8);
            } else {
                const uint2 w = *reinterpret_cast<const uint2 *>(qp + 64 * (s >> 2) + 16 * j + 4 * (s & 3));
                qa[s][0] = w.x;
                qa[s][1] = w.y;
            }
        }
        float m = -INFINITY, l = 0.0f;
        constexpr int kLo = G == 8 ? D / 16 : 1;
        float O[D / 16][4], Olo[kLo][4];
#pragma unroll
        for (int i = 0; i < D / 16; ++i) O[i][0] = O[i][1] = O[i][2] = O[i][3] = 0.0f;
#pragma unroll
        for (int i = 0; i < kLo; ++i) Olo[i][0] = Olo[i][1] = Olo[i][2] = Olo[i][3] = 0.0f;

        for (; tile < hi; tile += kMmWarps) {
            fetch();
            mm_wait<kStages - 1>();
            __syncwarp();
            const uint32_t sK = ring + stage * LT::kTileBytes, sV = sK + kMmTile * LT::kRow;
            const unsigned char *pK = ring_ptr + stage * LT::kTileBytes, *pV = pK + kMmTile * LT::kRow;
            const float *sc = reinterpret_cast<const float *>(pK + LT::kScaleOff);  // [K, V][block][token]
            const int t0 = static_cast<int>(tile - before) * kMmTile;
            // ---- scores of 16 tokens: two n-tiles of 8 ----
            float p[2][2];
            float mx = -INFINITY;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float sum[2] = {0.0f, 0.0f};
                if constexpr (!kQuant) {
                    float s0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, s1[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // even and odd k-steps
                    const int row = nt * 8 + (lane & 7);
                    const uint32_t kr = sK + row * LT::kRow;
#pragma unroll
                    for (int kk = 0; kk < D / 32; ++kk) {
                        uint32_t b[4];
                        ldsm4(b, kr + (((kk * 4 + (lane >> 3)) ^ LT::swz(row)) << 4));
                        mma_bf16(s0, qa[2 * kk][0], 0u, qa[2 * kk][1], 0u, b[0], b[1]);
                        mma_bf16(s1, qa[2 * kk + 1][0], 0u, qa[2 * kk + 1][1], 0u, b[2], b[3]);
                    }
                    sum[0] = s0[0] + s1[0];
                    sum[1] = s0[1] + s1[1];
                } else {
                    const int row = nt * 8 + g;
#pragma unroll
                    for (int b = 0; b < D / 64; ++b) {
                        float s0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, s1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                        if constexpr (KIND == HS_KV_INT8) {
                            const uint4 kv = *reinterpret_cast<const uint4 *>(pK + row * LT::kRow + (((4 * b + j) ^ LT::swz(row)) << 4));
                            const uint32_t kw[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                uint32_t b0, b1;
                                codes4_bf16(kw[s], b0, b1);
                                mma_bf16((s & 1) ? s1 : s0, qa[4 * b + s][0], 0u, qa[4 * b + s][1], 0u, b0, b1);
                            }
                        } else {
                            const int at = 32 * b + 8 * j;  // byte of the row; a byte's high nibble is its even element
                            const uint2 kv = *reinterpret_cast<const uint2 *>(pK + row * LT::kRow + (((at >> 4) ^ LT::swz(row)) << 4) + (at & 15));
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                const uint32_t w = s < 2 ? kv.x : kv.y;
                                const uint2 v0 = lut_pairs<kLutStride>(lut, w, 2 * (s & 1)), v1 = lut_pairs<kLutStride>(lut, w, 2 * (s & 1) + 1);
                                mma_bf16(s0, qa[4 * b + s][0], 0u, qa[4 * b + s][1], 0u, v0.x, v1.x);
                                if (two_terms) mma_bf16(s1, qa[4 * b + s][0], 0u, qa[4 * b + s][1], 0u, v0.y, v1.y);
                                if constexpr (EXACT) {
                                    if (two_terms)
                                        mma_bf16(s1, qa[4 * b + s][0], 0u, qa[4 * b + s][1], 0u, lut_third<kLut2Stride>(lut2, w, 2 * (s & 1)),
                                                 lut_third<kLut2Stride>(lut2, w, 2 * (s & 1) + 1));
                                }
                            }
                        }
                        const float2 ks = *reinterpret_cast<const float2 *>(sc + (b >> (kLog2(D / 64) - bpr_shift)) * kMmTile + nt * 8 + 2 * j);
                        sum[0] = fmaf(s0[0] + s1[0], ks.x, sum[0]);
                        sum[1] = fmaf(s0[1] + s1[1], ks.y, sum[1]);
                    }
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    p[nt][e] = t0 + nt * 8 + 2 * j + e < L ? sum[e] * scale_log2 : -INFINITY;
                    mx = fmaxf(mx, p[nt][e]);
                }
            }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float m_new = fmaxf(m, mx);
            const float corr = m_new == -INFINITY ? 1.0f : exp2f(m - m_new);
            m = m_new;
            float psum = 0.0f;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    p[nt][e] = m_new == -INFINITY ? 0.0f : exp2f(p[nt][e] - m_new);
                    psum += p[nt][e];
                }
            l = l * corr + psum;
            if (__any_sync(0xffffffffu, corr != 1.0f)) {
                // the accumulators' columns are heads 2j, 2j + 1: their factors are in the lanes of those score rows
                const float c0 = __shfl_sync(0xffffffffu, corr, 8 * j), c1 = __shfl_sync(0xffffffffu, corr, 8 * j + 4);
#pragma unroll
                for (int i = 0; i < D / 16; ++i) { O[i][0] *= c0; O[i][1] *= c1; O[i][2] *= c0; O[i][3] *= c1; }
                if constexpr (G == 8) {
#pragma unroll
                    for (int i = 0; i < kLo; ++i) { Olo[i][0] *= c0; Olo[i][1] *= c1; Olo[i][2] *= c0; Olo[i][3] *= c1; }
                }
            }
            // P (times V's scale of a block) as two bf16 terms; ph / pl: the B operands of the upper and lower term.  EXACT: three terms,
            // in 8 columns as far as they go: up to 2 heads, ph has them all; 4 heads, the third has an MMA of its own with pt, whose
            // upper columns must carry something of P too (an infinite value times zero would be NaN): half of the upper term in
            // this MMA and half in the first one's ph2; 8 heads, an MMA each.
            uint32_t ph[2], pl[2], pt[2], ph2[2];
            auto split_p = [&](float2 v0, float2 v1) {
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    const float a = p[nt][0] * (nt ? v1.x : v0.x), b = p[nt][1] * (nt ? v1.y : v0.y);
                    if constexpr (EXACT) {
                        const uint32_t half = pack_bf16(0.5f * a, 0.5f * b);
                        ph[nt] = pack_bf16(2.0f * bf16lo(half), 2.0f * bf16hi(half));
                        const float ra = a - bf16lo(ph[nt]), rb = b - bf16hi(ph[nt]);
                        pl[nt] = pack_bf16(ra, rb);
                        pt[nt] = pack_bf16(ra - bf16lo(pl[nt]), rb - bf16hi(pl[nt]));
                        if constexpr (G <= 2) {
                            ph[nt] = g < G ? ph[nt] : (g / G == 2 ? pt[nt] : pl[nt]);
                        } else if constexpr (G == 4) {
                            ph2[nt] = low_half ? pl[nt] : half;
                            pt[nt] = low_half ? pt[nt] : half;
                            if (low_half) ph[nt] = pl[nt];
                        }
                        continue;
                    }
                    ph[nt] = pack_bf16(a, b);
                    pl[nt] = pack_bf16(a - bf16lo(ph[nt]), b - bf16hi(ph[nt]));
                    if (low_half) ph[nt] = pl[nt];
                }
            };
            // EXACT: O^T += (all terms of A).P^T, the tile's sum on its own first: an MMA cuts its sum off at the accumulator's last
            // bit, which over thousands of tokens is more than the rounding of as many additions
            auto pv_exact = [&](int mt, const uint4 *a, int terms) {
                float t[4] = {0.0f, 0.0f, 0.0f, 0.0f}, tl[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int i = 2; i >= 0; --i) {
                    if (i >= terms) continue;
                    if constexpr (G == 8) {
                        if (i == 0) mma_bf16(tl, a[i].x, a[i].y, a[i].z, a[i].w, pt[0], pt[1]);
                        if (i <= 1) mma_bf16(tl, a[i].x, a[i].y, a[i].z, a[i].w, pl[0], pl[1]);
                    }
                    if (G == 4 && i == 0) {
                        mma_bf16(t, a[i].x, a[i].y, a[i].z, a[i].w, pt[0], pt[1]);
                        mma_bf16(t, a[i].x, a[i].y, a[i].z, a[i].w, ph2[0], ph2[1]);
                    } else {
                        mma_bf16(t, a[i].x, a[i].y, a[i].z, a[i].w, ph[0], ph[1]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    O[mt][i] += t[i];
                    if constexpr (G == 8) Olo[mt][i] += tl[i];
                }
            };
            // O^T += A.P^T; low: A is the lower term of the values
            auto pv = [&](int mt, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, bool low) {
                if constexpr (EXACT) {
                    const uint4 a = make_uint4(a0, a1, a2, a3);
                    pv_exact(mt, &a, 1);
                    return;
                }
                mma_bf16(O[mt], a0, a1, a2, a3, ph[0], ph[1]);
                if constexpr (G == 8) {
                    if (!low) mma_bf16(Olo[mt], a0, a1, a2, a3, pl[0], pl[1]);
                }
            };
            if constexpr (!kQuant) {
                split_p(make_float2(1.0f, 1.0f), make_float2(1.0f, 1.0f));
                const int row = ((lane >> 4) & 1) * 8 + (lane & 7);
                const uint32_t vr = sV + row * LT::kRow;
#pragma unroll
                for (int mt = 0; mt < D / 16; ++mt) {
                    uint32_t a[4];
                    ldsm4_t(a, vr + (((2 * mt + ((lane >> 3) & 1)) ^ LT::swz(row)) << 4));
                    pv(mt, a[0], a[1], a[2], a[3], false);
                }
            } else {
#pragma unroll
                for (int b = 0; b < D / 64; ++b) {
                    const float *vs = sc + kMaxBpr * kMmTile + (b >> (kLog2(D / 64) - bpr_shift)) * kMmTile + 2 * j;
                    split_p(*reinterpret_cast<const float2 *>(vs), *reinterpret_cast<const float2 *>(vs + 8));
                    if constexpr (KIND == HS_KV_INT8) {
                        // this lane's 8 codes d = 64 b + 8 g .. + 7 of its four tokens; word k, m-tile h of it: row g is d = 8 g + 4 k + 2 h,
                        // row g + 8 the next one
                        uint2 x[2][2];
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int row = nt * 8 + 2 * j + e, at = 64 * b + 8 * g;
                                x[nt][e] = *reinterpret_cast<const uint2 *>(pV + row * LT::kRow + (((at >> 4) ^ LT::swz(row)) << 4) + (at & 15));
                            }
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            uint32_t a01[2][2], a23[2][2];  // [nt][token e]: pairs (d, d + 1) and (d + 2, d + 3) of one token
#pragma unroll
                            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                                for (int e = 0; e < 2; ++e) codes4_bf16(k ? x[nt][e].y : x[nt][e].x, a01[nt][e], a23[nt][e]);
                            pv(4 * b + 2 * k, __byte_perm(a01[0][0], a01[0][1], 0x5410), __byte_perm(a01[0][0], a01[0][1], 0x7632),
                               __byte_perm(a01[1][0], a01[1][1], 0x5410), __byte_perm(a01[1][0], a01[1][1], 0x7632), false);
                            pv(4 * b + 2 * k + 1, __byte_perm(a23[0][0], a23[0][1], 0x5410), __byte_perm(a23[0][0], a23[0][1], 0x7632),
                               __byte_perm(a23[1][0], a23[1][1], 0x5410), __byte_perm(a23[1][0], a23[1][1], 0x7632), false);
                        }
                    } else {
                        // 4 bytes d = 64 b + 8 g .. + 7 of each token; the nibbles of a token pair are mixed first, so that a lookup gives
                        // the pair's two values of one element: byte k of `even` is d = 8 g + 2 k (row g of m-tile k), of `odd` the next
                        // element (row g + 8)
                        uint32_t even[2], odd[2];
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt) {
                            uint32_t x[2];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int row = nt * 8 + 2 * j + e, at = 32 * b + 4 * g;
                                x[e] = *reinterpret_cast<const uint32_t *>(pV + row * LT::kRow + (((at >> 4) ^ LT::swz(row)) << 4) + (at & 15));
                            }
                            even[nt] = (x[0] & 0xf0f0f0f0u) | ((x[1] >> 4) & 0x0f0f0f0fu);
                            odd[nt] = ((x[0] << 4) & 0xf0f0f0f0u) | (x[1] & 0x0f0f0f0fu);
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint2 a0 = lut_pairs<kLutStride>(lut, even[0], k), a1 = lut_pairs<kLutStride>(lut, odd[0], k);
                            const uint2 a2 = lut_pairs<kLutStride>(lut, even[1], k), a3 = lut_pairs<kLutStride>(lut, odd[1], k);
                            if constexpr (EXACT) {
                                uint4 a[3] = {make_uint4(a0.x, a1.x, a2.x, a3.x), make_uint4(a0.y, a1.y, a2.y, a3.y), make_uint4(0u, 0u, 0u, 0u)};
                                if (two_terms)
                                    a[2] = make_uint4(lut_third<kLut2Stride>(lut2, even[0], k), lut_third<kLut2Stride>(lut2, odd[0], k),
                                                      lut_third<kLut2Stride>(lut2, even[1], k), lut_third<kLut2Stride>(lut2, odd[1], k));
                                pv_exact(4 * b + k, a, two_terms ? 3 : 1);
                                continue;
                            }
                            pv(4 * b + k, a0.x, a1.x, a2.x, a3.x, false);
                            if (two_terms) pv(4 * b + k, a0.y, a1.y, a2.y, a3.y, true);
                        }
                    }
                }
            }
            __syncwarp();  // every lane has read the stage before the next fetch overwrites it
            stage = stage + 1 == kStages ? 0 : stage + 1;
        }

        // ---- the CTA's partial of this sequence: the warps' sums through shared memory ----
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        __syncthreads();  // the readers of the previous sequence's sums are done
        if (j == 0 && !low_half && g < G) {
            m_ml[(warp * G + g) * 2] = m;
            m_ml[(warp * G + g) * 2 + 1] = l;
        }
#pragma unroll
        for (int mt = 0; mt < D / 16; ++mt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float hi_sum = O[mt][i];
                float lo_sum;
                if constexpr (G == 8) lo_sum = Olo[mt][i];
                else if constexpr (EXACT && G == 2) lo_sum = __shfl_down_sync(0xffffffffu, hi_sum, 1) + __shfl_down_sync(0xffffffffu, hi_sum, 2);
                else if constexpr (EXACT && G == 1) lo_sum = __shfl_down_sync(0xffffffffu, hi_sum, 1) + O[mt][i | 1];
                else lo_sum = __shfl_xor_sync(0xffffffffu, hi_sum, 2);  // columns 4..7 are the low parts of heads 0..3
                const int hd = 2 * j + (i & 1);
                int d;  // element that row g (i < 2) or g + 8 of m-tile mt stands for
                if constexpr (!kQuant) d = 16 * mt + 8 * (i >> 1) + g;
                else if constexpr (KIND == HS_KV_INT8) d = 64 * (mt >> 2) + 8 * g + 4 * ((mt >> 1) & 1) + 2 * (mt & 1) + (i >> 1);
                else d = 64 * (mt >> 2) + 8 * g + 2 * (mt & 3) + (i >> 1);
                // (an infinite sum stands: its low part is 0 x inf)
                if (hd < G) m_o[(warp * G + hd) * LT::kORow + d] = fabsf(hi_sum) == INFINITY ? hi_sum : hi_sum + lo_sum;
            }
        __syncthreads();
        const int64_t slot = cta + r;
        for (int idx = threadIdx.x; idx < G * D; idx += kMmThreads) {
            const int gg = idx / D, d = idx % D;
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < kMmWarps; ++w) M = fmaxf(M, m_ml[(w * G + gg) * 2]);
            float num = 0.0f, den = 0.0f;
#pragma unroll
            for (int w = 0; w < kMmWarps; ++w) {
                const float mw = m_ml[(w * G + gg) * 2];
                const float wgt = mw == -INFINITY ? 0.0f : exp2f(mw - M);
                num = fmaf(wgt, m_o[(w * G + gg) * LT::kORow + d], num);
                den = fmaf(wgt, m_ml[(w * G + gg) * 2 + 1], den);
            }
            const int64_t hrow = slot * n_q_heads + kvh * G + gg;
            o_part[hrow * D + d] = den > 0.0f ? num / den : 0.0f;
            if (d == 0) lse_part[hrow] = den > 0.0f ? (M + log2f(den)) * 0.6931471805599453f : -INFINITY;
        }
        before += nt_seq;
    }
    mm_wait<0>();
}

template <int KIND, int D, int G, bool EXACT>
static int32_t launch_mma(const ViewDev &v, const uint16_t *q, const int32_t *seq_lens, int n_seqs, int n_q_heads, float scale_log2, float *o_part,
                          float *lse_part, int *err, int max_ctas, int *n_ctas_out, bool after_write, const AppendArgs &ap, cudaStream_t s) {
    using LT = MmLayout<KIND, D, G, EXACT>;
    auto kern = decode_mma_kernel<KIND, D, G, EXACT>;
    static PerDeviceState configured;
    const int dev = current_device();
    if (configured.get(dev) == 0) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LT::kTotal);
        if (e != cudaSuccess) return fail(static_cast<int32_t>(e), "hs_attn_decode: %s", cudaGetErrorString(e));
        configured.set(dev, 1);
    }
    // one wave: every resident CTA takes an equal share of the tile list of its kv head
    const int n_ctas = max(1, min(LT::kCtasPerSm * sm_count() / v.n_kv_heads, max_ctas));
    *n_ctas_out = n_ctas;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_ctas, v.n_kv_heads);
    cfg.blockDim = dim3(kMmThreads);
    cfg.dynamicSmemBytes = LT::kTotal;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = after_write ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, v, q, seq_lens, n_seqs, n_q_heads, scale_log2, o_part, lse_part, err, ap);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(static_cast<int32_t>(e), "hs_attn_decode: %s", cudaGetErrorString(e));
    }
    return HS_OK;
}

// `ap` (a bf16 cache of one sequence in one page, else k_new == NULL): the step's new token.  *n_ctas_out = CTAs per kv head, *tile_out = tokens per tile, as the merge kernel needs them.
// `exact`: the caller takes fp32 results.
int32_t decode_mma(const ViewDev &v, const uint16_t *q, const int32_t *seq_lens, int n_seqs, int n_q_heads, float scale_log2, float *o_part,
                   float *lse_part, int *err, int max_ctas, int *n_ctas_out, int *tile_out, bool after_write, bool exact, const AppendArgs &ap, cudaStream_t s) {
    *tile_out = kMmTile;
    const int G = n_q_heads / v.n_kv_heads;
#define HS_MMA_ARGS v, q, seq_lens, n_seqs, n_q_heads, scale_log2, o_part, lse_part, err, max_ctas, n_ctas_out, after_write, ap, s
#define HS_MMA_RUN(K, DD, GG) exact ? launch_mma<K, DD, GG, true>(HS_MMA_ARGS) : launch_mma<K, DD, GG, false>(HS_MMA_ARGS)
#define HS_MMA_G(K, DD) \
    switch (G) { \
        case 1: return HS_MMA_RUN(K, DD, 1); \
        case 2: return HS_MMA_RUN(K, DD, 2); \
        case 4: return HS_MMA_RUN(K, DD, 4); \
        case 8: return HS_MMA_RUN(K, DD, 8); \
        default: return fail(HS_ERR_UNSUPPORTED, "hs_attn_decode: n_q_heads / n_kv_heads = %d (supported: 1, 2, 4, 8)", G); \
    }
#define HS_MMA_D(K) \
    switch (v.head_dim) { \
        case 64: HS_MMA_G(K, 64) \
        case 128: HS_MMA_G(K, 128) \
        case 256: HS_MMA_G(K, 256) \
        default: return fail(HS_ERR_UNSUPPORTED, "hs_attn_decode: head_dim %d", v.head_dim); \
    }
    switch (v.kind) {
        case HS_KV_BF16: HS_MMA_D(HS_KV_BF16)
        case HS_KV_INT8: HS_MMA_D(HS_KV_INT8)
        default: HS_MMA_D(HS_KV_NF4)
    }
#undef HS_MMA_D
#undef HS_MMA_G
#undef HS_MMA_RUN
#undef HS_MMA_ARGS
}

}  // namespace hs
