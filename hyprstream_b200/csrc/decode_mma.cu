// Decode attention over a bf16 cache, any head_dim in {64, 128, 256} and 1 / 2 / 4 / 8 query heads per kv head, on the tensor
// cores.  Same partition, same partials and same merge kernel as the CUDA-core kernel of decode.cu, which it replaces for bf16.
//
// HBM bound: a cached token of one kv head is 4 * head_dim bytes and is read once.  What the CUDA-core form spent its time on
// instead: two tokens in flight per lane group (latency), and 2 * G fp32 FMAs plus the unpacking per element (issue).  Here
//   * a warp works by itself: 16 tokens of one kv head are one tile, its K and V rows come into the warp's own ring of shared
//     memory with 16-byte cp.async (rows XOR-swizzled, so that ldmatrix is free of bank conflicts); no block barrier inside a
//     sequence, any page size, rows past the end of a sequence filled with zeros;
//   * S = q.K^T on mma.sync m16n8k16 with the query heads as rows (bf16 operands as stored: exact products, fp32 sums) and
//     O^T += V^T.P^T with head_dim as rows, so that P's accumulator registers are the B operand as they are;
//   * P keeps 16 bits of mantissa: p = hi + lo, both bf16.  With up to 4 query heads the second half of the MMA's 8 columns is
//     free and carries lo (one MMA for both); with 8 heads lo takes an MMA and an accumulator of its own;
//   * the warps of a CTA merge their sums at the end of a sequence and write one partial per (CTA, sequence).
// Measured against the CUDA-core form (32 / 8 heads x 128, a cold launch by itself): 16 paged sequences of 100 to 6,000 tokens
// (247 MB) 150 -> 44.0 us = 5.6 TB/s; one sequence of 4,096 tokens 23.3 -> 9.3 us.
#include "hs_common.cuh"

namespace hs {

constexpr int kMmWarps = 4;
constexpr int kMmThreads = kMmWarps * 32;
constexpr int kMmTile = 16;  // tokens per tile of the flat partition = one warp step

template <int D, int G>
struct MmLayout {
    static constexpr int kRow = D * 2;                  // bytes of one (token, head) row
    static constexpr int kTileBytes = 2 * kMmTile * kRow;
    // bytes in flight: 6.5 TB/s / 148 SMs at ~1 us is ~44 KB per SM; the rings hold 160-192 KB per SM
    static constexpr int kStages = D == 128 ? 3 : (D == 256 ? 3 : 5);
    static constexpr int kCtasPerSm = D == 256 ? 1 : 2;
    static constexpr int kORow = D + 4;                 // floats between the heads of a warp's merge rows (bank spread)
    static constexpr int kMergeOff = kMmWarps * kStages * kTileBytes;
    static constexpr int kMlOff = kMergeOff + kMmWarps * G * kORow * 4;
    static constexpr int kTotal = kMlOff + kMmWarps * G * 2 * 4;
    static_assert(kCtasPerSm * (kTotal + 1024) <= 228 * 1024, "the CTAs of an SM must fit its shared memory");
};

__device__ __forceinline__ void mm_cp16(uint32_t dst, const void *src, int bytes) {  // bytes = 16, or 0: sixteen zero bytes, src not read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
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

template <int D, int G>
__global__ void __launch_bounds__(kMmThreads, MmLayout<D, G>::kCtasPerSm)
decode_bf16_mma_kernel(ViewDev view, const uint16_t *__restrict__ q, const int32_t *__restrict__ seq_lens, int n_seqs, int n_q_heads,
                       float scale_log2, float *__restrict__ o_part, float *__restrict__ lse_part, int *__restrict__ err) {
    using LT = MmLayout<D, G>;
    constexpr int kChunks = D / 8;                 // 16-byte chunks of a row
    constexpr int kStages = LT::kStages;
    extern __shared__ __align__(128) unsigned char mm_smem[];
    // the merge kernel that follows as a programmatic dependent may start; it waits for this grid before it reads anything
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kvh = blockIdx.y, H = view.n_kv_heads;
    const int64_t cta = blockIdx.x;
    const int cap = view.page_tokens * view.pages_per_seq;  // lengths beyond the view's pages are cut (and recorded)
    auto tiles_of = [&](int L) { return (min(max(L, 0), cap) + kMmTile - 1) / kMmTile; };

    // ---- the CTA's range of the concatenated tile list (every warp for itself, 32 lengths per load) ----
    int64_t total = 0;
    bool over = false;
    for (int base = 0; base < n_seqs; base += 32) {
        const int L = base + lane < n_seqs ? seq_lens[base + lane] : 0;
        over |= L > cap;
        total += __reduce_add_sync(0xffffffffu, static_cast<unsigned>(tiles_of(L)));
    }
    if (over && warp == 0 && cta == 0 && kvh == 0) atomicOr(err, HS_DEVERR_DECODE_RANGE);
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

    // ---- feeding the ring: this warp's tiles are t_begin + warp, + kMmWarps, ... ----
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(mm_smem)) + warp * (kStages * LT::kTileBytes);
    int64_t f_tile = t_begin + warp, f_before = before_first;  // next tile to fetch; tiles in front of sequence f_r
    int f_r = r_first, f_len = min(max(seq_lens[r_first], 0), cap), f_stage = 0;
    const bool whole_pages = view.pages_per_seq == 1 || view.page_tokens % kMmTile == 0;  // a tile lies in one page
    auto fetch = [&]() {
        if (f_tile < t_end) {
            int nt = (f_len + kMmTile - 1) / kMmTile;
            while (f_tile >= f_before + nt) {
                f_before += nt;
                f_len = min(max(seq_lens[++f_r], 0), cap);
                nt = (f_len + kMmTile - 1) / kMmTile;
            }
            const int t0 = static_cast<int>(f_tile - f_before) * kMmTile;
            void *const *kp = view.k_pages + static_cast<int64_t>(f_r) * view.pages_per_seq;
            void *const *vp = view.v_pages + static_cast<int64_t>(f_r) * view.pages_per_seq;
            const uint32_t sK = ring + f_stage * LT::kTileBytes;
            const int page0 = view.pages_per_seq == 1 ? 0 : t0 / view.page_tokens;
            const unsigned char *k0 = reinterpret_cast<const unsigned char *>(kp[page0]), *v0 = reinterpret_cast<const unsigned char *>(vp[page0]);
            constexpr int kPer = kMmTile * kChunks / 32, kRows = 32 / kChunks;  // copies per lane and operand; rows the warp covers per copy
            const int row0 = lane / kChunks, c = lane % kChunks;
            if (whole_pages) {
                const int64_t off = (static_cast<int64_t>(t0 - page0 * view.page_tokens + row0) * H + kvh) * LT::kRow + c * 16;
                const int64_t step = static_cast<int64_t>(kRows) * H * LT::kRow;
                const unsigned char *ka = k0 + off, *va = v0 + off;
#pragma unroll 4
                for (int i = 0; i < kPer; ++i, ka += step, va += step) {
                    const int row = i * kRows + row0;
                    const bool live = t0 + row < f_len;
                    const uint32_t dst = sK + row * LT::kRow + ((c ^ (row & 7)) << 4);
                    mm_cp16(dst, live ? ka : k0, live ? 16 : 0);
                    mm_cp16(dst + kMmTile * LT::kRow, live ? va : v0, live ? 16 : 0);
                }
            } else {
#pragma unroll 1
                for (int i = 0; i < kPer; ++i) {
                    const int row = i * kRows + row0, t = t0 + row;
                    const bool live = t < f_len;
                    const int page = live ? t / view.page_tokens : page0;
                    const int64_t off = live ? (static_cast<int64_t>(t - page * view.page_tokens) * H + kvh) * LT::kRow + c * 16 : 0;
                    const uint32_t dst = sK + row * LT::kRow + ((c ^ (row & 7)) << 4);
                    mm_cp16(dst, reinterpret_cast<const unsigned char *>(kp[page]) + off, live ? 16 : 0);
                    mm_cp16(dst + kMmTile * LT::kRow, reinterpret_cast<const unsigned char *>(vp[page]) + off, live ? 16 : 0);
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
        uint32_t qa[D / 16][2];
        const uint16_t *qp = q + (static_cast<int64_t>(r) * n_q_heads + kvh * G + head) * D + 2 * j;
#pragma unroll
        for (int s = 0; s < D / 16; ++s) {
            qa[s][0] = *reinterpret_cast<const uint32_t *>(qp + 16 * s);
            qa[s][1] = *reinterpret_cast<const uint32_t *>(qp + 16 * s + 8);
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
            const int t0 = static_cast<int>(tile - before) * kMmTile;
            // ---- scores of 16 tokens: two n-tiles of 8, even and odd k-steps in accumulators of their own ----
            float p[2][2];
            float mx = -INFINITY;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float s0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, s1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                const int row = nt * 8 + (lane & 7);
                const uint32_t kr = sK + row * LT::kRow;
#pragma unroll
                for (int kk = 0; kk < D / 32; ++kk) {
                    uint32_t b[4];
                    ldsm4(b, kr + (((kk * 4 + (lane >> 3)) ^ (row & 7)) << 4));
                    mma_bf16(s0, qa[2 * kk][0], 0u, qa[2 * kk][1], 0u, b[0], b[1]);
                    mma_bf16(s1, qa[2 * kk + 1][0], 0u, qa[2 * kk + 1][1], 0u, b[2], b[3]);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    p[nt][e] = t0 + nt * 8 + 2 * j + e < L ? (s0[e] + s1[e]) * scale_log2 : -INFINITY;
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
            uint32_t ph[2], pl[2];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                ph[nt] = pack_bf16(p[nt][0], p[nt][1]);
                pl[nt] = pack_bf16(p[nt][0] - bf16lo(ph[nt]), p[nt][1] - bf16hi(ph[nt]));
                if (low_half) ph[nt] = pl[nt];
            }
            // ---- O^T += V^T.P^T ----
            {
                const int row = ((lane >> 4) & 1) * 8 + (lane & 7);
                const uint32_t vr = sV + row * LT::kRow;
#pragma unroll
                for (int mt = 0; mt < D / 16; ++mt) {
                    uint32_t a[4];
                    ldsm4_t(a, vr + (((2 * mt + ((lane >> 3) & 1)) ^ (row & 7)) << 4));
                    mma_bf16(O[mt], a[0], a[1], a[2], a[3], ph[0], ph[1]);
                    if constexpr (G == 8) mma_bf16(Olo[mt], a[0], a[1], a[2], a[3], pl[0], pl[1]);
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
                else lo_sum = __shfl_xor_sync(0xffffffffu, hi_sum, 2);  // columns 4..7 are the low parts of heads 0..3
                const int hd = 2 * j + (i & 1), d = 16 * mt + 8 * (i >> 1) + g;
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

template <int D, int G>
static int32_t launch_mma(const ViewDev &v, const uint16_t *q, const int32_t *seq_lens, int n_seqs, int n_q_heads, float scale_log2, float *o_part,
                          float *lse_part, int *err, int max_ctas, int *n_ctas_out, bool after_write, cudaStream_t s) {
    using LT = MmLayout<D, G>;
    auto kern = decode_bf16_mma_kernel<D, G>;
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
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, v, q, seq_lens, n_seqs, n_q_heads, scale_log2, o_part, lse_part, err);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(static_cast<int32_t>(e), "hs_attn_decode: %s", cudaGetErrorString(e));
    }
    return HS_OK;
}

// The bf16 decode kernel; *n_ctas_out = CTAs per kv head, *tile_out = tokens per tile, as the merge kernel needs them.
int32_t decode_bf16_mma(const ViewDev &v, const uint16_t *q, const int32_t *seq_lens, int n_seqs, int n_q_heads, float scale_log2, float *o_part,
                        float *lse_part, int *err, int max_ctas, int *n_ctas_out, int *tile_out, bool after_write, cudaStream_t s) {
    *tile_out = kMmTile;
    const int G = n_q_heads / v.n_kv_heads;
#define HS_MMA_G(DD) \
    switch (G) { \
        case 1: return launch_mma<DD, 1>(v, q, seq_lens, n_seqs, n_q_heads, scale_log2, o_part, lse_part, err, max_ctas, n_ctas_out, after_write, s); \
        case 2: return launch_mma<DD, 2>(v, q, seq_lens, n_seqs, n_q_heads, scale_log2, o_part, lse_part, err, max_ctas, n_ctas_out, after_write, s); \
        case 4: return launch_mma<DD, 4>(v, q, seq_lens, n_seqs, n_q_heads, scale_log2, o_part, lse_part, err, max_ctas, n_ctas_out, after_write, s); \
        case 8: return launch_mma<DD, 8>(v, q, seq_lens, n_seqs, n_q_heads, scale_log2, o_part, lse_part, err, max_ctas, n_ctas_out, after_write, s); \
        default: return fail(HS_ERR_UNSUPPORTED, "hs_attn_decode: n_q_heads / n_kv_heads = %d (supported: 1, 2, 4, 8)", G); \
    }
    switch (v.head_dim) {
        case 64: HS_MMA_G(64)
        case 128: HS_MMA_G(128)
        case 256: HS_MMA_G(256)
        default: return fail(HS_ERR_UNSUPPORTED, "hs_attn_decode: head_dim %d", v.head_dim);
    }
#undef HS_MMA_G
}

}  // namespace hs
