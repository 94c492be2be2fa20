// Decode attention (one query token per sequence) over a bf16 / int8 / 4-bit KV cache view, with a
// flat split-KV partition over all sequences and a log-sum-exp merge.
//
// Fused replacement of cache.get() -> GQA expansion -> transposes -> fp32 upcast -> q@K^T*scale ->
// softmax -> @V (architectures/llama.rs:605-640,847-872,1023-1119; the batched ragged form
// llama.rs:710-844 with its padding mask 2540-2572; qwen3_5.rs:992-1059 for the gated variant).
// The cache is read exactly once, in its stored precision, and dequantised in registers.
//
// This file holds the entry points, the choice of the kernel (decode_tc.cu: quantised caches of the two served models' shapes;
// decode_mma.cu: everything else) and the merge kernel.
#include <mutex>

#include "hs_common.cuh"

namespace hs {

__device__ __forceinline__ int ceil_div_i(int a, int b) { return (a + b - 1) / b; }

// Merge the split-KV partials of one (sequence, query head) per CTA.  The CTAs that hold tiles of the sequence follow from
// seq_lens with the same partition arithmetic the decode kernel used: CTA c and sequence r share slot c + r, no CTA of the
// range is empty, so the partials are consecutive.  Latency bound (a few dozen partials of D floats from L2): D / 4 threads
// take a partial with 16-byte loads and the CTA's thread groups take every kMergeThreads / (D / 4)-th, so that a batch of one
// sequence has all its partials in flight at once.  One query head a CTA and closed-form ends of the range instead of four
// heads a CTA and one thread walking the CTA list with 64-bit divisions: 50.8 -> 8.2 us for 1 x 4096 tokens (a cold launch by itself).
constexpr int kMergeThreads = 256;
__global__ void __launch_bounds__(kMergeThreads)
decode_merge_kernel(const int32_t *__restrict__ seq_lens, int n_seqs, int n_q_heads, int D, int n_ctas, int tile, int cap,
                    const float *__restrict__ o_part, const float *__restrict__ lse_part, uint16_t *__restrict__ out,
                    const uint16_t *__restrict__ gate, float *__restrict__ o_shard, float *__restrict__ lse_shard) {
    __shared__ float4 s_num[kMergeThreads];
    const int r = blockIdx.x / n_q_heads, h = blockIdx.x - r * n_q_heads, lane = threadIdx.x & 31;
    // Tiles of all sequences, and of those in front of r, one coalesced load per 32 lengths.  A short list is summed by every warp for
    // itself, a long one (there are n_seqs * n_q_heads CTAs) by all warps together.  bf16 32 / 8 heads x 128, up to 64 tokens, the whole
    // call: 257 sequences 67.6 us together (256 by every warp: 85.4), 4,000 sequences 6,527 by every warp, 1,672 together.
    int64_t total = 0, before = 0;
    const bool together = n_seqs > 64;  // (one or two loads by every warp cost less than the barrier)
    for (int base = together ? threadIdx.x & ~31 : 0; base < n_seqs; base += together ? kMergeThreads : 32) {
        const int i = base + lane;
        const unsigned t = i < n_seqs ? ceil_div_i(min(max(seq_lens[i], 0), cap), tile) : 0;
        total += __reduce_add_sync(0xffffffffu, t);
        before += __reduce_add_sync(0xffffffffu, i < r ? t : 0u);
    }
    if (together) {
        __shared__ int64_t s_sum[2][kMergeThreads / 32];
        if (lane == 0) {
            s_sum[0][threadIdx.x >> 5] = total;
            s_sum[1][threadIdx.x >> 5] = before;
        }
        __syncthreads();
        total = before = 0;
#pragma unroll
        for (int w = 0; w < kMergeThreads / 32; ++w) {
            total += s_sum[0][w];
            before += s_sum[1][w];
        }
    }
    const int64_t nt = ceil_div_i(min(max(seq_lens[r], 0), cap), tile);
    if (total < n_ctas) n_ctas = total > 0 ? static_cast<int>(total) : 1;  // the decode kernels never use more CTAs than tiles
    int np = 0;
    int64_t slot0 = 0;
    if (nt > 0) {
        // tile t belongs to the last CTA c with floor(c * total / n_ctas) <= t, i.e. c * total < (t + 1) * n_ctas
        const int64_t c_lo = ((before + 1) * n_ctas - 1) / total, c_hi = ((before + nt) * n_ctas - 1) / total;
        np = static_cast<int>(c_hi - c_lo + 1);
        slot0 = c_lo + r;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // everything above overlaps with the decode kernel's end; its partials are read below
    const float *lse = lse_part + slot0 * n_q_heads + h;
    float M = -INFINITY;
    for (int i = lane; i < np; i += 32) M = fmaxf(M, lse[static_cast<int64_t>(i) * n_q_heads]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    float den = 0.0f;
    for (int i = lane; i < np; i += 32) {
        const float ls = lse[static_cast<int64_t>(i) * n_q_heads];
        den += ls == -INFINITY ? 0.0f : __expf(ls - M);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) den += __shfl_xor_sync(0xffffffffu, den, off);
    const int dt = D / 4, groups = kMergeThreads / dt;          // threads per partial, partials at a time
    const int grp = threadIdx.x / dt, d = (threadIdx.x - grp * dt) * 4;
    const float *op = o_part + (slot0 * n_q_heads + h) * D + d;
    const int64_t stride = static_cast<int64_t>(n_q_heads) * D;
    float4 num = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int i = grp; i < np; i += groups) {
        const float ls = lse[static_cast<int64_t>(i) * n_q_heads];
        const float4 v = *reinterpret_cast<const float4 *>(op + i * stride);
        const float w = ls == -INFINITY ? 0.0f : __expf(ls - M);
        num.x = fmaf(w, v.x, num.x); num.y = fmaf(w, v.y, num.y); num.z = fmaf(w, v.z, num.z); num.w = fmaf(w, v.w, num.w);
    }
    s_num[threadIdx.x] = num;
    __syncthreads();
    if (grp != 0) return;
    for (int k = 1; k < groups; ++k) {
        const float4 v = s_num[k * dt + threadIdx.x];
        num.x += v.x; num.y += v.y; num.z += v.z; num.w += v.w;
    }
    const int64_t row = static_cast<int64_t>(r) * n_q_heads + h;
    const float o[4] = {num.x, num.y, num.z, num.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float v = den > 0.0f ? o[i] / den : 0.0f;
        if (o_shard != nullptr) {
            o_shard[row * D + d + i] = v;
            continue;
        }
        float res = v;
        if (gate != nullptr) {
            const float gv = bf16_bits_to_f32(gate[row * D + d + i]);
            res = bf16_round(v) * bf16_round(1.0f / (1.0f + __expf(-gv)));  // ctx * sigmoid(gate) in bf16 (qwen3_5.rs:1056-1059)
        }
        out[row * D + d + i] = f32_to_bf16_bits(res);
    }
    if (o_shard != nullptr && d == 0) lse_shard[row] = den > 0.0f ? M + __logf(den) : -INFINITY;
}

// Merge of externally produced partials (KV-length shards from several GPUs, or a caller's own split).
// Part p's outputs start at o_parts + p * stride_o floats ([n_rows, D] dense), its log-sum-exps at lse_parts + p * stride_l.
__global__ void merge_parts_kernel(const float *__restrict__ o_parts, const float *__restrict__ lse_parts, int n_parts,
                                   int64_t stride_o, int64_t stride_l, int D, uint16_t *__restrict__ out,
                                   const uint16_t *__restrict__ gate) {
    const int64_t row = blockIdx.x;
    const int d = threadIdx.x;
    float M = -INFINITY;
    for (int p = 0; p < n_parts; ++p) M = fmaxf(M, lse_parts[p * stride_l + row]);
    float num = 0.0f, den = 0.0f;
    for (int p = 0; p < n_parts; ++p) {
        const float ls = lse_parts[p * stride_l + row];
        const float wgt = ls == -INFINITY ? 0.0f : __expf(ls - M);
        num = fmaf(wgt, o_parts[p * stride_o + row * D + d], num);
        den += wgt;
    }
    float res = den > 0.0f ? num / den : 0.0f;
    if (gate != nullptr) {
        const float gv = bf16_bits_to_f32(gate[row * D + d]);
        res = bf16_round(res) * bf16_round(1.0f / (1.0f + __expf(-gv)));
    }
    out[row * D + d] = f32_to_bf16_bits(res);
}

static int decode_max_ctas() { return 4 * sm_count(); }
constexpr int kMaxPartsPerPair = 2;

// decode_tc.cu: cooperative tensor-core kernel for the quantised caches of the two served models' shapes
int32_t decode_int8_tc_try(const ViewDev &v, const uint16_t *q, const int32_t *seq_lens, int n_seqs, int n_q_heads,
                           float softmax_scale, float *o_part, float *lse_part, int *err, cudaStream_t s, int *n_ctas_out,
                           uint16_t *out, const uint16_t *gate, float *o_shard, float *lse_shard, int *merged_out,
                           const ShardArgs *shard, int after_write, const AppendArgs *append);

// decode_mma.cu: tensor-core kernel for every kind, head_dim and query group
int32_t decode_mma(const ViewDev &v, const uint16_t *q, const int32_t *seq_lens, int n_seqs, int n_q_heads, float scale_log2, float *o_part,
                   float *lse_part, int *err, int max_ctas, int *n_ctas_out, int *tile_out, bool after_write, bool exact, const AppendArgs &ap, cudaStream_t s);

// ---- decode scratch that lives inside the library ------------------------------------------------
// Backing store of hs_attn_decode_static(): the split-KV partials go here instead of into a workspace the
// caller would have had to allocate.  Every GPU that loads the library holds these bytes until exit.
constexpr int64_t kStaticScratchBytes = 24ll << 20;  // 24 MiB
constexpr int kStaticMaxDevices = 64;
static __device__ __align__(256) unsigned char g_decode_static_scratch[kStaticScratchBytes];
// Device address of the array on each device.  The array's name is only a host-side handle: the address a
// kernel can use has to be asked for, per device, with that device current.
static void *g_static_scratch_ptr[kStaticMaxDevices] = {nullptr};
static std::mutex g_static_scratch_mutex;

static int32_t static_scratch_for_current_device(void **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(HS_ERR_DEVICE, "hs_attn_decode_static: no usable CUDA device: %s", cudaGetErrorString(e));
    }
    if (dev < 0 || dev >= kStaticMaxDevices) return fail(HS_ERR_DEVICE, "hs_attn_decode_static: device ordinal %d is beyond the table of %d", dev, kStaticMaxDevices);
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (g_static_scratch_ptr[dev] == nullptr) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_decode_static_scratch);
        if (e != cudaSuccess || p == nullptr) {
            cudaGetLastError();
            return fail(e != cudaSuccess ? static_cast<int32_t>(e) : HS_ERR_DEVICE, "hs_attn_decode_static: cudaGetSymbolAddress failed: %s",
                        cudaGetErrorString(e));
        }
        g_static_scratch_ptr[dev] = p;
    }
    *out = g_static_scratch_ptr[dev];
    return HS_OK;
}

int32_t decode_impl(const void *q, const hs_kv_view *view, const int32_t *seq_lens, int32_t n_seqs, int32_t n_q_heads, float softmax_scale,
                    void *out, const void *gate, void *workspace, int64_t workspace_bytes, float *o_shard, float *lse_shard,
                    const ShardArgs *shard, hs_stream_t stream, int after_write = 0, const AppendArgs *append = nullptr, int *appended = nullptr);

}  // namespace hs

using namespace hs;

extern "C" {

int64_t hs_attn_decode_workspace_bytes(int32_t n_seqs, int32_t n_q_heads, int32_t head_dim) {
    if (n_seqs < 0 || n_q_heads <= 0 || head_dim <= 0) return HS_ERR_ARG;
    const int64_t slots = (static_cast<int64_t>(decode_max_ctas()) + n_seqs) * kMaxPartsPerPair;
    return slots * n_q_heads * (static_cast<int64_t>(head_dim) + 1) * 4;
}

int32_t hs_attn_decode(const void *q, const hs_kv_view *view, const int32_t *seq_lens, int32_t n_seqs, int32_t n_q_heads,
                       float softmax_scale, void *out, const void *gate, void *workspace, int64_t workspace_bytes,
                       float *o_shard, float *lse_shard, hs_stream_t stream) {
    return hs::decode_impl(q, view, seq_lens, n_seqs, n_q_heads, softmax_scale, out, gate, workspace, workspace_bytes, o_shard, lse_shard,
                           nullptr, stream);
}

}  // extern "C"

// The body of hs_attn_decode; `shard` (optional) makes the tensor-core kernel exchange its result with the other GPUs of
// a shard group and merge again (hs_attn_decode_sharded); only that kernel can, so other shapes are refused then.
int32_t hs::decode_impl(const void *q, const hs_kv_view *view, const int32_t *seq_lens, int32_t n_seqs, int32_t n_q_heads,
                        float softmax_scale, void *out, const void *gate, void *workspace, int64_t workspace_bytes,
                        float *o_shard, float *lse_shard, const ShardArgs *shard, hs_stream_t stream, int after_write, const AppendArgs *append,
                        int *appended) {
    if (appended) *appended = 0;
    if (int32_t st = check_device()) return st;
    if (int32_t st = validate_view(view)) return st;
    if (n_seqs < 0 || n_q_heads <= 0) return fail(HS_ERR_ARG, "hs_attn_decode: bad sizes");
    if (n_seqs == 0) return HS_OK;
    if (n_q_heads % view->n_kv_heads != 0) return fail(HS_ERR_ARG, "hs_attn_decode: n_q_heads %d not a multiple of n_kv_heads %d", n_q_heads, view->n_kv_heads);
    if (!q || !seq_lens || !workspace) return fail(HS_ERR_ARG, "hs_attn_decode: NULL pointer");
    if ((o_shard == nullptr) != (lse_shard == nullptr)) return fail(HS_ERR_ARG, "hs_attn_decode: o_shard and lse_shard go together");
    if (!o_shard && !out && !(shard && shard->push_only)) return fail(HS_ERR_ARG, "hs_attn_decode: no output");
    if (!aligned(q, 16) || !aligned(workspace, 16) || (out && !aligned(out, 2)) || (gate && !aligned(gate, 2)) || !aligned(seq_lens, 4))
        return fail(HS_ERR_ARG, "hs_attn_decode: q and workspace must be 16-byte aligned");
    const int D = view->head_dim;
    const int64_t need = hs_attn_decode_workspace_bytes(n_seqs, n_q_heads, D);
    if (workspace_bytes < need) return fail(HS_ERR_WORKSPACE, "hs_attn_decode: workspace %lld < %lld bytes", (long long)workspace_bytes, (long long)need);
    int *err = device_error_word();
    if (!err) return fail(HS_ERR_DEVICE, "hs_attn_decode: device error word unavailable");

    ViewDev v = to_dev(view);
    const int64_t slots = (static_cast<int64_t>(decode_max_ctas()) + n_seqs) * kMaxPartsPerPair;
    float *o_part = reinterpret_cast<float *>(workspace);
    float *lse_part = o_part + slots * n_q_heads * D;
    const float scale_log2 = softmax_scale * 1.4426950408889634f;
    cudaStream_t s = as_stream(stream);
    const uint16_t *qp = reinterpret_cast<const uint16_t *>(q);
    int32_t st;
    int n_ctas = 0, tile = 0, tc_ctas = 0, merged = 0;
    prof_begin(s);
    st = decode_int8_tc_try(v, qp, seq_lens, n_seqs, n_q_heads, softmax_scale, o_part, lse_part, err, s, &tc_ctas,
                            reinterpret_cast<uint16_t *>(out), reinterpret_cast<const uint16_t *>(gate), o_shard, lse_shard, &merged, shard, after_write, append);
    if (st == HS_OK && append && tc_ctas == 0 && view->kind != HS_KV_BF16) {  // no kernel writes these codes itself: nothing was written, the caller writes
        prof_end(s);
        return HS_OK;
    }
    if (appended && append) *appended = 1;
    if (st == HS_OK && shard && tc_ctas == 0) {
        prof_end(s);
        return fail(HS_ERR_UNSUPPORTED, "hs_attn_decode_sharded: only the tensor-core decode kernel exchanges shard results (quantised cache, 8 kv heads x 128 "
                                        "with 32 query heads or 2 x 256 with 16, cooperative launch available); use hs_attn_decode with o_shard / lse_shard, an "
                                        "all-gather and hs_attn_merge_partials_strided for this shape");
    }
    if (st == HS_OK && tc_ctas == 0) {
        st = decode_mma(v, qp, seq_lens, n_seqs, n_q_heads, scale_log2, o_part, lse_part, err, decode_max_ctas(), &n_ctas, &tile, after_write != 0, o_shard != nullptr,
                        append ? *append : AppendArgs{}, s);
    }
    prof_end(s);
    if (st != HS_OK) return st;
    if (int32_t e = check_launch("hs_attn_decode")) return e;
    if (merged) return HS_OK;  // the decode kernel merged its own partials behind a grid barrier
    // the merge is launched as the decode kernel's programmatic dependent: its launch and its slot arithmetic overlap with it
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(n_seqs) * static_cast<unsigned>(n_q_heads));
    cfg.blockDim = dim3(kMergeThreads);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t me = cudaLaunchKernelEx(&cfg, decode_merge_kernel, seq_lens, static_cast<int>(n_seqs), static_cast<int>(n_q_heads), D, n_ctas, tile,
                                              v.page_tokens * v.pages_per_seq, static_cast<const float *>(o_part), static_cast<const float *>(lse_part),
                                              reinterpret_cast<uint16_t *>(out), reinterpret_cast<const uint16_t *>(gate), o_shard, lse_shard);
    if (me != cudaSuccess) {
        cudaGetLastError();
        return fail(static_cast<int32_t>(me), "hs_attn_decode (merge): %s", cudaGetErrorString(me));
    }
    return check_launch("hs_attn_decode (merge)");
}

extern "C" {

int32_t hs_attn_merge_partials_strided(const float *o_parts, const float *lse_parts, int32_t n_parts, int64_t part_stride_o,
                                       int64_t part_stride_lse, int64_t n_rows, int32_t head_dim, void *out, const void *gate,
                                       hs_stream_t stream) {
    if (int32_t st = check_device()) return st;
    if (n_parts <= 0 || n_rows < 0 || head_dim <= 0 || head_dim > 1024) return fail(HS_ERR_ARG, "hs_attn_merge_partials: bad sizes");
    if (part_stride_o < n_rows * head_dim || part_stride_lse < n_rows) return fail(HS_ERR_ARG, "hs_attn_merge_partials: part strides overlap");
    if (n_rows == 0) return HS_OK;
    if (!o_parts || !lse_parts || !out) return fail(HS_ERR_ARG, "hs_attn_merge_partials: NULL pointer");
    if (n_rows > 0x7fffffffLL) return fail(HS_ERR_ARG, "hs_attn_merge_partials: too many rows");
    merge_parts_kernel<<<static_cast<unsigned>(n_rows), head_dim, 0, as_stream(stream)>>>(
        o_parts, lse_parts, n_parts, part_stride_o, part_stride_lse, head_dim, reinterpret_cast<uint16_t *>(out),
        reinterpret_cast<const uint16_t *>(gate));
    return check_launch("hs_attn_merge_partials");
}

int32_t hs_attn_merge_partials(const float *o_parts, const float *lse_parts, int32_t n_parts, int64_t n_rows, int32_t head_dim,
                               void *out, const void *gate, hs_stream_t stream) {
    return hs_attn_merge_partials_strided(o_parts, lse_parts, n_parts, n_rows * head_dim, n_rows, n_rows, head_dim, out, gate, stream);
}


int64_t hs_attn_decode_static_max_bytes(void) { return kStaticScratchBytes; }

int32_t hs_attn_decode_static(const void *q, const hs_kv_view *view, const int32_t *seq_lens, int32_t n_seqs, int32_t n_q_heads,
                              float softmax_scale, void *out, const void *gate, hs_stream_t stream) {
    if (int32_t st = check_device()) return st;
    if (int32_t st = validate_view(view)) return st;
    if (n_seqs < 0 || n_q_heads <= 0) return fail(HS_ERR_ARG, "hs_attn_decode_static: bad sizes");
    const int64_t need = hs_attn_decode_workspace_bytes(n_seqs, n_q_heads, view->head_dim);
    if (need < 0 || need > kStaticScratchBytes)
        return fail(HS_ERR_WORKSPACE,
                    "hs_attn_decode_static: n_seqs %d x n_q_heads %d x head_dim %d needs %lld bytes of scratch, the built-in array holds "
                    "%lld; use hs_attn_decode with a caller-provided workspace",
                    n_seqs, n_q_heads, view->head_dim, (long long)need, (long long)kStaticScratchBytes);
    void *scratch = nullptr;
    if (int32_t st = static_scratch_for_current_device(&scratch)) return st;
    // Nothing in the scratch has to start at zero: each launch writes every partial slot it later reads.
    return hs_attn_decode(q, view, seq_lens, n_seqs, n_q_heads, softmax_scale, out, gate, scratch, kStaticScratchBytes, nullptr,
                          nullptr, stream);
}


int32_t hs_attn_decode_append(const void *q, const void *k_new, const void *v_new, const hs_kv_view *view, const int32_t *dst_pos,
                              const int32_t *seq_lens, int32_t n_seqs, int32_t n_q_heads, float softmax_scale, const void *sin, const void *cos,
                              int32_t rotary_dim, int32_t n_positions, void *out, const void *gate, void *workspace, int64_t workspace_bytes,
                              hs_stream_t stream) {
    if (!k_new || !v_new) return fail(HS_ERR_ARG, "hs_attn_decode_append: NULL new token");
    if (dst_pos == nullptr) {
        // The new token goes to position seq_lens[s] - 1: the attention kernel can write it itself - u8 caches on decode_tc.cu, and bf16
        // on decode_mma.cu for one sequence in one page; otherwise the write kernel runs first, at those positions.  (bf16 rows of a
        // batch may look at one another's new tokens, several tokens of one sequence handed in as rows, and a table may list a page
        // twice: the host cannot see either, so everything that could is written before anything is attended.  One launch against
        // two: 1 x 4,096 tokens 34.3 against 36.0 us, 16 paged sequences 53.9 against 55.4 us.)
        if (!seq_lens && n_seqs > 0) return fail(HS_ERR_ARG, "hs_attn_decode_append: NULL lengths");  // (before anything is written)
        if (!aligned(k_new, 16) || !aligned(v_new, 16)) return fail(HS_ERR_ARG, "hs_attn_decode_append: inputs must be 16-byte aligned");
        if (sin != nullptr && (!cos || rotary_dim <= 0 || rotary_dim % 16 != 0 || (view && rotary_dim > view->head_dim) || n_positions <= 0))
            return fail(HS_ERR_UNSUPPORTED, "hs_attn_decode_append: rotary_dim must be a positive multiple of 16 <= head_dim");
        AppendArgs ap{reinterpret_cast<const uint16_t *>(k_new), reinterpret_cast<const uint16_t *>(v_new), reinterpret_cast<const uint16_t *>(sin),
                      reinterpret_cast<const uint16_t *>(cos), rotary_dim, n_positions};
        int appended = 0;
        if (view && (view->kind == HS_KV_INT8 || (view->kind == HS_KV_BF16 && n_seqs == 1 && view->pages_per_seq == 1))) {
            if (int32_t st = decode_impl(q, view, seq_lens, n_seqs, n_q_heads, softmax_scale, out, gate, workspace, workspace_bytes, nullptr, nullptr,
                                         nullptr, stream, 0, &ap, &appended))
                return st;
            if (appended || n_seqs == 0) return HS_OK;
        }
        if (int32_t st = kv_write_at_end(view, k_new, v_new, n_seqs, seq_lens, sin, cos, rotary_dim, n_positions, stream)) return st;
        return decode_impl(q, view, seq_lens, n_seqs, n_q_heads, softmax_scale, out, gate, workspace, workspace_bytes, nullptr, nullptr, nullptr, stream, 1);
    }
    if (int32_t st = hs_kv_quantize_write(view, k_new, v_new, n_seqs, 1, dst_pos, sin, cos, rotary_dim, n_positions, stream)) return st;
    return decode_impl(q, view, seq_lens, n_seqs, n_q_heads, softmax_scale, out, gate, workspace, workspace_bytes, nullptr, nullptr, nullptr, stream, 1);
}

int32_t hs_attn_decode_step(const hs_kv_view *view, const void *host_in, void *dev_in, const int32_t *dst_pos, const int32_t *seq_lens,
                            int32_t n_seqs, int32_t n_q_heads, float softmax_scale, const void *sin, const void *cos, int32_t rotary_dim,
                            int32_t n_positions, void *dev_out, void *host_out, void *workspace, int64_t workspace_bytes, int32_t flags,
                            hs_stream_t stream) {
    if (int32_t st = check_device()) return st;
    if (int32_t st = validate_view(view)) return st;
    if (n_seqs < 0 || n_q_heads <= 0) return fail(HS_ERR_ARG, "hs_attn_decode_step: bad sizes");
    if (n_seqs == 0) return HS_OK;
    if (!host_in || !dev_in || !dev_out || !host_out || !seq_lens)
        return fail(HS_ERR_ARG, "hs_attn_decode_step: NULL pointer");
    if (!aligned(dev_in, 16)) return fail(HS_ERR_ARG, "hs_attn_decode_step: dev_in must be 16-byte aligned");
    const int64_t D = view->head_dim;
    const int64_t q_elems = static_cast<int64_t>(n_seqs) * n_q_heads * D, kv_elems = static_cast<int64_t>(n_seqs) * view->n_kv_heads * D;
    if ((q_elems * 2) % 16 != 0 || (kv_elems * 2) % 16 != 0) return fail(HS_ERR_ARG, "hs_attn_decode_step: q and k/v parts must be multiples of 16 bytes");
    cudaStream_t s = as_stream(stream);
    cudaError_t e = cudaMemcpyAsync(dev_in, host_in, static_cast<size_t>(q_elems + 2 * kv_elems) * 2, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return fail(static_cast<int32_t>(e), "hs_attn_decode_step: %s", cudaGetErrorString(e));
    uint16_t *qd = reinterpret_cast<uint16_t *>(dev_in), *kd = qd + q_elems, *vd = kd + kv_elems;
    // cache update + attention: where the attention kernel writes the tokens itself one launch less (see above), else the write kernel
    // and the attention kernel as its programmatic dependent; q came with the copy before both
    if (int32_t st = hs_attn_decode_append(qd, kd, vd, view, dst_pos, seq_lens, n_seqs, n_q_heads, softmax_scale, sin, cos, rotary_dim, n_positions, dev_out,
                                           nullptr, workspace, workspace_bytes, stream))
        return st;
    // (letting the kernel store into mapped host memory instead of this copy was measured: 9 us slower per step; copy kernels over
    // mapped pinned memory in place of the two cudaMemcpyAsync calls: 3 us faster of 102, not worth a second mechanism; the host
    // polling a word that the stream writes behind the copy, instead of cudaStreamSynchronize: 106 against 104 us)
    e = cudaMemcpyAsync(host_out, dev_out, static_cast<size_t>(q_elems) * 2, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && (flags & HS_STEP_SYNC)) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(static_cast<int32_t>(e), "hs_attn_decode_step: %s", cudaGetErrorString(e));
    return HS_OK;
}

}  // extern "C"
