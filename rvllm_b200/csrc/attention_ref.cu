// Plain paged attention: the reference kernel that every faster attention kernel is checked
// against, and the kernel of the float32 path.  One CTA per (token, query head); its eight warps take
// blocks of neighbouring keys in turn through the block table, each with an online softmax in float,
// and their results are merged in warp order.  Bound by the latency of a warp's chain (table, keys, sums
// over lanes, values): a block's loads are in flight together and its softmax is one step.  One warp per
// (token, head) and one key at a time, the form before, took 303 us a layer for three tokens of 28 heads
// at 200 keys; this takes 11.5.  The cut of the keys depends on a token's position and window alone.
//
// Rule (v3/kernels/paged_attention_sm89.cu:241-369 of the reference): the q_len tokens a
// sequence brings to a step are the tail of its ctx_len cached tokens.  The token with
// in-step index i sits at position p = ctx_len - q_len + i and sees keys [0, p]; with a
// window of W keys it sees (p - W, p].  kv_head = head * nkv / nh.  A decoded token is the
// case q_len = 1.  ctx_len <= 0 marks a padded row: zeros are written, no table is read.
//
// Options for mixers that want them: `softcap` > 0 replaces a scaled score s by
// softcap * tanh(s / softcap); `sinks` (one float per query head) adds exp(sink_h) to the softmax
// denominator - a key without a value, neither scaled nor capped; `gate` (float [tokens, heads])
// multiplies each head's output; `dist` (float [nkv, dist_n, nh / nkv]) is added to a (scaled, capped) score by the distance
// between query and key, a distance beyond the last reading the last.
//
// Cache layer layout: [num_pages, planes, nkv, page_size, hd].  planes = 2: keys in plane 0, values in plane 1.
// planes = 1: one row per token and kv head; the key is the whole row and the value its leading `vd` elements
// (a latent that keys and values are projections of).  The output row of a head has `vd` elements (hd with two planes).
#include "common.cuh"

#define REF_WARPS 8

// DPL: elements of a row that one lane holds (row <= 32 * DPL); KEYS: keys of a block
template <typename T, int DPL, int KEYS>
__global__ void __launch_bounds__(REF_WARPS * 32)
paged_attention_ref_kernel(const T* __restrict__ q, const T* __restrict__ cache,
                           const int* __restrict__ block_tables, const int* __restrict__ cu_seqlens,
                           const int* __restrict__ ctx_lens, const int* __restrict__ token_seq,
                           T* __restrict__ out, int n_tokens, int nh, int nkv, int hd,
                           int page_size, int max_blocks, float scale, int window,
                           float softcap, const float* __restrict__ sinks, const float* __restrict__ gate,
                           int planes, int vd, const float* __restrict__ dist, int dist_n) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    __shared__ float sh_acc[REF_WARPS][32 * DPL];
    __shared__ float sh_m[REF_WARPS], sh_l[REF_WARPS];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int t = blockIdx.x / nh, h = blockIdx.x % nh;
    const int seq = token_seq[t];
    T* o = out + ((size_t)t * nh + h) * vd;
    const int ctx = seq >= 0 ? ctx_lens[seq] : 0;
    if (ctx <= 0) {
        for (int d = threadIdx.x; d < vd; d += blockDim.x) o[d] = rv_from_float<T>(0.f);
        return;
    }
    const int q_start = cu_seqlens[seq];
    const int q_len = cu_seqlens[seq + 1] - q_start;
    const int pos = ctx - q_len + (t - q_start);
    const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    const int kvh = (int)(((long long)h * nkv) / nh);

    float qv[DPL], acc[DPL];
    const T* qp = q + ((size_t)t * nh + h) * hd;
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
        const int d = lane + 32 * i;
        qv[i] = d < hd ? rv_to_float(qp[d]) * scale : 0.f;
        acc[i] = 0.f;
    }
    float m = -INFINITY, l = 0.f;
    const int* table = block_tables + (size_t)seq * max_blocks;
    const int G = nh / nkv;
    const float* bias = dist ? dist + (size_t)kvh * dist_n * G + (h - kvh * G) : nullptr;
    const size_t page_stride = (size_t)planes * nkv * page_size * hd;
    const size_t v_off = planes == 2 ? (size_t)nkv * page_size * hd : 0;
    for (int j0 = lo + warp * KEYS; j0 <= pos; j0 += REF_WARPS * KEYS) {
        const T* kp[KEYS];
        float kv[KEYS][DPL], s[KEYS];
#pragma unroll
        for (int n = 0; n < KEYS; ++n) {                    // (a key beyond the last repeats it and gets no weight)
            const int j = min(j0 + n, pos);
            kp[n] = cache + (size_t)table[j / page_size] * page_stride + ((size_t)kvh * page_size + (j % page_size)) * hd;
        }
#pragma unroll
        for (int n = 0; n < KEYS; ++n)
#pragma unroll
            for (int i = 0; i < DPL; ++i) { const int d = lane + 32 * i; kv[n][i] = d < hd ? rv_to_float(kp[n][d]) : 0.f; }
#pragma unroll
        for (int n = 0; n < KEYS; ++n) {
            s[n] = 0.f;
#pragma unroll
            for (int i = 0; i < DPL; ++i) s[n] = fmaf(qv[i], kv[n][i], s[n]);
        }
        if (planes == 2) {                                  // the values are on their way while the sums over the lanes run
#pragma unroll
            for (int n = 0; n < KEYS; ++n)
#pragma unroll
                for (int i = 0; i < DPL; ++i) { const int d = lane + 32 * i; kv[n][i] = d < vd ? rv_to_float(kp[n][v_off + d]) : 0.f; }
        }
        float m_new = m;
#pragma unroll
        for (int n = 0; n < KEYS; ++n) {
            s[n] = rv_warp_sum(s[n]);
            if (softcap > 0.f) s[n] = softcap * tanhf(s[n] / softcap);
            if (bias) s[n] += bias[(size_t)max(0, min(pos - j0 - n, dist_n - 1)) * G];
            if (j0 + n > pos) s[n] = -INFINITY;
            m_new = fmaxf(m_new, s[n]);
        }
        const float corr = expf(m - m_new);                 // exp(-inf) = 0 at the first block
        l *= corr;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[i] *= corr;
#pragma unroll
        for (int n = 0; n < KEYS; ++n) {
            if (j0 + n > pos) continue;                     // (also keeps a value of infinity or NaN past the end out)
            const float p = expf(s[n] - m_new);
            l += p;
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[i] = fmaf(p, kv[n][i], acc[i]);
        }
        m = m_new;
    }
    if (lane == 0) { sh_m[warp] = m; sh_l[warp] = l; }
#pragma unroll
    for (int i = 0; i < DPL; ++i) sh_acc[warp][lane + 32 * i] = acc[i];
    __syncthreads();
    float top = sinks ? sinks[h] : -INFINITY;
    for (int w = 0; w < REF_WARPS; ++w)
        if (lo + w * KEYS <= pos) top = fmaxf(top, sh_m[w]);
    float sum = 0.f, corr[REF_WARPS];
#pragma unroll
    for (int w = 0; w < REF_WARPS; ++w) {
        corr[w] = lo + w * KEYS <= pos ? expf(sh_m[w] - top) : 0.f;      // a warp without keys adds nothing
        sum += sh_l[w] * corr[w];
    }
    if (sinks) sum += expf(sinks[h] - top);
    float inv = sum > 0.f ? 1.0f / sum : 0.f;
    if (gate) inv *= gate[(size_t)t * nh + h];
    for (int d = threadIdx.x; d < vd; d += blockDim.x) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < REF_WARPS; ++w) v = fmaf(sh_acc[w][d], corr[w], v);
        o[d] = rv_from_float<T>(v * inv);
    }
}

template <int DPL, int KEYS>
static int launch_ref(const void* q, const void* cache, const int* block_tables, const int* cu_seqlens, const int* ctx_lens,
                      const int* token_seq, void* out, int n_tokens, int nh, int nkv, int hd, int page_size, int max_blocks,
                      float scale, int window, float softcap, const float* sinks, const float* gate, int planes, int vd,
                      int dtype, const float* dist, int dist_n, cudaStream_t stream) {
    if ((long long)n_tokens * nh > 0x7fffffffLL) return RV_ERR_BAD_SIZE;
    const dim3 grid((unsigned)n_tokens * (unsigned)nh);
    if (dtype == RV_DTYPE_F32)
        RV_LAUNCH_ST = rv_launch(paged_attention_ref_kernel<float, DPL, KEYS>, dim3(grid), dim3(REF_WARPS * 32), 0, stream,
            (const float*)q, (const float*)cache, block_tables, cu_seqlens, ctx_lens, token_seq, (float*)out,
            n_tokens, nh, nkv, hd, page_size, max_blocks, scale, window, softcap, sinks, gate, planes, vd, dist, dist_n);
    else if (dtype == RV_DTYPE_BF16)
        RV_LAUNCH_ST = rv_launch(paged_attention_ref_kernel<__nv_bfloat16, DPL, KEYS>, dim3(grid), dim3(REF_WARPS * 32), 0, stream,
            (const __nv_bfloat16*)q, (const __nv_bfloat16*)cache, block_tables, cu_seqlens, ctx_lens, token_seq,
            (__nv_bfloat16*)out, n_tokens, nh, nkv, hd, page_size, max_blocks, scale, window, softcap, sinks, gate, planes, vd, dist, dist_n);
    else
        return RV_ERR_BAD_DTYPE;
    return rv_launch_status();
}

// planes 2: keys and values in their planes, output rows of hd; planes 1: the value is the leading vd elements of the key row.
RV_EXPORT int rv_paged_attention_ref_ex(const void* q, const void* cache, const int* block_tables,
                                        const int* cu_seqlens, const int* ctx_lens, const int* token_seq,
                                        void* out, int n_tokens, int nh, int nkv, int hd, int page_size,
                                        int max_blocks, float scale, int window, float softcap, const float* sinks,
                                        const float* gate, int planes, int vd, int dtype, const float* dist, int dist_n,
                                        cudaStream_t stream) {
    if (dist && (dist_n <= 0 || nkv <= 0 || nh % nkv)) return RV_ERR_BAD_SIZE;
    if (n_tokens < 0 || nh <= 0 || nkv <= 0 || hd <= 0 || page_size <= 0 || max_blocks <= 0) return RV_ERR_BAD_SIZE;
    if ((planes != 1 && planes != 2) || vd <= 0 || vd > hd || (planes == 2 && vd != hd)) return RV_ERR_BAD_SIZE;
    if (hd > 32 * 32) return RV_ERR_UNSUPPORTED;
    if (n_tokens == 0) return RV_OK;
    if (hd <= 32 * 4)
        return launch_ref<4, 8>(q, cache, block_tables, cu_seqlens, ctx_lens, token_seq, out, n_tokens, nh, nkv, hd, page_size,
                                max_blocks, scale, window, softcap, sinks, gate, planes, vd, dtype, dist, dist_n, stream);
    if (hd <= 32 * 8)
        return launch_ref<8, 4>(q, cache, block_tables, cu_seqlens, ctx_lens, token_seq, out, n_tokens, nh, nkv, hd, page_size,
                             max_blocks, scale, window, softcap, sinks, gate, planes, vd, dtype, dist, dist_n, stream);
    return launch_ref<32, 1>(q, cache, block_tables, cu_seqlens, ctx_lens, token_seq, out, n_tokens, nh, nkv, hd, page_size,
                          max_blocks, scale, window, softcap, sinks, gate, planes, vd, dtype, dist, dist_n, stream);
}

RV_EXPORT int rv_paged_attention_ref(const void* q, const void* cache, const int* block_tables,
                                     const int* cu_seqlens, const int* ctx_lens, const int* token_seq,
                                     void* out, int n_tokens, int nh, int nkv, int hd, int page_size,
                                     int max_blocks, float scale, int window, float softcap, const float* sinks,
                                     const float* gate, int dtype, cudaStream_t stream) {
    if (hd > 32 * 8) return RV_ERR_UNSUPPORTED;
    return rv_paged_attention_ref_ex(q, cache, block_tables, cu_seqlens, ctx_lens, token_seq, out, n_tokens, nh, nkv, hd,
                                     page_size, max_blocks, scale, window, softcap, sinks, gate, 2, hd, dtype, nullptr, 0, stream);
}
