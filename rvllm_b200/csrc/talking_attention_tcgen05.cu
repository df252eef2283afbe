// Attention whose softmax weights are mixed across the heads, for prompt portions in bfloat16, with the mixing BEHIND the sum over
// the keys (same cache layout, arguments and rule as talking_attention.cu):
//
//     o_h = sum_j (sum_g talk[h, g] p_g(j)) v_kv(h)(j) = sum_g talk[h, g] U[g][kv(h)],     U[g][c] = sum_j p_g(j) v_c(j)
//
// so the walk over the keys is a flash attention with running maxima whose value is the rows of ALL key/value heads, and nothing
// needs the heads of a token together before U is there: the tensor cores do nkv times the second product and the walk has no
// mixing, no second pass over the keys and no float32 work beyond a softmax.
//
//   talking_wide_kernel   a CTA owns 128 rows ((token, head) pairs of one key/value head) and the values of up to
//                         384 / V_DIM key/value heads: S = Q K^T and O += P V by tcgen05.mma as in attention_tcgen05.cu (S double
//                         buffered, P back into tensor memory over its S, O [128 x heads x V_DIM] float in the other
//                         384 columns).  U is O over the row's sum of weights, float32.
//   talking_mix_kernel    out[t, h] = sum_g talk[h, g] U[t][kv(h)][g], float32 sums in the order of g, rounded once.
//
// A weight goes into the products as TWO bfloat16 numbers, its rounding and what the rounding left (16 bits and more of the float32
// weight).  The mixing may take heads that attend alike from one another: then the weights cancel and what they were rounded by does
// not.  Error against float64 (2-norms; 16 heads on 4, 32 on 8, 8 on 8; contexts of 150 to 4,000), mixing by the identity, at random,
// and by differences of heads whose scores are 0.3 to 0.005 of themselves apart: 1.6e-3 to 1.8e-3, where the rounding of the result
// alone is 1.6e-3 and the kernel that mixes inside the walk (talking_attention_mma.cu: mixed weights rounded once) has 2.3e-3 to
// 2.4e-3.  With one bfloat16 number a weight it was 2.0e-3 to 2.4e-3 for the first two, 6e-3 to 3.5e-1 for the differences.
//
// Against the kernel that mixes inside the walk (heads of 128, L2 flushed): 16 heads on 4, 2,048 tokens 475 -> 160 us,
// 80 tokens 31 -> 21, 100 tokens behind 3,990 keys 960 -> 110 to 160; 32 heads on 8, 2,048 tokens 975 -> 490, 100 behind 3,990 1,329 -> 185.  (One
// number a weight and no look at the values: 118, 19, 97; 392, 114.  The softmax warps, one a scheduler, bind the walk: forming the rests and
// storing them takes 25 us of 2,048 tokens of 16 heads, the second products 12, the look at the values 5.)
//
// The distance bias r1 ln(1 + r2 d) takes a logarithm per (head, distance), not per score: a warp's 32 rows are few tokens, so
// a tile of 64 keys meets only 63 + tokens distances, whose biases the warp forms in shared memory while the tile's Q K^T runs.
#include "common.cuh"
#include "tcgen05_attention.cuh"

#define ROWS 128
#define KV_TILE 64
#define SOFTMAX_WARPS 4
#define LOADER_WARP SOFTMAX_WARPS               // Q and the keys (and the tensor memory's allocation)
#define VLOADER_WARP (SOFTMAX_WARPS + 1)       // the values
#define QK_WARP (SOFTMAX_WARPS + 2)            // issues S = Q K^T
#define PV_WARP (SOFTMAX_WARPS + 3)            // issues O += P V
#define NUM_THREADS (32 * (SOFTMAX_WARPS + 4))
#define TMEM_COLS 512
#define S_COL 0                                // two S buffers of 64 columns; P (two bf16 numbers a weight) reuses them
#define O_COL 128
#define O_COLS (TMEM_COLS - O_COL)
#define MAX_GROUP 16                           // heads on one key/value head
#define BIAS_FLOATS ((KV_TILE - 1 + 2) * MAX_GROUP)      // a warp's biases of a tile: (63 + 32 / G) distances x G heads
#define NK 3
#define NV 2
#define B_Q 0
#define B_K 1                                  // keys of a stage have landed [NK]
#define B_KFREE (B_K + NK)                     // the S product that read a stage has finished [NK]
#define B_V (B_KFREE + NK)                     // values of a stage have landed [NV]
#define B_VFREE (B_V + NV)                     // the P V products that read a stage have finished [NV]
#define B_SFULL (B_VFREE + NV)                 // [2] each from here on
#define B_OFULL (B_SFULL + 2)
#define B_PFULL (B_OFULL + 2)
#define NUM_BARS (B_PFULL + 2)
static_assert(NUM_BARS <= 30, "the barriers, the tensor-memory address and the abort flag share 256 bytes");
#define RESCALE_LOG2 8.0f

struct WideParams {
    const int* block_tables;
    const int* cu_seqlens;
    const int* ctx_lens;
    float* u;                      // [tokens tok_lo .. tok_hi][nkv][nh][V_DIM]
    const __nv_bfloat16* values;   // of page 0; a page has page_elems elements
    size_t page_elems;
    int* status;
    int nh, nkv, page_shift, page_size, max_blocks, chunk;
    int per_block, blocks;         // value heads of a CTA, and how many such blocks there are
    int tok_lo, tok_hi;            // the step's tokens whose rows are stored
    float scale_log2e;
    const float* r1;               // or null
    const float* r2;
};

template <int HD, int VD>
struct WideSizes {
    static constexpr int HALVES = HD / 64, V_HALVES = VD / 64, MAX_V = O_COLS / VD;
    static constexpr int Q_BYTES = ROWS * HD * 2, K_BYTES = KV_TILE * HD * 2, V_BYTES = KV_TILE * MAX_V * VD * 2;
    static constexpr int SMEM = Q_BYTES + NK * K_BYTES + NV * V_BYTES + 256 + SOFTMAX_WARPS * BIAS_FLOATS * 4;
};

template <int W> struct WideVec { using type = float4; };
template <> struct WideVec<2> { using type = float2; };

__device__ __forceinline__ float fast_log2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// G: heads on one key/value head (a constant, so that the reads of the biases have constant offsets: 64 registers of addresses less; 2,048
// tokens, with one number a weight, 134 -> 118 and 406 -> 392 us)
template <int HD, int VD, int G>
__global__ void __launch_bounds__(NUM_THREADS, 1)
talking_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const WideParams p) {
    using Z = WideSizes<HD, VD>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* q_s = smem_raw;                           // [HALVES][128 rows x 128 B]
    unsigned char* k_s = q_s + Z::Q_BYTES;                   // [NK stages][HALVES][KV_TILE keys x 128 B]
    unsigned char* v_s = k_s + NK * Z::K_BYTES;              // [NV stages][value heads][V_HALVES][KV_TILE keys x 128 B]
    uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + NV * Z::V_BYTES);
    uint32_t& tmem_base_slot = *reinterpret_cast<uint32_t*>(bars + 30);
    volatile int& abort_flag = *reinterpret_cast<volatile int*>(bars + 31);
    volatile int& left_out = *(reinterpret_cast<volatile int*>(bars + 31) + 1);     // 1: values that are not finite stayed out of a product
    float* bias_s = reinterpret_cast<float*>(bars + 32);     // [SOFTMAX_WARPS][BIAS_FLOATS]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) { tma_prefetch_descriptor(&map_q); tma_prefetch_descriptor(&map_k); tma_prefetch_descriptor(&map_v); }
    const uint32_t bar_q = smem_u32(&bars[B_Q]), bar_k0 = smem_u32(&bars[B_K]);
    const uint32_t bar_kfree0 = smem_u32(&bars[B_KFREE]), bar_v0 = smem_u32(&bars[B_V]);
    const uint32_t bar_vfree0 = smem_u32(&bars[B_VFREE]);
    const uint32_t bar_s_full0 = smem_u32(&bars[B_SFULL]);
    const uint32_t bar_o_full0 = smem_u32(&bars[B_OFULL]), bar_p_full0 = smem_u32(&bars[B_PFULL]);

    // the row tile is the slowest index, counted down: the tiles with the most keys start first (attention_tcgen05.cu)
    const int kvh = blockIdx.x / p.blocks, c0 = (blockIdx.x % p.blocks) * p.per_block, nv = min(p.per_block, p.nkv - c0);
    const int seq = blockIdx.y, tile_m = gridDim.z - 1 - blockIdx.z;
    rv_pdl_wait();
    const int ctx = p.ctx_lens[seq];
    const int q_start = p.cu_seqlens[seq];
    const int q_len = p.cu_seqlens[seq + 1] - q_start;
    constexpr int tile_tokens = ROWS / G;
    const int tok0 = tile_m * tile_tokens, n_tok = min(tile_tokens, q_len - tok0);      // this CTA's tokens of the portion
    if (n_tok <= 0 || q_start + tok0 >= p.tok_hi || q_start + tok0 + n_tok <= p.tok_lo) return;
    if (ctx <= 0) {                                          // padding: its result is zero
        for (int i = tid; i < n_tok * nv * G * VD; i += NUM_THREADS) {
            const int e = i % VD, hh = (i / VD) % G, b = (i / (VD * G)) % nv, t = q_start + tok0 + i / (VD * G * nv);
            if (t >= p.tok_lo && t < p.tok_hi) p.u[(((size_t)(t - p.tok_lo) * p.nkv + c0 + b) * p.nh + kvh * G + hh) * VD + e] = 0.f;
        }
        return;
    }
    const int pos_first = ctx - q_len + tok0, pos_last = pos_first + n_tok - 1;
    const int key_lo = p.chunk > 0 ? (pos_first / p.chunk) * p.chunk : 0;
    const int key_hi = pos_last + 1;
    const int t_begin = key_lo / KV_TILE, t_end = (key_hi + KV_TILE - 1) / KV_TILE;
    const int n_it = t_end - t_begin;
    const int* table = p.block_tables + (size_t)seq * p.max_blocks;
    // Tiles with a key that some row of the CTA does not see: those of the portion's own keys and, where it crosses a chunk's border, those
    // of the chunk before.  A hidden key's weight is zero, and zero times a value that is not finite is no number: such values of
    // these tiles stay out of the products, and the rows that do see them get them added behind the walk.  (Looking for them, by the warp
    // that issues the products: 2,048 tokens of 16 heads on 4 155 -> 160 us, of 32 on 8 475 -> 500.)
    const int lo_last = p.chunk > 0 ? (pos_last / p.chunk) * p.chunk : 0;
    auto partly_seen = [&](int t) { return t * KV_TILE + KV_TILE - 1 > pos_first || t * KV_TILE < lo_last; };

    if (tid == 0) {
        abort_flag = 0;
        left_out = 0;
        mbar_init(bar_q, 1);
        for (int i = 0; i < NK; ++i) { mbar_init(bar_k0 + 8 * i, 1); mbar_init(bar_kfree0 + 8 * i, 1); }
        for (int i = 0; i < NV; ++i) { mbar_init(bar_v0 + 8 * i, 1); mbar_init(bar_vfree0 + 8 * i, 1); }
        mbar_init(bar_s_full0, 1); mbar_init(bar_s_full0 + 8, 1);
        mbar_init(bar_p_full0, SOFTMAX_WARPS); mbar_init(bar_p_full0 + 8, SOFTMAX_WARPS);
        mbar_init(bar_o_full0, 1); mbar_init(bar_o_full0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == LOADER_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    // value tiles start as zeros: a page that is not loaded (beyond the context, or given back) must not meet a weight of zero with a NaN
    for (int i = tid; i < NV * Z::V_BYTES / 16; i += NUM_THREADS) reinterpret_cast<uint4*>(v_s)[i] = make_uint4(0, 0, 0, 0);
    fence_async_smem();
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    rv_pdl_launch_dependents();                              // only now that this CTA holds its tensor memory (attention_tcgen05.cu)

    const int box_keys = p.page_size < KV_TILE ? p.page_size : KV_TILE;     // keys one TMA box brings
    const int boxes = KV_TILE / box_keys;
    int tiles_issued = 0;             // by this warp, if it is a loader
    if (warp == LOADER_WARP || warp == VLOADER_WARP) {
        // ------------------------------------------------------------ loader warps: one for keys, one for values
        // Lane i looks up the page of box i of a tile (a tile ahead); the lanes share the (head, box) pairs of a tile.
        const bool keys = warp == LOADER_WARP;
        const int stages = keys ? NK : NV, heads = keys ? 1 : nv, slabs = keys ? Z::HALVES : Z::V_HALVES;
        const uint32_t stage_bytes = keys ? Z::K_BYTES : Z::V_BYTES;
        const uint32_t bar_full0 = keys ? bar_k0 : bar_v0, bar_free0 = keys ? bar_kfree0 : bar_vfree0;
        const uint32_t ring = smem_u32(keys ? k_s : v_s);
        const CUtensorMap* map = keys ? &map_k : &map_v;
        auto wait_all = [&](uint32_t bar, uint32_t parity, int code) -> bool {
            int ok_l = 1;
            if (lane == 0) ok_l = mbar_wait(bar, parity, &abort_flag, code) ? 1 : 0;
            return __shfl_sync(0xffffffffu, ok_l, 0) != 0;
        };
        auto lookup = [&](int t) -> int {               // the page of box `lane` of tile t, or -1
            const int key = t * KV_TILE + lane * box_keys;
            return (lane < boxes && key < key_hi && key + box_keys > key_lo) ? __ldg(table + (key >> p.page_shift)) : -1;
        };
        auto issue = [&](int t, int stage, int page) {
            const uint32_t bar = bar_full0 + 8 * stage;
            const unsigned mask = __ballot_sync(0xffffffffu, page >= 0);
            if (lane == 0) mbar_expect_tx(bar, (uint32_t)__popc(mask) * (uint32_t)(heads * slabs) * (uint32_t)box_keys * 128u);
            __syncwarp();
            for (int i0 = 0; i0 < boxes * heads; i0 += 32) {
                const int i = i0 + lane, box = i % boxes, b = i / boxes;
                const int pg = __shfl_sync(0xffffffffu, page, box);
                if (b < heads && pg >= 0) {
                    const int key = t * KV_TILE + box * box_keys;
                    const int row = (keys ? kvh : c0 + b) * p.page_size + (key & (p.page_size - 1));
                    const uint32_t dst = ring + (uint32_t)stage * stage_bytes + (uint32_t)(b * slabs) * (KV_TILE * 128) + (uint32_t)box * box_keys * 128u;
                    for (int h = 0; h < slabs; ++h) tma_load_3d(dst + (uint32_t)h * (KV_TILE * 128), map, h * 64, row, pg, bar);
                }
            }
            __syncwarp();
        };
        if (keys && lane == 0) {                        // Q: one box of [64 elements, G heads, whole tokens] per slab
            mbar_expect_tx(bar_q, (uint32_t)Z::Q_BYTES);                    // (whole boxes count, also where they reach beyond the step)
#pragma unroll
            for (int h = 0; h < Z::HALVES; ++h)
                tma_load_3d(smem_u32(q_s) + h * (ROWS * 128), &map_q, h * 64, kvh * G, q_start + tok0, bar_q);
        }
        for (int i = 0; i < stages && i < n_it; ++i, ++tiles_issued) issue(t_begin + i, i, lookup(t_begin + i));
        int page = stages < n_it ? lookup(t_begin + stages) : -1;
        int stage = 0;
        uint32_t phase = 0;
        for (int e = 0; e + stages < n_it; ++e) {
            const int next = e + 1 + stages < n_it ? lookup(t_begin + e + 1 + stages) : -1;
            if (!wait_all(bar_free0 + 8 * stage, phase, keys ? 3 : 4)) break;
            issue(t_begin + e + stages, stage, page);
            ++tiles_issued;
            page = next;
            if (++stage == stages) { stage = 0; phase ^= 1; }
        }
    } else if (warp == QK_WARP) {
        // ------------------------------------------------------------ S = Q K^T into buffer i mod 2, over P(i - 2)
        if (lane == 0) {
            const uint32_t idesc_s = umma_idesc_bf16(ROWS, KV_TILE);
            bool ok = mbar_wait(bar_q, 0, &abort_flag, 1);
            int k_stage = 0;
            uint32_t k_phase = 0;
            for (int i = 0; i < n_it && ok; ++i) {
                const int buf = i & 1;
                if (!(ok = mbar_wait(bar_k0 + 8 * k_stage, k_phase, &abort_flag, 5))) break;
                if (i >= 2 && !(ok = mbar_wait(bar_o_full0 + 8 * buf, ((i - 2) >> 1) & 1, &abort_flag, 6))) break;
                tcgen05_fence_after();
#pragma unroll
                for (int h = 0; h < Z::HALVES; ++h) {
                    const uint64_t dq = umma_desc(smem_u32(q_s) + h * (ROWS * 128));
                    const uint64_t dk = umma_desc(smem_u32(k_s) + k_stage * Z::K_BYTES + h * (KV_TILE * 128));
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        tcgen05_mma_bf16(tmem_base + S_COL + buf * KV_TILE, dq + (uint64_t)(2 * j), dk + (uint64_t)(2 * j), idesc_s, (h | j) != 0);
                }
                tcgen05_commit(bar_s_full0 + 8 * buf);
                tcgen05_commit(bar_kfree0 + 8 * k_stage);
                if (++k_stage == NK) { k_stage = 0; k_phase ^= 1; }
            }
        }
    } else if (warp == PV_WARP) {
        // ------------------------------------------------------------ O += P V, head by head of the CTA's values
        const uint32_t idesc_o = umma_idesc_bf16(ROWS, VD) | (1u << 16);                 // B is MN-major
        const int valid = key_hi - (t_end - 1) * KV_TILE;        // keys of the last tile
        bool ok = true;
        auto products = [&](int it) {                            // one thread
            const int b = it & 1, v_stage = it % NV;
            if (!(ok = mbar_wait(bar_p_full0 + 8 * b, (it >> 1) & 1, &abort_flag, 8))) return;
            tcgen05_fence_after();
            const uint32_t tp = tmem_base + S_COL + b * KV_TILE;         // P(it) over S buffer b: of 32 keys 16 columns of roundings and 16 of rests
            for (int c = 0; c < nv; ++c) {
                const uint64_t dv = umma_desc_mn(smem_u32(v_s) + v_stage * Z::V_BYTES + c * (Z::V_HALVES * KV_TILE * 128), KV_TILE * 128);
#pragma unroll
                for (int j = 0; j < 8; ++j) {            // 16 keys per MMA: 8 columns along P's rows, 2048 bytes down V
                    const int keys = 2 * (j >> 2) + (j & 1);
                    tcgen05_mma_bf16_ts(tmem_base + O_COL + c * VD, tp + 8 * j, dv + (uint64_t)(128 * keys), idesc_o, (it | j) != 0);
                }
            }
            tcgen05_commit(bar_vfree0 + 8 * v_stage);
            tcgen05_commit(bar_o_full0 + 8 * b);
        };
        for (int it = 0; it < n_it; ++it) {
            if (!partly_seen(t_begin + it)) {
                if (lane == 0 && ok && (ok = mbar_wait(bar_v0 + 8 * (it % NV), (it / NV) & 1, &abort_flag, 7))) products(it);
                continue;
            }
            __syncwarp();
            if (ok) ok = mbar_wait(bar_v0 + 8 * (it % NV), (it / NV) & 1, &abort_flag, 7);
            if (__all_sync(0xffffffffu, ok)) {                   // (while the softmax warps form this tile's weights)
                uint4* tile = reinterpret_cast<uint4*>(v_s + (it % NV) * Z::V_BYTES);
                if (it + 1 == n_it) {
                    // rows of the last tile's pages beyond the portion's last key may hold anything: zeros in their place
                    const int words = (KV_TILE - valid) * 8;     // of 16 bytes, per slab
                    for (int i = lane; i < nv * Z::V_HALVES * words; i += 32)
                        tile[(i / words) * (KV_TILE * 8) + valid * 8 + i % words] = make_uint4(0, 0, 0, 0);
                    __syncwarp();
                }
                constexpr int head_words = Z::V_HALVES * KV_TILE * 8;
                const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
                __nv_bfloat162 sum[4] = {zero, zero, zero, zero};        // of zero times every value
#pragma unroll 8
                for (int i = lane; i < nv * head_words; i += 32) {
                    const uint4 w = tile[i];
                    sum[0] = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w.x), zero, sum[0]);
                    sum[1] = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w.y), zero, sum[1]);
                    sum[2] = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w.z), zero, sum[2]);
                    sum[3] = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w.w), zero, sum[3]);
                }
                const float2 all = __bfloat1622float2(__hadd2(__hadd2(sum[0], sum[1]), __hadd2(sum[2], sum[3])));
                if (__any_sync(0xffffffffu, !(all.x + all.y == 0.f))) {
                    auto finite = [](uint32_t x) { return x & ~(((((x & 0x7f807f80u) + 0x00800080u) >> 15) & 0x00010001u) * 0xffffu); };
                    for (int i = lane; i < nv * head_words; i += 32) {
                        const uint4 w = tile[i];
                        tile[i] = make_uint4(finite(w.x), finite(w.y), finite(w.z), finite(w.w));
                    }
                    if (lane == 0) left_out = 1;
                }
                fence_async_smem();
                __syncwarp();
            }
            if (lane == 0 && ok) products(it);
        }
    } else {
        // ------------------------------------------------------------ softmax warps: one thread per row
        const int row_l = warp * 32 + lane;                  // row of the tile = TMEM lane: (token, head in group)
        const int tok_i = row_l / G;
        const bool in_range = tok_i < n_tok;
        const int head = kvh * G + row_l - tok_i * G;
        const int pos = in_range ? pos_first + tok_i : -1;
        const int lo = p.chunk > 0 && in_range ? (pos / p.chunk) * p.chunk : 0;
        const uint32_t t_lane = tmem_base + ((uint32_t)(warp * 32) << 16);
        // the warp's tokens and their biases of a tile: entry (distance - nearest) * G + head; the rows of a token read neighbours
        const int w_tok0 = warp * 32 / G;
        constexpr int w_toks = 32 / G, b_step = 32 / G;
        const int w_pos0 = pos_first + w_tok0;               // (also of rows beyond the portion: their scores are masked)
        float* bias = bias_s + warp * BIAS_FLOATS;
        const bool biased = p.r1 != nullptr;
        // distances of a tile at key0: w_pos0 - key0 - 63 ... w_pos0 - key0 + w_toks - 1
        const int b_head = lane % G;                         // a lane forms the biases of one head
        const float b_r1 = biased ? -p.r1[kvh * G + b_head] : 0.f, b_r2 = biased ? p.r2[kvh * G + b_head] : 0.f;
        const float* my_bias = bias + (KV_TILE - 1 + tok_i - w_tok0) * G + (row_l - tok_i * G);      // of the tile's first key; a key on is G back
        float m_ref = -INFINITY, l_run = 0.f;
        bool ok = true;
        for (int t = t_begin; t < t_end; ++t) {
            const int it = t - t_begin;
            const int sb = it & 1;
            const int key0 = t * KV_TILE;
            if (biased) {
                const int d0 = w_pos0 - key0 - (KV_TILE - 1);
                __syncwarp();                                // (the tile before has been read)
#pragma unroll
                for (int e0 = 0; e0 < KV_TILE - 1 + w_toks; e0 += b_step) {
                    const int e = e0 + lane / G;
                    if (e < KV_TILE - 1 + w_toks) bias[e * G + b_head] = b_r1 * fast_log2(fmaf(b_r2, (float)max(d0 + e, 0), 1.0f));
                }
                __syncwarp();
            }
            if (!mbar_wait(bar_s_full0 + 8 * sb, (it >> 1) & 1, &abort_flag, 9)) { ok = false; break; }
            tcgen05_fence_after();
            uint32_t s0[32], s1[32];
            tmem_ld_32x32(t_lane + S_COL + sb * KV_TILE, s0);
            tmem_ld_32x32(t_lane + S_COL + sb * KV_TILE + 32, s1);
            tmem_ld_wait();
            tcgen05_fence_before();
            __syncwarp();
            if (biased) {
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    s0[e] = __float_as_uint(fmaf(__uint_as_float(s0[e]), p.scale_log2e, my_bias[-e * G]));
                    s1[e] = __float_as_uint(fmaf(__uint_as_float(s1[e]), p.scale_log2e, my_bias[-(e + 32) * G]));
                }
            }
            const float eff_scale = biased ? 1.f : p.scale_log2e;
            if (!(key0 + KV_TILE - 1 <= pos && key0 >= lo)) {
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    const int ka = key0 + e, kb = key0 + 32 + e;
                    if (!(ka <= pos && ka >= lo)) s0[e] = 0xff800000u;        // -inf
                    if (!(kb <= pos && kb >= lo)) s1[e] = 0xff800000u;
                }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
                mx[0] = max3(mx[0], __uint_as_float(s0[e]), __uint_as_float(s0[e + 1]));
                mx[1] = max3(mx[1], __uint_as_float(s0[e + 2]), __uint_as_float(s0[e + 3]));
                mx[2] = max3(mx[2], __uint_as_float(s1[e]), __uint_as_float(s1[e + 1]));
                mx[3] = max3(mx[3], __uint_as_float(s1[e + 2]), __uint_as_float(s1[e + 3]));
            }
            const float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * eff_scale;     // the scale is positive: the maximum commutes
            // raise the reference maximum only when it is far behind: O then needs a pass
            const bool raise = (m_ref == -INFINITY && m_tile > -INFINITY) || m_tile > m_ref + RESCALE_LOG2;
            float factor = 1.f;
            if (raise) {
                factor = m_ref == -INFINITY ? 0.f : fast_exp2(m_ref - m_tile);
                m_ref = m_tile;
                l_run *= factor;
            }
            if (__any_sync(0xffffffffu, raise && it > 0)) {
                if (!mbar_wait(bar_o_full0 + 8 * ((it - 1) & 1), ((it - 1) >> 1) & 1, &abort_flag, 11)) { ok = false; break; }
                tcgen05_fence_after();
                for (int c = 0; c < nv * VD; c += 32) {
                    uint32_t o[32];
                    tmem_ld_32x32(t_lane + O_COL + c, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * factor);
                    tmem_st_32x32(t_lane + O_COL + c, o);
                }
                tmem_st_wait();
                tcgen05_fence_before();
            }
            const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
            float l_tile = 0.f, l_tile2 = 0.f;
#pragma unroll
            for (int half = 0; half < 2; ++half) {           // 32 keys: 16 columns of their roundings, 16 of the rests (a store of each
                const uint32_t* s = half ? s1 : s0;          // half as it is done: 2,048 tokens of 16 heads on 4 163 -> 153 us, of 32 on 8 490 -> 472)
                uint32_t pk[32];
#pragma unroll
                for (int j = 0; j < 16; ++j) {               // keys 2j and 2j + 1
                    float a0, a1;
                    fma2(a0, a1, __uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1]), eff_scale, neg_m);
                    const float x0 = fast_exp2(a0), x1 = fast_exp2(a1);
                    add2(l_tile, l_tile2, x0, x1);
                    __nv_bfloat162 h2 = __floats2bfloat162_rn(x0, x1);
                    pk[j] = *reinterpret_cast<uint32_t*>(&h2);
                    h2 = __floats2bfloat162_rn(x0 - __uint_as_float(pk[j] << 16), x1 - __uint_as_float(pk[j] & 0xffff0000u));
                    pk[16 + j] = *reinterpret_cast<uint32_t*>(&h2);
                }
                tmem_st_32x32(t_lane + S_COL + sb * KV_TILE + 32 * half, pk);
            }
            l_run += l_tile + l_tile2;
            tmem_st_wait();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p_full0 + 8 * sb);
        }
        if (ok) {
            ok = mbar_wait(bar_o_full0 + 8 * ((n_it - 1) & 1), ((n_it - 1) >> 1) & 1, &abort_flag, 10);
            tcgen05_fence_after();
            if (ok) {
                const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
                const int t = q_start + tok0 + tok_i;
                const bool store = in_range && t >= p.tok_lo && t < p.tok_hi;
                float* dst = p.u + (((size_t)(store ? t - p.tok_lo : 0) * p.nkv + c0) * p.nh + head) * VD;
                for (int c = 0; c < nv; ++c, dst += (size_t)p.nh * VD) {
#pragma unroll
                    for (int e0 = 0; e0 < VD; e0 += 32) {
                        uint32_t o[32];
                        tmem_ld_32x32(t_lane + O_COL + c * VD + e0, o);
                        tmem_ld_wait();
                        if (store) {
#pragma unroll
                            for (int v = 0; v < 4; ++v)      // whole sectors
                                asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + e0 + 8 * v),
                                             "f"(__uint_as_float(o[8 * v]) * inv), "f"(__uint_as_float(o[8 * v + 1]) * inv),
                                             "f"(__uint_as_float(o[8 * v + 2]) * inv), "f"(__uint_as_float(o[8 * v + 3]) * inv),
                                             "f"(__uint_as_float(o[8 * v + 4]) * inv), "f"(__uint_as_float(o[8 * v + 5]) * inv),
                                             "f"(__uint_as_float(o[8 * v + 6]) * inv), "f"(__uint_as_float(o[8 * v + 7]) * inv) : "memory");
                        }
                    }
                }
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if (abort_flag != 0) {
        // A wait gave up somewhere: the loaders wait (bounded, without touching the flag) for what is still on its way into shared memory.
        if ((warp == LOADER_WARP || warp == VLOADER_WARP) && lane == 0) {
            volatile int ignore = 0;
            const int stages = warp == LOADER_WARP ? NK : NV;
            const uint32_t full0 = warp == LOADER_WARP ? bar_k0 : bar_v0;
            if (warp == LOADER_WARP) mbar_wait(bar_q, 0, &ignore, 0);
            for (int i = max(0, tiles_issued - stages); i < tiles_issued; ++i)
                mbar_wait(full0 + 8 * (i % stages), (i / stages) & 1, &ignore, 0);
        }
        __syncthreads();
    }
    if (left_out != 0 && abort_flag == 0 && warp < SOFTMAX_WARPS) {
        // A warp has the tokens of its rows, a lane some columns of each head: one walk over the keys of those tiles, whose sum up to a
        // token's own key is what its rows are due.
        constexpr int W = VD / 32;
        using Vec = typename WideVec<W>::type;
        const int first = pos_first + warp * 32 / G, last = pos_first + min(n_tok, (warp + 1) * 32 / G) - 1;
        const int skip_lo = (lo_last + KV_TILE - 1) / KV_TILE * KV_TILE, skip_hi = (pos_first + 1) / KV_TILE * KV_TILE;      // between: seen by all
        for (int c = 0; c < nv; ++c) {
            float sum[W] = {};
            int j = p.chunk > 0 ? (first / p.chunk) * p.chunk : 0;
            auto take = [&](int end) {
#pragma unroll 8
                for (; j < end; ++j) {
                    const __nv_bfloat16* v = p.values + (size_t)__ldg(table + (j >> p.page_shift)) * p.page_elems +
                                             ((size_t)(c0 + c) * p.page_size + (j & (p.page_size - 1))) * VD + lane * W;
#pragma unroll
                    for (int w = 0; w < W; w += 2) {
                        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(v + w));
                        if (!(fabsf(x.x) < INFINITY)) sum[w] += x.x;
                        if (!(fabsf(x.y) < INFINITY)) sum[w + 1] += x.y;
                    }
                }
            };
            for (int pos = first; pos <= last; ++pos) {
                if (p.chunk > 0 && pos % p.chunk == 0) {     // a chunk begins here
#pragma unroll
                    for (int w = 0; w < W; ++w) sum[w] = 0.f;
                    j = pos;
                }
                take(min(pos + 1, skip_lo));
                if (j >= skip_lo) j = max(j, skip_hi);
                take(pos + 1);
                const int t = q_start + tok0 + pos - pos_first;
                bool due = false;
#pragma unroll
                for (int w = 0; w < W; ++w) due |= sum[w] != 0.f;                // (also where it is no number)
                if (!due || t < p.tok_lo || t >= p.tok_hi) continue;
                float* dst = p.u + (((size_t)(t - p.tok_lo) * p.nkv + c0 + c) * p.nh + kvh * G) * VD + lane * W;
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    Vec x = *reinterpret_cast<const Vec*>(dst + h * VD);
#pragma unroll
                    for (int w = 0; w < W; ++w) reinterpret_cast<float*>(&x)[w] += sum[w];
                    *reinterpret_cast<Vec*>(dst + h * VD) = x;
                }
            }
        }
    }
    if (warp == LOADER_WARP) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
    }
    if (tid == 0 && abort_flag != 0 && p.status) atomicCAS(p.status, 0, abort_flag);
}

// A warp per (token, key/value head): the G heads on it, V_DIM elements, from the nh rows of U that share its values.  Bound by
// reading U.
template <int G, int VD>
__global__ void __launch_bounds__(256)
talking_mix_kernel(const float* __restrict__ u, const float* __restrict__ talk, __nv_bfloat16* __restrict__ out, int tokens, int tok_lo,
                   int nh, int nkv) {
    rv_pdl_launch_dependents();
    extern __shared__ float mix_talk[];                     // [nh][G]: the weights of this block's heads
    const int c = blockIdx.y, lane = threadIdx.x & 31, t = blockIdx.x * 8 + (threadIdx.x >> 5);
    for (int i = threadIdx.x; i < nh * G; i += 256) mix_talk[i] = talk[(size_t)(c * G + i % G) * nh + i / G];
    __syncthreads();
    rv_pdl_wait();
    if (t >= tokens) return;
    constexpr int W = VD / 32;                              // floats a lane
    const float* row = u + ((size_t)t * nkv + c) * nh * VD + lane * W;
    float acc[G][W];
#pragma unroll
    for (int h = 0; h < G; ++h)
#pragma unroll
        for (int w = 0; w < W; ++w) acc[h][w] = 0.f;
#pragma unroll 8
    for (int g = 0; g < nh; ++g) {
        float v[W];
        if constexpr (W == 4) { const float4 x = __ldcs(reinterpret_cast<const float4*>(row + (size_t)g * VD)); v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }
        else { const float2 x = __ldcs(reinterpret_cast<const float2*>(row + (size_t)g * VD)); v[0] = x.x; v[1] = x.y; }
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const float k = mix_talk[g * G + h];
#pragma unroll
            for (int w = 0; w < W; ++w) acc[h][w] = fmaf(k, v[w], acc[h][w]);
        }
    }
    __nv_bfloat16* dst = out + ((size_t)(tok_lo + t) * nh + c * G) * VD + lane * W;
#pragma unroll
    for (int h = 0; h < G; ++h)
#pragma unroll
        for (int w = 0; w < W; w += 2) *reinterpret_cast<__nv_bfloat162*>(dst + (size_t)h * VD + w) = __floats2bfloat162_rn(acc[h][w], acc[h][w + 1]);
}

// A map of one kind of rows (keys, or values) of a cache whose pages hold [nkv][page][hd] keys and then [nkv][page][vd] values.
static int make_page_map(CUtensorMap* map, const void* base, int width, int rows, long long num_pages, long long page_elems, int box_rows) {
    RvEncodeTiledFn fn = rv_encode_fn();
    if (!fn) return RV_ERR_UNSUPPORTED;
    const cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)rows, (cuuint64_t)num_pages};
    const cuuint64_t strides[2] = {(cuuint64_t)width * 2, (cuuint64_t)page_elems * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? RV_OK : RV_ERR_BAD_SIZE;
}

static int make_query_map(CUtensorMap* map, const void* q, int n_tokens, int nh, int hd, int G) {
    RvEncodeTiledFn fn = rv_encode_fn();
    if (!fn) return RV_ERR_UNSUPPORTED;
    const cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)nh, (cuuint64_t)n_tokens};
    const cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)nh * hd * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)(ROWS / G)};
    const cuuint32_t elem[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? RV_OK : RV_ERR_BAD_SIZE;
}

template <int HD, int VD, int G>
static int launch_wide_group(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const WideParams& p, dim3 grid, cudaStream_t stream) {
    static RvPerDevice once;
    if (int st = rv_configure_smem(once, talking_wide_kernel<HD, VD, G>, WideSizes<HD, VD>::SMEM)) return st;
    return rv_launch(talking_wide_kernel<HD, VD, G>, grid, dim3(NUM_THREADS), WideSizes<HD, VD>::SMEM, stream, mq, mk, mv, p);
}

template <int HD, int VD>
static int launch_wide(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const WideParams& p, dim3 grid, cudaStream_t stream) {
    switch (p.nh / p.nkv) {
        case 1: return launch_wide_group<HD, VD, 1>(mq, mk, mv, p, grid, stream);
        case 2: return launch_wide_group<HD, VD, 2>(mq, mk, mv, p, grid, stream);
        case 4: return launch_wide_group<HD, VD, 4>(mq, mk, mv, p, grid, stream);
        case 8: return launch_wide_group<HD, VD, 8>(mq, mk, mv, p, grid, stream);
        default: return launch_wide_group<HD, VD, 16>(mq, mk, mv, p, grid, stream);
    }
}

template <int VD>
static int launch_mix(int G, const float* u, const float* talk, void* out, int tokens, int tok_lo, int nh, int nkv, cudaStream_t stream) {
    auto kernel = G == 1 ? talking_mix_kernel<1, VD> : G == 2 ? talking_mix_kernel<2, VD> : G == 4 ? talking_mix_kernel<4, VD>
                : G == 8 ? talking_mix_kernel<8, VD> : talking_mix_kernel<16, VD>;
    return rv_launch(kernel, dim3((tokens + 7) / 8, nkv), dim3(256), sizeof(float) * nh * G, stream, u, talk, (__nv_bfloat16*)out, tokens, tok_lo, nh, nkv);
}

// 1 if the sizes fit this build.
RV_EXPORT int rv_talking_wide_fits(int nh, int nkv, int hd, int vd, int page_size) {
    if (nh <= 0 || nkv <= 0 || nh % nkv || nh > 64) return 0;
    const int G = nh / nkv;
    if (G > MAX_GROUP || (G & (G - 1))) return 0;
    if ((hd != 64 && hd != 128) || (vd != 64 && vd != 128)) return 0;
    return page_size >= 8 && (page_size & (page_size - 1)) == 0;
}

// The step's tokens [tok_lo, tok_hi) of all sequences, single tokens among them; u: float [tok_hi - tok_lo][nkv][nh][vd].
// Arguments else as of rv_talking_attention_mma; `talk` is not null.
RV_EXPORT int rv_talking_wide(const void* q, const void* cache, long long num_pages, const int* block_tables, const int* cu_seqlens,
                              const int* ctx_lens, void* out, float* u, int n_tokens, int tok_lo, int tok_hi, int n_seqs, int max_q_len,
                              int nh, int nkv, int hd, int vd, int page_size, int max_blocks, float scale, const float* r1, const float* r2,
                              const float* talk, int chunk, int* status, cudaStream_t stream) {
    if (!rv_talking_wide_fits(nh, nkv, hd, vd, page_size)) return RV_ERR_UNSUPPORTED;
    if (n_seqs < 0 || max_q_len < 0 || max_blocks <= 0 || n_seqs > 65535 || num_pages <= 0 || tok_lo < 0 || tok_hi > n_tokens || chunk < 0 ||
        !(scale > 0.f) || !talk || !u)
        return RV_ERR_BAD_SIZE;
    if ((r1 == nullptr) != (r2 == nullptr)) return RV_ERR_BAD_SIZE;
    if (((uintptr_t)cache | (uintptr_t)q | (uintptr_t)out) % 16 || (uintptr_t)u % 32) return RV_ERR_ALIGNMENT;
    if (n_seqs == 0 || max_q_len == 0 || tok_hi <= tok_lo) return RV_OK;
    const int G = nh / nkv, box_rows = page_size < KV_TILE ? page_size : KV_TILE;
    const long long page_elems = (long long)nkv * page_size * (hd + vd);
    alignas(64) CUtensorMap mq, mk, mv;
    int st = make_query_map(&mq, q, n_tokens, nh, hd, G);
    if (st == RV_OK) st = make_page_map(&mk, cache, hd, nkv * page_size, num_pages, page_elems, box_rows);
    if (st == RV_OK) st = make_page_map(&mv, (const __nv_bfloat16*)cache + (size_t)nkv * page_size * hd, vd, nkv * page_size, num_pages, page_elems, box_rows);
    if (st != RV_OK) return st;
    WideParams p;
    p.block_tables = block_tables; p.cu_seqlens = cu_seqlens; p.ctx_lens = ctx_lens; p.u = u; p.status = status;
    p.values = (const __nv_bfloat16*)cache + (size_t)nkv * page_size * hd; p.page_elems = (size_t)page_elems;
    p.nh = nh; p.nkv = nkv; p.page_size = page_size; p.max_blocks = max_blocks; p.chunk = chunk;
    p.page_shift = 0;
    while ((1 << p.page_shift) < page_size) ++p.page_shift;
    p.blocks = (nkv + O_COLS / vd - 1) / (O_COLS / vd);
    p.per_block = (nkv + p.blocks - 1) / p.blocks;
    p.tok_lo = tok_lo; p.tok_hi = tok_hi;
    p.scale_log2e = scale * 1.4426950408889634f;
    p.r1 = r1; p.r2 = r2;
    const int tile_tokens = ROWS / G;
    const dim3 grid(nkv * p.blocks, n_seqs, (max_q_len + tile_tokens - 1) / tile_tokens);
    if (grid.z > 65535) return RV_ERR_UNSUPPORTED;
    if (hd == 128) RV_LAUNCH_ST = vd == 128 ? launch_wide<128, 128>(mq, mk, mv, p, grid, stream) : launch_wide<128, 64>(mq, mk, mv, p, grid, stream);
    else RV_LAUNCH_ST = vd == 128 ? launch_wide<64, 128>(mq, mk, mv, p, grid, stream) : launch_wide<64, 64>(mq, mk, mv, p, grid, stream);
    if (RV_LAUNCH_ST != RV_OK) return rv_launch_status();
    RV_LAUNCH_ST = vd == 128 ? launch_mix<128>(G, u, talk, out, tok_hi - tok_lo, tok_lo, nh, nkv, stream)
                             : launch_mix<64>(G, u, talk, out, tok_hi - tok_lo, tok_lo, nh, nkv, stream);
    return rv_launch_status();
}
