// A mixture of experts whose choice per token is given (a table lookup by token id, a router's top-k): every token runs
// `top` experts and adds them, with one weight for all or one per (token, slot).  An expert is gated,
// down_e( silu(gate_e x) * up_e x ), or plain, down_e( relu(up_e x)^2 ).
//
// Layout: gate_up [experts, 2 ff, width] (an expert's gate rows, then its up rows; plain experts: up [experts, ff, width]),
// down [experts, width, ff], chosen [tokens, top] int32 expert numbers (numbers outside 0 .. experts-1 contribute
// nothing - or, with `identity`, numbers from `experts` on contribute the token's own vector x_t), weights float
// [tokens, top] or null.
//
//   moe_route_top act on a router's float32 logits: s = sigmoid(z); the choice is made among s + correction, within the best
//                 `keep` of `groups` equal groups of neighbouring experts (a group counts by the sum of its two largest
//                 corrected scores - or, with `group_max`, by the largest); chosen [tokens, top], weights = the chosen s over
//                 their sum (+ eps).  Mode 1: the choice is made among z + correction itself and the weights are the softmax
//                 over the chosen ones.  Mode 2: as mode 0 with s = softmax(z) over all experts
//   moe_gate_up   act[t * top + k, f] = silu(gate_e[f] . x_t) * (up_e[f] . x_t)  or  relu(up_e[f] . x_t)^2,  e = chosen[t, k]
//   moe_down      out[t, n] = (add_scale[t] add[t, n]) + weight * sum_k weights[t, k] down_e(k)[n] . act[t * top + k]
//
// One CTA per (token, slot) and block of features keeps the token's vector in shared memory as float; a warp owns a
// feature at a time and its lanes walk the weight row (16-byte loads where rows are aligned).  The weights of an
// expert are read once per token that chose it: the kernels serve decoded tokens and short portions, where the step
// is bound by reading the chosen experts' weights; sums are float, in one order whatever the batch.
//
// Many tokens take another way, on the tensor cores: the (token, slot) pairs are sorted by expert into a buffer in
// which every expert's rows are padded to whole row tiles, and two grouped products (gemm_tcgen05.cu: row tile t is
// multiplied with the matrices of expert tile_group[t]) run over it.  The kernels here do the sorting and the sum:
//
//   moe_route     row_of[pair], src_of[row] and the products' work units (tile_group, tile_rows) from chosen (one CTA:
//                 counts, padded offsets, places)
//   moe_gather    xs[row] = x[src_of[row]], zeros in the padding
//   moe_combine   out[t] = (add_scale[t] add[t]) + weight * sum_k weights[t, k] ys[row_of[t * top + k]]   (slots in their order: one sum per element)
#include "common.cuh"

// N rows of W against one vector at a time: the lanes walk all rows together, so N loads are in flight per lane and step
// (one row after the other left the memory idle between a row's reduction and the next row's first load).
template <typename T, int N>
__device__ __forceinline__ void moe_dot_rows(const T* const (&w)[N], const float* __restrict__ x, int n, int lane, float (&out)[N]) {
    float s[N];
#pragma unroll
    for (int r = 0; r < N; ++r) s[r] = 0.f;
    constexpr int V = 16 / sizeof(T);                      // elements of a 16-byte load
    bool aligned = (n % V) == 0;
#pragma unroll
    for (int r = 0; r < N; ++r) aligned = aligned && ((uintptr_t)w[r] & 15) == 0;
    if (aligned) {
        for (int i = lane * V; i < n; i += 32 * V) {
            uint4 v[N];
#pragma unroll
            for (int r = 0; r < N; ++r) v[r] = __ldg(reinterpret_cast<const uint4*>(w[r] + i));
#pragma unroll
            for (int r = 0; r < N; ++r) {
                if constexpr (sizeof(T) == 4) {
                    const float* f = reinterpret_cast<const float*>(&v[r]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[r] = fmaf(f[j], x[i + j], s[r]);
                } else {
                    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[r]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = __bfloat1622float2(h[j]);
                        s[r] = fmaf(f.x, x[i + 2 * j], s[r]);
                        s[r] = fmaf(f.y, x[i + 2 * j + 1], s[r]);
                    }
                }
            }
        }
    } else {
        for (int i = lane; i < n; i += 32)
#pragma unroll
            for (int r = 0; r < N; ++r) s[r] = fmaf(rv_to_float(w[r][i]), x[i], s[r]);
    }
#pragma unroll
    for (int r = 0; r < N; ++r) out[r] = rv_warp_sum(s[r]);
}

#define MOE_WARPS 8
#define MOE_FEATURES 32      // features of one CTA
#define MOE_PER_WARP (MOE_FEATURES / MOE_WARPS)

// grid (tokens * top, feature blocks).  GATED: an expert's first matrix holds gate rows and up rows, a CTA covers MOE_FEATURES
// features; plain: up rows only, a CTA covers twice as many (the same number of weight rows walked together).
template <typename T, bool GATED>
__global__ void __launch_bounds__(MOE_WARPS * 32)
moe_gate_up_kernel(const T* __restrict__ x, const int* __restrict__ chosen, const T* __restrict__ gate_up, T* __restrict__ act,
                   int top, int experts, int ff, int width) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ float xs[];
    const int pair = blockIdx.x, t = pair / top;
    const int e = chosen[pair];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int FEATURES = GATED ? MOE_FEATURES : 2 * MOE_FEATURES;
    const int f0 = blockIdx.y * FEATURES;
    if (e < 0 || e >= experts) {
        for (int f = f0 + threadIdx.x; f < min(ff, f0 + FEATURES); f += blockDim.x) act[(size_t)pair * ff + f] = rv_from_float<T>(0.f);
        return;
    }
    for (int i = threadIdx.x; i < width; i += blockDim.x) xs[i] = rv_to_float(x[(size_t)t * width + i]);
    __syncthreads();
    if constexpr (!GATED) {
        const T* wu = gate_up + (size_t)e * ff * width;
        const T* rows[2 * MOE_PER_WARP];
#pragma unroll
        for (int j = 0; j < 2 * MOE_PER_WARP; ++j) rows[j] = wu + (size_t)min(ff - 1, f0 + warp + j * MOE_WARPS) * width;
        float r[2 * MOE_PER_WARP];
        moe_dot_rows<T, 2 * MOE_PER_WARP>(rows, xs, width, lane, r);
#pragma unroll
        for (int j = 0; j < 2 * MOE_PER_WARP; ++j) {
            const int f = f0 + warp + j * MOE_WARPS;
            const float v = fmaxf(r[j], 0.f);
            if (lane == 0 && f < ff) act[(size_t)pair * ff + f] = rv_from_float<T>(v * v);
        }
        return;
    }
    const T* wg = gate_up + (size_t)e * 2 * ff * width;
    const T* wu = wg + (size_t)ff * width;
    // a warp's features f0 + warp, + MOE_WARPS, ...: their gate and up rows are walked together (a feature beyond ff reads
    // the last row again and is not stored)
    const T* rows[2 * MOE_PER_WARP];
#pragma unroll
    for (int j = 0; j < MOE_PER_WARP; ++j) {
        const int f = min(ff - 1, f0 + warp + j * MOE_WARPS);
        rows[2 * j] = wg + (size_t)f * width;
        rows[2 * j + 1] = wu + (size_t)f * width;
    }
    float r[2 * MOE_PER_WARP];
    moe_dot_rows<T, 2 * MOE_PER_WARP>(rows, xs, width, lane, r);
#pragma unroll
    for (int j = 0; j < MOE_PER_WARP; ++j) {
        const int f = f0 + warp + j * MOE_WARPS;
        if (lane == 0 && f < ff) act[(size_t)pair * ff + f] = rv_from_float<T>(r[2 * j] / (1.0f + expf(-r[2 * j])) * r[2 * j + 1]);
    }
}

// grid (tokens, feature blocks)
template <typename T, typename TO>
__global__ void __launch_bounds__(MOE_WARPS * 32)
moe_down_kernel(const T* __restrict__ act, const int* __restrict__ chosen, const T* __restrict__ down, const float* add,
                TO* out, int top, int experts, int ff, int width, float weight, const float* __restrict__ weights,
                const float* __restrict__ add_scale, const T* __restrict__ identity_x) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ float as[];                 // [top][ff]
    const int t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < top * ff; i += blockDim.x) as[i] = rv_to_float(act[(size_t)t * top * ff + i]);
    __syncthreads();
    const int n0 = blockIdx.y * MOE_FEATURES;
    float sum[MOE_PER_WARP];
#pragma unroll
    for (int j = 0; j < MOE_PER_WARP; ++j) sum[j] = 0.f;
    for (int k = 0; k < top; ++k) {                       // the slots in their order: one sum per element, whatever the batch
        const int e = chosen[t * top + k];
        if (e >= experts && identity_x) {
            const float wk = weights ? weights[t * top + k] : 1.f;
#pragma unroll
            for (int j = 0; j < MOE_PER_WARP; ++j)
                sum[j] = fmaf(wk, rv_to_float(identity_x[(size_t)t * width + min(width - 1, n0 + warp + j * MOE_WARPS)]), sum[j]);
            continue;
        }
        if (e < 0 || e >= experts) continue;
        const T* rows[MOE_PER_WARP];
#pragma unroll
        for (int j = 0; j < MOE_PER_WARP; ++j) rows[j] = down + ((size_t)e * width + min(width - 1, n0 + warp + j * MOE_WARPS)) * ff;
        float r[MOE_PER_WARP];
        moe_dot_rows<T, MOE_PER_WARP>(rows, as + (size_t)k * ff, ff, lane, r);
        const float wk = weights ? weights[t * top + k] : 1.f;
#pragma unroll
        for (int j = 0; j < MOE_PER_WARP; ++j) sum[j] = fmaf(wk, r[j], sum[j]);
    }
#pragma unroll
    for (int j = 0; j < MOE_PER_WARP; ++j) {
        const int n = n0 + warp + j * MOE_WARPS;
        if (lane == 0 && n < width) {
            float v = sum[j] * weight;
            if (add) v += add_scale ? add_scale[t] * add[(size_t)t * width + n] : add[(size_t)t * width + n];
            out[(size_t)t * width + n] = rv_from_float<TO>(v);
        }
    }
}

static RvPerDevice g_once[8];

template <typename T>
static int moe_launch(const void* x, const int* chosen, const float* weights, const void* gate_up, const void* down, void* act,
                      const float* add, const float* add_scale, void* out, int out_f32, int tokens, int top, int experts, int ff,
                      int width, float weight, int gated, int identity, int slot, cudaStream_t stream) {
    const int smem_a = width * 4, smem_b = top * ff * 4;
    if (smem_a > 200 * 1024 || smem_b > 200 * 1024) return RV_ERR_UNSUPPORTED;
    int st;
    if (gated) {
        st = rv_configure_smem(g_once[slot], moe_gate_up_kernel<T, true>, 200 * 1024);
        if (st != RV_OK) return st;
        RV_LAUNCH_ST = rv_launch(moe_gate_up_kernel<T, true>, dim3(tokens * top, (ff + MOE_FEATURES - 1) / MOE_FEATURES), dim3(MOE_WARPS * 32),
                                 (size_t)smem_a, stream, (const T*)x, chosen, (const T*)gate_up, (T*)act, top, experts, ff, width);
    } else {
        st = rv_configure_smem(g_once[slot + 3], moe_gate_up_kernel<T, false>, 200 * 1024);
        if (st != RV_OK) return st;
        RV_LAUNCH_ST = rv_launch(moe_gate_up_kernel<T, false>, dim3(tokens * top, (ff + 2 * MOE_FEATURES - 1) / (2 * MOE_FEATURES)),
                                 dim3(MOE_WARPS * 32), (size_t)smem_a, stream, (const T*)x, chosen, (const T*)gate_up, (T*)act, top,
                                 experts, ff, width);
    }
    st = rv_launch_status();
    if (st != RV_OK) return st;
    const dim3 grid(tokens, (width + MOE_FEATURES - 1) / MOE_FEATURES);
    if (out_f32) {
        st = rv_configure_smem(g_once[slot + 1], moe_down_kernel<T, float>, 200 * 1024);
        if (st != RV_OK) return st;
        RV_LAUNCH_ST = rv_launch(moe_down_kernel<T, float>, dim3(grid), dim3(MOE_WARPS * 32), (size_t)smem_b, stream, (const T*)act,
                                 chosen, (const T*)down, add, (float*)out, top, experts, ff, width, weight, weights, add_scale,
                                 identity ? (const T*)x : (const T*)nullptr);
    } else {
        st = rv_configure_smem(g_once[slot + 2], moe_down_kernel<T, T>, 200 * 1024);
        if (st != RV_OK) return st;
        RV_LAUNCH_ST = rv_launch(moe_down_kernel<T, T>, dim3(grid), dim3(MOE_WARPS * 32), (size_t)smem_b, stream, (const T*)act,
                                 chosen, (const T*)down, add, (T*)out, top, experts, ff, width, weight, weights, add_scale,
                                 identity ? (const T*)x : (const T*)nullptr);
    }
    return rv_launch_status();
}

// ------------------------------------------------------------------ few bfloat16 tokens on the tensor cores
// A step of few tokens is bound by reading the matrices of the experts that any of them chose.  The kernels above read them
// once per (token, slot) pair; these read each once: the pairs of an expert are the columns of an mma.sync (m16n8k16, float
// accumulators; the rate needed is one per 23 clocks and SM), sixteen rows of the matrix its rows.  The order of k inside a
// product is free, so a lane takes 8 neighbouring k of its row and of its pair as one 16-byte load each (k = 32 c + 8 (lane & 3))
// and these four words are the operands of two products: nothing passes through shared memory on the way in.
//   moe_mma_gate_up   a CTA per (expert, 16 features, or 2 x 16): eight warps share k (gated: four on the gate rows, four on the up rows),
//                     their sums meet in shared memory
//   moe_mma_down      a CTA per 16 columns of the result: its warps share the (expert, quarter of k) items, and the sums of a
//                     token's slots are added in the slots' order; a launch per block of tokens whose sums fit the shared memory
// 32 experts (4096 x 2048, gated), 4 of them for each of 8 / 64 tokens, both products: 290 / 1,411 us with the kernels above, 179 /
// 291 us (5.6 TB/s) with these.  The cuts of k depend on the sizes alone, so a row's result does not depend on the rest of
// the batch, as far as these kernels serve it (the caller takes grouped products from 128 tokens on).
__device__ __forceinline__ void moe_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Weights are read once: they leave the first-level cache to the vectors.
__device__ __forceinline__ uint4 moe_ld_weight(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// The same with c = 0.
__device__ __forceinline__ void moe_mma_new(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// acc[n]: 16 matrix rows (this lane's rows wlo, whi) against NT blocks of 8 vectors (this lane's x[n]), over the 32-wide blocks
// c0 .. c1 - 1 of k, U of them in flight (4 with one CTA more per SM: 10 % slower).  The pointers stand at 8 (lane & 3)
// elements of their row.
template <int NT>
__device__ __forceinline__ void moe_mma_span(const uint4* wlo, const uint4* whi, const uint4* const (&x)[NT], int c0, int c1, float (&acc)[NT][4]) {
    constexpr int U = NT > 2 ? 4 : 8;
    int c = c0;
    for (; c + U <= c1; c += U) {
        uint4 lo[U], hi[U];
#pragma unroll
        for (int u = 0; u < U; ++u) { lo[u] = moe_ld_weight(wlo + (c + u) * 4); hi[u] = moe_ld_weight(whi + (c + u) * 4); }
#pragma unroll
        for (int u0 = 0; u0 < U; u0 += 4)                   // sums of 128 k from zero, then added in float: the tensor cores cut off what
#pragma unroll                                              // float rounds, so no sum runs through all of k there
            for (int n = 0; n < NT; ++n) {
                float part[4];
#pragma unroll
                for (int u = u0; u < u0 + 4; ++u) {
                    const uint4 b = x[n][(c + u) * 4];
                    if (u == u0) moe_mma_new(part, lo[u].x, hi[u].x, lo[u].y, hi[u].y, b.x, b.y);
                    else moe_mma(part, lo[u].x, hi[u].x, lo[u].y, hi[u].y, b.x, b.y);
                    moe_mma(part, lo[u].z, hi[u].z, lo[u].w, hi[u].w, b.z, b.w);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[n][j] += part[j];
            }
    }
    for (; c < c1; ++c) {
        const uint4 lo = moe_ld_weight(wlo + c * 4), hi = moe_ld_weight(whi + c * 4);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const uint4 b = x[n][c * 4];
            moe_mma(acc[n], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
            moe_mma(acc[n], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
        }
    }
}

#define MM_WARPS 8
#define MM_PASS 32              // pairs of one expert that one pass over its rows serves

// NT blocks of 8 pairs from list[p0] on: the products of this warp's rows (gated experts: the first half of the warps takes the
// gate rows, the second the up rows) and part of k, left in red[warp][row][pair].
template <bool GATED, int NT>
__device__ __forceinline__ void moe_gate_up_pass(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* w0,
                                                 const int* list, int count, int p0, int f0, int top, int ff, int width, float* red) {
    constexpr int PARTS = GATED ? MM_WARPS / 2 : MM_WARPS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3, part = warp % PARTS;
    const __nv_bfloat16* w = w0 + (warp >= PARTS ? (size_t)ff * width : 0);
    const uint4* wlo = reinterpret_cast<const uint4*>(w + (size_t)min(ff - 1, f0 + g) * width) + q;
    const uint4* whi = reinterpret_cast<const uint4*>(w + (size_t)min(ff - 1, f0 + g + 8) * width) + q;
    const uint4* xr[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n)                            // (a column beyond the list repeats its last pair and is not stored)
        xr[n] = reinterpret_cast<const uint4*>(x + (size_t)(list[min(count - 1, p0 + n * 8 + g)] / top) * width) + q;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[n][j] = 0.f;
    const int blocks = width / 32;
    moe_mma_span<NT>(wlo, whi, xr, part * blocks / PARTS, (part + 1) * blocks / PARTS, acc);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) red[(warp * 16 + g + 8 * (j >> 1)) * MM_PASS + n * 8 + 2 * q + (j & 1)] = acc[n][j];
}

// grid (at most min(pairs, experts) experts in use, feature blocks); shared memory: presence bits, the expert's pairs, the sums
template <bool GATED>
__global__ void __launch_bounds__(MM_WARPS * 32, 2)
moe_mma_gate_up_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ chosen, const __nv_bfloat16* __restrict__ gate_up,
                       __nv_bfloat16* __restrict__ act, int pairs, int top, int experts, int ff, int width) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ __align__(16) float mm_smem[];
    constexpr int MT = GATED ? 2 : 1, PARTS = MM_WARPS / MT;
    float* red = mm_smem;                                   // [warps][16][MM_PASS]
    int* bits = reinterpret_cast<int*>(red + MM_WARPS * 16 * MM_PASS);
    int* list = bits + (experts + 31) / 32;
    __shared__ int expert_s, count_s;
    const int words = (experts + 31) / 32, tid = threadIdx.x;
    if (tid == 0) { expert_s = -1; count_s = 0; }
    for (int i = tid; i < words; i += blockDim.x) bits[i] = 0;
    __syncthreads();
    for (int i = tid; i < pairs; i += blockDim.x) {
        const int e = chosen[i];
        if (e >= 0 && e < experts) atomicOr(&bits[e >> 5], 1 << (e & 31));
    }
    __syncthreads();
    if (tid < 32) {                                         // the blockIdx.x-th expert in use
        int before = 0;
        for (int w0 = 0; w0 < words; w0 += 32) {
            const unsigned b = w0 + tid < words ? (unsigned)bits[w0 + tid] : 0u;
            int n = __popc(b), at = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, at, o); if (tid >= o) at += v; }
            const int first = before + at - n;
            if ((int)blockIdx.x >= first && (int)blockIdx.x < first + n) expert_s = (w0 + tid) * 32 + __fns(b, 0, blockIdx.x - first + 1);
            before += __shfl_sync(0xffffffffu, at, 31);
        }
    }
    __syncthreads();
    const int e = expert_s;
    if (e < 0) return;
    for (int i = tid; i < pairs; i += blockDim.x)
        if (chosen[i] == e) list[atomicAdd(&count_s, 1)] = i;
    __syncthreads();
    const int count = count_s;
    const __nv_bfloat16* w = gate_up + (size_t)e * MT * ff * width;
    for (int f0 = blockIdx.y * 16; f0 < ff; f0 += gridDim.y * 16)
    for (int p0 = 0; p0 < count; p0 += MM_PASS) {
        const int left = min(MM_PASS, count - p0);
        if (left <= 8) moe_gate_up_pass<GATED, 1>(x, w, list, count, p0, f0, top, ff, width, red);
        else if (left <= 16) moe_gate_up_pass<GATED, 2>(x, w, list, count, p0, f0, top, ff, width, red);
        else moe_gate_up_pass<GATED, 4>(x, w, list, count, p0, f0, top, ff, width, red);
        __syncthreads();
        for (int i = tid; i < left * 16; i += blockDim.x) {
            const int row = i & 15, p = i >> 4, f = f0 + row;
            float s[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                double sum = 0.0;                           // (the parts meet with one rounding)
#pragma unroll
                for (int w = 0; w < PARTS; ++w) sum += (double)red[((m * PARTS + w) * 16 + row) * MM_PASS + p];
                s[m] = (float)sum;
            }
            float v;
            if constexpr (GATED) v = s[0] / (1.0f + expf(-s[0])) * s[MT - 1];
            else { v = fmaxf(s[0], 0.f); v *= v; }
            if (f < ff) act[(size_t)list[p0 + p] * ff + f] = __float2bfloat16_rn(v);
        }
        __syncthreads();
    }
}

#define MM_QUARTERS 4

template <int NT>
__device__ __forceinline__ void moe_down_pass(const __nv_bfloat16* __restrict__ act, const __nv_bfloat16* wd, const int* list, int count,
                                              int p0, int n0, int quarter, int ff, int width, float* part, int pairs) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const uint4* wlo = reinterpret_cast<const uint4*>(wd + (size_t)min(width - 1, n0 + g) * ff) + q;
    const uint4* whi = reinterpret_cast<const uint4*>(wd + (size_t)min(width - 1, n0 + g + 8) * ff) + q;
    const uint4* xr[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) xr[n] = reinterpret_cast<const uint4*>(act + (size_t)list[min(count - 1, p0 + n * 8 + g)] * ff) + q;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[n][j] = 0.f;
    const int blocks = ff / 32;
    moe_mma_span<NT>(wlo, whi, xr, quarter * blocks / MM_QUARTERS, (quarter + 1) * blocks / MM_QUARTERS, acc);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = p0 + n * 8 + 2 * q + (j & 1);
            if (p < count) part[((size_t)quarter * pairs + list[p]) * 16 + g + 8 * (j >> 1)] = acc[n][j];
        }
}

// grid: blocks of 16 columns; shared memory: partial sums [quarters][pairs][16], counts and offsets per expert, experts in use, sorted pairs
template <typename TO>
__global__ void __launch_bounds__(MM_WARPS * 32, 2)
moe_mma_down_kernel(const __nv_bfloat16* __restrict__ act, const int* __restrict__ chosen, const __nv_bfloat16* __restrict__ down,
                    const float* add, TO* out, int tokens, int top, int experts, int ff, int width, float weight,
                    const float* __restrict__ weights, const float* __restrict__ add_scale, const __nv_bfloat16* __restrict__ identity_x) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ __align__(16) float mm_smem[];
    const int pairs = tokens * top, tid = threadIdx.x, n0 = blockIdx.x * 16;
    float* part = mm_smem;
    int* counts = reinterpret_cast<int*>(part + (size_t)MM_QUARTERS * pairs * 16);
    int* offsets = counts + experts;
    int* used = offsets + experts;                          // at most min(pairs, experts)
    int* list = used + min(pairs, experts);
    __shared__ int used_s;
    for (int i = tid; i < experts; i += blockDim.x) counts[i] = 0;
    __syncthreads();
    for (int i = tid; i < pairs; i += blockDim.x) {
        const int e = chosen[i];
        if (e >= 0 && e < experts) atomicAdd(&counts[e], 1);
    }
    __syncthreads();
    if (tid < 32) {
        int rows = 0, n_used = 0;
        for (int e0 = 0; e0 < experts; e0 += 32) {
            const int n = e0 + tid < experts ? counts[e0 + tid] : 0;
            int at = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, at, o); if (tid >= o) at += v; }
            const unsigned has = __ballot_sync(0xffffffffu, n > 0);
            if (n > 0) used[n_used + __popc(has & ((1u << tid) - 1u))] = e0 + tid;
            if (e0 + tid < experts) offsets[e0 + tid] = rows + at - n;
            rows += __shfl_sync(0xffffffffu, at, 31);
            n_used += __popc(has);
        }
        if (tid == 0) used_s = n_used;
    }
    __syncthreads();
    for (int i = tid; i < pairs; i += blockDim.x) {
        const int e = chosen[i];
        if (e >= 0 && e < experts) list[atomicAdd(&offsets[e], 1)] = i;      // (afterwards offsets[e] is the end of e's pairs)
    }
    __syncthreads();
    const int items = used_s * MM_QUARTERS;
    for (int item = tid >> 5; item < items; item += MM_WARPS) {
        const int e = used[item / MM_QUARTERS], quarter = item % MM_QUARTERS, count = counts[e];
        const int* mine = list + offsets[e] - count;
        const __nv_bfloat16* wd = down + (size_t)e * width * ff;
        for (int p0 = 0; p0 < count; p0 += MM_PASS) {
            const int left = min(MM_PASS, count - p0);
            if (left <= 8) moe_down_pass<1>(act, wd, mine, count, p0, n0, quarter, ff, width, part, pairs);
            else if (left <= 16) moe_down_pass<2>(act, wd, mine, count, p0, n0, quarter, ff, width, part, pairs);
            else moe_down_pass<4>(act, wd, mine, count, p0, n0, quarter, ff, width, part, pairs);
        }
    }
    __syncthreads();
    for (int i = tid; i < tokens * 16; i += blockDim.x) {
        const int t = i >> 4, n = n0 + (i & 15);
        if (n >= width) continue;
        double sum = 0.0;                                   // quarters, slots and `add` meet with one rounding: the parts' cut sums are a little
        for (int k = 0; k < top; ++k) {                     // further from 64 bits than float chains, and these roundings were as large
            const int pair = t * top + k, e = chosen[pair];
            const double wk = weights ? (double)weights[pair] : 1.0;
            if (e >= experts && identity_x) sum = fma(wk, (double)__bfloat162float(identity_x[(size_t)t * width + n]), sum);
            if (e < 0 || e >= experts) continue;
            const float* p = part + (size_t)pair * 16 + (i & 15);
            const size_t step = (size_t)pairs * 16;
            sum = fma(wk, ((double)p[0] + (double)p[step]) + ((double)p[2 * step] + (double)p[3 * step]), sum);
        }
        double v = sum * (double)weight;
        if (add) v += (add_scale ? (double)add_scale[t] : 1.0) * (double)add[(size_t)t * width + n];
        out[(size_t)t * width + n] = rv_from_float<TO>((float)v);
    }
}

// Whether the kernels above serve the sizes: rows of whole 32-wide blocks, and sums and lists that fit shared memory.
static size_t moe_mma_gate_up_smem(int pairs, int experts) {
    return (size_t)MM_WARPS * 16 * MM_PASS * 4 + (size_t)((experts + 31) / 32 + pairs) * 4;
}
static size_t moe_mma_down_smem(int pairs, int experts) {
    return (size_t)MM_QUARTERS * pairs * 16 * 4 + (size_t)(2 * experts + (pairs < experts ? pairs : experts) + pairs) * 4;
}
#define MM_SMEM_MAX (160 * 1024)
// The launches of moe_mma_down for `tokens` tokens (0: the sums of one token do not fit).  A second reads the matrices again, but the
// kernels above read them once per pair: 80 tokens of 8 of 64 experts of 2048 x 1408, 640 pairs, 455 us so and 1,324 with those; 127
// tokens of 8 of 32 of 4096 x 2048 742 and 5,146.
RV_EXPORT int rv_moe_down_blocks(int tokens, int top, int experts) {
    int fit = tokens;
    while (fit > 0 && moe_mma_down_smem(fit * top, experts) > MM_SMEM_MAX) --fit;
    return fit > 0 ? (tokens + fit - 1) / fit : 0;
}

static int moe_mma_launch(const __nv_bfloat16* x, const int* chosen, const float* weights, const __nv_bfloat16* gate_up,
                          const __nv_bfloat16* down, __nv_bfloat16* act, const float* add, const float* add_scale, void* out, int out_f32,
                          int tokens, int top, int experts, int ff, int width, float weight, int gated, int identity, cudaStream_t stream) {
    static RvPerDevice once[4];
    const int pairs = tokens * top;
    // Two feature blocks a CTA where one each would be more than the SMs hold at a time (two CTAs): finding the expert and its pairs
    // costs less (16 pairs on 13 experts of 2048 x 4096, both kernels: 80.1 -> 77.2 us; four blocks 81.6).  2 pairs on 88
    // blocks: 15.1 us so, 16.5 with two.
    const int used = pairs < experts ? pairs : experts, blocks = (ff + 15) / 16;
    const dim3 grid(used, (long long)used * blocks > 2LL * rv_sm_count() ? (blocks + 1) / 2 : blocks);
    const size_t smem_a = moe_mma_gate_up_smem(pairs, experts);
    // The first kernel waits for its predecessors at the launch: its loads go through L1, and CTAs that came in early, beside a product
    // whose stages fill the SM's shared memory, kept the SM in that division, with no room for what they ask for (8 tokens
    // of 4 experts, 2048 x 4096, behind the shared expert's products: 312 us for both kernels, 171 us launched so).
    int st;
    if (gated) {
        if ((st = rv_configure_smem(once[0], moe_mma_gate_up_kernel<true>, MM_SMEM_MAX)) != RV_OK) return st;
        st = rv_launch_alone(moe_mma_gate_up_kernel<true>, grid, dim3(MM_WARPS * 32), smem_a, stream, x, chosen, gate_up, act, pairs, top, experts, ff, width);
    } else {
        if ((st = rv_configure_smem(once[1], moe_mma_gate_up_kernel<false>, MM_SMEM_MAX)) != RV_OK) return st;
        st = rv_launch_alone(moe_mma_gate_up_kernel<false>, grid, dim3(MM_WARPS * 32), smem_a, stream, x, chosen, gate_up, act, pairs, top, experts, ff, width);
    }
    if (st != RV_OK) return st;
    const dim3 grid_b((width + 15) / 16);
    const int blocks_b = rv_moe_down_blocks(tokens, top, experts), per = (tokens + blocks_b - 1) / blocks_b;
    st = out_f32 ? rv_configure_smem(once[2], moe_mma_down_kernel<float>, MM_SMEM_MAX) : rv_configure_smem(once[3], moe_mma_down_kernel<__nv_bfloat16>, MM_SMEM_MAX);
    for (int t0 = 0; t0 < tokens && st == RV_OK; t0 += per) {
        const int n = tokens - t0 < per ? tokens - t0 : per;
        const size_t first = (size_t)t0 * top, at = (size_t)t0 * width, smem_b = moe_mma_down_smem(n * top, experts);
        const float* w = weights ? weights + first : nullptr;
        const float* a = add ? add + at : nullptr;
        const float* scale = add_scale ? add_scale + t0 : nullptr;
        const __nv_bfloat16* own = identity ? x + at : nullptr;
        if (out_f32)
            st = rv_launch(moe_mma_down_kernel<float>, grid_b, dim3(MM_WARPS * 32), smem_b, stream, act + first * ff, chosen + first, down, a, (float*)out + at,
                           n, top, experts, ff, width, weight, w, scale, own);
        else
            st = rv_launch(moe_mma_down_kernel<__nv_bfloat16>, grid_b, dim3(MM_WARPS * 32), smem_b, stream, act + first * ff, chosen + first, down, a,
                           (__nv_bfloat16*)out + at, n, top, experts, ff, width, weight, w, scale, own);
    }
    RV_LAUNCH_ST = st;
    return rv_launch_status();
}

// x [tokens, width], act [tokens * top, ff] (scratch of the weights' type), add float [tokens, width] or null, add_scale float
// [tokens] or null (1),
// weights float [tokens, top] or null, out [tokens, width] float (out_f32) or of the weights' type.  gated: 1 the experts'
// first matrix is [gate | up] with SiLU, 0 it is the up matrix with a squared relu.  Two launches.
RV_EXPORT int rv_moe_experts_ex(const void* x, const int* chosen, const float* weights, const void* gate_up, const void* down, void* act,
                                const float* add, const float* add_scale, void* out, int out_f32, int tokens, int top, int experts,
                                int ff, int width, float weight, int gated, int identity, int dtype, cudaStream_t stream) {
    if (tokens < 0 || top <= 0 || experts <= 0 || ff <= 0 || width <= 0) return RV_ERR_BAD_SIZE;
    if ((long long)tokens * top > 0x7fffffffLL || ff > 65535 * MOE_FEATURES || width > 65535 * MOE_FEATURES) return RV_ERR_BAD_SIZE;
    if (tokens == 0) return RV_OK;
    if (dtype == RV_DTYPE_F32)
        return moe_launch<float>(x, chosen, weights, gate_up, down, act, add, add_scale, out, 1, tokens, top, experts, ff, width, weight, gated, identity, 0,
                                 stream);
    if (dtype == RV_DTYPE_BF16 && width % 32 == 0 && ff % 32 == 0 && (long long)tokens * top <= 4096 && experts <= 4096 && (ff + 15) / 16 <= 65535 &&
        ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(down) | reinterpret_cast<uintptr_t>(act)) & 15) == 0 &&
        moe_mma_gate_up_smem(tokens * top, experts) <= MM_SMEM_MAX && rv_moe_down_blocks(tokens, top, experts) > 0)
        return moe_mma_launch((const __nv_bfloat16*)x, chosen, weights, (const __nv_bfloat16*)gate_up, (const __nv_bfloat16*)down, (__nv_bfloat16*)act,
                              add, add_scale, out, out_f32, tokens, top, experts, ff, width, weight, gated, identity, stream);
    if (dtype == RV_DTYPE_BF16)
        return moe_launch<__nv_bfloat16>(x, chosen, weights, gate_up, down, act, add, add_scale, out, out_f32, tokens, top, experts, ff, width,
                                         weight, gated, identity, 4, stream);
    return RV_ERR_BAD_DTYPE;
}

RV_EXPORT int rv_moe_experts(const void* x, const int* chosen, const void* gate_up, const void* down, void* act, const float* add,
                             void* out, int out_f32, int tokens, int top, int experts, int ff, int width, float weight,
                             int dtype, cudaStream_t stream) {
    return rv_moe_experts_ex(x, chosen, nullptr, gate_up, down, act, add, nullptr, out, out_f32, tokens, top, experts, ff, width, weight, 1, 0,
                             dtype, stream);
}

// ------------------------------------------------------------------ sorting pairs by expert for the grouped products
// One CTA.  Shared memory: counts[experts], offsets[experts], cursor[experts], first unit[experts].
// Rows: expert e gets ceil(count / block) blocks of `block` rows from offsets[e] on.  Work units of the grouped product:
// `ranks` blocks of one expert each (the CTAs of a tile); where an expert's blocks run out, the unit's last entries are -1.
// order_a / order_b: the work lists of the two products (nt_a / nt_b column tiles per unit), see GemmParams::tile_order.
__global__ void __launch_bounds__(1024)
moe_route_kernel(const int* __restrict__ chosen, int pairs, int top, int experts, int block, int max_rows, int ranks, int max_units,
                 int* __restrict__ row_of, int* __restrict__ src_of, int* __restrict__ tile_group, int* __restrict__ tile_rows,
                 int nt_a, int* __restrict__ order_a, int nt_b, int* __restrict__ order_b) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ int sm[];
    int* counts = sm;
    int* offsets = sm + experts;
    int* cursor = sm + 2 * experts;
    int* unit0 = sm + 3 * experts;
    for (int e = threadIdx.x; e < experts; e += blockDim.x) { counts[e] = 0; cursor[e] = 0; }
    for (int r = threadIdx.x; r < max_rows; r += blockDim.x) src_of[r] = -1;
    for (int t = threadIdx.x; t < max_units; t += blockDim.x) tile_group[t] = -1;
    for (int t = threadIdx.x; t < max_units * ranks; t += blockDim.x) tile_rows[t] = -1;
    for (int t = threadIdx.x; t < max_units * nt_a; t += blockDim.x) order_a[t] = -1;
    for (int t = threadIdx.x; t < max_units * nt_b; t += blockDim.x) order_b[t] = -1;
    __syncthreads();
    for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
        const int e = chosen[i];
        if (e >= 0 && e < experts) atomicAdd(&counts[e], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int at = 0, unit = 0;
        for (int e = 0; e < experts; ++e) {
            const int blocks = (counts[e] + block - 1) / block;
            offsets[e] = at;
            unit0[e] = unit;
            at += blocks * block;
            unit += (blocks + ranks - 1) / ranks;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < experts; e += blockDim.x) {
        const int blocks = (counts[e] + block - 1) / block;
        for (int b = 0; b < blocks; ++b) {
            const int unit = unit0[e] + b / ranks;
            if (unit >= max_units) break;
            tile_group[unit] = e;
            tile_rows[unit * ranks + b % ranks] = offsets[e] + b * block;
        }
        // the order of the two products' work: this expert's entries lie together, column tile by column tile, its units within
        const int units = min((blocks + ranks - 1) / ranks, max(0, max_units - unit0[e]));
        for (int i = 0; i < units * nt_a; ++i) order_a[unit0[e] * nt_a + i] = ((unit0[e] + i % units) << 16) | (i / units);
        for (int i = 0; i < units * nt_b; ++i) order_b[unit0[e] * nt_b + i] = ((unit0[e] + i % units) << 16) | (i / units);
    }
    for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
        const int e = chosen[i];
        int row = -1;
        if (e >= 0 && e < experts) {
            row = offsets[e] + atomicAdd(&cursor[e], 1);
            if (row < max_rows) src_of[row] = i / top; else row = -1;
        }
        row_of[i] = row;
    }
}

// xs[row, :] = x[src_of[row], :] or zeros; 16-byte words (`words` per row)
__global__ void moe_gather_kernel(const uint4* __restrict__ x, const int* __restrict__ src_of, uint4* __restrict__ xs, int words,
                                  size_t total) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t row = i / words;
        const int src = src_of[row];
        xs[i] = src >= 0 ? x[(size_t)src * words + (i - row * words)] : make_uint4(0u, 0u, 0u, 0u);
    }
}

template <typename TO>
__global__ void moe_combine_kernel(const float* __restrict__ ys, const int* __restrict__ row_of, const float* add, TO* out,
                                   int top, int width, float weight, size_t total, const float* __restrict__ weights,
                                   const float* __restrict__ add_scale, const __nv_bfloat16* __restrict__ identity_x,
                                   const int* __restrict__ chosen, int experts) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / width;
        const int n = (int)(i - t * width);
        float s = 0.f;
        for (int k = 0; k < top; ++k) {
            const int row = row_of[t * top + k];
            if (row >= 0) s = fmaf(weights ? weights[t * top + k] : 1.f, ys[(size_t)row * width + n], s);
            else if (identity_x && chosen[t * top + k] >= experts)
                s = fmaf(weights ? weights[t * top + k] : 1.f, __bfloat162float(identity_x[i]), s);
        }
        float v = s * weight;
        if (add) v += add_scale ? add_scale[t] * add[i] : add[i];
        out[i] = rv_from_float<TO>(v);
    }
}

// The same for widths in multiples of 4: a block per token, its rows and weights in shared memory, four columns a thread and four
// rows in flight; the sums in the same order.
template <typename TO>
__global__ void __launch_bounds__(256)
moe_combine_vec_kernel(const float* __restrict__ ys, const int* __restrict__ row_of, const float* add, TO* out, int top, int width,
                       float weight, const float* __restrict__ weights, const float* __restrict__ add_scale,
                       const __nv_bfloat16* __restrict__ identity_x, const int* __restrict__ chosen, int experts) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ float mc_smem[];                    // weights [top], rows [top] (-1: nothing, -2: the token itself)
    int* rows = reinterpret_cast<int*>(mc_smem + top);
    const size_t t = blockIdx.x;
    for (int k = threadIdx.x; k < top; k += blockDim.x) {
        const int r = row_of[t * top + k];
        rows[k] = r >= 0 ? r : (identity_x && chosen[t * top + k] >= experts ? -2 : -1);
        mc_smem[k] = weights ? weights[t * top + k] : 1.f;
    }
    __syncthreads();
    const float scale = add && add_scale ? add_scale[t] : 1.f;
    for (int q = threadIdx.x; q < width / 4; q += blockDim.x) {
        const size_t at = t * width + 4 * (size_t)q;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), s = a;
        if (add) a = *reinterpret_cast<const float4*>(add + at);
        for (int k0 = 0; k0 < top; k0 += 4) {
            float4 y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int r = k0 + j < top ? rows[k0 + j] : -1;
                if (r >= 0) {
                    y[j] = *reinterpret_cast<const float4*>(ys + (size_t)r * width + 4 * (size_t)q);
                } else if (r == -2) {
                    const uint2 u = *reinterpret_cast<const uint2*>(identity_x + at);
                    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
                    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
                    y[j] = make_float4(lo.x, lo.y, hi.x, hi.y);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (k0 + j < top && rows[k0 + j] != -1) {
                    const float w = mc_smem[k0 + j];
                    s.x = fmaf(w, y[j].x, s.x); s.y = fmaf(w, y[j].y, s.y);
                    s.z = fmaf(w, y[j].z, s.z); s.w = fmaf(w, y[j].w, s.w);
                }
            }
        }
        s.x = fmaf(scale, a.x, s.x * weight); s.y = fmaf(scale, a.y, s.y * weight);
        s.z = fmaf(scale, a.z, s.z * weight); s.w = fmaf(scale, a.w, s.w * weight);
        if constexpr (sizeof(TO) == 4) {
            *reinterpret_cast<float4*>(out + at) = s;
        } else {
            __nv_bfloat162 lo = __floats2bfloat162_rn(s.x, s.y), hi = __floats2bfloat162_rn(s.z, s.w);
            uint2 pk;
            pk.x = *reinterpret_cast<uint32_t*>(&lo); pk.y = *reinterpret_cast<uint32_t*>(&hi);
            *reinterpret_cast<uint2*>(out + at) = pk;
        }
    }
}

RV_EXPORT int rv_moe_route(const int* chosen, int pairs, int top, int experts, int block, int max_rows, int ranks, int max_units,
                           int* row_of, int* src_of, int* tile_group, int* tile_rows, int nt_a, int* order_a, int nt_b, int* order_b,
                           cudaStream_t stream) {
    if (pairs < 0 || top <= 0 || experts <= 0 || block <= 0 || max_rows <= 0 || ranks <= 0 || max_units <= 0) return RV_ERR_BAD_SIZE;
    if (nt_a <= 0 || nt_b <= 0 || nt_a > 65535 || nt_b > 65535 || max_units > 32767 || !order_a || !order_b) return RV_ERR_BAD_SIZE;
    if (experts > 4096) return RV_ERR_UNSUPPORTED;
    if ((long long)max_rows < (long long)pairs) return RV_ERR_BAD_SIZE;
    RV_LAUNCH_ST = rv_launch(moe_route_kernel, dim3(1), dim3(1024), (size_t)4 * experts * sizeof(int), stream, chosen, pairs, top, experts,
                             block, max_rows, ranks, max_units, row_of, src_of, tile_group, tile_rows, nt_a, order_a, nt_b, order_b);
    return rv_launch_status();
}

RV_EXPORT int rv_moe_gather(const void* x, const int* src_of, void* xs, int rows, int width_bytes, cudaStream_t stream) {
    if (rows < 0 || width_bytes <= 0 || width_bytes % 16) return RV_ERR_BAD_SIZE;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(xs)) % 16) return RV_ERR_ALIGNMENT;
    if (rows == 0) return RV_OK;
    const size_t total = (size_t)rows * (width_bytes / 16);
    const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    RV_LAUNCH_ST = rv_launch(moe_gather_kernel, dim3(blocks), dim3(256), 0, stream, (const uint4*)x, src_of, (uint4*)xs, width_bytes / 16, total);
    return rv_launch_status();
}

RV_EXPORT int rv_moe_combine(const float* ys, const int* row_of, const float* add, void* out, int out_f32, int tokens, int top,
                             int width, float weight, const float* weights, const float* add_scale, const void* identity_x,
                             const int* chosen, int experts, cudaStream_t stream) {
    if (identity_x && (!chosen || experts <= 0)) return RV_ERR_BAD_SIZE;
    if (tokens < 0 || top <= 0 || width <= 0) return RV_ERR_BAD_SIZE;
    if (tokens == 0) return RV_OK;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(ys) | reinterpret_cast<uintptr_t>(add) | reinterpret_cast<uintptr_t>(out) |
                           reinterpret_cast<uintptr_t>(identity_x);
    if (width % 4 == 0 && bits % 16 == 0 && top <= 4096) {
        const size_t smem = (size_t)top * 8;
        const int threads = width >= 1024 ? 256 : 128;
        if (out_f32)
            RV_LAUNCH_ST = rv_launch(moe_combine_vec_kernel<float>, dim3(tokens), dim3(threads), smem, stream, ys, row_of, add, (float*)out, top,
                                     width, weight, weights, add_scale, (const __nv_bfloat16*)identity_x, chosen, experts);
        else
            RV_LAUNCH_ST = rv_launch(moe_combine_vec_kernel<__nv_bfloat16>, dim3(tokens), dim3(threads), smem, stream, ys, row_of, add,
                                     (__nv_bfloat16*)out, top, width, weight, weights, add_scale, (const __nv_bfloat16*)identity_x, chosen, experts);
        return rv_launch_status();
    }
    const size_t total = (size_t)tokens * width;
    const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    if (out_f32)
        RV_LAUNCH_ST = rv_launch(moe_combine_kernel<float>, dim3(blocks), dim3(256), 0, stream, ys, row_of, add, (float*)out, top, width, weight, total, weights, add_scale,
                                 (const __nv_bfloat16*)identity_x, chosen, experts);
    else
        RV_LAUNCH_ST = rv_launch(moe_combine_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, ys, row_of, add, (__nv_bfloat16*)out, top,
                                 width, weight, total, weights, add_scale, (const __nv_bfloat16*)identity_x, chosen, experts);
    return rv_launch_status();
}

// ------------------------------------------------------------------ the router's choice
// One warp per token.  Shared memory per warp: s[experts], c[experts], group scores[groups].
#define MR_WARPS 4

__device__ __forceinline__ void mr_argmax(const float* v, int n, int lane, float& best, int& at) {
    best = -INFINITY; at = 0x7fffffff;
    for (int i = lane; i < n; i += 32) {
        const float x = v[i];
        if (x > best || (x == best && i < at)) { best = x; at = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
}

__global__ void __launch_bounds__(MR_WARPS * 32)
moe_route_top_kernel(const float* __restrict__ logits, int stride, const float* __restrict__ correction, int* __restrict__ chosen,
                     float* __restrict__ weights, float* __restrict__ gate_out, int tokens, int experts, int top, int groups, int keep,
                     float weight_eps, int mode, int group_max) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ float mr_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x * MR_WARPS + warp;
    if (t >= tokens) return;
    float* s = mr_smem + (size_t)warp * (2 * experts + groups);
    float* c = s + experts;
    float* gs = c + experts;
    const float* z = logits + (size_t)t * stride;
    const bool softmax = mode == 1;
    if (mode == 2) {                                        // a softmax over all experts; every lane keeps to its own entries
        float most = -INFINITY, total = 0.f;
        for (int e = lane; e < experts; e += 32) most = fmaxf(most, z[e]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
        for (int e = lane; e < experts; e += 32) { s[e] = expf(z[e] - most); total += s[e]; }
        total = rv_warp_sum(total);
        for (int e = lane; e < experts; e += 32) { s[e] = s[e] / total; c[e] = s[e] + correction[e]; }
    } else {
        for (int e = lane; e < experts; e += 32) {
            const float v = softmax ? z[e] + correction[e] : 1.0f / (1.0f + expf(-z[e]));
            s[e] = v;
            c[e] = softmax ? v : v + correction[e];
        }
    }
    if (gate_out && lane == 0) gate_out[t] = 1.0f / (1.0f + expf(-z[experts]));
    __syncwarp();
    if (keep < groups) {
        const int per = experts / groups;
        for (int g = lane; g < groups; g += 32) {           // a group counts by its two largest corrected scores, or the largest
            float a = -INFINITY, b = -INFINITY;
            for (int i = 0; i < per; ++i) {
                const float v = c[g * per + i];
                if (v > a) { b = a; a = v; } else if (v > b) b = v;
            }
            gs[g] = per > 1 && !group_max ? a + b : a;
        }
        __syncwarp();
        for (int k = 0; k < keep; ++k) {                    // the kept groups are marked +inf, then the others are closed
            float best; int at;
            mr_argmax(gs, groups, lane, best, at);
            if (lane == 0 && at < groups) gs[at] = -INFINITY;
            __syncwarp();
        }
        for (int e = lane; e < experts; e += 32)
            if (gs[e / per] != -INFINITY) c[e] = -INFINITY;  // (a kept group was set to -inf when it was taken)
        __syncwarp();
    }
    float sum = 0.f, mine = 0.f, largest = 0.f;
    for (int k = 0; k < top; ++k) {
        float best; int at;
        mr_argmax(c, experts, lane, best, at);
        if (at >= experts) at = 0;                           // (cannot happen: top <= the experts of the kept groups)
        if (k == 0) largest = s[at];                         // (with one score per expert the first choice has the largest)
        const float w = softmax ? expf(s[at] - largest) : s[at];
        sum += w;
        if (lane == k % 32 && k < 32) mine = w;
        if (lane == 0) {
            chosen[(size_t)t * top + k] = at;
            if (k >= 32) weights[(size_t)t * top + k] = w;    // (beyond a warp's lanes: scaled below through memory)
            c[at] = -INFINITY;
        }
        __syncwarp();
    }
    const float inv = 1.0f / (sum + weight_eps);
    if (lane < top && lane < 32) weights[(size_t)t * top + lane] = mine * inv;
    if (lane == 0)
        for (int k = 32; k < top; ++k) weights[(size_t)t * top + k] *= inv;
}

// logits float [tokens, stride]: the experts' logits and, with gate_out, one more column whose sigmoid goes to gate_out.
RV_EXPORT int rv_moe_route_top(const float* logits, int stride, const float* correction, int* chosen, float* weights, float* gate_out,
                               int tokens, int experts, int top, int groups, int keep, float weight_eps, int mode, int group_max, cudaStream_t stream) {
    if (mode < 0 || mode > 2) return RV_ERR_UNSUPPORTED;
    if (tokens < 0 || experts <= 0 || top <= 0 || top > experts || groups <= 0 || experts % groups || keep <= 0 || keep > groups)
        return RV_ERR_BAD_SIZE;
    if (stride < experts + (gate_out ? 1 : 0) || top > (experts / groups) * keep) return RV_ERR_BAD_SIZE;
    if (experts > 1024) return RV_ERR_UNSUPPORTED;
    if (tokens == 0) return RV_OK;
    const size_t smem = (size_t)MR_WARPS * (2 * experts + groups) * sizeof(float);
    RV_LAUNCH_ST = rv_launch(moe_route_top_kernel, dim3((tokens + MR_WARPS - 1) / MR_WARPS), dim3(MR_WARPS * 32), smem, stream, logits,
                             stride, correction, chosen, weights, gate_out, tokens, experts, top, groups, keep, weight_eps, mode, group_max);
    return rv_launch_status();
}
