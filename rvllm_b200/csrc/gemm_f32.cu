// True 32-bit linear layer: out[M, N] = x[M, K] . W[N, K]^T (+ bias[N]) (+ residual[M, N]).
// Plain FFMA on the CUDA cores: no tensor-core instruction is used, so no operand is ever
// rounded to TF32.  Any M, N, K.
//
// One order of summation for every M, so that a row's result is bitwise the same whatever else is in
// the batch and whichever kernel serves it: K is cut into at most 16 segments of equal length (a
// multiple of 32), each segment is one chain of FMAs in ascending k from zero, four consecutive
// segments are added in order, and the four groups as (g0 + g1) + (g2 + g3).  Then bias, then residual.
//
//   gemm_f32_stream_kernel   up to 32 rows (more in blocks of 32 where the product is small): bound by the stream of weights.  A CTA takes 16 rows of W whole;
//                            each half warp walks one segment, a lane one row of W, against all rows of x,
//                            from a ring of warp-private stages that cp.async fills (no CTA barrier in the loop;
//                            the first weights are asked for before griddepcontrol.wait).
//   gemm_f32_tile_kernel     more rows: bound by the FMA rate.  128 x 128 tiles, 8 x 8 outputs a thread with packed
//                            two-float FMAs, the groups of segments dealt out to a cluster of 1, 2 or 4 CTAs where
//                            the tiles alone would leave SMs idle.
//
// Measured against one 64 x 64 tile kernel for every M (4 x 4 outputs a thread), which this replaced: 3 rows of 3584 x 18944
// 2,120 -> 72 us (3.8 TB/s), of 37888 x 3584 836 -> 105 us (5.2 TB/s), of 152064 x 3584 3,235 -> 349 us (6.2 TB/s); 433 rows of
// 37888 x 3584 5,381 -> 2,803 us (42 TFLOP/s; the loop over shared memory with nothing brought there reaches 61); error against float64 1.1e-6 -> 2.7e-7 (2-norms, K = 3,584).
//
// Shapes of the layer's five products: v3/crates/rvllm-runtime/src/layer_exec.rs:240-266,
// 433-444, 478-488, 511-522 of the reference (which calls cuBLASLt there); bias as a row
// broadcast and the residual as beta = 1 follow cublaslt.rs:335-368.
#include "common.cuh"

#define MAX_SEGMENTS 16

__host__ __device__ __forceinline__ int segment_length(int K) { return ((K + 32 * MAX_SEGMENTS - 1) / (32 * MAX_SEGMENTS)) * 32; }

// ------------------------------------------------------------------------------------- few rows: the stream of weights
#define ST_K 32                 // k per stage: 128 bytes of a row, eight 16-byte chunks
#define ST_WARPS 8

__device__ __forceinline__ void cp_async_16(void* dst, const void* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 16 : 0;                       // 0: the destination is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void cp_async_4(void* dst, const void* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(d), "l"(src), "r"(bytes) : "memory");
}

// MB: rows of x (padded); stages are per half warp: [16 rows of W | MB rows of x] x 128 bytes,
// the chunk c of row r at place c ^ (r & 7) (16 lanes on one chunk of 16 rows meet no bank twice).
template <int MB, int STAGES>
__global__ void __launch_bounds__(ST_WARPS * 32)
gemm_f32_stream_kernel(const float* __restrict__ x, const float* __restrict__ w, const void* __restrict__ bias,
                       int bias_dtype, const float* __restrict__ residual, float* __restrict__ out,
                       int M, int N, int K) {
    extern __shared__ __align__(128) float smem[];
    if (blockIdx.y) {                                       // (rows beyond the first MB)
        const size_t m0 = (size_t)blockIdx.y * MB;
        x += m0 * K;
        out += m0 * N;
        if (residual) residual += m0 * N;
        M -= (int)m0;
    }
    constexpr int WROWS = 16;
    constexpr int STAGE = (WROWS + MB) * ST_K;              // floats of a half warp's stage
    const int tid = threadIdx.x, half = tid >> 4, l16 = tid & 15;
    const int n0 = blockIdx.x * WROWS;
    const int seg = segment_length(K);
    const int k_begin = half * seg, k_end = min(K, k_begin + seg);
    const int steps = seg / ST_K;                           // the same for all half warps: a segment past K reads zeros
    float* ring = smem + (size_t)half * STAGES * STAGE;
    const int chunk = l16 & 7, row_of = l16 >> 3;           // a half warp copies two rows of 128 bytes at a time
    const int turn = (half & 1) << 2;                       // x of a warp's two halves lies in different banks

    auto load_w = [&](int s) {
        float* st = ring + (s % STAGES) * STAGE;
        const int k = k_begin + s * ST_K + chunk * 4;
#pragma unroll
        for (int r = 0; r < WROWS; r += 2) {
            const int row = r + row_of, n = n0 + row;
            const bool ok = k < k_end && n < N;
            cp_async_16(st + row * ST_K + ((chunk ^ (row & 7)) << 2), ok ? w + (size_t)n * K + k : w, ok);
        }
    };
    auto load_x = [&](int s) {
        float* st = ring + (s % STAGES) * STAGE + WROWS * ST_K;
        const int k = k_begin + s * ST_K + chunk * 4;
#pragma unroll
        for (int r = 0; r < MB; r += 2) {
            const int row = r + row_of;
            if (MB == 1 && row_of) continue;
            const bool ok = k < k_end && row < M;
            cp_async_16(st + row * ST_K + ((chunk ^ turn) << 2), ok ? x + (size_t)row * K + k : x, ok);
        }
    };
    rv_pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
        if (s < steps) load_w(s);
    rv_pdl_wait();
    // the weights of the first stages and their x are one group for the first of them, so stage 0 waits for all
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load_x(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[MB];
#pragma unroll
    for (int m = 0; m < MB; ++m) acc[m] = 0.f;

    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 2) : "memory");
        __syncwarp();                                       // the half warps' stages are filled by the lanes of their own warp
        if (s + STAGES - 1 < steps) { load_w(s + STAGES - 1); load_x(s + STAGES - 1); }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* ws = ring + (s % STAGES) * STAGE;
        const float* xs = ws + WROWS * ST_K;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float4 wv = *reinterpret_cast<const float4*>(ws + l16 * ST_K + ((c ^ (l16 & 7)) << 2));
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                const float4 xv = *reinterpret_cast<const float4*>(xs + m * ST_K + ((c ^ turn) << 2));
                acc[m] = fmaf(xv.x, wv.x, acc[m]);
                acc[m] = fmaf(xv.y, wv.y, acc[m]);
                acc[m] = fmaf(xv.z, wv.z, acc[m]);
                acc[m] = fmaf(xv.w, wv.w, acc[m]);
            }
        }
        __syncwarp();                                       // read before the next turn's copies overwrite the oldest stage
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the segments' sums meet in shared memory: [segment][m][row of W]
#pragma unroll
    for (int m = 0; m < MB; ++m) smem[(half * MB + m) * WROWS + l16] = acc[m];
    __syncthreads();
    for (int i = tid; i < MB * WROWS; i += ST_WARPS * 32) {
        const int m = i / WROWS, n = n0 + i % WROWS;
        if (m >= M || n >= N) continue;
        float g[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            g[q] = smem[(4 * q) * MB * WROWS + i];
#pragma unroll
            for (int j = 1; j < 4; ++j) g[q] += smem[(4 * q + j) * MB * WROWS + i];
        }
        float v = (g[0] + g[1]) + (g[2] + g[3]);
        if (bias) v += rv_load_param(bias, bias_dtype, n);
        if (residual) v += residual[(size_t)m * N + n];
        out[(size_t)m * N + n] = v;
    }
}

template <int MB, int STAGES>
static int launch_stream(const float* x, const float* w, const void* bias, int bias_dtype, const float* residual, float* out,
                         int M, int N, int K, cudaStream_t stream) {
    constexpr int ring = MAX_SEGMENTS * STAGES * (16 + MB) * ST_K * 4;
    static_assert(ring >= MAX_SEGMENTS * MB * 16 * 4, "the sums fit the ring");
    static RvPerDevice configured;
    if (int st = rv_configure_smem(configured, gemm_f32_stream_kernel<MB, STAGES>, ring)) return st;
    return rv_launch(gemm_f32_stream_kernel<MB, STAGES>, dim3((N + 15) / 16, (M + MB - 1) / MB), dim3(ST_WARPS * 32), ring, stream,
                     x, w, bias, bias_dtype, residual, out, M, N, K);
}

// ------------------------------------------------------------------------------------------ many rows: the FMA rate
#define TB 128                  // tile rows and columns
#define TK 16
#define TPITCH (TB + 4)         // floats between k rows: k and k + 4 lie 16 banks apart

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// blockIdx.x = tile * splits + part (the parts of a tile form a cluster), tile = column tile * row tiles + row tile: the CTAs
// that share rows of W run side by side (column tiles first, W came from memory once per row tile, and the way of
// a tile from there was longer than the work on one).  Part p of S walks the segments of groups p * 4 / S .. (p + 1) * 4 / S - 1.
template <bool VEC>
__global__ void __launch_bounds__(256, 1)
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, const void* __restrict__ bias,
                     int bias_dtype, const float* __restrict__ residual, float* __restrict__ out,
                     int M, int N, int K, int splits, int row_tiles) {
    extern __shared__ __align__(128) float smem[];           // two stages of xs | ws [TK][TPITCH], two parked groups, two stages of words
                                                            // on their way from memory; later a part's sums [128][TPITCH]
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = blockIdx.x % splits, tile = blockIdx.x / splits;
    const int m0 = (tile % row_tiles) * TB, n0 = (tile / row_tiles) * TB;
    // a warp covers 32 x 64 outputs (4 x 8 lanes of 8 x 8, as two halves of 4 each way); the two warps of a scheduler lie 64 rows
    // apart, so a last row tile of up to 64 rows takes half the time
    const int wm = (warp >> 2) * 64 + (warp & 1) * 32, wn = ((warp >> 1) & 1) * 64;
    const bool active = m0 + wm < M;
    const int am = wm + (lane >> 3) * 4, bn = wn + (lane & 7) * 4;       // and +16 rows, +32 columns
    const int seg = segment_length(K), per = MAX_SEGMENTS / splits;
    const int k_first = part * per * seg, k_last = min(K, k_first + per * seg);

    // two lanes bring 8 consecutive k of a row: whole 32-byte sectors in, conflict-free columns out
    const int ld_row = (warp >> 1) * 16 + (lane >> 1) , ld_k = (warp & 1) * 8 + (lane & 1) * 4;      // rows +0, +64
    // the words wait in shared memory, each in its thread's own places ([stage][4][256 threads] x 16 bytes), until the thread puts
    // them down by column: in registers the compiler moved the loads to where they are used, and a fifth of the time
    // was spent waiting for them
    float4* mail = reinterpret_cast<float4*>(smem + 4 * TK * TPITCH + 2 * 64 * 256);
    auto fetch = [&](int t) {
        const int k = k_first + t * TK + ld_k;
        float4* to = mail + (t & 1) * 4 * 256 + tid;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + ld_row + h * 64, n = n0 + ld_row + h * 64;
            const float* px = x + (size_t)m * K + k;
            const float* pw = w + (size_t)n * K + k;
            if (VEC) {
                const bool okx = m < M && k < k_last, okw = n < N && k < k_last;
                cp_async_16(to + h * 256, okx ? px : x, okx);
                cp_async_16(to + (2 + h) * 256, okw ? pw : w, okw);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool okx = m < M && k + j < k_last, okw = n < N && k + j < k_last;
                    cp_async_4(reinterpret_cast<float*>(to + h * 256) + j, okx ? px + j : x, okx);
                    cp_async_4(reinterpret_cast<float*>(to + (2 + h) * 256) + j, okw ? pw + j : w, okw);
                }
            }
        }
    };
    auto store = [&](int t, int i) {                         // one of the thread's four words of tile t: x for i < 2, w for the others
        float* to = smem + ((t & 1) * 2 + (i >> 1)) * TK * TPITCH + ld_k * TPITCH + ld_row + (i & 1) * 64;
        const float4 v = mail[(t & 1) * 4 * 256 + tid + i * 256];
        to[0] = v.x; to[TPITCH] = v.y; to[2 * TPITCH] = v.z; to[3 * TPITCH] = v.w;
    };

    // acc: the running segment; group: the running group of four; total: the groups of this part (all packed column pairs)
    unsigned long long acc[8][4];
    float total[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) { acc[i][j] = 0ull; total[i][2 * j] = total[i][2 * j + 1] = 0.f; }
    const int n_tiles = k_first < k_last ? (k_last - k_first + TK - 1) / TK : 0;
    const int seg_tiles = seg / TK;
    if (n_tiles) fetch(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (n_tiles > 1) fetch(1);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
    if (n_tiles) { store(0, 0); store(0, 1); store(0, 2); store(0, 3); }
    __syncthreads();
    int in_seg = 0, seg_i = 0;
    // the sums of a tile: groups of four segments; the first group's sum waits in shared memory behind the stages while the
    // second of a pair is formed (a part of four groups does that twice, and once more for the pairs)
    float* park = smem + 4 * TK * TPITCH;                   // [2][64 values][256 threads]
    for (int t = 0; t < n_tiles; ++t) {
        const int buf = t & 1;
        if (t + 2 < n_tiles) fetch(t + 2);                  // (its places were read, by this thread, before the last barrier)
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
        const float* xs = smem + buf * 2 * TK * TPITCH;
        const float* ws = xs + TK * TPITCH;
        const bool more = t + 1 < n_tiles;
        auto products = [&](int k) {
            const float4 a0 = *reinterpret_cast<const float4*>(xs + k * TPITCH + am);
            const float4 a1 = *reinterpret_cast<const float4*>(xs + k * TPITCH + am + 16);
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(ws + k * TPITCH + bn);
            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(ws + k * TPITCH + bn + 32);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const unsigned long long b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long aa = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) fma2(acc[i][j], aa, b[j]);
            }
        };
        // the next tile's words go to their columns between the products (the other stage has not been read since the last barrier);
        // behind them, with every warp at it and the multiply-adds idle, they took 4 to 5 % of the time
        if (active && more) {
#pragma unroll
            for (int k = 0; k < TK; ++k) {
                products(k);
                if ((k & 3) == 3) store(t + 1, k >> 2);
            }
        } else if (active) {
#pragma unroll
            for (int k = 0; k < TK; ++k) products(k);
        } else if (more) {
            store(t + 1, 0); store(t + 1, 1); store(t + 1, 2); store(t + 1, 3);
        }
        if (++in_seg == seg_tiles || t + 1 == n_tiles) {    // a segment is done
            in_seg = 0;
            const bool first = (seg_i & 3) == 0;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float lo, hi;
                    unpack2(acc[i][j], lo, hi);
                    total[i][2 * j] = first ? lo : total[i][2 * j] + lo;
                    total[i][2 * j + 1] = first ? hi : total[i][2 * j + 1] + hi;
                    acc[i][j] = 0ull;
                }
            ++seg_i;
            if ((seg_i & 3) == 0 || t + 1 == n_tiles) {     // a group is done: even ones wait, odd ones join the one before
                const int g = (seg_i - 1) >> 2;
                if (g & 1) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) total[i][j] = park[(i * 8 + j) * 256 + tid] + total[i][j];
                }
                if (g == 3) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) total[i][j] = park[(64 + i * 8 + j) * 256 + tid] + total[i][j];
                } else if (t + 1 < n_tiles) {
                    float* p = park + (g == 1 ? 64 * 256 : 0);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) p[(i * 8 + j) * 256 + tid] = total[i][j];
                } else if (g == 2) {                        // K ends within the third group: (g0 + g1) + g2
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) total[i][j] = park[(64 + i * 8 + j) * 256 + tid] + total[i][j];
                }
            }
        }
        __syncthreads();
    }

    if (splits == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int m = m0 + am + (i & 3) + (i >> 2) * 16;
            if (m >= M) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int n = n0 + bn + (j & 3) + (j >> 2) * 32;
                if (n >= N) continue;
                float v = total[i][j];
                if (bias) v += rv_load_param(bias, bias_dtype, n);
                if (residual) v += residual[(size_t)m * N + n];
                out[(size_t)m * N + n] = v;
            }
        }
        return;
    }
    // the parts' sums through the cluster's shared memory: part p finishes rows p * 128 / splits .. of the tile
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            *reinterpret_cast<float4*>(smem + (am + (i & 3) + (i >> 2) * 16) * TPITCH + bn + h * 32) =
                make_float4(total[i][4 * h], total[i][4 * h + 1], total[i][4 * h + 2], total[i][4 * h + 3]);
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
    const int rows = TB / splits;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    for (int i = tid; i < rows * (TB / 4); i += 256) {
        const int row = part * rows + i / (TB / 4), col = (i % (TB / 4)) * 4;
        float4 g[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            if (p >= splits) break;
            uint32_t addr;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(base + (uint32_t)(row * TPITCH + col) * 4u), "r"(p));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(g[p].x), "=f"(g[p].y), "=f"(g[p].z), "=f"(g[p].w) : "r"(addr) : "memory");
        }
        const int m = m0 + row;
        if (m >= M) continue;
        float v[4] = {g[0].x + g[1].x, g[0].y + g[1].y, g[0].z + g[1].z, g[0].w + g[1].w};
        if (splits == 4) {
            v[0] += g[2].x + g[3].x; v[1] += g[2].y + g[3].y; v[2] += g[2].z + g[3].z; v[3] += g[2].w + g[3].w;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + col + j;
            if (n >= N) continue;
            float r = v[j];
            if (bias) r += rv_load_param(bias, bias_dtype, n);
            if (residual) r += residual[(size_t)m * N + n];
            out[(size_t)m * N + n] = r;
        }
    }
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");   // no CTA leaves while others read it
}

RV_EXPORT int rv_gemm_f32(const float* x, const float* w, const void* bias, int bias_dtype,
                          const float* residual, float* out, int M, int N, int K, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0) return RV_ERR_BAD_SIZE;
    if (M == 0) return RV_OK;
    const bool vec = (K & 3) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    // Up to 32 rows the weights' stream is the longer side (8 rows) or level with the FMAs (32); beyond, W would be
    // read once per 32 rows.  The ring needs rows of whole 16-byte words.  Products of up to 512 k (one step of the ring) whose
    // blocks of 32 rows are one CTA an SM at most are all latency, of which a tile has more (64 rows of 64 x 64: 9.0 us).
    const bool small = K <= ST_K * MAX_SEGMENTS && (long long)((N + 15) / 16) * ((M + 31) / 32) <= rv_sm_count();
    if (vec && (M <= 32 || small)) {
        int st;
        if (M == 1) st = launch_stream<1, 3>(x, w, bias, bias_dtype, residual, out, M, N, K, stream);
        else if (M == 2) st = launch_stream<2, 3>(x, w, bias, bias_dtype, residual, out, M, N, K, stream);
        else if (M <= 4) st = launch_stream<4, 2>(x, w, bias, bias_dtype, residual, out, M, N, K, stream);
        else if (M <= 8) st = launch_stream<8, 2>(x, w, bias, bias_dtype, residual, out, M, N, K, stream);
        else if (M <= 16) st = launch_stream<16, 3>(x, w, bias, bias_dtype, residual, out, M, N, K, stream);
        else st = launch_stream<32, 2>(x, w, bias, bias_dtype, residual, out, M, N, K, stream);
        RV_LAUNCH_ST = st;
        return rv_launch_status();
    }
    const long long rows = (M + TB - 1) / TB, cols = (N + TB - 1) / TB;
    if (rows * cols > 0x7fffffffll / 4) return RV_ERR_BAD_SIZE;
    // K over a cluster of 1, 2 or 4 CTAs (one per SM): the fewest rounds of work, counted in a whole tile's time (a last row tile of
    // up to 64 rows is half of one), and of ones within a twentieth the fewest parts.  433 rows of 3584 x 18944, 112 tiles: one round of
    // 1,913 us whole, 1,734 in parts of four; 300 of 4095 x 1023 146 and 119.
    const int sms = rv_sm_count();
    const long long halves = cols * (2 * rows - (M - (rows - 1) * TB <= TB / 2 ? 1 : 0));
    int splits = 1;
    for (int s = 2; s <= 4; s *= 2)
        if ((halves * s + 2 * sms - 1) / (2 * sms) * splits * 20 < (halves * splits + 2 * sms - 1) / (2 * sms) * s * 19) splits = s;
    const int smem = (4 * TK * TPITCH + 2 * 64 * 256) * 4 + 2 * 4 * 256 * 16;       // stages, two parked groups (>= a part's sums), words on their way
    static_assert(4 * TK * TPITCH + 2 * 64 * 256 >= TB * TPITCH, "a part's sums fit");
    static RvPerDevice conf_v, conf_s;
    const dim3 grid((unsigned)(rows * cols * splits));
    if (vec) {
        if (int st = rv_configure_smem(conf_v, gemm_f32_tile_kernel<true>, smem)) return st;
        RV_LAUNCH_ST = splits == 1 ? rv_launch(gemm_f32_tile_kernel<true>, grid, dim3(256), smem, stream, x, w, bias, bias_dtype, residual, out, M, N, K, splits, (int)rows)
                                   : rv_launch_cluster(gemm_f32_tile_kernel<true>, grid, dim3(256), smem, stream, splits, x, w, bias, bias_dtype, residual, out, M, N, K, splits, (int)rows);
    } else {
        if (int st = rv_configure_smem(conf_s, gemm_f32_tile_kernel<false>, smem)) return st;
        RV_LAUNCH_ST = splits == 1 ? rv_launch(gemm_f32_tile_kernel<false>, grid, dim3(256), smem, stream, x, w, bias, bias_dtype, residual, out, M, N, K, splits, (int)rows)
                                   : rv_launch_cluster(gemm_f32_tile_kernel<false>, grid, dim3(256), smem, stream, splits, x, w, bias, bias_dtype, residual, out, M, N, K, splits, (int)rows);
    }
    return rv_launch_status();
}
