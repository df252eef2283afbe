// The gated delta rule of ssm.cu over long portions of bfloat16 rows, chunk by chunk.  With g_t the decays, G_t the product of a chunk's
// first t of them, D_ts the product of those behind s up to t, and S the state before the chunk,
//     u_t = beta_t (v_t - G_t S^T k_t - sum_{s < t} D_ts (k_t . k_s) u_s),     so   U = T beta (V - G K S),  T = (1 + beta D (K K^T))^-1
//     o_t = G_t S^T q_t + sum_{s <= t} D_ts (q_t . k_s) u_s
//     S   <- G_C S + sum_s D_Cs k_s u_s^T
// so that the chain from token to token runs through matrices of 16 x 16 that the state has no part in.  Token by token the walk of
// ssm.cu is one chain: a sum over the lanes, u, the state, 370 to 500 cycles a token, whatever stands idle beside it.
//
// Grid (blocks of 32 columns, heads, sequences).  Four warps hold the state as the walk does - a lane 8 of its rows by 4 columns, the
// rows in pairs for the packed multiply-adds - and take a chunk of 16 tokens at a time: sums of S with k and with q, four tokens at a
// time, dealt out to the lanes by a reduction of 15 shuffles (all independent); the small products with T and with M = D (Q K^T); the
// update.  Four others bring the next chunk: unit vectors, the products of the raw rows on the tensor cores (exact for bfloat16,
// each 16 elements from zero and added in float), the decays, T by substitution.  Everything that the state meets is float32.
// Bound by shared memory, which hands a lane k and q twice a chunk, about two thirds of the multiply-adds' rate.
#include "common.cuh"

#define DC 16                       // tokens of a chunk
#define DC_COLS 32                  // columns of a block
#define RAW_PITCH (128 + 8)         // elements between raw rows: eight rows of a column fall on different banks

__device__ __forceinline__ void dc_mma_new(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void dc_ldsm(uint32_t (&r)[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
typedef unsigned long long dc_pair;  // two floats
__device__ __forceinline__ dc_pair dc_pack(float lo, float hi) {
    dc_pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void dc_unpack(dc_pair v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ dc_pair dc_fma(dc_pair a, dc_pair b, dc_pair c) {
    dc_pair d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ dc_pair dc_mul(dc_pair a, dc_pair b) {
    dc_pair d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

template <int PARTS>
struct ChunkStage {
    static constexpr int ROW = PARTS * 12;                  // 8 elements a part, 12 floats apart: the reads of a token's parts fall on banks of their own
    float q[DC][ROW], k[DC][ROW];                           // unit vectors (q with its scale)
    float v[DC][DC_COLS];
    float T[DC][DC + 4], M[DC][DC + 4];                     // rows t; entries s > t are not read
    float decay[DC], beta[DC], left[DC];                    // G_t, beta_t, D_Cs
};
template <int PARTS>
struct ChunkShared {
    ChunkStage<PARTS> stage[2];
    __nv_bfloat16 raw_q[DC][RAW_PITCH], raw_k[DC][RAW_PITCH];
    float A[DC][DC + 4];
    float g[DC], scale_q[DC], scale_k[DC];
    float r[4][8][DC + 4], u[4][DC][8];                     // per walking warp: [column][token] and [token][column]
    float uc[4][8][DC + 4];
};

// 16 sums over 16 lanes, dealt out: lane p of the 16 gets sum number p.
__device__ __forceinline__ float dc_sum16_dealt(float (&v)[16], int p) {
#pragma unroll
    for (int h = 8; h > 0; h >>= 1) {
        const bool up = p & h;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float mine = up ? v[i + h] : v[i], theirs = up ? v[i] : v[i + h];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, h);
        }
    }
    return v[0];
}
__global__ void __launch_bounds__(256, 1)
delta_chunk_kernel(const __nv_bfloat16* __restrict__ qkv, int qkv_stride, const float* __restrict__ proj, int proj_stride, int b_col0, int a_col0,
                   const float* __restrict__ a_log, const float* __restrict__ dt_bias, const int* __restrict__ cu_seqlens,
                   const int* __restrict__ state_slots, float* __restrict__ state, size_t state_stride, float* __restrict__ out, int heads,
                   int qk_heads, int vd, float unit_eps, int least) {
    constexpr int PARTS = 16, D = 8 * PARTS;
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ __align__(16) unsigned char dc_raw[];
    ChunkShared<PARTS>& sm = *reinterpret_cast<ChunkShared<PARTS>*>(dc_raw);
    const int seq = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * DC_COLS;
    const int slot = state_slots[seq];
    if (slot < 0) return;
    const int start = cu_seqlens[seq], n_tok = cu_seqlens[seq + 1] - start;
    if (n_tok < least) return;                             // (ssm.cu's)
    const int chunks = (n_tok + DC - 1) / DC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 4) {                                        // ---- the state
        const int part = lane & 15, group = lane >> 4;
        const int cg = group * 4, cb = warp * 8 + cg, col = col0 + cb;         // (vd is a multiple of 4: a group's columns are all there or none)
        const bool live = col < vd;
        const int n0 = part * 8, to = part >> 2, mine = part & 3;              // after a reduction: token 4 q + to, column `mine` of the group's four
        dc_pair S[4][4];                                   // rows n0 + 2 i and n0 + 2 i + 1, column j
        float* srow = state + (size_t)slot * state_stride + (size_t)h * D * vd + col;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (live) {
                a = *reinterpret_cast<const float4*>(srow + (size_t)(n0 + 2 * i) * vd);
                b = *reinterpret_cast<const float4*>(srow + (size_t)(n0 + 2 * i + 1) * vd);
            }
            S[i][0] = dc_pack(a.x, b.x); S[i][1] = dc_pack(a.y, b.y); S[i][2] = dc_pack(a.z, b.z); S[i][3] = dc_pack(a.w, b.w);
        }
        auto row8 = [&](const float* p, dc_pair (&x)[4]) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p), b = *reinterpret_cast<const ulonglong2*>(p + 4);
            x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        };
        __syncthreads();                                   // the first chunk is staged
        for (int c = 0; c < chunks; ++c) {
            const ChunkStage<PARTS>& st = sm.stage[c & 1];
            // ---- S^T k and S^T q of the chunk's tokens: this lane keeps tokens 4 q + to of its column
            float w[4], z[4];
            auto sums = [&](const float (&rows)[DC][ChunkStage<PARTS>::ROW], float (&kept)[4]) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float v[16];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        dc_pair x[4];
                        row8(&rows[4 * q + t][part * 12], x);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            dc_pair s = dc_mul(S[0][j], x[0]);
#pragma unroll
                            for (int i = 1; i < 4; ++i) s = dc_fma(S[i][j], x[i], s);
                            float lo, hi;
                            dc_unpack(s, lo, hi);
                            v[4 * t + j] = lo + hi;
                        }
                    }
                    kept[q] = dc_sum16_dealt(v, part);
                }
            };
            sums(st.k, w);
            // ---- R = beta (v - G S^T k)
            float (&rc)[8][DC + 4] = sm.r[warp];
            float (&uc)[8][DC + 4] = sm.uc[warp];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int t = 4 * q + to;
                rc[cg + mine][t] = st.beta[t] * fmaf(-st.decay[t], w[q], st.v[t][cb + mine]);
            }
            __syncwarp();
            // a row of a lower triangle times a column: entries beyond the diagonal, and what they would meet, are not looked at
            auto lower = [&](const float (&rows)[DC][DC + 4], const float (&cols)[8][DC + 4], float (&acc)[4]) {
                float x[DC];
#pragma unroll
                for (int s = 0; s < DC; s += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(&cols[cg + mine][s]);
                    x[s] = v.x; x[s + 1] = v.y; x[s + 2] = v.z; x[s + 3] = v.w;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float a[2] = {0.f, 0.f};
#pragma unroll
                    for (int s4 = 0; s4 <= q; ++s4) {
                        const float4 v = *reinterpret_cast<const float4*>(&rows[4 * q + to][4 * s4]);
                        const float m[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int s = 0; s < 4; ++s)
                            if (s4 < q || s <= to) a[s & 1] = fmaf(m[s], x[4 * s4 + s], a[s & 1]);
                    }
                    acc[q] = a[0] + a[1];
                }
            };
            float u[4];
            lower(st.T, rc, u);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int t = 4 * q + to;
                uc[cg + mine][t] = u[q];
                sm.u[warp][t][cg + mine] = st.left[t] * u[q];
            }
            sums(st.q, z);
            __syncwarp();
            float o[4];
            lower(st.M, uc, o);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int t = c * DC + 4 * q + to;
                if (t < n_tok && live) out[((size_t)(start + t) * heads + h) * vd + col + mine] = fmaf(st.decay[4 * q + to], z[q], o[q]);
            }
            // ---- the state
            const float all = st.decay[DC - 1];
            const dc_pair all2 = dc_pack(all, all);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) S[i][j] = dc_mul(S[i][j], all2);
#pragma unroll
            for (int s = 0; s < DC; ++s) {
                dc_pair x[4];
                row8(&st.k[s][part * 12], x);
                const float4 uu = *reinterpret_cast<const float4*>(&sm.u[warp][s][cg]);
                const dc_pair u2[4] = {dc_pack(uu.x, uu.x), dc_pack(uu.y, uu.y), dc_pack(uu.z, uu.z), dc_pack(uu.w, uu.w)};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) S[i][j] = dc_fma(x[i], u2[j], S[i][j]);
            }
            __syncthreads();                               // this chunk is done, the next one staged
        }
        if (live) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float4 a, b;
                dc_unpack(S[i][0], a.x, b.x); dc_unpack(S[i][1], a.y, b.y); dc_unpack(S[i][2], a.z, b.z); dc_unpack(S[i][3], a.w, b.w);
                *reinterpret_cast<float4*>(srow + (size_t)(n0 + 2 * i) * vd) = a;
                *reinterpret_cast<float4*>(srow + (size_t)(n0 + 2 * i + 1) * vd) = b;
            }
        }
        return;
    }
    // ---- staging: a warp per token for q and k (four elements a lane), the block's columns of v, a thread per token for g and beta
    const int tid = threadIdx.x - 128, sw = warp - 4;
    const int kh = h / (heads / qk_heads), qk = qk_heads * D;
    const float q_scale = 1.0f / sqrtf((float)D);
    const float decay_rate = expf(a_log[h]), a_bias = dt_bias[h];
    uint2 pq[DC / 4], pk[DC / 4];
    unsigned short pv[DC * DC_COLS / 128];
    float pb = 0.f, pa = 0.f;
    auto load_chunk = [&](int c) {
        const int t0 = c * DC, nt = min(DC, n_tok - t0);
#pragma unroll
        for (int x = 0; x < DC / 4; ++x) {
            const int tt = sw + 4 * x;
            const __nv_bfloat16* row = qkv + (size_t)(start + t0 + tt) * qkv_stride + (size_t)kh * D + 4 * lane;
            pq[x] = pk[x] = make_uint2(0u, 0u);
            if (tt < nt) {
                pq[x] = *reinterpret_cast<const uint2*>(row);
                pk[x] = *reinterpret_cast<const uint2*>(row + qk);
            }
        }
#pragma unroll
        for (int y = 0; y < DC * DC_COLS / 128; ++y) {
            const int i = tid + 128 * y, tt = i / DC_COLS, cc = col0 + i % DC_COLS;
            pv[y] = 0;
            if (tt < nt && cc < vd) pv[y] = reinterpret_cast<const unsigned short*>(qkv)[(size_t)(start + t0 + tt) * qkv_stride + 2 * qk + (size_t)h * vd + cc];
        }
        if (tid < nt) {
            const size_t row = (size_t)(start + t0 + tid) * proj_stride;
            pb = proj[row + b_col0 + h];
            pa = proj[row + a_col0 + h];
        }
    };
    auto low = [](uint32_t v) { return __uint_as_float(v << 16); };
    auto high = [](uint32_t v) { return __uint_as_float(v & 0xffff0000u); };
    const int mi = lane >> 3, mr = lane & 7;               // ldmatrix: this lane's matrix and row
    auto stage = [&](int c) {
        ChunkStage<PARTS>& st = sm.stage[c & 1];
        const int nt = min(DC, n_tok - c * DC);
        float sq[DC / 4], sk[DC / 4];
#pragma unroll
        for (int x = 0; x < DC / 4; ++x) {                 // (beyond the sequence: zeros)
            const float q0 = low(pq[x].x), q1 = high(pq[x].x), q2 = low(pq[x].y), q3 = high(pq[x].y);
            const float k0 = low(pk[x].x), k1 = high(pk[x].x), k2 = low(pk[x].y), k3 = high(pk[x].y);
            sq[x] = fmaf(q3, q3, fmaf(q2, q2, fmaf(q1, q1, q0 * q0)));
            sk[x] = fmaf(k3, k3, fmaf(k2, k2, fmaf(k1, k1, k0 * k0)));
            *reinterpret_cast<uint2*>(&sm.raw_q[sw + 4 * x][4 * lane]) = pq[x];
            *reinterpret_cast<uint2*>(&sm.raw_k[sw + 4 * x][4 * lane]) = pk[x];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int x = 0; x < DC / 4; ++x) {
                sq[x] += __shfl_xor_sync(0xffffffffu, sq[x], o);
                sk[x] += __shfl_xor_sync(0xffffffffu, sk[x], o);
            }
#pragma unroll
        for (int x = 0; x < DC / 4; ++x) {
            const int tt = sw + 4 * x, at = (lane >> 1) * 12 + (lane & 1) * 4;
            const float rq = tt < nt ? q_scale / sqrtf(sq[x] + unit_eps) : 0.f, rk = tt < nt ? 1.0f / sqrtf(sk[x] + unit_eps) : 0.f;
            if (lane == 0) { sm.scale_q[tt] = rq; sm.scale_k[tt] = rk; }
            *reinterpret_cast<float4*>(&st.q[tt][at]) = make_float4(low(pq[x].x) * rq, high(pq[x].x) * rq, low(pq[x].y) * rq, high(pq[x].y) * rq);
            *reinterpret_cast<float4*>(&st.k[tt][at]) = make_float4(low(pk[x].x) * rk, high(pk[x].x) * rk, low(pk[x].y) * rk, high(pk[x].y) * rk);
        }
#pragma unroll
        for (int y = 0; y < DC * DC_COLS / 128; ++y) st.v[(tid + 128 * y) / DC_COLS][(tid + 128 * y) % DC_COLS] = __uint_as_float((uint32_t)pv[y] << 16);
        if (tid < DC) {                                    // (beyond the sequence: nothing decays and nothing is written)
            const float a = pa + a_bias;
            const float sp = a > 20.f ? a : log1pf(expf(a));
            st.beta[tid] = tid < nt ? 1.0f / (1.0f + expf(-pb)) : 0.f;
            sm.g[tid] = tid < nt ? expf(-decay_rate * sp) : 1.f;
        }
        asm volatile("bar.sync 2, 128;" ::: "memory");
        if (sw >= 2) return;
        // ---- one warp: A = beta D (K K^T) below the diagonal and T; the other: M = D (Q K^T) up to the diagonal, and the decays
        float P[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) P[n][0] = P[n][1] = P[n][2] = P[n][3] = 0.f;
        const __nv_bfloat16 (&left)[DC][RAW_PITCH] = sw == 0 ? sm.raw_k : sm.raw_q;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            uint32_t a[4], b[4];
            dc_ldsm(a, &left[(mi & 1) * 8 + mr][kk * 16 + (mi >> 1) * 8]);
            dc_ldsm(b, &sm.raw_k[(mi >> 1) * 8 + mr][kk * 16 + (mi & 1) * 8]);
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                float p[4];
                dc_mma_new(p, a, b[2 * n], b[2 * n + 1]);
#pragma unroll
                for (int j = 0; j < 4; ++j) P[n][j] += p[j];
            }
        }
        // lane s of each half walks D_ts down its column (t from s on); the products of an entry are picked up by the lanes that hold it
        const int s16 = lane & 15;
        float run = 1.f, all = 1.f;
        float (&to_rows)[DC][DC + 4] = sw == 0 ? sm.A : st.M;
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            const float g = sm.g[t];
            if (t > s16) run *= g;
            all *= g;
            if (lane < 16) to_rows[t][s16] = run;          // D_ts (t >= s)
            if (sw == 1 && lane == 0) st.decay[t] = all;
        }
        if (sw == 1 && lane < 16) st.left[s16] = run;
        __syncwarp();
        const int r0 = lane >> 2, c0 = 2 * (lane & 3);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = r0 + 8 * (j >> 1), s = 8 * n + c0 + (j & 1);
                if (s > t) continue;
                const float e = to_rows[t][s] * (P[n][j] * (sw == 0 ? sm.scale_k[t] * st.beta[t] : sm.scale_q[t]) * sm.scale_k[s]);
                to_rows[t][s] = e;
            }
        if (sw == 1) return;
        __syncwarp();
        // T: column s of (1 + A)^-1, row by row
        float x[DC];
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            float acc[2] = {t == s16 ? 1.f : 0.f, 0.f};
#pragma unroll
            for (int s = 0; s < t; ++s) acc[s & 1] = fmaf(-sm.A[t][s], x[s], acc[s & 1]);
            x[t] = acc[0] + acc[1];
            if (lane < 16) st.T[t][s16] = x[t];
        }
    };
    if (chunks > 0) { load_chunk(0); stage(0); }
    if (chunks > 1) load_chunk(1);
    __syncthreads();
    for (int c = 0; c < chunks; ++c) {                     // while chunk c is at work: c + 1 in, c + 2 on its way
        if (c + 1 < chunks) {
            stage(c + 1);
            if (c + 2 < chunks) load_chunk(c + 2);
        }
        __syncthreads();
    }
}

// Arguments as of rv_delta_rule (ssm.cu), qkv bfloat16; sequences of fewer than `least` tokens are left alone.  RV_ERR_UNSUPPORTED for what
// the kernel does not serve: keys of other than 128 elements, rows and states that are not whole words of four.
RV_EXPORT int rv_delta_chunk(const void* qkv, int qkv_stride, const float* proj, int proj_stride, int b_col0, int a_col0, const float* a_log,
                             const float* dt_bias, const int* cu_seqlens, const int* state_slots, float* state, long long state_stride, float* out,
                             int n_seqs, int heads, int qk_heads, int d, int vd, float unit_eps, int least, cudaStream_t stream) {
    if (n_seqs < 0 || heads <= 0 || qk_heads <= 0 || heads % qk_heads || d <= 0 || vd <= 0 || n_seqs > 65535 || heads > 65535) return RV_ERR_BAD_SIZE;
    if (qkv_stride < 2 * qk_heads * d + heads * vd || b_col0 < 0 || a_col0 < 0 || b_col0 + heads > proj_stride || a_col0 + heads > proj_stride ||
        state_stride < (long long)heads * d * vd)
        return RV_ERR_BAD_SIZE;
    if (d != 128 || vd % 4 || qkv_stride % 4 || state_stride % 4 || (reinterpret_cast<uintptr_t>(qkv) & 7) || (reinterpret_cast<uintptr_t>(state) & 15))
        return RV_ERR_UNSUPPORTED;
    if (n_seqs == 0) return RV_OK;
    constexpr int smem = (int)sizeof(ChunkShared<16>);
    static RvPerDevice once;
    if (int st = rv_configure_smem(once, delta_chunk_kernel, smem)) return st;
    RV_LAUNCH_ST = rv_launch(delta_chunk_kernel, dim3((vd + DC_COLS - 1) / DC_COLS, heads, n_seqs), dim3(256), smem, stream, (const __nv_bfloat16*)qkv,
                             qkv_stride, proj, proj_stride, b_col0, a_col0, a_log, dt_bias, cu_seqlens, state_slots, state, (size_t)state_stride,
                             out, heads, qk_heads, vd, unit_eps, least);
    return rv_launch_status();
}
