// The selective-state recurrence of ssm.cu over long portions of bfloat16 rows, chunk by chunk on the tensor cores.  With
// a_t = -exp(A_log_h) dt_t, c_t the running sum of a from the chunk's first token on, and S the state before the chunk,
//     y_t   = e^(c_t) S^T C_t + sum_{s <= t} (C_t . B_s) e^(c_t - c_s) dt_s x_s + D_h x_t
//     S_new = e^(c_L) S + sum_s (e^(c_L - c_s) dt_s) B_s x_s^T
// which is four products per chunk of 64 tokens instead of 64 dependent updates of the whole state: 2,048 tokens of 128 heads
// of 64 x 128 take 330 us in place of 1,040, portions of 1,228 and 820 tokens 227 in place of 713.
//
// x, B and C are bfloat16 as they come, so products among them are exact; the float factors (the state, the weighted
// scores, the weighted x) go in as three bfloat16 terms each (24 bits: v = hi + mid + lo), so nothing is rounded below
// float.  The running sums c are formed in double and kept as two floats, so a difference of two of them is as exact as
// a sum of the few terms between; an exponential makes up for its argument's rounding.  The tensor cores cut sums off where float
// rounds them: products of leading terms start from zero and are added in float.  Against float64 (2-norms, decays of dt 0.001
// to 0.1, rates 1 to 16): y 0.9e-7, state 0.8e-7 to 1.3e-7; the walk 1.4e-7 to 7e-7 and 1.4e-7 to 2e-6.  With one accumulator for
// all terms and plain exponentials they were 1.8e-7 to 4.6e-7 and up to 8.6e-7, above the walk's for some heads, in 296 us.
//
// A product multiplies the masked zeros of a block of scores with the x of later tokens, infinities do not split into terms, and
// a running sum that a single step size dominates does not tell the others' decays any more.  So a chunk with numbers that
// are not finite, or with a sum of decays beyond 10^5, is walked token by token, as ssm.cu does (the columns of a warp where it
// is an x or the state, else the whole block): what is not finite stays with its token and those after it.
//
// Grid (blocks of 64 columns p, heads, sequences), four warps, one per 16 columns: S^T of them (16 x N) lives in the
// accumulators' layout in registers, which is also the layout of an A operand, so y needs no pass of S through shared
// memory.  The scores of a chunk are formed by all four warps (16 tokens each) and meet in shared memory as their three
// terms.  The next chunk's rows are on their way (cp.async) while a chunk is computed.
#include "common.cuh"

#define CH 64                    // tokens of a chunk
#define XP (64 + 8)              // elements between rows of x and of the scores: 16-byte rows fall on different banks

__device__ __forceinline__ void ch_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same from zero: the tensor cores cut their sums off, they do not round them, so the products of leading terms are kept from
// running through one accumulator and added in float.
__device__ __forceinline__ void ch_mma_new(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void ch_mma_add(float (&sum)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    float c[4];
    ch_mma_new(c, a, b0, b1);
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[j] += c[j];
}
// e^v of a double as a float, to float's last place: the argument's own rounding is made up for
__device__ __forceinline__ float ch_exp(double v) {
    const float hi = (float)v, e = expf(hi);
    return fmaf(e, (float)(v - (double)hi), e);
}
__device__ __forceinline__ void ch_ldsm(uint32_t (&r)[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ch_ldsm_t(uint32_t (&r)[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ uint32_t ch_pack(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float ch_low(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float ch_high(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// two floats as three pairs of bfloat16 whose sums are the floats (to the last bit or two of a float)
__device__ __forceinline__ void ch_split(float a, float b, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
    t0 = ch_pack(a, b);
    a -= ch_low(t0); b -= ch_high(t0);
    t1 = ch_pack(a, b);
    a -= ch_low(t1); b -= ch_high(t1);
    t2 = ch_pack(a, b);
}
__device__ __forceinline__ void ch_copy16(void* dst, const void* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ float ch_any(const void* p, int dtype, size_t i) {
    return dtype == RV_DTYPE_F32 ? ((const float*)p)[i] : __bfloat162float(((const __nv_bfloat16*)p)[i]);
}

template <int N>
struct ChunkSmem {
    __nv_bfloat16 b[2][CH][N];      // the 16-byte word w of row t at place w ^ (t & 7): a column of eight rows meets no bank twice
    __nv_bfloat16 c[2][CH][N];
    __nv_bfloat16 x[2][CH][XP];
    __nv_bfloat16 m[3][CH][XP];     // the chunk's weighted scores [t][s], three terms
    float dt[CH], cum[CH], cum_lo[CH], decay[CH], weight[CH];        // e^(c_t); e^(c_L - c_s) dt_s
    double part[2];
    float last;                                                       // e^(c_L)
};

template <int N>
__device__ __forceinline__ __nv_bfloat16* ch_word(__nv_bfloat16 (&rows)[CH][N], int t, int w) { return &rows[t][(w ^ (t & 7)) * 8]; }

template <int N>
__global__ void __launch_bounds__(128, 2)
ssm_chunk_kernel(const __nv_bfloat16* __restrict__ xbc, int channels, const void* __restrict__ dt_in, int dt_dtype, int dt_stride, int dt_col0,
                 const void* __restrict__ dt_bias, const void* __restrict__ a_log, const void* __restrict__ d_skip, int p_dtype,
                 const int* __restrict__ cu_seqlens, const int* __restrict__ state_slots, float* __restrict__ state,
                 size_t state_stride, float* __restrict__ y, int heads, int P, int groups, int least) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    extern __shared__ __align__(16) unsigned char ch_raw[];
    ChunkSmem<N>& sm = *reinterpret_cast<ChunkSmem<N>*>(ch_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int seq = blockIdx.z, h = blockIdx.y, p0 = blockIdx.x * 64;
    const int start = cu_seqlens[seq], n_tok = cu_seqlens[seq + 1] - start;
    if (n_tok < least) return;                             // (ssm.cu's)
    const int slot = state_slots[seq];
    const int inner = heads * P, cols = min(64, P - p0);
    if (slot < 0) {                                        // a padding row: no state; its output is zero
        for (int i = tid; i < n_tok * cols; i += 128) y[(size_t)(start + i / cols) * inner + h * P + p0 + i % cols] = 0.f;
        return;
    }
    if (n_tok <= 0) return;
    const float A = -expf(rv_load_param(a_log, p_dtype, h));
    const float bias = rv_load_param(dt_bias, p_dtype, h);
    const float Dh = rv_load_param(d_skip, p_dtype, h);
    const int group = h / (heads / groups);
    const size_t b_col = (size_t)inner + (size_t)group * N, c_col = (size_t)inner + (size_t)(groups + group) * N;

    auto fetch = [&](int t0, int buf) {                    // rows past the sequence's end are zeros
        constexpr int V = N / 8;
        for (int i = tid; i < CH * V; i += 128) {
            const int t = i / V, k = i % V;
            const bool ok = t0 + t < n_tok;
            const __nv_bfloat16* row = xbc + (size_t)(start + (ok ? t0 + t : 0)) * channels;
            ch_copy16(ch_word<N>(sm.b[buf], t, k), row + b_col + k * 8, ok);
            ch_copy16(ch_word<N>(sm.c[buf], t, k), row + c_col + k * 8, ok);
        }
        for (int i = tid; i < CH * 8; i += 128) {
            const int t = i >> 3, k = i & 7;
            const bool ok = t0 + t < n_tok && k * 8 < cols;
            ch_copy16(&sm.x[buf][t][k * 8], ok ? xbc + (size_t)(start + t0 + t) * channels + h * P + p0 + k * 8 : xbc, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto raw_dt = [&](int t0) { return tid < CH && t0 + tid < n_tok ? ch_any(dt_in, dt_dtype, (size_t)(start + t0 + tid) * dt_stride + dt_col0 + h) : 0.f; };

    // S^T: this warp's columns p0 + 16 warp .. (rows g and g + 8 of the fragment), N in tiles of 8
    float S[N / 8][4];
    const int pr = p0 + warp * 16 + g;
    float* state_row = state + (size_t)slot * state_stride + (size_t)h * N * P;
#pragma unroll
    for (int n = 0; n < N / 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = pr + 8 * (j >> 1), nn = n * 8 + 2 * q + (j & 1);
            S[n][j] = p < P ? state_row[(size_t)nn * P + p] : 0.f;
        }
    fetch(0, 0);
    float dt_next = raw_dt(0);
    const int mi = lane >> 3, mr = lane & 7;               // ldmatrix: this lane's matrix and row
    for (int t0 = 0, buf = 0; t0 < n_tok; t0 += CH, buf ^= 1) {
        const bool more = t0 + CH < n_tok;
        // ---- step sizes and running sums of the chunk's decays
        const float raw = dt_next + bias;
        const float dt = tid < CH && t0 + tid < n_tok ? (raw > 20.f ? raw : log1pf(expf(raw))) : 0.f;
        double c = (double)(A * dt);
        if (more) dt_next = raw_dt(t0 + CH);
        if (warp < 2) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const double v = __shfl_up_sync(0xffffffffu, c, o); if (lane >= o) c += v; }
            if (lane == 31) sm.part[warp] = c;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                   // rows of this chunk are here; the chunk before has been read
        if (more) fetch(t0 + CH, buf ^ 1);
        if (warp < 2) {
            const double total = sm.part[0] + sm.part[1];
            if (warp == 1) c += sm.part[0];
            const float hi = (float)c;
            sm.dt[tid] = dt;
            sm.cum[tid] = hi;
            sm.cum_lo[tid] = (float)(c - (double)hi);
            sm.decay[tid] = ch_exp(c);
            sm.weight[tid] = ch_exp(total - c) * dt;
            if (tid == 0) sm.last = ch_exp(total);
        }
        // ---- scores of this warp's 16 tokens: C_t . B_s for s up to the warp's last token
        float G[CH / 8][4];
#pragma unroll
        for (int s = 0; s < CH / 8; ++s) G[s][0] = G[s][1] = G[s][2] = G[s][3] = 0.f;
#pragma unroll
        for (int k = 0; k < N / 16; ++k) {
            uint32_t a[4];
            ch_ldsm(a, ch_word<N>(sm.c[buf], warp * 16 + (mi & 1) * 8 + mr, 2 * k + (mi >> 1)));
#pragma unroll
            for (int s = 0; s < CH / 16; ++s) {
                if (s > warp) break;
                uint32_t b[4];
                ch_ldsm(b, ch_word<N>(sm.b[buf], s * 16 + (mi >> 1) * 8 + mr, 2 * k + (mi & 1)));
                ch_mma_add(G[2 * s], a, b[0], b[1]);
                ch_mma_add(G[2 * s + 1], a, b[2], b[3]);
            }
        }
        float odd_g = 0.f;                                 // B_t . C_t is not finite where B_t or C_t is not
#pragma unroll
        for (int s = 0; s < CH / 8; ++s)
#pragma unroll
            for (int j = 0; j < 4; ++j) odd_g = fmaf(G[s][j], 0.f, odd_g);
        // (and the sums of the decays are written)
        bool odd = __syncthreads_or(odd_g != odd_g || !(sm.part[0] + sm.part[1] > -1e5));
#pragma unroll
        for (int s = 0; s < CH / 8; ++s) {
            if (s > 2 * warp + 1) break;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = warp * 16 + g + 8 * r, s0 = s * 8 + 2 * q;
                float v[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int ss = s0 + j;
                    v[j] = 0.f;
                    if (ss <= t) {                          // (|c_t| >= |c_s|: what the subtractions round off is known exactly)
                        const float d = sm.cum[t] - sm.cum[ss], lo = ((sm.cum[t] - d) - sm.cum[ss]) + (sm.cum_lo[t] - sm.cum_lo[ss]);
                        const float arg = d + lo, e = expf(arg);
                        v[j] = G[s][2 * r + j] * fmaf(e, lo - (arg - d), e) * sm.dt[ss];
                    }
                    if (ss == t) v[j] += Dh;
                }
                uint32_t w0, w1, w2;
                ch_split(v[0], v[1], w0, w1, w2);
                *reinterpret_cast<uint32_t*>(&sm.m[0][t][s0]) = w0;
                *reinterpret_cast<uint32_t*>(&sm.m[1][t][s0]) = w1;
                *reinterpret_cast<uint32_t*>(&sm.m[2][t][s0]) = w2;
            }
        }
        // ---- whether this warp's columns hold only finite numbers (zero times anything else is NaN)
        const uint32_t odd_x = [&] {
            uint32_t zeros = 0u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {                  // rows lane and lane + 32, eight columns a word
                const uint4 v = *reinterpret_cast<const uint4*>(&sm.x[buf][lane + 32 * (i >> 1)][warp * 16 + 8 * (i & 1)]);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    __nv_bfloat162 z = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]), __nv_bfloat162(0.f, 0.f), *reinterpret_cast<const __nv_bfloat162*>(&zeros));
                    zeros = *reinterpret_cast<const uint32_t*>(&z);
                }
            }
            return zeros & 0x7fff7fffu;
        }();
        float odd_s = 0.f;
#pragma unroll
        for (int n = 0; n < N / 8; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) odd_s = fmaf(S[n][j], 0.f, odd_s);
        odd = odd || __any_sync(0xffffffffu, odd_x != 0u || odd_s != odd_s);
        // ---- what the state before the chunk gives: Y^T = S^T C^T, then each token's decay.  The leading terms' products are summed
        // in Y, those of the others, 2^-8 of them and less, in Z.  (Eight independent sums stand between two products of one,
        // about the unit's latency.)
        float Y[CH / 8][4], Z[CH / 8][4];
#pragma unroll
        for (int t = 0; t < CH / 8; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) Y[t][j] = Z[t][j] = 0.f;
        if (!odd) {
#pragma unroll
        for (int k = 0; k < N / 16; ++k) {
            uint32_t a0[4], a1[4], a2[4], b[CH / 16][4];
            ch_split(S[2 * k][0], S[2 * k][1], a0[0], a1[0], a2[0]);
            ch_split(S[2 * k][2], S[2 * k][3], a0[1], a1[1], a2[1]);
            ch_split(S[2 * k + 1][0], S[2 * k + 1][1], a0[2], a1[2], a2[2]);
            ch_split(S[2 * k + 1][2], S[2 * k + 1][3], a0[3], a1[3], a2[3]);
#pragma unroll
            for (int t = 0; t < CH / 16; ++t) ch_ldsm(b[t], ch_word<N>(sm.c[buf], t * 16 + (mi >> 1) * 8 + mr, 2 * k + (mi & 1)));
#pragma unroll
            for (int t = 0; t < CH / 16; ++t) { ch_mma(Z[2 * t], a2, b[t][0], b[t][1]); ch_mma(Z[2 * t + 1], a2, b[t][2], b[t][3]); }
#pragma unroll
            for (int t = 0; t < CH / 16; ++t) { ch_mma_add(Y[2 * t], a0, b[t][0], b[t][1]); ch_mma_add(Y[2 * t + 1], a0, b[t][2], b[t][3]); }
#pragma unroll
            for (int t = 0; t < CH / 16; ++t) { ch_mma(Z[2 * t], a1, b[t][0], b[t][1]); ch_mma(Z[2 * t + 1], a1, b[t][2], b[t][3]); }
        }
#pragma unroll
        for (int t = 0; t < CH / 8; ++t) {
            const float d0 = sm.decay[t * 8 + 2 * q], d1 = sm.decay[t * 8 + 2 * q + 1];
            Y[t][0] *= d0; Y[t][1] *= d1; Y[t][2] *= d0; Y[t][3] *= d1;
            Z[t][0] *= d0; Z[t][1] *= d1; Z[t][2] *= d0; Z[t][3] *= d1;
        }
        }
        __syncthreads();                                   // the scores are written
        if (odd) {
            for (int t = 0; t < min(CH, n_tok - t0); ++t) {
                const float step = sm.dt[t], keep = expf(A * step);
                const float x0 = __bfloat162float(sm.x[buf][t][warp * 16 + g]), x1 = __bfloat162float(sm.x[buf][t][warp * 16 + g + 8]);
                const float u0 = step * x0, u1 = step * x1;
                float y0 = 0.f, y1 = 0.f;
#pragma unroll
                for (int n = 0; n < N / 8; ++n) {
                    const uint32_t b = *reinterpret_cast<const uint32_t*>(ch_word<N>(sm.b[buf], t, n) + 2 * q);
                    const uint32_t c2 = *reinterpret_cast<const uint32_t*>(ch_word<N>(sm.c[buf], t, n) + 2 * q);
                    S[n][0] = fmaf(keep, S[n][0], ch_low(b) * u0); S[n][1] = fmaf(keep, S[n][1], ch_high(b) * u0);
                    S[n][2] = fmaf(keep, S[n][2], ch_low(b) * u1); S[n][3] = fmaf(keep, S[n][3], ch_high(b) * u1);
                    y0 = fmaf(S[n][1], ch_high(c2), fmaf(S[n][0], ch_low(c2), y0));
                    y1 = fmaf(S[n][3], ch_high(c2), fmaf(S[n][2], ch_low(c2), y1));
                }
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) { y0 += __shfl_xor_sync(0xffffffffu, y0, o); y1 += __shfl_xor_sync(0xffffffffu, y1, o); }
                float* row = y + (size_t)(start + t0 + t) * inner + h * P;
                if (q == 0 && pr < P) row[pr] = fmaf(Dh, x0, y0);
                if (q == 0 && pr + 8 < P) row[pr + 8] = fmaf(Dh, x1, y1);
            }
            continue;
        }
        // ---- the chunk's own tokens: Y^T += x^T M^T
#pragma unroll
        for (int k = 0; k < CH / 16; ++k) {
            uint32_t xa[4];
            ch_ldsm_t(xa, &sm.x[buf][k * 16 + (mi >> 1) * 8 + mr][warp * 16 + (mi & 1) * 8]);
#pragma unroll
            for (int term = 2; term >= 0; --term)
#pragma unroll
                for (int t = 0; t < CH / 16; ++t) {
                    if (k > t) continue;                   // tokens before the block see nothing of it
                    uint32_t b[4];
                    ch_ldsm(b, &sm.m[term][t * 16 + (mi >> 1) * 8 + mr][k * 16 + (mi & 1) * 8]);
                    if (term) { ch_mma(Z[2 * t], xa, b[0], b[1]); ch_mma(Z[2 * t + 1], xa, b[2], b[3]); }
                    else { ch_mma_add(Y[2 * t], xa, b[0], b[1]); ch_mma_add(Y[2 * t + 1], xa, b[2], b[3]); }
                }
        }
#pragma unroll
        for (int t = 0; t < CH / 8; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int p = pr + 8 * (j >> 1), tt = t0 + t * 8 + 2 * q + (j & 1);
                if (p < P && tt < n_tok) y[(size_t)(start + tt) * inner + h * P + p] = Y[t][j] + Z[t][j];
            }
        // ---- the state: S^T = e^(c_L) S^T + (weight x)^T B, 64 of its rows n at a time (sums of the leading terms and of the others)
        const float last = sm.last;
#pragma unroll
        for (int n0 = 0; n0 < N / 16; n0 += 4) {
            float U[8][4], V[8][4];
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) U[n][j] = V[n][j] = 0.f;
#pragma unroll
            for (int k = 0; k < CH / 16; ++k) {
                uint32_t xa[4], a0[4], a1[4], a2[4], b[4][4];
                ch_ldsm_t(xa, &sm.x[buf][k * 16 + (mi >> 1) * 8 + mr][warp * 16 + (mi & 1) * 8]);
#pragma unroll
                for (int n = 0; n < 4; ++n) ch_ldsm_t(b[n], ch_word<N>(sm.b[buf], k * 16 + (mi & 1) * 8 + mr, 2 * (n0 + n) + (mi >> 1)));
                const float w0 = sm.weight[k * 16 + 2 * q], w1 = sm.weight[k * 16 + 2 * q + 1];
                const float w2 = sm.weight[k * 16 + 8 + 2 * q], w3 = sm.weight[k * 16 + 8 + 2 * q + 1];
                ch_split(ch_low(xa[0]) * w0, ch_high(xa[0]) * w1, a0[0], a1[0], a2[0]);
                ch_split(ch_low(xa[1]) * w0, ch_high(xa[1]) * w1, a0[1], a1[1], a2[1]);
                ch_split(ch_low(xa[2]) * w2, ch_high(xa[2]) * w3, a0[2], a1[2], a2[2]);
                ch_split(ch_low(xa[3]) * w2, ch_high(xa[3]) * w3, a0[3], a1[3], a2[3]);
#pragma unroll
                for (int n = 0; n < 4; ++n) { ch_mma(V[2 * n], a2, b[n][0], b[n][1]); ch_mma(V[2 * n + 1], a2, b[n][2], b[n][3]); }
#pragma unroll
                for (int n = 0; n < 4; ++n) { ch_mma_add(U[2 * n], a0, b[n][0], b[n][1]); ch_mma_add(U[2 * n + 1], a0, b[n][2], b[n][3]); }
#pragma unroll
                for (int n = 0; n < 4; ++n) { ch_mma(V[2 * n], a1, b[n][0], b[n][1]); ch_mma(V[2 * n + 1], a1, b[n][2], b[n][3]); }
            }
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) S[2 * n0 + n][j] = fmaf(last, S[2 * n0 + n][j], U[n][j] + V[n][j]);
        }
    }
#pragma unroll
    for (int n = 0; n < N / 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = pr + 8 * (j >> 1), nn = n * 8 + 2 * q + (j & 1);
            if (p < P) state_row[(size_t)nn * P + p] = S[n][j];
        }
}

template <int N>
static int launch_chunk(const void* xbc, int channels, const void* dt_in, int dt_dtype, int dt_stride, int dt_col0, const void* dt_bias,
                        const void* a_log, const void* d_skip, int p_dtype, const int* cu_seqlens, const int* state_slots, float* state,
                        size_t state_stride, float* y, int n_seqs, int heads, int P, int groups, int least, cudaStream_t stream) {
    static RvPerDevice once;
    if (int st = rv_configure_smem(once, ssm_chunk_kernel<N>, (int)sizeof(ChunkSmem<N>))) return st;
    return rv_launch(ssm_chunk_kernel<N>, dim3((P + 63) / 64, heads, n_seqs), dim3(128), sizeof(ChunkSmem<N>), stream, (const __nv_bfloat16*)xbc,
                     channels, dt_in, dt_dtype, dt_stride, dt_col0, dt_bias, a_log, d_skip, p_dtype, cu_seqlens, state_slots, state,
                     state_stride, y, heads, P, groups, least);
}

// Arguments as of rv_ssm_scan (ssm.cu), xbc bfloat16; sequences of fewer than `least` tokens are left alone.  RV_ERR_UNSUPPORTED for sizes that the kernel does not serve: state sizes
// other than 64 and 128, rows that are not whole 16-byte words.
RV_EXPORT int rv_ssm_chunk(const void* xbc, int channels, const void* dt_in, int dt_dtype, int dt_stride, int dt_col0, const void* dt_bias,
                           const void* a_log, const void* d_skip, int p_dtype, const int* cu_seqlens, const int* state_slots, float* state,
                           long long state_stride, float* y, int n_seqs, int heads, int P, int N, int groups, int least, cudaStream_t stream) {
    if (n_seqs < 0 || heads <= 0 || P <= 0 || N <= 0 || groups <= 0 || heads % groups) return RV_ERR_BAD_SIZE;
    if (channels < heads * P + 2 * groups * N || dt_stride < dt_col0 + heads || dt_col0 < 0) return RV_ERR_BAD_SIZE;
    if ((dt_dtype | p_dtype) & ~1) return RV_ERR_BAD_DTYPE;
    if (heads > 65535 || n_seqs > 65535 || (P & 7) || (channels & 7) || (reinterpret_cast<uintptr_t>(xbc) & 15)) return RV_ERR_UNSUPPORTED;
    if (n_seqs == 0) return RV_OK;
    if (N == 128)
        RV_LAUNCH_ST = launch_chunk<128>(xbc, channels, dt_in, dt_dtype, dt_stride, dt_col0, dt_bias, a_log, d_skip, p_dtype, cu_seqlens,
                                         state_slots, state, (size_t)state_stride, y, n_seqs, heads, P, groups, least, stream);
    else if (N == 64)
        RV_LAUNCH_ST = launch_chunk<64>(xbc, channels, dt_in, dt_dtype, dt_stride, dt_col0, dt_bias, a_log, d_skip, p_dtype, cu_seqlens,
                                        state_slots, state, (size_t)state_stride, y, n_seqs, heads, P, groups, least, stream);
    else
        return RV_ERR_UNSUPPORTED;
    return rv_launch_status();
}
