// Sampling over float logits [R, V]: greedy (lowest index wins ties, NaN never wins) and
// seeded temperature sampling with optional top-k / top-p, one block per row.
//
// Parameters per row as the reference's SamplingParams {temperature, top_k, top_p, seed}
// (v3/crates/rvllm-sampling/src/params.rs:7-28): temperature 0 means greedy.  The reference
// ships only an argmax kernel (kernels/argmax.cu:66-117; tie rule of its oracle,
// v3/crates/rvllm-fused/src/reference.rs:131-146); the rest is defined here:
//   p = softmax(logits / T) in float with the maximum subtracted;
//   top-k keeps the tokens at least as likely as the k-th most likely one;
//   top-p keeps the most likely tokens up to the first whose cumulated mass reaches top_p
//   (tokens exactly as likely as the last kept one stay in);
//   the draw is the first token, in vocabulary order, whose cumulated kept mass exceeds
//   u * (kept mass), with u = Philox4x32-10(key = seed, counter = index of the output token).
// The uniform depends on (seed, output index) only, never on the batch a row is sampled in.
//
// Rows with a top-k or a top-p take two passes over the row (maximum + counts per bin of the top 12 bits of
// the ordered bit pattern, then the tokens from a bin upwards and the whole mass); the at most
// 2,048 candidates are sorted and cut exactly in the first CTA's shared memory.  Rows under a top-p alone whose cut
// lies below their 2,048 most likely tokens take three passes over the masses (`sample_mass_way`).  The general search, eight
// passes of four bits over the row, is left with: rows under a top-k with fewer than k tokens that are numbers, or
// more than 2,048 tokens down to the end of the k-th one's bin (k beyond 2,048, or a flat row); under a top-p alone, rows whose maximum is
// infinite, a share above 2 M tokens a CTA, a top-p that no fixed-point mass is small enough for.  All sums that decide anything are integers or
// are added in a fixed order, so a token depends neither on the run nor on how many CTAs share the row.
#include "common.cuh"
#include <string.h>

#define SAMPLE_THREADS 1024

__device__ __forceinline__ uint32_t order_key(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// Block-wide (value, index) arg-max: larger value wins, then lower index.
__device__ __forceinline__ void argmax_combine(float& v, int& i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

// ---------------------------------------------------------------------------------------------
// One to eight CTAs per row.  A row is always cut into SAMPLE_SLICES contiguous slices of the
// vocabulary; every reduction over the row (arg-max, mass, the 16 + 16 sums of a pass of the
// threshold search, the kept mass) is done slice by slice by one block of SAMPLE_THREADS threads and
// the slices' results are combined in slice order.  With several CTAs per row (a thread-block
// cluster; each CTA owns SAMPLE_SLICES / CTAs neighbouring slices) each CTA writes its slices'
// results into every CTA's shared memory (st.shared::cluster), and one cluster barrier later all CTAs
// combine the same numbers in the same order and take the same decision.  So the sampled token does
// not depend on how many CTAs share the row, which the host chooses by the number of rows: one block
// per row is bound by its own instruction rate (125 tokens per thread and pass at a vocabulary of
// 128,256), eight CTAs make a pass eight times shorter.  The exchange buffers alternate between two
// copies, so that a CTA that is one step ahead never overwrites what a slower one still reads.
#define SAMPLE_SLICES 8

__device__ __forceinline__ uint32_t sc_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t sc_map(const void* p, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void sc_store(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void sc_store(uint32_t addr, int v) { asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sc_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// What the CTAs of a row tell one another, per slice; two copies, used in turn.
struct SampleExchange {
    float val[SAMPLE_SLICES];                // arg-max value / mass / kept mass of a slice
    int idx[SAMPLE_SLICES];                  // arg-max index / last kept token of a slice
    int cnt[SAMPLE_SLICES][16];              // a pass of the threshold search: tokens per digit
    float mass[SAMPLE_SLICES][16];           // ... and their mass
};

// The chunk of slice [lo_s, hi_s) that thread `tid` owns.
__device__ __forceinline__ void slice_chunk(int lo_s, int hi_s, int tid, int& lo, int& hi) {
    const int C = (hi_s - lo_s + SAMPLE_THREADS - 1) / SAMPLE_THREADS;
    lo = min(hi_s, lo_s + tid * C);
    hi = min(hi_s, lo + C);
}

// Kept mass of the `per` slices from `first` on, in vocabulary order: thread t owns a contiguous chunk of each.  On return
// s_incl[sl][t] is slice first + sl's kept mass up to the end of thread t's chunk, s_last[sl] its last kept token (-1: none).  (The
// slices side by side: one after the other, each with its own barriers, four of 16,032 tokens took 12 us.)
__device__ void slices_scan(const float* row, int V, int S, int first, int per, uint32_t tau, float m, float inv_t, float (*s_scan)[SAMPLE_THREADS / 32],
                            float (*s_incl)[SAMPLE_THREADS], int* s_last) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float incl[SAMPLE_SLICES];
    int last_kept[SAMPLE_SLICES];
    __syncthreads();                                       // the previous use of the shared arrays is over
    if (tid < per) s_last[tid] = -1;
#pragma unroll
    for (int sl = 0; sl < SAMPLE_SLICES; ++sl) {
        if (sl >= per) break;
        const int lo_s = min(V, (first + sl) * S), hi_s = min(V, lo_s + S);
        int lo, hi, last = -1;
        slice_chunk(lo_s, hi_s, tid, lo, hi);
        float local = 0.f;
        auto take = [&](float v, int i) {
            if (order_key(v) >= tau && !(v != v)) { local += expf((v - m) * inv_t); last = i; }
        };
        if (((lo | hi) & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
#pragma unroll 4
            for (int i = lo; i < hi; i += 4) {
                const float4 q = *reinterpret_cast<const float4*>(row + i);
                take(q.x, i); take(q.y, i + 1); take(q.z, i + 2); take(q.w, i + 3);
            }
        } else {
            for (int i = lo; i < hi; ++i) take(row[i], i);
        }
        float in = local;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float n = __shfl_up_sync(0xffffffffu, in, o);
            if (lane >= o) in += n;
        }
        if (lane == 31) s_scan[sl][warp] = in;
        incl[sl] = in;
        last_kept[sl] = last;
    }
    __syncthreads();
#pragma unroll
    for (int sl = 0; sl < SAMPLE_SLICES; ++sl)
        if (sl < per && last_kept[sl] >= 0) atomicMax(&s_last[sl], last_kept[sl]);
    if (warp < per) {
        static_assert(SAMPLE_THREADS / 32 == 32, "a warp adds up the warps of a slice");
        const float w = s_scan[warp][lane];
        float wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float n = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += n;
        }
        s_scan[warp][lane] = wi - w;                       // exclusive prefix of the warps
    }
    __syncthreads();
    // inclusive prefixes in shared memory, so that neighbouring chunks tile [0, kept mass)
    // without gaps or overlaps whatever the rounding
#pragma unroll
    for (int sl = 0; sl < SAMPLE_SLICES; ++sl)
        if (sl < per) s_incl[sl][tid] = s_scan[sl][warp] + incl[sl];
    __syncthreads();
}

// ---------------------------------------------------------------------------------------------
// The short way to the top-k / top-p threshold: two passes over the row instead of eleven.
//
// A histogram counts the row's tokens over the top 12 bits of the ordered bit pattern (sign, exponent, three bits of
// mantissa: 4,096 bins); the CTAs of a row add their bins into the first CTA's histogram through distributed shared
// memory.  The threshold lies in the bin of the k-th token, or in the one in which the cumulated mass exp((v - m) / T)
// reaches top_p x (the whole mass); masses are 40-bit fixed-point integers, so their sums do not depend on the order of the
// additions, on the number of CTAs that share the row or on the run.  Every token from the threshold's bin upwards is a
// candidate.  If there are at most FAST_CANDIDATES of them (a peaked distribution, or a small k), they are gathered
// - ordered bit pattern and index, in any order - in the first CTA's shared memory, where they are sorted (bitonic, by
// value then index: a total order, so the result is the same whatever order they arrived in), cut exactly by count and by
// cumulated mass, sorted back into vocabulary order and drawn from.  Otherwise the kernel goes on below: a flat row under
// top-p alone by its masses, any other by the general search.
#define FAST_BINS 4096
#define FAST_CANDIDATES 2048
#define FAST_SCALE 1099511627776.0f      // 2^40

__device__ __forceinline__ void sc_red_add(uint32_t addr, unsigned int v) { asm volatile("red.shared::cluster.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sc_red_add(uint32_t addr, unsigned long long v) { asm volatile("red.shared::cluster.add.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory"); }
__device__ __forceinline__ void sc_store(uint32_t addr, unsigned long long v) { asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory"); }
__device__ __forceinline__ float key_value(uint32_t key) {
    return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

__device__ __forceinline__ unsigned long long sort_keep(unsigned long long x, unsigned long long y, bool larger) { return (x > y) == larger ? x : y; }

// Bitonic sort of n_pad (a power of two, SORT_LEAST ... FAST_CANDIDATES) 64-bit keys in shared memory, descending: eight neighbouring
// keys a thread, so that most pairs meet in a thread's registers or by shuffles, and only those 256 and more apart through
// shared memory, behind a barrier of the few warps that take part.  (A key a thread, every pair through shared memory behind a barrier of
// 1,024 threads: 64 keys 3.5 us, 1,024 keys 11; with shuffles within a warp 1,024 still 8.5.)
#define SORT_LEAST 256
__device__ void sort_desc(unsigned long long* a, int n_pad) {
    const int t = threadIdx.x, threads = n_pad / 8;
    if (t < threads) {                                     // (whole warps)
        unsigned long long x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = a[8 * t + e];
        auto in_thread = [&](int j, auto&& down) {          // pairs j < 8 apart
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if ((e & j) == 0 && (x[e] < x[e | j]) == down(e)) { const unsigned long long s = x[e]; x[e] = x[e | j]; x[e | j] = s; }
        };
        in_thread(1, [](int e) { return (e & 2) == 0; });
        in_thread(2, [](int e) { return (e & 4) == 0; });
        in_thread(1, [](int e) { return (e & 4) == 0; });
        for (int k = 8; k <= n_pad; k <<= 1) {
            const bool is_down = ((8 * t) & k) == 0;
            auto down = [&](int) { return is_down; };
            int j = k >> 1;
            for (; j >= 256; j >>= 1) {
#pragma unroll
                for (int e = 0; e < 8; ++e) a[8 * t + e] = x[e];
                asm volatile("bar.sync 1, %0;" :: "r"(threads) : "memory");
                const int other = 8 * (t ^ (j >> 3));
                const bool larger = ((8 * t & j) == 0) == is_down;
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = sort_keep(x[e], a[other + e], larger);
                asm volatile("bar.sync 1, %0;" :: "r"(threads) : "memory");
            }
            for (; j >= 8; j >>= 1) {
                const bool larger = ((8 * t & j) == 0) == is_down;
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = sort_keep(x[e], __shfl_xor_sync(0xffffffffu, x[e], j >> 3), larger);
            }
            in_thread(4, down);
            in_thread(2, down);
            in_thread(1, down);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) a[8 * t + e] = x[e];
    }
    __syncthreads();
}

// The same for 64 keys of one warp: keys l and l + 32 of lane l.
__device__ __forceinline__ void sort_desc_64(unsigned long long& x, unsigned long long& y) {
    const int l = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 64; k <<= 1) {
        const bool up_x = (l & k) == 0, up_y = ((l + 32) & k) == 0;
        if (k == 64 && x < y) { const unsigned long long s = x; x = y; y = s; }
#pragma unroll
        for (int j = k == 64 ? 16 : k >> 1; j > 0; j >>= 1) {
            const bool first = (l & j) == 0;
            x = sort_keep(x, __shfl_xor_sync(0xffffffffu, x, j), first == up_x);
            y = sort_keep(y, __shfl_xor_sync(0xffffffffu, y, j), first == up_y);
        }
    }
}

// Inclusive sums of n (<= 2 * SAMPLE_THREADS) floats in shared memory, in place, in index order: thread t owns
// elements 2t and 2t + 1; warp scans by shuffles, warp totals through s_scan.  The same order every time.
__device__ void scan_inclusive(float* a, int n, float* s_scan) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float x0 = 2 * tid < n ? a[2 * tid] : 0.f, x1 = 2 * tid + 1 < n ? a[2 * tid + 1] : 0.f;
    float incl = x0 + x1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    __syncthreads();
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        float w = s_scan[lane], wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float v = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += v;
        }
        s_scan[lane] = wi - w;
    }
    __syncthreads();
    const float before = s_scan[warp] + incl - (x0 + x1);
    if (2 * tid < n) a[2 * tid] = before + x0;
    if (2 * tid + 1 < n) a[2 * tid + 1] = before + x0 + x1;
    __syncthreads();
}

struct FastShared {
    unsigned int n_cand;        // candidates gathered so far (in the first CTA)
    int go;                     // 1: the short way serves the row; 0: the general search
    int bin;                    // candidates are the tokens from this bin upwards
    int kept, pick;
    unsigned long long z_q;     // the row's whole mass, fixed point
};

// `scan_inclusive` of 64 floats by one warp, in the same order: lane l owns elements 2l (x0) and 2l + 1 (x1).
__device__ __forceinline__ void scan_inclusive_64(float& x0, float& x1) {
    const int lane = threadIdx.x & 31;
    const float pair = x0 + x1;
    float incl = pair;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const float all = __shfl_sync(0xffffffffu, incl, 31);
    const float before = (all - all) + incl - pair;
    x1 = before + x0 + x1;
    x0 = before + x0;
}

// `short_way_finish` for at most 64 candidates: one warp, nothing to wait for (the same sums in the same order).
__device__ void short_way_finish_64(unsigned long long* cand, int n, float m, float inv_t, int k, float pp, bool use_k, bool use_p,
                                    unsigned long long seed, long long draw, int* out_token, unsigned long long z_q) {
    const int lane = threadIdx.x & 31;
    auto relay = [&](unsigned long long& x, unsigned long long& y) {     // from keys l and l + 32 to keys 2l and 2l + 1
        cand[lane] = x; cand[lane + 32] = y;
        __syncwarp();
        x = cand[2 * lane]; y = cand[2 * lane + 1];
        __syncwarp();
    };
    unsigned long long x = lane < n ? cand[lane] : 0ull, y = lane + 32 < n ? cand[lane + 32] : 0ull;
    __syncwarp();
    sort_desc_64(x, y);
    relay(x, y);
    auto mass = [&](unsigned long long c) { return expf((key_value((uint32_t)(c >> 32)) - m) * inv_t); };
    const bool hx = 2 * lane < n, hy = 2 * lane + 1 < n;
    const float mx = hx ? mass(x) : 0.f, my = hy ? mass(y) : 0.f;
    float sx = mx, sy = my;
    scan_inclusive_64(sx, sy);
    uint32_t tau = 0u;
    if (use_k) {
        const int at = min(k, n) - 1;
        const uint32_t kx = __shfl_sync(0xffffffffu, (uint32_t)(x >> 32), at >> 1), ky = __shfl_sync(0xffffffffu, (uint32_t)(y >> 32), at >> 1);
        tau = at & 1 ? ky : kx;
    }
    if (use_p) {
        const float target = pp * (float)((double)z_q * (1.0 / (double)FAST_SCALE));
        const float before = __shfl_up_sync(0xffffffffu, sy, 1);
        const unsigned int ox = __ballot_sync(0xffffffffu, hx && sx >= target && (lane == 0 || before < target));
        const unsigned int oy = __ballot_sync(0xffffffffu, hy && sy >= target && sx < target);
        const int lx = ox ? __ffs(ox) - 1 : 32, ly = oy ? __ffs(oy) - 1 : 32;
        const uint32_t kx = __shfl_sync(0xffffffffu, (uint32_t)(x >> 32), lx & 31), ky = __shfl_sync(0xffffffffu, (uint32_t)(y >> 32), ly & 31);
        if (lx < 32 && lx <= ly) tau = max(tau, kx);
        else if (ly < 32) tau = max(tau, ky);
    }
    // kept: the candidates whose value is at least the threshold - a prefix of the sorted list; back into vocabulary order
    const bool kept_x = hx && (uint32_t)(x >> 32) >= tau, kept_y = hy && (uint32_t)(y >> 32) >= tau;
    const int L = __popc(__ballot_sync(0xffffffffu, kept_x)) + __popc(__ballot_sync(0xffffffffu, kept_y));
    x = kept_x ? ((unsigned long long)(uint32_t)x << 32) | (unsigned long long)__float_as_uint(mx) : 0ull;
    y = kept_y ? ((unsigned long long)(uint32_t)y << 32) | (unsigned long long)__float_as_uint(my) : 0ull;
    sort_desc_64(x, y);
    relay(x, y);
    sx = 2 * lane < L ? __uint_as_float((uint32_t)x) : 0.f;
    sy = 2 * lane + 1 < L ? __uint_as_float((uint32_t)y) : 0.f;
    scan_inclusive_64(sx, sy);
    uint32_t c4[4] = {(uint32_t)(draw & 0xffffffffll), (uint32_t)((unsigned long long)draw >> 32), 0u, 0u};
    philox4x32_10(c4, (uint32_t)(seed & 0xffffffffull), (uint32_t)(seed >> 32));
    const float u = (float)(c4[0] >> 8) * (1.0f / 16777216.0f);
    const float all_x = __shfl_sync(0xffffffffu, sx, (L - 1) >> 1), all_y = __shfl_sync(0xffffffffu, sy, (L - 1) >> 1);
    const float t_draw = u * ((L - 1) & 1 ? all_y : all_x);
    const float before = __shfl_up_sync(0xffffffffu, sy, 1);
    const unsigned int ox = __ballot_sync(0xffffffffu, 2 * lane < L && sx > t_draw && (lane == 0 || before <= t_draw));
    const unsigned int oy = __ballot_sync(0xffffffffu, 2 * lane + 1 < L && sy > t_draw && sx <= t_draw);
    int pick = L - 1;                                     // rounding put the target at the kept mass: the last kept token
    if (ox || oy) {
        const int px = ox ? 2 * (__ffs(ox) - 1) : 64, py = oy ? 2 * (__ffs(oy) - 1) + 1 : 64;
        pick = min(px, py);
    }
    const uint32_t ix = __shfl_sync(0xffffffffu, (uint32_t)(x >> 32), pick >> 1), iy = __shfl_sync(0xffffffffu, (uint32_t)(y >> 32), pick >> 1);
    if (lane == 0) *out_token = (int)(0xffffffffu - (pick & 1 ? iy : ix));
}

// The first CTA's end of the short way: sort the gathered candidates, cut by count and by mass, draw.
__device__ void short_way_finish(unsigned long long* cand, float* cmass, int n, float m, float inv_t, int k, float pp, bool use_k,
                                 bool use_p, unsigned long long seed, long long draw, int* out_token, float* s_scan, FastShared* fs) {
    const int tid = threadIdx.x;
    int n_pad = SORT_LEAST;
    while (n_pad < n) n_pad <<= 1;
    for (int i = n + tid; i < n_pad; i += SAMPLE_THREADS) cand[i] = 0ull;       // sorts behind every candidate
    __syncthreads();
    sort_desc(cand, n_pad);
    // masses in descending order of value and their running sums
    for (int i = tid; i < n; i += SAMPLE_THREADS) cmass[i] = expf((key_value((uint32_t)(cand[i] >> 32)) - m) * inv_t);
    __syncthreads();
    scan_inclusive(cmass, n, s_scan);
    // the threshold: the value of the k-th candidate, and of the first whose running sum reaches top_p x the whole mass
    __shared__ unsigned int s_tau_k, s_tau_p;
    if (tid == 0) {
        s_tau_k = use_k ? (uint32_t)(cand[min(k, n) - 1] >> 32) : 0u;
        s_tau_p = 0u;
    }
    __syncthreads();
    if (use_p) {
        const float target = pp * (float)((double)fs->z_q * (1.0 / (double)FAST_SCALE));
        for (int i = tid; i < n; i += SAMPLE_THREADS)
            if (cmass[i] >= target && (i == 0 || cmass[i - 1] < target)) s_tau_p = (uint32_t)(cand[i] >> 32);
    }
    __syncthreads();
    const uint32_t tau = max(s_tau_k, s_tau_p);
    // kept: the candidates whose value is at least the threshold - a prefix of the sorted list
    for (int i = tid; i < n; i += SAMPLE_THREADS)
        if ((uint32_t)(cand[i] >> 32) >= tau && (i + 1 == n || (uint32_t)(cand[i + 1] >> 32) < tau)) fs->kept = i + 1;
    __syncthreads();
    const int L = fs->kept;
    // back into vocabulary order: (index, mass bits), ascending = descending of the complement
    int l_pad = SORT_LEAST;
    while (l_pad < L) l_pad <<= 1;
    for (int i = tid; i < l_pad; i += SAMPLE_THREADS) {
        unsigned long long w = 0ull;
        if (i < L) {
            const uint32_t key = (uint32_t)(cand[i] >> 32), inv_idx = (uint32_t)cand[i];
            w = ((unsigned long long)inv_idx << 32) | (unsigned long long)__float_as_uint(expf((key_value(key) - m) * inv_t));
        }
        cand[i] = w;
    }
    __syncthreads();
    sort_desc(cand, l_pad);                               // descending complemented index = ascending index; padding (0) last
    for (int i = tid; i < L; i += SAMPLE_THREADS) cmass[i] = __uint_as_float((uint32_t)cand[i]);
    __syncthreads();
    scan_inclusive(cmass, L, s_scan);
    uint32_t c4[4] = {(uint32_t)(draw & 0xffffffffll), (uint32_t)((unsigned long long)draw >> 32), 0u, 0u};
    philox4x32_10(c4, (uint32_t)(seed & 0xffffffffull), (uint32_t)(seed >> 32));
    const float u = (float)(c4[0] >> 8) * (1.0f / 16777216.0f);
    const float t_draw = u * cmass[L - 1];
    for (int i = tid; i < L; i += SAMPLE_THREADS)
        if (cmass[i] > t_draw && (i == 0 || cmass[i - 1] <= t_draw)) fs->pick = i;
    __syncthreads();
    if (tid == 0) {
        const int pick = fs->pick >= 0 ? fs->pick : L - 1;           // rounding put the target at the kept mass: the last kept token
        *out_token = (int)(0xffffffffu - (uint32_t)(cand[pick] >> 32));
    }
}

// f(value, index) for every token of [lo, hi) that is a thread's: four 16-byte words in flight where the share is made of such words
// (one word at a time left the memory idle between a pass's steps), else token by token; indices rise within a thread.
template <typename F>
__device__ __forceinline__ void sample_walk(const float* __restrict__ row, int lo, int hi, const F& f) {
    if (((lo | hi) & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
        const float4* r4 = reinterpret_cast<const float4*>(row);
        const int end = hi >> 2;
        for (int i0 = (lo >> 2) + threadIdx.x; i0 < end; i0 += 4 * SAMPLE_THREADS) {
            float4 q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i0 + j * SAMPLE_THREADS < end) q[j] = r4[i0 + j * SAMPLE_THREADS];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = i0 + j * SAMPLE_THREADS;
                if (i >= end) break;
                f(q[j].x, 4 * i); f(q[j].y, 4 * i + 1); f(q[j].z, 4 * i + 2); f(q[j].w, 4 * i + 3);
            }
        }
        return;
    }
    for (int i = lo + threadIdx.x; i < hi; i += SAMPLE_THREADS) f(row[i], i);
}

// The CTAs' candidates (n_cand of them in `cand`, at most FAST_CANDIDATES in all) side by side in the first CTA's memory; it gets their number,
// the others 0.
__device__ __forceinline__ int gather_in_first(unsigned long long* cand, const unsigned int* n_cand, int CL, int rank) {
    __shared__ unsigned int x_cnt[8];
    const int tid = threadIdx.x;
    __syncthreads();
    if (CL == 1) return (int)min(*n_cand, (unsigned int)FAST_CANDIDATES);
    if (tid < CL) sc_store(sc_map(&x_cnt[rank], tid), (int)*n_cand);
    sc_sync();
    unsigned int base = 0u, all = 0u;
    for (int c = 0; c < CL; ++c) { if (c < rank) base += x_cnt[c]; all += x_cnt[c]; }
    if (rank != 0) {
        const uint32_t to = sc_map(cand, 0);
        for (unsigned int i = tid; i < x_cnt[rank] && base + i < FAST_CANDIDATES; i += SAMPLE_THREADS) sc_store(to + (base + i) * 8u, cand[i]);
    }
    sc_sync();
    return rank == 0 ? (int)min(all, (unsigned int)FAST_CANDIDATES) : 0;
}

// A token among the candidates of this CTA.  (Gathered in the CTA's own memory: a count in another CTA's kept the warp waiting.)
__device__ __forceinline__ void gather_one(unsigned long long* cand, unsigned int* n_cand, uint32_t key, int i) {
    const int lane = threadIdx.x & 31;
    const unsigned int now = __activemask(), first = __ffs(now) - 1;           // one add for the lanes that are here together
    unsigned int pos = 0u;
    if (lane == (int)first) pos = atomicAdd(n_cand, __popc(now));
    pos = __shfl_sync(now, pos, first) + __popc(now & ((1u << lane) - 1u));
    if (pos < FAST_CANDIDATES) cand[pos] = ((unsigned long long)key << 32) | (unsigned long long)(0xffffffffu - (uint32_t)i);
}

// The short way: TWO passes over the row.  Pass A finds the row's maximum (larger value, then lower index - the same whatever
// the order) and counts the tokens per bin; no exponential, no mass.  With a top-k the bin of the k-th token follows from the
// counts alone; with a top-p alone, pass B takes the tokens of as many bins from the top as hold at most FAST_CANDIDATES.
// Pass B gathers the tokens from that bin upwards and adds up the row's whole mass as 40-bit fixed-point integers in registers.
// A top-p cut behind a top-k lies among the candidates or below them all; a top-p cut alone is then found among the bins of the
// candidates, by their masses: where these do not reach it, the tokens down to it are more than FAST_CANDIDATES.  (The masses
// of all tokens, added per bin by 64-bit atomics in shared memory, took three passes: 64 rows of 128,256 tokens 134 us, now 42;
// one of 152,064 52, now 25; behind a top-k 40 and 34.)  `m_out` / `best_out` carry the maximum on to the general search where the candidates are too many.
__device__ bool sample_short_way(const float* __restrict__ row, int V, float inv_t, int k, float pp, bool use_k, bool use_p,
                                 unsigned long long seed, long long draw, int* out_token, unsigned char* s_dyn, float* s_scan,
                                 float* s_val, int* s_idx, FastShared* fs, float& m_out, int& best_out) {
    const int CL = gridDim.x, rank = (int)sc_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned int* h_cnt = reinterpret_cast<unsigned int*>(s_dyn);                                   // [FAST_BINS]
    unsigned int* h_low = h_cnt + FAST_BINS;               // [FAST_BINS], [FAST_BINS]: the candidates' masses, low 20 bits and the others, added
    unsigned int* h_high = h_low + FAST_BINS;              // apart (2,048 times 2^20 fit 32 bits: adds of 64 bits in shared memory are loops)
    unsigned long long* cand = reinterpret_cast<unsigned long long*>(h_high + FAST_BINS);           // [FAST_CANDIDATES]
    float* cmass = reinterpret_cast<float*>(cand + FAST_CANDIDATES);                                // [FAST_CANDIDATES]
    __shared__ float x_val[8];
    __shared__ int x_idx[8];
    for (int b = tid; b < FAST_BINS; b += SAMPLE_THREADS) h_cnt[b] = 0u;
    if (tid == 0) { fs->n_cand = 0u; fs->go = 0; fs->bin = 0; fs->kept = 0; fs->pick = -1; fs->z_q = 0ull; }
    __syncthreads();
    const int per = (((V + CL - 1) / CL) + 3) & ~3;
    const int lo = min(V, rank * per), hi = min(V, lo + per);
    // ---- pass A: maximum and counts
    float bv = __int_as_float(0x7fc00000);                // (the first token that is not NaN is larger than nothing, also -inf)
    int bi = 0x7fffffff;
    sample_walk(row, lo, hi, [&](float v, int i) {
        if (v != v) return;
        if (!(v <= bv)) { bv = v; bi = i; }               // indices rise within a thread: equal values keep the lowest
        atomicAdd(&h_cnt[order_key(v) >> 20], 1u);
    });
    if (bi == 0x7fffffff) bv = -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        argmax_combine(bv, bi, ov, oi);
    }
    if (lane == 0) { s_val[warp] = bv; s_idx[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        bv = s_val[lane]; bi = s_idx[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            argmax_combine(bv, bi, ov, oi);
        }
        if (lane < CL) { sc_store(sc_map(&x_val[rank], lane), bv); sc_store(sc_map(&x_idx[rank], lane), bi); }
    }
    sc_sync();                                            // maxima exchanged, every CTA's counts complete
    float m = -INFINITY;
    int best = 0x7fffffff;
    for (int c = 0; c < CL; ++c) argmax_combine(m, best, x_val[c], x_idx[c]);
    if (best == 0x7fffffff) best = 0;
    m_out = m; best_out = best;
    if (rank != 0) {
        for (int b = tid; b < FAST_BINS; b += SAMPLE_THREADS)
            if (h_cnt[b]) sc_red_add(sc_map(&h_cnt[b], 0), h_cnt[b]);
    }
    sc_sync();
    if (rank == 0) {
        // the bin of the k-th token, counted from the top bin down: thread t owns the bins 4095 - 4t ... 4092 - 4t
        unsigned int c_own = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) c_own += h_cnt[FAST_BINS - 1 - 4 * tid - j];
        unsigned int c_inc = c_own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int cv = __shfl_up_sync(0xffffffffu, c_inc, o);
            if (lane >= o) c_inc += cv;
        }
        __shared__ unsigned int w_cnt[32];
        __shared__ int s_bk;
        __shared__ unsigned int s_n;
        if (lane == 31) w_cnt[warp] = c_inc;
        if (tid == 0) { s_bk = use_k ? -1 : FAST_BINS; s_n = 0u; }
        __syncthreads();
        unsigned int c_run = c_inc - c_own;
        for (int w = 0; w < warp; ++w) c_run += w_cnt[w];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int b = FAST_BINS - 1 - 4 * tid - j;
            const unsigned int c = h_cnt[b];
            if (use_k) {
                if (c_run < (unsigned int)k && c_run + c >= (unsigned int)k) { s_bk = b; s_n = c_run + c; }
            } else if (c_run + c <= FAST_CANDIDATES) {      // (all bins from the top down to the lowest of these)
                atomicMin(&s_bk, b);
                atomicMax(&s_n, c_run + c);
            }
            c_run += c;
        }
        __syncthreads();
        // (fewer than k tokens in the row, or more than FAST_CANDIDATES in its first bins: the general search)
        bool go = use_k ? s_bk >= 0 && s_n <= FAST_CANDIDATES : s_n > 0u;
        if (!use_k && go) {
            // a flat row: the counts and the edges of the bins bound the candidates' mass from above and the whole mass
            // from below; where these cannot meet, pass B would be for nothing (empty bins and edges that are no numbers add nothing)
            float most = 0.f, least = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int b = FAST_BINS - 1 - 4 * tid - j;
                if (!h_cnt[b]) continue;
                const float c = (float)h_cnt[b], low = key_value((uint32_t)b << 20), high = key_value(((uint32_t)b << 20) | 0xfffffu);
                if (low == low) least += c * expf((low - m) * inv_t);
                if (b >= s_bk) most += c * (high == high ? expf((fminf(high, m) - m) * inv_t) : 1.f);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                most += __shfl_xor_sync(0xffffffffu, most, o);
                least += __shfl_xor_sync(0xffffffffu, least, o);
            }
            if (lane == 0) { s_val[warp] = most; s_scan[warp] = least; }
            __syncthreads();
            most = least = 0.f;
            for (int w = 0; w < SAMPLE_THREADS / 32; ++w) { most += s_val[w]; least += s_scan[w]; }
            go = !(most * 1.001f < pp * least);            // (a thousandth: far above what the sums' rounding can do)
        }
        if (tid < CL) { sc_store(sc_map(&fs->go, tid), go ? 1 : 0); sc_store(sc_map(&fs->bin, tid), s_bk); }
    }
    sc_sync();
    if (!fs->go) return false;
    // ---- pass B: candidates to the first CTA; the whole mass, if a top-p cut wants it
    {
        const uint32_t bin = (uint32_t)fs->bin;
        unsigned long long z = 0ull;
        sample_walk(row, lo, hi, [&](float v, int i) {
            if (v != v) return;
            const uint32_t key = order_key(v);
            if (use_p) z += __float2ull_rz(expf((v - m) * inv_t) * FAST_SCALE);
            if ((key >> 20) >= bin) gather_one(cand, &fs->n_cand, key, i);
        });
        if (use_p) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
            if (lane == 0) sc_red_add(sc_map(&fs->z_q, 0), z);
        }
    }
    int n = gather_in_first(cand, &fs->n_cand, CL, rank);
    if (!use_k) {
        // ---- the bin in which the candidates' masses, from the top down, reach top_p x the whole mass
        if (rank == 0) {
            __shared__ unsigned long long w_mass[32];
            __shared__ int s_bp, s_kept;
            for (int b = tid; b < FAST_BINS; b += SAMPLE_THREADS) h_low[b] = h_high[b] = 0u;
            if (tid == 0) { s_bp = -1; s_kept = 0; }
            __syncthreads();
            for (int i = tid; i < n; i += SAMPLE_THREADS) {
                const uint32_t key = (uint32_t)(cand[i] >> 32);
                const unsigned long long q = __float2ull_rz(expf((key_value(key) - m) * inv_t) * FAST_SCALE);
                atomicAdd(&h_low[key >> 20], (uint32_t)q & 0xfffffu);
                atomicAdd(&h_high[key >> 20], (uint32_t)(q >> 20));
            }
            __syncthreads();
            auto mass_of = [&](int b) { return ((unsigned long long)h_high[b] << 20) + h_low[b]; };
            unsigned long long m_own = 0ull;               // thread t owns the bins 4095 - 4t ... 4092 - 4t
#pragma unroll
            for (int j = 0; j < 4; ++j) m_own += mass_of(FAST_BINS - 1 - 4 * tid - j);
            unsigned long long m_inc = m_own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long mv = __shfl_up_sync(0xffffffffu, m_inc, o);
                if (lane >= o) m_inc += mv;
            }
            if (lane == 31) w_mass[warp] = m_inc;
            __syncthreads();
            unsigned long long m_run = m_inc - m_own;
            for (int w = 0; w < warp; ++w) m_run += w_mass[w];
            const unsigned long long target = (unsigned long long)((double)pp * (double)fs->z_q);
#pragma unroll
            for (int j = 0; j < 4; ++j) {                  // exactly one thread finds it
                const int b = FAST_BINS - 1 - 4 * tid - j;
                const unsigned long long mm = mass_of(b);
                if (target > 0ull && m_run < target && m_run + mm >= target) s_bp = b;
                m_run += mm;
            }
            __syncthreads();
            // (a row whose maximum is +inf has masses that are no numbers: its infinities are the candidates)
            if (tid == 0 && m == INFINITY) s_bp = fs->z_q ? (int)(order_key(INFINITY) >> 20) : -1;
            __syncthreads();
            // candidates below that bin are none: the others close ranks (what is sorted is what a cut can keep)
            unsigned long long own[2] = {tid < n ? cand[tid] : 0ull, tid + SAMPLE_THREADS < n ? cand[tid + SAMPLE_THREADS] : 0ull};
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (tid + j * SAMPLE_THREADS < n && (int)(own[j] >> 52) >= s_bp) {
                    const unsigned int now = __activemask(), first = __ffs(now) - 1;
                    int pos = 0;
                    if (lane == (int)first) pos = atomicAdd(&s_kept, __popc(now));
                    cand[__shfl_sync(now, pos, first) + __popc(now & ((1u << lane) - 1u))] = own[j];
                }
            __syncthreads();
            n = s_kept;
            if (tid < CL) sc_store(sc_map(&fs->go, tid), s_bp >= 0 ? 1 : 0);
        }
        sc_sync();
        if (!fs->go) return false;                         // (not reached, or rounding keeps the mass below the target)
    }
    if (rank != 0) return true;                           // the first CTA finishes the row; nobody's shared memory is touched from outside any more
    if (n <= 64) {
        if (warp == 0) short_way_finish_64(cand, n, m, inv_t, k, pp, use_k, use_p, seed, draw, out_token, fs->z_q);
        return true;
    }
    short_way_finish(cand, cmass, n, m, inv_t, k, pp, use_k, use_p, seed, draw, out_token, s_scan, fs);
    return true;
}

// The threshold of a top-p alone whose cut lies below FAST_CANDIDATES tokens (a flat row): the key tau with
// mass(key >= tau) >= top_p x (the whole mass) > mass(key > tau), masses as 40-bit fixed-point integers.  One pass adds up the masses (and
// counts) of 16 groups of neighbouring bins, each about a sixteenth of the tokens by the histogram that the short way left in the
// first CTA; a group of more than FAST_CANDIDATES tokens is divided again, by key; the tokens of the last group are gathered, sorted and
// cut.  Every thread adds in places of its own (16 sums of 64 bits, the count above the mass), so nothing is atomic and the sums
// are exact.  Three passes over the row in place of the search's eight: a step of 64 rows
// of 128,256 tokens with one such row 212 -> 101 us, 36 without.
#define MASS_GROUPS 16
#define MASS_BITS 52                       // of a thread's sum: 4,096 masses of 2^40; the count above
struct MassShared {
    unsigned long long mass[2][MASS_GROUPS];               // of the row's groups; two copies, used in turn
    unsigned int count[2][MASS_GROUPS];
    unsigned int group_of[FAST_BINS / 4];                  // per bin, a byte each (255: no token)
    uint32_t lo, hi, tau;
};

__device__ bool sample_mass_way(const float* __restrict__ row, int V, float inv_t, float pp, float m, unsigned char* s_dyn, float* s_scan,
                                FastShared* fs, MassShared* ms, uint32_t& tau) {
    const int CL = gridDim.x, rank = (int)sc_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = (((V + CL - 1) / CL) + 3) & ~3;
    const int lo_v = min(V, rank * per), hi_v = min(V, lo_v + per);
    if (per > (SAMPLE_THREADS << 11) || !(fabsf(m) < INFINITY)) return false;  // (every CTA alike)
    unsigned long long* slots = reinterpret_cast<unsigned long long*>(s_dyn);  // [MASS_GROUPS][SAMPLE_THREADS]
    unsigned long long* cand = slots;                                           // later
    if (tid < 2 * MASS_GROUPS) { ms->mass[tid / MASS_GROUPS][tid % MASS_GROUPS] = 0ull; ms->count[tid / MASS_GROUPS][tid % MASS_GROUPS] = 0u; }
    if (tid == 0) { ms->lo = 0xffffffffu; ms->hi = 0u; fs->n_cand = 0u; }
    __syncthreads();
    sc_sync();                                             // (every CTA's places are zero)
    if (rank == 0) {
        // the group of a bin, by the tokens above it: thread t owns the bins 4095 - 4t ... 4092 - 4t
        const unsigned int* h_cnt = reinterpret_cast<const unsigned int*>(s_dyn);
        unsigned int* w_cnt = reinterpret_cast<unsigned int*>(s_scan);
        unsigned int own = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) own += h_cnt[FAST_BINS - 1 - 4 * tid - j];
        unsigned int inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const unsigned int v = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += v; }
        if (lane == 31) w_cnt[warp] = inc;
        __syncthreads();
        unsigned int run = inc - own, all = 0u;
        for (int w = 0; w < SAMPLE_THREADS / 32; ++w) { if (w < warp) run += w_cnt[w]; all += w_cnt[w]; }
        unsigned int word = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned int g = (unsigned int)(((unsigned long long)run * MASS_GROUPS) / max(all, 1u));
            const unsigned int c = h_cnt[FAST_BINS - 1 - 4 * tid - j];
            word |= (c ? min(g, MASS_GROUPS - 1u) : 0xffu) << (8 * (3 - j));          // (empty bins are nobody's: a group's keys are those of its tokens)
            run += c;
        }
        for (int c = 0; c < CL; ++c) sc_store(sc_map(&ms->group_of[FAST_BINS / 4 - 1 - tid], c), (int)word);
    }
    sc_sync();                                             // the groups are known; the histogram is read
    const unsigned char* group_of = reinterpret_cast<const unsigned char*>(ms->group_of);
    auto clear = [&]() {
#pragma unroll
        for (int g = 0; g < MASS_GROUPS; ++g) slots[g * SAMPLE_THREADS + tid] = 0ull;
    };
    auto add = [&](int g, float v) {
        slots[g * SAMPLE_THREADS + tid] += __float2ull_rz(expf((v - m) * inv_t) * FAST_SCALE) + (1ull << MASS_BITS);
    };
    auto meet = [&](int turn) {                            // a warp adds up a group and tells every CTA
        __syncthreads();
        if (warp < MASS_GROUPS) {
            unsigned long long mass = 0ull;
            unsigned int count = 0u;
            for (int i = lane; i < SAMPLE_THREADS; i += 32) {
                const unsigned long long v = slots[warp * SAMPLE_THREADS + i];
                mass += v & ((1ull << MASS_BITS) - 1);
                count += (unsigned int)(v >> MASS_BITS);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                mass += __shfl_xor_sync(0xffffffffu, mass, o);
                count += __shfl_xor_sync(0xffffffffu, count, o);
            }
            if (lane < CL) { sc_red_add(sc_map(&ms->mass[turn][warp], lane), mass); sc_red_add(sc_map(&ms->count[turn][warp], lane), count); }
        }
        sc_sync();
    };
    clear();
    sample_walk(row, lo_v, hi_v, [&](float v, int) {
        if (v == v) add(group_of[order_key(v) >> 20], v);
    });
    meet(0);
    unsigned long long z = 0ull, above = 0ull;
    for (int g = 0; g < MASS_GROUPS; ++g) z += ms->mass[0][g];
    const unsigned long long target = (unsigned long long)((double)pp * (double)z);
    if (target == 0ull) return false;
    int g = 0;
    while (g < MASS_GROUPS - 1 && above + ms->mass[0][g] < target) above += ms->mass[0][g++];
    unsigned int count = ms->count[0][g];
    // the group's keys
    for (int b = tid; b < FAST_BINS; b += SAMPLE_THREADS)
        if (group_of[b] == g) { atomicMin(&ms->lo, (uint32_t)b << 20); atomicMax(&ms->hi, ((uint32_t)b << 20) | 0xfffffu); }
    __syncthreads();
    uint32_t lo = ms->lo, hi = ms->hi;
    int turn = 0;
    while (count > FAST_CANDIDATES && hi > lo) {           // (every CTA decides alike)
        const int shift = max(0, 28 - __clz(hi - lo));     // sixteen parts at most, counted from the top
        clear();
        turn ^= 1;
        if (tid < MASS_GROUPS && turn == 0) { ms->mass[0][tid] = 0ull; ms->count[0][tid] = 0u; }
        if (turn == 0) sc_sync();                          // (read by everyone, and zero again)
        sample_walk(row, lo_v, hi_v, [&](float v, int) {
            if (v != v) return;
            const uint32_t key = order_key(v);
            if (key >= lo && key <= hi) add((int)((hi - key) >> shift), v);
        });
        meet(turn);
        g = 0;
        while (g < MASS_GROUPS - 1 && above + ms->mass[turn][g] < target) above += ms->mass[turn][g++];
        count = ms->count[turn][g];
        const uint32_t top = hi - ((uint32_t)g << shift);
        lo = max(lo, top - min(top, (1u << shift) - 1u));
        hi = top;
        if (turn == 1) {                                   // the next turn's places
            sc_sync();
            if (tid < MASS_GROUPS) { ms->mass[1][tid] = 0ull; ms->count[1][tid] = 0u; }
        }
    }
    if (count > FAST_CANDIDATES) { tau = hi; return true; }                     // many tokens of one value
    __syncthreads();
    sample_walk(row, lo_v, hi_v, [&](float v, int i) {
        if (v != v) return;
        const uint32_t key = order_key(v);
        if (key >= lo && key <= hi) gather_one(cand, &fs->n_cand, key, i);
    });
    const int n = gather_in_first(cand, &fs->n_cand, CL, rank);
    if (rank == 0) {
        int n_pad = SORT_LEAST;
        while (n_pad < n) n_pad <<= 1;
        for (int i = n + tid; i < n_pad; i += SAMPLE_THREADS) cand[i] = 0ull;
        if (tid == 0) ms->tau = 0u;
        __syncthreads();
        sort_desc(cand, n_pad);
        // the first whose running mass, behind what lies above, reaches the target: thread t owns keys 2t and 2t + 1
        unsigned long long* w_mass = cand + FAST_CANDIDATES;
        unsigned long long q[2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
            q[j] = 2 * tid + j < n ? __float2ull_rz(expf((key_value((uint32_t)(cand[2 * tid + j] >> 32)) - m) * inv_t) * FAST_SCALE) : 0ull;
        unsigned long long inc = q[0] + q[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const unsigned long long v = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += v; }
        if (lane == 31) w_mass[warp] = inc;
        __syncthreads();
        unsigned long long run = above + inc - q[0] - q[1];
        for (int w = 0; w < warp; ++w) run += w_mass[w];
#pragma unroll
        for (int j = 0; j < 2; ++j) {                      // (exactly one finds it)
            if (2 * tid + j < n && run < target && run + q[j] >= target) ms->tau = (uint32_t)(cand[2 * tid + j] >> 32);
            run += q[j];
        }
        __syncthreads();
        const uint32_t found = ms->tau;
        __syncthreads();
        if (tid < CL) sc_store(sc_map(&ms->tau, tid), (int)found);
    }
    sc_sync();
    tau = ms->tau;
    return tau != 0u;
}

__device__ int g_sample_short_way = 1;      // 0: always the general search (tests compare the two), 2: rows the short way leaves get -1, 3: rows left to the search do

// Where a row's parameters are: in arrays on the device (null: greedy, or off), or, for up to SAMPLE_VALUE_ROWS rows whose
// parameters the host has, in the launch itself: no buffer on the device, no copy of 1.8 KB that the host prepares and the kernel waits
// for (64 rows: 76 us of the host's time with them, 23 without).
#define SAMPLE_VALUE_ROWS 128               // 28 bytes each: with the other arguments below the 4 KB that every launch may carry
struct SampleArrays {
    const float* temperature;
    const int* top_k;
    const float* top_p;
    const unsigned long long* seeds;
    const long long* draw_index;
    __device__ __forceinline__ float t(int r) const { return temperature ? temperature[r] : 0.f; }
    __device__ __forceinline__ int k(int r) const { return top_k ? top_k[r] : 0; }
    __device__ __forceinline__ float p(int r) const { return top_p ? top_p[r] : 1.0f; }
    __device__ __forceinline__ unsigned long long seed(int r) const { return seeds[r]; }
    __device__ __forceinline__ long long draw(int r) const { return draw_index[r]; }
};
struct SampleValues {
    unsigned long long seeds[SAMPLE_VALUE_ROWS];
    long long draw_index[SAMPLE_VALUE_ROWS];
    float temperature[SAMPLE_VALUE_ROWS], top_p[SAMPLE_VALUE_ROWS];
    int top_k[SAMPLE_VALUE_ROWS];
    __device__ __forceinline__ float t(int r) const { return temperature[r]; }
    __device__ __forceinline__ int k(int r) const { return top_k[r]; }
    __device__ __forceinline__ float p(int r) const { return top_p[r]; }
    __device__ __forceinline__ unsigned long long seed(int r) const { return seeds[r]; }
    __device__ __forceinline__ long long draw(int r) const { return draw_index[r]; }
};

template <typename Rows>
__global__ void __launch_bounds__(SAMPLE_THREADS, 1)
sample_kernel(const float* __restrict__ logits, const __grid_constant__ Rows rows, int* __restrict__ out, int V) {
    rv_pdl_launch_dependents();
    rv_pdl_wait();
    __shared__ float s_val[33];
    __shared__ int s_idx[33];
    __shared__ float s_scan[SAMPLE_THREADS / 32 + 1];
    __shared__ int s_result, s_last[SAMPLE_SLICES];
    __shared__ float s_incl[SAMPLE_SLICES][SAMPLE_THREADS], s_warps[SAMPLE_SLICES][SAMPLE_THREADS / 32];
    __shared__ int s_cnt[2][16];
    __shared__ float s_mass[2][16];
    __shared__ SampleExchange xch[2];
    __shared__ FastShared fast_shared;
    __shared__ MassShared mass_shared;
    extern __shared__ __align__(16) unsigned char s_dyn_fast[];      // the dynamic shared memory, as the short way lays it out
    // gridDim.x CTAs (1, 2, 4 or 8: the cluster) share row blockIdx.y; this one owns the slices [first, first + per)
    const int CL = gridDim.x, rank = (int)sc_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = SAMPLE_SLICES / CL, first = rank * per;
    const int r = blockIdx.y;
    const float* row = logits + (size_t)r * V;
    const int S = (((V + SAMPLE_SLICES - 1) / SAMPLE_SLICES) + 3) & ~3;     // slices of an aligned row start on 16-byte boundaries
    const float T = rows.t(r);
    int turn = 0;                                        // which copy of the exchange buffers is written next
    sc_sync();                                           // every CTA of the cluster runs before its memory is written

    const int k_row = rows.k(r);
    const float p_row = rows.p(r);
    const bool uk_row = k_row > 0 && k_row < V, up_row = p_row < 1.0f;
    const float inv_t = fminf(1.0f / T, 3.402823466e38f);      // (a temperature below 2.9e-39 would make the maximum's own mass 0 x infinity)
    float m = -INFINITY;
    int best = 0x7fffffff;
    bool have_max = false, have_tau = false;
    uint32_t tau = 0;
    if (T > 0.f && (uk_row || up_row) && g_sample_short_way) {
        // maximum, counts and candidates in two passes; too many candidates: the maximum is kept, the search below goes on
        if (sample_short_way(row, V, inv_t, k_row, p_row, uk_row, up_row, rows.seed(r), rows.draw(r), out + r, s_dyn_fast, s_scan,
                               s_val, s_idx, &fast_shared, m, best))
            return;
        have_max = true;
        sc_sync();                                       // (the first CTA's shared memory is no longer written from outside)
        if (g_sample_short_way == 2) {
            if (rank == 0 && tid == 0) out[r] = -1;
            return;
        }
        if (!uk_row) have_tau = sample_mass_way(row, V, inv_t, p_row, m, s_dyn_fast, s_scan, &fast_shared, &mass_shared, tau);
        if (g_sample_short_way == 3 && !have_tau) {
            if (rank == 0 && tid == 0) out[r] = -1;
            return;
        }
    }
    if (!have_max) {
    // ---- arg-max of the row: this CTA's slices lie side by side
    float bv = __int_as_float(0x7fc00000);                // (as in the short way)
    int bi = 0x7fffffff;
    sample_walk(row, min(V, first * S), min(V, (first + per) * S), [&](float v, int i) {
        if (v == v && !(v <= bv)) { bv = v; bi = i; }
    });
    if (bi == 0x7fffffff) bv = -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        argmax_combine(bv, bi, ov, oi);
    }
    if (lane == 0) { s_val[warp] = bv; s_idx[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        bv = s_val[lane]; bi = s_idx[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            argmax_combine(bv, bi, ov, oi);
        }
        if (lane < CL) { sc_store(sc_map(&xch[turn].val[rank], lane), bv); sc_store(sc_map(&xch[turn].idx[rank], lane), bi); }
    }
    sc_sync();
    for (int c = 0; c < CL; ++c) argmax_combine(m, best, xch[turn].val[c], xch[turn].idx[c]);   // larger value, then lower index
    if (best == 0x7fffffff) best = 0;
    turn ^= 1;
    }
    if (!(T > 0.f)) {
        if (rank == 0 && tid == 0) out[r] = best;
        return;
    }

    // ---- mass of everything, where a top-p is measured by it
    float total = 0.f;
    if (up_row && !have_tau) {
    for (int sl = first; sl < first + per; ++sl) {
        const int lo_s = min(V, sl * S), hi_s = min(V, lo_s + S);
        float part = 0.f;
        for (int i = lo_s + tid; i < hi_s; i += SAMPLE_THREADS) {
            const float v = row[i];
            if (v == v) part += expf((v - m) * inv_t);   // (with a NaN among them the target was none, and everything was kept)
        }
        part = rv_block_sum(part, s_val);
        if (tid < CL) sc_store(sc_map(&xch[turn].val[sl], tid), part);
    }
    sc_sync();
    for (int sl = 0; sl < SAMPLE_SLICES; ++sl) total += xch[turn].val[sl];
    turn ^= 1;
    }

    // ---- threshold key: keep tokens whose order key is >= tau.  tau is the largest key c with
    // count(key >= c) >= k (top-k), or with mass(key >= c) >= top_p * total (top-p); it is found four
    // bits at a time, eight passes over the row: every thread counts its tokens (and adds their mass)
    // by the next four bits of the key in 16 slots of its own in shared memory, for the tokens that
    // agree with the bits decided so far; the block adds the slots up in a fixed order, the slices'
    // sums are added in slice order, and the largest digit that still satisfies the condition is
    // taken.  No atomics: the same result in every run.  NaN is never kept.
    const int k = k_row;
    const float pp = p_row;
    bool use_k = k > 0 && k < V;
    bool use_p = pp < 1.0f;
    if (!have_tau && (use_k || use_p)) {
        extern __shared__ __align__(16) unsigned char s_dyn[];
        int* h_cnt = reinterpret_cast<int*>(s_dyn);                                   // [16][SAMPLE_THREADS]
        float* h_mass = reinterpret_cast<float*>(s_dyn) + 16 * SAMPLE_THREADS;       // [16][SAMPLE_THREADS]
        uint32_t pre_k = 0, pre_p = 0;        // the bits decided so far
        int above_cnt = 0;                    // tokens whose decided bits are greater than pre_k
        float above_mass = 0.f;               // mass of the tokens whose decided bits are greater than pre_p
        const float target = pp * total;
        for (int shift = 28; shift >= 0; shift -= 4) {
            for (int sl = first; sl < first + per; ++sl) {
                const int lo_s = min(V, sl * S), hi_s = min(V, lo_s + S);
#pragma unroll
                for (int d = 0; d < 16; ++d) { h_cnt[d * SAMPLE_THREADS + tid] = 0; h_mass[d * SAMPLE_THREADS + tid] = 0.f; }
                // four loads in flight per thread
                for (int i0 = lo_s + tid; i0 < hi_s; i0 += 4 * SAMPLE_THREADS) {
                    float vs[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int i = i0 + j * SAMPLE_THREADS;
                        vs[j] = i < hi_s ? row[i] : __int_as_float(0x7fc00000);      // NaN: skipped below
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float v = vs[j];
                        if (v != v) continue;
                        const uint32_t key = order_key(v);
                        const int d = (int)((key >> shift) & 15u);
                        const bool top = shift == 28;
                        if (use_k && (top || (key >> (shift + 4)) == (pre_k >> (shift + 4)))) h_cnt[d * SAMPLE_THREADS + tid] += 1;
                        if (use_p && (top || (key >> (shift + 4)) == (pre_p >> (shift + 4)))) h_mass[d * SAMPLE_THREADS + tid] += expf((v - m) * inv_t);
                    }
                }
                __syncthreads();
                {   // warp w adds digit w % 16 over one half of the threads, lanes in a fixed order
                    const int d = warp & 15, half = warp >> 4;
                    int c = 0;
                    float ms = 0.f;
                    for (int j = lane; j < SAMPLE_THREADS / 2; j += 32) {
                        c += h_cnt[d * SAMPLE_THREADS + half * (SAMPLE_THREADS / 2) + j];
                        ms += h_mass[d * SAMPLE_THREADS + half * (SAMPLE_THREADS / 2) + j];
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        c += __shfl_xor_sync(0xffffffffu, c, o);
                        ms += __shfl_xor_sync(0xffffffffu, ms, o);
                    }
                    if (lane == 0) { s_cnt[half][d] = c; s_mass[half][d] = ms; }
                }
                __syncthreads();
                // this slice's 16 + 16 sums go to every CTA of the row
                if (tid < 16 * CL) {
                    const int d = tid & 15, to = tid >> 4;
                    sc_store(sc_map(&xch[turn].cnt[sl][d], to), s_cnt[0][d] + s_cnt[1][d]);
                    sc_store(sc_map(&xch[turn].mass[sl][d], to), s_mass[0][d] + s_mass[1][d]);
                }
            }
            sc_sync();
            // every thread of every CTA takes the same decision from the same sums
            if (use_k) {
                int run = above_cnt, found = -1;
                for (int d = 15; d >= 0; --d) {
                    int c = 0;
                    for (int sl = 0; sl < SAMPLE_SLICES; ++sl) c += xch[turn].cnt[sl][d];
                    if (run + c >= k) { found = d; break; }
                    run += c;
                }
                if (found < 0) { use_k = false; pre_k = 0; }          // fewer than k tokens (NaN rows): keep all
                else { pre_k |= (uint32_t)found << shift; above_cnt = run; }
            }
            if (use_p) {
                float run = above_mass;
                int found = -1;
                for (int d = 15; d >= 0; --d) {
                    float c = 0.f;
                    for (int sl = 0; sl < SAMPLE_SLICES; ++sl) c += xch[turn].mass[sl][d];
                    if (run + c >= target) { found = d; break; }
                    run += c;
                }
                if (found < 0) { use_p = false; pre_p = 0; }          // rounding left the sum just below the target: keep all
                else { pre_p |= (uint32_t)found << shift; above_mass = run; }
            }
            turn ^= 1;
            if (!use_k && !use_p) break;
        }
        tau = pre_k > pre_p ? pre_k : pre_p;
    }

    // ---- kept mass and last kept token of every slice, to every CTA
    slices_scan(row, V, S, first, per, tau, m, inv_t, s_warps, s_incl, s_last);
    for (int i = tid; i < per * CL; i += SAMPLE_THREADS) {
        const int sl = i % per, to = i / per;
        sc_store(sc_map(&xch[turn].val[first + sl], to), s_incl[sl][SAMPLE_THREADS - 1]);
        sc_store(sc_map(&xch[turn].idx[first + sl], to), s_last[sl]);
    }
    sc_sync();
    float kept_total = 0.f;
    for (int sl = 0; sl < SAMPLE_SLICES; ++sl) kept_total += xch[turn].val[sl];

    // ---- the draw: the first token, in vocabulary order, whose cumulated kept mass exceeds u * (kept mass)
    const unsigned long long seed = rows.seed(r), draw = (unsigned long long)rows.draw(r);
    uint32_t c4[4] = {(uint32_t)draw, (uint32_t)(draw >> 32), 0u, 0u};
    philox4x32_10(c4, (uint32_t)seed, (uint32_t)(seed >> 32));
    const float u = (float)(c4[0] >> 8) * (1.0f / 16777216.0f);
    const float target = u * kept_total;
    // the slice the target falls into (the same arithmetic in every CTA); if rounding put the target at
    // or beyond the kept mass, the slice of the last kept token
    int resp = -1;
    float off = 0.f, resp_off = 0.f;
    for (int sl = 0; sl < SAMPLE_SLICES; ++sl) {
        const float kc = xch[turn].val[sl];
        if (resp < 0 && kc > 0.f && target < off + kc) { resp = sl; resp_off = off; }
        off += kc;
    }
    bool beyond = false;
    if (resp < 0) {
        beyond = true;
        for (int sl = SAMPLE_SLICES - 1; sl >= 0; --sl)
            if (xch[turn].idx[sl] >= 0) { resp = sl; break; }
    }
    if (resp < 0) {                                       // nothing was kept at all (a row of NaN): the arg-max
        if (rank == 0 && tid == 0) out[r] = best;
        return;
    }
    if (resp / per != rank) return;                       // (nothing of another CTA is touched after the barrier above)
    {
        const int own = resp - first, lo_s = min(V, resp * S), hi_s = min(V, lo_s + S);
        if (tid == 0) s_result = -1;
        __syncthreads();
        const float t_loc = target - resp_off, excl = tid > 0 ? s_incl[own][tid - 1] : 0.f, upto = s_incl[own][tid];
        if (!beyond && upto > excl && excl <= t_loc && t_loc < upto) {
            int lo, hi;
            slice_chunk(lo_s, hi_s, tid, lo, hi);
            float run = excl;
            int pick = -1;
            bool found = false;
            for (int i0 = lo; i0 < hi && !found; i0 += 16) {             // sixteen values in flight: one thread does this, the others wait
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = i0 + j < hi ? row[i0 + j] : __int_as_float(0x7fc00000);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (found || order_key(v[j]) < tau || v[j] != v[j]) continue;
                    run += expf((v[j] - m) * inv_t);
                    pick = i0 + j;                        // (none passes it, by rounding: the chunk's last kept token)
                    found = run > t_loc;
                }
            }
            atomicMax(&s_result, pick);   // at most one thread matches; max is only a tie guard
        }
        __syncthreads();
        // no chunk took it (rounding): the last kept token of the slice
        if (tid == 0) out[r] = s_result >= 0 ? s_result : (s_last[own] >= 0 ? s_last[own] : best);
    }
}

static int g_sample_cluster = 0;
// CTAs per row: 0 chosen by the number of rows, else 1, 2, 4 or 8 (for tests: the result is the same).
RV_EXPORT void rv_sample_set_cluster(int ctas_per_row) { g_sample_cluster = ctas_per_row; }
// 1 (default): top-k / top-p rows try the short way first; 0: always the general search; 2: the short way alone, rows that it
// does not serve get the id -1; 3: rows left to the general search get -1 (for tests).
RV_EXPORT int rv_sample_set_short_way(int mode) {
    const int v = mode == 2 || mode == 3 ? mode : (mode ? 1 : 0);
    return (int)cudaMemcpyToSymbol(g_sample_short_way, &v, sizeof(int));
}

// `filtered`: some row has a top-k or a top-p.
template <typename Rows>
static int launch_sample(const float* logits, const Rows& rows, int* out, int n_rows, int vocab, bool filtered, cudaStream_t stream) {
    // the threshold search of top-k / top-p keeps 16 counters and 16 sums per thread in shared memory
    const size_t smem = filtered ? (size_t)2 * 16 * SAMPLE_THREADS * 4 : 0;
    static RvPerDevice configured;
    if (smem) {
        if (int e = rv_configure_smem(configured, sample_kernel<Rows>, (int)(2 * 16 * SAMPLE_THREADS * 4))) return e;
    }
    // CTAs per row: as many (8, 4, 2 or 1) as keep rows x CTAs within the SMs; the result is the same for each
    const int sms = rv_sm_count();
    int cl = g_sample_cluster > 0 ? g_sample_cluster : (n_rows * 8 <= sms ? 8 : (n_rows * 4 <= sms ? 4 : (n_rows * 2 <= sms ? 2 : 1)));
    if (cl != 1 && cl != 2 && cl != 4 && cl != 8) return RV_ERR_BAD_SIZE;
    RV_LAUNCH_ST = rv_launch_cluster(sample_kernel<Rows>, dim3(cl, n_rows), dim3(SAMPLE_THREADS), smem, stream, (unsigned)cl, logits, rows, out, vocab);
    return rv_launch_status();
}

// temperature, top_k, top_p may be null (greedy / disabled).  seeds and draw_index are read
// only for rows with temperature > 0.
RV_EXPORT int rv_sample(const float* logits, const float* temperature, const int* top_k, const float* top_p,
                        const unsigned long long* seeds, const long long* draw_index, int* out,
                        int n_rows, int vocab, cudaStream_t stream) {
    if (n_rows < 0 || vocab <= 0) return RV_ERR_BAD_SIZE;
    if (n_rows == 0) return RV_OK;
    if (temperature && (!seeds || !draw_index)) return RV_ERR_BAD_SIZE;
    if (n_rows > 65535) return RV_ERR_BAD_SIZE;
    return launch_sample(logits, SampleArrays{temperature, top_k, top_p, seeds, draw_index}, out, n_rows, vocab,
                         temperature && (top_k || top_p), stream);
}

RV_EXPORT int rv_sample_value_rows() { return SAMPLE_VALUE_ROWS; }

// The same for up to SAMPLE_VALUE_ROWS rows whose parameters lie packed on the HOST: seeds (64 bits) of all rows, draw indices (64
// bits), temperatures, top-p, top-k (32 bits each).  They are read before the call returns.
RV_EXPORT int rv_sample_rows(const float* logits, const unsigned char* packed, int* out, int n_rows, int vocab, cudaStream_t stream) {
    if (n_rows < 0 || n_rows > SAMPLE_VALUE_ROWS || vocab <= 0 || !packed) return RV_ERR_BAD_SIZE;
    if (n_rows == 0) return RV_OK;
    SampleValues v;
    const size_t n = (size_t)n_rows;
    memcpy(v.seeds, packed, 8 * n);
    memcpy(v.draw_index, packed + 8 * n, 8 * n);
    memcpy(v.temperature, packed + 16 * n, 4 * n);
    memcpy(v.top_p, packed + 20 * n, 4 * n);
    memcpy(v.top_k, packed + 24 * n, 4 * n);
    bool filtered = false;
    for (int r = 0; r < n_rows; ++r) filtered = filtered || v.top_k[r] > 0 || v.top_p[r] < 1.0f;
    return launch_sample(logits, v, out, n_rows, vocab, filtered, stream);
}
