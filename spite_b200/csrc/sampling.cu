// Token sampling on the device.  A row of logits is worked on by a cluster of eight blocks that keep
// it in their shared memory (an eighth each; distributed shared memory carries the sums between them),
// so the passes of the pipeline below read shared memory, not L2; a row too long for that (more than
// 8 x 49,152 logits) is worked on by one block through a scratch row in global memory.
//
// The pipeline and its order are those of giveen/spite's sampler
// (crates/spite-sampling/src/lib.rs:273-296): repetition penalty over the distinct
// tokens of the trailing context (lib.rs:208-231), temperature (117-125), min-p
// (178-189), top-k (128-143), top-p (146-174), then the argmax when temperature <= 0
// (236-243; of equal maxima the highest index wins, as Rust's `max_by` returns the
// last) or a multinomial draw against unnormalised masses exp(l - max) with the
// 64-bit LCG of lib.rs:343-348 (first index whose running sum reaches u * total,
// 247-265).  Sums are float32 and are added in a fixed order (a thread's elements, the threads of
// a warp, the warps of a block, the blocks of a cluster by rank), so a row's result does not depend on
// the other rows or on timing.
#include <cmath>
#include <cstring>

#include "common.cuh"

namespace {

constexpr int THREADS = 1024;

__device__ __forceinline__ unsigned order_key(float v) {
    const unsigned u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float block_max(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < (THREADS >> 5) ? scratch[lane] : -INFINITY;
        t = warp_max(t);
        if (lane == 0) scratch[32] = t;
    }
    __syncthreads();
    return scratch[32];
}

// Largest index holding the maximum (argmax with ties to the highest index).
__device__ int block_argmax_last(const float* l, int n, float* fscratch, int* iscratch) {
    float best = -INFINITY;
    int idx = -1;
    for (int i = threadIdx.x; i < n; i += THREADS) {
        const float v = l[i];
        if (v > best || (v == best && i > idx) || idx < 0) { best = v; idx = i; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (oi >= 0 && (idx < 0 || ov > best || (ov == best && oi > idx))) { best = ov; idx = oi; }
    }
    __syncthreads();
    if (lane == 0) { fscratch[warp] = best; iscratch[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        best = lane < (THREADS >> 5) ? fscratch[lane] : -INFINITY;
        idx = lane < (THREADS >> 5) ? iscratch[lane] : -1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (oi >= 0 && (idx < 0 || ov > best || (ov == best && oi > idx))) { best = ov; idx = oi; }
        }
        if (lane == 0) iscratch[32] = idx;
    }
    __syncthreads();
    return iscratch[32];
}

// First index i (ascending) at which the running sum of f(0..i) reaches `target`;
// -1 if it never does.  Every thread owns a contiguous range of indices.
template <typename F>
__device__ int block_first_reaching(int n, float target, F f, float* fscratch, int* iscratch) {
    const int chunk = (n + THREADS - 1) / THREADS;
    const int lo = min(n, (int)threadIdx.x * chunk), hi = min(n, lo + chunk);
    float mine = 0.f;
    for (int i = lo; i < hi; ++i) mine += f(i);
    // exclusive scan of the per-thread sums: within a warp by shuffles, across warps serially
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) fscratch[warp] = incl;
    if (threadIdx.x == 0) iscratch[32] = 0x7fffffff;
    __syncthreads();
    float before = 0.f;
    for (int w = 0; w < warp; ++w) before += fscratch[w];
    float run = before + (incl - mine);
    if (threadIdx.x == 0 || run < target) {
        // the crossing may lie in this range: walk it
        for (int i = lo; i < hi; ++i) {
            run += f(i);
            if (run >= target) { atomicMin(&iscratch[32], i); break; }
        }
    } else if (lo < hi) {
        // the sum before this range has reached the target already; if rounding kept the
        // owner of the crossing from seeing it, this range's first index stands in
        atomicMin(&iscratch[32], lo);
    }
    __syncthreads();
    const int r = iscratch[32];
    __syncthreads();
    return r == 0x7fffffff ? -1 : r;
}

struct SampleParams {
    const float* logits;          // [rows, vocab], not modified
    float* work;                  // [rows, vocab] scratch
    const float* temperature;     // per row; <= 0: argmax
    const int* top_k;             // per row; 0: off
    const float* top_p;           // per row; >= 1: off
    const float* min_p;           // per row; <= 0: off
    const float* repetition_penalty;  // per row; 1: off
    const int* context;           // tokens of all rows, row r at [context_offsets[r], context_offsets[r+1])
    const int* context_offsets;   // the window (`repeat_last_n`) is applied by the caller
    unsigned long long* rng_state;    // per row, advanced once per multinomial draw
    int* out_tokens;              // [rows]
    int vocab;
};

__global__ void __launch_bounds__(THREADS) sample_kernel(const SampleParams p) {
    __shared__ float fs[33];
    __shared__ int is[33];
    __shared__ int hist[256];
    const int r = blockIdx.x;
    const int V = p.vocab;
    const float* in = p.logits + (size_t)r * V;
    float* l = p.work + (size_t)r * V;
    const float T = p.temperature[r];

    for (int i = threadIdx.x; i < V; i += THREADS) l[i] = in[i];
    __syncthreads();
    const float pen = p.repetition_penalty ? p.repetition_penalty[r] : 1.f;
    if (fabsf(pen - 1.f) >= 1.1920929e-07f && p.context) {
        // every occurrence writes the same function of the unmodified logit
        for (int i = p.context_offsets[r] + threadIdx.x; i < p.context_offsets[r + 1]; i += THREADS) {
            const int tok = p.context[i];
            if (tok >= 0 && tok < V) { const float v = in[tok]; l[tok] = v > 0.f ? v / pen : v * pen; }
        }
        __syncthreads();
    }
    if (T > 0.f)
        for (int i = threadIdx.x; i < V; i += THREADS) l[i] = l[i] / T;
    __syncthreads();

    const float minp = p.min_p ? p.min_p[r] : 0.f;
    if (minp > 0.f) {
        float mx = -INFINITY;
        for (int i = threadIdx.x; i < V; i += THREADS) mx = fmaxf(mx, l[i]);
        mx = block_max(mx, fs);
        const float thresh = mx + logf(minp);
        for (int i = threadIdx.x; i < V; i += THREADS) if (l[i] < thresh) l[i] = -INFINITY;
        __syncthreads();
    }

    const int k = p.top_k ? p.top_k[r] : 0;
    if (k > 0 && k < V) {
        // k-th largest key by radix selection, 8 bits a pass
        unsigned prefix = 0, mask = 0;
        int remaining = k;
        for (int shift = 24; shift >= 0; shift -= 8) {
            for (int b = threadIdx.x; b < 256; b += THREADS) hist[b] = 0;
            __syncthreads();
            for (int i = threadIdx.x; i < V; i += THREADS) {
                const unsigned key = order_key(l[i]);
                if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255], 1);
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                int b = 255, rem = remaining;
                for (; b > 0; --b) { if (hist[b] >= rem) break; rem -= hist[b]; }
                is[0] = b; is[1] = rem;
            }
            __syncthreads();
            prefix |= (unsigned)is[0] << shift;
            mask |= 255u << shift;
            remaining = is[1];
            __syncthreads();
        }
        for (int i = threadIdx.x; i < V; i += THREADS) if (order_key(l[i]) < prefix) l[i] = -INFINITY;
        __syncthreads();
    }

    float mx = -INFINITY;
    for (int i = threadIdx.x; i < V; i += THREADS) mx = fmaxf(mx, l[i]);
    mx = block_max(mx, fs);

    const float topp = p.top_p ? p.top_p[r] : 1.f;
    if (topp < 1.f && mx > -INFINITY) {
        float tot = 0.f;
        for (int i = threadIdx.x; i < V; i += THREADS) tot += expf(l[i] - mx);
        tot = block_sum(tot, fs);
        const float want = topp * tot;
        // largest key K with mass(key >= K) >= want, by bisection on the key bits
        unsigned K = 0;
        for (int bit = 31; bit >= 0; --bit) {
            const unsigned cand = K | (1u << bit);
            float m = 0.f;
            for (int i = threadIdx.x; i < V; i += THREADS) if (order_key(l[i]) >= cand) m += expf(l[i] - mx);
            m = block_sum(m, fs);
            if (m >= want) K = cand;
        }
        float above = 0.f, tie_mass = 0.f, ties = 0.f;
        for (int i = threadIdx.x; i < V; i += THREADS) {
            const unsigned key = order_key(l[i]);
            if (key > K) above += expf(l[i] - mx);
            else if (key == K) { ties += 1.f; tie_mass = expf(l[i] - mx); }
        }
        above = block_sum(above, fs);
        ties = block_sum(ties, fs);
        tie_mass = block_max(tie_mass, fs);
        // of equal logits at the cut, the sorted order keeps the lower indices first
        float keep = tie_mass > 0.f ? ceilf((want - above) / tie_mass) : ties;
        keep = fminf(fmaxf(keep, 1.f), ties);
        int last_tie = V;
        if (keep < ties) {
            auto is_tie = [&](int i) { return order_key(l[i]) == K ? 1.f : 0.f; };
            last_tie = block_first_reaching(V, keep, is_tie, fs, is);
        }
        for (int i = threadIdx.x; i < V; i += THREADS) {
            const unsigned key = order_key(l[i]);
            if (key < K || (key == K && i > last_tie)) l[i] = -INFINITY;
        }
        __syncthreads();
    }

    int token;
    if (T <= 0.f) {
        token = block_argmax_last(l, V, fs, is);
    } else {
        unsigned long long s = p.rng_state[r];
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        const float u = (float)(s >> 33) / 2147483648.0f;
        float tot = 0.f;
        for (int i = threadIdx.x; i < V; i += THREADS) tot += expf(l[i] - mx);
        tot = block_sum(tot, fs);
        const float target = u * tot;
        auto mass = [&](int i) { return expf(l[i] - mx); };
        token = block_first_reaching(V, target, mass, fs, is);
        if (token < 0) token = block_argmax_last(l, V, fs, is);
        if (threadIdx.x == 0) p.rng_state[r] = s;
    }
    if (threadIdx.x == 0) p.out_tokens[r] = token;
}

// ---------------------------------------------------------------------------------
// The same pipeline with a row spread over a cluster of CL blocks.  Block `rank` holds the elements
// [rank * per, rank * per + per) of the row in shared memory.  Whatever the blocks must agree on goes
// through `Shared::pub`: every block publishes one value (or its histogram), the cluster meets at a
// barrier, every block reads all CL values through distributed shared memory and combines them in
// rank order.  Two sets of slots are used in turn, so one barrier per exchange is enough: a block
// that writes a set again has passed the barrier of the exchange between, which every block reaches
// only after it has read the set.
// ---------------------------------------------------------------------------------
constexpr int CL = 8;
constexpr int CLUSTER_MAX_PER_BLOCK = 49152;                 // floats of a row a block can hold (192 KiB)

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned cl_load_u32(const void* own_smem, unsigned rank) {
    unsigned addr = (unsigned)__cvta_generic_to_shared(own_smem), remote, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(remote) : "memory");
    return v;
}

// A block of the cluster has 512 threads: two blocks a multiprocessor with 64 registers a thread hold 32 rows of 202,048 logits at once
// (256 blocks).  The order of every sum is that of 1,024 threads: a thread adds up the elements of two of them, its own and its own + 512.
constexpr int ST = 512;
constexpr int BINS = 2048;                                   // bins of a narrowing pass, four a thread
constexpr int LIST = 1024;                                   // candidates that are sorted, two a thread
constexpr int NARROWINGS = 4;
constexpr int CUT_TRIES = 6;
static_assert(BINS == 4 * ST && LIST == 2 * ST && THREADS == 2 * ST && ST / 64 == CL, "shares of a thread, of a warp");

struct ClusterShared {
    float fs[33];
    int is[33];
    float parts[2][32];
    float sums_pub[2][2], sums[2];
    unsigned pub[2][2];           // two sets of two published words (a value, an index)
    int turn;                     // which set the next exchange uses (the same in every block)
    int n_list;
    int found[3];                 // what the threads of a narrowing pass find: first bin, last bin, elements in them
    float scan[2][ST / 32];
    __align__(16) unsigned hist[BINS];    // bins of a pass; the row's candidates; counts of the radix selection and what it publishes
    __align__(16) unsigned list[LIST];    // keys of this block's candidates
};

// All of a block's shared memory; the functions below name it themselves, so that they address it as shared memory.
extern __shared__ __align__(16) unsigned char sample_shared[];
#define sh (*reinterpret_cast<ClusterShared*>(sample_shared))
static_assert(sizeof(ClusterShared) % 16 == 0, "the row behind it is copied 16 bytes at a time");
__device__ __forceinline__ float* row_shared() { return reinterpret_cast<float*>(sample_shared + sizeof(ClusterShared)); }

// Two words of every block: lane q (of every warp of every block) receives those of block q & 7.
__device__ __noinline__ uint2 cl_exchange(unsigned mine0, unsigned mine1) {
    const int t = sh.turn;
    __syncthreads();                                         // everyone has read `turn` (and the last results)
    if (threadIdx.x == 0) { sh.pub[t][0] = mine0; sh.pub[t][1] = mine1; sh.turn = t ^ 1; }
    cl_sync();
    const unsigned q = threadIdx.x & (CL - 1);
    return make_uint2(cl_load_u32(&sh.pub[t][0], q), cl_load_u32(&sh.pub[t][1], q));
}

// Two sums over the row (every thread of every block receives them): the elements of each of 1,024 threads in ascending order (a0, b0:
// of the first 512, a1, b1: of the others), the threads of a warp, the 32 warps, the blocks by rank.
__device__ __forceinline__ float2 cl_sums(float a0, float a1, float b0, float b1) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = sh.turn;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        b0 += __shfl_xor_sync(0xffffffffu, b0, o);
        b1 += __shfl_xor_sync(0xffffffffu, b1, o);
    }
    __syncthreads();                                         // everyone has read `turn` and the last results
    if (lane == 0) {
        sh.parts[0][warp] = a0;
        sh.parts[0][warp + ST / 32] = a1;
        sh.parts[1][warp] = b0;
        sh.parts[1][warp + ST / 32] = b1;
    }
    if (threadIdx.x == 0) sh.turn = t ^ 1;
    __syncthreads();
    float x = warp_sum(sh.parts[warp & 1][lane]);
    if (lane == 0 && warp < 2) sh.sums_pub[t][warp] = x;
    cl_sync();
    // a lane for each sum of each block
    const float of = __uint_as_float(cl_load_u32(&sh.sums_pub[t][(lane >> 3) & 1], lane & (CL - 1)));
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < CL; ++r) { sum.x += __shfl_sync(0xffffffffu, of, r); sum.y += __shfl_sync(0xffffffffu, of, 8 + r); }
    return sum;
}

__device__ __forceinline__ void clear_bins() { reinterpret_cast<uint4*>(sh.hist)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u); }

__device__ __forceinline__ unsigned key_of_bits(unsigned u) { return u ^ ((unsigned)((int)u >> 31) | 0x80000000u); }

__device__ __forceinline__ float key_value(unsigned key) {
    return __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
}

// This block's part of the row in shared memory.  PAD: a thread's share of it (see cl_first_reaching) is an even number of elements, and an
// unused word behind every 32 keeps the lanes' shares in different banks.
template <int PAD>
struct Part {
    int n, lo;
    __device__ __forceinline__ float& operator[](int i) const { return row_shared()[PAD ? i + (i >> 5) : i]; }
    // f(index, address, element, 0 or 1: which of the thread's two sums) over the thread's elements in ascending order for each of the two;
    // of BATCH elements, read together, that are all below `least` none is looked at.
    static constexpr int BATCH = 4, STEP = ST + PAD * (ST / 32);
    template <typename F>
    __device__ __forceinline__ void each(float least, F f) const {
        float* x = row_shared() + threadIdx.x + PAD * (threadIdx.x >> 5);
        const int whole = n / (BATCH * ST);
#pragma unroll 2
        for (int m = 0; m < whole; ++m) {
            float v[BATCH], top = -INFINITY;
#pragma unroll
            for (int j = 0; j < BATCH; ++j) { v[j] = x[j * STEP]; top = fmaxf(top, v[j]); }
            if (!(top < least))
#pragma unroll
                for (int j = 0; j < BATCH; ++j) f((BATCH * m + j) * ST + (int)threadIdx.x, x + j * STEP, v[j], j & 1);
            x += BATCH * STEP;
        }
        const int i = BATCH * ST * whole + threadIdx.x;
#pragma unroll
        for (int j = 0; j < BATCH; ++j) if (i + j * ST < n) f(i + j * ST, x + j * STEP, x[j * STEP], j & 1);
    }
    // The same over all elements, with their keys: for rows with numbers that are not finite and for cuts at zero (whose signs a
    // comparison of numbers does not tell apart).  Read as integers: a NaN keeps its bits.
    template <typename F>
    __device__ __forceinline__ void each_key(F f) const {
        unsigned* x = reinterpret_cast<unsigned*>(row_shared()) + threadIdx.x + PAD * (threadIdx.x >> 5);
#pragma unroll 1
        for (int i = threadIdx.x; i < n; i += 2 * ST, x += 2 * STEP) {
            f(i, reinterpret_cast<float*>(x), __uint_as_float(x[0]), key_of_bits(x[0]), 0);
            if (i + ST < n) f(i + ST, reinterpret_cast<float*>(x + STEP), __uint_as_float(x[STEP]), key_of_bits(x[STEP]), 1);
        }
    }
};

// Divides the elements by `by` (1: as they are); their maximum, and whether there is a NaN among them.
template <int PAD>
__device__ __forceinline__ float row_max(const Part<PAD> row, float by, bool& nan) {
    float mx = -INFINITY;
    int bad = 0;
    row.each(-INFINITY, [&](int, float* at, float x, int) {
        x /= by;
        *at = x;
        mx = fmaxf(mx, x);
        bad |= x != x;
    });
    mx = warp_max(mx);
    bad = __syncthreads_or(bad);
    if ((threadIdx.x & 31) == 0) sh.fs[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = warp_max(sh.fs[threadIdx.x & (ST / 32 - 1)]);
    const uint2 all = cl_exchange(__float_as_uint(mx), (unsigned)bad);
    nan = __any_sync(0xffffffffu, all.y != 0u);
    return warp_max(__uint_as_float(all.x));
}

// A narrowing pass's bins: bin b holds the elements whose distance d = mx - x from the row's maximum rounds to b steps of 1 / scale from
// lo.  An element's bin never falls as the element falls; below 0 are the elements above the bins, from BINS on those below.
struct Bins {
    float lo, scale;                                         // scale: a power of two
    __host__ __device__ __forceinline__ int of(float d) const {
        // The integer part of 2^23 + t stands in the low bits; more than 2^23 steps above the bins the sum is negative, whose bits
        // would be a number above all others.
        const float sum = fmaxf(fmaf(d - lo, scale, 8388608.f), 0.f);
#ifdef __CUDA_ARCH__
        const unsigned bits = __float_as_uint(sum);
#else
        unsigned bits;
        memcpy(&bits, &sum, sizeof bits);
#endif
        return (int)(bits - 0x4b000000u);
    }
};

// One pass over the row: the masses (ONES: the numbers) of the elements above `high`, and from `low` on; low <= high.  BIN: the elements
// from `low` on are counted into the bins, and those above the bins are summed in the place of those above `high`.  LISTED: the keys of
// the elements from `low` to `high` are listed.
constexpr int BIN = 1, LISTED = 2, ONES = 4;
template <int WHAT, int PAD>
__device__ __forceinline__ float2 masses(const Part<PAD> row, float mx, float low, float high, Bins bins) {
    float above[2] = {0.f, 0.f}, from[2] = {0.f, 0.f};
    row.each(low, [&](int, float*, float x, int h) {
        const float d = mx - x, e = WHAT & ONES ? 1.f : expf(-d);
        if (x >= low) from[h] += e;
        if (WHAT & BIN) {
            const int b = bins.of(d);
            if (x >= low && b < 0) above[h] += e;
            if (x >= low && (unsigned)b < BINS) atomicAdd(&sh.hist[b], 1u);
        } else {
            if (x > high) above[h] += e;
        }
        if ((WHAT & LISTED) && x >= low && x <= high) {
            const int at = atomicAdd(&sh.n_list, 1);
            if (at < LIST) sh.list[at] = key_of_bits(__float_as_uint(x));
        }
    });
    return cl_sums(above[0], above[1], from[0], from[1]);
}
// The masses (ones: the numbers) of the elements with keys above `high`, and from `low` on, of those with keys of at least `floor`.
template <int PAD>
__device__ __noinline__ float2 masses_by_key(const Part<PAD> row, float mx, unsigned floor, unsigned low, unsigned high, bool ones) {
    float above[2] = {0.f, 0.f}, from[2] = {0.f, 0.f};
    row.each_key([&](int, float*, float x, unsigned key, int h) {
        const float e = key >= floor && key >= low ? (ones ? 1.f : expf(x - mx)) : 0.f;
        from[h] += e;
        above[h] += key > high ? e : 0.f;
    });
    return cl_sums(above[0], above[1], from[0], from[1]);
}

// The sum over the warps before this one.
__device__ __forceinline__ float warps_before(const float (&of_warp)[ST / 32]) {
    const int lane = threadIdx.x & 31;
    return warp_sum(lane < (threadIdx.x >> 5) ? of_warp[lane & (ST / 32 - 1)] : 0.f);
}

// Reads the bins of all blocks (they are complete and the cluster has met since) and finds the bins [first, last] of which one holds the
// cut: the element at which the count from the top reaches `want`, or (by_mass) the mass does, `base` being what lies above the first
// bin.  The mass of a bin is known between its count times the masses of its edges.  False if no bin reaches it.
__device__ __forceinline__ bool find_bins(const Bins bins, bool by_mass, float want, float base, int& first, int& last,
                                          int& count) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b0 = 4 * threadIdx.x;
    unsigned v[CL][4];
#pragma unroll
    for (int r = 0; r < CL; ++r) {
        unsigned addr = (unsigned)__cvta_generic_to_shared(&sh.hist[b0]), remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(addr), "r"(r));
        asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];\n"
                     : "=r"(v[r][0]), "=r"(v[r][1]), "=r"(v[r][2]), "=r"(v[r][3]) : "r"(remote) : "memory");
    }
    if (threadIdx.x == 0) { sh.found[0] = sh.found[1] = BINS; sh.found[2] = 0; sh.n_list = 0; }
    // upper and lower bound of the thread's mass (or its count, twice), and their sums over the threads before
    const float slack = by_mass ? 1e-5f : 0.f;               // far above what d, expf and these sums round off (4e-6)
    const float width = 1.f / bins.scale;
    float edge = by_mass ? expf(-(bins.lo + ((float)b0 - 0.5f) * width)) : 1.f, up[4], low[4];
    const float fall = by_mass ? expf(-width) : 1.f;
    int c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        c[j] = 0;
#pragma unroll
        for (int r = 0; r < CL; ++r) c[j] += (int)v[r][j];
        up[j] = (float)c[j] * edge * (1.f + slack);
        edge *= fall;
        low[j] = (float)c[j] * edge * (1.f - slack);
        if (j) { up[j] += up[j - 1]; low[j] += low[j - 1]; }
    }
    float su = up[3], sl = low[3];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float tu = __shfl_up_sync(0xffffffffu, su, o), tl = __shfl_up_sync(0xffffffffu, sl, o);
        if (lane >= o) { su += tu; sl += tl; }
    }
    if (lane == 31) { sh.scan[0][warp] = su; sh.scan[1][warp] = sl; }
    __syncthreads();
    const float pu = base * (1.f + slack) + warps_before(sh.scan[0]) + (su - up[3]), pl = base * (1.f - slack) + warps_before(sh.scan[1]) + (sl - low[3]);
    // a thread's first bins with elements that reach the goal
    int f = BINS, g = BINS;
#pragma unroll
    for (int j = 3; j >= 0; --j) {
        if (c[j] && pu + up[j] >= want * (1.f - slack)) f = b0 + j;
        if (c[j] && pl + low[j] >= want * (1.f + slack)) g = b0 + j;
    }
    f = __reduce_min_sync(0xffffffffu, f);
    g = __reduce_min_sync(0xffffffffu, g);
    if (lane == 0) { atomicMin(&sh.found[0], f); atomicMin(&sh.found[1], g); }
    __syncthreads();
    first = sh.found[0];
    last = sh.found[1];
    int mine = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) if (b0 + j >= first && b0 + j <= last) mine += c[j];
    if (mine) atomicAdd(&sh.found[2], mine);
    __syncthreads();
    count = sh.found[2];
    return first <= last && last < BINS;
}

// The candidates of all blocks, sorted in descending order into sh.hist (the cluster has met since they were listed); their number, or
// LIST + 1 if they are more than LIST.
__device__ __forceinline__ int gather_sorted() {
    unsigned* const c = sh.hist;
    // two warps a block of the cluster; each sums up the counts of the blocks before its own
    const int lane = threadIdx.x & 31, of = threadIdx.x >> 6;
    const int n_lane = lane < CL ? (int)cl_load_u32(&sh.n_list, lane) : 0;
    const int count = __reduce_add_sync(0xffffffffu, n_lane), at = __reduce_add_sync(0xffffffffu, lane < of ? n_lane : 0);
    const int n = __shfl_sync(0xffffffffu, n_lane, of);
    if (count > LIST) return LIST + 1;
    int size = 64;
#pragma unroll 1
    while (size < count) size <<= 1;
#pragma unroll 1
    for (int j = threadIdx.x & 63; j < n; j += 64) c[at + j] = cl_load_u32(&sh.list[j], of);
#pragma unroll 1
    for (int j = count + threadIdx.x; j < size; j += ST) c[j] = 0u;
    __syncthreads();
    // bitonic: a thread compares one pair a step; pairs at most 32 apart stay within 64 elements, which are one warp's
#pragma unroll 1
    for (int k = 2; k <= size; k <<= 1) {
#pragma unroll 1
        for (int s = k >> 1; s > 0; s >>= 1) {
            const int i = 2 * threadIdx.x - (threadIdx.x & (s - 1));
            if (i + s < size) {
                const unsigned x = c[i], y = c[i + s];
                if ((x < y) == ((i & k) == 0)) { c[i] = y; c[i + s] = x; }
            }
            if (s > 32 || (s == 1 && k >= 64)) __syncthreads(); else __syncwarp();
        }
    }
    __syncthreads();
    return count;
}

// First index of the sorted keys (of `count`) at which base + the running sum of their masses reaches `want`; count - 1 if none does.
__device__ __forceinline__ int first_by_mass(int count, float mx, float base, float want) {
    const int lane = threadIdx.x & 31, i = 2 * threadIdx.x;
    const float a = i < count ? expf(key_value(sh.hist[i]) - mx) : 0.f, b = i + 1 < count ? expf(key_value(sh.hist[i + 1]) - mx) : 0.f;
    float s = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += t;
    }
    if (lane == 31) sh.scan[0][threadIdx.x >> 5] = s;
    if (threadIdx.x == 0) sh.found[0] = count - 1;
    __syncthreads();
    const float p = base + warps_before(sh.scan[0]) + (s - (a + b));
    if (i < count && p + a >= want) atomicMin(&sh.found[0], i);
    else if (i + 1 < count && p + a + b >= want) atomicMin(&sh.found[0], i + 1);
    __syncthreads();
    return sh.found[0];
}

// A search for the cut of a row whose maximum is mx (a finite number, and there is no NaN): of the elements from `floor` on, the one at which
// the count from the top reaches k, or (k = 0) the mass reaches want = topp * the mass of all of them.
struct Found {
    int count;                    // candidates: their keys stand sorted in sh.hist, downwards; 0: they were not found
    float above, want;            // what lies above them: elements or mass
    float low, high;              // where they were not found: the cut should lie between these
};
template <bool MASS, int PAD>
__device__ __forceinline__ Found narrow(const Part<PAD> row, float mx, float floor, int k, float topp) {
    Bins bins{0.f, 128.f};
    constexpr int what = MASS ? 0 : ONES;
    Found found{0, 0.f, (float)k, -INFINITY, INFINITY};
    const float& want = found.want;
    int before = 0;
#pragma unroll 1
    for (int round = 0; round < NARROWINGS; ++round) {
        if (round) {
            cl_sync();                                       // the others have read the bins
            clear_bins();
            __syncthreads();
        }
        const float2 sum = masses<BIN | what>(row, mx, floor, 0.f, bins);
        if (MASS && !round) found.want = topp * sum.y;
        if (!(want > 0.f)) break;
        int first, last, count;
        if (!find_bins(bins, MASS, want, sum.x, first, last, count)) {
            if (round) break;
            bins.scale = 8.f;                                // the cut is further down than 16 from the maximum
            continue;
        }
        // from edge to edge of these bins and a little beyond: what the distances were rounded by
        const float lo = bins.lo + ((float)first - 0.5f) / bins.scale, hi = bins.lo + ((float)last + 0.5f) / bins.scale;
        const float more = 1e-6f * (fabsf(mx) + hi);
        found.low = fmaxf(floor, mx - hi - more);
        found.high = fmaxf(found.low, mx - lo + more);
        if (count <= LIST * 7 / 8) {
            found.above = masses<LISTED | what>(row, mx, found.low, found.high, bins).x;
            count = gather_sorted();
            found.count = count <= LIST ? count : 0;
            break;
        }
        if (count == before) break;                          // equal logits: narrower bins do not part them
        before = count;
        bins.lo = lo;
#pragma unroll 1
        for (int wide = last - first + 1; wide * 2 <= BINS - 2; wide *= 2) bins.scale *= 2.f;
    }
    return found;
}

// Largest key K with mass(key >= K) >= want, two bits of it at a time.  For rows whose cut the narrowing passes do not find (many equal logits around
// it, numbers that are not finite).
template <int PAD>
__device__ __noinline__ unsigned cut_by_bits(const Part<PAD> row, float mx, float want, unsigned floor, float low, float high) {
    unsigned K = 0u;
    int shift = 30;
    // if the cut does lie from `low` to `high`, the bits that these have in common are known
    if (low > -INFINITY && high < INFINITY && low != 0.f && high != 0.f) {
        const unsigned a = key_of_bits(__float_as_uint(low)), b = key_of_bits(__float_as_uint(high));
        const float2 m = masses_by_key(row, mx, floor, a, b, false);
        if (m.y >= want && m.x < want) {
            shift = a == b ? 0 : (31 - __clz(a ^ b)) / 2 * 2;
            K = a & ~((4u << shift) - 1u);
        }
    }
#pragma unroll 1
    for (; shift >= 0; shift -= 2) {
        // a pass gives the masses from two of the three values on that the next two bits can have; the third is asked for where it decides
        const unsigned c1 = K | (1u << shift), c2 = K | (2u << shift), c3 = K | (3u << shift);
        const float2 m = masses_by_key(row, mx, floor, c1, c2 - 1u, false);
        if (m.x >= want) K = masses_by_key(row, mx, floor, c3, 0xffffffffu, false).y >= want ? c3 : c2;
        else if (m.y >= want) K = c1;
    }
    return K;
}

// The k-th largest key by radix selection, 8 bits a pass; the histograms of the blocks are added.
template <int PAD>
__device__ __noinline__ unsigned kth_by_bits(const Part<PAD> row, int k) {
    unsigned* const hist = sh.hist;
    unsigned prefix = 0, mask = 0;
    int remaining = k;
    cl_sync();                                               // the others may still read the bins of a narrowing pass
#pragma unroll 1
    for (int shift = 24; shift >= 0; shift -= 8) {
        if (threadIdx.x < 256) hist[threadIdx.x] = 0;
        __syncthreads();
        row.each_key([&](int, float*, float, unsigned key, int) {
            if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255], 1u);
        });
        __syncthreads();
        const int t = sh.turn;
        unsigned* const pub = hist + 256 + 256 * t;
        if (threadIdx.x < 256) pub[threadIdx.x] = hist[threadIdx.x];
        __syncthreads();
        if (threadIdx.x == 0) sh.turn = t ^ 1;
        cl_sync();
        if (threadIdx.x < 256) {
            unsigned total = 0;
#pragma unroll
            for (int q = 0; q < CL; ++q) total += cl_load_u32(&pub[threadIdx.x], q);
            hist[threadIdx.x] = total;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int b = 255, rem = remaining;
            for (; b > 0; --b) { if ((int)hist[b] >= rem) break; rem -= (int)hist[b]; }
            sh.is[0] = b; sh.is[1] = rem;
        }
        __syncthreads();
        prefix |= (unsigned)sh.is[0] << shift;
        mask |= 255u << shift;
        remaining = sh.is[1];
        __syncthreads();
    }
    cl_sync();                                               // ... and what was published here, before the bins are used again
    return prefix;
}

// What of the row is kept: the elements above the key K and those of the key K up to the global index `last_tie`, if their key is at
// least `floor`.
struct Kept {
    unsigned floor, K;
    int last_tie;
    __device__ __forceinline__ bool has(unsigned key, int i) const { return key >= floor && (key > K || (key == K && i <= last_tie)); }
};
template <int PAD>
__device__ __noinline__ float kept_mass(const Part<PAD> row, float mx, const Kept kept) {
    float s[2] = {0.f, 0.f};
    row.each_key([&](int i, float*, float x, unsigned key, int h) { if (kept.has(key, row.lo + i)) s[h] += expf(x - mx); });
    return cl_sums(s[0], s[1], 0.f, 0.f).x;
}
// First global index (ascending) at which the running sum of f over the row reaches `target`; -1 if never.  Each of 1,024 threads
// owns a contiguous range, a thread here the ranges of two.
template <int PAD, typename F>
__device__ __forceinline__ int cl_first_reaching(const Part<PAD> row, float target, F f) {
    const int chunk = (row.n + THREADS - 1) / THREADS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float mine[2], incl[2];
    const int lo0 = min(row.n, (int)threadIdx.x * chunk), hi0 = min(row.n, lo0 + chunk);
    const int lo1 = min(row.n, ((int)threadIdx.x + ST) * chunk), hi1 = min(row.n, lo1 + chunk);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        mine[h] = 0.f;
        const int hi = h ? hi1 : hi0;
#pragma unroll 4
        for (int i = h ? lo1 : lo0; i < hi; ++i) mine[h] += f(i);
    }
    incl[0] = mine[0];
    incl[1] = mine[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t0 = __shfl_up_sync(0xffffffffu, incl[0], o), t1 = __shfl_up_sync(0xffffffffu, incl[1], o);
        if (lane >= o) { incl[0] += t0; incl[1] += t1; }
    }
    __syncthreads();
    if (lane == 31) { sh.fs[warp] = incl[0]; sh.fs[warp + ST / 32] = incl[1]; }
    if (threadIdx.x == 0) sh.is[32] = 0x7fffffff;
    __syncthreads();
    float before[2] = {0.f, 0.f}, block_total = 0.f;
#pragma unroll 4
    for (int w = 0; w < (THREADS >> 5); ++w) {
        const float x = sh.fs[w];
        if (w == warp) before[0] = block_total;
        if (w == warp + ST / 32) before[1] = block_total;
        block_total += x;
    }
    // the sums of the blocks before this one, in rank order
    const float of_block = __uint_as_float(cl_exchange(__float_as_uint(block_total), 0u).x);
    float base = 0.f;
    const unsigned rank = cl_rank();
#pragma unroll
    for (int r = 0; r < CL; ++r) {
        const float x = __shfl_sync(0xffffffffu, of_block, r);
        if ((unsigned)r < rank) base += x;
    }
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const int lo = h ? lo1 : lo0, hi = h ? hi1 : hi0;
        const float own = h ? mine[1] : mine[0];
        float run = base + (h ? before[1] : before[0]) + ((h ? incl[1] : incl[0]) - own);
        if ((rank == 0 && threadIdx.x == 0 && h == 0) || run < target) {
            // the crossing may lie in this range: walk it, unless its sum falls short by more than the walk could round off
            if (!((run + own) * (1.f + 1e-4f) < target))
#pragma unroll 1
                for (int i = lo; i < hi; ++i) {
                    run += f(i);
                    if (run >= target) { atomicMin(&sh.is[32], row.lo + i); break; }
                }
        } else if (lo < hi) {
            // the sum before this range has reached the target already; if rounding kept the owner of the
            // crossing from seeing it, this range's first index stands in
            atomicMin(&sh.is[32], row.lo + lo);
        }
    }
    __syncthreads();
    const int r = __reduce_min_sync(0xffffffffu, (int)cl_exchange((unsigned)sh.is[32], 0u).x);
    return r == 0x7fffffff ? -1 : r;
}

// Twice what cl_first_reaching is called with where more than a smallest element decides what is kept: the kept masses, or (ties) the
// elements of the key K, one each.
template <int PAD>
__device__ __noinline__ int first_reaching_kept(const Part<PAD> row, float target, float mx, const Kept kept, bool ties) {
    return cl_first_reaching(row, target, [&](int i) {
        const float x = row[i], e = ties ? 1.f : expf(x - mx);
        const unsigned key = key_of_bits(__float_as_uint(x));
        return kept.has(key, row.lo + i) && (key == kept.K || !ties) ? e : 0.f;
    });
}

// The row's largest element (of equal ones the last), after what is not kept has been set to -infinity.
template <int PAD>
__device__ __noinline__ int row_argmax_last(const Part<PAD> row, const Kept kept) {
    row.each_key([&](int i, float* at, float, unsigned key, int) {
        if (!kept.has(key, row.lo + i)) *at = -INFINITY;
    });
    float best2[2] = {-INFINITY, -INFINITY}, best;
    int idx2[2] = {-1, -1}, idx;
    row.each_key([&](int i, float*, float v, unsigned, int h) {
        if (v > best2[h] || (v == best2[h] && i > idx2[h]) || idx2[h] < 0) { best2[h] = v; idx2[h] = i; }
    });
    auto of_warp = [&](float& bv, int& bi) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (oi >= 0 && (bi < 0 || ov > bv || (ov == bv && oi > bi))) { bv = ov; bi = oi; }
        }
    };
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        of_warp(best2[h], idx2[h]);
        if ((threadIdx.x & 31) == 0) { sh.fs[(threadIdx.x >> 5) + h * (ST / 32)] = best2[h]; sh.is[(threadIdx.x >> 5) + h * (ST / 32)] = idx2[h]; }
    }
    __syncthreads();
    best = sh.fs[threadIdx.x & 31];
    idx = sh.is[threadIdx.x & 31];
    of_warp(best, idx);
    const uint2 all = cl_exchange(__float_as_uint(best), (unsigned)(idx >= 0 ? row.lo + idx : -1));
    float bv = -INFINITY;
    int bi = -1;
#pragma unroll
    for (int q = 0; q < CL; ++q) {                               // ties go to the highest index: later ranks win
        const float v = __uint_as_float(__shfl_sync(0xffffffffu, all.x, q));
        const int i = (int)__shfl_sync(0xffffffffu, all.y, q);
        if (i >= 0 && (bi < 0 || v >= bv)) { bv = v; bi = i; }
    }
    return bi;
}

// What bounds it: passes over the row's part in shared memory (25,280 elements a block for 202,048 logits, an expf each in four of them),
// the cluster's barriers, and the fetching of code that runs once.  So the cuts of top-k and top-p are found from one histogram each: the
// bin of an element is its distance from the maximum in steps of 1/128, the counts of the bins bound the masses, and only the few
// hundred elements of the bins that can hold the cut are sorted and summed.  What is found that way is then proved: the masses above and from the
// cut on are summed in the order of every other sum of the row and must enclose the wanted mass, else the next candidate is tried.
// So the cut, and with it the token, is the one that the search bit by bit (cut_by_bits) would give.  Where the bins are still too full
// after NARROWINGS passes, that search runs.
// Measured against the form before (1,024 threads; top-p's cut in eleven passes of seven sums, top-k's in four of 256 counts), us: 32 rows of
// 202,048 logits with top-p, every second with top-k 40, 167 -> 63, top-p alone 211 -> 69, neither 37 -> 32; 8 rows 91 -> 42; one 68 -> 33;
// 32 rows of 32,768 88 -> 44; 32 rows of equal logits 219 -> 167.  With one histogram for counts and the elements' keys compared as integers
// 91 (twice the instructions); with four elements a batch not read ahead 102.
template <int PAD>
__global__ void __launch_bounds__(ST, 2) sample_cluster_kernel(const SampleParams p, const int per) {
    const unsigned rank = cl_rank();
    const int r = blockIdx.x / CL;
    const int V = p.vocab;
    Part<PAD> row;
    row.lo = (int)rank * per;
    row.n = max(0, min(per, V - row.lo));
    const int n = row.n, lo = row.lo;
    const float* in = p.logits + (size_t)r * V;
    // 16 bytes a copy where the row and its part's layout allow it
    if (!PAD && n % 4 == 0 && ((uintptr_t)(in + lo) & 15) == 0) {
#pragma unroll 4
        for (int i = threadIdx.x * 4; i < n; i += 4 * ST)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(&row_shared()[i])), "l"(in + lo + i));
    } else {
#pragma unroll 4
        for (int i = threadIdx.x; i < n; i += ST)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(&row[i])), "l"(in + lo + i));
    }
    if (threadIdx.x == 0) { sh.turn = 0; sh.n_list = 0; }
    clear_bins();
    const float T = p.temperature[r];
    const unsigned long long state = p.rng_state[r];
    const float pen = p.repetition_penalty ? p.repetition_penalty[r] : 1.f, minp = p.min_p ? p.min_p[r] : 0.f, topp = p.top_p ? p.top_p[r] : 1.f;
    const int k = p.top_k ? p.top_k[r] : 0;
    const bool penalty = fabsf(pen - 1.f) >= 1.1920929e-07f && p.context;
    int at = 0, end = 0, tok = -1;
    float of_tok = 0.f;
    if (penalty) {                                           // the thread's first token and its logit, while the row is on its way
        at = p.context_offsets[r] + threadIdx.x;
        end = p.context_offsets[r + 1];
        if (at < end) tok = p.context[at];
        if (tok >= lo && tok < lo + n) of_tok = in[tok];
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    if (penalty) {
        // every occurrence writes the same function of the unmodified logit
#pragma unroll 1
        while (at < end) {
            if (tok >= lo && tok < lo + n) row[tok - lo] = of_tok > 0.f ? of_tok / pen : of_tok * pen;
            at += ST;
            tok = at < end ? p.context[at] : -1;
            if (tok >= lo && tok < lo + n) of_tok = in[tok];
        }
        __syncthreads();
    }
    bool nan;
    float mx = row_max(row, T > 0.f ? T : 1.f, nan);         // (x / 1 is x)
    if (minp > 0.f) {
        const float thresh = mx + logf(minp);
        row.each_key([&](int, float* at, float x, unsigned, int) { if (x < thresh) *at = -INFINITY; });
        __syncthreads();
        if (minp >= 1.f) mx = row_max(row, 1.f, nan);        // (nothing may be left)
    }
    const bool plain = !nan && mx > -INFINITY && mx < INFINITY;

    Kept kept{0u, 0u, V};
    if (k > 0 && k < V) {
        Found found{0, 0.f, 0.f, 0.f, 0.f};
        if (plain && k < (1 << 24)) found = narrow<false>(row, mx, -INFINITY, k, 0.f);
        const int at_k = found.count ? k - (int)found.above - 1 : -1;
        if (at_k >= 0 && at_k < found.count) {
            kept.floor = sh.hist[at_k];
            __syncthreads();                                 // (read before the bins are cleared)
        } else {
            kept.floor = kth_by_bits(row, k);
        }
        clear_bins();
        __syncthreads();
        if (!plain) {                                        // a NaN alone may be left
            row.each_key([&](int, float* at, float, unsigned key, int) { if (key < kept.floor) *at = -INFINITY; });
            __syncthreads();
            mx = row_max(row, 1.f, nan);
        }
    }
    // the smallest element that is kept, where numbers tell what is kept and what is not
    float least = kept.floor ? key_value(kept.floor) : -INFINITY;
    bool simple = plain && least != 0.f;

    float tot = 0.f;
    bool have_tot = false;
    if (topp < 1.f && mx > -INFINITY) {
        Found found{0, 0.f, 0.f, -INFINITY, INFINITY};
        if (simple) found = narrow<true>(row, mx, least, 0, topp);
        float want = found.want;
        unsigned K = 0u;
        float2 at_cut;                                       // the masses above the cut and from it on
        bool proved = false;
        if (found.count) {
            int at = first_by_mass(found.count, mx, found.above, want);
#pragma unroll 1
            for (int t = 0; t < CUT_TRIES && !proved; ++t) {
                K = sh.hist[at];
                const float cut = key_value(K);
                if (cut == 0.f) break;
                at_cut = masses<0>(row, mx, cut, cut, Bins{0.f, 1.f});
                if (at_cut.x >= want) {                      // the cut is higher
                    while (at >= 0 && sh.hist[at] == K) --at;
                    if (at < 0) break;
                } else if (at_cut.y < want) {                // ... or lower
                    while (at < found.count && sh.hist[at] == K) ++at;
                    if (at >= found.count) break;
                } else {
                    proved = true;
                }
            }
        }
        float ties;
        if (proved) {                                        // they are all among the candidates
            const int i = 2 * threadIdx.x;
            ties = (float)(__syncthreads_count(i < found.count && sh.hist[i] == K) + __syncthreads_count(i + 1 < found.count && sh.hist[i + 1] == K));
            least = key_value(K);
        } else {
            simple = false;
            if (!(want > 0.f)) want = topp * masses_by_key(row, mx, kept.floor, 0u, 0xffffffffu, false).y;
            K = cut_by_bits(row, mx, want, kept.floor, found.low, found.high);
            at_cut = masses_by_key(row, mx, kept.floor, K, K, false);
            const float2 numbers = masses_by_key(row, mx, kept.floor, K, K, true);
            ties = numbers.y - numbers.x;
        }
        tot = at_cut.y;
        have_tot = true;
        kept.K = K;
        const float tie_mass = ties > 0.f ? expf(key_value(K) - mx) : 0.f;
        // of equal logits at the cut, the sorted order keeps the lower indices first
        float keep = tie_mass > 0.f ? ceilf((want - at_cut.x) / tie_mass) : ties;
        keep = fminf(fmaxf(keep, 1.f), ties);
        if (keep < ties) {
            kept.last_tie = first_reaching_kept(row, keep, mx, kept, true);
            simple = have_tot = false;
        }
    }

    int token;
    if (T <= 0.f) {
        token = row_argmax_last(row, kept);
    } else {
        const unsigned long long s = state * 6364136223846793005ull + 1442695040888963407ull;
        const float u = (float)(s >> 33) / 2147483648.0f;
        if (!have_tot) tot = simple ? masses<0>(row, mx, least, least, Bins{0.f, 1.f}).y : kept_mass(row, mx, kept);
        if (simple)
            token = cl_first_reaching(row, u * tot, [&](int i) { const float x = row[i], e = expf(x - mx); return x >= least ? e : 0.f; });
        else
            token = first_reaching_kept(row, u * tot, mx, kept, false);
        if (token < 0) token = row_argmax_last(row, kept);
        if (rank == 0 && threadIdx.x == 0) p.rng_state[r] = s;   // (every block has read the state before the cluster met)
    }
    if (rank == 0 && threadIdx.x == 0) p.out_tokens[r] = token;
    cl_sync();                                                   // no block leaves while another may still read its shared memory
}
#undef sh

__global__ void __launch_bounds__(THREADS) argmax_kernel(const float* logits, int vocab, int* out) {
    __shared__ float fs[33];
    __shared__ int is[33];
    const int idx = block_argmax_last(logits + (size_t)blockIdx.x * vocab, vocab, fs, is);
    if (threadIdx.x == 0) out[blockIdx.x] = idx;
}

// The same with a row spread over a cluster of CL blocks, an eighth each: one block alone reads a row of
// 202,048 logits in 25 us, which a decode step of one request would wait for.  The blocks' results meet in
// block 0 through distributed shared memory, in rank order, with the same rule for equal values.
__global__ void __launch_bounds__(THREADS) argmax_cluster_kernel(const float* logits, int vocab, int per, int* out) {
    __shared__ float fs[33];
    __shared__ int is[33];
    __shared__ unsigned pub[2];
    const unsigned rank = cl_rank();
    const int row = blockIdx.x / CL;
    const float* l = logits + (size_t)row * vocab;
    const int lo = min(vocab, (int)rank * per), n = min(vocab, lo + per) - lo;
    const int mine = n > 0 ? block_argmax_last(l + lo, n, fs, is) : -1;
    if (threadIdx.x == 0) {
        pub[0] = __float_as_uint(mine >= 0 ? l[lo + mine] : -INFINITY);
        pub[1] = (unsigned)(mine >= 0 ? lo + mine : -1);
    }
    cl_sync();
    if (rank == 0 && threadIdx.x == 0) {
        float best = -INFINITY;
        int idx = -1;
        for (unsigned r = 0; r < CL; ++r) {
            const float ov = __uint_as_float(cl_load_u32(&pub[0], r));
            const int oi = (int)cl_load_u32(&pub[1], r);
            if (oi >= 0 && (idx < 0 || ov > best || (ov == best && oi > idx))) { best = ov; idx = oi; }
        }
        out[row] = idx;
    }
    cl_sync();                                                   // no block leaves while block 0 may still read its shared memory
}

}  // namespace

SPITE_API int spite_argmax(const float* logits, int rows, int vocab, int* out, void* stream) {
    if (!logits || !out || rows < 0 || vocab < 1) return SPITE_BAD_ARG;
    if (rows == 0) return SPITE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (vocab >= 16384 && rows <= 0x7fffffff / CL) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)rows * CL);
        cfg.blockDim = dim3(THREADS);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CL;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        (void)cudaLaunchKernelEx(&cfg, argmax_cluster_kernel, logits, vocab, (vocab + CL - 1) / CL, out);
        return spite_launch_status();
    }
    argmax_kernel<<<rows, THREADS, 0, st>>>(logits, vocab, out);
    return spite_launch_status();
}

// Both entry points launch through here, so they give the same tokens: a cluster of eight blocks per row where
// a row fits their shared memory (`p.work` is not touched then), else one block per row on `p.work`.
// bins[i] = the bin of a logit `distances[i]` below its row's maximum in a pass whose bins begin at `lo`, `scale` bins a unit (on the host,
// for tests)
SPITE_API int spite_sample_bins(const float* distances, int n, float lo, float scale, int* bins) {
    if (!distances || !bins || n < 0) return SPITE_BAD_ARG;
    const Bins b{lo, scale};
    for (int i = 0; i < n; ++i) bins[i] = b.of(distances[i]);
    return SPITE_OK;
}

static int launch_sample(const SampleParams& p, int rows, cudaStream_t st) {
    int per = ((p.vocab + CL - 1) / CL + 31) / 32 * 32;
    if (per <= CLUSTER_MAX_PER_BLOCK && rows <= 0x7fffffff / CL) {
        const bool pad = (per + THREADS - 1) / THREADS % 2 == 0;      // see Part
        const size_t smem = sizeof(ClusterShared) + (size_t)(per + (pad ? per / 32 : 0)) * sizeof(float);
        void (*kernel)(SampleParams, int) = pad ? sample_cluster_kernel<1> : sample_cluster_kernel<0>;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return SPITE_LAUNCH_FAILED;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)rows * CL);
        cfg.blockDim = dim3(ST);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CL;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        (void)cudaLaunchKernelEx(&cfg, kernel, p, per);
        return spite_launch_status();
    }
    sample_kernel<<<rows, THREADS, 0, st>>>(p);
    return spite_launch_status();
}

SPITE_API int spite_sample(const SampleParams* p, int rows, void* stream) {
    if (!p || !p->logits || !p->work || !p->temperature || !p->rng_state || !p->out_tokens) return SPITE_BAD_ARG;
    if (rows < 0 || p->vocab < 1) return SPITE_BAD_ARG;
    if (p->context && !p->context_offsets) return SPITE_BAD_ARG;
    if (rows == 0) return SPITE_OK;
    return launch_sample(*p, rows, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------
// spite_sample_noalloc: the same kernel with its scratch rows in a fixed array of
// this library instead of memory the caller allocates.  See sampling_noalloc.h for
// who needs this, the size limit, and the rules on sharing and on the first call.
// ---------------------------------------------------------------------------------
#include "sampling_noalloc.h"
#include <atomic>

// Scratch of the no-allocation entry point.  In host code this name is only a handle
// for cudaGetSymbolAddress; it is never passed to a kernel as if it were a pointer.
static __device__ __align__(256) float g_sample_noalloc_scratch[SPITE_SAMPLE_NOALLOC_MAX_FLOATS];

namespace {

constexpr int NOALLOC_MAX_DEVICES = 64;
// device address of the array, per device; atomic, since the first calls of two host threads may both look it
// up (they store the same value)
std::atomic<float*> g_noalloc_scratch_addr[NOALLOC_MAX_DEVICES] = {};

// The device address of the scratch array on the current device; looked up once per
// device with that device current.  Returns null if the runtime refuses.
float* noalloc_scratch_for_current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return nullptr;
    float* ptr = g_noalloc_scratch_addr[dev].load(std::memory_order_acquire);
    if (!ptr) {
        if (cudaGetSymbolAddress((void**)&ptr, g_sample_noalloc_scratch) != cudaSuccess) {
            (void)cudaGetLastError();
            return nullptr;
        }
        g_noalloc_scratch_addr[dev].store(ptr, std::memory_order_release);
    }
    return ptr;
}

}  // namespace

SPITE_API int spite_sample_noalloc(const SpiteSampleNoAllocArgs* a, void* stream) {
    if (!a || !a->logits || !a->temperature || !a->rng_state || !a->out_tokens) return SPITE_BAD_ARG;
    if (a->rows < 0 || a->vocab < 1) return SPITE_BAD_ARG;
    if (a->context && !a->context_offsets) return SPITE_BAD_ARG;
    if ((long long)a->rows * (long long)a->vocab > (long long)SPITE_SAMPLE_NOALLOC_MAX_FLOATS)
        return SPITE_UNSUPPORTED;                            // beyond the fixed scratch: nothing runs
    if (a->rows == 0) return SPITE_OK;
    float* scratch = noalloc_scratch_for_current_device();
    if (!scratch) return SPITE_LAUNCH_FAILED;
    SampleParams p;
    p.logits = a->logits;
    p.work = scratch;                                        // every element is written before it is read
    p.temperature = a->temperature;
    p.top_k = a->top_k;
    p.top_p = a->top_p;
    p.min_p = a->min_p;
    p.repetition_penalty = a->repetition_penalty;
    p.context = a->context;
    p.context_offsets = a->context_offsets;
    p.rng_state = a->rng_state;
    p.out_tokens = a->out_tokens;
    p.vocab = a->vocab;
    return launch_sample(p, a->rows, (cudaStream_t)stream);
}
