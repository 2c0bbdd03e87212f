// The gated delta rule: a mixer whose state is a matrix per head, S [dim, vdim], carried from token to token in
// float32 in the request's state slot:
//     g_t    = exp(-exp(A_h) * softplus(a_t + dt_h))         a_t, b_t: two columns of the projection per head
//     beta_t = sigmoid(b_t)
//     k_t <- k_t / sqrt(|k_t|^2 + unit_eps),   q_t <- q_t / sqrt(|q_t|^2 + unit_eps) * q_scale
//     S <- g_t S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
// A state of zeros is the start of a sequence.  `heads` value heads share `kv_heads` query/key heads (head h reads
// q/k head h / (heads / kv_heads)).  Everything is float32: the inputs are float32 (the projection's sums after the
// short convolution), and nothing in the recurrence is rounded below that.
//
// Token by token.  A block owns 32, 16 or 8 value columns of one (segment, head); a warp a quarter of them; a lane one
// column and a contiguous share of the key rows, RP rows in registers.  The sums over the key rows are a thread's own
// RP terms and two to four shuffles.  One pass over the state per token gives S^T k, S^T q and k . q together
// (o_t = g S_old^T q + u (k . q) is the read-out after the write, regrouped), a second one renews the state.  What
// does not depend on the state (the unit vectors' factors, beta, the decay) comes from a kernel that runs before.  The
// tokens' inputs come through a ring of shared-memory stages filled by asynchronous copies several tokens ahead, so
// the walk waits for arithmetic, not for memory.
//
// Or 32 tokens at a time, on the tensor cores (chunk.cuh), for prompts and their portions.  With b_t the sum of the log decays of a
// chunk's tokens up to t, k and q unit vectors, A[t, s] = beta_t k_t . k_s (s < t) and T = (1 + A)^-1, the rule unrolls to
//     u = T' beta V - e^(b_t) (T beta K) S0,   T'[t, s] = T[t, s] e^(b_t - b_s)
//     o = e^(b_t) Q S0 + P u,   P[t, s] = q_t . k_s e^(b_t - b_s) (s <= t);   S = e^(b_last) S0 + K^T (e^(b_last - b_s) u_s)
// T itself holds no decays (they cancel), so |T[t, s]| <= 1 and the rows of T beta K are no longer than one: unit steps
// 1 - beta k k^T never lengthen a vector.  `delta_chunk_kernel` makes Q, K, T beta K, P and T' beta V for all chunks and heads at once.
#include "chunk.cuh"

SPITE_WAIT_CONTROLS(delta, chunk::walk_error)

struct DeltaParams {
    const float* x;             // [tokens, stride]
    long long stride;
    int q_col, k_col, v_col, b_col, a_col;   // first columns of q, k [kv_heads * dim], v [heads * vdim], b, a [heads]
    const float* a_log;         // [heads]
    const float* dt_bias;       // [heads]
    float* out;                 // [tokens, heads * vdim]
    float* state;               // state + slot * slot_stride + head * dim * vdim: S row-major [dim, vdim]
    long long slot_stride;
    const int* cu_seqlens;      // [segments + 1]
    const int* slots;           // [segments]
    int n_segments, heads, kv_heads, dim, vdim;
    float q_scale, unit_eps;
    float* gates;               // scratch [tokens, 2 * kv_heads + 2 * heads]: per q/k head the factors that make k and q unit
                                // vectors (q's with q_scale), per head beta and the decay; written before the walk
    int n_tokens;
    int n_long;                 // the walk in chunks: how many segments it takes, if that is known (else 0)
};

namespace {

using namespace chunk;

constexpr int NBUF = 8;                                        // tokens in flight

// grid (ceil(vdim / (4 CW)), heads, segments), block 128, shared memory NBUF * stage floats.
// What a token brings besides q, k, v does not depend on the state: one small kernel computes it for all tokens of the
// step, so that the walk's chain per token is multiply-adds and shuffles alone.  grid tokens, block 128: warp w takes
// the q/k heads w, w + 4, ... (sums over dim) and the heads w, w + 4, ... (beta, decay).
__global__ void __launch_bounds__(128) delta_gates_kernel(const DeltaParams p) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* row = p.x + (size_t)t * p.stride;
    float* out = p.gates + (size_t)t * (2 * p.kv_heads + 2 * p.heads);
    for (int g = warp; g < p.kv_heads; g += 4) {
        float k2 = 0.f, q2 = 0.f;
        for (int i = lane; i < p.dim; i += 32) {
            const float kv = row[p.k_col + g * p.dim + i], qv = row[p.q_col + g * p.dim + i];
            k2 = fmaf(kv, kv, k2); q2 = fmaf(qv, qv, q2);
        }
        k2 = warp_sum(k2); q2 = warp_sum(q2);
        if (lane == 0) {
            out[g] = 1.0f / sqrtf(k2 + p.unit_eps);
            out[p.kv_heads + g] = p.q_scale / sqrtf(q2 + p.unit_eps);
        }
    }
    for (int h = threadIdx.x; h < p.heads; h += blockDim.x) {
        const float zb = row[p.b_col + h], za = row[p.a_col + h] + p.dt_bias[h];
        const float softplus = fmaxf(za, 0.f) + log1pf(expf(-fabsf(za)));
        out[2 * p.kv_heads + h] = 1.0f / (1.0f + expf(-zb));
        out[2 * p.kv_heads + p.heads + h] = expf(-expf(p.a_log[h]) * softplus);
    }
}

// CW: value columns a warp owns (8, 4 or 2); its 32 / CW lanes per column split the key rows, RP contiguous rows a lane
// (zeros beyond dim).  Fewer columns a warp means more and smaller blocks and fewer instructions a token and warp, which
// is what a long segment wants (the walk is bound by what one warp can issue); whole sectors of the state per row
// (CW = 8) is what a decode step wants.
template <int RP, int CW>
__global__ void __launch_bounds__(128) delta_scan_kernel(const DeltaParams p, const Leftovers left) {
    extern __shared__ __align__(16) float ring[];
    pdl_wait();
    constexpr int RS = 32 / CW, COLS = 4 * CW, DPAD = RS * RP;
    constexpr int STAGE = 2 * DPAD + ((COLS + 4 + 3) & ~3);    // k [DPAD], q [DPAD], v [COLS], rk, rq, beta, decay
    const int seg = blockIdx.z, head = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r = lane / CW, cc = lane % CW;
    const int dim = p.dim, vdim = p.vdim;
    const int c0 = blockIdx.x * COLS;
    const int j = c0 + warp * CW + cc;                         // this thread's value column
    const bool col_ok = j < vdim;
    const int t0 = p.cu_seqlens[seg], t1 = p.cu_seqlens[seg + 1];
    if (t0 >= t1) return;
    const int what = left_over(left, p.cu_seqlens, seg, head, p.heads, c0, COLS);
    if (what == NOTHING) return;
    const bool mine = col_ok && left_column(left, what, seg, head, p.heads, j);
    const int slot = p.slots[seg];
    // A captured step pads its rows with copies of its first row: a copy would renew the first row's state a second
    // time.  It leaves zeros instead (its results are never read).
    if (seg > 0 && slot == p.slots[0]) {
        if (r == 0 && col_ok)
            for (int t = t0; t < t1; ++t) p.out[(size_t)t * p.heads * vdim + (size_t)head * vdim + j] = 0.f;
        return;
    }
    const int kvh = head / (p.heads / p.kv_heads);
    float* st = p.state + (size_t)slot * p.slot_stride + (size_t)head * dim * vdim;
    float S[RP];
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        const int row = r * RP + i;
        S[i] = (row < dim && col_ok) ? st[(size_t)row * vdim + j] : 0.f;
    }
    const int n_gates = 2 * p.kv_heads + 2 * p.heads;
    // the rows of k and q beyond dim stay zero in every stage
    for (int e = threadIdx.x; e < NBUF * 2 * (DPAD - dim); e += blockDim.x) {
        const int s = e / (2 * (DPAD - dim)), i = e % (2 * (DPAD - dim));
        ring[(size_t)s * STAGE + (i < DPAD - dim ? dim + i : DPAD + dim + i - (DPAD - dim))] = 0.f;
    }

    auto issue = [&](int t) {
        if (t < t1) {
            float* dst = ring + (size_t)((t - t0) % NBUF) * STAGE;
            const float* row = p.x + (size_t)t * p.stride;
            for (int e = threadIdx.x; e < dim; e += blockDim.x) {
                copy4(dst + e, row + p.k_col + kvh * dim + e);
                copy4(dst + DPAD + e, row + p.q_col + kvh * dim + e);
            }
            if (threadIdx.x < COLS) {
                const int c = c0 + threadIdx.x;
                copy4(dst + 2 * DPAD + threadIdx.x, row + p.v_col + head * vdim + (c < vdim ? c : vdim - 1));
            } else if (threadIdx.x < COLS + 4) {
                const int w = threadIdx.x - COLS;              // rk, rq of the q/k head; beta, decay of the head
                const float* gt = p.gates + (size_t)t * n_gates;
                copy4(dst + 2 * DPAD + threadIdx.x, gt + (w == 0 ? kvh : w == 1 ? p.kv_heads + kvh : w == 2 ? 2 * p.kv_heads + head
                                                                                                            : 2 * p.kv_heads + p.heads + head));
            }
        }
        copy_commit();
    };
#pragma unroll 1
    for (int s = 0; s < NBUF - 1; ++s) issue(t0 + s);

#pragma unroll 1
    for (int t = t0; t < t1; ++t) {
        copy_wait<NBUF - 2>();
        __syncthreads();                                       // token t has landed, and every thread is done with token t - 1
        issue(t + NBUF - 1);                                   // (into the stage that token t - 1 had)
        const float* in = ring + (size_t)((t - t0) % NBUF) * STAGE;
        const float4* kk = (const float4*)(in + r * RP);
        const float4* qq = (const float4*)(in + DPAD + r * RP);
        // (four partial sums each: a sum's multiply-adds would otherwise wait for one another)
        float a4[4] = {0.f, 0.f, 0.f, 0.f}, b4[4] = {0.f, 0.f, 0.f, 0.f}, kq4[4] = {0.f, 0.f, 0.f, 0.f};
        float kr[RP];
#pragma unroll
        for (int i = 0; i < RP / 4; ++i) {
            const float4 kv = kk[i], qv = qq[i];
            kr[4 * i] = kv.x; kr[4 * i + 1] = kv.y; kr[4 * i + 2] = kv.z; kr[4 * i + 3] = kv.w;
            a4[0] = fmaf(S[4 * i], kv.x, a4[0]); a4[1] = fmaf(S[4 * i + 1], kv.y, a4[1]);
            a4[2] = fmaf(S[4 * i + 2], kv.z, a4[2]); a4[3] = fmaf(S[4 * i + 3], kv.w, a4[3]);
            b4[0] = fmaf(S[4 * i], qv.x, b4[0]); b4[1] = fmaf(S[4 * i + 1], qv.y, b4[1]);
            b4[2] = fmaf(S[4 * i + 2], qv.z, b4[2]); b4[3] = fmaf(S[4 * i + 3], qv.w, b4[3]);
            kq4[0] = fmaf(kv.x, qv.x, kq4[0]); kq4[1] = fmaf(kv.y, qv.y, kq4[1]);
            kq4[2] = fmaf(kv.z, qv.z, kq4[2]); kq4[3] = fmaf(kv.w, qv.w, kq4[3]);
        }
        float a = (a4[0] + a4[1]) + (a4[2] + a4[3]), b = (b4[0] + b4[1]) + (b4[2] + b4[3]), kq = (kq4[0] + kq4[1]) + (kq4[2] + kq4[3]);
#pragma unroll
        for (int o = CW; o < 32; o <<= 1) {                    // over the lanes that share a column
            a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o);
            kq += __shfl_xor_sync(0xffffffffu, kq, o);
        }
        const float vj = in[2 * DPAD + warp * CW + cc];
        const float rk = in[2 * DPAD + COLS], rq = in[2 * DPAD + COLS + 1], beta = in[2 * DPAD + COLS + 2], g = in[2 * DPAD + COLS + 3];
        const float u = beta * (vj - g * (a * rk));
        const float o = g * (b * rq) + u * (kq * rk * rq);
        const float ku = u * rk;
#pragma unroll
        for (int i = 0; i < RP; ++i) S[i] = fmaf(kr[i], ku, g * S[i]);
        if (r == 0 && mine) p.out[(size_t)t * p.heads * vdim + (size_t)head * vdim + j] = o;
    }
    copy_wait<0>();
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        const int row = r * RP + i;
        if (row < dim && mine) st[(size_t)row * vdim + j] = S[i];
    }
    pdl_launch_dependents();                                   // (late: the next kernel's blocks would only sit and wait)
}

template <int RP, int CW>
static int launch_scan(const DeltaParams& p, const Leftovers& left, cudaStream_t st) {
    constexpr int RS = 32 / CW, COLS = 4 * CW, DPAD = RS * RP;
    constexpr int STAGE = 2 * DPAD + ((COLS + 4 + 3) & ~3);
    dim3 grid((p.vdim + COLS - 1) / COLS, p.heads, p.n_segments);
    // Launched in the ordinary way, not as a programmatic dependent: started early, the walk's few blocks take whatever
    // multiprocessors the kernel before frees first, several to one, and stay there for the whole walk (2,048 tokens
    // of 16 heads of 128 x 128: 1.40 to 1.78 ms against 1.14 ms).
    delta_scan_kernel<RP, CW><<<grid, 128, (size_t)NBUF * STAGE * sizeof(float), st>>>(p, left);
    return spite_launch_status();
}

// What the walk in chunks needs that does not depend on the state.  A block has one chunk and HB heads that share q and k, four warps a
// head.  Left in working memory: the unit q and k and P as split tiles (of size one), W = T beta K alike, its rows divided by their token's
// beta's size (a row is no longer than its beta), U0 = T' beta V in float32.
template <int DP, int HB>
struct DeltaChunkSmem {
    __half qk[4][CT * DP];                                // as in working memory: q high, q low, k high, k low
    float kk[CT][36], qk_scores[CT][36];                  // k_t . k_s, q_t . k_s
    struct Head {
        __half decayed[2][CT * CT], plain[2][CT * CT];    // T' beta and T beta, split
        float T[CT][36], X[16][20];
        double b[CT];
        float beta[CT], size[CT];                         // `size`: of beta (Scale), by which the rows of T' beta, T beta and W are divided
    } head[HB];
    int bad[HB];
};

template <int DP, int HB>
__global__ void __launch_bounds__(128 * HB) delta_chunk_kernel(const DeltaParams p, const Made out) {
    using Rec = Record<DELTA, DP>;
    using SM = DeltaChunkSmem<DP, HB>;
    constexpr int WARPS = 4 * HB, THREADS = 32 * WARPS;
    extern __shared__ __align__(16) unsigned char smem[];
    SM& sm = *reinterpret_cast<SM*>(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int team = warp >> 2, tw = warp & 3, tt = tid & 127;       // the head's four warps, and a thread's place among them
    const int group = p.heads / p.kv_heads, blocks = group / HB, kvh = blockIdx.y / blocks;
    const int head0 = kvh * group + (blockIdx.y % blocks) * HB, head = head0 + team;
    typename SM::Head& hd = sm.head[team];
    pdl_wait();
    pdl_launch_dependents();
    Place pl;
    if (!find_chunk<ALL>(out.numbering, p.cu_seqlens, p.n_segments, blockIdx.x, pl)) return;
    const int first = pl.first, len = min(CT, pl.end - first), dim = p.dim, vdim = p.vdim;
    const bool brief = pl.at < 0;                         // walked token by token: the tokens' scalars alone
    const float* rows = p.x + (size_t)first * p.stride;
    const int n_gates = 2 * p.kv_heads + 2 * p.heads;
    if (!brief && first == pl.begin) clear_marks(out.columns, out.column_groups, pl.seg, head, p.heads, tt, 128);
    if (tid < HB) sm.bad[tid] = 0;

    // ---- unit vectors: a warp has the tokens warp, warp + WARPS, ..., a lane the elements lane, lane + 32, ...
    constexpr int E = DP / 32, TW = CT / WARPS;
    float kv[TW][E], qv[TW][E];
#pragma unroll
    for (int i = 0; i < TW; ++i) {
        const int t = warp + WARPS * i;
        const float* row = rows + (size_t)t * p.stride + kvh * dim;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const bool on = t < len && lane + 32 * e < dim;
            kv[i][e] = on ? row[p.k_col + lane + 32 * e] : 0.f;
            qv[i][e] = on ? row[p.q_col + lane + 32 * e] : 0.f;
        }
    }
    bool bad = false;
    if (tw == 0) {                                        // a lane a token: beta, the decays' running sum
        float beta = 0.f, log_decay = 0.f;
        if (lane < len) {
            const float* row = rows + (size_t)lane * p.stride;
            const float zb = row[p.b_col + head], za = row[p.a_col + head] + p.dt_bias[head];
            const float softplus = fmaxf(za, 0.f) + log1pf(expf(-fabsf(za)));
            beta = 1.0f / (1.0f + expf(-zb));
            log_decay = -expf(p.a_log[head]) * softplus;
            bad = !(beta >= 0.f) || !(log_decay <= 0.f);
            float* gates = p.gates + (size_t)(first + lane) * n_gates;
            gates[2 * p.kv_heads + head] = beta;
            gates[2 * p.kv_heads + p.heads + head] = expf(log_decay);
        }
        hd.beta[lane] = beta;
        hd.size[lane] = scale_of(abs_bits(beta)).size;
        hd.b[lane] = prefix_sum((double)bounded_log(log_decay), lane);
    }
    // the values of the warp's first two groups of sixteen columns, as left operands: columns g, g + 8, tokens 2 t4, + 1, + 8, + 9
    const float* v_rows = rows + p.v_col + (size_t)head * vdim;
    const auto load_values = [&](int tile, float (&v)[2][4][2]) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int t = 16 * k + 2 * t4 + e + 8 * (i >> 1), col = 16 * tile + g + 8 * (i & 1);
                    v[k][i][e] = t < len && col < vdim ? v_rows[(size_t)t * p.stride + col] : 0.f;
                }
    };
#pragma unroll
    for (int i = 0; i < TW; ++i) {
        const int t = warp + WARPS * i;
        float k2 = 0.f, q2 = 0.f;
#pragma unroll
        for (int e = 0; e < E; ++e) { k2 = fmaf(kv[i][e], kv[i][e], k2); q2 = fmaf(qv[i][e], qv[i][e], q2); }
        k2 = warp_sum(k2); q2 = warp_sum(q2);
        const float rk = 1.0f / sqrtf(k2 + p.unit_eps), rq = 1.0f / sqrtf(q2 + p.unit_eps);
        if (t < len) {
            bad |= !(k2 < 3e38f) || !(q2 < 3e38f) || !(rk < 3e38f) || !(rq < 3e38f);
            if (lane == 0 && head0 % group == 0) {
                float* gates = p.gates + (size_t)(first + t) * n_gates;
                gates[kvh] = rk;
                gates[p.kv_heads + kvh] = p.q_scale * rq;
            }
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int at = tile_at<DP>(t, lane + 32 * e);
            split1(t < len ? qv[i][e] * rq * UP : 0.f, sm.qk[0][at], sm.qk[1][at]);
            split1(t < len ? kv[i][e] * rk * UP : 0.f, sm.qk[2][at], sm.qk[3][at]);
        }
    }
    if (brief) return;
    float va[2][2][4][2];
    load_values(tw, va[0]);
    load_values(tw + 4, va[1]);
    const size_t at_head = (size_t)pl.at * p.heads + head;
    float* rec = out.records + at_head * Rec::FLOATS;
    __syncthreads();

    // ---- k_t . k_s and q_t . k_s: sixteen tokens t a warp (k for the first half of four, q for the other), 32 / HB tokens s
    {
        constexpr int N = 4 / HB;                         // groups of eight tokens s
        const bool of_q = tw >= 2;
        const int m = tw & 1, n0 = team * N;
        float main[N][4] = {}, cross[N][4] = {};
        const __half* a = sm.qk[of_q ? 0 : 2];
#pragma unroll 4
        for (int k = 0; k < DP / 16; ++k) {
            unsigned ah[4], al[4];
            ldsm_left<DP>(ah, a, 16 * m, 16 * k, lane);
            ldsm_left<DP>(al, a + CT * DP, 16 * m, 16 * k, lane);
#pragma unroll
            for (int n = 0; n < N; n += 2) {
                const int row = 8 * (n0 + n) + 8 * (lane >> 4) + (lane & 7), col = 16 * k + 8 * ((lane >> 3) & 1);
                unsigned bh[4], bl[4];
                ldsm(bh, sm.qk[2] + tile_at<DP>(row, col));
                ldsm(bl, sm.qk[3] + tile_at<DP>(row, col));
                mma3(main[n], cross[n], ah, al, bh[0], bh[1], bl[0], bl[1]);
                mma3(main[n + 1], cross[n + 1], ah, al, bh[2], bh[3], bl[2], bl[3]);
            }
        }
        float (*to)[36] = of_q ? sm.qk_scores : sm.kk;
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int r = 0; r < 2; ++r)
                *(float2*)&to[16 * m + g + 8 * r][8 * (n0 + n) + 2 * t4] =
                    make_float2(sum2(main[n][2 * r], cross[n][2 * r]), sum2(main[n][2 * r + 1], cross[n][2 * r + 1]));
    }
    if (head0 % group == 0) {                             // q and k of the group's heads are the same
        uint4* dst = reinterpret_cast<uint4*>(out.qk + ((size_t)pl.at * p.kv_heads + kvh) * (4 * CT * DP));
        const uint4* src = reinterpret_cast<const uint4*>(sm.qk[0]);
#pragma unroll 4
        for (int e = tid; e < 4 * CT * DP / 8; e += THREADS) dst[e] = src[e];
    }
    __syncthreads();
    // ---- T = (1 + A)^-1, A[t, s] = beta_t kk[t, s]: its two diagonal blocks, a column a lane of one warp; the other three make P
    if (tw == 0) {
        const int o = lane & 16, col = lane & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int k = 0; k < i; k += 2) {
                const float2 a = *(const float2*)&sm.kk[o + i][o + k];
                s0 = fmaf(a.x, x[k], s0);
                if (k + 1 < i) s1 = fmaf(a.y, x[k + 1], s1);
            }
            x[i] = fmaf(-hd.beta[o + i], s0 + s1, i == col ? 1.f : 0.f);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) hd.T[o + i][o + col] = x[i];
    } else {
        __half* scores = out.scores + at_head * (2 * CT * CT);
        for (int e = tt - 32; e < CT * CT / 2; e += 96) {
            const int t = e >> 4, s = 2 * (e & 15);
            float x[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) x[i] = s + i <= t && t < len ? sm.qk_scores[t][s + i] * expf((float)(hd.b[t] - hd.b[s + i])) * UP : 0.f;
            unsigned h, l;
            split2(x[0], x[1], h, l);
            *(unsigned*)(scores + score_at(t, s)) = h;
            *(unsigned*)(scores + CT * CT + score_at(t, s)) = l;
        }
    }
    __syncthreads();
    // ... and the block below them, T21 = -T22 A21 T11
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int i = (tt >> 4) + 8 * r, j = tt & 15;
        float x = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) x = fmaf(sm.kk[16 + i][k], hd.T[k][j], x);
        hd.X[i][j] = hd.beta[16 + i] * x;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int i = (tt >> 4) + 8 * r, j = tt & 15;
        float x = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) x = fmaf(hd.T[16 + i][16 + k], hd.X[k][j], x);
        hd.T[16 + i][j] = -x;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int e = tt + 128 * r, t = e >> 4, s = 2 * (e & 15), at = score_at(t, s);
        const float up = UP / hd.size[t];                 // (a power of two)
        float x[2], y[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            x[i] = s + i <= t ? hd.T[t][s + i] * hd.beta[s + i] * up : 0.f;
            y[i] = s + i <= t ? x[i] * expf((float)(hd.b[t] - hd.b[s + i])) : 0.f;
        }
        split2(x[0], x[1], *(unsigned*)&hd.plain[0][at], *(unsigned*)&hd.plain[1][at]);
        split2(y[0], y[1], *(unsigned*)&hd.decayed[0][at], *(unsigned*)&hd.decayed[1][at]);
    }
    __syncthreads();
    // ---- U0^T = V^T (T' beta)^T, sixteen columns at a time
    const auto u0_tile = [&](int tile, const float (&v)[2][4][2]) {
        Scale sc[2];                                      // of the columns g and g + 8
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            unsigned largest = 0;
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = c; i < 4; i += 2) largest = max(largest, max(abs_bits(v[k][i][0]), abs_bits(v[k][i][1])));
            largest = quad_max(largest);
            bad |= largest >= 0x7f800000u;
            sc[c] = scale_of(largest);
        }
        unsigned ah[2][4], al[2][4];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) split2(v[k][i][0] * sc[i & 1].up, v[k][i][1] * sc[i & 1].up, ah[k][i], al[k][i]);
        float* u0 = out.u0 + (size_t)first * p.heads * vdim + (size_t)head * vdim;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            float main[4] = {}, cross[4] = {};
            unsigned bh[4], bl[4];
            ldsm(bh, hd.decayed[0] + score_at(8 * n + (lane & 7), 8 * (lane >> 3)));
            ldsm(bl, hd.decayed[1] + score_at(8 * n + (lane & 7), 8 * (lane >> 3)));
            mma3(main, cross, ah[0], al[0], bh[0], bh[1], bl[0], bl[1]);
            if (n >= 2) mma3(main, cross, ah[1], al[1], bh[2], bh[3], bl[2], bl[3]);       // (T is lower triangular)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = 8 * n + 2 * t4 + (i & 1), col = 16 * tile + g + 8 * (i >> 1);
                if (t < len && col < vdim) u0[(size_t)t * p.heads * vdim + col] = sum2(main[i], cross[i]) * sc[i >> 1].size * hd.size[t];
            }
        }
    };
    if (16 * tw < vdim) u0_tile(tw, va[0]);
    if (16 * (tw + 4) < vdim) u0_tile(tw + 4, va[1]);
    for (int tile = tw + 8; 16 * tile < vdim; tile += 4) {
        load_values(tile, va[0]);
        u0_tile(tile, va[0]);
    }
    // ---- W = (T beta) K, a quarter of the keys a warp
    __half* w = out.w + at_head * (2 * CT * DP);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        constexpr int NW = DP / 32;
        float main[NW][4] = {}, cross[NW][4] = {};
#pragma unroll
        for (int k = 0; k <= m; ++k) {
            unsigned ah[4], al[4];
            ldsm_left_scores(ah, hd.plain[0], 16 * m, 16 * k, lane);
            ldsm_left_scores(al, hd.plain[1], 16 * m, 16 * k, lane);
#pragma unroll
            for (int n = 0; n < NW; n += 2) {
                const int row = 16 * k + 8 * ((lane >> 3) & 1) + (lane & 7), cc = DP / 4 * tw + 8 * n + 8 * (lane >> 4);
                unsigned bh[4], bl[4];
                ldsm_t(bh, sm.qk[2] + tile_at<DP>(row, cc));
                ldsm_t(bl, sm.qk[3] + tile_at<DP>(row, cc));
                mma3(main[n], cross[n], ah, al, bh[0], bh[1], bl[0], bl[1]);
                mma3(main[n + 1], cross[n + 1], ah, al, bh[2], bh[3], bl[2], bl[3]);
            }
        }
#pragma unroll
        for (int n = 0; n < NW; ++n)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int at = tile_at<DP>(16 * m + g + 8 * r, DP / 4 * tw + 8 * n + 2 * t4);
                unsigned h, l;
                split2(sum2(main[n][2 * r], cross[n][2 * r]) * UP, sum2(main[n][2 * r + 1], cross[n][2 * r + 1]) * UP, h, l);
                *(unsigned*)(w + at) = h;
                *(unsigned*)(w + CT * DP + at) = l;
            }
    }
    if (bad) sm.bad[team] = 1;
    __syncthreads();
    if (tw == 0) {
        const double last = hd.b[len - 1];
        rec[Rec::G + lane] = lane < len ? expf((float)hd.b[lane]) : 0.f;
        rec[Rec::W + lane] = lane < len ? expf((float)(last - hd.b[lane])) : 0.f;
        rec[Rec::W_SIZE + lane] = hd.size[lane];
        if (lane < 8) {
            bool any = false;
            for (int h = 0; h < HB; ++h) any |= sm.bad[h] != 0;       // (a block's heads share q and k)
            rec[Rec::SCALARS + lane] = lane == DECAY ? expf((float)last) : lane == BAD && any ? 1.f : 0.f;
        }
    }
}

inline Layout delta_layout(int dim, int vdim, int heads, int kv_heads, int n_tokens, int n_chunks, int n_segments) {
    return layout_of(dim <= 64 ? 64 : 128, Record<DELTA, 64>::FLOATS, heads, kv_heads, vdim, n_chunks, n_segments, true,
                     (long long)n_tokens * heads * vdim);
}

template <int DP, int HB>
int launch_delta_prepare(const DeltaParams& p, const Made& out, cudaStream_t st) {
    auto kernel = delta_chunk_kernel<DP, HB>;
    constexpr int bytes = (int)sizeof(DeltaChunkSmem<DP, HB>);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return SPITE_LAUNCH_FAILED;
    // (every chunk of the step, also of segments that go token by token: their tokens' scalars come from here)
    SPITE_LAUNCH(kernel, dim3(p.n_tokens / CT + p.n_segments, p.heads / HB), 128 * HB, bytes, st, p, out);
    return spite_launch_status();
}

template <int DP>
int launch_delta_chunks(const DeltaParams& p, const Made& out, cudaStream_t st) {
    const int rc = p.heads / p.kv_heads % 2 == 0 ? launch_delta_prepare<DP, 2>(p, out, st) : launch_delta_prepare<DP, 1>(p, out, st);
    if (rc != SPITE_OK) return rc;
    Walk w = walk_of(out);
    w.v = out.u0; w.v_stride = (long long)p.heads * p.vdim;
    w.out = p.out; w.out_stride = (long long)p.heads * p.vdim;
    w.state = p.state; w.slot_stride = p.slot_stride; w.head_stride = (long long)p.dim * p.vdim;
    w.key_stride = p.vdim; w.col_stride = 1;
    w.cu_seqlens = p.cu_seqlens; w.slots = p.slots;
    w.n_segments = p.n_segments; w.heads = p.heads; w.qk_heads = p.kv_heads; w.dim = p.dim; w.vdim = p.vdim;
    w.out_scale = p.q_scale;
    // 16 columns a block while that leaves every multiprocessor one block at most, else 32.  2,048 tokens, us of the walk alone: 16 heads
    // (128 blocks of 16 columns) 130, 32 heads (128 blocks of 32) 176.  The kernel before it: 41 and 74.  Measured with one scale a tile:
    // 124, with 16 keys a warp and twice the warps 135; the kernel before it 39 and 70, with a block a head instead of two 69 and 111.
    if ((long long)((p.vdim + 15) / 16) * p.heads * out.numbering.segments <= 148) return launch_walk<32, DP / 32, 1, DELTA>(w, s_waits, st);
    return launch_walk<32, DP / 32, 2, DELTA>(w, s_waits, st);
}

int check_delta(const DeltaParams* p) {
    if (!p || !p->x || !p->a_log || !p->dt_bias || !p->out || !p->state || !p->cu_seqlens || !p->slots || !p->gates) return SPITE_BAD_ARG;
    if (p->n_tokens < 0) return SPITE_BAD_ARG;
    if (p->n_segments < 0 || p->heads < 1 || p->kv_heads < 1 || p->heads % p->kv_heads || p->dim < 1 || p->vdim < 1) return SPITE_BAD_ARG;
    if (p->slot_stride < (long long)p->heads * p->dim * p->vdim || !(p->unit_eps >= 0.f)) return SPITE_BAD_ARG;
    const long long need = (long long)p->kv_heads * p->dim;
    if (p->q_col < 0 || p->k_col < 0 || p->v_col < 0 || p->b_col < 0 || p->a_col < 0) return SPITE_BAD_ARG;
    if (p->stride < p->q_col + need || p->stride < p->k_col + need || p->stride < p->v_col + (long long)p->heads * p->vdim ||
        p->stride < p->b_col + p->heads || p->stride < p->a_col + p->heads) return SPITE_BAD_ARG;
    if (p->dim > 512 || p->heads > 65535 || p->n_segments > 65535) return SPITE_UNSUPPORTED;
    return SPITE_OK;
}

int launch_token_walk(const DeltaParams* p, const Leftovers& left, int split_rows, cudaStream_t st) {
    const int dim = p->dim;
    if (split_rows) {
        if (dim <= 32) return launch_scan<4, 4>(*p, left, st);
        if (dim <= 64) return launch_scan<8, 4>(*p, left, st);
        if (dim <= 128) return launch_scan<8, 2>(*p, left, st);
        if (dim <= 256) return launch_scan<16, 2>(*p, left, st);
        return launch_scan<32, 2>(*p, left, st);
    }
    if (dim <= 32) return launch_scan<8, 8>(*p, left, st);
    if (dim <= 64) return launch_scan<16, 8>(*p, left, st);
    if (dim <= 128) return launch_scan<32, 8>(*p, left, st);
    if (dim <= 256) return launch_scan<64, 8>(*p, left, st);
    return launch_scan<128, 8>(*p, left, st);
}

}  // namespace

// `split_rows`: more lanes a value column and fewer columns a block (for steps with long segments); without it a warp
// owns 8 columns, whole sectors of every row of the state (for decode steps).  The two differ in the order of sums.
SPITE_API int spite_delta_scan(const DeltaParams* p, int split_rows, void* stream) {
    const int chk = check_delta(p);
    if (chk != SPITE_OK) return chk;
    if (p->n_segments == 0 || p->n_tokens == 0) return SPITE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    SPITE_LAUNCH(delta_gates_kernel, p->n_tokens, 128, 0, st, *p);
    if (cudaGetLastError() != cudaSuccess) return SPITE_LAUNCH_FAILED;
    return launch_token_walk(p, Leftovers{}, split_rows, st);
}

// Bytes of working memory that `spite_delta_scan_chunked` needs for a step of `n_chunks` chunks of 32 tokens (the sum over the long segments
// of ceil(tokens / 32), or more); -2: sizes that it does not take.
SPITE_API long long spite_delta_chunk_bytes(int dim, int vdim, int heads, int kv_heads, int n_tokens, int n_chunks, int n_segments) {
    if (dim < 1 || vdim < 1 || heads < 1 || kv_heads < 1 || n_tokens < 0 || n_chunks < 0 || n_segments < 0) return SPITE_BAD_ARG;
    if (dim > 128) return SPITE_UNSUPPORTED;
    return delta_layout(dim, vdim, heads, kv_heads, n_tokens, n_chunks, n_segments).bytes;
}

// Segments of at least `min_tokens` tokens in chunks of 32, the others token by token, and those that the working memory, made for
// `n_chunks` chunks, has no place for.
SPITE_API int spite_delta_scan_chunked(const DeltaParams* p, void* scratch, int n_chunks, int min_tokens, void* stream) {
    const int chk = check_delta(p);
    if (chk != SPITE_OK) return chk;
    if (!scratch || ((uintptr_t)scratch & 15) || n_chunks < 1 || min_tokens < 1) return SPITE_BAD_ARG;
    if (p->dim > 128) return SPITE_UNSUPPORTED;
    if (p->n_segments == 0 || p->n_tokens == 0) return SPITE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const Layout l = delta_layout(p->dim, p->vdim, p->heads, p->kv_heads, p->n_tokens, n_chunks, p->n_segments);
    const Made out = made_at(scratch, l, min_tokens, n_chunks, p->n_segments, p->n_long);
    const int rc = p->dim <= 64 ? launch_delta_chunks<64>(*p, out, st) : launch_delta_chunks<128>(*p, out, st);
    if (rc != SPITE_OK) return rc;
    return launch_token_walk(p, leftovers_of(out, l, p->heads, Record<DELTA, 64>::SCALARS), 0, st);
}
