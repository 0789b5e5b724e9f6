// Linear recurrences over a matrix state per (request, head), carried from token to token in 32-bit:
//   * the gated matrix memory (mLSTM):       S = a S + b k v^T,  n = a n + b k,  o = S^T q / (max(|n . q|, exp(-m)) + 1e-6)
//                                            with log gates i, f, the running maximum m' = max(f + m, i) (m starts at 0),
//                                            a = exp(f + m - m'), b = exp(i - m');
//   * the generalised delta rule:            S = diag(w) S - (r u)(u^T S) + k v^T,  o = S^T q,  u = k / sqrt(sum k^2 + 1e-6),
//                                            both terms reading the old S, w a decay and r a removal rate per key channel;
//   * gated linear attention:                S = diag(a) S + k v^T,  o = S^T q,  a = sigmoid(z)^(1/tau) = exp(logsigmoid(z) / tau)
//                                            a decay per key channel from the pre-activation z;
// (what follows them is in gated_norm.cu)
//
// A block owns a tile of value columns of one (request, head) (32, 16 or 8 of them: whatever gives the SMs a block each) and
// walks the request's tokens of this step in order, with its part of S in registers.  The columns of S do not depend on one
// another, so the tiles of a head run side by side; the vector n and the maximum m, which all tiles of a head need, are
// kept and updated by each tile for itself (dk + 1 numbers for every 8 columns in the state record: no tile ever reads
// what another writes, whenever their blocks happen to run).  Two kernels: one for steps with prompt portions (scan_kernel),
// whose arithmetic for a token does not depend on where a portion starts or ends, and one for steps in which every request
// brings one token (scan_decode_kernel: `longest` = 1), whose sums over a column's rows run in another order.  Long portions are taken in
// chunks of tokens instead (see "runs of tokens as products"), whose results depend on where a portion starts, and on whether the other long requests of
// its step let it take chunks, to a few roundings of 32 bits.
//
// Inputs are columns of one 32-bit activation matrix `proj` [T, ld] (the fused projection of the mixer's input).
#include "common.cuh"

SPY_MODULE(spy_recurrence)

constexpr int CT = 32;   // value columns a block of the decode kernel owns, and the widest tile of the other

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float log_sigmoidf_(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

__device__ __forceinline__ void cp_async16(float* smem_dst, const float* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(float* smem_dst, const float* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct ScanArgs {
    const float* proj;      // [T, ld]
    long long ld;
    int off_q, off_k, off_v, off_x1, off_x2;   // columns of q (or r), k, v; mLSTM: i and f pre-activations; delta: the removal rate's pre-activation (x2 unused)
    const float* extra;     // delta, gated linear attention: the decay's pre-activation [T, H * dk]
    const float* bias1;     // mLSTM: bias of i [H];   delta: bias of the removal rate [H * dk]
    const float* bias2;     // mLSTM: bias of f [H];   delta: the decay's offset [H * dk];   gated linear attention: the decay's bias [H * dk]
    float* state;           // [slots, H, record]
    long long record;       // floats a head: mLSTM dk * dv + (dk + 1) for every 8 columns (padded to 4); delta dk * dv
    int num_slots;
    const int* q_start;     // [S + 1]
    const int* state_slot;  // [S]
    float* out;             // [T, H * dv]
    int H, dk, dv;
    float q_scale, cap;     // cap: mLSTM: the gates' cap;   gated linear attention: 1 / tau
    int* status;
    const int* flags;       // null, or what the chunks' kernels left (see "runs of tokens as products"): the requests that those took are not walked here
};

// Which form a request takes where both run: see "runs of tokens as products" below.
// In a step that takes chunks every request of chunk_min tokens and more does.  A step takes them for two such requests, or for one of chunk_alone tokens: a
// little above where the forms meet for one request (us, tokens / chunks: matrix memory of 4 heads, 96 tokens 26 / 28, 112 30 / 28, 128 33 / 28; delta rule of 32
// heads, 100 tokens 34 / 43, 128 42 / 42, 160 51 / 44; linear attention of 8 heads, 160 tokens 48 / 52, 192 56 / 52, 256 73 / 56).
__host__ __device__ constexpr int chunk_min(int mode) { return mode == 0 ? 96 : (mode == 1 ? 128 : 160); }
__host__ __device__ constexpr int chunk_alone(int mode) { return mode == 0 ? 112 : (mode == 1 ? 128 : 192); }
template <int MODE> struct ChunkOf { static constexpr int C = MODE == 1 ? 32 : 64; };   // tokens of a chunk
// The place in the scratch of the first chunk of a request that starts at token t: its chunks take the places from there on.  The places run ahead of
// the chunks by a factor with which requests of chunk_min tokens and more never meet, however many shorter ones lie between them:
// floor(n f) is at least the n / C chunks, rounded up, of n tokens (f C = 3/2, 5/4 and 4/3).
__host__ __device__ constexpr int chunk_slot(int mode, int t)
{
    return (int)(mode == 0 ? 3LL * t / (2 * 64) : (mode == 1 ? 5LL * t / (4 * 32) : 4LL * t / (3 * 64)));
}
// Whether head h of a request takes the products: every block that asks gets the same answer.
template <int MODE>
__device__ __forceinline__ bool takes_chunks(const ScanArgs& A, int h, int t_begin, int t_end)
{
    constexpr int C = ChunkOf<MODE>::C;
    if (A.flags == nullptr || t_end - t_begin < chunk_min(MODE)) return false;
    const int first = chunk_slot(MODE, t_begin), n = (t_end - t_begin + C - 1) / C;
    int bad = 0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) bad |= A.flags[(size_t)(first + j) * A.H + h];
    return __syncthreads_or(bad) == 0;
}

constexpr int THREADS = 256;      // 8 warps; warp w owns the columns 4w .. 4w + 3 of the tile, lane = 4 * (row group) + (column of the four)

// A thread keeps its part of S in registers for the whole kernel: NR consecutive rows (row group rg owns the rows
// rg * NR .. rg * NR + NR - 1; 8 * NR >= dk) of one column.  The tokens of the request are walked in chunks of TC: a
// chunk's vectors (k, q, and for the delta rule the removal rate and the decay, with their sigmoids and exponentials)
// are brought into shared memory by all threads at once, in rows of 8 * NR floats whose tail beyond dk is zero (so the
// loops over a thread's rows need no bounds); then every warp walks the chunk's tokens on its own four columns without
// a barrier (an element of S belongs to one thread, a sum over the rows is three shuffles inside the warp); the chunk's
// outputs are scaled and stored together.  The state enters and leaves through a tile in shared memory, so that global
// memory is read and written in whole rows of the tile.
// Four tokens are walked at a time: their sums over the rows are reduced together afterwards, so that the shuffles of one
// token run beside those of the others and beside the next token's rows (nothing in S waits for them).
// RG row groups share a warp's lanes (8, 16 or 32), so a warp owns 32 / RG columns and a block CTB = 8 * 32 / RG of them:
// with few requests and heads the tiles are made narrow, so that there are blocks for every SM, and a thread's rows few.
template <int MODE, int NR, int RG>   // MODE 0: gated matrix memory, 1: delta rule, 2: gated linear attention
__global__ void __launch_bounds__(THREADS, NR <= 8 ? 2 : 1) scan_kernel(ScanArgs A, int TC)
{
    constexpr int CW = 32 / RG, CTB = 8 * CW, SPB = CTB + 4;   // columns a warp and a block own; floats between the rows of the state tile in shared memory
    extern __shared__ __align__(16) float sm[];
    // Launched in plain stream order (spy_launch_in_order): it runs long on about a block an SM, and started early its
    // blocks piled up on the SMs that the product ahead left first (a prompt step was a sixth slower).
    pdl_wait();
    constexpr int KS = RG * NR;                     // floats a staged vector takes
    constexpr int V4 = NR >= 4 ? 4 : NR;           // elements a load of a thread's rows brings
    const int dk = A.dk, dv = A.dv, H = A.H;
    // two stages of a chunk's vectors (the next chunk's arrive while this one's tokens are walked), then what a chunk makes
    constexpr int NVEC = MODE == 1 ? 4 : (MODE == 2 ? 3 : 2);     // staged vectors of dk a token: k, q, then the removal rate (delta) and the decay (delta, gated linear attention)
    const size_t stage_floats = (size_t)NVEC * TC * KS + (size_t)TC * CTB + 2 * (size_t)TC;
    float* o_s = sm + 2 * stage_floats;            // [TC][CTB]
    float* m_s = o_s + TC * CTB;                   // [TC] memory: the running maximum after each token
    float* nqp = m_s + TC;                         // [TC][8] memory: n . q, one partial sum a warp
    float* a_s = nqp + TC * 8;                     // [TC] memory: what a token keeps of the state, exp(f + m_before - m_after)
    float* b_s = a_s + TC;                         // [TC] memory: what it adds, exp(i - m_after)
    float* tile = sm;                              // [dk][SPB], only before the first and after the last chunk

    const int seq = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * CTB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col = warp * CW + lane % CW, rg = lane / CW, r0 = rg * NR;
    const int t_begin = A.q_start[seq], t_end = A.q_start[seq + 1];
    if (t_begin >= t_end || takes_chunks<MODE>(A, h, t_begin, t_end)) return;
    const int slot = A.state_slot[seq];
    if (slot < 0 || slot >= A.num_slots) {
        if (tid == 0) report_status(A.status, SPY_STATUS_BAD_PAGE, t_begin);
        return;
    }
    float* st = A.state + ((size_t)slot * H + h) * A.record;
    for (int idx = tid; idx < dk * CTB; idx += THREADS) {
        const int r = idx / CTB, c = idx % CTB;
        tile[r * SPB + c] = c0 + c < dv ? st[(size_t)r * dv + c0 + c] : 0.f;
    }
    // n and m: a copy for every 8 columns of the state (the narrowest tile); a block reads the copy of its first 8 columns and
    // writes those of all its columns, so that every copy is the same whatever tiles the steps before and after use
    float* st_nm = st + (size_t)dk * dv + (size_t)(c0 / 8) * (dk + 1);
    const int copies = min(CTB / 8, (dv + 7) / 8 - c0 / 8);
    float m = 0.f, n_reg[4] = {0.f, 0.f, 0.f, 0.f};                           // n: the rows tid, tid + 256, ... (dk <= 1024)
    if (MODE == 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (tid + j * THREADS < dk) n_reg[j] = st_nm[tid + j * THREADS];
        m = st_nm[dk];
    }
    __syncthreads();
    float Sr[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) Sr[i] = r0 + i < dk ? tile[(r0 + i) * SPB + col] : 0.f;

    // whether a token's vectors start on 16-byte boundaries in the projection (and in the decay's pre-activation)
    const bool aligned = (dk & 3) == 0 && (A.ld & 3) == 0 && ((A.off_k | A.off_q) & 3) == 0 && (reinterpret_cast<uintptr_t>(A.proj) & 15) == 0 &&
                         (MODE == 0 || (((MODE == 1 ? A.off_x1 : 0) & 3) == 0 && (reinterpret_cast<uintptr_t>(A.extra) & 15) == 0));
    // Requests a chunk's vectors into a stage: 16-byte asynchronous copies where the columns allow it (all under way at once),
    // else plain loads; v and the gates' pre-activations by 4-byte copies.  What is made of them (the scaled q, the sigmoid of
    // the removal rate, the decay, the capped gates) is worked out in place once they have landed.
    auto request = [&](int t0, int stage) {
        const int n_tok = min(TC, t_end - t0);
        float* k_s = sm + stage * stage_floats;
        float* q_s = k_s + (size_t)TC * KS;
        float* x1_s = q_s + (size_t)TC * KS;
        float* x2_s = x1_s + (MODE == 1 ? (size_t)TC * KS : 0);
        float* v_s = x2_s + (MODE != 0 ? (size_t)TC * KS : 0);
        float* g1_s = v_s + TC * CTB;
        float* g2_s = g1_s + TC;
        if (aligned) {
            const int quads = dk >> 2;
            for (int idx = tid; idx < n_tok * quads; idx += THREADS) {
                const int tt = idx / quads, qd = idx - tt * quads, c = h * dk + 4 * qd;
                const float* row = A.proj + (size_t)(t0 + tt) * A.ld;
                cp_async16(k_s + tt * KS + 4 * qd, row + A.off_k + c);
                cp_async16(q_s + tt * KS + 4 * qd, row + A.off_q + c);
                if (MODE == 1) cp_async16(x1_s + tt * KS + 4 * qd, row + A.off_x1 + c);
                if (MODE != 0) cp_async16(x2_s + tt * KS + 4 * qd, A.extra + (size_t)(t0 + tt) * H * dk + c);
            }
        } else {
            for (int idx = tid; idx < n_tok * dk; idx += THREADS) {
                const int tt = idx / dk, r = idx - tt * dk, c = h * dk + r;
                const float* row = A.proj + (size_t)(t0 + tt) * A.ld;
                cp_async4(k_s + tt * KS + r, row + A.off_k + c);
                cp_async4(q_s + tt * KS + r, row + A.off_q + c);
                if (MODE == 1) cp_async4(x1_s + tt * KS + r, row + A.off_x1 + c);
                if (MODE != 0) cp_async4(x2_s + tt * KS + r, A.extra + (size_t)(t0 + tt) * H * dk + c);
            }
        }
        if (KS > dk) {
            const int pad = KS - dk;
            for (int idx = tid; idx < n_tok * pad; idx += THREADS) {
                const int tt = idx / pad, r = dk + idx - tt * pad;
                k_s[tt * KS + r] = 0.f;
                q_s[tt * KS + r] = 0.f;
                if (MODE == 1) x1_s[tt * KS + r] = 0.f;
                if (MODE != 0) x2_s[tt * KS + r] = 0.f;
            }
        }
        for (int idx = tid; idx < n_tok * CTB; idx += THREADS) {
            const int tt = idx / CTB, c = idx % CTB;
            if (c0 + c < dv) cp_async4(v_s + idx, A.proj + (size_t)(t0 + tt) * A.ld + A.off_v + h * dv + c0 + c);
            else v_s[idx] = 0.f;
        }
        if (MODE == 0 && tid < n_tok) {
            const float* row = A.proj + (size_t)(t0 + tid) * A.ld;
            cp_async4(g1_s + tid, row + A.off_x1 + h);
            cp_async4(g2_s + tid, row + A.off_x2 + h);
        }
    };
    __syncthreads();                               // the tile has been read: its place is the stages' now
    request(t_begin, 0);
    int stage = 0;
    for (int t0 = t_begin; t0 < t_end; t0 += TC, stage ^= 1) {
        const int n_tok = min(TC, t_end - t0);
        float* k_s = sm + stage * stage_floats;
        float* q_s = k_s + (size_t)TC * KS;
        float* x1_s = q_s + (size_t)TC * KS;
        float* x2_s = x1_s + (MODE == 1 ? (size_t)TC * KS : 0);
        float* v_s = x2_s + (MODE != 0 ? (size_t)TC * KS : 0);
        float* g1_s = v_s + TC * CTB;
        float* g2_s = g1_s + TC;
        cp_async_wait_all();
        __syncthreads();                           // this chunk's vectors have landed; the chunk before has been stored
        for (int idx = tid; idx < n_tok * dk; idx += THREADS) {
            const int tt = idx / dk, r = idx - tt * dk, c = h * dk + r;
            if (MODE == 0) {
                q_s[tt * KS + r] *= A.q_scale;
            } else if (MODE == 2) {
                q_s[tt * KS + r] *= A.q_scale;
                x2_s[tt * KS + r] = expf(log_sigmoidf_(x2_s[tt * KS + r] + A.bias2[c]) * A.cap);
            } else {
                x1_s[tt * KS + r] = sigmoidf_(x1_s[tt * KS + r] + A.bias1[c]);
                x2_s[tt * KS + r] = expf(-0.60653065971263342f * sigmoidf_(x2_s[tt * KS + r] + A.bias2[c]));   // exp(-1/2) = 0.6065...
            }
        }
        if (MODE == 0 && tid < n_tok) {
            g1_s[tid] = A.cap * tanhf((g1_s[tid] + A.bias1[h]) / A.cap);
            g2_s[tid] = log_sigmoidf_(A.cap * tanhf((g2_s[tid] + A.bias2[h]) / A.cap));
        }
        __syncthreads();
        if (MODE == 1) {
            for (int tt = warp; tt < n_tok; tt += THREADS / 32) {
                float ksq = 0.f;
                for (int r = lane; r < dk; r += 32) ksq += k_s[tt * KS + r] * k_s[tt * KS + r];
                ksq = warp_sum(ksq);
                if (lane == 0) g1_s[tt] = 1.0f / sqrtf(ksq + 1e-6f);
            }
            __syncthreads();
        }
        if (MODE == 0) {
            // The running maximum is a chain through the chunk's tokens (an addition and a maximum each), walked by one
            // lane; the two exponentials of every token, which need only the maxima before and after it, are then worked
            // out by a lane each.  The numbers are those of a token-by-token walk.
            if (warp == 0) {         // a chunk has at most 32 tokens: lane tt keeps token tt's gates, the chain runs through shuffles
                const float ig = lane < n_tok ? g1_s[lane] : 0.f, fg = lane < n_tok ? g2_s[lane] : 0.f;
                float mm = m, before = m, after = m;
                for (int tt = 0; tt < n_tok; ++tt) {
                    const float f_t = __shfl_sync(0xffffffffu, fg, tt), i_t = __shfl_sync(0xffffffffu, ig, tt);
                    const float next = fmaxf(f_t + mm, i_t);
                    if (lane == tt) {
                        before = mm;
                        after = next;
                    }
                    mm = next;
                }
                if (lane < n_tok) {
                    m_s[lane] = after;
                    a_s[lane] = expf(fg + before - after);
                    b_s[lane] = expf(ig - after);
                }
            }
            __syncthreads();
            m = m_s[n_tok - 1];
        }
        if (t0 + TC < t_end) request(t0 + TC, stage ^ 1);     // the stage that the chunk before used; every thread is past that chunk
        constexpr int U = NR <= 8 ? 8 : 4;         // tokens walked at a time (their reductions run together); fewer when a thread's rows take many registers
        for (int tt0 = 0; tt0 < n_tok; tt0 += U) {
            float acc[U], nq[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int tt = tt0 + u;
                acc[u] = 0.f;
                nq[u] = 0.f;
                if (tt >= n_tok) continue;         // the same for every thread
                const float* __restrict__ k = k_s + tt * KS + r0;
                const float* __restrict__ q = q_s + tt * KS + r0;
                const float v_c = v_s[tt * CTB + col];
                if (MODE == 0) {
                    const float a_t = a_s[tt], b_t = b_s[tt];
                    float part[4] = {0.f, 0.f, 0.f, 0.f};     // several short chains of sums instead of one long one
#pragma unroll
                    for (int i0 = 0; i0 < NR; i0 += V4) {
                        float kk[V4], qq[V4];
                        if (V4 == 4) {
                            *reinterpret_cast<float4*>(kk) = *reinterpret_cast<const float4*>(k + i0);
                            *reinterpret_cast<float4*>(qq) = *reinterpret_cast<const float4*>(q + i0);
                        } else {
#pragma unroll
                            for (int e = 0; e < V4; ++e) { kk[e] = k[i0 + e]; qq[e] = q[i0 + e]; }
                        }
#pragma unroll
                        for (int e = 0; e < V4; ++e) {
                            const float s = a_t * Sr[i0 + e] + (b_t * kk[e]) * v_c;
                            Sr[i0 + e] = s;
                            part[e & 3] = fmaf(s, qq[e], part[e & 3]);
                        }
                    }
                    acc[u] = (part[0] + part[1]) + (part[2] + part[3]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int r = tid + j * THREADS;
                        if (r < dk) {
                            n_reg[j] = a_t * n_reg[j] + b_t * k_s[tt * KS + r];
                            nq[u] += n_reg[j] * q_s[tt * KS + r];
                        }
                    }
                } else if (MODE == 2) {
                    const float* __restrict__ decay = x2_s + tt * KS + r0;
                    float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int i0 = 0; i0 < NR; i0 += V4) {
                        float kk[V4], qq[V4], dd[V4];
                        if (V4 == 4) {
                            *reinterpret_cast<float4*>(kk) = *reinterpret_cast<const float4*>(k + i0);
                            *reinterpret_cast<float4*>(qq) = *reinterpret_cast<const float4*>(q + i0);
                            *reinterpret_cast<float4*>(dd) = *reinterpret_cast<const float4*>(decay + i0);
                        } else {
#pragma unroll
                            for (int e = 0; e < V4; ++e) { kk[e] = k[i0 + e]; qq[e] = q[i0 + e]; dd[e] = decay[i0 + e]; }
                        }
#pragma unroll
                        for (int e = 0; e < V4; ++e) {
                            const float s = fmaf(dd[e], Sr[i0 + e], kk[e] * v_c);
                            Sr[i0 + e] = s;
                            part[e & 3] = fmaf(s, qq[e], part[e & 3]);
                        }
                    }
                    acc[u] = (part[0] + part[1]) + (part[2] + part[3]);
                } else {
                    const float inv = g1_s[tt];
                    const float* __restrict__ rate = x1_s + tt * KS + r0;
                    const float* __restrict__ decay = x2_s + tt * KS + r0;
                    float part[4] = {0.f, 0.f, 0.f, 0.f};     // several short chains of sums instead of one long one
#pragma unroll
                    for (int i = 0; i < NR; ++i) part[i & 3] = fmaf(k[i] * inv, Sr[i], part[i & 3]);
                    float us = (part[0] + part[1]) + (part[2] + part[3]);
                    part[0] = part[1] = part[2] = part[3] = 0.f;
#pragma unroll
                    for (int o = CW; o <= 16; o <<= 1) us += __shfl_xor_sync(0xffffffffu, us, o);
#pragma unroll
                    for (int i0 = 0; i0 < NR; i0 += V4) {
                        float kk[V4], qq[V4], rr[V4], dd[V4];
                        if (V4 == 4) {
                            *reinterpret_cast<float4*>(kk) = *reinterpret_cast<const float4*>(k + i0);
                            *reinterpret_cast<float4*>(qq) = *reinterpret_cast<const float4*>(q + i0);
                            *reinterpret_cast<float4*>(rr) = *reinterpret_cast<const float4*>(rate + i0);
                            *reinterpret_cast<float4*>(dd) = *reinterpret_cast<const float4*>(decay + i0);
                        } else {
#pragma unroll
                            for (int e = 0; e < V4; ++e) { kk[e] = k[i0 + e]; qq[e] = q[i0 + e]; rr[e] = rate[i0 + e]; dd[e] = decay[i0 + e]; }
                        }
#pragma unroll
                        for (int e = 0; e < V4; ++e) {
                            const float u_r = kk[e] * inv;
                            const float s = dd[e] * Sr[i0 + e] - (rr[e] * u_r) * us + kk[e] * v_c;
                            Sr[i0 + e] = s;
                            part[e & 3] = fmaf(s, qq[e], part[e & 3]);
                        }
                    }
                    acc[u] = (part[0] + part[1]) + (part[2] + part[3]);
                }
            }
#pragma unroll
            for (int o = CW; o <= 16; o <<= 1) {
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
            }
            if (MODE == 0) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                    for (int u = 0; u < U; ++u) nq[u] += __shfl_xor_sync(0xffffffffu, nq[u], o);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (tt0 + u < n_tok) {
                    if (rg == 0) o_s[(tt0 + u) * CTB + col] = acc[u];
                    if (MODE == 0 && lane == 0) nqp[(tt0 + u) * 8 + warp] = nq[u];
                }
            }
        }
        __syncthreads();
        for (int idx = tid; idx < n_tok * CTB; idx += THREADS) {
            const int tt = idx / CTB, c = idx % CTB;
            if (c0 + c >= dv) continue;
            float o = o_s[idx];
            if (MODE == 0) {
                float nq = 0.f;
#pragma unroll
                for (int w = 0; w < 8; ++w) nq += nqp[tt * 8 + w];
                o = o / (fmaxf(fabsf(nq), expf(-m_s[tt])) + 1e-6f);
            }
            A.out[(size_t)(t0 + tt) * H * dv + h * dv + c0 + c] = o;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NR; ++i)
        if (r0 + i < dk) tile[(r0 + i) * SPB + col] = Sr[i];
    __syncthreads();
    for (int idx = tid; idx < dk * CTB; idx += THREADS) {
        const int r = idx / CTB, c = idx % CTB;
        if (c0 + c < dv) st[(size_t)r * dv + c0 + c] = tile[r * SPB + c];
    }
    if (MODE == 0) {
        for (int cp = 0; cp < copies; ++cp) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (tid + j * THREADS < dk) st_nm[(size_t)cp * (dk + 1) + tid + j * THREADS] = n_reg[j];
            if (tid == 0) st_nm[(size_t)cp * (dk + 1) + dk] = m;
        }
    }
    pdl_launch_dependents();
}

// Decoding (every request brings one token): the state's way through memory is all there is to do, so the kernel is built
// to keep much of it under way: a lane owns a column of the tile (a warp reads and writes whole 128-byte rows), a warp owns
// NR consecutive rows, the loads of a thread's rows are issued before anything else, and several blocks share an SM.  Sums
// over the rows cross the warps through shared memory.
template <int MODE, int NR>
__global__ void __launch_bounds__(THREADS, NR <= 16 ? 4 : 1) scan_decode_kernel(ScanArgs A)
{
    __shared__ float red[8][CT], red2[8][CT], part[8], nqp[8];
    extern __shared__ __align__(16) float vec[];      // k, q and, for the delta rule, the removal rate and the decay: dk each
    pdl_enter();
    const int dk = A.dk, dv = A.dv, H = A.H;
    const int seq = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * CT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r0 = warp * NR;
    const int t = A.q_start[seq];
    if (A.q_start[seq + 1] <= t) return;
    const int slot = A.state_slot[seq];
    if (slot < 0 || slot >= A.num_slots) {
        if (tid == 0) report_status(A.status, SPY_STATUS_BAD_PAGE, t);
        return;
    }
    const bool col_ok = c0 + lane < dv;
    float* st = A.state + ((size_t)slot * H + h) * A.record;
    float Sr[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) Sr[i] = (r0 + i < dk && col_ok) ? st[(size_t)(r0 + i) * dv + c0 + lane] : 0.f;
    const float* row = A.proj + (size_t)t * A.ld;
    float *k_s = vec, *q_s = vec + dk, *x1_s = vec + 2 * dk, *x2_s = vec + (MODE == 1 ? 3 : 2) * dk;     // gated linear attention has no x1
    float a = 1.f, b = 0.f, m_new = 0.f, ksq = 0.f, nq = 0.f;
    float* st_nm = st + (size_t)dk * dv + (size_t)(c0 / 8) * (dk + 1);      // n and m: a copy for every 8 columns; the first of this tile's is read, all of them are written
    const int copies = min(CT / 8, (dv + 7) / 8 - c0 / 8);
    if (MODE == 0) {
        const float ig = A.cap * tanhf((row[A.off_x1 + h] + A.bias1[h]) / A.cap);
        const float fg = log_sigmoidf_(A.cap * tanhf((row[A.off_x2 + h] + A.bias2[h]) / A.cap));
        const float m = st_nm[dk];
        m_new = fmaxf(fg + m, ig);
        a = expf(fg + m - m_new);
        b = expf(ig - m_new);
    }
    for (int r = tid; r < dk; r += THREADS) {
        const int c = h * dk + r;
        const float kr = row[A.off_k + c], qr = row[A.off_q + c] * A.q_scale;
        k_s[r] = kr;
        q_s[r] = qr;
        if (MODE == 0) {
            const float n = a * st_nm[r] + b * kr;
            for (int cp = 0; cp < copies; ++cp) st_nm[(size_t)cp * (dk + 1) + r] = n;
            nq += n * qr;
        } else if (MODE == 2) {
            x2_s[r] = expf(log_sigmoidf_(A.extra[(size_t)t * H * dk + c] + A.bias2[c]) * A.cap);
        } else {
            x1_s[r] = sigmoidf_(row[A.off_x1 + c] + A.bias1[c]);
            x2_s[r] = expf(-0.60653065971263342f * sigmoidf_(A.extra[(size_t)t * H * dk + c] + A.bias2[c]));
            ksq += kr * kr;
        }
    }
    if (MODE == 0) {
        nq = warp_sum(nq);
        if (lane == 0) nqp[warp] = nq;
    } else if (MODE == 1) {
        ksq = warp_sum(ksq);
        if (lane == 0) part[warp] = ksq;
    }
    __syncthreads();
    const float v_c = col_ok ? row[A.off_v + h * dv + c0 + lane] : 0.f;
    float acc = 0.f;
    if (MODE == 0) {
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int r = r0 + i;
            if (r < dk) {
                const float s = a * Sr[i] + (b * k_s[r]) * v_c;
                if (col_ok) st[(size_t)r * dv + c0 + lane] = s;
                acc = fmaf(s, q_s[r], acc);
            }
        }
        red[warp][lane] = acc;
        __syncthreads();
        if (warp == 0 && col_ok) {
            float o = 0.f, n = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) { o += red[w][lane]; n += nqp[w]; }
            A.out[(size_t)t * H * dv + h * dv + c0 + lane] = o / (fmaxf(fabsf(n), expf(-m_new)) + 1e-6f);
        }
        if (tid == 0)
            for (int cp = 0; cp < copies; ++cp) st_nm[(size_t)cp * (dk + 1) + dk] = m_new;
    } else if (MODE == 2) {
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int r = r0 + i;
            if (r < dk) {
                const float s = fmaf(x2_s[r], Sr[i], k_s[r] * v_c);
                if (col_ok) st[(size_t)r * dv + c0 + lane] = s;
                acc = fmaf(s, q_s[r], acc);
            }
        }
        red2[warp][lane] = acc;
        __syncthreads();
        if (warp == 0 && col_ok) {
            float o = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) o += red2[w][lane];
            A.out[(size_t)t * H * dv + h * dv + c0 + lane] = o;
        }
    } else {
        float sq = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) sq += part[w];
        const float inv = 1.0f / sqrtf(sq + 1e-6f);
        float us = 0.f;
#pragma unroll
        for (int i = 0; i < NR; ++i)
            if (r0 + i < dk) us = fmaf(k_s[r0 + i] * inv, Sr[i], us);
        red[warp][lane] = us;
        __syncthreads();
        us = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) us += red[w][lane];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int r = r0 + i;
            if (r < dk) {
                const float u = k_s[r] * inv;
                const float s = x2_s[r] * Sr[i] - (x1_s[r] * u) * us + k_s[r] * v_c;
                if (col_ok) st[(size_t)r * dv + c0 + lane] = s;
                acc = fmaf(s, q_s[r], acc);
            }
        }
        red2[warp][lane] = acc;
        __syncthreads();
        if (warp == 0 && col_ok) {
            float o = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) o += red2[w][lane];
            A.out[(size_t)t * H * dv + h * dv + c0 + lane] = o;
        }
    }
}

// ---- runs of tokens as products --------------------------------------------------------------------------------------------
//
// A request that brings many tokens (chunk_min and more) is walked in chunks of C tokens instead of token by token.  Written out over a
// chunk, each recurrence gives the chunk's outputs and the state behind it as products with the state S ahead of it and the
// chunk's values V, whose other factors do not depend on S:
//   matrix memory:  o_t = (alpha_t (P V)_t + beta_t S^T q_t) / ...,   S' = g S + K^T diag(kappa) V,   P_ts = exp(F_t - F_s + i_s - l_t) q_t . k_s
//                   (F: the forget gates' sums from the chunk's start, l: the running maximum as if the chunk were the first; the true
//                   maximum is max(F_t + m, l_t), alpha and beta are what is left of l and of F + m under it: every exponent is at most 0);
//   linear attention:  o_t = (P V)_t + S^T (q_t a_1..a_t),   S' = diag(a_1..a_C) S + (k_s a_s+1..a_C)^T V,   P_ts = sum over channels of q_t k_s a_s+1..a_t;
//   delta rule:     with A_t = w_1..w_t, p_t = u_t A_t-1, b_s = r_s u_s / A_s, c_s = k_s / A_s, g_t = q_t A_t (w is above exp(-exp(-1/2)) = 0.545, so A_32
//                   above 3.7e-9) and (I + L) [P' | M'] = [p | M], L = p b^T and M = p c^T below the diagonal:
//                   [o; S'] = W [S; V] with the rows g - X P' and Y - X M' (X = g b^T, Y = g c^T up to the diagonal) for the outputs and
//                   A_C (I - b^T P') and A_C (c^T - b^T M') for the state.
// (The delta rule's form inverts a unit triangular matrix, as the published chunked forms of delta rules do, after Yang et al., 2024; the
// decays of linear attention are taken relative to sub-blocks of 16 tokens, so that no factor exceeds 1.)
//
// Two kernels: chunk_*_kernel makes these factors, a block a (chunk, head), all chunks side by side; walk_*_kernel carries S through a
// request's chunks, a block 16 value columns of a (request, head).  What bounds the walk is the way through a chunk on eight warps (a chunk of
// 64 tokens at 128 x 16 takes 4.7 us; the counters show shared memory busy for 64 % of the time and the FMA pipes for 33); the token-by-token kernel above
// spends 270 to 300 ns a token on one request, nearly all of it waiting.  Measured, chunks' kernels and walk together (us, by tokens / in chunks):
//   matrix memory, 8 heads of 128 x 256: one request of 256 tokens 76 / 38, of 2,047 570 / 179; 8 of 100 to 400 417 / 212; 16 of 1,024 2,585 / 1,523;
//   delta rule, 32 heads of 64: one request of 256 79 / 50, of 2,047 610 / 351; 16 heads 80 / 49 and 614 / 250;
//   linear attention, 16 heads of 128 x 256: one of 256 103 / 71, of 2,047 777 / 378; 8 of 100 to 400 632 / 445; 16 of 1,024 4,109 / 2,988.
// Error against 64 bits, tokens / chunks, 2,047 tokens (2-norm; matrix memory: the median token's): matrix memory of 128 x 48 1.85e-7 / 1.12e-7, linear attention 1.73e-7 /
// 1.70e-7 (decays near nothing 1.03e-7 / 0.94e-7), delta rule 1.04e-7 / 0.99e-7 (1.13e-7 / 1.08e-7).  What is summed into a chunk's factors is what counts:
// with the delta rule's 64-term sums and the linear attention's sums inside sub-blocks in 32-bit, and chains of 128 terms between sub-blocks, the chunks'
// errors were 1.74e-7 and 2.02e-7.  So those sums are taken in 64-bit (delta rule of 2,047 tokens 298 us with 32-bit ones, 351 now; linear attention 373
// and 378) or in short chains; products of decays are taken in 64-bit and rounded once; all else is in 32-bit.
//
// Which form a request takes in a step that takes chunks (chunk_work_floats) is decided on the device, head by head, by one rule (takes_chunks) in both
// kernels: runs of fewer than chunk_min tokens, and heads of a request with a number among their q, k and v that is not below HUGE_INPUT in magnitude
// or with a NaN among these or their gates and decays (whose infinities saturate), are walked token by token: in the products an infinity of a
// later token would meet the zeros of an earlier one.
constexpr float HUGE_INPUT = 1e10f;
constexpr int WALK_COLS = 16;          // value columns a block of the walk owns
constexpr int WALK_LD = WALK_COLS + 4; // floats between the rows of a tile of them in shared memory

struct ChunkArgs {
    ScanArgs s;
    float* work;       // [slots][H][chunk_floats(mode, dk)]
    int* flags;        // [slots][H]: the chunk holds a number that keeps its request off the products
    int num_seqs;
};

// what a chunk of one head takes of the scratch, in floats
__host__ __device__ constexpr int chunk_floats(int mode, int dk)
{
    return mode == 0 ? 64 * 64 + 4 * 64 + dk : (mode == 2 ? 64 * 64 + 2 * 64 * dk + dk : (dk + 32) * (dk + 32));
}

// The chunk at a place in the scratch (its first token and its tokens); false where there is none.
template <int MODE>
__device__ __forceinline__ bool chunk_of_slot(const ChunkArgs& A, int slot, int& t0, int& n_tok)
{
    constexpr int C = ChunkOf<MODE>::C;
    int lo = 0, hi = A.num_seqs;           // the last request whose first place is at most `slot`: none behind a place's request starts before its end
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (chunk_slot(MODE, A.s.q_start[mid]) <= slot) lo = mid;
        else hi = mid;
    }
    const int t_begin = A.s.q_start[lo], t_end = A.s.q_start[lo + 1];
    t0 = t_begin + (slot - chunk_slot(MODE, t_begin)) * C;
    n_tok = min(C, t_end - t0);
    return t0 < t_end && t_end - t_begin >= chunk_min(MODE);
}

// The request of a block of the walk: the x-th of those with chunk_min tokens and more; -1 where there are fewer.  Every warp finds it for itself.
template <int MODE>
__device__ __forceinline__ int long_request(const ChunkArgs& A, int x)
{
    const int lane = threadIdx.x & 31;
    for (int s0 = 0; s0 < A.num_seqs; s0 += 32) {
        const int s = s0 + lane;
        unsigned found = __ballot_sync(0xffffffffu, s < A.num_seqs && A.s.q_start[s + 1] - A.s.q_start[s] >= chunk_min(MODE));
        const int n = __popc(found);
        if (x < n) {
            for (; x > 0; --x) found &= found - 1;
            return s0 + __ffs(found) - 1;
        }
        x -= n;
    }
    return -1;
}

__device__ __forceinline__ bool huge(float x) { return !(fabsf(x) < HUGE_INPUT); }
__device__ __forceinline__ bool huge4(float4 v) { return huge(v.x) | huge(v.y) | huge(v.z) | huge(v.w); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float dot4(float4 a, float4 b, float s) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s)))); }

// Brings rows [0, n_tok) of DK columns into shared memory (rows of LD floats), zeros up to C rows; true if a number is huge.
template <int C, int DK, int LD>
__device__ __forceinline__ bool load_rows(float* dst, const float* src, long long ld, int n_tok)
{
    bool bad = false;
    for (int idx = threadIdx.x; idx < C * (DK / 4); idx += THREADS) {
        const int t = idx / (DK / 4), c = 4 * (idx - t * (DK / 4));
        const float4 v = t < n_tok ? ld4(src + (size_t)t * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        bad |= huge4(v);
        st4(dst + t * LD + c, v);
    }
    return bad;
}
__device__ __forceinline__ bool huge_values(const ScanArgs& A, int h, int t0, int n_tok)
{
    bool bad = false;
    const int quads = A.dv >> 2;
    for (int idx = threadIdx.x; idx < n_tok * quads; idx += THREADS) {
        const int t = idx / quads, c = 4 * (idx - t * quads);
        bad |= huge4(ld4(A.proj + (size_t)(t0 + t) * A.ld + A.off_v + (size_t)h * A.dv + c));
    }
    return bad;
}

template <int DK>
__global__ void __launch_bounds__(THREADS, 2) chunk_memory_kernel(ChunkArgs A)
{
    constexpr int C = 64, LD = DK + 4;
    extern __shared__ __align__(16) float sm[];
    float *q_s = sm, *k_s = sm + C * LD;
    __shared__ double from_s[C], to_s[C];          // i_s - F_s and F_t - l_t
    __shared__ float kappa_s[C];
    pdl_enter();
    int t0, n_tok;
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!chunk_of_slot<0>(A, blockIdx.x, t0, n_tok)) return;
    const ScanArgs& a = A.s;
    float* mine = A.work + ((size_t)blockIdx.x * a.H + h) * chunk_floats(0, DK);
    float *P = mine, *F = mine + C * C, *loc = F + C, *kap = loc + C, *psum = kap + C, *ksum = psum + C;
    const float* rows = a.proj + (size_t)t0 * a.ld;
    bool bad = load_rows<C, DK, LD>(q_s, rows + a.off_q + h * DK, a.ld, n_tok);
    bad |= load_rows<C, DK, LD>(k_s, rows + a.off_k + h * DK, a.ld, n_tok);
    bad |= huge_values(a, h, t0, n_tok);
    if (warp == 0) {
        // the gates' sums and the running maximum in 64-bit (differences of sums are taken below); a lane owns tokens 2 lane and 2 lane + 1
        double f[2], e[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = 2 * lane + j;
            float ig = -INFINITY, fg = 0.f;
            if (t < n_tok) {
                const float x1 = rows[(size_t)t * a.ld + a.off_x1 + h] + a.bias1[h], x2 = rows[(size_t)t * a.ld + a.off_x2 + h] + a.bias2[h];
                bad |= isnan(x1) || isnan(x2);
                ig = a.cap * tanhf(x1 / a.cap);
                fg = log_sigmoidf_(a.cap * tanhf(x2 / a.cap));
            }
            f[j] = fg;
            e[j] = ig;
        }
        double sum = f[0] + f[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
        }
        const double F0 = sum - f[1], F1 = sum;
        e[0] -= F0;
        e[1] -= F1;
        double most = fmax(e[0], e[1]);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, most, o);
            if (lane >= o) most = fmax(most, up);
        }
        double before = __shfl_up_sync(0xffffffffu, most, 1);
        if (lane == 0) before = -INFINITY;
        const double l0 = F0 + fmax(before, e[0]), l1 = F1 + most;
        const double F_end = __shfl_sync(0xffffffffu, F1, 31), l_end = __shfl_sync(0xffffffffu, l1, 31);     // padding tokens change neither
        from_s[2 * lane] = e[0];
        from_s[2 * lane + 1] = e[1];
        to_s[2 * lane] = F0 - l0;
        to_s[2 * lane + 1] = F1 - l1;
        const float k0 = expf((float)(F_end - l_end + e[0])), k1 = expf((float)(F_end - l_end + e[1]));
        kappa_s[2 * lane] = k0;
        kappa_s[2 * lane + 1] = k1;
        *reinterpret_cast<float2*>(F + 2 * lane) = make_float2((float)F0, (float)F1);
        *reinterpret_cast<float2*>(loc + 2 * lane) = make_float2((float)l0, (float)l1);
        *reinterpret_cast<float2*>(kap + 2 * lane) = make_float2(k0, k1);
    }
    const int any = __syncthreads_or(bad);
    if (tid == 0) A.flags[(size_t)blockIdx.x * a.H + h] = any;
    // P: a thread has 4 x 4 of the 64 x 64, rows 4 ty + i, columns tx + 16 j, each in two chains of sums
    const int tx = tid & 15, ty = tid >> 4;
    float acc[4][4] = {}, acc2[4][4] = {};
    for (int c = 0; c < DK; c += 4) {
        float4 kk[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) kk[j] = ld4(k_s + (tx + 16 * j) * LD + c);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 qq = ld4(q_s + (4 * ty + i) * LD + c);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[i][j] = fmaf(qq.x, kk[j].x, fmaf(qq.y, kk[j].y, acc[i][j]));
                acc2[i][j] = fmaf(qq.z, kk[j].z, fmaf(qq.w, kk[j].w, acc2[i][j]));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = 4 * ty + i;
        float row = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int s = tx + 16 * j;
            const float p = s <= t ? expf((float)(to_s[t] + from_s[s])) * ((acc[i][j] + acc2[i][j]) * a.q_scale) : 0.f;
            P[t * C + s] = p;
            row += p;
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) row += __shfl_xor_sync(0xffffffffu, row, o);
        if (tx == 0) psum[t] = row;
    }
    for (int c = tid; c < DK; c += THREADS) {
        float s = 0.f;
#pragma unroll 8
        for (int t = 0; t < C; ++t) s = fmaf(kappa_s[t], k_s[t * LD + c], s);
        ksum[c] = s;
    }
}

template <int DK>
__global__ void __launch_bounds__(THREADS, 2) chunk_linear_kernel(ChunkArgs A)
{
    constexpr int C = 64, LD = DK + 4, B = 16;     // sub-blocks of 16 tokens
    extern __shared__ __align__(16) float sm[];
    float *q_s = sm, *k_s = q_s + C * LD, *a_s = k_s + C * LD;
    pdl_enter();
    int t0, n_tok;
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!chunk_of_slot<2>(A, blockIdx.x, t0, n_tok)) return;
    const ScanArgs& a = A.s;
    float* mine = A.work + ((size_t)blockIdx.x * a.H + h) * chunk_floats(2, DK);
    float *P = mine, *Q = mine + C * C, *K = Q + C * DK, *dec = K + C * DK;
    const float* rows = a.proj + (size_t)t0 * a.ld;
    bool bad = load_rows<C, DK, LD>(q_s, rows + a.off_q + h * DK, a.ld, n_tok);
    bad |= load_rows<C, DK, LD>(k_s, rows + a.off_k + h * DK, a.ld, n_tok);
    bad |= huge_values(a, h, t0, n_tok);
    for (int idx = tid; idx < C * DK; idx += THREADS) {
        const int t = idx / DK, c = idx - t * DK;
        float d = 1.f;
        if (t < n_tok) {
            const float z = a.extra[(size_t)(t0 + t) * a.H * DK + h * DK + c] + a.bias2[h * DK + c];
            bad |= isnan(z);
            d = expf(log_sigmoidf_(z) * a.cap);
        }
        a_s[t * LD + c] = d;
    }
    const int any = __syncthreads_or(bad);
    if (tid == 0) A.flags[(size_t)blockIdx.x * a.H + h] = any;
    // inside a sub-block: k_s carried from its token on, a decay at a time; a warp takes every eighth token, a lane DK / 32 channels
    for (int s = warp; s < C; s += THREADS / 32) {
        const int b0 = s & ~(B - 1), first = s - b0;
        constexpr int E = DK / 32;
        float w[E], d[B];
#pragma unroll
        for (int e = 0; e < E; ++e) w[e] = k_s[s * LD + lane + 32 * e];
#pragma unroll
        for (int i = 0; i < B; ++i) {
            d[i] = 0.f;
            if (i >= first) {                      // the same for the whole warp
                const float* at = a_s + (b0 + i) * LD + lane;
                const float* qt = q_s + (b0 + i) * LD + lane;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    if (i > first) w[e] *= at[32 * e];
                    d[i] = fmaf(w[e], qt[32 * e], d[i]);
                }
            }
        }
        // the sixteen sums over the warp together, in 64-bit: with every step a lane keeps half of its sums
        int mine = 0;
        double wide[B];
#pragma unroll
        for (int i = 0; i < B; ++i) wide[i] = d[i];
#pragma unroll
        for (int o = 16, n = B / 2; n > 0; o >>= 1, n >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const double own = up ? wide[i + n] : wide[i], give = up ? wide[i] : wide[i + n];
                wide[i] = own + __shfl_xor_sync(0xffffffffu, give, o);
            }
            mine += up ? n : 0;
        }
        wide[0] += __shfl_xor_sync(0xffffffffu, wide[0], 1);
        if ((lane & 1) == 0) P[(b0 + mine) * C + s] = (float)(wide[0] * a.q_scale);       // zero above the diagonal
    }
    for (int idx = tid; idx < C * C; idx += THREADS)
        if ((idx & (C - 1)) / B > idx / C / B) P[idx] = 0.f;
    __syncthreads();
    // q from its sub-block's start, k to its sub-block's end; a_s's last row of a sub-block then holds the sub-block's product
    for (int idx = tid; idx < DK * (C / B); idx += THREADS) {
        const int c = idx % DK, b0 = idx / DK * B;
        double run = 1.0, back = 1.0;              // products of up to sixteen decays, rounded once
#pragma unroll
        for (int i = 0; i < B; ++i) {
            run *= a_s[(b0 + i) * LD + c];
            q_s[(b0 + i) * LD + c] *= (float)run * a.q_scale;
        }
#pragma unroll
        for (int i = B - 1; i >= 0; --i) {
            k_s[(b0 + i) * LD + c] *= (float)back;
            back *= a_s[(b0 + i) * LD + c];
        }
        a_s[(b0 + B - 1) * LD + c] = (float)run;
    }
    __syncthreads();
    // across sub-blocks, one after the other: the keys so far reach the end of the sub-block ahead.  A thread has row t = b B + tid / 16
    // and the columns tid % 16 + 16 j.
    for (int b = 1; b < C / B; ++b) {
        const int t = b * B + (tid >> 4), s0 = tid & 15;
        float acc[C / B - 1][4] = {};              // four short chains of sums instead of one of DK terms
        for (int c = 0; c < DK; c += 4) {
            const float4 qq = ld4(q_s + t * LD + c);
#pragma unroll
            for (int j = 0; j < C / B - 1; ++j)
                if (j < b) {
                    const float4 kk = ld4(k_s + (s0 + 16 * j) * LD + c);
                    acc[j][0] = fmaf(qq.x, kk.x, acc[j][0]);
                    acc[j][1] = fmaf(qq.y, kk.y, acc[j][1]);
                    acc[j][2] = fmaf(qq.z, kk.z, acc[j][2]);
                    acc[j][3] = fmaf(qq.w, kk.w, acc[j][3]);
                }
        }
#pragma unroll
        for (int j = 0; j < C / B - 1; ++j)
            if (j < b) P[t * C + s0 + 16 * j] = (acc[j][0] + acc[j][1]) + (acc[j][2] + acc[j][3]);
        __syncthreads();
        for (int idx = tid; idx < b * B * DK; idx += THREADS) {
            const int s = idx / DK, c = idx - s * DK;
            k_s[s * LD + c] *= a_s[(b * B + B - 1) * LD + c];
        }
        __syncthreads();
    }
    for (int idx = tid; idx < C * DK; idx += THREADS) {
        const int t = idx / DK, c = idx - t * DK;
        float q = q_s[t * LD + c];
        for (int b = 0; b < t / B; ++b) q *= a_s[(b * B + B - 1) * LD + c];
        Q[idx] = q;
        K[idx] = k_s[t * LD + c];
        if (t == 0) {
            float d = 1.f;
#pragma unroll
            for (int b = 0; b < C / B; ++b) d *= a_s[(b * B + B - 1) * LD + c];
            dec[c] = d;
        }
    }
}

__global__ void __launch_bounds__(THREADS, 2) chunk_delta_kernel(ChunkArgs A)
{
    constexpr int C = 32, D = 64, LD = D + 2, R = D + C, LDM = R + 4;
    extern __shared__ __align__(16) float sm[];
    double* pg = reinterpret_cast<double*>(sm);   // [2 C][LD]: p, then g (first: q)
    double* bc = pg + 2 * C * LD;      // [2 C][LD]: b, then c (first: the rates, k)
    float* PM = reinterpret_cast<float*>(bc + 2 * C * LD);   // [C][LDM]: P' | M' (first: the decays)
    float* XB = PM + C * LDM;          // [C][LDM]: token s: X_ts of the outputs t, then b_s of the state's rows
    float* L = XB + C * LDM;           // [C][C + 1]
    float* Y = L + C * (C + 1);        // [C][C + 1]
    __shared__ float inv_s[C], last_s[D];
    pdl_enter();
    int t0, n_tok;
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!chunk_of_slot<1>(A, blockIdx.x, t0, n_tok)) return;
    const ScanArgs& a = A.s;
    float* W = A.work + ((size_t)blockIdx.x * a.H + h) * chunk_floats(1, D);
    const float* rows = a.proj + (size_t)t0 * a.ld;
    bool bad = huge_values(a, h, t0, n_tok);
#pragma unroll 4
    for (int idx = tid; idx < C * D; idx += THREADS) {
        const int t = idx / D, c = idx - t * D;
        float q = 0.f, k = 0.f, rate = 0.f, w = 1.f;
        if (t < n_tok) {
            const float* row = rows + (size_t)t * a.ld + h * D + c;
            q = row[a.off_q];
            k = row[a.off_k];
            const float x1 = row[a.off_x1] + a.bias1[h * D + c];
            const float x2 = a.extra[(size_t)(t0 + t) * a.H * D + h * D + c] + a.bias2[h * D + c];
            bad |= huge(q) | huge(k) | isnan(x1) | isnan(x2);
            rate = sigmoidf_(x1);
            w = expf(-0.60653065971263342f * sigmoidf_(x2));     // exp(-1/2) = 0.6065...
        }
        pg[(C + t) * LD + c] = q;
        bc[(C + t) * LD + c] = k;
        bc[t * LD + c] = rate;
        PM[t * LDM + c] = w;
    }
    const int any = __syncthreads_or(bad);
    if (tid == 0) A.flags[(size_t)blockIdx.x * a.H + h] = any;
    for (int t = warp; t < C; t += THREADS / 32) {
        const float k0 = (float)bc[(C + t) * LD + lane], k1 = (float)bc[(C + t) * LD + lane + 32];
        const float sq = warp_sum(k0 * k0 + k1 * k1);
        if (lane == 0) inv_s[t] = 1.0f / sqrtf(sq + 1e-6f);
    }
    __syncthreads();
    if (tid < D) {
        double product = 1.0;                      // of the decays so far, rounded where it is used
        float run = 1.f;
#pragma unroll 8
        for (int t = 0; t < C; ++t) {
            const float k = (float)bc[(C + t) * LD + tid], u = k * inv_s[t], rate = (float)bc[t * LD + tid];
            pg[t * LD + tid] = u * run;
            product *= PM[t * LDM + tid];
            run = (float)product;
            pg[(C + t) * LD + tid] = (float)pg[(C + t) * LD + tid] * run;
            const float b = rate * u / run;
            bc[t * LD + tid] = b;
            bc[(C + t) * LD + tid] = k / run;
            XB[t * LDM + C + tid] = b;
        }
        last_s[tid] = run;
    }
    __syncthreads();
    {
        // [p; g] [b; c]^T, 64 x 64, summed in 64-bit (what these sums round off, every output and the state carry on: with 32-bit sums the outputs' error
        // was half as large again as the walk's by tokens): rows 4 ty + i, columns tx + 16 j; a warp whose rows are tokens below 16
        // leaves out the columns of the later tokens
        const int tx = tid & 15, ty = tid >> 4;
        const bool early = (ty & 7) < 4;
        double acc[4][4] = {};
#pragma unroll 2
        for (int c = 0; c < D; c += 2) {
            double2 kk[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (!early || (j & 1) == 0) kk[j] = *reinterpret_cast<const double2*>(bc + (tx + 16 * j) * LD + c);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 qq = *reinterpret_cast<const double2*>(pg + (4 * ty + i) * LD + c);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (!early || (j & 1) == 0) acc[i][j] = fma(qq.x, kk[j].x, fma(qq.y, kk[j].y, acc[i][j]));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int row = 4 * ty + i, s = (tx + 16 * j) & (C - 1), t = row & (C - 1);
                const float v = (float)acc[i][j];
                if (row < C) {
                    if (j < 2) L[t * (C + 1) + s] = s < t ? v : 0.f;
                    else PM[t * LDM + D + s] = s < t ? v : 0.f;
                } else {
                    if (j < 2) XB[s * LDM + t] = s <= t ? v : 0.f;
                    else Y[t * (C + 1) + s] = s <= t ? v : 0.f;
                }
            }
    }
    for (int idx = tid; idx < C * D; idx += THREADS) PM[idx / D * LDM + idx % D] = (float)pg[idx / D * LD + idx % D];     // the decays have been used
    __syncthreads();
    if (tid < R) {
        float x[C];
#pragma unroll
        for (int t = 0; t < C; ++t) {
            float v = PM[t * LDM + tid];
#pragma unroll
            for (int s = 0; s < t; ++s) v = fmaf(-L[t * (C + 1) + s], x[s], v);
            x[t] = v;
            PM[t * LDM + tid] = v;
        }
    }
    __syncthreads();
    {
        // [X; b^T] [P' | M'], 96 x 96: rows 6 ty + i (outputs, then the state's rows), columns 6 tx + j
        const int tx = tid & 15, ty = tid >> 4;
        float acc[6][6] = {};
#pragma unroll 4
        for (int s = 0; s < C; ++s) {
            float x[6], m[6];
#pragma unroll
            for (int i = 0; i < 6; i += 2) {
                *reinterpret_cast<float2*>(x + i) = *reinterpret_cast<const float2*>(XB + s * LDM + 6 * ty + i);
                *reinterpret_cast<float2*>(m + i) = *reinterpret_cast<const float2*>(PM + s * LDM + 6 * tx + i);
            }
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int j = 0; j < 6; ++j) acc[i][j] = fmaf(x[i], m[j], acc[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const int row = 6 * ty + i;
            float v[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const int col = 6 * tx + j;
                if (row < C) v[j] = (col < D ? (float)pg[(C + row) * LD + col] : Y[row * (C + 1) + col - D]) - acc[i][j];
                else v[j] = last_s[row - C] * ((col < D ? (row - C == col ? 1.f : 0.f) : (float)bc[(C + col - D) * LD + row - C]) - acc[i][j]);
            }
#pragma unroll
            for (int j = 0; j < 6; j += 2) *reinterpret_cast<float2*>(W + row * R + 6 * tx + j) = make_float2(v[j], v[j + 1]);
        }
    }
}

// Sums the eight warps' parts of a tile of ROWS x 16 that a thread's accumulators hold (rows g + 8 j, columns 4 cg ..): through shared memory.
template <int NJ>
__device__ __forceinline__ void put_parts(float* red, int warp, int g, int cg, const float (&acc)[NJ][4])
{
#pragma unroll
    for (int j = 0; j < NJ; ++j) st4(red + ((size_t)warp * 8 * NJ + g + 8 * j) * WALK_COLS + 4 * cg, make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]));
}
template <int ROWS>
__device__ __forceinline__ float4 sum_parts(const float* red, int row, int cg)
{
    float4 v[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) v[w] = ld4(red + ((size_t)w * ROWS + row) * WALK_COLS + 4 * cg);
#pragma unroll
    for (int n = 4; n > 0; n >>= 1)              // as a tree: three roundings a number instead of seven
#pragma unroll
        for (int w = 0; w < n; ++w) v[w] = make_float4(v[w].x + v[w + n].x, v[w].y + v[w + n].y, v[w].z + v[w + n].z, v[w].w + v[w + n].w);
    return v[0];
}
// acc[j][c] += sum over four k of x[row g + 8 j][k ..] * y[k ..][4 cg + c]; x rows LDX floats apart, y rows WALK_LD
template <int NJ, int LDX>
__device__ __forceinline__ void tile_fma(float (&acc)[NJ][4], const float* x, const float* y)
{
    float yy[4][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) *reinterpret_cast<float4*>(yy[k]) = ld4(y + k * WALK_LD);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        float xx[4];
        *reinterpret_cast<float4*>(xx) = ld4(x + (size_t)8 * j * LDX);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[j][c] = fmaf(xx[k], yy[k][c], acc[j][c]);
    }
}

// Matrix memory and linear attention: a warp owns DK / 8 rows of the block's 16 columns of S.
template <int MODE, int DK> struct WalkSmem {
    static constexpr int C = 64, LDK = DK + 4, LDP = C + 4;
    static constexpr int Q = 0, P = Q + C * LDK, K = P + C * LDP, V = K + C * LDK, X = V + C * WALK_LD;     // floats; X: F, l, kappa, psum, ksum | the decays
    static constexpr int STAGE = X + (MODE == 0 ? 4 * C + DK : DK);
    static constexpr int S = 2 * STAGE, N = S + DK * WALK_LD, RED = N + DK, TOTAL = RED + 8 * C * WALK_COLS;      // N: n; RED: the warps' parts of the outputs
    static constexpr size_t BYTES = TOTAL * sizeof(float);
    static_assert(BYTES <= 227 * 1024, "a block's shared memory");
};

template <int MODE, int DK>
__global__ void __launch_bounds__(THREADS, 1) walk_kernel(ChunkArgs A)
{
    using L = WalkSmem<MODE, DK>;
    constexpr int C = L::C, LDK = L::LDK, LDP = L::LDP, KW = DK / 8;       // KW: rows of S a warp owns
    extern __shared__ __align__(16) float sm[];
    float *S_s = sm + L::S, *n_s = sm + L::N, *red = sm + L::RED;
    pdl_enter();
    const ScanArgs& a = A.s;
    const int seq = long_request<MODE>(A, blockIdx.x), h = blockIdx.y, c0 = blockIdx.z * WALK_COLS, dv = a.dv;
    if (seq < 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, cg = lane & 3;
    const int t_begin = a.q_start[seq], t_end = a.q_start[seq + 1];
    if (!takes_chunks<MODE>(a, h, t_begin, t_end)) return;
    const int slot = a.state_slot[seq];
    if (slot < 0 || slot >= a.num_slots) {
        if (tid == 0) report_status(a.status, SPY_STATUS_BAD_PAGE, t_begin);
        return;
    }
    float* st = a.state + ((size_t)slot * a.H + h) * a.record;
    float* st_nm = st + (size_t)DK * dv + (size_t)(c0 / 8) * (DK + 1);      // two copies of n and m: one for every 8 columns
    for (int idx = tid; idx < DK * 4; idx += THREADS) st4(S_s + (idx >> 2) * WALK_LD + 4 * (idx & 3), ld4(st + (size_t)(idx >> 2) * dv + c0 + 4 * (idx & 3)));
    float m = 0.f;
    if (MODE == 0) {
        for (int r = tid; r < DK; r += THREADS) n_s[r] = st_nm[r];
        m = st_nm[DK];
    }
    const int first_slot = chunk_slot(MODE, t_begin);
    auto request = [&](int t0, int stage) {
        const int n_tok = min(C, t_end - t0);
        float* base = sm + stage * L::STAGE;
        const float* mine = A.work + ((size_t)(first_slot + (t0 - t_begin) / C) * a.H + h) * chunk_floats(MODE, DK);
        const float* rows = a.proj + (size_t)t0 * a.ld;
        for (int idx = tid; idx < C * (DK / 4); idx += THREADS) {
            const int t = idx / (DK / 4), c = 4 * (idx - t * (DK / 4));
            if (MODE == 2) {
                cp_async16(base + L::Q + t * LDK + c, mine + C * C + t * DK + c);
                cp_async16(base + L::K + t * LDK + c, mine + C * C + C * DK + t * DK + c);
            } else if (t < n_tok) {
                cp_async16(base + L::Q + t * LDK + c, rows + (size_t)t * a.ld + a.off_q + h * DK + c);
                cp_async16(base + L::K + t * LDK + c, rows + (size_t)t * a.ld + a.off_k + h * DK + c);
            } else {
                st4(base + L::Q + t * LDK + c, make_float4(0.f, 0.f, 0.f, 0.f));
                st4(base + L::K + t * LDK + c, make_float4(0.f, 0.f, 0.f, 0.f));
            }
        }
        for (int idx = tid; idx < C * C / 4; idx += THREADS) cp_async16(base + L::P + (idx >> 4) * LDP + 4 * (idx & 15), mine + 4 * idx);
        for (int idx = tid; idx < C * 4; idx += THREADS) {
            const int t = idx >> 2, c = 4 * (idx & 3);
            if (t < n_tok) cp_async16(base + L::V + t * WALK_LD + c, rows + (size_t)t * a.ld + a.off_v + h * dv + c0 + c);
            else st4(base + L::V + t * WALK_LD + c, make_float4(0.f, 0.f, 0.f, 0.f));
        }
        const float* extra = mine + C * C + (MODE == 2 ? 2 * C * DK : 0);
        for (int idx = tid; idx < (MODE == 0 ? 4 * C + DK : DK) / 4; idx += THREADS) cp_async16(base + L::X + 4 * idx, extra + 4 * idx);
    };
    request(t_begin, 0);
    int stage = 0;
    for (int t0 = t_begin; t0 < t_end; t0 += C, stage ^= 1) {
        const int n_tok = min(C, t_end - t0);
        float* base = sm + stage * L::STAGE;
        float *Q = base + L::Q, *K = base + L::K, *P = base + L::P, *V = base + L::V, *X = base + L::X;
        cp_async_wait_all();
        __syncthreads();                           // this chunk has landed, the chunk before is done with
        if (t0 + C < t_end) request(t0 + C, stage ^ 1);
        float keep = 1.f, add = 1.f, nq = 0.f;     // of the old state and of the chunk's sum; n . q of token tid / 4
        const auto taken = [&](int t, float& alpha, float& beta) {     // what a token's output takes of the chunk and of the state ahead
            const float l = X[C + t], f = X[t] + m, top = fmaxf(f, l);
            alpha = expf(l - top);
            beta = expf(f - top);
        };
        if (MODE == 0) {
            taken(C - 1, add, keep);               // behind the chunk (padding tokens change nothing)
            const int t = tid >> 2, part = tid & 3;
#pragma unroll
            for (int c = 0; c < DK / 4; c += 4) nq = dot4(ld4(Q + t * LDK + 4 * c + 4 * part), ld4(n_s + 4 * c + 4 * part), nq);
            nq += __shfl_xor_sync(0xffffffffu, nq, 1);
            nq += __shfl_xor_sync(0xffffffffu, nq, 2);
        }
        // what the state ahead of the chunk gives: this warp's rows of it; then this warp's share of the chunk's own tokens
        float acc[8][4] = {};
#pragma unroll
        for (int k = 0; k < KW; k += 4) tile_fma<8, LDK>(acc, Q + g * LDK + warp * KW + k, S_s + (warp * KW + k) * WALK_LD + 4 * cg);
        if (MODE == 0) {
            float own[8][4] = {};
#pragma unroll
            for (int k = 0; k < C / 8; k += 4) tile_fma<8, LDP>(own, P + g * LDP + warp * (C / 8) + k, V + (warp * (C / 8) + k) * WALK_LD + 4 * cg);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float alpha, beta;
                taken(g + 8 * j, alpha, beta);
                beta *= a.q_scale;
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[j][c] = fmaf(beta, acc[j][c], alpha * own[j][c]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < C / 8; k += 4) tile_fma<8, LDP>(acc, P + g * LDP + warp * (C / 8) + k, V + (warp * (C / 8) + k) * WALK_LD + 4 * cg);
        }
        put_parts<8>(red, warp, g, cg, acc);
        // The state behind the chunk.  A warp's rows (no other warp reads them): a lane has half of them and four columns, over every fourth
        // token; the four sums meet by shuffles, each lane keeping a quarter.
        __syncwarp();
        {
            constexpr int RL = KW / 2;             // rows of a lane
            const int rg = lane >> 4, sg = lane >> 2 & 3, r0 = warp * KW + rg * RL;
            float u[RL][4] = {};
#pragma unroll 4
            for (int s = sg; s < C; s += 4) {
                float kk[RL], vv[4];
#pragma unroll
                for (int r = 0; r < RL; r += 4) *reinterpret_cast<float4*>(kk + r) = ld4(K + s * LDK + r0 + r);
                *reinterpret_cast<float4*>(vv) = ld4(V + s * WALK_LD + 4 * cg);
                if (MODE == 0) {
                    const float f = X[2 * C + s] * add;
#pragma unroll
                    for (int c = 0; c < 4; ++c) vv[c] *= f;
                }
#pragma unroll
                for (int r = 0; r < RL; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) u[r][c] = fmaf(kk[r], vv[c], u[r][c]);
            }
            // lanes sg and sg ^ 2 halve the rows, then sg and sg ^ 1: a lane ends with RL / 4 rows
            constexpr int H2 = RL / 2, H4 = RL / 4;
            const bool up2 = (sg & 2) != 0, up1 = (sg & 1) != 0;
            float half[H2][4], mine[H4][4];
#pragma unroll
            for (int r = 0; r < H2; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float give = up2 ? u[r][c] : u[r + H2][c], own = up2 ? u[r + H2][c] : u[r][c];
                    half[r][c] = own + __shfl_xor_sync(0xffffffffu, give, 8);
                }
#pragma unroll
            for (int r = 0; r < H4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float give = up1 ? half[r][c] : half[r + H4][c], own = up1 ? half[r + H4][c] : half[r][c];
                    mine[r][c] = own + __shfl_xor_sync(0xffffffffu, give, 4);
                }
#pragma unroll
            for (int r = 0; r < H4; ++r) {
                const int row = r0 + (up2 ? H2 : 0) + (up1 ? H4 : 0) + r;
                float* s = S_s + row * WALK_LD + 4 * cg;
                const float d = MODE == 0 ? keep : X[row];
                float4 o = ld4(s);
                st4(s, make_float4(fmaf(d, o.x, mine[r][0]), fmaf(d, o.y, mine[r][1]), fmaf(d, o.z, mine[r][2]), fmaf(d, o.w, mine[r][3])));
            }
        }
        __syncthreads();                           // the outputs' parts are there; n has been read
        {
            const int t = tid >> 2, part = tid & 3;
            float4 o = sum_parts<C>(red, t, part);
            if (MODE == 0) {
                float alpha, beta;
                taken(t, alpha, beta);
                nq = fmaf(beta * a.q_scale, nq, alpha * X[3 * C + t]);
                const float d = fmaxf(fabsf(nq), expf(-fmaxf(X[t] + m, X[C + t]))) + 1e-6f;
                o = make_float4(o.x / d, o.y / d, o.z / d, o.w / d);
            }
            if (t < n_tok) st4(a.out + (size_t)(t0 + t) * a.H * dv + h * dv + c0 + 4 * part, o);
        }
        if (MODE == 0) {
            for (int r = tid; r < DK; r += THREADS) n_s[r] = fmaf(keep, n_s[r], add * X[4 * C + r]);
            m = fmaxf(X[C - 1] + m, X[C + C - 1]);
        }
    }
    __syncthreads();
    for (int idx = tid; idx < DK * 4; idx += THREADS) st4(st + (size_t)(idx >> 2) * dv + c0 + 4 * (idx & 3), ld4(S_s + (idx >> 2) * WALK_LD + 4 * (idx & 3)));
    if (MODE == 0) {
        for (int cp = 0; cp < 2; ++cp) {
            for (int r = tid; r < DK; r += THREADS) st_nm[(size_t)cp * (DK + 1) + r] = n_s[r];
            if (tid == 0) st_nm[(size_t)cp * (DK + 1) + DK] = m;
        }
    }
}

// Delta rule: [outputs of 32 tokens; the state's 64 rows] = W [the state; the values], a warp 12 of the 96 columns of W.
struct DeltaSmem {
    static constexpr int C = 32, D = 64, R = C + D, LDW = R + 4;
    static constexpr int W = 0, V = W + R * LDW, STAGE = V + C * WALK_LD;
    static constexpr int S = 2 * STAGE, RED = S + D * WALK_LD, TOTAL = RED + 8 * R * WALK_COLS;
    static constexpr size_t BYTES = TOTAL * sizeof(float);
};

__global__ void __launch_bounds__(THREADS, 1) walk_delta_kernel(ChunkArgs A)
{
    using L = DeltaSmem;
    constexpr int C = L::C, D = L::D, R = L::R, LDW = L::LDW, KW = R / 8;
    extern __shared__ __align__(16) float sm[];
    float *S_s = sm + L::S, *red = sm + L::RED;
    pdl_enter();
    const ScanArgs& a = A.s;
    const int seq = long_request<1>(A, blockIdx.x), h = blockIdx.y, c0 = blockIdx.z * WALK_COLS;
    if (seq < 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, cg = lane & 3;
    const int t_begin = a.q_start[seq], t_end = a.q_start[seq + 1];
    if (!takes_chunks<1>(a, h, t_begin, t_end)) return;
    const int slot = a.state_slot[seq];
    if (slot < 0 || slot >= a.num_slots) {
        if (tid == 0) report_status(a.status, SPY_STATUS_BAD_PAGE, t_begin);
        return;
    }
    float* st = a.state + ((size_t)slot * a.H + h) * a.record;
    st4(S_s + (tid >> 2) * WALK_LD + 4 * (tid & 3), ld4(st + (size_t)(tid >> 2) * D + c0 + 4 * (tid & 3)));      // 64 rows of four quads: one a thread
    const int first_slot = chunk_slot(1, t_begin);
    auto request = [&](int t0, int stage) {
        const int n_tok = min(C, t_end - t0);
        float* base = sm + stage * L::STAGE;
        const float* W = A.work + ((size_t)(first_slot + (t0 - t_begin) / C) * a.H + h) * chunk_floats(1, D);
        for (int idx = tid; idx < R * R / 4; idx += THREADS) cp_async16(base + L::W + idx / (R / 4) * LDW + 4 * (idx % (R / 4)), W + 4 * idx);
        if (tid < C * 4) {
            const int t = tid >> 2, c = 4 * (tid & 3);
            if (t < n_tok) cp_async16(base + L::V + t * WALK_LD + c, a.proj + (size_t)(t0 + t) * a.ld + a.off_v + h * D + c0 + c);
            else st4(base + L::V + t * WALK_LD + c, make_float4(0.f, 0.f, 0.f, 0.f));
        }
    };
    request(t_begin, 0);
    int stage = 0;
    for (int t0 = t_begin; t0 < t_end; t0 += C, stage ^= 1) {
        const int n_tok = min(C, t_end - t0);
        const float *W = sm + stage * L::STAGE + L::W, *V = sm + stage * L::STAGE + L::V;
        cp_async_wait_all();
        __syncthreads();                           // this chunk has landed, the state of the chunk before is written
        if (t0 + C < t_end) request(t0 + C, stage ^ 1);
        float acc[R / 8][4] = {};
#pragma unroll
        for (int i = 0; i < KW; i += 4) {
            const int k = warp * KW + i;           // 4 consecutive columns of W: all of the state or all of the values
            tile_fma<R / 8, LDW>(acc, W + g * LDW + k, (k < D ? S_s + k * WALK_LD : V + (k - D) * WALK_LD) + 4 * cg);
        }
        put_parts<R / 8>(red, warp, g, cg, acc);
        __syncthreads();
        for (int idx = tid; idx < R * 4; idx += THREADS) {
            const int row = idx >> 2, part = idx & 3;
            const float4 o = sum_parts<R>(red, row, part);
            if (row >= C) st4(S_s + (row - C) * WALK_LD + 4 * part, o);
            else if (row < n_tok) st4(a.out + (size_t)(t0 + row) * a.H * D + h * D + c0 + 4 * part, o);
        }
    }
    __syncthreads();
    st4(st + (size_t)(tid >> 2) * D + c0 + 4 * (tid & 3), ld4(S_s + (tid >> 2) * WALK_LD + 4 * (tid & 3)));
}

// Which steps take chunks: keys of 64 or 128 channels (the delta rule's states of 64 x 64), value columns in sixteens, requests long enough (chunk_alone),
// factors that fit 512 MB (130 K tokens of 8 heads of the matrix memory).  Only the long requests count: those of a token or a few beside
// them take no place in the scratch and no blocks of these kernels, and are walked by tokens behind them.  Measured, the step's kernels together (us, by tokens / in chunks): one prompt
// portion of 1,501 tokens beside 47 replies, matrix memory of 8 heads 705 / 290, delta rule of 32 heads 739 / 341, linear attention of 16 heads 1,023 / 454; of 200 beside 8
// 98 / 59, 101 / 61, 142 / 95; of 200 beside 250 866 / 811, 389 / 363, 945 / 926; 60 tokens each of 16 beside one of 200 276 / 221, 182 / 169, 392 / 375.
// The delta rule with up to 32 (long request, head) pairs: with more, the walk by tokens has work for most SMs and does fewer additions (32 heads, by tokens / in
// chunks: one request of 160 tokens 51 / 44, two 64 / 73; one of 1,024 313 / 190, two 385 / 354).
static long long chunk_work_floats(int mode, int tokens, int long_requests, int longest, int H, int dk, int dv)
{
    if (long_requests <= 0 || longest < (long_requests > 1 ? chunk_min(mode) : chunk_alone(mode)) || dv % WALK_COLS != 0 || dv / WALK_COLS > 65535) return 0;
    if (mode == 1 ? dk != 64 || dv != 64 || (long long)long_requests * H > 32 : dk != 64 && dk != 128) return 0;
    const long long floats = (long long)chunk_slot(mode, tokens) * H * (chunk_floats(mode, dk) + 4LL);
    return floats <= (128LL << 20) ? floats : 0;
}

// walks: the most requests of chunk_min tokens that there can be.
template <int MODE> static int launch_chunks(ScanArgs& S, int tokens, int num_seqs, int walks, float* work, cudaStream_t stream)
{
    const int slots = chunk_slot(MODE, tokens);
    ChunkArgs A = {S, work, nullptr, num_seqs};
    A.flags = reinterpret_cast<int*>(work + (size_t)slots * S.H * chunk_floats(MODE, S.dk));
    A.s.flags = S.flags = A.flags;
    const dim3 chunks(slots, S.H), walk(walks, S.H, S.dv / WALK_COLS), threads(THREADS);
    if constexpr (MODE == 1) {
        constexpr int C = 32, D = 64, R = C + D;
        constexpr size_t factors = 4 * C * (D + 2) * sizeof(double) + (2 * C * (R + 4) + 2 * C * (C + 1)) * sizeof(float);
        SPY_ONCE_PER_DEVICE {
            SPY_CUDA(cudaFuncSetAttribute(chunk_delta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)factors));
            SPY_CUDA(cudaFuncSetAttribute(walk_delta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DeltaSmem::BYTES));
        }
        spy_launch(chunk_delta_kernel, chunks, threads, factors, stream, A);
        spy_launch(walk_delta_kernel, walk, threads, DeltaSmem::BYTES, stream, A);
    } else {
        void (*const chunk64)(ChunkArgs) = MODE == 0 ? chunk_memory_kernel<64> : chunk_linear_kernel<64>;
        void (*const chunk128)(ChunkArgs) = MODE == 0 ? chunk_memory_kernel<128> : chunk_linear_kernel<128>;
        const auto factors = [](int dk) { return (MODE == 0 ? 2 : 3) * 64 * (size_t)(dk + 4) * sizeof(float); };
        SPY_ONCE_PER_DEVICE {
            SPY_CUDA(cudaFuncSetAttribute(chunk64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)factors(64)));
            SPY_CUDA(cudaFuncSetAttribute(chunk128, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)factors(128)));
            SPY_CUDA(cudaFuncSetAttribute(walk_kernel<MODE, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WalkSmem<MODE, 64>::BYTES));
            SPY_CUDA(cudaFuncSetAttribute(walk_kernel<MODE, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WalkSmem<MODE, 128>::BYTES));
        }
        spy_launch(S.dk == 64 ? chunk64 : chunk128, chunks, threads, factors(S.dk), stream, A);
        if (S.dk == 64) spy_launch(walk_kernel<MODE, 64>, walk, threads, WalkSmem<MODE, 64>::BYTES, stream, A);
        else spy_launch(walk_kernel<MODE, 128>, walk, threads, WalkSmem<MODE, 128>::BYTES, stream, A);
    }
    SPY_CHECK_LAUNCH("recurrence (chunks)");
    return 0;
}

template <int MODE, int RG> static int launch_scan_rg(ScanArgs& A, int num_seqs, int longest, cudaStream_t stream)
{
    constexpr int CTB = 8 * (32 / RG);
    const int tiles = (A.dv + CTB - 1) / CTB;
    int nr = 2;
    while (RG * nr < A.dk) nr *= 2;
    if (nr > 64) SPY_FAIL("recurrence: a key size of %d exceeds the kernel's %d", A.dk, 64 * RG);
    // tokens a chunk: 32, fewer when a request never brings that many or when the vectors of 32 would not fit
    int tc = 32;
    while (tc > 1 && tc / 2 >= longest) tc /= 2;
    auto bytes = [&](int n) {
        const size_t stage = (MODE == 1 ? 4 : (MODE == 2 ? 3 : 2)) * (size_t)n * RG * nr + (size_t)n * CTB + 2 * (size_t)n;      // one stage of a chunk's vectors
        const size_t staged = (2 * stage + (size_t)n * CTB + 11 * (size_t)n) * sizeof(float);
        const size_t tile = (size_t)A.dk * (CTB + 4) * sizeof(float);
        return staged > tile ? staged : tile;
    };
    while (tc > 1 && bytes(tc) > 100 * 1024) tc /= 2;
    const size_t smem = bytes(tc);
    if (smem > 227 * 1024) SPY_FAIL("recurrence: a key size of %d does not fit a block's shared memory", A.dk);
    void (*kernel)(ScanArgs, int) = nullptr;
    switch (nr) {
        case 2: kernel = scan_kernel<MODE, 2, RG>; break;
        case 4: kernel = scan_kernel<MODE, 4, RG>; break;
        case 8: kernel = scan_kernel<MODE, 8, RG>; break;
        case 16: kernel = scan_kernel<MODE, 16, RG>; break;
        case 32: kernel = scan_kernel<MODE, 32, RG>; break;
        default: kernel = scan_kernel<MODE, 64, RG>; break;
    }
    if (smem > 48 * 1024) SPY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    spy_launch_in_order(kernel, dim3(num_seqs, A.H, tiles), dim3(THREADS), smem, stream, A, tc);
    SPY_CHECK_LAUNCH("recurrence scan");
    return 0;
}

template <int MODE> static int launch_scan_mode(ScanArgs& A, int num_seqs, int longest, cudaStream_t stream)
{
    if (longest <= 1) {     // every request brings one token
        const int tiles = (A.dv + CT - 1) / CT;
        int nr = 2;
        while (8 * nr < A.dk) nr *= 2;
        if (nr > 64) SPY_FAIL("recurrence: a key size of %d exceeds the kernel's 512", A.dk);
        void (*dk_kernel)(ScanArgs) = nullptr;
        switch (nr) {
            case 2: dk_kernel = scan_decode_kernel<MODE, 2>; break;
            case 4: dk_kernel = scan_decode_kernel<MODE, 4>; break;
            case 8: dk_kernel = scan_decode_kernel<MODE, 8>; break;
            case 16: dk_kernel = scan_decode_kernel<MODE, 16>; break;
            case 32: dk_kernel = scan_decode_kernel<MODE, 32>; break;
            default: dk_kernel = scan_decode_kernel<MODE, 64>; break;
        }
        const size_t vec_bytes = (MODE == 1 ? 4 : (MODE == 2 ? 3 : 2)) * (size_t)A.dk * sizeof(float);
        spy_launch(dk_kernel, dim3(num_seqs, A.H, tiles), dim3(THREADS), vec_bytes, stream, A);
        SPY_CHECK_LAUNCH("recurrence scan (decoding)");
        return 0;
    }
    // the widest tiles (32, 16 or 8 columns a block) that still give (nearly) every SM a block; key sizes above 512 need the narrower ones
    const int sms = spy_sm_count();
    const long long heads = (long long)num_seqs * A.H;
    static int forced = -1;                      // SPYINFER_SCAN_RG = 8, 16 or 32 in the environment fixes the tile width (for measurements)
    if (forced < 0) {
        const char* e = getenv("SPYINFER_SCAN_RG");
        forced = e != nullptr ? atoi(e) : 0;
    }
    if (forced == 8 && A.dk <= 512) return launch_scan_rg<MODE, 8>(A, num_seqs, longest, stream);
    if (forced == 16 && A.dk <= 1024) return launch_scan_rg<MODE, 16>(A, num_seqs, longest, stream);
    if (forced == 32) return launch_scan_rg<MODE, 32>(A, num_seqs, longest, stream);
    // measured on one request of 8 heads, 128 x 256: 64 blocks of 32 columns 0.79 ms, 128 of 16 columns 0.64, 256 of 8 columns 0.75
    if (A.dk <= 512 && heads * ((A.dv + 31) / 32) >= sms) return launch_scan_rg<MODE, 8>(A, num_seqs, longest, stream);
    if (A.dk <= 1024 && 4 * heads * ((A.dv + 15) / 16) >= 3 * sms) return launch_scan_rg<MODE, 16>(A, num_seqs, longest, stream);
    return launch_scan_rg<MODE, 32>(A, num_seqs, longest, stream);
}

// work: null (every request is walked by tokens), or scratch of spy_scan_chunk_floats floats for `tokens` tokens, 16-byte aligned;
// walks: the most requests that can bring chunk_min tokens in any step that this launch serves.
static int launch_scan(int mode, ScanArgs& A, int num_seqs, int longest, int tokens, float* work, long long work_floats, int walks, cudaStream_t stream)
{
    if (num_seqs <= 0) return 0;
    if (A.H <= 0 || A.dk <= 0 || A.dv <= 0) SPY_FAIL("recurrence: heads %d, key size %d and value size %d must be positive", A.H, A.dk, A.dv);
    if (A.H > 65535) SPY_FAIL("recurrence: %d heads exceed the grid limit", A.H);
    if ((A.dv + CT - 1) / CT > 65535) SPY_FAIL("recurrence: a value size of %d exceeds the grid limit", A.dv);
    // chunks want whole 16-byte pieces of every row, state and output
    const bool aligned = ((A.ld | A.off_q | A.off_k | A.off_v | (mode == 1 ? A.off_x1 : 0)) & 3) == 0 && A.record % 4 == 0 &&
                         ((reinterpret_cast<uintptr_t>(A.proj) | reinterpret_cast<uintptr_t>(A.state) | reinterpret_cast<uintptr_t>(A.out) |
                           reinterpret_cast<uintptr_t>(work)) & 15) == 0;
    if (work != nullptr && walks > 0 && aligned) {
        const long long need = chunk_work_floats(mode, tokens, 1, tokens, A.H, A.dk, A.dv);
        if (need <= 0 || need > work_floats) SPY_FAIL("recurrence: %lld floats of scratch for %d tokens, %lld are needed", work_floats, tokens, need);
        const int rc = mode == 0 ? launch_chunks<0>(A, tokens, num_seqs, walks, work, stream)
                       : mode == 1 ? launch_chunks<1>(A, tokens, num_seqs, walks, work, stream) : launch_chunks<2>(A, tokens, num_seqs, walks, work, stream);
        if (rc) return rc;
    }
    if (mode == 2) return launch_scan_mode<2>(A, num_seqs, longest, stream);
    return mode == 0 ? launch_scan_mode<0>(A, num_seqs, longest, stream) : launch_scan_mode<1>(A, num_seqs, longest, stream);
}

// The tokens from which on a request is walked in chunks where its step takes them.
extern "C" int spy_scan_chunk_min(int mode) { return chunk_min(mode); }

// Floats of scratch with which a step of `tokens` tokens takes chunks, `long_requests` of its requests bringing chunk_min tokens or more and the longest
// `longest`; 0: it does not take them.
extern "C" long long spy_scan_chunk_floats(int mode, int tokens, int long_requests, int longest, int H, int dk, int dv)
{
    return chunk_work_floats(mode, tokens, long_requests, longest, H, dk, dv);
}

// State record of one head, in floats.
extern "C" long long spy_mlstm_record(int dk, int dv) { return ((long long)dk * dv + (long long)((dv + 7) / 8) * (dk + 1) + 3) / 4 * 4; }

extern "C" int spy_mlstm_scan(const float* proj, long long ld, int off_q, int off_k, int off_v, int off_i, int off_f, const float* bias_i, const float* bias_f,
                              float* state, int num_slots, const int* q_start, const int* state_slot, int num_seqs, int longest, float* out, int H, int dk,
                              int dv, float q_scale, float cap, int* status, cudaStream_t stream, int tokens, float* work, long long work_floats,
                              int walks)
{
    if (!(cap > 0.f)) SPY_FAIL("mlstm: the gates' cap must be positive");
    ScanArgs A = {proj, ld, off_q, off_k, off_v, off_i, off_f, nullptr, bias_i, bias_f, state, spy_mlstm_record(dk, dv), num_slots, q_start, state_slot, out,
                  H, dk, dv, q_scale, cap, status, nullptr};
    return launch_scan(0, A, num_seqs, longest, tokens, work, work_floats, walks, stream);
}

extern "C" int spy_delta_scan(const float* proj, long long ld, int off_r, int off_k, int off_v, int off_a, const float* decay_pre, const float* bias_a,
                              const float* decay_offset, float* state, int num_slots, const int* q_start, const int* state_slot, int num_seqs, int longest,
                              float* out, int H, int dk, int* status, cudaStream_t stream, int tokens, float* work, long long work_floats,
                              int walks)
{
    ScanArgs A = {proj, ld, off_r, off_k, off_v, off_a, 0, decay_pre, bias_a, decay_offset, state, (long long)dk * dk, num_slots, q_start, state_slot, out,
                  H, dk, dk, 1.0f, 1.0f, status, nullptr};
    return launch_scan(1, A, num_seqs, longest, tokens, work, work_floats, walks, stream);
}

// Gated linear attention with a decay per key channel: proj holds q, k, v at `off_*`; decay_pre [T, H * dk] the decay's
// pre-activation z, to which decay_bias [H * dk] is added: a = exp(logsigmoid(z + bias) / tau).  q is scaled by q_scale.
extern "C" int spy_gla_scan(const float* proj, long long ld, int off_q, int off_k, int off_v, const float* decay_pre, const float* decay_bias, float inv_tau,
                            float* state, int num_slots, const int* q_start, const int* state_slot, int num_seqs, int longest, float* out, int H, int dk, int dv,
                            float q_scale, int* status, cudaStream_t stream, int tokens, float* work, long long work_floats,
                              int walks)
{
    if (!(inv_tau > 0.f)) SPY_FAIL("gated linear attention: tau must be positive");
    ScanArgs A = {proj, ld, off_q, off_k, off_v, 0, 0, decay_pre, nullptr, decay_bias, state, (long long)dk * dv, num_slots, q_start, state_slot, out,
                  H, dk, dv, q_scale, inv_tau, status, nullptr};
    return launch_scan(2, A, num_seqs, longest, tokens, work, work_floats, walks, stream);
}

// out[t, j] = act(proj[t, off + j]) for j < n: the inner activation of a two-step (low-rank) projection; act 0: tanh, 1: none.
template <typename TO>
__global__ void tanh_cols_kernel(const float* __restrict__ proj, long long ld, int off, int n, TO* __restrict__ out, long long total, int act)
{
    pdl_enter();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (; i < total; i += stride) {
        const long long t = i / n;
        const float x = proj[t * ld + off + (i - t * n)];
        out[i] = from_f32<TO>(act == 0 ? tanhf(x) : x);
    }
}

extern "C" int spy_tanh_cols(const float* proj, long long ld, int off, int n, void* out, int out_dtype, int tokens, cudaStream_t stream, int act)
{
    if (tokens <= 0 || n <= 0) return 0;
    if (act != 0 && act != 1) SPY_FAIL("tanh_cols: activation %d (0: tanh, 1: none)", act);
    const long long total = (long long)tokens * n;
    long long blocks = (total + 255) / 256;
    const long long most = (long long)spy_sm_count() * 32;
    if (blocks > most) blocks = most;
    SPY_DISPATCH_DTYPE(out_dtype, TO, {
        spy_launch(tanh_cols_kernel<TO>, dim3((int)blocks), dim3(256), 0, stream, proj, ld, off, n, (TO*)out, total, act);
    })
    SPY_CHECK_LAUNCH("tanh_cols");
    return 0;
}
