// Attention over the paged cache for any mix of queries, every head size, every page size, 32-bit
// or bfloat16 storage, everything computed in 32-bit with expf.  Two kernels: head sizes up to 128 in
// quads take the one for several query rows a block (attention_rows_kernel), the others one block per
// (query token, head).  It is the
// engine's float32 path and the fallback of the bfloat16 path for sizes its fast kernels
// refuse.  A cache of one plane (`planes` = 1) holds keys only and the values are the keys
// themselves (a latent that both are made of): V rows are then read from the K plane.  Head
// sizes that are no multiple of 4 take element-wise loads.
//
// A query at position p of sequence s sees the keys j with lo <= j <= p, lo = 0 or
// p - window + 1; key j lies in page block_table[s, j / page_size], slot j % page_size.
// kv head = head / (nh / nkv); score = (q . k) * scale; p = exp(score - max) / sum;
// o = sum p v.  Formula: spymaster2h/spyinfer src/backends/cpu/cpu_attention.cpp:89-135.
// Keys are processed in chunks of 128 that start at multiples of 128 of the absolute
// position, so the result of a query does not depend on how the batch was cut.
// Two options of the mask and the softmax: with a window, `keep_first` > 0 lets every query also see
// the keys at the sequence's first keep_first positions (at their true positions); `sink` != 0 adds one
// to the softmax's denominator (a key of score 0 that has no value): p = exp(score) / (1 + sum exp(score)).
// SpyScores (common.cuh) caps the scores, takes a distance bias off, adds a learned sink a head, scales the result.
#include "common.cuh"

SPY_MODULE(spy_attention_generic)

constexpr int CHUNK = 128;
constexpr int ACC = 8;       // output elements a thread owns: head sizes up to ACC * CHUNK

template <typename T> struct Vec4;
template <> struct Vec4<float> {
    static __device__ __forceinline__ void load(const float* p, float (&v)[4])
    {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    }
};
template <> struct Vec4<bf16> {
    static __device__ __forceinline__ void load(const bf16* p, float (&v)[4])
    {
        const uint2 x = *reinterpret_cast<const uint2*>(p);
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&x.x);
        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&x.y);
        v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
    }
};

template <typename TA, typename TC>
__global__ void __launch_bounds__(CHUNK)
attention_generic_kernel(const TA* __restrict__ q, long long q_row_stride, TA* __restrict__ out, const TC* __restrict__ pages,
                         const int* __restrict__ block_table, int table_width, int page_size, int num_pages, int nh, int nkv, int hd,
                         const int* __restrict__ positions, const int* __restrict__ seq_of_token, int window, float scale, int* status, int planes,
                         int keep_first, int sink, SpyScores sc)
{
    extern __shared__ float smem[];
    pdl_enter();
    float* q_s = smem;                       // hd
    float* p_s = q_s + hd;                   // CHUNK
    long long* row_s = (long long*)(p_s + CHUNK + (hd & 1));  // CHUNK offsets of K rows (elements); 8-byte aligned: hd + (hd & 1) and CHUNK are even
    float* scratch = (float*)(row_s + CHUNK);      // 33

    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int pos = positions[t];
    const int seq = seq_of_token[t];
    const int kvh = h / (nh / nkv);
    const int* bt = block_table + (size_t)seq * table_width;
    const long long v_offset = planes == 2 ? (long long)nkv * page_size * hd : 0;  // from a K row to its V row (one plane: the values are the keys)
    const bool quads = (hd & 3) == 0;

    const TA* q_row = q + (size_t)t * q_row_stride + (size_t)h * hd;
    for (int d = tid; d < hd; d += CHUNK) q_s[d] = to_f32(q_row[d]);

    const int lo = spy_first_key(pos, window);
    float m = -INFINITY, l = 0.f;
    float acc[ACC];                       // dims tid, tid + 128, tid + 256, ...
#pragma unroll
    for (int r = 0; r < ACC; ++r) acc[r] = 0.f;
    __syncthreads();

    const int kept = min(keep_first, lo);             // the keys 0 .. kept - 1 lie before the window and are seen all the same
    const int kept_chunks = (kept + CHUNK - 1) / CHUNK;
    for (int c = 0; c <= pos / CHUNK; ++c) {
        if (c >= kept_chunks && c < lo / CHUNK) {
            c = lo / CHUNK - 1;                       // nothing to see between the kept keys and the window
            continue;
        }
        const int j = c * CHUNK + tid;
        bool valid = (j >= lo || j < kept) && j <= pos;
        long long row = 0;
        if (valid) {
            const int lp = j / page_size;
            const int page = lp < table_width ? bt[lp] : -1;
            if (page < 0 || page >= num_pages) {
                report_status(status, SPY_STATUS_BAD_PAGE, t);
                valid = false;
            } else {
                row = ((((long long)page * planes) * nkv + kvh) * page_size + j % page_size) * hd;
            }
        }
        float s = -INFINITY;
        if (valid) {
            const TC* k = pages + row;
            float dot = 0.f;
            if (quads) {
                for (int d = 0; d < hd; d += 4) {
                    float kv[4];
                    Vec4<TC>::load(k + d, kv);
                    dot = fmaf(q_s[d], kv[0], dot);
                    dot = fmaf(q_s[d + 1], kv[1], dot);
                    dot = fmaf(q_s[d + 2], kv[2], dot);
                    dot = fmaf(q_s[d + 3], kv[3], dot);
                }
            } else {
                for (int d = 0; d < hd; ++d) dot = fmaf(q_s[d], to_f32(k[d]), dot);
            }
            s = dot * scale;
            if (sc.softcap > 0.f) s = sc.softcap * tanhf(s / sc.softcap);
            if (sc.slopes != nullptr) s -= sc.slopes[h] * (float)(pos - j);
        }
        const float chunk_max = block_max(s, scratch);
        const float m_new = fmaxf(m, chunk_max);
        if (m_new == -INFINITY) continue;  // every key of the chunk was refused: nothing to add (uniform over the block)
        const float p = valid ? expf(s - m_new) : 0.f;
        const float alpha = m == -INFINITY ? 0.f : expf(m - m_new);
        p_s[tid] = p;
        row_s[tid] = row;
        const float chunk_sum = block_sum(p, scratch);  // its barriers also publish p_s and row_s
        l = l * alpha + chunk_sum;
        m = m_new;
        const int first = (c < kept_chunks ? 0 : max(lo, c * CHUNK) - c * CHUNK), last = min(pos, c * CHUNK + CHUNK - 1) - c * CHUNK;
        const int gap_first = c < kept_chunks ? kept - c * CHUNK : CHUNK, gap_end = c < kept_chunks ? lo - c * CHUNK : 0;   // [gap_first, gap_end): unseen keys inside the chunk
#pragma unroll
        for (int r = 0; r < ACC; ++r) {
            const int d = tid + r * CHUNK;
            if (d < hd) {
                float a = acc[r] * alpha;
                for (int jj = first; jj <= last; ++jj) {
                    if (jj >= gap_first && jj < gap_end) continue;
                    a = fmaf(p_s[jj], to_f32(pages[row_s[jj] + v_offset + d]), a);
                }
                acc[r] = a;
            }
        }
        __syncthreads();  // p_s and row_s are rewritten by the next chunk
    }
    if (sink) l += m == -INFINITY ? 1.f : expf(-m);      // the key of score 0 without a value
    if (sc.sinks != nullptr) l += m == -INFINITY ? 1.f : expf(sc.sinks[h] - m);      // (too large for 32-bit: the result is 0, as it should be)
    const float os = sc.out_scale != nullptr ? sc.out_scale[(size_t)t * nh + h] : 1.f;
    TA* o_row = out + ((size_t)t * nh + h) * hd;
#pragma unroll
    for (int r = 0; r < ACC; ++r) {
        const int d = tid + r * CHUNK;
        if (d < hd) o_row[d] = from_f32<TA>(l > 0.f ? acc[r] / l * os : 0.f);
    }
}

// ---- head sizes up to 128 in quads: a block takes several query rows of one kv head -----------------------------------------
// The kernel above reads every key and value once a (token, head) and waits for each: 179 us a layer for 4 requests with up to 700
// keys (32 heads, 8 kv heads of 128, 32-bit), where the cache takes 5 us to read, and 290 us for a prompt of 300 tokens.  Here a
// block takes R query rows (the heads of a kv head, times up to 16 / heads tokens of one sequence where tokens outnumber the
// sequences), so a key row serves all of them: staged through shared memory in whole rows, half a head at a time, one key a thread for
// the scores (its row read in quads, the queries broadcast), one dimension a thread for the values, eight of them requested ahead.
// With few rows (decoding) the chunks of a row go to blocks of their own and attention_merge_kernel adds them: 33 us for those 4 requests,
// 114 us for the 300 tokens (both with the merge).
//
// A chunk's maximum, sum and value sum are formed for themselves and added to the row's in the order of the chunks, whether one
// block walks them or many, and a row's numbers do not depend on the rows beside it: results do not depend on the cut.
// Value sums are formed with probabilities divided by CHUNK (a power of two: the same bits), so that a chunk's never exceed its largest value: relative to
// the chunk's own maximum they could overflow where the chunk weighs next to nothing in its row.
// A key that a row does not see is left out (p_s = -1), not multiplied by zero: what lies there may not be a finite number.
struct AttnArgs {
    long long q_row_stride;
    const int* block_table;
    int table_width, page_size, num_pages, nh, nkv, hd;
    const int* positions;
    const int* seq_of_token;
    int tokens, window;
    float scale;
    int* status;
    int planes, keep_first, sink;
    SpyScores sc;
    int heads, per_tile, head_groups;   // heads and tokens of a block, blocks a kv head
    float* partial;                     // [tokens][nh][max_chunks][hd + 2]: value sums, then the maximum and the sum
    int max_chunks;
};

constexpr int KD = 64;                  // dimensions of the keys staged at a time
constexpr int KLD = KD + 4;

// The running softmax of a row takes a chunk's: the factors of what was there and of what comes; false: there is no score above -inf so
// far, nothing to add (as attention_generic_kernel leaves out chunks until one has such a score).  A chunk without one behind others is
// added as it is: its probabilities are 0, or NaN where a score is NaN; a row with a NaN in its sum is stored as 0.
__device__ __forceinline__ bool take_chunk(float& m, float& l, float mc, float lc, float& alpha, float& beta)
{
    const float m_new = fmaxf(m, mc);
    if (m_new == -INFINITY) return false;
    alpha = m == -INFINITY ? 0.f : expf(m - m_new);
    beta = mc == -INFINITY ? 1.f : expf(mc - m_new);
    l = fmaf(l, alpha, lc * beta);
    m = m_new;
    return true;
}

template <typename TA>
__device__ __forceinline__ void store_row(const AttnArgs& A, TA* out, int t, int h, int d, float acc, float m, float l)
{
    if (A.sink) l += m == -INFINITY ? 1.f : expf(-m);
    if (A.sc.sinks != nullptr) l += m == -INFINITY ? 1.f : expf(A.sc.sinks[h] - m);
    const float os = A.sc.out_scale != nullptr ? A.sc.out_scale[(size_t)t * A.nh + h] : 1.f;
    out[((size_t)t * A.nh + h) * A.hd + d] = from_f32<TA>(l > 0.f ? acc / l * os : 0.f);
}

// The keys [j0, j1) of a chunk into the value sums of a thread's dimension, in order, 16 values requested at a time.  CHECK: a row
// leaves out the keys whose p is below zero.
template <int R, bool CHECK, typename TC>
__device__ __forceinline__ void add_values(int j0, int j1, const TC* __restrict__ values, const long long* row_s, const float (*p_s)[R], float (&vs)[R])
{
    constexpr int AHEAD = 16;
    for (; j0 < j1; j0 += AHEAD) {
        float v[AHEAD];
#pragma unroll
        for (int e = 0; e < AHEAD; ++e) {
            const long long at = j0 + e < j1 ? row_s[j0 + e] : -1;
            v[e] = at >= 0 ? to_f32(values[at]) : 0.f;
        }
#pragma unroll
        for (int e = 0; e < AHEAD; ++e) {
            if (j0 + e >= j1) break;
            float p[R];
#pragma unroll
            for (int r = 0; r < R; r += 4) *reinterpret_cast<float4*>(p + r) = *reinterpret_cast<const float4*>(&p_s[j0 + e][r]);
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (!CHECK || !(p[r] < 0.f)) vs[r] = fmaf(p[r], v[e], vs[r]);
        }
    }
}

template <typename TA, typename TC, int R, bool SPLIT>
__global__ void __launch_bounds__(CHUNK, 4)
attention_rows_kernel(const TA* __restrict__ q, TA* __restrict__ out, const TC* __restrict__ pages, AttnArgs A)
{
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float p_s[CHUNK][R];
    __shared__ long long row_s[CHUNK];
    __shared__ float red[2][4][R];
    __shared__ int pos_s[R], lo_s[R], kept_s[R];
    pdl_enter();
    const int hd = A.hd, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* q_s = sm;                    // [R][hd]
    float* k_s = sm + R * hd;           // [CHUNK][KLD]
    const int kvh = blockIdx.y / A.head_groups, G = A.nh / A.nkv;
    const int h0 = kvh * G + (blockIdx.y % A.head_groups) * A.heads, nheads = min(A.heads, (kvh + 1) * G - h0);
    const int t_end = min(A.tokens, (int)(blockIdx.x + 1) * A.per_tile);
    const long long v_offset = A.planes == 2 ? (long long)A.nkv * A.page_size * hd : 0;

    for (int t0 = blockIdx.x * A.per_tile, t1; t0 < t_end; t0 = t1) {            // runs of tokens of one sequence
        const int seq = A.seq_of_token[t0];
        t1 = t0 + 1;
        while (t1 < t_end && A.seq_of_token[t1] == seq) ++t1;
        const int rows = (t1 - t0) * nheads;
        const int* bt = A.block_table + (size_t)seq * A.table_width;
        __syncthreads();                                                         // the run before is done with the shared arrays
        if (tid < R) {
            const int pos = tid < rows ? A.positions[t0 + tid / nheads] : -1, lo = tid < rows ? spy_first_key(pos, A.window) : 0;
            pos_s[tid] = pos;
            lo_s[tid] = lo;
            kept_s[tid] = min(A.keep_first, lo);
        }
        for (int i = tid; i < R * hd; i += CHUNK) {
            const int r = i / hd;
            q_s[i] = r < rows ? to_f32(q[(size_t)(t0 + r / nheads) * A.q_row_stride + (size_t)(h0 + r % nheads) * hd + (i - r * hd)]) : 0.f;
        }
        __syncthreads();
        int pos_max = -1, pos_min = 0x7fffffff, lo_min = 0x7fffffff, lo_max = 0, kept_max = 0;
        for (int r = 0; r < rows; r += nheads) {
            pos_max = max(pos_max, pos_s[r]);
            pos_min = min(pos_min, pos_s[r]);
            lo_min = min(lo_min, lo_s[r]);
            lo_max = max(lo_max, lo_s[r]);
            kept_max = max(kept_max, kept_s[r]);
        }
        const int kept_chunks = (kept_max + CHUNK - 1) / CHUNK;
        // A position beyond the table sees keys that have no page: the first such token is reported and its keys are left out, and no
        // chunk beyond the table's is walked (there is no scratch for one).
        if (pos_max / CHUNK >= A.max_chunks && tid == 0 && (!SPLIT || blockIdx.z == 0))
            for (int r = 0; r < rows; r += nheads)
                if (pos_s[r] / CHUNK >= A.max_chunks) report_status(A.status, SPY_STATUS_BAD_PAGE, t0 + r / nheads);
        const int last_chunk = pos_max < 0 ? -1 : min(pos_max / CHUNK, A.max_chunks - 1);
        float m[R], l[R], acc[R];                                                // of the row, acc of this thread's dimension
#pragma unroll
        for (int r = 0; r < R; ++r) {
            m[r] = -INFINITY;
            l[r] = acc[r] = 0.f;
        }
        for (int c = SPLIT ? blockIdx.z : 0; c <= last_chunk; c += SPLIT ? gridDim.z : 1) {
            if (c >= kept_chunks && c < lo_min / CHUNK) continue;                // nothing to see between the kept keys and the windows
            const int j = c * CHUNK + tid;
            bool any = false;
            int first_seer = 0;                                                  // the first row whose token sees the key
            for (int r = rows - nheads; r >= 0; r -= nheads)
                if ((j >= lo_s[r] || j < kept_s[r]) && j <= pos_s[r]) {
                    any = true;
                    first_seer = r;
                }
            long long row = -1;
            if (any) {
                const int lp = j / A.page_size;
                const int page = lp < A.table_width ? bt[lp] : -1;
                if (page < 0 || page >= A.num_pages) report_status(A.status, SPY_STATUS_BAD_PAGE, t0 + first_seer / nheads);
                else row = ((((long long)page * A.planes) * A.nkv + kvh) * A.page_size + j % A.page_size) * hd;
            }
            row_s[tid] = row;
            const bool bad = __syncthreads_or(any && row < 0) != 0;              // a page that is none: its key is left out by every row
            float s[R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = 0.f;
            for (int d0 = 0; d0 < hd; d0 += KD) {
                const int dims = min(KD, hd - d0), quads = dims >> 2;
                __syncthreads();                                                 // row_s is there; the half before has been read
                const int qd = tid % (KD / 4);                                   // half a warp a key, eight keys requested at a time
                for (int k0 = tid / (KD / 4); k0 < CHUNK; k0 += 8 * (CHUNK / (KD / 4))) {
                    float kv[8][4];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const long long at = row_s[k0 + e * (CHUNK / (KD / 4))];
                        if (at >= 0 && qd < quads) Vec4<TC>::load(pages + at + d0 + 4 * qd, kv[e]);
                        else kv[e][0] = kv[e][1] = kv[e][2] = kv[e][3] = 0.f;
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        *reinterpret_cast<float4*>(k_s + (k0 + e * (CHUNK / (KD / 4))) * KLD + 4 * qd) = make_float4(kv[e][0], kv[e][1], kv[e][2], kv[e][3]);
                }
                __syncthreads();
#pragma unroll 2
                for (int d = 0; d < dims; d += 4) {
                    const float4 kv = *reinterpret_cast<const float4*>(k_s + tid * KLD + d);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 qv = *reinterpret_cast<const float4*>(q_s + r * hd + d0 + d);
                        s[r] = fmaf(qv.x, kv.x, s[r]);
                        s[r] = fmaf(qv.y, kv.y, s[r]);
                        s[r] = fmaf(qv.z, kv.z, s[r]);
                        s[r] = fmaf(qv.w, kv.w, s[r]);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const bool sees = row >= 0 && r < rows && (j >= lo_s[r] || j < kept_s[r]) && j <= pos_s[r];
                float v = s[r] * A.scale;
                if (A.sc.softcap > 0.f) v = A.sc.softcap * tanhf(v / A.sc.softcap);
                if (A.sc.slopes != nullptr && r < rows) v -= A.sc.slopes[h0 + r % nheads] * (float)(pos_s[r] - j);
                s[r] = sees ? v : -INFINITY;
                const float top = warp_max(s[r]);
                if (lane == 0) red[0][warp][r] = top;
            }
            __syncthreads();
            float mc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                mc[r] = fmaxf(fmaxf(red[0][0][r], red[0][1][r]), fmaxf(red[0][2][r], red[0][3][r]));
                const bool sees = row >= 0 && r < rows && (j >= lo_s[r] || j < kept_s[r]) && j <= pos_s[r];
                const float p = !sees ? 0.f : mc[r] != -INFINITY ? expf(s[r] - mc[r]) : isnan(s[r]) ? s[r] : 0.f;
                p_s[tid][r] = sees || r >= rows ? p * (1.f / CHUNK) : -1.f;
                const float sum = warp_sum(p);
                if (lane == 0) red[1][warp][r] = sum;
            }
            __syncthreads();
            const int first = c < kept_chunks ? 0 : max(lo_min - c * CHUNK, 0), last = min(pos_max - c * CHUNK, CHUNK - 1);
            float vs[R];
#pragma unroll
            for (int r = 0; r < R; ++r) vs[r] = 0.f;
            if (tid < hd) {
                // [fa, fb): keys that every row of the block sees
                const int fa = min(max(first, lo_max - c * CHUNK), last + 1), fb = bad ? fa : max(fa, min(last, pos_min - c * CHUNK) + 1);
                add_values<R, true>(first, fa, pages + v_offset + tid, row_s, p_s, vs);
                add_values<R, false>(fa, fb, pages + v_offset + tid, row_s, p_s, vs);
                add_values<R, true>(fb, last + 1, pages + v_offset + tid, row_s, p_s, vs);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float lc = ((red[1][0][r] + red[1][1][r]) + red[1][2][r]) + red[1][3][r];
                if (SPLIT) {
                    if (r < rows) {
                        float* part = A.partial + (((size_t)(t0 + r / nheads) * A.nh + h0 + r % nheads) * A.max_chunks + c) * (hd + 2);
                        if (tid < hd) part[tid] = vs[r];
                        if (tid == 0) {
                            part[hd] = mc[r];
                            part[hd + 1] = lc;
                        }
                    }
                } else {
                    float alpha, beta;
                    if (take_chunk(m[r], l[r], mc[r], lc, alpha, beta)) acc[r] = fmaf(acc[r], alpha, vs[r] * (CHUNK * beta));
                }
            }
            __syncthreads();                                                     // the shared arrays are rewritten by the next chunk
        }
        if (!SPLIT && tid < hd) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r < rows) store_row(A, out, t0 + r / nheads, h0 + r % nheads, tid, acc[r], m[r], l[r]);
        }
    }
}

template <typename TA>
__global__ void __launch_bounds__(CHUNK) attention_merge_kernel(TA* __restrict__ out, AttnArgs A)
{
    pdl_enter();
    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, hd = A.hd;
    const int pos = A.positions[t], lo = spy_first_key(pos, A.window), kept_chunks = (min(A.keep_first, lo) + CHUNK - 1) / CHUNK;
    const float* part = A.partial + ((size_t)t * A.nh + h) * A.max_chunks * (hd + 2);
    const int last_chunk = pos < 0 ? -1 : min(pos / CHUNK, A.max_chunks - 1);    // the chunks that attention_rows_kernel walks
    float m = -INFINITY, l = 0.f, acc = 0.f;
#pragma unroll 4
    for (int c = 0; c <= last_chunk; ++c) {
        if (c >= kept_chunks && c < lo / CHUNK) continue;
        const float* p = part + (size_t)c * (hd + 2);
        const float mc = p[hd], lc = p[hd + 1], v = tid < hd ? p[tid] : 0.f;
        float alpha, beta;
        if (take_chunk(m, l, mc, lc, alpha, beta)) acc = fmaf(acc, alpha, v * (CHUNK * beta));
    }
    if (tid < hd) store_row(A, out, t, h, tid, acc, m, l);
}

template <typename TA, typename TC, int R>
static int launch_rows(const void* q, void* out, const void* pages, const AttnArgs& A, dim3 grid, bool split, cudaStream_t stream)
{
    const size_t smem = (size_t)(R * A.hd + CHUNK * KLD) * sizeof(float);
    SPY_ONCE_PER_DEVICE
    {
        const int most = (int)((R * CHUNK + CHUNK * KLD) * sizeof(float));       // with the static arrays more than the 48 KB that need no attribute
        SPY_CUDA(cudaFuncSetAttribute(attention_rows_kernel<TA, TC, R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        SPY_CUDA(cudaFuncSetAttribute(attention_rows_kernel<TA, TC, R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    }
    if (split) {
        spy_launch(attention_rows_kernel<TA, TC, R, true>, grid, dim3(CHUNK), smem, stream, (const TA*)q, (TA*)out, (const TC*)pages, A);
        spy_launch(attention_merge_kernel<TA>, dim3(A.tokens, A.nh), dim3(CHUNK), 0, stream, (TA*)out, A);
    } else {
        spy_launch(attention_rows_kernel<TA, TC, R, false>, grid, dim3(CHUNK), smem, stream, (const TA*)q, (TA*)out, (const TC*)pages, A);
    }
    return 0;
}

// Tokens of a block: several where they outnumber the sequences by far (prompts), one where most tokens are their sequence's only one.
static int tokens_of_block(int heads, int tokens, int num_seqs) { return tokens > 2 * num_seqs ? (16 / heads > 0 ? 16 / heads : 1) : 1; }
static int heads_of_block(int group) { return group < 16 ? group : 16; }

// Floats of scratch with which the chunks of a row may go to blocks of their own (0: one block walks them all).  Worth it while
// the device holds the blocks about twice at most (300 tokens: 145 us where each row group has one block, the last tokens' with three chunks) and
// a row may have more than two chunks (a launch more costs what a second chunk does); the results are the same to the last bit.
extern "C" long long spy_attention_generic_scratch(int tokens, int num_seqs, int nh, int nkv, int hd, int table_width, int page_size)
{
    if (tokens <= 0 || nh <= 0 || nkv <= 0 || nh % nkv != 0 || hd <= 0 || hd > CHUNK || hd % 4 != 0) return 0;
    const int heads = heads_of_block(nh / nkv), per_tile = tokens_of_block(heads, tokens, num_seqs);
    const long long blocks = (long long)((tokens + per_tile - 1) / per_tile) * nkv * ((nh / nkv + heads - 1) / heads);
    const long long chunks = ((long long)table_width * page_size + CHUNK - 1) / CHUNK;
    const long long floats = (long long)tokens * nh * chunks * (hd + 2);
    return blocks < 8 * spy_sm_count() && chunks > 2 && floats <= (16LL << 20) ? floats : 0;
}

// q: [T, ...] rows of q_row_stride elements whose first nh*hd elements are the query heads;
// out: [T, nh*hd]; pages: one cache [num_pages][planes][nkv][page_size][hd] of cache_dtype.
extern "C" int spy_attention_generic(const void* q, long long q_row_stride, void* out, int act_dtype, const void* pages, int cache_dtype,
                                     const int* block_table, int table_width, int page_size, int num_pages, int nh, int nkv, int hd,
                                     const int* positions, const int* seq_of_token, int tokens, int window, float scale, int* status,
                                     cudaStream_t stream, int planes, int keep_first, int sink, float softcap, const float* slopes, const float* sinks,
                                     const float* out_scale, int num_seqs, float* scratch, long long scratch_floats)
{
    if (softcap < 0.f) SPY_FAIL("attention: a cap of %g on the scores", softcap);
    const SpyScores scores = {softcap, slopes, sinks, out_scale};
    if (keep_first < 0 || (keep_first > 0 && window <= 0)) SPY_FAIL("attention: kept first keys (%d) go with a window", keep_first);
    if (tokens <= 0) return 0;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0) SPY_FAIL("attention: %d query heads do not group over %d key/value heads", nh, nkv);
    if (hd <= 0 || hd > ACC * CHUNK) SPY_FAIL("attention: head_dim %d must be positive and at most %d", hd, ACC * CHUNK);
    if (planes != 1 && planes != 2) SPY_FAIL("attention: a cache of %d planes (1: keys that are the values too, 2: keys and values)", planes);
    if (page_size <= 0 || num_pages <= 0 || table_width <= 0) SPY_FAIL("attention: page_size, num_pages and table_width must be positive");
    if (nh > 65535) SPY_FAIL("attention: %d heads exceed the grid limit", nh);
    if (hd <= CHUNK && hd % 4 == 0) {
        AttnArgs A = {q_row_stride, block_table, table_width, page_size, num_pages, nh, nkv, hd, positions, seq_of_token, tokens, window, scale, status,
                      planes, keep_first, sink, scores, 0, 0, 0, scratch, 0};
        const int group = nh / nkv;
        A.heads = heads_of_block(group);
        A.per_tile = tokens_of_block(A.heads, tokens, num_seqs);
        A.head_groups = (group + A.heads - 1) / A.heads;
        A.max_chunks = (int)(((long long)table_width * page_size + CHUNK - 1) / CHUNK);
        const long long need = spy_attention_generic_scratch(tokens, num_seqs, nh, nkv, hd, table_width, page_size);
        const bool split = need > 0 && scratch != nullptr && scratch_floats >= need;
        if ((long long)nkv * A.head_groups > 65535) SPY_FAIL("attention: %d heads exceed the grid limit", nh);
        const dim3 grid((tokens + A.per_tile - 1) / A.per_tile, nkv * A.head_groups, split ? (A.max_chunks < 64 ? A.max_chunks : 64) : 1);
        const int rows = A.heads * A.per_tile;
        SPY_DISPATCH_DTYPE(act_dtype, TA, {
            SPY_DISPATCH_DTYPE(cache_dtype, TC, {
                const int rc = rows <= 4 ? launch_rows<TA, TC, 4>(q, out, pages, A, grid, split, stream)
                               : rows <= 8 ? launch_rows<TA, TC, 8>(q, out, pages, A, grid, split, stream)
                                           : launch_rows<TA, TC, 16>(q, out, pages, A, grid, split, stream);
                if (rc) return rc;
            })
        })
        SPY_CHECK_LAUNCH("attention_rows");
        return 0;
    }
    const size_t smem = (size_t)(hd + (hd & 1) + CHUNK + 33) * sizeof(float) + (size_t)CHUNK * sizeof(long long);
    dim3 grid(tokens, nh);
    SPY_DISPATCH_DTYPE(act_dtype, TA, {
        SPY_DISPATCH_DTYPE(cache_dtype, TC, {
            spy_launch(attention_generic_kernel<TA, TC>, grid, dim3(CHUNK), smem, stream,
                (const TA*)q, q_row_stride, (TA*)out, (const TC*)pages, block_table, table_width, page_size, num_pages, nh, nkv, hd,
                positions, seq_of_token, window, scale, status, planes, keep_first, sink, scores);
        })
    })
    SPY_CHECK_LAUNCH("attention_generic");
    return 0;
}
