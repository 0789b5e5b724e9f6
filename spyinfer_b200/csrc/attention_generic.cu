// Attention over the paged cache for any mix of queries, every head size, every page size, 32-bit
// or bfloat16 storage, everything computed in 32-bit with expf.  Three kernels: head sizes up to 128 in
// quads take one of two for several query rows a block (attention_rows_kernel; attention_wide_kernel for prompts), the others one block per
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
// The kernel above reads every key and value once a (token, head) and waits for each.  Here a block takes up to R query rows (the heads
// of a kv head, times several tokens of one sequence where tokens outnumber the sequences), so a key row serves all of them: keys and values are copied
// to shared memory behind the block's back (cp.async), one key a thread for the scores (its row read in quads, the queries broadcast), one
// dimension a thread for the values.  Head sizes up to 64 and 32 leave threads over for those: the rows are then shared out over two and four
// groups of threads.  With few rows (decoding) the chunks of a row go to blocks of their own and attention_merge_kernel adds them.
//
// Bounds: with few keys the way through a block, whose steps wait for one another and whose instructions come cold (loads
// unrolled into registers, three times the code, took 16 us where this takes 11); with many rows shared-memory reads and multiply-adds in about equal parts.
// Measured with the merge, 32 heads over 8 of 128, 32-bit, kernel above / rows read through registers one batch at a time / this one (us): decoding
// 4 requests of 100 keys 13.6 / 16.8 / 11, of 640 71 / 25 / 17, of 8,192 1,835 / 121 / 101; prompts of 7 tokens 5.9 / 24 / 6.8, of 37 12.7 / 28 / 9, of 300
// 287 / 105 / 91.
//
// A chunk's maximum, sum and value sum are formed for themselves and added to the row's in the order of the chunks, whether one
// block walks them or many, and a row's numbers do not depend on the rows beside it: results do not depend on the cut.
// A key that a row does not see is left out (p_s = -1), not multiplied by zero: what lies there may not be a finite number.
// Value sums are formed with probabilities divided by CHUNK (a power of two: the same bits), so that a chunk's never exceed its largest value: relative to
// the chunk's own maximum they could overflow where the chunk weighs next to nothing in its row.
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
    int heads, per_tile, head_groups;   // heads and tokens of a block (at most 32 tokens), blocks a kv head
    int max_chunks;                     // of the block table
    int page_shift;                     // log2 of the page size, -1 where that is no power of two
    int kld, area;                      // numbers between the keys in shared memory, from one area to the other
    float* partial;                     // [tokens][nh][slots][hd + 2]: value sums, then the maximum and the sum
    int slots;                          // rows of 2 to `slots` chunks have their chunks on blocks of their own (0: none)
};

constexpr int KD = 64;                  // dimensions of the keys staged at a time

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

// What a row's sum becomes with the sinks.
__device__ __forceinline__ float with_sinks(const AttnArgs& A, int h, float m, float l)
{
    if (A.sink) l += m == -INFINITY ? 1.f : expf(-m);
    if (A.sc.sinks != nullptr) l += m == -INFINITY ? 1.f : expf(A.sc.sinks[h] - m);
    return l;
}

// A tile's tokens, one a lane of every warp, and a run of them that belong to one sequence.
struct TileTokens {
    int n, seq, pos, lo, kept;          // tokens of the tile; of this lane's token: sequence, position, first key, keys kept before it
};
struct Run {
    int first, len, seq;                // tokens of the tile
    int pos_max, pos_min, lo_min, lo_max, kept_max;
    int last_chunk;                     // that any of them sees and the table holds; -1: none
};

__device__ __forceinline__ TileTokens load_tile(const AttnArgs& A, int t_first)
{
    TileTokens T;
    const int lane = threadIdx.x & 31;
    T.n = min(A.per_tile, A.tokens - t_first);
    T.seq = lane < T.n ? A.seq_of_token[t_first + lane] : 0;
    T.pos = lane < T.n ? A.positions[t_first + lane] : -1;
    T.lo = spy_first_key(T.pos, A.window);
    T.kept = min(A.keep_first, T.lo);
    return T;
}

// The run that begins at token `first` of the tile.
__device__ __forceinline__ Run run_from(const AttnArgs& A, const TileTokens& T, int first)
{
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    Run R;
    R.first = first;
    R.seq = __shfl_sync(all, T.seq, first);
    const unsigned others = __ballot_sync(all, lane >= first && (lane >= T.n || T.seq != R.seq));
    R.len = (others != 0 ? __ffs(others) - 1 : 32) - first;
    const bool mine = lane >= first && lane < first + R.len;
    R.pos_max = __reduce_max_sync(all, mine ? T.pos : -1);
    R.pos_min = __reduce_min_sync(all, mine ? T.pos : 0x7fffffff);
    R.lo_min = __reduce_min_sync(all, mine ? T.lo : 0x7fffffff);
    R.lo_max = __reduce_max_sync(all, mine ? T.lo : 0);
    R.kept_max = __reduce_max_sync(all, mine ? T.kept : 0);
    R.last_chunk = R.pos_max < 0 ? -1 : min(R.pos_max / CHUNK, A.max_chunks - 1);
    return R;
}

// Whether a run's chunks go to blocks of their own (one chunk is stored as it is, more than there is room for are walked by one block).
__device__ __forceinline__ bool in_parts(const AttnArgs& A, const Run& R) { return R.last_chunk >= 1 && R.last_chunk < A.slots; }

struct TakeMax { static __device__ __forceinline__ float of(float a, float b) { return fmaxf(a, b); } };
struct TakeSum { static __device__ __forceinline__ float of(float a, float b) { return a + b; } };

// v[0..R) of every lane over the warp, each row in the order of warp_sum (lanes 16 apart, then 8, 4, 2, 1), in R + 3 or fewer shuffles
// instead of 5 R: with every step a lane keeps half of its rows.  The result is row `*row`'s in lanes whose `*row` is not negative.
template <int R, typename OP>
__device__ __forceinline__ float reduce_rows(float (&v)[R], int* row)
{
    const int lane = threadIdx.x & 31;
    int at = 0;
#pragma unroll
    for (int o = 16, n = R; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int r = 0; r < n; ++r) {
                const float keep = upper ? v[r + n] : v[r], give = upper ? v[r] : v[r + n];
                v[r] = OP::of(keep, __shfl_xor_sync(0xffffffffu, give, o));
            }
            at += upper ? n : 0;
        } else {
            v[0] = OP::of(v[0], __shfl_xor_sync(0xffffffffu, v[0], o));
        }
    }
    constexpr int SPARE = 32 / R - 1;                      // the lowest bits tell no rows apart
    *row = (lane & SPARE) == 0 ? at : -1;
    return v[0];
}

template <int RG>
__device__ __forceinline__ void load_probabilities(const float* src, float (&p)[RG])
{
    if constexpr (RG >= 4) {
#pragma unroll
        for (int r = 0; r < RG; r += 4) *reinterpret_cast<float4*>(p + r) = *reinterpret_cast<const float4*>(src + r);
    } else if constexpr (RG == 2) {
        *reinterpret_cast<float2*>(p) = *reinterpret_cast<const float2*>(src);
    } else {
        p[0] = src[0];
    }
}

// Four elements on their way from global to shared memory.
template <typename TC>
__device__ __forceinline__ void copy_quad(uint32_t dst, const TC* src)
{
    if constexpr (sizeof(TC) == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

template <typename TA, typename TC, int R, int GROUPS>
__global__ void __launch_bounds__(CHUNK, 4)
attention_rows_kernel(const TA* __restrict__ q, TA* __restrict__ out, const TC* __restrict__ pages, AttnArgs A)
{
    constexpr int RG = R / GROUPS, DG = CHUNK / GROUPS;     // rows of a group of threads, dimensions it takes
    constexpr int PLD = R == 4 ? 4 : R + 4;                // four lanes' quads of probabilities meet no bank twice
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float p_s[CHUNK][PLD];
    __shared__ __align__(16) float red[2][R][4];           // by row and warp: maxima, sums
    __shared__ long long row_s[CHUNK];
    __shared__ int pos_s[R], lo_s[R], kept_s[R];
    __shared__ float slope_s[R];
    __shared__ long long at_s[R];                          // token * nh + head
    __shared__ float2 take_s[R], end_s[R];                 // how the row takes a chunk: factors of what was there and what comes; its sum and scale in the end
    pdl_wait();
    pdl_launch_dependents();                               // behind the wait: a kernel launched early may read this one's inputs (attention_merge_kernel does)
    const int hd = A.hd, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kld = A.kld;
    const int group = tid / DG, dim = tid - group * DG;    // of the value sums
    float* q_s = sm;                    // [R][hd]
    // Two areas.  Head sizes up to 64: a chunk's keys [CHUNK][kld] and its values [CHUNK][hd].  Above: the keys' halves [CHUNK][kld], and when those have
    // been read the values of the chunk's halves [CHUNK / 2][hd] in their place.
    TC* const area0 = reinterpret_cast<TC*>(sm + R * hd);
    TC* const area1 = area0 + A.area;
    const bool halves = hd > KD;
    const int kvh = blockIdx.y / A.head_groups, G = A.nh / A.nkv;
    const int h0 = kvh * G + (blockIdx.y % A.head_groups) * A.heads, nheads = min(A.heads, (kvh + 1) * G - h0);
    const int t_first = blockIdx.x * A.per_tile;
    const long long v_offset = A.planes == 2 ? (long long)A.nkv * A.page_size * hd : 0;
    // keys or values [j0, j1) of the chunk, `dims` numbers from d0 on, to rows of ld: half a warp a row, a whole one for wide ones
    const auto copy_rows = [&](TC* dst, int ld, int j0, int j1, long long offset, int d0, int dims) {
        const int lanes = dims > KD ? 32 : 16, quad = 4 * (tid & (lanes - 1));
        if (quad < dims) {
#pragma unroll 4
            for (int j = j0 + tid / lanes; j < j1; j += CHUNK / lanes) {
                const long long at = row_s[j];
                if (at >= 0) copy_quad((uint32_t)__cvta_generic_to_shared(dst + (j - j0) * ld + quad), pages + at + offset + d0 + quad);
            }
        }
        copy_commit();
    };
    const TileTokens T = load_tile(A, t_first);

    for (int i = 0; i < T.n;) {                                                  // runs of tokens of one sequence
        const Run run = run_from(A, T, i);
        i += run.len;
        // A position beyond the table sees keys that have no page: such a token is reported and its keys are left out, and no
        // chunk beyond the table's is walked (there is no scratch for one).
        if (warp == 0 && blockIdx.z == 0 && lane >= run.first && lane < i && T.pos / CHUNK >= A.max_chunks)
            report_status(A.status, SPY_STATUS_BAD_PAGE, t_first + lane);
        const bool parts = in_parts(A, run);
        if (blockIdx.z > 0 && (!parts || (int)blockIdx.z > run.last_chunk)) continue;
        const int kept_chunks = (run.kept_max + CHUNK - 1) / CHUNK, lo_chunk = run.lo_min / CHUNK, step = parts ? gridDim.z : 1;
        const auto seen_from = [&](int c) {                                      // nothing to see between the kept keys and the windows
            return c >= kept_chunks && c < lo_chunk ? c + (lo_chunk - c + step - 1) / step * step : c;
        };
        const int* bt = A.block_table + (size_t)run.seq * A.table_width;
        const auto page_index = [&](int key) { return A.page_shift >= 0 ? key >> A.page_shift : key / A.page_size; };
        const auto page_of = [&](int c) {
            const int lp = c <= run.last_chunk ? page_index(c * CHUNK + tid) : A.table_width;
            return lp < A.table_width ? bt[lp] : -1;
        };
        int c = seen_from(parts ? blockIdx.z : 0);
        if (parts && c > run.last_chunk) continue;

        const int rows = run.len * nheads;
        int page = page_of(c);
        {
            float x[R / 4][4];                                                   // a warp a row, everything requested at once
#pragma unroll
            for (int k = 0; k < R / 4; ++k) {
                const int r = warp + 4 * k, t = r / nheads;
                const TA* src = q + (size_t)(t_first + run.first + t) * A.q_row_stride + (size_t)(h0 + r - t * nheads) * hd;
#pragma unroll
                for (int e = 0; e < 4; ++e) x[k][e] = r < rows && lane + 32 * e < hd ? to_f32(src[lane + 32 * e]) : 0.f;
            }
            __syncthreads();                                                     // the run before is done with the shared arrays
#pragma unroll
            for (int k = 0; k < R / 4; ++k)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (lane + 32 * e < hd) q_s[(warp + 4 * k) * hd + lane + 32 * e] = x[k][e];
        }
        int my_head = 0;                                                         // of warp 0's lanes, a row each
        float m = -INFINITY, l = 0.f;                                            // the row's maximum and sum
        if (warp == 0) {
            const int t = run.first + lane / nheads;
            my_head = h0 + lane % nheads;
            const int pos = __shfl_sync(0xffffffffu, T.pos, t & 31), lo = __shfl_sync(0xffffffffu, T.lo, t & 31), kept = __shfl_sync(0xffffffffu, T.kept, t & 31);
            if (lane < R) {
                pos_s[lane] = lane < rows ? pos : -1;
                lo_s[lane] = lane < rows ? lo : 0;
                kept_s[lane] = lane < rows ? kept : 0;
                slope_s[lane] = A.sc.slopes != nullptr && lane < rows ? A.sc.slopes[my_head] : 0.f;
                at_s[lane] = (long long)(t_first + t) * A.nh + my_head;
            }
        }
        __syncthreads();
        float acc[RG];                                                           // of the group's rows, this thread's dimension
#pragma unroll
        for (int r = 0; r < RG; ++r) acc[r] = 0.f;
        while (c <= run.last_chunk) {
            const int c0 = c * CHUNK, j = c0 + tid, c_next = seen_from(c + step);
            const int first = c < kept_chunks ? 0 : max(run.lo_min - c0, 0), last = min(run.pos_max - c0, CHUNK - 1);   // of the keys that any row sees
            bool any = j >= run.lo_max && j <= run.pos_min;                      // every row sees it
            int first_seer = 0;                                                  // the first row whose token sees the key
            if (!any)
                for (int r = rows - nheads; r >= 0; r -= nheads)
                    if ((j >= lo_s[r] || j < kept_s[r]) && j <= pos_s[r]) {
                        any = true;
                        first_seer = r;
                    }
            long long row = -1;
            if (any) {
                if (page < 0 || page >= A.num_pages) report_status(A.status, SPY_STATUS_BAD_PAGE, t_first + run.first + first_seer / nheads);
                else row = ((((long long)page * A.planes) * A.nkv + kvh) * A.page_size + (j - page_index(j) * A.page_size)) * hd;
            }
            row_s[tid] = row;
            page = page_of(c_next);
            const bool bad = __syncthreads_or(any && row < 0) != 0;              // a page that is none: its key is left out by every row
            const bool all_see = !bad && c0 >= run.lo_max && c0 + CHUNK - 1 <= run.pos_min;
            const bool warp_sees = warp * 32 <= last && warp * 32 + 31 >= first;
            float s[R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = 0.f;
            copy_rows(area0, kld, 0, last + 1, 0, 0, min(KD, hd));
            if (halves) copy_rows(area1, kld, 0, last + 1, 0, KD, hd - KD);
            else copy_rows(area1, hd, 0, last + 1, v_offset, 0, hd);
#pragma unroll 1
            for (int d0 = 0; d0 < hd; d0 += KD) {
                copy_wait<1>();
                __syncthreads();
                if (warp_sees) {
                    const TC* key = (d0 == 0 ? area0 : area1) + tid * kld;
                    const float* query = q_s + d0;
                    const int dims = min(KD, hd - d0);
#pragma unroll(R == 4 ? 4 : 2)
                    for (int d = 0; d < dims; d += 4) {
                        float kq[4];
                        Vec4<TC>::load(key + d, kq);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const float4 qv = *reinterpret_cast<const float4*>(query + r * hd + d);
                            s[r] = fmaf(qv.x, kq[0], s[r]);
                            s[r] = fmaf(qv.y, kq[1], s[r]);
                            s[r] = fmaf(qv.z, kq[2], s[r]);
                            s[r] = fmaf(qv.w, kq[3], s[r]);
                        }
                    }
                }
                if (halves) {
                    __syncthreads();                                             // this half of the keys has been read
                    if (d0 == 0) copy_rows(area0, hd, 0, min(last + 1, CHUNK / 2), v_offset, 0, hd);
                    else copy_rows(area1, hd, CHUNK / 2, last + 1, v_offset, 0, hd);
                }
            }
            unsigned seen = (1u << rows) - 1;                                    // of this thread's key, a bit a row
            if (!all_see) {
                seen = 0;
#pragma unroll
                for (int r = 0; r < R; ++r) seen |= (row >= 0 && (j >= lo_s[r] || j < kept_s[r]) && j <= pos_s[r] ? 1u : 0u) << r;   // rows beyond the run's: pos_s = -1
            }
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] *= A.scale;
            if (A.sc.softcap > 0.f) {
#pragma unroll
                for (int r = 0; r < R; ++r) s[r] = A.sc.softcap * tanhf(s[r] / A.sc.softcap);
            }
            if (A.sc.slopes != nullptr) {
#pragma unroll
                for (int r = 0; r < R; ++r) s[r] -= slope_s[r] * (float)(pos_s[r] - j);
            }
            float w[R];
#pragma unroll
            for (int r = 0; r < R; ++r) w[r] = s[r] = (seen >> r & 1) != 0 ? s[r] : -INFINITY;
            int mine;
            const float top = reduce_rows<R, TakeMax>(w, &mine);
            if (mine >= 0) red[0][mine][warp] = top;
            __syncthreads();
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float4 x = *reinterpret_cast<const float4*>(red[0][r]);
                const float mc = fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w));
                const float p = mc != -INFINITY ? expf(s[r] - mc) : isnan(s[r]) ? s[r] : 0.f;
                w[r] = (seen >> r & 1) != 0 ? p : 0.f;
                s[r] = (seen >> r & 1) != 0 || r >= rows ? w[r] * (1.f / CHUNK) : -1.f;
            }
#pragma unroll
            for (int r = 0; r < R; r += 4) *reinterpret_cast<float4*>(&p_s[tid][r]) = make_float4(s[r], s[r + 1], s[r + 2], s[r + 3]);
            const float sum = reduce_rows<R, TakeSum>(w, &mine);
            if (mine >= 0) red[1][mine][warp] = sum;
            if (halves) copy_wait<1>();
            else copy_wait<0>();
            __syncthreads();
            if (warp == 0 && lane < R) {
                const float4 x = *reinterpret_cast<const float4*>(red[0][lane]), y = *reinterpret_cast<const float4*>(red[1][lane]);
                const float mc = fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)), lc = ((y.x + y.y) + y.z) + y.w;
                if (parts) {
                    if (lane < rows) {
                        float* part = A.partial + ((size_t)at_s[lane] * A.slots + c) * (hd + 2) + hd;
                        part[0] = mc;
                        part[1] = lc;
                    }
                } else {
                    float alpha = -1.f, beta = 0.f;                              // alpha below zero: there is nothing to take
                    if (!take_chunk(m, l, mc, lc, alpha, beta)) alpha = -1.f;
                    take_s[lane] = make_float2(alpha, CHUNK * beta);
                }
            }
            float vs[RG];
#pragma unroll
            for (int r = 0; r < RG; ++r) vs[r] = 0.f;
            {
                // [fa, fb): keys that every row of the block sees; elsewhere a row leaves out the keys whose p is below zero
                const int fa = max(first, run.lo_max - c0), fb = bad ? 0 : min(run.pos_min - c0, last) + 1;
                const float* p_g = &p_s[0][group * RG];
                const TC* v_s = (halves ? area0 : area1) + (dim < hd ? dim : 0);
                int j = first, end = halves ? min(CHUNK / 2, last + 1) : last + 1;
#pragma unroll 1
                while (true) {
#pragma unroll 1
                    while (j < end) {
                        if (j >= fa && j < fb) {
                            const int whole = min(fb, end);
#pragma unroll 8
                            for (; j < whole; ++j) {
                                const float v = to_f32(v_s[j * hd]);
                                float p[RG];
                                load_probabilities<RG>(p_g + j * PLD, p);
#pragma unroll
                                for (int r = 0; r < RG; ++r) vs[r] = fmaf(p[r], v, vs[r]);
                            }
                        } else {
                            const float v = to_f32(v_s[j * hd]);
                            float p[RG];
                            load_probabilities<RG>(p_g + j * PLD, p);
#pragma unroll
                            for (int r = 0; r < RG; ++r)
                                if (!(p[r] < 0.f)) vs[r] = fmaf(p[r], v, vs[r]);
                            ++j;
                        }
                    }
                    if (end > last) break;
                    copy_wait<0>();
                    __syncthreads();
                    v_s = area1 + (dim < hd ? dim : 0) - (CHUNK / 2) * hd;
                    end = last + 1;
                }
            }
            __syncthreads();                                                     // take_s is there; the next chunk rewrites the shared arrays
#pragma unroll
            for (int rr = 0; rr < RG; ++rr) {
                const int r = group * RG + rr;
                if (parts) {
                    if (r < rows && dim < hd) A.partial[((size_t)at_s[r] * A.slots + c) * (hd + 2) + dim] = vs[rr];
                } else {
                    const float2 f = take_s[r];
                    if (!(f.x < 0.f)) acc[rr] = fmaf(acc[rr], f.x, vs[rr] * f.y);
                }
            }
            c = c_next;
        }
        if (parts) continue;
        if (warp == 0 && lane < R)
            end_s[lane] = make_float2(with_sinks(A, my_head, m, l), A.sc.out_scale != nullptr && lane < rows ? A.sc.out_scale[at_s[lane]] : 1.f);
        __syncthreads();
        if (dim < hd) {
#pragma unroll
            for (int rr = 0; rr < RG; ++rr) {
                const int r = group * RG + rr;
                const float2 f = end_s[r];
                if (r < rows) out[at_s[r] * hd + dim] = from_f32<TA>(f.x > 0.f ? acc[rr] / f.x * f.y : 0.f);
            }
        }
    }
}

// ---- prompts with head sizes above 64: 32 rows a block, four rows by four keys (or dimensions) a thread -------------------------
// The kernel above reads shared memory more than it multiplies: a key's quad and 16 queries' for 64 multiply-adds.  Here a thread reads four
// keys' quads and four queries' for as many, and in the value sums a quad of probabilities and one of values for 16, so that the multiply-adds
// are what is left, and a block's keys and values serve twice the rows.  Every sum runs in the same order as above: the bits are the same.
// Measured with the merge, 32 heads over 8 of 128, 32-bit, kernel above with 16 rows / this one (us): prompts of 150 tokens 52 / 40, of 300 95 / 66, of 600
// 286 / 178, of 2,000 2,266 / 1,405; 64 tokens behind 2,000 183 / 113; 8 of 100 115 / 76.  What is left beside the multiply-adds (the FMA pipes are busy for 14 us
// of the 300 tokens' 66, 20 on the busiest SM): a block's copies, maxima and sums wait for one another, and two blocks an SM are what shared memory holds.
constexpr int WIDE_ROWS = 32, WIDE_THREADS = 256, WIDE_PLD = WIDE_ROWS + 4;

// v[0..4) over the eight lanes whose numbers differ in their lowest three bits; the result is row `*row`'s in lanes whose `*row` is not negative.
template <typename OP>
__device__ __forceinline__ float reduce_four(float (&v)[4], int* row)
{
    const int lane = threadIdx.x & 31;
    const bool up2 = (lane & 4) != 0, up1 = (lane & 2) != 0;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float keep = up2 ? v[r + 2] : v[r], give = up2 ? v[r] : v[r + 2];
        v[r] = OP::of(keep, __shfl_xor_sync(0xffffffffu, give, 4));
    }
    const float keep = up1 ? v[1] : v[0], give = up1 ? v[0] : v[1];
    float x = OP::of(keep, __shfl_xor_sync(0xffffffffu, give, 2));
    x = OP::of(x, __shfl_xor_sync(0xffffffffu, x, 1));
    *row = (lane & 1) == 0 ? (up2 ? 2 : 0) + (up1 ? 1 : 0) : -1;
    return x;
}

template <typename TA, typename TC>
__global__ void __launch_bounds__(WIDE_THREADS, 2)
attention_wide_kernel(const TA* __restrict__ q, TA* __restrict__ out, const TC* __restrict__ pages, AttnArgs A)
{
    constexpr int R = WIDE_ROWS, PLD = WIDE_PLD;
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float p_s[CHUNK][PLD];
    __shared__ __align__(16) float red[2][R][4];           // by row and quarter of the chunk: maxima, sums
    __shared__ long long row_s[CHUNK];
    __shared__ int pos_s[R], lo_s[R], kept_s[R];
    __shared__ float slope_s[R];
    __shared__ long long at_s[R];                          // token * nh + head
    __shared__ float2 take_s[R], end_s[R];
    pdl_wait();
    pdl_launch_dependents();                               // behind the wait, as above
    const int hd = A.hd, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kld = A.kld, qld = hd + 4;
    // Scores: a warp takes 16 rows and a quarter of the chunk; a lane's rows are four apart, its keys eight (lanes side by side then read rows of
    // shared memory that meet no bank twice).  Value sums: four rows side by side and four dimensions.
    const int half = warp >> 2, quarter = warp & 3, row_lane = lane >> 3, key_lane = lane & 7;
    const int quad = 4 * ((warp & 3) * 8 + (lane & 7)), v_row = 4 * ((warp >> 2) * 4 + (lane >> 3));
    const bool has_quad = quad < hd;
    float* q_s = sm;                    // [R][qld]
    TC* const area0 = reinterpret_cast<TC*>(sm + R * qld);          // the keys' halves, then the values of the chunk's halves in their place
    TC* const area1 = area0 + A.area;
    const int kvh = blockIdx.y / A.head_groups, G = A.nh / A.nkv;
    const int h0 = kvh * G + (blockIdx.y % A.head_groups) * A.heads, nheads = min(A.heads, (kvh + 1) * G - h0);
    const int t_first = blockIdx.x * A.per_tile;
    const long long v_offset = A.planes == 2 ? (long long)A.nkv * A.page_size * hd : 0;
    const auto copy_rows = [&](TC* dst, int ld, int j0, int j1, long long offset, int d0, int dims) {
        const int lanes = dims > KD ? 32 : 16, d = 4 * (tid & (lanes - 1));
        if (d < dims) {
#pragma unroll 4
            for (int j = j0 + tid / lanes; j < j1; j += WIDE_THREADS / lanes) {
                const long long at = row_s[j];
                if (at >= 0) copy_quad((uint32_t)__cvta_generic_to_shared(dst + (j - j0) * ld + d), pages + at + offset + d0 + d);
            }
        }
        copy_commit();
    };
    const TileTokens T = load_tile(A, t_first);

    for (int i = 0; i < T.n;) {                                                  // runs of tokens of one sequence
        const Run run = run_from(A, T, i);
        i += run.len;
        if (warp == 0 && blockIdx.z == 0 && lane >= run.first && lane < i && T.pos / CHUNK >= A.max_chunks)
            report_status(A.status, SPY_STATUS_BAD_PAGE, t_first + lane);        // as above: a position beyond the table
        const bool parts = in_parts(A, run);
        if (blockIdx.z > 0 && (!parts || (int)blockIdx.z > run.last_chunk)) continue;
        const int kept_chunks = (run.kept_max + CHUNK - 1) / CHUNK, lo_chunk = run.lo_min / CHUNK, step = parts ? gridDim.z : 1;
        const auto seen_from = [&](int c) { return c >= kept_chunks && c < lo_chunk ? c + (lo_chunk - c + step - 1) / step * step : c; };
        const int* bt = A.block_table + (size_t)run.seq * A.table_width;
        const auto page_index = [&](int key) { return A.page_shift >= 0 ? key >> A.page_shift : key / A.page_size; };
        const auto page_of = [&](int c) {
            const int lp = tid < CHUNK && c <= run.last_chunk ? page_index(c * CHUNK + tid) : A.table_width;
            return lp < A.table_width ? bt[lp] : -1;
        };
        int c = seen_from(parts ? blockIdx.z : 0);
        if (parts && c > run.last_chunk) continue;

        const int rows = run.len * nheads;
        int page = page_of(c);
        {
            constexpr int WARPS = WIDE_THREADS / 32;
            float x[R / WARPS][4];                                               // a warp a row, everything requested at once
#pragma unroll
            for (int k = 0; k < R / WARPS; ++k) {
                const int r = warp + WARPS * k, t = r / nheads;
                const TA* src = q + (size_t)(t_first + run.first + t) * A.q_row_stride + (size_t)(h0 + r - t * nheads) * hd;
#pragma unroll
                for (int e = 0; e < 4; ++e) x[k][e] = r < rows && lane + 32 * e < hd ? to_f32(src[lane + 32 * e]) : 0.f;
            }
            __syncthreads();                                                     // the run before is done with the shared arrays
#pragma unroll
            for (int k = 0; k < R / WARPS; ++k)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (lane + 32 * e < hd) q_s[(warp + WARPS * k) * qld + lane + 32 * e] = x[k][e];
        }
        int my_head = 0;                                                         // of warp 0's lanes, a row each
        float m = -INFINITY, l = 0.f;                                            // the row's maximum and sum
        if (warp == 0) {
            const int t = run.first + lane / nheads;
            my_head = h0 + lane % nheads;
            const int pos = __shfl_sync(0xffffffffu, T.pos, t & 31), lo = __shfl_sync(0xffffffffu, T.lo, t & 31), kept = __shfl_sync(0xffffffffu, T.kept, t & 31);
            pos_s[lane] = lane < rows ? pos : -1;
            lo_s[lane] = lane < rows ? lo : 0;
            kept_s[lane] = lane < rows ? kept : 0;
            slope_s[lane] = A.sc.slopes != nullptr && lane < rows ? A.sc.slopes[my_head] : 0.f;
            at_s[lane] = (long long)(t_first + t) * A.nh + my_head;
        }
        __syncthreads();
        float acc[4][4];                                                         // of rows v_row + r, dimensions quad + e
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[r][e] = 0.f;
        while (c <= run.last_chunk) {
            const int c0 = c * CHUNK, c_next = seen_from(c + step);
            const int first = c < kept_chunks ? 0 : max(run.lo_min - c0, 0), last = min(run.pos_max - c0, CHUNK - 1);   // of the keys that any row sees
            bool any = false;
            long long key_row = -1;
            if (tid < CHUNK) {
                const int j = c0 + tid;
                any = j >= run.lo_max && j <= run.pos_min;                       // every row sees it
                int first_seer = 0;                                              // the first row whose token sees the key
                if (!any)
                    for (int r = rows - nheads; r >= 0; r -= nheads)
                        if ((j >= lo_s[r] || j < kept_s[r]) && j <= pos_s[r]) {
                            any = true;
                            first_seer = r;
                        }
                if (any) {
                    if (page < 0 || page >= A.num_pages) report_status(A.status, SPY_STATUS_BAD_PAGE, t_first + run.first + first_seer / nheads);
                    else key_row = ((((long long)page * A.planes) * A.nkv + kvh) * A.page_size + (j - page_index(j) * A.page_size)) * hd;
                }
                row_s[tid] = key_row;
            }
            page = page_of(c_next);
            const bool bad = __syncthreads_or(any && key_row < 0) != 0;          // a page that is none: its key is left out by every row
            const bool all_see = !bad && rows == R && c0 >= run.lo_max && c0 + CHUNK - 1 <= run.pos_min;
            const bool warp_sees = quarter * 32 <= last && quarter * 32 + 31 >= first && half * 16 < rows;
            float s[4][4];                                                       // of rows 16 half + 4 r + row_lane, keys 32 quarter + 8 e + key_lane
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[r][e] = 0.f;
            copy_rows(area0, kld, 0, last + 1, 0, 0, KD);
            copy_rows(area1, kld, 0, last + 1, 0, KD, hd - KD);
#pragma unroll 1
            for (int d0 = 0; d0 < hd; d0 += KD) {
                copy_wait<1>();
                __syncthreads();
                if (warp_sees) {
                    const TC* key = (d0 == 0 ? area0 : area1) + (quarter * 32 + key_lane) * kld;
                    const float* query = q_s + (half * 16 + row_lane) * qld + d0;
                    const int dims = min(KD, hd - d0);
#pragma unroll 2
                    for (int d = 0; d < dims; d += 4) {
                        float kq[4][4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) Vec4<TC>::load(key + 8 * e * kld + d, kq[e]);
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const float4 qv = *reinterpret_cast<const float4*>(query + 4 * r * qld + d);
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                s[r][e] = fmaf(qv.x, kq[e][0], s[r][e]);
                                s[r][e] = fmaf(qv.y, kq[e][1], s[r][e]);
                                s[r][e] = fmaf(qv.z, kq[e][2], s[r][e]);
                                s[r][e] = fmaf(qv.w, kq[e][3], s[r][e]);
                            }
                        }
                    }
                }
                __syncthreads();                                                 // this half of the keys has been read
                if (d0 == 0) copy_rows(area0, hd, 0, min(last + 1, CHUNK / 2), v_offset, 0, hd);
                else copy_rows(area1, hd, CHUNK / 2, last + 1, v_offset, 0, hd);
            }
            unsigned seen = 0xffffu;                                             // bit 4 r + e
            if (!all_see) {
                seen = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int at = quarter * 32 + 8 * e + key_lane, j = c0 + at;
                    const bool there = row_s[at] >= 0;
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int row = half * 16 + 4 * r + row_lane;            // beyond the run's: pos_s = -1
                        seen |= (there && (j >= lo_s[row] || j < kept_s[row]) && j <= pos_s[row] ? 1u : 0u) << (4 * r + e);
                    }
                }
            }
            int mine;
            {
                float tops[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int row = half * 16 + 4 * r + row_lane;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float x = __fmul_rn(s[r][e], A.scale);                   // rounded before the bias comes off, as above
                        if (A.sc.softcap > 0.f) x = __fmul_rn(A.sc.softcap, tanhf(x / A.sc.softcap));
                        if (A.sc.slopes != nullptr) x = fmaf(-slope_s[row], (float)(pos_s[row] - (c0 + quarter * 32 + 8 * e + key_lane)), x);
                        s[r][e] = (seen >> (4 * r + e) & 1) != 0 ? x : -INFINITY;
                    }
                    tops[r] = fmaxf(fmaxf(s[r][0], s[r][2]), fmaxf(s[r][1], s[r][3]));
                }
                const float top = reduce_four<TakeMax>(tops, &mine);
                if (mine >= 0) red[0][half * 16 + 4 * mine + row_lane][quarter] = top;
            }
            __syncthreads();
            {
                float sums[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int row = half * 16 + 4 * r + row_lane;
                    const float4 x = *reinterpret_cast<const float4*>(red[0][row]);
                    const float mc = fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w));
                    float w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const bool sees = (seen >> (4 * r + e) & 1) != 0;
                        const float p = mc != -INFINITY ? expf(s[r][e] - mc) : isnan(s[r][e]) ? s[r][e] : 0.f;
                        w[e] = sees ? p : 0.f;
                        p_s[quarter * 32 + 8 * e + key_lane][row] = sees || row >= rows ? w[e] * (1.f / CHUNK) : -1.f;
                    }
                    sums[r] = (w[0] + w[2]) + (w[1] + w[3]);                     // keys 16 apart, then 8: the order of a warp's sum
                }
                const float sum = reduce_four<TakeSum>(sums, &mine);
                if (mine >= 0) red[1][half * 16 + 4 * mine + row_lane][quarter] = sum;
            }
            copy_wait<1>();
            __syncthreads();
            if (warp == 0) {
                const float4 x = *reinterpret_cast<const float4*>(red[0][lane]), y = *reinterpret_cast<const float4*>(red[1][lane]);
                const float mc = fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)), lc = ((y.x + y.y) + y.z) + y.w;
                if (parts) {
                    if (lane < rows) {
                        float* part = A.partial + ((size_t)at_s[lane] * A.slots + c) * (hd + 2) + hd;
                        part[0] = mc;
                        part[1] = lc;
                    }
                } else {
                    float alpha = -1.f, beta = 0.f;                              // alpha below zero: there is nothing to take
                    if (!take_chunk(m, l, mc, lc, alpha, beta)) alpha = -1.f;
                    take_s[lane] = make_float2(alpha, CHUNK * beta);
                }
            }
            float vs[4][4];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int e = 0; e < 4; ++e) vs[r][e] = 0.f;
            {
                // [fa, fb): keys that every row of the block sees; elsewhere a row leaves out the keys whose p is below zero
                const int fa = max(first, run.lo_max - c0), fb = bad ? 0 : min(run.pos_min - c0, last) + 1;
                const float* p_g = &p_s[0][v_row];
                const TC* v_s = area0 + (has_quad ? quad : 0);
                int j = first, end = min(CHUNK / 2, last + 1);
#pragma unroll 1
                while (true) {
#pragma unroll 1
                    while (j < end) {
                        float v[4];
                        if (j >= fa && j < fb) {
                            const int whole = min(fb, end);
#pragma unroll 4
                            for (; j < whole; ++j) {
                                Vec4<TC>::load(v_s + j * hd, v);
                                const float4 p = *reinterpret_cast<const float4*>(p_g + j * PLD);
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    vs[0][e] = fmaf(p.x, v[e], vs[0][e]);
                                    vs[1][e] = fmaf(p.y, v[e], vs[1][e]);
                                    vs[2][e] = fmaf(p.z, v[e], vs[2][e]);
                                    vs[3][e] = fmaf(p.w, v[e], vs[3][e]);
                                }
                            }
                        } else {
                            Vec4<TC>::load(v_s + j * hd, v);
                            float p[4];
                            load_probabilities<4>(p_g + j * PLD, p);
#pragma unroll
                            for (int r = 0; r < 4; ++r)
                                if (!(p[r] < 0.f)) {
#pragma unroll
                                    for (int e = 0; e < 4; ++e) vs[r][e] = fmaf(p[r], v[e], vs[r][e]);
                                }
                            ++j;
                        }
                    }
                    if (end > last) break;
                    copy_wait<0>();
                    __syncthreads();
                    v_s = area1 + (has_quad ? quad : 0) - (CHUNK / 2) * hd;
                    end = last + 1;
                }
            }
            __syncthreads();                                                     // take_s is there; the next chunk rewrites the shared arrays
#pragma unroll
            for (int rr = 0; rr < 4; ++rr) {
                const int r = v_row + rr;
                if (parts) {
                    if (r < rows && has_quad) {
                        float* part = A.partial + ((size_t)at_s[r] * A.slots + c) * (hd + 2) + quad;
#pragma unroll
                        for (int e = 0; e < 4; ++e) part[e] = vs[rr][e];
                    }
                } else {
                    const float2 f = take_s[r];
                    if (!(f.x < 0.f)) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[rr][e] = fmaf(acc[rr][e], f.x, vs[rr][e] * f.y);
                    }
                }
            }
            c = c_next;
        }
        if (parts) continue;
        if (warp == 0) end_s[lane] = make_float2(with_sinks(A, my_head, m, l), A.sc.out_scale != nullptr && lane < rows ? A.sc.out_scale[at_s[lane]] : 1.f);
        __syncthreads();
        if (has_quad) {
#pragma unroll
            for (int rr = 0; rr < 4; ++rr) {
                const int r = v_row + rr;
                const float2 f = end_s[r];
                if (r < rows) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) out[at_s[r] * hd + quad + e] = from_f32<TA>(f.x > 0.f ? acc[rr][e] / f.x * f.y : 0.f);
                }
            }
        }
    }
}

// The rows whose chunks went to blocks of their own: the chunks added in order.
template <typename TA>
__global__ void __launch_bounds__(CHUNK) attention_merge_kernel(TA* __restrict__ out, AttnArgs A)
{
    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, hd = A.hd, t_first = t / A.per_tile * A.per_tile;
    const TileTokens T = load_tile(A, t_first);
    int i = 0;
    Run run = run_from(A, T, 0);
    while (t_first + i + run.len <= t) {                                         // the run that holds the token
        i += run.len;
        run = run_from(A, T, i);
    }
    pdl_enter();                                                                 // what is read above was complete when attention_rows_kernel let this one start
    if (!in_parts(A, run)) return;                                               // one block has stored it
    const int pos = __shfl_sync(0xffffffffu, T.pos, t - t_first), lo = __shfl_sync(0xffffffffu, T.lo, t - t_first);
    const int kept_chunks = (__shfl_sync(0xffffffffu, T.kept, t - t_first) + CHUNK - 1) / CHUNK;
    const int last_chunk = pos < 0 ? -1 : min(pos / CHUNK, A.max_chunks - 1);    // the chunks that attention_rows_kernel walks
    const float* part = A.partial + ((size_t)t * A.nh + h) * A.slots * (hd + 2);
    float m = -INFINITY, l = 0.f, acc = 0.f;
#pragma unroll 4
    for (int c = 0; c <= last_chunk; ++c) {
        if (c >= kept_chunks && c < lo / CHUNK) continue;
        const float* p = part + (size_t)c * (hd + 2);
        const float mc = p[hd], lc = p[hd + 1], v = tid < hd ? p[tid] : 0.f;
        float alpha, beta;
        if (take_chunk(m, l, mc, lc, alpha, beta)) acc = fmaf(acc, alpha, v * (CHUNK * beta));
    }
    if (tid < hd) {
        const long long row = (long long)t * A.nh + h;
        l = with_sinks(A, h, m, l);
        out[row * hd + tid] = from_f32<TA>(l > 0.f ? acc / l * (A.sc.out_scale != nullptr ? A.sc.out_scale[row] : 1.f) : 0.f);
    }
}

template <typename TA, typename TC, int R, int GROUPS>
static int launch_rows(const void* q, void* out, const void* pages, const AttnArgs& A, dim3 grid, cudaStream_t stream)
{
    const size_t smem = R * A.hd * sizeof(float) + (size_t)2 * A.area * sizeof(TC);
    SPY_ONCE_PER_DEVICE
    {
        const int most = (int)(R * CHUNK * sizeof(float) + 2 * CHUNK * (KD + 4) * sizeof(TC));   // with the static arrays more than the 48 KB that need no attribute
        SPY_CUDA(cudaFuncSetAttribute(attention_rows_kernel<TA, TC, R, GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    }
    spy_launch(attention_rows_kernel<TA, TC, R, GROUPS>, grid, dim3(CHUNK), smem, stream, (const TA*)q, (TA*)out, (const TC*)pages, A);
    if (A.slots > 0) spy_launch(attention_merge_kernel<TA>, dim3(A.tokens, A.nh), dim3(CHUNK), 0, stream, (TA*)out, A);
    return 0;
}

template <typename TA, typename TC>
static int launch_wide(const void* q, void* out, const void* pages, const AttnArgs& A, dim3 grid, cudaStream_t stream)
{
    const size_t smem = WIDE_ROWS * (A.hd + 4) * sizeof(float) + (size_t)2 * A.area * sizeof(TC);
    SPY_ONCE_PER_DEVICE
    {
        const int most = (int)(WIDE_ROWS * (CHUNK + 4) * sizeof(float) + 2 * CHUNK * (KD + 4) * sizeof(TC));
        SPY_CUDA(cudaFuncSetAttribute(attention_wide_kernel<TA, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    }
    spy_launch(attention_wide_kernel<TA, TC>, grid, dim3(WIDE_THREADS), smem, stream, (const TA*)q, (TA*)out, (const TC*)pages, A);
    if (A.slots > 0) spy_launch(attention_merge_kernel<TA>, dim3(A.tokens, A.nh), dim3(CHUNK), 0, stream, (TA*)out, A);
    return 0;
}

// How the rows are shared out; the results are the same to the last bit whatever is chosen here.
struct RowsPlan {
    int rows, heads, per_tile, head_groups;   // of a block: rows at most (4, 8, 16, 32), heads, tokens; blocks a kv head
    long long blocks;                         // without the split
    int chunks, slots, split;                 // of the table; chunks a row that the scratch holds (0: no scratch); blocks a row group's chunks are dealt to
};

static RowsPlan plan_rows(int tokens, int num_seqs, int nh, int nkv, int hd, int table_width, int page_size)
{
    RowsPlan P;
    const int group = nh / nkv, sms = spy_sm_count();
    P.chunks = (int)(((long long)table_width * page_size + CHUNK - 1) / CHUNK);
    const long long all_rows = (long long)tokens * nh;
    // Rows a block: few where a block's way through one chunk is what counts, more where blocks share the reading of many chunks.  Measured
    // with 4 / 8 / 16 (us): 16 heads a kv head, 100 keys, 1 to 16 requests 11.5 / 14 / 20; 16 requests of 4,096 keys 83 / 78 / 62; 4 of 4,096 40 / 32 / 37;
    // prompts of 32 heads over 8: 37 tokens 9.3 / 12 / 17, 300 tokens 116 / 112 / 92, 20 tokens behind 8,000 326 / 304 / 233: two blocks an SM are kept busy
    // by the wider choice.  Prompts with head sizes above 64 take 32 rows in place of 16 (attention_wide_kernel) wherever 16 would be chosen: at the least work
    // there (300 tokens of 5 heads over 1) 38.4 with 16 and 37.7, from there on 0.59 to 0.86 of the time.  A table of more than 64 chunks tells little about the contexts in it: 16 are assumed, for prompts their own length.
    const bool prompts = tokens > 2 * (long long)num_seqs;
    const long long work = all_rows * (P.chunks <= 64 ? P.chunks : prompts ? tokens / (num_seqs > 0 ? num_seqs : 1) / CHUNK + 1 : 16);
    const int most = work < 16LL * sms ? 4 : work < 32LL * sms ? 8 : hd > KD && prompts && work >= 32LL * sms ? WIDE_ROWS : 16;
    P.head_groups = (group + most - 1) / most;
    P.heads = (group + P.head_groups - 1) / P.head_groups;
    // several tokens a block where they outnumber the sequences by far (prompts), one where most tokens are their sequence's only one
    P.per_tile = prompts ? most / P.heads : 1;
    const int rows = P.heads * P.per_tile;
    P.rows = rows <= 4 ? 4 : rows <= 8 ? 8 : rows <= 16 ? 16 : WIDE_ROWS;
    P.blocks = ((long long)tokens + P.per_tile - 1) / P.per_tile * nkv * P.head_groups;
    // Chunks on blocks of their own: worth it while the device holds the blocks about twice at most and a row may have more than two
    // chunks (a launch more costs what a second chunk does).  The table says how many chunks there may be, not how many there are: the
    // blocks of a row group take its chunks in turns, as many blocks as fill the device, and rows longer than the scratch has room for
    // (64 MB) stay with one block.
    const long long room = (16LL << 20) / (all_rows * (hd + 2));
    P.slots = P.blocks < 8LL * sms && P.chunks > 2 && room > 2 ? (int)(room < P.chunks ? room : P.chunks) : 0;
    const long long fill = (16LL * sms + P.blocks - 1) / P.blocks;
    P.split = P.slots > 0 ? (int)(fill < P.slots ? fill : P.slots) : 1;
    return P;
}

// Floats of scratch with which the chunks of a row may go to blocks of their own (0: one block walks them all).
extern "C" long long spy_attention_generic_scratch(int tokens, int num_seqs, int nh, int nkv, int hd, int table_width, int page_size)
{
    if (tokens <= 0 || nh <= 0 || nkv <= 0 || nh % nkv != 0 || hd <= 0 || hd > CHUNK || hd % 4 != 0 || table_width <= 0 || page_size <= 0) return 0;
    return (long long)plan_rows(tokens, num_seqs, nh, nkv, hd, table_width, page_size).slots * tokens * nh * (hd + 2);
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
        const RowsPlan P = plan_rows(tokens, num_seqs, nh, nkv, hd, table_width, page_size);
        const long long need = (long long)P.slots * tokens * nh * (hd + 2);
        const bool split = need > 0 && scratch != nullptr && scratch_floats >= need;
        const int quads = (hd < KD ? hd : KD) / 4;                               // an odd number of quads between the keys: eight lanes meet no bank twice
        const int kld = 4 * (quads + 1 - quads % 2), area = CHUNK * kld;         // values: at most CHUNK * 64 numbers, in either layout
        const int page_shift = (page_size & (page_size - 1)) == 0 ? __builtin_ctz((unsigned)page_size) : -1;
        const AttnArgs A = {q_row_stride, block_table, table_width, page_size, num_pages, nh, nkv, hd, positions, seq_of_token, tokens, window, scale, status,
                            planes, keep_first, sink, scores, P.heads, P.per_tile, P.head_groups, P.chunks, page_shift, kld, area, scratch, split ? P.slots : 0};
        if ((long long)nkv * P.head_groups > 65535) SPY_FAIL("attention: %d heads exceed the grid limit", nh);
        const dim3 grid((tokens + P.per_tile - 1) / P.per_tile, nkv * P.head_groups, split ? P.split : 1);
#define SPY_ROWS_LAUNCH(R_) (hd <= 32 ? launch_rows<TA, TC, R_, 4>(q, out, pages, A, grid, stream) \
                             : hd <= 64 ? launch_rows<TA, TC, R_, 2>(q, out, pages, A, grid, stream) : launch_rows<TA, TC, R_, 1>(q, out, pages, A, grid, stream))
        SPY_DISPATCH_DTYPE(act_dtype, TA, {
            SPY_DISPATCH_DTYPE(cache_dtype, TC, {
                const int rc = P.rows == WIDE_ROWS ? launch_wide<TA, TC>(q, out, pages, A, grid, stream) : P.rows == 4 ? SPY_ROWS_LAUNCH(4) : P.rows == 8 ? SPY_ROWS_LAUNCH(8) : SPY_ROWS_LAUNCH(16);
                if (rc) return rc;
            })
        })
#undef SPY_ROWS_LAUNCH
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
