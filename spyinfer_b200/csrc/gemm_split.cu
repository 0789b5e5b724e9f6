// The float32 path's matrix product on the 5th-generation tensor cores:  C[M, N] = A[M, K] . W[N, K]^T with 32-bit A and C and
// bfloat16 W.  A finite 32-bit number is exactly the sum of three bfloat16 numbers (24 bits of mantissa in runs of eight, cut, not
// rounded), the second and third scaled by powers of two where they are stored, so three tensor-core products with the same weight tile give every term
// of the 32-bit product exactly; what is left is how the terms are summed.
//
// The sums.  The tensor core adds into its accumulator by cutting, which leans toward zero a little at every step (measured:
// 2.4e-8 of the result after 16 terms of K, 6.7e-8 after 64, 2.3e-7 after 256).  So the leading pieces' accumulator is taken
// out of tensor memory every 64 terms of K (one K block) and added to a sum in registers by an ordinary rounded addition; the other two
// pieces are 2^-8 and 2^-16 of the size and are accumulated through.
// Relative error (2-norm) against 64 bits at K = 256, 4,096 and 12,288: 0.7e-7, 1.1e-7 and 1.4e-7, where the CUDA-core kernel, one
// chain over K, has 2.9e-7, 1.1e-6 and 2.0e-6.  (Every 32 terms: 0.7e-7, 1.6e-7 and 2.6e-7, twice as many rounded additions.)
//
// A row's result does not depend on M or on its neighbours: K is cut into slices by N, K and the device (plan_slices), a slice's sum
// runs over its K blocks of 64 in order, and the slices are added in order.
//
// Bounds.  Few tokens: the weights' way through memory (2 bytes a weight).  Many: the tensor cores (three passes).  Measured with
// the pieces' kernel, from a graph, weights not in L2 (the CUDA-core kernel took 822 us a product on average at 4 tokens of these
// sizes, 1,690 at 300):   N x K = 6,144 x 4,096: 15 us at 4 tokens, 72 at 300;   4,096 x 4,096: 12 and 62;   24,576 x 4,096: 41
// (4.9 TB/s) and 191 (317 TFLOP/s of 32-bit product, three times that on the tensor cores);   4,096 x 12,288: 23 and 113;
// 151,936 x 4,096: 200 (6.2 TB/s).
// Tiles: up to 128 weight rows in the instruction's M slot and 16, 32 or 64 tokens in its N slot, each token three times (a
// product with the leading pieces, N = BN, and one with the two others side by side, N = 2 BN), two blocks an SM up to 32
// tokens so that enough weight bytes are under way; beyond 64 tokens 256 weight rows as two halves over 64 tokens (56 KB a
// stage for 24 products), where a half's sums are taken out while the other half multiplies.  A thread that waits, issues and
// commits needs about 60 to 100 cycles for each, more than these small products take, so the leading and the other pieces of each
// half are issued by a warp of their own (one warp for all: 27 us where this takes 20), and sums are handed over once a K block
// (every 32 terms: 221 us where this takes 191).
// The slices of a tile are the blocks of a cluster: their partial tiles meet through shared memory, no scratch, no second kernel.
//
// An element whose sum is no finite number is summed again from the operands term by term in 32-bit, so that infinities and
// NaN come out as a plain sum gives them (a zero piece times an infinite weight would make NaN of an infinity).
//
// Counterpart: the reference computes this path in 32-bit on the CPU (spymaster2h/spyinfer src/backends/cpu/x64/kernels.cpp:95-166).
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"

SPY_MODULE(spy_gemm_split)

namespace {

using namespace tc;

constexpr int BK = 64;            // 64 bfloat16 = 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
constexpr int MAX_STAGES = 8;
constexpr int MAX_SLICES = 8;     // blocks of a cluster
constexpr float PIECE_SCALE = 256.f;   // of the second piece; of the third its square (split3)

template <int BN, int HALVES> struct Shape {
    static constexpr int ISSUERS = 2 * HALVES;             // warps that issue products: a half's leading pieces, a half's two others
    static constexpr int FIRST_SUM_WARP = 1 + ISSUERS;     // warp 0: TMA and tensor memory; then the issuers; then four warps a half that sum
    static constexpr int THREADS = 32 * FIRST_SUM_WARP + 128 * HALVES;
    static constexpr int ROWS = 128 * HALVES;              // weight rows of a tile, at most
    static constexpr int Y_BYTES = BN * BK * 2;            // one piece of the tokens
    static constexpr int COLS = (HALVES == 1 ? 8 : 4) * BN;   // tensor-memory columns of a half: buffers of the leading pieces' sums, then the two other pieces'
    static constexpr int BUFFERS = COLS / BN - 2;          // blocks of K whose sums may wait to be taken out
    static constexpr int PER_SM = HALVES == 1 && BN <= 32 ? 2 : 1;
    static constexpr int AREA = (PER_SM == 2 ? 110 : 224) * 1024;
    static constexpr size_t SMEM = (size_t)AREA + 1024 /* alignment */ + 512 /* barriers */;
    static constexpr int LD = ROWS + 4;                    // floats between the tokens of the staged result
    __host__ __device__ static constexpr int x_bytes(int rows) { return (rows * BK * 2 + 1023) & ~1023; }
    // The tensor core reads 128 rows a half: spare ones come from what lies behind and feed sums that are never stored; the area ends with room for that
    __host__ __device__ static constexpr int stages(int rows)
    {
        const int n = (AREA - (ROWS * BK * 2 - x_bytes(rows))) / (x_bytes(rows) + 3 * Y_BYTES);
        return n < MAX_STAGES ? n : MAX_STAGES;
    }
    static_assert(BN * LD * 4 <= AREA, "the staged result fits the stages' place");
    static_assert(COLS * HALVES * PER_SM <= 512, "tensor memory");
};

__device__ __forceinline__ float4 ld_cluster4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// One element, term by term in 32-bit in order, when its sum is no finite number; it ends with the first NaN, which stays one.  Sixteen terms
// are requested at a time (K is a multiple of 8, weight rows start on 16-byte borders).  4, 64 and 300 rows by 4,096 x 4,096 (us): of NaN 20, 35 and
// 85 (one term after the other to the end 1,340 and 8,000 for the first two), with an infinity in each 410, 1,800 and 5,400; without 14, 25 and 63.
__device__ __noinline__ float plain_sum(const float* a, const bf16* w, int K)
{
    float s = 0.f;
    for (int k = 0; k < K && !isnan(s); k += 16) {
        const bool both = k + 8 < K;
        uint4 wv[2];
        float av[16];
        wv[0] = *reinterpret_cast<const uint4*>(w + k);
        wv[1] = *reinterpret_cast<const uint4*>(w + k + (both ? 8 : 0));
#pragma unroll
        for (int e = 0; e < 16; ++e) av[e] = a[k + (e < 8 || both ? e : 0)];
#pragma unroll
        for (int e = 0; e < 16; ++e)
            if (e < 8 || both) s = fmaf(av[e], __bfloat162float(reinterpret_cast<const bf16*>(wv)[e]), s);
    }
    return s;
}

// W [n_rows, K] through map_w (boxes of tile_rows rows), the pieces [3][m_rows][K] through map_a (boxes of BN rows).
template <int BN, int HALVES>
__global__ void __launch_bounds__(Shape<BN, HALVES>::THREADS, Shape<BN, HALVES>::PER_SM)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, float* __restrict__ out, long long ldc,
                  const float* __restrict__ A, long long lda, const bf16* __restrict__ W, long long ldw, int n_rows, int m_rows, int K,
                  int k_blocks_per_slice, int tile_rows, int* status)
{
    using S = Shape<BN, HALVES>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + S::AREA);
    uint64_t* empty_bar = full_bar + MAX_STAGES;
    constexpr int NB = S::BUFFERS;
    uint64_t* sum_full = empty_bar + MAX_STAGES;           // [HALVES][NB] a K block's sums of the leading pieces are complete
    uint64_t* sum_empty = sum_full + NB * HALVES;          // [HALVES][NB] they have been taken out
    uint64_t* done_bar = sum_empty + NB * HALVES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int x0 = blockIdx.y * tile_rows, y0 = blockIdx.x * BN;
    const int x_bytes = S::x_bytes(tile_rows), stage_bytes = x_bytes + 3 * S::Y_BYTES, stages = S::stages(tile_rows);
    const uint32_t stage_tx = (uint32_t)tile_rows * BK * 2 + 3 * S::Y_BYTES;
    const int k_blocks = (K + BK - 1) / BK;
    const int kb0 = blockIdx.z * k_blocks_per_slice;
    const int num_kb = min(k_blocks - kb0, k_blocks_per_slice);      // at least one (plan_slices)
    const int slices = gridDim.z;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full_bar + s, 1);
            mbar_init(empty_bar + s, S::ISSUERS);
        }
        for (int i = 0; i < NB * HALVES; ++i) {
            mbar_init(sum_full + i, 1);
            mbar_init(sum_empty + i, 4);
        }
        mbar_init(done_bar, S::ISSUERS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(tmem_slot, (uint32_t)(S::COLS * HALVES));
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    pdl_launch_dependents();
    if (warp == 0) {
        if (lane == 0) {
            // the weights depend on no earlier kernel: the first stages' are requested before the wait for the kernels ahead
            const int pre = min(num_kb, stages);
            for (int i = 0; i < pre; ++i) {
                mbar_expect_tx(full_bar + i, stage_tx);
                tma_load_2d(smem_u32(tiles + (size_t)i * stage_bytes), &map_w, (kb0 + i) * BK, x0, full_bar + i);
            }
            pdl_wait();
            for (int i = 0; i < pre; ++i) {
                uint8_t* ys = tiles + (size_t)i * stage_bytes + x_bytes;
                for (int p = 0; p < 3; ++p) tma_load_2d(smem_u32(ys + p * S::Y_BYTES), &map_a, (kb0 + i) * BK, y0 + p * m_rows, full_bar + i);
            }
            int s = 0;
            uint32_t phase = 0;
            for (int i = pre; i < num_kb; ++i) {
                if (!mbar_wait(empty_bar + s, phase, abort_flag)) break;
                uint8_t* xs = tiles + (size_t)s * stage_bytes;
                mbar_expect_tx(full_bar + s, stage_tx);
                tma_load_2d(smem_u32(xs), &map_w, (kb0 + i) * BK, x0, full_bar + s);
                for (int p = 0; p < 3; ++p) tma_load_2d(smem_u32(xs + x_bytes + p * S::Y_BYTES), &map_a, (kb0 + i) * BK, y0 + p * m_rows, full_bar + s);
                if (++s == stages) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
    } else if (warp < S::FIRST_SUM_WARP) {
        if (lane == 0) {
            const int half = (warp - 1) >> 1;
            const bool lead = ((warp - 1) & 1) == 0;
            const uint32_t acc = tmem + (uint32_t)(half * S::COLS), x_off = (uint32_t)(half * 128 * BK * 2);
            int s = 0;
            uint32_t phase = 0;
            if (lead) {
                const uint32_t idesc = instr_desc_bf16(128, BN, false, false);
                uint64_t* full = sum_full + NB * half;
                uint64_t* empty = sum_empty + NB * half;
                int b = 0;
                uint32_t taken = 1;                        // the parity of a buffer's release that its next use waits for
                for (int i = 0; i < num_kb; ++i) {
                    if (!mbar_wait(full_bar + s, phase, abort_flag)) break;
                    const uint32_t xs = smem_u32(tiles + (size_t)s * stage_bytes);
                    const uint64_t dx = desc_k_major(xs + x_off), dy = desc_k_major(xs + x_bytes);
                    if (i >= NB && !mbar_wait(empty + b, taken, abort_flag)) break;
                    fence_after_sync();
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        umma(acc + (uint32_t)(b * BN), dx + (uint64_t)(k * UMMA_K * 2 >> 4), dy + (uint64_t)(k * UMMA_K * 2 >> 4), idesc, k > 0 ? 1u : 0u);
                    umma_commit(full + b);
                    if (++b == NB) {
                        b = 0;
                        taken ^= 1;
                    }
                    umma_commit(empty_bar + s);
                    if (++s == stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            } else {
                const uint32_t idesc = instr_desc_bf16(128, 2 * BN, false, false);
                for (int i = 0; i < num_kb; ++i) {
                    if (!mbar_wait(full_bar + s, phase, abort_flag)) break;
                    fence_after_sync();
                    const uint32_t xs = smem_u32(tiles + (size_t)s * stage_bytes);
                    const uint64_t dx = desc_k_major(xs + x_off), dy = desc_k_major(xs + x_bytes + S::Y_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        umma(acc + NB * BN, dx + (uint64_t)(k * UMMA_K * 2 >> 4), dy + (uint64_t)(k * UMMA_K * 2 >> 4), idesc, (i > 0 || k > 0) ? 1u : 0u);
                    umma_commit(empty_bar + s);
                    if (++s == stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
            umma_commit(done_bar);
        }
    } else {
        const int half = (warp - S::FIRST_SUM_WARP) >> 2, quarter = warp & 3;
        const uint32_t acc = tmem + (uint32_t)(half * S::COLS) + ((uint32_t)(quarter * 32) << 16);
        constexpr int C = BN < 32 ? BN : 32;
        float sum[BN];
#pragma unroll
        for (int c = 0; c < BN; ++c) sum[c] = 0.f;
        int b = 0;
        uint32_t phase = 0;
        for (int n = 0; n < num_kb; ++n) {
            if (!mbar_wait_warp(sum_full + NB * half + b, phase, abort_flag)) break;
            fence_after_sync();
#pragma unroll
            for (int c = 0; c < BN; c += C) {
                uint32_t r[C];
                tmem_load<C>(acc + (uint32_t)(b * BN + c), r);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < C; ++e) sum[c + e] += __uint_as_float(r[e]);
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(sum_empty + NB * half + b);
            if (++b == NB) {
                b = 0;
                phase ^= 1;
            }
        }
        mbar_wait_warp(done_bar, 0, abort_flag);           // every product is complete: the stages are free as well
        fence_after_sync();
        float* staged = reinterpret_cast<float*>(tiles) + half * 128 + quarter * 32 + lane;
#pragma unroll
        for (int c = 0; c < BN; c += C) {
            uint32_t r1[C], r2[C];
            tmem_load<C>(acc + (uint32_t)(NB * BN + c), r1);
            tmem_load<C>(acc + (uint32_t)((NB + 1) * BN + c), r2);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < C; ++e) staged[(size_t)(c + e) * S::LD] =
                fmaf(fmaf(__uint_as_float(r2[e]), 1.f / PIECE_SCALE, __uint_as_float(r1[e])), 1.f / PIECE_SCALE, sum[c + e]);   // the scales are powers of two: two rounded additions
        }
        fence_before_sync();
    }
    __syncwarp();
    if (slices > 1) cluster_sync();
    else __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        // a wait ran out: copies that may still be in flight get time to land before the shared memory is released
        const unsigned long long t0 = global_timer();
        while (global_timer() - t0 < 2000000ull) { }
        report_status(status, SPY_STATUS_WAIT_TIMEOUT, (int)(blockIdx.x + blockIdx.y * gridDim.x));
    }
    pdl_wait();   // the output may still be in use by a kernel ahead in the stream
    {
        // the slices' partial tiles, added in order; block z of a cluster finishes every slices-th run of the tile
        const int outs = min(tile_rows, n_rows - x0), rows = min(BN, m_rows - y0);
        const uint32_t own = smem_u32(tiles);
        uint32_t part[MAX_SLICES];
#pragma unroll
        for (int z = 0; z < MAX_SLICES; ++z) part[z] = map_to_rank(own, z < slices ? z : 0);
        float* gout = out + (size_t)y0 * ldc + x0;
        const int first = blockIdx.z * S::THREADS + threadIdx.x, step = slices * S::THREADS;
        if ((outs & 3) == 0 && (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(gout) & 15) == 0) {
            const int quads = outs >> 2;
            for (int u = first; u < rows * quads; u += step) {
                const int t = u / quads, q = 4 * (u - t * quads);
                const uint32_t off = (uint32_t)(t * S::LD + q) * 4;
                float4 p[MAX_SLICES];
#pragma unroll
                for (int z = 0; z < MAX_SLICES; ++z)
                    if (z < slices) p[z] = ld_cluster4(part[z] + off);
                float v[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
                for (int z = 1; z < MAX_SLICES; ++z)
                    if (z < slices) {
                        v[0] += p[z].x;
                        v[1] += p[z].y;
                        v[2] += p[z].z;
                        v[3] += p[z].w;
                    }
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (!isfinite(v[e])) v[e] = plain_sum(A + (size_t)(y0 + t) * lda, W + (size_t)(x0 + q + e) * ldw, K);
                *reinterpret_cast<float4*>(gout + (size_t)t * ldc + q) = make_float4(v[0], v[1], v[2], v[3]);
            }
        } else {
            for (int u = first; u < rows * outs; u += step) {
                const int t = u / outs, q = u - t * outs;
                const uint32_t off = (uint32_t)(t * S::LD + q) * 4;
                float v = ld_cluster(part[0] + off);
                for (int z = 1; z < slices; ++z) v += ld_cluster(map_to_rank(own, z) + off);
                if (!isfinite(v)) v = plain_sum(A + (size_t)(y0 + t) * lda, W + (size_t)(x0 + q) * ldw, K);
                gout[(size_t)t * ldc + q] = v;
            }
        }
    }
    __syncwarp();
    if (slices > 1) cluster_sync();   // no block leaves while another reads its shared memory
    else __syncthreads();
    if (warp == 0) {
        fence_after_sync();
        tmem_dealloc(tmem, (uint32_t)(S::COLS * HALVES));
    }
}

// The three pieces of 32-bit rows: pieces[p][m][k], eight numbers a thread.  Numbers that are not finite go into the first piece alone.
// The second piece is stored 2^PIECE_SHIFT times as large, the third 2^(2 PIECE_SHIFT): as they are, their last bits would lie below the smallest
// bfloat16 number (2^-133) for numbers under 2^-110.
__device__ __forceinline__ void split3(float a, uint32_t& p0, uint32_t& p1, uint32_t& p2)
{
    const uint32_t u = __float_as_uint(a);
    if ((u & 0x7f800000u) == 0x7f800000u) {
        p0 = (u >> 16) | ((u & 0x7fffffu) != 0 ? 0x40u : 0u);      // a NaN stays one
        p1 = p2 = 0;
        return;
    }
    p0 = u >> 16;
    const float r = (a - __uint_as_float(u & 0xffff0000u)) * PIECE_SCALE;        // exact: the low 16 bits of the mantissa, below 2^-7 of the number
    const uint32_t ur = __float_as_uint(r);
    p1 = ur >> 16;
    p2 = __float_as_uint((r - __uint_as_float(ur & 0xffff0000u)) * PIECE_SCALE) >> 16;   // what is left has at most eight bits
}

__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ A, long long lda, bf16* __restrict__ pieces, int m_rows, int K, int vec)
{
    pdl_enter();
    const long long eights = K / 8, total = eights * m_rows, plane = (long long)m_rows * K;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / eights, k = 8 * (i - m * eights);
        const float* src = A + m * lda + k;
        float v[8];
        if (vec) {
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src);
            *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(src + 4);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = src[e];
        }
        uint32_t p[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            uint32_t a[3], b[3];
            split3(v[2 * e], a[0], a[1], a[2]);
            split3(v[2 * e + 1], b[0], b[1], b[2]);
#pragma unroll
            for (int j = 0; j < 3; ++j) p[j][e] = a[j] | (b[j] << 16);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<uint4*>(pieces + j * plane + m * K + k) = make_uint4(p[j][0], p[j][1], p[j][2], p[j][3]);
    }
}

int make_map(CUtensorMap* map, const void* base, long long rows, int K, long long ld, int box_rows)
{
    EncodeTiledFn encode = encode_tiled_fn();
    if (encode == nullptr) SPY_FAIL("gemm_split: the driver has no cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult rc = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) SPY_FAIL("gemm_split: tensor map for %lld x %d (row stride %lld) failed with code %d", rows, K, ld, (int)rc);
    return 0;
}

template <int BN, int HALVES> int set_up()
{
    SPY_ONCE_PER_DEVICE
    {
        SPY_CUDA(cudaFuncSetAttribute(gemm_split_kernel<BN, HALVES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<BN, HALVES>::SMEM));
        SPY_CUDA(cudaFuncSetAttribute(gemm_split_kernel<BN, HALVES>, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
    }
    return 0;
}

template <int BN, int HALVES> void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], dim3 grid, int slices, cudaStream_t stream)
{
    cfg.gridDim = grid;
    cfg.blockDim = dim3(Shape<BN, HALVES>::THREADS);
    cfg.dynamicSmemBytes = Shape<BN, HALVES>::SMEM;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = slices;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = spy_pdl_enabled() ? 2 : 1;
}

// How many clusters of `slices` blocks the device holds at a time with `per_sm` blocks an SM, asked once per device.  The
// occupancy query counts one block an SM for every kernel that uses tensor memory, although two share one (seen in their start
// times), so the clusters of two blocks an SM are those of half as many blocks of one an SM.
int resident_clusters(int slices, int per_sm, int* count)
{
    static int known[SPY_MAX_DEVICES][MAX_SLICES + 1] = {};
    const bool halve = per_sm == 2 && slices % 2 == 0;
    const int ask = halve ? slices / 2 : slices;
    int& c = known[spy_device()][ask];
    if (c == 0) {
        if (int rc = set_up<16, 1>()) return rc;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        configure<16, 1>(cfg, attr, dim3(1, 1, ask), ask, nullptr);
        cfg.numAttrs = 1;
        int n = 0;
        SPY_CUDA(cudaOccupancyMaxActiveClusters(&n, gemm_split_kernel<16, 1>, &cfg));
        if (n <= 0) SPY_FAIL("gemm_split: no cluster of %d blocks fits the device", ask);
        c = n;
    }
    *count = per_sm == 2 && !halve ? 2 * c : c;
    return 0;
}

// Weight rows of a tile (a multiple of 8) for which `n_rows` weight rows in `slices` slices of `per` K blocks take the least
// time, and that time in cycles: rounds of `clusters` tiles, a round's K blocks at the memory's rate (3,400 bytes a cycle once
// five sixths of the places are taken) but no faster than a block's chain of waits and issues allows (720 cycles a K block
// measured), and 5,500 cycles for its start and end.
double plan_rows(int n_rows, int slices, int clusters, int per, int* rows_out)
{
    double best = 0;
    const auto round = [&](int tiles, int rows) {
        const double blocks = (double)tiles * slices, places = (double)clusters * slices * 5.0 / 6.0;
        const double memory = rows * 128.0 * (blocks > places ? blocks : places) / 3400.0;
        return per * (memory > 720.0 ? memory : 720.0) + 5500.0;
    };
    for (int rows = 128; rows >= 64; rows -= 8) {
        const int tiles = (n_rows + rows - 1) / rows, full = tiles / clusters, left = tiles - full * clusters;
        const double cost = full * round(clusters, rows) + (left > 0 ? round(left, rows) : 0.0);
        if (rows == 128 || cost < best) {
            best = cost;
            *rows_out = rows;
        }
    }
    return best;
}

// Into how many slices K is cut: by N, K and what the device holds, for a step of few tokens (whose blocks should fill the device and whose
// weights should arrive evenly); steps of many tokens use the same slices, so that a row's sums never depend on its company.
int plan_slices(int n_rows, int k_blocks, int* slices_out)
{
    double best = 0;
    for (int z = 1; z <= MAX_SLICES; ++z) {
        const int per = (k_blocks + z - 1) / z;
        if (z > 1 && (per < 4 || (k_blocks + per - 1) / per != z)) continue;
        int clusters = 0, rows = 0;
        if (int rc = resident_clusters(z, 2, &clusters)) return rc;
        const double cost = plan_rows(n_rows, z, clusters, per, &rows) + 250.0 * (z - 1);
        if (z == 1 || cost < best) {
            best = cost;
            *slices_out = z;
        }
    }
    return 0;
}

template <int BN, int HALVES>
int launch(const CUtensorMap& mw, const CUtensorMap& ma, float* C, long long ldc, const float* A, long long lda, const bf16* W, long long ldw, int N, int M, int K,
           int slices, int per, int tile_rows, int* status, cudaStream_t stream)
{
    if (int rc = set_up<BN, HALVES>()) return rc;
    const int tiles = (N + tile_rows - 1) / tile_rows;
    if (tiles > 65535) SPY_FAIL("gemm_split: %d weight rows exceed the grid", N);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    configure<BN, HALVES>(cfg, attr, dim3((M + BN - 1) / BN, tiles, slices), slices, stream);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_split_kernel<BN, HALVES>, mw, ma, C, ldc, A, lda, W, ldw, N, M, K, per, tile_rows, status);
    if (e != cudaSuccess) SPY_FAIL("gemm_split: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

}  // namespace

// Slices of K that a weight of this shape is cut into (for the tests).
extern "C" int spy_gemm_split_slices(int N, int K, int* slices) { return plan_slices(N, (K + BK - 1) / BK, slices); }

// A [M, K] and C [M, N] float32, W [N, K] bfloat16, rows lda/ldc/ldw elements apart (W's on 16-byte borders; K a multiple of 8).
// pieces: scratch of 3 * M * K bfloat16, 16-byte aligned.
extern "C" int spy_gemm_split(const float* A, long long lda, const void* W, long long ldw, float* C, long long ldc, int M, int N, int K, void* pieces,
                              int* status, cudaStream_t stream)
{
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 8 != 0) SPY_FAIL("gemm_split: K %d must be a positive multiple of 8 (16-byte rows for TMA)", K);
    if (lda < K || ldw < K || ldc < N) SPY_FAIL("gemm_split: row strides %lld/%lld/%lld are shorter than the rows", lda, ldw, ldc);
    if (ldw % 8 != 0 || (reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(pieces) & 15) || pieces == nullptr)
        SPY_FAIL("gemm_split: weight rows and pieces must start on 16-byte borders");
    if (M > (0x7fffffff - 64) / 3) SPY_FAIL("gemm_split: %d rows", M);
    const int vec = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    long long blocks = ((long long)M * (K / 8) + 255) / 256;
    if (blocks > 8LL * spy_sm_count()) blocks = 8LL * spy_sm_count();
    spy_launch(split_rows_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, A, lda, (bf16*)pieces, M, K, vec);
    SPY_CHECK_LAUNCH("gemm_split (pieces)");

    const int k_blocks = (K + BK - 1) / BK;
    int slices = 1;
    if (int rc = plan_slices(N, k_blocks, &slices)) return rc;
    const int per = (k_blocks + slices - 1) / slices;
    // 64 tokens and fewer: one token tile, as narrow as it may be.  More: 256 weight rows under every 64 tokens.
    const int bn = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
    int tile_rows = 256;
    if (M <= 64) {
        int clusters = 0;
        if (int rc = resident_clusters(slices, bn == 64 ? 1 : 2, &clusters)) return rc;
        plan_rows(N, slices, clusters, per, &tile_rows);
    }
    CUtensorMap mw, ma;
    if (make_map(&mw, W, N, K, ldw, tile_rows) || make_map(&ma, pieces, 3LL * M, K, K, bn)) return 1;
#define SPY_SPLIT_LAUNCH(BN_, H_) launch<BN_, H_>(mw, ma, C, ldc, A, lda, (const bf16*)W, ldw, N, M, K, slices, per, tile_rows, status, stream)
    if (M > 64) return SPY_SPLIT_LAUNCH(64, 2);
    if (bn == 16) return SPY_SPLIT_LAUNCH(16, 1);
    if (bn == 32) return SPY_SPLIT_LAUNCH(32, 1);
    return SPY_SPLIT_LAUNCH(64, 1);
#undef SPY_SPLIT_LAUNCH
}
