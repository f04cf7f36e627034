// sgemm_tc.cu — SGEMM on the tcgen05 tensor cores at single precision: every
// operand is split into three bf16 terms, x = h + m + l (24 = 8 + 8 + 8
// significant bits, each term the rounding of what the ones before leave, so
// the sum is exact), and the six products
//     h h' + (h m' + m h') + (m m' + h l' + l h')
// are formed by bf16 MMAs with FP32 accumulators.  The products left out (m l',
// l m', l l') are below 2^-26 of |x x'| each.  bf16 has the exponent range of
// FP32, so no operand needs scaling and every element of C keeps the error
// bound of a single-precision product, relative to sum_k |a_ik b_kj|.
//
// Accuracy.  A tensor-core accumulation rounds towards zero, so long sums in
// one accumulator would drift.  h h' therefore has accumulators of its own that
// take at most 128 values of k (eight rounded steps); then the drain warps add
// them to an FP32 sum in registers, rounded to nearest.  The other five
// products are below 2^-8 of it and keep two accumulators through all of k.
// Measured against 64 bits, relative Frobenius
// error for uniform[-1,1] operands, k = 8 / 256 / 4096 / 16384: 3.8e-8 / 7.7e-8
// / 1.5e-7 / 2.4e-7 (SIMT core: 5.4e-8 / 2.9e-7 / 1.1e-6 / 2.3e-6); for
// operands of one sign 3.9e-8 / 8.7e-8 / 1.7e-7 / 2.1e-7 (4.6e-8 / 2.2e-7 /
// 8.5e-7 / 1.7e-6).
//
// Operands the split does not cover are found by the splitting kernel, which marks
// them; the tensor kernel then returns at once and the SIMT kernel queued behind
// it, which otherwise returns at once, computes the product.  No host
// synchronisation is needed.  Covered are zeros and magnitudes in [2^-90, 2^60]:
// above, sums of products could overflow before a later term brings them back (and
// Inf and NaN have no split); below, products could be subnormal, where six of them
// are rounded for the SIMT core's one.  For the same reason the other operand
// must not go below 2^-34 where one goes below 2^-60 (no product below 2^-124:
// relative error 6e-8 there, the SIMT core's 1.1e-6).  The lower ends matter for
// operands with a few tiny entries, exp(-x) among them: the SIMT core takes seven
// times as long.
// Kernel layout: persistent, one CTA per SM and 128 x 128 tile of C, 576
// threads: warp 0 issues the TMA loads, warp 1 the MMAs, warps 2-17 drain (one
// row and 32 columns per thread).  The planes of B lie side by side as 384 rows
// of one 48 KB stage, h, m, l, so that one MMA multiplies a plane of A by two
// of them:
//     A_m [h' m'] -> [D1 D2]   A_l [h'] -> D2   A_h [m' l'] -> [D1 D2]   A_h [h'] -> D0
// with D1 = h m' + m h' and D2 = h l' + m m' + l h'.  An MMA costs the issuing
// thread about 70 cycles for up to 128 columns, so six products of 128 columns
// left the tensor pipe waiting for instructions (1.4 us per 64 values of k
// against 1.06 us now; 0.75 us of tensor time at the full clock).  D0 alternates between two
// accumulators, so its hand-over to the drain warps overlaps the next MMAs.
// CTA pairs (256 x 256 tiles) were slower, 648 us at 4096^3: the hand-overs
// between the two SMs take longer than the planes that fit can cover.
// Bound by the tensor pipe (74 % of the cycles active): 4096^3 takes 0.54 ms in a
// stream of calls, 0.59 through sgemm_, which waits for each; 54 us of them are the
// splitting (5.2 TB/s, bound by instruction issue) and 480 the products, 1.72 PFLOP/s
// of bf16 against a measured cuBLAS burst of 1.92.  SIMT core: 4.6 ms.
#include "gbx_internal.h"
#include "gemm_host.h"
#include "tc_ptx.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <atomic>
#include <mutex>

using namespace gbx_gemm;
using namespace gbx_tc;

namespace {

constexpr int ST_T = 128;             // tile of C
constexpr int ST_BK = 64;             // bf16 values per k block: 128-byte rows
constexpr int ST_PLANE = ST_T * ST_BK * 2;              // 16 KB: one plane of a k block
constexpr int ST_ASLOTS = 5, ST_BSTAGES = 3;            // A plane by plane, B all three planes together
constexpr int ST_DRAIN_WARPS = 16, ST_THREADS = 64 + 32 * ST_DRAIN_WARPS;
constexpr size_t ST_DATA = (size_t)(ST_ASLOTS + 3 * ST_BSTAGES) * ST_PLANE;
constexpr size_t ST_SMEM = ST_DATA + 1024 /*align*/ + 256 /*barriers*/;
constexpr int ST_D0 = 0, ST_D12 = 2 * ST_T;   // TMEM columns: D0 twice, then D1, D2
constexpr int ST_GROUP_M = 16;  // tile order: groups of 16 row tiles, row tile fastest
static_assert(ST_SMEM <= 227 * 1024, "opt-in shared memory");

inline cudaStream_t S(gbx_ctx *ctx) { return (cudaStream_t)gbx_ctx_get_stream(ctx); }

// ---------------------------------------------------------------- splitting
struct SplitOp {
    const float *X;
    long long ld;
    int row_k;            // 1: element (r, k) is X[r * ld + k]; 0: X[k * ld + r]
    int rows;
    __nv_bfloat16 *P;     // planes [3][rows][pitch]: h, m, l
    int tiles_r;
};

// Two floats as packed bf16 (a in the low half), and back.
__device__ __forceinline__ uint32_t pack_bf16(float a, float b)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ float lo_f(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi_f(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// Both operands, 64 x 64 tiles through shared memory: read along the
// contiguous index, written as 16-byte pieces along k: 4 bytes read and 6 written
// per element.  Bound by instruction issue (84 % of the slots) at 5.2 TB/s.
__global__ void __launch_bounds__(256)
split_bf16x3(SplitOp a, SplitOp b, int K, long long pitch, int blocks_a, unsigned *marks,
             unsigned tag)
{
    __shared__ float s[64][65];
    const bool is_a = (int)blockIdx.x < blocks_a;
    const SplitOp o = is_a ? a : b;
    const int blk = is_a ? blockIdx.x : blockIdx.x - blocks_a;
    const int r0 = (blk % o.tiles_r) * 64, k0 = (blk / o.tiles_r) * 64;
    const int t = threadIdx.x;
    unsigned least = 0xffffffffu, most = 0u;   // of the magnitudes' bit patterns; the least less one, without zeros
    float v[16];
#pragma unroll
    for (int u = 0; u < 16; u++) {
        const int x = t & 63, y = (t >> 6) + 4 * u;
        const int r = r0 + (o.row_k ? y : x), k = k0 + (o.row_k ? x : y);
        v[u] = r < o.rows && k < K ? (o.row_k ? o.X[(long long)r * o.ld + k] : o.X[(long long)k * o.ld + r]) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < 16; u++) {
        const uint32_t m = __float_as_uint(v[u]) & 0x7fffffffu;
        least = min(least, m - 1u);
        most = max(most, m);
        const int x = t & 63, y = (t >> 6) + 4 * u;
        if (o.row_k) s[y][x] = v[u];
        else s[x][y] = v[u];
    }
    __syncthreads();
    auto below = [&](int e) { return least < ((unsigned)(127 + e) << 23) - 1u; };   // an element below 2^e
    if (below(-34)) marks[is_a ? SPLIT_A_SMALL : SPLIT_B_SMALL] = tag;
    if (below(-60)) marks[is_a ? SPLIT_A_TINY : SPLIT_B_TINY] = tag;
    if (below(-90) || most > (127u + 60u) << 23) marks[SPLIT_UNCOVERED] = tag;
    const size_t plane = (size_t)o.rows * pitch;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int r = (t >> 3) + 32 * q, k = (t & 7) * 8;
        if (r0 + r >= o.rows || k0 + k >= pitch) continue;
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float x0 = s[r][k + 2 * j], x1 = s[r][k + 2 * j + 1];
            h[j] = pack_bf16(x0, x1);
            const float y0 = x0 - lo_f(h[j]), y1 = x1 - hi_f(h[j]);   // exact
            m[j] = pack_bf16(y0, y1);
            l[j] = pack_bf16(y0 - lo_f(m[j]), y1 - hi_f(m[j]));       // exact
        }
        __nv_bfloat16 *d = o.P + (size_t)(r0 + r) * pitch + k0 + k;
        *(uint4 *)d = make_uint4(h[0], h[1], h[2], h[3]);
        *(uint4 *)(d + plane) = make_uint4(m[0], m[1], m[2], m[3]);
        *(uint4 *)(d + 2 * plane) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

// ------------------------------------------------------------------ product
struct StParams {
    int M, N, nkb;
    int chunk;            // k blocks per D0 accumulator
    int tiles_m, tiles_n;
    float alpha, beta;
    float *C;
    long long ldc;
    const unsigned *marks;
    unsigned tag;
    int *status, *status_host;
};

// D[tmem] (+)= A[smem desc] * B[smem desc], kind::f16, one CTA.
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// kind::f16, dense: D = F32, A = B = BF16, both K-major, shape M x N
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void st_tile(const StParams &p, int t, int &tm, int &tn)
{
    const int per_group = ST_GROUP_M * p.tiles_n;
    const int g = t / per_group, r = t - g * per_group;
    const int rows = min(ST_GROUP_M, p.tiles_m - g * ST_GROUP_M);
    tm = g * ST_GROUP_M + r % rows;
    tn = r / rows;
}

// acc += this thread's row of 32 accumulator columns at taddr
__device__ __forceinline__ void st_add(float (&acc)[32], uint32_t taddr)
{
    uint32_t r[32];
    tmem_ld_32x32b_x32(taddr, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 32; j++) acc[j] += __uint_as_float(r[j]);
}

// C = alpha acc + beta C for 32 columns of one row (neighbouring lanes hold
// neighbouring rows); the loads of 16 columns are issued together.
__device__ __forceinline__ void st_store(const StParams &p, const float (&acc)[32], int row, int col)
{
    if (row >= p.M) return;
    float *c = p.C + (long long)col * p.ldc + row;
    const bool beta0 = p.beta == 0.0f;
#pragma unroll
    for (int b = 0; b < 32; b += 16) {
        float old[16];
        if (!beta0) {
#pragma unroll
            for (int j = 0; j < 16; j++) old[j] = col + b + j < p.N ? c[j * p.ldc] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 16; j++)
            if (col + b + j < p.N)
                c[j * p.ldc] =
                    beta0 ? Ops<float>::mul(p.alpha, acc[b + j]) : Ops<float>::axpby(p.alpha, acc[b + j], p.beta, old[j]);
        c += 16 * p.ldc;
    }
}

__global__ void __launch_bounds__(ST_THREADS, 1)
sgemm_bf16x3(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, StParams p)
{
    if (gbx_gemm::split_uncovered(p.marks, p.tag)) return;   // the SIMT kernel behind this one computes the product
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *smB = smem + ST_ASLOTS * ST_PLANE;
    uint64_t *bars = (uint64_t *)(smem + ST_DATA);
    uint64_t *fullA = bars, *emptyA = fullA + ST_ASLOTS, *fullB = emptyA + ST_ASLOTS, *emptyB = fullB + ST_BSTAGES;
    uint64_t *tfull = emptyB + ST_BSTAGES, *tempty = tfull + 2, *sempty = tempty + 2;
    uint32_t *tmem_slot = (uint32_t *)(sempty + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntiles = p.tiles_m * p.tiles_n;
    volatile int *status = p.status;

    if (threadIdx.x == 0) {
        for (int i = 0; i < ST_ASLOTS; i++) { mbar_init(&fullA[i], 1); mbar_init(&emptyA[i], 1); }
        for (int i = 0; i < ST_BSTAGES; i++) { mbar_init(&fullB[i], 1); mbar_init(&emptyB[i], 1); }
        for (int i = 0; i < 2; i++) { mbar_init(&tfull[i], 1); mbar_init(&tempty[i], ST_DRAIN_WARPS); }
        mbar_init(sempty, ST_DRAIN_WARPS);
        fence_barrier_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            int as = 0, bs = 0;
            uint32_t ap = 0, bp = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                int tm, tn;
                st_tile(p, t, tm, tn);
                for (int kb = 0; kb < p.nkb && ok; kb++) {
                    ok = mbar_wait(&emptyB[bs], bp ^ 1u, status, TC_TIMEOUT_EMPTY);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&fullB[bs], 3 * ST_PLANE);
                    tma_load_3d(smB + bs * 3 * ST_PLANE, &tmB, &fullB[bs], kb * ST_BK, tn * ST_T, 0);
                    if (++bs == ST_BSTAGES) { bs = 0; bp ^= 1u; }
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const int plane = i == 0 ? 1 : (i == 1 ? 2 : 0);   // m, l, h: the order of use
                        ok = ok && mbar_wait(&emptyA[as], ap ^ 1u, status, TC_TIMEOUT_EMPTY);
                        if (!ok) continue;
                        mbar_arrive_expect_tx(&fullA[as], ST_PLANE);
                        tma_load_3d(smem + as * ST_PLANE, &tmA, &fullA[as], kb * ST_BK, tm * ST_T, plane);
                        if (++as == ST_ASLOTS) { as = 0; ap ^= 1u; }
                    }
                }
            }
            // wait (bounded) until every load has landed and been used
            for (int i = 0; i < ST_ASLOTS; i++) {
                mbar_wait(&emptyA[as], ap ^ 1u, status, TC_TIMEOUT_EMPTY);
                if (++as == ST_ASLOTS) { as = 0; ap ^= 1u; }
            }
            for (int i = 0; i < ST_BSTAGES; i++) {
                mbar_wait(&emptyB[bs], bp ^ 1u, status, TC_TIMEOUT_EMPTY);
                if (++bs == ST_BSTAGES) { bs = 0; bp ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            int as = 0, bs = 0, buf = 0;
            uint32_t ap = 0, bp = 0, tp = 0, sp = 0;
            bool ok = true;
            const uint64_t a0 = smem_desc_k128(smem_u32(smem)), b0 = smem_desc_k128(smem_u32(smB));
            const uint32_t d12 = tmem_base + ST_D12, d2 = d12 + ST_T;
            constexpr uint32_t wide = idesc_bf16_f32(ST_T, 2 * ST_T), one = idesc_bf16_f32(ST_T, ST_T);
            constexpr uint64_t PL = ST_PLANE >> 4;   // a plane in descriptor address units
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                int left = 0;   // k blocks until D0 is handed over
                uint32_t d0 = 0;
                for (int kb = 0; kb < p.nkb; kb++) {
                    auto take_a = [&]() {
                        const bool r = mbar_wait(&fullA[as], ap, status, TC_TIMEOUT_FULL);
                        tc_fence_after();
                        return r;
                    };
                    auto next_a = [&]() {
                        mma_commit(&emptyA[as]);
                        if (++as == ST_ASLOTS) { as = 0; ap ^= 1u; }
                    };
                    // the tile's first products start D1 and D2, once the drain has read the last tile's
                    ok = (kb > 0 || mbar_wait(sempty, sp ^ 1u, status, TC_TIMEOUT_TMEM_EMPTY)) &&
                         mbar_wait(&fullB[bs], bp, status, TC_TIMEOUT_FULL) && take_a();
                    if (!ok) break;
                    const uint64_t db = b0 + (uint64_t)(bs * 3) * PL;
                    uint64_t da = a0 + (uint64_t)as * PL;
#pragma unroll
                    for (int kk = 0; kk < ST_BK / 16; kk++)
                        mma_f16(d12, da + 2 * kk, db + 2 * kk, wide, kb || kk ? 1u : 0u);   // m [h' m']
                    next_a();
                    if (!(ok = take_a())) break;
                    da = a0 + (uint64_t)as * PL;
#pragma unroll
                    for (int kk = 0; kk < ST_BK / 16; kk++)
                        mma_f16(d2, da + 2 * kk, db + 2 * kk, one, 1u);                     // l h'
                    next_a();
                    if (!(ok = take_a())) break;
                    da = a0 + (uint64_t)as * PL;
#pragma unroll
                    for (int kk = 0; kk < ST_BK / 16; kk++)
                        mma_f16(d12, da + 2 * kk, db + PL + 2 * kk, wide, 1u);              // h [m' l']
                    const bool first = left == 0;
                    if (first) {
                        ok = mbar_wait(&tempty[buf], tp ^ 1u, status, TC_TIMEOUT_TMEM_EMPTY);
                        if (!ok) break;
                        tc_fence_after();
                        left = min(p.chunk, p.nkb - kb);
                        d0 = tmem_base + ST_D0 + (uint32_t)(buf * ST_T);
                    }
#pragma unroll
                    for (int kk = 0; kk < ST_BK / 16; kk++)
                        mma_f16(d0, da + 2 * kk, db + 2 * kk, one, !first || kk ? 1u : 0u); // h h'
                    next_a();
                    mma_commit(&emptyB[bs]);
                    if (++bs == ST_BSTAGES) { bs = 0; bp ^= 1u; }
                    if (--left == 0) {
                        mma_commit(&tfull[buf]);
                        if (++buf == 2) { buf = 0; tp ^= 1u; }
                    }
                }
                sp ^= 1u;
            }
        }
    } else {
        // ---------------- drain (warps 2..17) ----------------
        const int quarter = warp & 3;         // TMEM lane window of this warp
        const int part = (warp - 2) >> 2;     // which 32 columns of an accumulator
        int buf = 0;
        uint32_t tp = 0;
        bool ok = true;
        const uint32_t tl = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * 32);
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
            int tm, tn;
            st_tile(p, t, tm, tn);
            float acc[32];
#pragma unroll
            for (int j = 0; j < 32; j++) acc[j] = 0.0f;
            for (int kb = 0; kb < p.nkb; kb += p.chunk) {
                // warp-uniform outcome: tcgen05.ld is .sync.aligned
                ok = __all_sync(0xffffffffu, mbar_wait(&tfull[buf], tp, status, TC_TIMEOUT_TMEM_FULL));
                if (!ok) break;
                tc_fence_after();
                st_add(acc, tl + ST_D0 + (uint32_t)(buf * ST_T));
                const bool last = kb + p.chunk >= p.nkb;
                if (last) {
                    st_add(acc, tl + ST_D12);
                    st_add(acc, tl + ST_D12 + ST_T);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {   // one arrival per warp
                    mbar_arrive(&tempty[buf]);
                    if (last) mbar_arrive(sempty);
                }
                if (++buf == 2) { buf = 0; tp ^= 1u; }
            }
            if (!ok) break;
            st_store(p, acc, tm * ST_T + quarter * 32 + lane, tn * ST_T + part * 32);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if (threadIdx.x == 0 && *status != 0) {
        *(volatile int *)p.status_host = *status;
        __threadfence_system();
    }
}

// --------------------------------------------------------------------- host
typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                             const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn()
{
    static EncodeFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *q = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &q, 12000, cudaEnableDefault, &r) == cudaSuccess &&
            r == cudaDriverEntryPointSuccess)
            fn = (EncodeFn)q;
    });
    return fn;
}

// Planes as a (k, row, plane) tensor; rows and k beyond the operand read as
// zero, so the planes need no padding.
bool plane_map(CUtensorMap *map, void *base, int rows, int K, long long pitch, int box_planes)
{
    EncodeFn enc = encode_fn();
    if (!enc) return false;
    cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, 3};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)rows * pitch * 2};
    cuuint32_t box[3] = {ST_BK, ST_T, (cuuint32_t)box_planes}, estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

constexpr size_t ST_WS_MAX = (size_t)2 << 30;   // planes held at once

size_t st_plane_bytes(int m, int n, int k, size_t *a_bytes)
{
    const size_t pitch = ((size_t)k + 7) / 8 * 8;
    const size_t a = (6 * (size_t)m * pitch + 255) / 256 * 256;
    if (a_bytes) *a_bytes = a;
    return a + 6 * (size_t)n * pitch;
}

// What marks are set to: different in every call of the process, so that
// scratch need not be cleared.  (Scratch that happens to hold it costs the SIMT
// kernel's time, no more.)
unsigned next_tag()
{
    static std::atomic<unsigned> n{0x9d3c5a7eu};
    return ++n;
}

// The product with its scratch at ws.
gbx_status run_planes(gbx_ctx *ctx, const GemmArgs<float> &g, const char *what, char *ws, size_t a_bytes, int *words,
                      int *mirror)
{
    const long long pitch = ((long long)g.k + 7) / 8 * 8;
    __nv_bfloat16 *pa = (__nv_bfloat16 *)(ws + 256), *pb = (__nv_bfloat16 *)(ws + 256 + a_bytes);
    CUtensorMap tmA, tmB;
    if (!plane_map(&tmA, pa, g.m, g.k, pitch, 1) || !plane_map(&tmB, pb, g.n, g.k, pitch, 3))
        return gbx_fail(ctx, GBX_ERR_CUDA, "%s: cuTensorMapEncodeTiled failed", what);
    unsigned *marks = (unsigned *)ws;
    const unsigned tag = next_tag();

    SplitOp a{}, b{};
    a.X = g.A; a.ld = g.lda; a.row_k = g.ta; a.rows = g.m; a.P = pa; a.tiles_r = (g.m + 63) / 64;
    b.X = g.B; b.ld = g.ldb; b.row_k = !g.tb; b.rows = g.n; b.P = pb; b.tiles_r = (g.n + 63) / 64;
    const int kt = (g.k + 63) / 64;
    split_bf16x3<<<(unsigned)(kt * (a.tiles_r + b.tiles_r)), 256, 0, S(ctx)>>>(a, b, g.k, pitch, kt * a.tiles_r, marks,
                                                                               tag);
    StParams p{};
    p.M = g.m; p.N = g.n;
    p.nkb = (g.k + ST_BK - 1) / ST_BK;
    p.tiles_m = (g.m + ST_T - 1) / ST_T;
    p.tiles_n = (g.n + ST_T - 1) / ST_T;
    p.chunk = p.nkb > 4 ? 2 : 1;
    p.alpha = g.alpha; p.beta = g.beta;
    p.C = g.C; p.ldc = g.ldc;
    p.marks = marks; p.tag = tag;
    p.status = words + 4;
    p.status_host = mirror;
    // a per-device function attribute; setting it is a cheap host call
    if (cudaFuncSetAttribute(sgemm_bf16x3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ST_SMEM) != cudaSuccess)
        return gbx_fail(ctx, GBX_ERR_CUDA, "%s: shared memory attribute", what);
    const int grid = std::min(p.tiles_m * p.tiles_n, gbx_ctx_sms(ctx));
    gbx_timer_begin(ctx, GBX_TIMER_GEMM_FP64);
    sgemm_bf16x3<<<grid, ST_THREADS, ST_SMEM, S(ctx)>>>(tmA, tmB, p);
    gbx_timer_end(ctx);
    gbx_count_launch(ctx, 2);
    gbx_status st = gbx_check_launch(ctx, what);
    if (st != GBX_OK) return st;
    return launch_gemm_if(ctx, g, what, marks, tag);
}

}  // namespace

// Whether an m x n x k product is faster on the tensor cores than on the SIMT
// core.  Splitting, product and conditional SIMT launch take about 15 us
// however small the product is, and a tile's k loop 16 ns per k; a SIMT call
// takes 6 us and 32 ns per k for its 16 x 16 tiles, more once several of them
// share an SM, and its larger tiles (two of 32 x 32 per SM and up) are slow on
// short k.  Measured, tensor / SIMT us: 64 x 64 x 1024 31 / 35, 64 x 64 x 4096 78 /
// 131, 300^3 21 / 19, 384^3 22 / 27, 32 x 4096 x 256 21 / 19, 4096 x 16 x 512 27 / 23,
// 256 x 256 x 1024 31 / 41, 8 x 4096 x 4096 107 / 153, 1024 x 1024 x 16 17 / 86,
// 2000 x 2000 x 8 23 / 116, 128^3 18 / 8.
extern "C" int gbx_sgemm_tensor_choice(int m, int n, int k, int sms)
{
    const double work = (double)m * n * k;
    if (k >= 1024) return work >= 4e6;
    const long long tiles32 = ((m + 31LL) / 32) * ((n + 31) / 32);
    return work >= 4e7 || (k >= 8 && tiles32 >= 2LL * sms);
}

namespace gbx_gemm {

gbx_status sgemm_tensor(gbx_ctx *ctx, const GemmArgs<float> &g, const char *what, bool *done)
{
    *done = false;
    if (!gbx_sgemm_tensor_choice(g.m, g.n, g.k, gbx_ctx_sms(ctx))) return GBX_OK;
    // A capture gets the SIMT core: its replays outlive this call, may run on any
    // stream, and must not use scratch that other calls use too.
    if (gbx_capturing(ctx)) return GBX_OK;
    size_t a_bytes;
    const size_t planes = st_plane_bytes(g.m, g.n, g.k, &a_bytes);
    if (planes > ST_WS_MAX) {
        // halve the longer side: the pieces are independent products
        const bool rows = g.m >= g.n;
        const int len = rows ? g.m : g.n, h = (len / 2 + 255) / 256 * 256;
        if (h <= 0 || h >= len) return GBX_OK;
        for (int part = 0; part < 2; part++) {
            GemmArgs<float> q = g;
            const long long o = part ? h : 0;
            const int w = part ? len - h : h;
            if (rows) {
                q.m = w;
                q.A += g.ta ? o * g.lda : o;
                q.C += o;
            } else {
                q.n = w;
                q.B += g.tb ? o : o * g.ldb;
                q.C += o * g.ldc;
            }
            bool d = false;
            gbx_status st = sgemm_tensor(ctx, q, what, &d);
            if (st == GBX_OK && !d) st = launch_gemm<float>(ctx, q, what);
            if (st != GBX_OK) return st;
        }
        *done = true;
        return GBX_OK;
    }
    int *words, *mirror;
    if (gbx_ctx_status(ctx, &words, &mirror) != GBX_OK) return GBX_OK;
    // 256 bytes of marks, then the planes; where they cannot be had the SIMT core
    // takes the call
    void *ws;
    int block;
    if (gbx_scratch_get(ctx, 256 + planes, &ws, &block) != GBX_OK) return GBX_OK;
    *done = true;
    const gbx_status st = run_planes(ctx, g, what, (char *)ws, a_bytes, words, mirror);
    const gbx_status put = gbx_scratch_put(ctx, block);
    return st != GBX_OK ? st : put;
}

}  // namespace gbx_gemm
