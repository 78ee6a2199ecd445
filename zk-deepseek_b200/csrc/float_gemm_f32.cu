// float32 linear layers of more than 16 rows on the tensor cores: out = epilogue(A W^T) from exact bfloat16 thirds.
//
// A float times 2^24 is the sum of three bfloat16 numbers exactly, subnormal ones too: the nearest one, the nearest to what that leaves,
// and the rest.  (Without the factor, which the sums lose again at the end, bfloat16's smallest numbers cut the last third of what is
// below 2^-110: error 9e-6 at 2^-118, 2e-3 at 2^-126, where now it is 9e-8 as at 1.)  Operands from 2^104 and sums from 2^80 on leave the
// range and are taken by multiply-adds, see again_by_fma.  Of the nine products of thirds the six largest are taken: what is dropped is
// up to 2^-24 of a product, as much as a float's own rounding, of either sign, and 2^-27 on average.  On the CUDA cores these layers are
// bound by FMAs at 64 lanes an SM and clock; here by the pieces of both operands that have to be in flight (loads of floats, cut into
// thirds by the threads, 3 x 64 bytes a row and stage) and by 6 MMAs of 128 x NT x 16 for 16 k, a third of what those FMAs take.
//
// Precision: the tensor memory's sums are cut, not rounded, which takes 1.45e-8 of a sum of positive numbers for every 16 k.  So
// the products of the first thirds are collected after one or two stages (32 or 64 k) and added up in 32 bits, rounded; the other
// products are 2^-8 of them and less, of either sign, and stay.  Relative error against 64 bits (2-norm), this kernel and the FMAs, 17 to
// 300 rows, 128 to 16384 columns: normal operands, K 128 to 1024 6e-8 to 1.1e-7 and 1.5e-7 to 4.1e-7, K 2048 9.8e-8 to 1.3e-7 and 2.9e-7 to
// 4.1e-7, K 8192 1.2e-7 to 2.5e-7 and 5.7e-7 to 8.1e-7.  Positive operands are where FMAs in clusters that share a K below 2048 are good
// (6.5e-8 to 8e-8): a share of up to 512 there is collected after every stage, 5.6e-8 to 8e-8, where two stages have 8.7e-8 to 9.6e-8 and
// everywhere would cost 5 % (and more additions: K 8192 1.4e-7 -> 1.6e-7).  From K 2048 on positive operands have 8.7e-8 to 1.9e-7, FMAs
// 9.9e-8 to 3.5e-7.  Above the FMAs: 64 rows, 8192 x 1536 9.0e-8 (8.0e-8) and 33 rows, 16384 x 3072 1.2e-7 (1.0e-7).
// (One sum for all products: 1.8e-6 where the FMAs have 1.2e-6.)
//
// Weights take the MMA's 128 rows, up to 160 rows of A its columns: three sets of sums in 480 of 512 columns of tensor memory.
// Clusters of up to eight CTAs share K and add their sums through each other's shared memory, in rank order.
// 300 rows, 2048 x 2048: 80 -> 32 us; 16384 x 2048: 477 -> 158 us; 17 rows, 1344 x 2048: 19 -> 13 us; a prompt of 300 tokens at
// width 2048 2.69 -> 1.30 ms, 1.10 with attention_f32_kernel.
#include <float.h>
#include <math.h>

#include <atomic>

#include "float_common.cuh"
#include "tcgen05.cuh"

namespace zkds {

namespace {

constexpr int kSplitN = 128;                       // weight rows of a CTA: the MMA's 128 rows
constexpr int kSplitK = 32;                        // k of a stage: rows of 64 bytes, 64-byte swizzle
constexpr int kSplitWarps = 12;                    // warps that cut operands into thirds and finish the sums
constexpr int kSplitThreads = 32 * (kSplitWarps + 5);   // one more issues the MMAs, four collect their sums
constexpr int kSplitNT = 160;                      // most rows of A in a tile: three sets of sums in tensor memory
constexpr int kSplitStages = 4;
constexpr int kSplitPitch = kSplitN + 4;           // floats between the tokens of the finished sums
constexpr float kSplitScale = 16777216.f;          // 2^24: the last bit of any float is then a normal number
constexpr uint32_t kSplitW = kSplitN * kSplitK * 2;     // bytes of one third of the weights in a stage

__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr)
{
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}

// the bfloat16 nearest to each of eight numbers, and what that leaves (exactly: of a float, 16 bits; of those, 8)
__device__ __forceinline__ void nearest_halves(const uint64_t (&x)[4], uint32_t (&half)[4], uint64_t (&left)[4])
{
    const uint64_t minus = twice(-1.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        asm("{\n\t.reg .f32 a, b;\n\tmov.b64 {a, b}, %1;\n\tcvt.rn.bf16x2.f32 %0, b, a;\n\t}" : "=r"(half[i]) : "l"(x[i]));
        uint64_t h;
        asm("mov.b64 %0, {%1, %2};" : "=l"(h) : "r"(half[i] << 16), "r"(half[i] & 0xFFFF0000u));
        left[i] = x[i];
        fma2(left[i], h, minus);
    }
}

__device__ __forceinline__ float4 peer_sums(uint32_t own, unsigned rank)
{
    float4 v;
    asm volatile("{\n\t.reg .b32 p;\n\tmapa.shared::cluster.u32 p, %4, %5;\n\t"
                 "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [p];\n\t}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(own), "r"(rank) : "memory");
    return v;
}

// Outputs whose sum is not finite, once more: thirds of an infinity are no number.  `again` marks them, eight columns a bit, 16 bits a
// row, of `rows` rows from m0 on.  What has a NaN in its row or its weights is none; the rest, finite neighbours in the same eight
// among it, is taken by multiply-adds, 512 threads with eight columns of five rows each, 32 k at a time through shared memory.
// 300 rows, 16384 x 2048, against a thread an output that walked all of K by itself: rows of NaN 24.9 -> 0.31 ms, one of them 0.85 -> 0.30,
// an infinity in every row 25.0 -> 1.33 (finite 0.17; linear_f32_kernel 0.48 on any of them); 2048 x 8192: 12.9 -> 0.26, 2.0 -> 0.25, 12.9 ->
// 1.71 (0.09; 0.29).
constexpr int kAgainPitch = kSplitNT + 4, kAgainTile = kSplitN + kSplitNT;
__device__ __noinline__ void again_by_fma(const float* A, long long lda, const float* W, long long ldw, int M, int N, int K, int m0, int n0,
                                          int rows, const uint32_t* again, const LinEpi& e)
{
    extern __shared__ __align__(16) uint8_t raw[];             // (a pointer from outside would make every access a generic one)
    constexpr int kRows = kSplitNT / 32, kPieces = (kAgainTile * 8 + kSplitThreads - 1) / kSplitThreads;
    float *sw = reinterpret_cast<float*>(raw), *sa = sw + 32 * kSplitPitch;    // [k][weight rows], [k][rows of A]
    uint8_t* nan = raw + 32 * (kSplitPitch + kAgainPitch) * 4;                 // of the weights' rows, then A's
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    for (int row = warp; row < kSplitN + rows; row += kSplitThreads / 32) {
        const bool is_w = row < kSplitN, in = is_w ? n0 + row < N : m0 + row - kSplitN < M;
        const float* x = is_w ? W + (long long)(n0 + row) * ldw : A + (long long)(m0 + row - kSplitN) * lda;
        bool found = false;
#pragma unroll 4
        for (int k = lane * 4; in && k < K; k += 128) {
            const float4 v = *reinterpret_cast<const float4*>(x + k);
            found |= v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
        }
        found = __any_sync(0xffffffffu, found);
        if (lane == 0) nan[row] = found;
    }
    __syncthreads();
    uint32_t wanted = 0, left = 0, no_number = 0;             // rows of this thread: marked, for multiply-adds; its columns that are NaN
    if (ty < 32) {
#pragma unroll
        for (int i = 0; i < 8; ++i) no_number |= (uint32_t)nan[8 * tx + i] << i;
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            const int r = ty + 32 * j, it = r * (kSplitN / 8) + tx;
            if (r >= rows || !(again[it >> 5] >> (it & 31) & 1u)) continue;
            wanted |= 1u << j;
            if (!nan[kSplitN + r] && no_number != 255u) left |= 1u << j;
        }
    }
    uint64_t acc[kRows][4] = {};
    if (__syncthreads_or(left != 0)) {
        const int half = (kSplitN + rows) * 4;
        float4 x[kPieces];
        auto fetch = [&](int k0) {
#pragma unroll
            for (int u = 0; u < kPieces; ++u) {
                const int i = tid + u * kSplitThreads, at = i < half ? i : i - half, row = at >> 2, c = (at & 3) * 4 + (i < half ? 0 : 16);
                x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k0 + c >= K || at >= half) continue;
                if (row < kSplitN && n0 + row < N) x[u] = *reinterpret_cast<const float4*>(W + (long long)(n0 + row) * ldw + k0 + c);
                if (row >= kSplitN && m0 + row - kSplitN < M)
                    x[u] = *reinterpret_cast<const float4*>(A + (long long)(m0 + row - kSplitN) * lda + k0 + c);
            }
        };
        fetch(0);
        for (int k0 = 0; k0 < K; k0 += 32) {
            __syncthreads();
#pragma unroll
            for (int u = 0; u < kPieces; ++u) {
                const int i = tid + u * kSplitThreads, at = i < half ? i : i - half, row = at >> 2, c = (at & 3) * 4 + (i < half ? 0 : 16);
                if (at >= half) continue;
                // weights: the first four of every eight columns, then the others, so that 16 threads read them side by side
                const int pitch = row < kSplitN ? kSplitPitch : kAgainPitch;
                float* s = row < kSplitN ? sw + c * pitch + (row >> 3) * 4 + (row & 3) + (row & 4) * 16 : sa + c * pitch + row - kSplitN;
                s[0] = x[u].x; s[pitch] = x[u].y; s[2 * pitch] = x[u].z; s[3 * pitch] = x[u].w;
            }
            __syncthreads();
            if (k0 + 32 < K) fetch(k0 + 32);
            if (!left) continue;
            const int nk = min(32, K - k0);
#pragma unroll 4
            for (int k = 0; k < nk; ++k) {
                const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(sw + k * kSplitPitch + 4 * tx);
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(sw + k * kSplitPitch + 64 + 4 * tx);
#pragma unroll
                for (int j = 0; j < kRows; ++j)
                    if (32 * j < rows) {
                        const uint64_t a = twice(sa[k * kAgainPitch + ty + 32 * j]);
                        fma2(acc[j][0], a, u.x); fma2(acc[j][1], a, u.y);
                        fma2(acc[j][2], a, v.x); fma2(acc[j][3], a, v.y);
                    }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kRows; ++j)
        if (wanted >> j & 1u) {
            const int r = ty + 32 * j, m = m0 + r;
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                v[i] = nan[kSplitN + r] || (no_number >> i & 1u) ? NAN : __uint_as_float((uint32_t)(acc[j][i >> 1] >> (32 * (i & 1))));
            epilogue8(e, e.kind == ZKFP_EPI_ROTATE ? epi_position(e, m) : 0, m, n0 + 8 * tx, v);
        }
}

// U: pieces of eight k that a thread cuts per stage
template <int U>
__global__ void __launch_bounds__(kSplitThreads, 1)
linear_split_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W, long long ldw, int M, int N, int K,
                    int NT, int m_tiles, int ksplit, int stages, uint32_t tmem_cols, int* error_flag, const __grid_constant__ LinEpi e)
{
    extern __shared__ __align__(16) uint8_t raw[];
    uint8_t* base = (uint8_t*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t s_full[kSplitStages], s_empty[kSplitStages], s_sum, s_taken, s_done;
    __shared__ uint32_t s_tmem, s_again[kSplitNT * (kSplitN / 8) / 32];
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int share = blockIdx.x % ksplit, tile = blockIdx.x / ksplit;
    const int n0 = tile / m_tiles * kSplitN, m0 = tile % m_tiles * NT;
    const int kblocks = (K + kSplitK - 1) / kSplitK, per = (kblocks + ksplit - 1) / ksplit;
    const int kb0 = share * per, kb1 = min(kblocks, kb0 + per);
    const uint32_t a_third = (uint32_t)NT * kSplitK * 2, stage_bytes = 3 * (kSplitW + a_third), smem0 = smem_u32(base);
    const int chunk_stages = K < 2048 && per <= 16 ? 1 : 2;      // stages after which the products of the first thirds are collected
    volatile int* abort_flag = &s_abort;

    if (tid < kSplitNT * (kSplitN / 8) / 32) s_again[tid] = 0;
    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < stages; ++i) {
            mbar_init(smem_u32(&s_full[i]), kSplitWarps);
            mbar_init(smem_u32(&s_empty[i]), 1);
        }
        mbar_init(smem_u32(&s_sum), 1);
        mbar_init(smem_u32(&s_taken), 4);
        mbar_init(smem_u32(&s_done), 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == kSplitWarps) tmem_alloc(smem_u32(&s_tmem), tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    float* sums = reinterpret_cast<float*>(base);          // [token][kSplitPitch], over the stages once they are done with

    // tensor memory: [0, NT) products of the first thirds of a chunk, [NT, 2 NT) all other products, [2 NT, 3 NT) sums of chunks
    if (warp == kSplitWarps) {
        const uint32_t one = elect_one(), tm = uniform(tmem);
        {
            const uint32_t idesc = idesc_bf16(kSplitN, NT);
            int s = 0;
            uint32_t phase = 0, chunk = 0, sums_made = 0;
            bool ok = true;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!(ok = mbar_wait_warp(smem_u32(&s_full[s]), phase, abort_flag))) break;
                tc_fence_after();
                const uint32_t sw = smem0 + (uint32_t)s * stage_bytes, sa = sw + 3 * kSplitW;
                uint64_t w[3], a[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    w[i] = smem_desc_sw64(sw + (uint32_t)i * kSplitW);
                    a[i] = smem_desc_sw64(sa + (uint32_t)i * a_third);
                }
                const uint32_t rest = tm + (uint32_t)NT;
#pragma unroll
                for (int k = 0; k < kSplitK / 16; ++k) {
                    const uint64_t at = (uint64_t)(k * 2);
                    umma_bf16(rest, w[2] + at, a[0] + at, idesc, kb > kb0 || k ? 1u : 0u, one);
                    umma_bf16(rest, w[1] + at, a[1] + at, idesc, 1u, one);
                    umma_bf16(rest, w[0] + at, a[2] + at, idesc, 1u, one);
                    umma_bf16(rest, w[1] + at, a[0] + at, idesc, 1u, one);
                    umma_bf16(rest, w[0] + at, a[1] + at, idesc, 1u, one);
                }
                const int in_chunk = (kb - kb0) % chunk_stages;
                if (in_chunk == 0 && kb > kb0) {          // the chunk in front has been collected under these
                    if (!(ok = mbar_wait_warp(smem_u32(&s_taken), chunk & 1u, abort_flag))) break;
                    tc_fence_after();
                    ++chunk;
                }
#pragma unroll
                for (int k = 0; k < kSplitK / 16; ++k)
                    umma_bf16(tm, w[0] + (uint64_t)(k * 2), a[0] + (uint64_t)(k * 2), idesc, in_chunk || k ? 1u : 0u, one);
                umma_commit(smem_u32(&s_empty[s]), one);
                if (in_chunk == chunk_stages - 1 || kb == kb1 - 1) { umma_commit(smem_u32(&s_sum), one); ++sums_made; }
                if (++s == stages) { s = 0; phase ^= 1u; }
            }
            if (!ok) {                                     // no MMA in flight when tensor memory goes back
                umma_commit(smem_u32(&s_sum), one);
                for (uint32_t i = 0; i < kSpinLimit; ++i)
                    if (mbar_try(smem_u32(&s_sum), sums_made & 1u)) break;
            }
        }
    } else if (warp > kSplitWarps) {
        // the sums of a chunk, 32 rows of tensor memory a warp
        const uint32_t tq = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const int chunks = kb1 > kb0 ? (kb1 - kb0 + chunk_stages - 1) / chunk_stages : 0;
        bool ok = true;
        for (int c = 0; c < chunks && ok; ++c) {
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_sum), (uint32_t)c & 1u, abort_flag));
            if (!ok) break;
            tc_fence_after();
            for (int n = 0; n < NT; n += 16) {
                int32_t x[16], t[16];
                tmem_ldn(tq + (uint32_t)n, x);
                if (c) tmem_ldn(tq + (uint32_t)(2 * NT + n), t);
                tmem_ld_wait();
                if (c)
#pragma unroll
                    for (int i = 0; i < 16; ++i) x[i] = __float_as_int(__int_as_float(t[i]) + __int_as_float(x[i]));
                tmem_st16(tq + (uint32_t)(2 * NT + n), reinterpret_cast<uint32_t(&)[16]>(x));
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(c == chunks - 1 ? &s_done : &s_taken));
        }
    } else {
        const float* src[U];
        uint32_t dst[U], third[U];
        const int c8 = (tid & 3) * 8;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int row = (tid + u * 32 * kSplitWarps) >> 2, r = row < kSplitN ? row : row - kSplitN;
            const bool is_w = row < kSplitN;
            dst[u] = (is_w ? 0u : 3 * kSplitW) + (uint32_t)(r * 64 + (((tid & 3) ^ ((r >> 1) & 3)) << 4));
            third[u] = is_w ? kSplitW : a_third;
            src[u] = is_w ? (n0 + r < N ? W + (long long)(n0 + r) * ldw + c8 : nullptr)
                          : (r < NT && m0 + r < M ? A + (long long)(m0 + r) * lda + c8 : nullptr);
            if (!is_w && r >= NT) third[u] = 0;            // nothing to write
        }
        auto fetch = [&](float4 (&v)[U][2], int kb) {
            const int k = kb * kSplitK;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                v[u][0] = v[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (src[u] && kb < kb1 && k + c8 < K) {
                    v[u][0] = __ldg(reinterpret_cast<const float4*>(src[u] + k));
                    v[u][1] = __ldg(reinterpret_cast<const float4*>(src[u] + k) + 1);
                }
            }
        };
        int s = 0;
        uint32_t phase = 0;
        bool ok = true;
        auto put = [&](const float4 (&v)[U][2]) {
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[s]), phase ^ 1u, abort_flag));
            if (!ok) return;
            const uint32_t st = smem0 + (uint32_t)s * stage_bytes;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!third[u]) continue;
                uint64_t x[4], m[4], l[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    asm("mov.b64 %0, {%1, %2};\n\tmul.rn.f32x2 %0, %0, %3;" : "=&l"(x[i])
                        : "f"(i & 1 ? v[u][i >> 1].z : v[u][i >> 1].x), "f"(i & 1 ? v[u][i >> 1].w : v[u][i >> 1].y), "l"(twice(kSplitScale)));
                uint32_t t[3][4];
                nearest_halves(x, t[0], m);
                nearest_halves(m, t[1], l);
                nearest_halves(l, t[2], m);
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(st + dst[u] + (uint32_t)j * third[u]),
                                 "r"(t[j][0]), "r"(t[j][1]), "r"(t[j][2]), "r"(t[j][3])
                                 : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_full[s]));
            if (++s == stages) { s = 0; phase ^= 1u; }
        };
        constexpr int AHEAD = U == 2 ? 3 : 2;              // stages whose loads are in flight
        float4 v[AHEAD][U][2];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) fetch(v[i], kb0 + i);
        for (int kb = kb0; kb < kb1 && ok; kb += AHEAD)
#pragma unroll
            for (int i = 0; i < AHEAD; ++i)
                if (kb + i < kb1 && ok) {
                    put(v[i]);
                    fetch(v[i], kb + i + AHEAD);
                }
        // the sums: a lane holds a column of the output, a column of tensor memory is a token
        const bool some = kb0 < kb1;
        if (some && ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_done), 0, abort_flag));
        tc_fence_after();
        const int q = warp & 3;
        const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16);
        if (ok) {
            for (int c = (warp >> 2) * 16; c < NT; c += 16 * (kSplitWarps / 4)) {
                int32_t x[16] = {}, y[16] = {};
                if (some) {
                    tmem_ldn(tq + (uint32_t)(2 * NT + c), x);
                    tmem_ldn(tq + (uint32_t)(NT + c), y);
                    tmem_ld_wait();
                }
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    sums[(c + i) * kSplitPitch + q * 32 + lane] = __int_as_float(x[i]) + __int_as_float(y[i]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kSplitWarps) tmem_dealloc(tmem, tmem_cols);
    if (tid == 0 && s_abort) *(volatile int*)error_flag = 1;
    if (ksplit > 1) asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    // a slice of the tokens each, the shares of K added in a fixed order
    const int rows = (NT + ksplit - 1) / ksplit;
    int again = 0;
    for (int it = tid; it < rows * (kSplitN / 8); it += kSplitThreads) {
        const int r = share * rows + it / (kSplitN / 8), c = it % (kSplitN / 8) * 8, m = m0 + r, n = n0 + c;
        if (r >= NT || m >= M || n >= N) continue;
        const float* own = sums + r * kSplitPitch + c;
        float v[8];
        if (ksplit == 1) {
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(own);
            *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(own + 4);
        } else {
            const uint32_t at = smem_u32(own);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = 0.f;
            for (int p = 0; p < ksplit; ++p) {
                const float4 x = peer_sums(at, p), y = peer_sums(at + 16, p);
                v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
                v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
            }
        }
        bool finite = true;
#pragma unroll
        for (int i = 0; i < 8; ++i) finite &= fabsf(v[i]) <= FLT_MAX;
        if (!finite) {
            atomicOr(&s_again[it >> 5], 1u << (it & 31));
            again = 1;
            continue;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] *= 1.f / (kSplitScale * kSplitScale);
        epilogue8(e, e.kind == ZKFP_EPI_ROTATE ? epi_position(e, m) : 0, m, n, v);
    }
    if (ksplit > 1) asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    // (the peers are done with the sums here)
    if (__syncthreads_or(again)) again_by_fma(A, lda, W, ldw, M, N, K, m0 + share * rows, n0, rows, s_again, e);
}

}  // namespace

// clusters of so many CTAs that the current device holds at a time, one CTA to an SM
static int split_clusters(int size)
{
    static std::atomic<int> known[64][4];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fp_sm_count() / size;
    std::atomic<int>& held = known[dev][size == 1 ? 0 : size == 2 ? 1 : size == 4 ? 2 : 3];
    int n = held.load(std::memory_order_relaxed);
    if (n) return n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(size * fp_sm_count()));
    cfg.blockDim = dim3(kSplitThreads);
    cfg.dynamicSmemBytes = 200 * 1024;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(linear_split_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedMax - 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, linear_split_kernel<3>, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = fp_sm_count() / size;
    }
    held.store(n, std::memory_order_relaxed);
    return n;
}

namespace {

struct SplitPlan {
    long long n_tiles, m_tiles;
    int nt, ksplit;
};

// tiles and shares of K with the least time of a wave times waves: an SM's start and end, and for each stage what the slower of the
// threads that cut operands and the MMAs takes (clocks, fitted to sweeps of both)
SplitPlan split_plan(const zkfp_linear_args& a)
{
    const long long kb = (a.K + kSplitK - 1) / kSplitK, n_tiles = (a.N + kSplitN - 1) / kSplitN;
    const long long few = (a.M + kSplitNT - 1) / kSplitNT;
    SplitPlan best{n_tiles, few, 16, 1};
    long long least = 0;
    for (long long mt = few; mt <= few + 1; ++mt) {
        const int nt = (int)(((a.M + mt - 1) / mt + 15) / 16 * 16);
        for (int s = 1; s <= 8; s *= 2) {
            if (s > 1 && kb / s < 4) break;
            const long long held = split_clusters(s), waves = (n_tiles * mt + held - 1) / held;
            const long long block = 576 + 9 * nt / 2 > 6 * nt ? 576 + 9 * nt / 2 : 6 * nt;
            const long long cost = waves * (8000 + 10 * nt + (s > 1 ? 2000 : 0) + (kb + s - 1) / s * block);
            if (least == 0 || cost < least) { least = cost; best = {n_tiles, mt, nt, s}; }
        }
    }
    return best;
}

}  // namespace

// What stays with linear_f32_kernel, whose CTAs start and end sooner: K < 128 (8192 x 64: 100 rows 8.8 us there, 9.3 here, 700 rows
// 25 and 27; from K 128 on 9.0 and 8.7, 41 and 33); a handful of CTAs for more rows than that kernel's tiles need to fill the chip
// (640 x 328: 300 rows 14.1 and 16.2 us with 20 CTAs, 700 rows 18.9 and 16.9 with 50); up to 32 rows, which it has a tile for,
// where more than half and fewer than three quarters of the SMs would hold a tile (17 rows, 10304 x 2048: 51 to 56 and 60 us;
// 2048 x 2048 23 and 17, 16384 x 2048 78 and 66); and what it refuses.  With 34 to 48 tiles up to 32 rows are slower here (4384 x 2048
// 33.3 and 35.4 us, 6144 x 2048 33.3 and 37.2, 4384 x 8192 112 and 121) and stay for their error, a third of the FMAs'.
bool linear_split_takes(const zkfp_linear_args& a)
{
    if (a.K < 128 || (a.M + 63) / 64 > 65535) return false;
    const SplitPlan p = split_plan(a);
    const long long ctas = p.n_tiles * p.m_tiles * p.ksplit, sms = fp_sm_count();
    if (a.M > 128 && ctas * 4 < sms) return false;
    return a.M > 32 || p.n_tiles * 2 <= sms || p.n_tiles * 4 >= 3 * sms;
}

int launch_linear_split(const zkfp_linear_args& a, const LinEpi& e, cudaStream_t st)
{
    const SplitPlan plan = split_plan(a);
    const int nt = plan.nt, ksplit = plan.ksplit;
    const long long n_tiles = plan.n_tiles, m_tiles = plan.m_tiles;
    const size_t stage = 3 * (size_t)(kSplitN + nt) * kSplitK * 2;
    int stages = (int)((kSharedMax - 2048) / stage);
    if (stages > kSplitStages) stages = kSplitStages;
    size_t smem = stage * stages;
    if (smem < (size_t)nt * kSplitPitch * 4) smem = (size_t)nt * kSplitPitch * 4;
    smem += 1024;
    uint32_t cols = 32;
    while (cols < 3u * (uint32_t)nt) cols <<= 1;
    const long long grid = n_tiles * m_tiles * ksplit;
    if (grid > 0x7fffffffll) return ZKDS_ERR_UNSUPPORTED;
    int* flag = fp_error_flag();
    if (!flag) return ZKDS_ERR_WORKSPACE;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kSplitThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)ksplit;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    auto kernel = (kSplitN + nt) * 4 <= 2 * 32 * kSplitWarps ? linear_split_kernel<2> : linear_split_kernel<3>;
    ZKDS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedMax - 1024));
    const cudaError_t rc = cudaLaunchKernelEx(&cfg, kernel, (const float*)a.A, a.lda, (const float*)a.W, a.ldw, (int)a.M, (int)a.N,
                                              (int)a.K, nt, (int)m_tiles, ksplit, stages, cols, flag, e);
    if (rc != cudaSuccess) return set_cuda_error(rc);
    return fp_launched();
}

}  // namespace zkds
