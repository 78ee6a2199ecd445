// Linear layers of the floating-point decoders: out = epilogue(A W^T) with 32-bit accumulation.
//   few rows (decode)   linear_stream_kernel: every weight is read once, sixteen bytes a lane
//   up to 32, bfloat16  linear_skinny_kernel: the same with warp-level tensor-core products
//   many rows, bfloat16 linear_tc_kernel (float_gemm_tc.cu): tcgen05 tiles fed by TMA
//   many rows, float32  linear_split_kernel (float_gemm_f32.cu): tcgen05 products of bfloat16 thirds; what that leaves,
//                       linear_f32_kernel: 32-bit products on the CUDA cores
#include "float_common.cuh"

namespace zkds {

namespace {

// ---- float32 tiles: BM x 128 x 16, TM x 8 outputs a thread ------------------------------------------------
// Bound by the 128 multiply-adds a clock of an SM's CUDA cores.  Two products an instruction (fma.rn.f32x2, both rounded
// like fmaf) leave the issue slots that fetching operands and doubling the values of A need; tiles are transposed on their
// way into shared memory, with the columns turned by 8 per four k so that neither side of the transposition has conflicts.
// The CTAs of a cluster share the tile's K: each sums its share, then adds up a slice of rows of all of them in a fixed
// order through distributed shared memory, so a split needs no workspace and calls on several streams stay independent.
// 300 rows, against 64 x 64 tiles of single products without a split: 16384 x 2048 480 us (42 TFLOP/s) against 932, 2048 x
// 8192 295 against 918, 2048 x 2048 86 against 235; 17 rows, 2048 x 8192: 96 against 704.
constexpr int kFN = 128, kFK = 16, kFPitch = kFN + 4;

__device__ __forceinline__ float4 peer_float4(uint32_t own, unsigned rank)
{
    float4 v;
    asm volatile("{\n\t.reg .b32 p;\n\tmapa.shared::cluster.u32 p, %4, %5;\n\t"
                 "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [p];\n\t}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(own), "r"(rank) : "memory");
    return v;
}

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

template <int TM>                        // rows a thread: 8 (64-row tiles) or 4 (32-row tiles)
__global__ void __launch_bounds__(128, TM == 8 ? 3 : 4)
linear_f32_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W, long long ldw, int M, int N, int K,
                  int ksplit, const LinEpi e)
{
    constexpr int BM = TM * 8, NA = BM / 32, kStage = kFK * (BM + kFN);
    constexpr int kWords = 2 * kStage > BM * kFPitch ? 2 * kStage : BM * kFPitch;
    __shared__ __align__(16) float sm[kWords];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;   // columns tx * 4 and 64 + tx * 4, rows ty * TM
    const int share = blockIdx.x % ksplit, n0 = blockIdx.x / ksplit * kFN, m0 = blockIdx.y * BM;
    const int per = ((K + kFK - 1) / kFK + ksplit - 1) / ksplit * kFK;
    const int k_begin = share * per, k_end = min(K, k_begin + per);
    const int lrow = tid >> 2, lk = (tid & 3) * 4;               // loader: rows lrow + 32 j, four k
    uint64_t acc[TM][4] = {};
    float4 va[NA], vw[4];
    auto fetch = [&](int k0) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const bool in = k0 + lk < k_end;
#pragma unroll
        for (int j = 0; j < NA; ++j)
            va[j] = in && m0 + lrow + 32 * j < M
                        ? *reinterpret_cast<const float4*>(A + (long long)(m0 + lrow + 32 * j) * lda + k0 + lk) : zero;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            vw[j] = in && n0 + lrow + 32 * j < N
                        ? *reinterpret_cast<const float4*>(W + (long long)(n0 + lrow + 32 * j) * ldw + k0 + lk) : zero;
    };
    auto put = [&](float* s) {
        const int turn = (tid & 3) * 8;
#pragma unroll
        for (int j = 0; j < NA; ++j) {
            float* d = s + lk * BM + ((lrow + 32 * j) ^ turn);
            d[0] = va[j].x; d[BM] = va[j].y; d[2 * BM] = va[j].z; d[3 * BM] = va[j].w;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float* d = s + kFK * BM + lk * kFN + ((lrow + 32 * j) ^ turn);
            d[0] = vw[j].x; d[kFN] = vw[j].y; d[2 * kFN] = vw[j].z; d[3 * kFN] = vw[j].w;
        }
    };
    if (k_begin < k_end) {
        fetch(k_begin);
        put(sm);
        __syncthreads();
        int buf = 0;
        for (int k0 = k_begin; k0 < k_end; k0 += kFK, buf ^= 1) {
            const bool more = k0 + kFK < k_end;
            if (more) fetch(k0 + kFK);
            const float *As = sm + buf * kStage, *Ws = As + kFK * BM;
#pragma unroll
            for (int k = 0; k < kFK; ++k) {
                const int turn = (k >> 2) * 8;
                float a[TM];
#pragma unroll
                for (int i = 0; i < TM; i += 4)
                    *reinterpret_cast<float4*>(a + i) = *reinterpret_cast<const float4*>(As + k * BM + ((ty * TM) ^ turn) + i);
                const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(Ws + k * kFN + ((tx * 4) ^ turn));
                const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(Ws + k * kFN + 64 + ((tx * 4) ^ turn));
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const uint64_t aa = twice(a[i]);
                    fma2(acc[i][0], aa, w0.x); fma2(acc[i][1], aa, w0.y);
                    fma2(acc[i][2], aa, w1.x); fma2(acc[i][3], aa, w1.y);
                }
            }
            if (more) put(sm + (buf ^ 1) * kStage);
            __syncthreads();
        }
    }
    // the sums through shared memory, so that eight columns of a row come together and peers can read them
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        float* d = sm + (ty * TM + i) * kFPitch + tx * 4;
        *reinterpret_cast<ulonglong2*>(d) = make_ulonglong2(acc[i][0], acc[i][1]);
        *reinterpret_cast<ulonglong2*>(d + 64) = make_ulonglong2(acc[i][2], acc[i][3]);
    }
    if (ksplit > 1) cluster_barrier();
    else __syncthreads();
    const int rows = BM / ksplit;
    for (int it = tid; it < rows * (kFN / 8); it += 128) {
        const int r = share * rows + it / (kFN / 8), c = it % (kFN / 8) * 8, m = m0 + r, n = n0 + c;
        if (m >= M || n >= N) continue;
        const float* own = sm + r * kFPitch + c;
        float v[8];
        if (ksplit == 1) {
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(own);
            *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(own + 4);
        } else {
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(own);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = 0.f;
            for (int s = 0; s < ksplit; ++s) {
                const float4 x = peer_float4(at, s), y = peer_float4(at + 16, s);
                v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
                v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
            }
        }
        epilogue8(e, e.kind == ZKFP_EPI_ROTATE ? epi_position(e, m) : 0, m, n, v);
    }
    if (ksplit > 1) cluster_barrier();      // a peer may still be reading this block's sums
}

// ---- weight streaming ---------------------------------------------------------------------------------------
// A warp accumulates eight weight rows against MT activation rows over its share of K; `ksplit` warps of the
// block share the eight rows.  The butterfly leaves column (lane >> 2) of a token's eight sums in its lane.
__device__ __forceinline__ float reduce8(float (&v)[8], int lane)
{
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool up = lane & 16;
        const float send = up ? v[i] : v[i + 4], keep = up ? v[i + 4] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const bool up = lane & 8;
        const float send = up ? v[i] : v[i + 2], keep = up ? v[i + 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    const bool up = lane & 4;
    const float send = up ? v[0] : v[1], keep = up ? v[1] : v[0];
    float s = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

template <typename T, int MT>
__global__ void __launch_bounds__(256)
linear_stream_kernel(const T* A, long long lda, const T* W, long long ldw, int M, int N, int K, int ksplit, int early,
                     const LinEpi e)
{
    __shared__ float part[8][MT][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = 8 / ksplit, ks = warp % ksplit;
    const int n = (blockIdx.x * groups + warp / ksplit) * 8;
    const int m0 = blockIdx.y * MT;
    if (early && n < N) {            // this warp's first weights on their way into L2 while the kernel in front ends
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int k = (ks + u * ksplit) * 256 + lane * 8;
            if (k < K && (lane * 8 * (int)sizeof(T)) % 128 == 0) {
#pragma unroll
                for (int r = 0; r < 8; ++r)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (long long)(n + r) * ldw + k) : "memory");
            }
        }
    }
    chain_enter();
    float acc[MT][8] = {};
    if (n < N) {
        const T* w = W + (long long)n * ldw;
        const T* a = A + (long long)m0 * lda;
        const int step = 256 * ksplit;
#pragma unroll 2
        for (int k = ks * 256 + lane * 8; k < K; k += step) {
            float x[MT][8];
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                if (m0 + t < M) load8(a + t * lda + k, x[t]);
                else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[t][i] = 0.f;
                }
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                float v[8];
                load8(w + r * ldw + k, v);
#pragma unroll
                for (int t = 0; t < MT; ++t)
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[t][r] = fmaf(v[i], x[t][i], acc[t][r]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < MT; ++t) {
        const float s = reduce8(acc[t], lane);
        if ((lane & 3) == 0) part[warp][t][lane >> 2] = s;
    }
    __syncthreads();
    if (threadIdx.x < groups * MT) {
        const int g = threadIdx.x / MT, t = threadIdx.x % MT;
        const int ng = (blockIdx.x * groups + g) * 8, m = m0 + t;
        if (ng < N && m < M) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = 0.f;
                for (int s = 0; s < ksplit; ++s) v[i] += part[g * ksplit + s][t][i];
            }
            epilogue8(e, e.kind == ZKFP_EPI_ROTATE ? epi_position(e, m) : 0, m, ng, v);
        }
    }
}

// ---- few rows, bfloat16: weights streamed through warp-level tensor-core products -----------------------------------
// out^T = W A^T in 16 x 8 x 16 products: a warp owns sixteen weight rows, the rows of A are the eight columns of a
// product.  The order of K inside a product is free as long as both operands agree, so a lane takes eight consecutive k
// of its row (one 16-byte load) as the fragments of two products: no shared memory and no shuffles on the way in.
// Bound by the bytes of the weights; a warp keeps two blocks of 128 k (4 KB each) in flight.  4 rows, against the tcgen05
// tiles that these sizes took before (split sums, a start of 18 us): 4096 x 4096 9.8 us against 23.1, 10304 x 2048 13.1
// against 18.8, 28672 x 4096 46 (5.1 TB/s) against 68, 36864 x 7168 86 (6.1 TB/s) against 119.
__device__ __forceinline__ uint4 stream16(const bf16* p)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int kSkinnyRows = 32;
constexpr int kSkinnyK = 128;            // k of a block: four 16-byte loads a lane and weight row

template <int NT>                        // tiles of eight rows of A
__global__ void __launch_bounds__(256, NT <= 2 ? 2 : 1)
linear_skinny_kernel(const bf16* A, long long lda, const bf16* W, long long ldw, int M, int N, int K, int ksplit, int early,
                     const LinEpi e)
{
    if (!early) chain_enter();
    __shared__ float part[8][16][NT * 8 + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int groups = 8 / ksplit, ks = warp % ksplit;
    const int n0 = (blockIdx.x * groups + warp / ksplit) * 16;
    float acc[NT][4] = {}, sum[NT][4] = {};
    if (n0 < N) {
        // rows beyond the last are read as the last one; what they give is not stored
        const bf16 *w0 = W + (long long)min(n0 + g, N - 1) * ldw + t * 8, *w1 = W + (long long)min(n0 + g + 8, N - 1) * ldw + t * 8;
        const bf16* a[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) a[j] = A + (long long)min(j * 8 + g, M - 1) * lda + t * 8;
        const uint4 zero = make_uint4(0, 0, 0, 0);
        uint4 cur[2][4], nxt[2][4];
        auto fetch = [&](uint4 (&v)[2][4], int k) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = k + u * 32 + t * 8 < K;
                v[0][u] = in ? stream16(w0 + k + u * 32) : zero;
                v[1][u] = in ? stream16(w1 + k + u * 32) : zero;
            }
        };
        const int step = ksplit * kSkinnyK;
        int k = ks * kSkinnyK;
        if (k < K) fetch(cur, k);
        if (early) chain_enter();        // its first weights are on their way while the kernel in front ends
        for (; k < K; k += step) {
            if (k + step < K) fetch(nxt, k + step);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = k + u * 32 + t * 8 < K;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const uint4 x = in ? *reinterpret_cast<const uint4*>(a[j] + k + u * 32) : zero;
                    mma_16816(acc[j], cur[0][u].x, cur[1][u].x, cur[0][u].y, cur[1][u].y, x.x, x.y);
                    mma_16816(acc[j], cur[0][u].z, cur[1][u].z, cur[0][u].w, cur[1][u].w, x.z, x.w);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) { cur[0][u] = nxt[0][u]; cur[1][u] = nxt[1][u]; }
            // fresh accumulators for every block of 128 k: a product's own additions are cut off rather than rounded
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    sum[j][i] += acc[j][i];
                    acc[j][i] = 0.f;
                }
        }
    } else if (early) chain_enter();
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) part[warp][g + (i >> 1) * 8][j * 8 + t * 2 + (i & 1)] = sum[j][i];
    __syncthreads();
    // eight columns of one row an item, the shares of K added in a fixed order
    for (int it = threadIdx.x; it < groups * 2 * M; it += 256) {
        const int m = it % M, o = it / M, grp = o >> 1, n = (blockIdx.x * groups + grp) * 16 + (o & 1) * 8;
        if (n >= N) continue;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[i] = 0.f;
            for (int s = 0; s < ksplit; ++s) v[i] += part[grp * ksplit + s][(o & 1) * 8 + i][m];
        }
        epilogue8(e, e.kind == ZKFP_EPI_ROTATE ? epi_position(e, m) : 0, m, n, v);
    }
}

template <typename T>
int linear_stream(const zkfp_linear_args& a, const LinEpi& e, bool early, cudaStream_t st)
{
    int ksplit = 1;
    while (ksplit < 8 && (long long)ksplit * 512 < a.K) ksplit *= 2;
    // narrow outputs: more warps on the same rows until every SM has work
    while (ksplit < 8 && a.N / 8 * ksplit < 8LL * fp_sm_count() && ksplit * 256 < a.K) ksplit *= 2;
    const int groups = 8 / ksplit;
    const unsigned gx = (unsigned)((a.N / 8 + groups - 1) / groups);
    const T *A = (const T*)a.A, *W = (const T*)a.W;
    const int M = (int)a.M, N = (int)a.N, K = (int)a.K;
    if (M == 1) fp_launch(linear_stream_kernel<T, 1>, dim3(gx, 1), dim3(256), 0, st, A, a.lda, W, a.ldw, M, N, K, ksplit, early, e);
    else if (M == 2) fp_launch(linear_stream_kernel<T, 2>, dim3(gx, 1), dim3(256), 0, st, A, a.lda, W, a.ldw, M, N, K, ksplit, early, e);
    else fp_launch(linear_stream_kernel<T, 4>, dim3(gx, (M + 3) / 4), dim3(256), 0, st, A, a.lda, W, a.ldw, M, N, K, ksplit, early, e);
    return fp_launched();
}

}  // namespace

bool linear_skinny_takes(const zkfp_linear_args& a)
{
    // Up to eight rows always.  Beyond, every eight rows cost a product and a load of A per sixteen bytes of weights, and
    // the tcgen05 tiles win once the weights are large enough to hide their start and split sums (16 rows: 7168 x 18432
    // 60 against 65 us, 36864 x 7168 104 against 96; 32 rows: 2048 x 8192 20 against 30, 10304 x 2048 26 against 19).  Beyond
    // 8192 columns the tiles fill the SMs without a split and win sooner (32 rows: 16384 x 512 13.3 against 13.5, 12288 x 1024
    // 18.7 against 15.6, 65536 x 256 28.2 against 23.8).
    const long long weights = a.N * a.K;
    return a.M <= 8 || (a.M <= 16 && weights <= 140000000) ||
           (a.M <= kSkinnyRows && weights <= (a.N <= 8192 ? 20000000 : 10000000));
}

int launch_linear_skinny(const zkfp_linear_args& a, const LinEpi& e, bool early, cudaStream_t st)
{
    // warps on the same rows until every SM has a block.  More of them leave a last wave that is nearly empty and cost
    // more reductions (16384 x 2048, 4 rows: 2 shares 15.5 us, 4: 17.5, 8: 20.5), fewer leave SMs idle (4096 x 4096:
    // 8 shares 10.3 us, 4: 12.8, 2: 18.4)
    const long long tiles = (a.N + 15) / 16;
    int ksplit = 1;
    while (ksplit < 8 && tiles * ksplit < 8LL * fp_sm_count() && (long long)ksplit * kSkinnyK < a.K) ksplit *= 2;
    const int groups = 8 / ksplit;
    const unsigned grid = (unsigned)((tiles + groups - 1) / groups);
    const bf16 *A = (const bf16*)a.A, *W = (const bf16*)a.W;
    const int M = (int)a.M, N = (int)a.N, K = (int)a.K;
    if (M <= 8) fp_launch(linear_skinny_kernel<1>, dim3(grid), dim3(256), 0, st, A, a.lda, W, a.ldw, M, N, K, ksplit, early, e);
    else if (M <= 16) fp_launch(linear_skinny_kernel<2>, dim3(grid), dim3(256), 0, st, A, a.lda, W, a.ldw, M, N, K, ksplit, early, e);
    else if (M <= kSkinnyRows) fp_launch(linear_skinny_kernel<4>, dim3(grid), dim3(256), 0, st, A, a.lda, W, a.ldw, M, N, K, ksplit, early, e);
    else return ZKDS_ERR_UNSUPPORTED;
    return fp_launched();
}

int launch_linear_f32(const zkfp_linear_args& a, const LinEpi& e, cudaStream_t st)
{
    // 32-row tiles for the rows that would leave half of a 64-row tile empty, while there are few tiles of rows, and for a K
    // that is too shallow to be shared, where a CTA's start and end are the time (64 x 2048, K = 16: 4.9 us, in
    // 64-row tiles 6.9)
    const bool small = a.M <= 32 || (a.M > 64 && a.M <= 96) ||
                       (a.K <= 128 && (a.M + 63) / 64 * ((a.N + kFN - 1) / kFN) <= fp_sm_count());
    const long long bm = small ? 32 : 64, kb = (a.K + kFK - 1) / kFK;
    const long long tiles = (a.M + bm - 1) / bm * ((a.N + kFN - 1) / kFN);
    // shares of K: the fewest blocks of K that an SM works through one after the other, with 6 more for a CTA's start and
    // its part of the sums.  One or two CTAs on an SM cannot keep its units busy.
    int ksplit = 1;
    long long best = 0;
    for (int s = 1; s <= 8; s *= 2) {
        if (s > 1 && kb / s < 4) break;
        const long long each = (tiles * s + fp_sm_count() - 1) / fp_sm_count();
        const long long cost = each * ((kb + s - 1) / s + 6) * (each == 1 ? 20 : each == 2 ? 13 : 10);
        if (s == 1 || cost < best) { best = cost; ksplit = s; }
    }
    const long long gx = (a.N + kFN - 1) / kFN * ksplit, gy = (a.M + bm - 1) / bm;
    if (gx > 0x7fffffffll || gy > 65535) return ZKDS_ERR_UNSUPPORTED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)gx, (unsigned)gy);
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)ksplit;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const float *A = (const float*)a.A, *W = (const float*)a.W;
    const int M = (int)a.M, N = (int)a.N, K = (int)a.K;
    const cudaError_t rc = small ? cudaLaunchKernelEx(&cfg, linear_f32_kernel<4>, A, a.lda, W, a.ldw, M, N, K, ksplit, e)
                                 : cudaLaunchKernelEx(&cfg, linear_f32_kernel<8>, A, a.lda, W, a.ldw, M, N, K, ksplit, e);
    if (rc != cudaSuccess) return set_cuda_error(rc);
    return fp_launched();
}

int launch_linear_stream(const zkfp_linear_args& a, const LinEpi& e, bool early, cudaStream_t st)
{
    return a.dtype == ZKFP_BF16 ? linear_stream<bf16>(a, e, early, st) : linear_stream<float>(a, e, early, st);
}

}  // namespace zkds
