// True 32-bit matrix product on the FP32 pipes (FFMA only; no tensor-core or TF32 mode):
//   C[M,N] = alpha * A[M,K] * W[N,K]^T (+ bias[N])
// A and W are row-major with K contiguous (the layout of activations and of checkpoint weights).
//
// One order of summation for every shape, so that a row's result is bit-identical whatever else is in the batch: K is cut
// into chunks of 64; in a chunk the products at even and at odd k are two chains of fused multiply-adds in the order of k
// (one packed instruction serves both), the chunk's sum is even + odd, the chunks' sums are added in their order over the first
// f32_share(K) chunks and over the others, and the two shares' sums are added. Chunks are what the kernels below spread over threads and
// shares what they spread over blocks: no sum ever waits for K products in a row, and the rounding error is that of chains of 32 and
// K / 128 (up to 1,024 columns, one share: K / 64) instead of one of K.
//
// Up to 16 rows the kernel is bound by the bytes of W (gemm_f32_rows_kernel); beyond, by the FP32 pipes and, where there
// are few tiles, by how many SMs get one (gemm_f32_tile_kernel).
#include "common.cuh"

constexpr int F32_CHUNK = 64;
__host__ __device__ constexpr int f32_share(int K) { return K <= 16 * F32_CHUNK ? 16 : 16 * ((K + 32 * F32_CHUNK - 1) / (32 * F32_CHUNK)); }

__device__ __forceinline__ void f32_cp16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void f32_cp4(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void f32_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void f32_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Four floats row[k .. k+3] to shared memory, zeros past K. VEC: row + k is 16-byte aligned. (A copy of no bytes still names
// an address inside the row.)
template <bool VEC>
__device__ __forceinline__ void f32_cp_piece(uint32_t dst, const float* row, int k, int K) {
    if (VEC) {
        const int left = K - k;
        f32_cp16(dst, row + (left > 0 ? k : 0), left >= 4 ? 16 : left > 0 ? left * 4 : 0);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) f32_cp4(dst + 4 * i, row + (k + i < K ? k + i : 0), k + i < K ? 4 : 0);
    }
}

struct F32Pair { il_f2 lo, hi; };                 // floats k, k+1 and k+2, k+3
__device__ __forceinline__ F32Pair f32_ld4(const float* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return F32Pair{v.x, v.y};
}
__device__ __forceinline__ float f32_halves(il_f2 v) {
    float a, b;
    il_f2_get(v, a, b);
    return __fadd_rn(a, b);
}

// ---- up to 16 rows: W streamed once -------------------------------------------------------------------------------------
// A block owns 8 rows of W. K is taken in rounds of 16 chunks: asynchronous copies bring the round's 32 KB of W (and the rows of
// A) to shared memory, a thread sums one chunk of one W row with all M rows of A, and the chunk sums are added in order.
// The next round's copies are in flight meanwhile, and the first round's W is asked for before the wait for the kernel in
// front where the caller says that W is no kernel's output (`early`). Rows and chunks are padded so that the eight lanes of a load phase hit eight banks groups.
// Measured, one row, weights not in cache: 8,192 x 1,024 in 10.5 us (3.2 TB/s), 73,448 x 1,024 in 76 us (4.0 TB/s); one accumulator
// that walked all of K with plain loads took 740 us on average over a step's products of 1,024 and 4,096 k.
constexpr int FR_ROWS = 8, FR_CHUNKS = 16, FR_ROUND = FR_CHUNKS * F32_CHUNK, FR_CS = F32_CHUNK + 4;
constexpr int FR_WS = FR_CHUNKS * FR_CS + 4, FR_XS = FR_CHUNKS * FR_CS, FR_THREADS = FR_ROWS * FR_CHUNKS;
__host__ __device__ constexpr int fr_stage_floats(int M) { return FR_ROWS * FR_WS + M * FR_XS; }
__host__ __device__ constexpr int fr_smem_floats(int M, int stages) { return stages * fr_stage_floats(M) + M * FR_CHUNKS * FR_ROWS; }

// GLU: W holds N gate rows and then N up rows; a block's 8 rows are 4 gate rows and the 4 up rows that go with them, and the output is
// act(gate) * up as the SwiGLU kernel computes it from the two products (one launch less between a step's products).
template <int MT, bool VEC, bool GLU>
__global__ void __launch_bounds__(FR_THREADS) gemm_f32_rows_kernel(const float* A, int lda, const float* __restrict__ W, int ldw,
                                                                   float* __restrict__ C, int ldc, const float* __restrict__ bias, float alpha,
                                                                   int M, int N, int K, int stages, int early, int act, float limit, float act_alpha) {
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, n0 = blockIdx.x * (GLU ? FR_ROWS / 2 : FR_ROWS);
    const int n = tid & 7, c = tid >> 3;
    const int stage_f = fr_stage_floats(M);
    float* red = sm + (size_t)stages * stage_f;   // [M][FR_CHUNKS][FR_ROWS]
    const int rounds = (K + FR_ROUND - 1) / FR_ROUND;

    auto load_w = [&](int r) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm + (size_t)(r % stages) * stage_f);
#pragma unroll 4
        for (int i = 0; i < FR_ROWS * FR_ROUND / 4 / FR_THREADS; ++i) {
            const int idx = tid + i * FR_THREADS, row = idx / (FR_ROUND / 4), kk = (idx % (FR_ROUND / 4)) * 4;
            // rows past the end are computed and dropped
            const int gn = GLU ? (row < FR_ROWS / 2 ? 0 : N) + min(n0 + row % (FR_ROWS / 2), N - 1) : min(n0 + row, N - 1);
            f32_cp_piece<VEC>(base + 4u * (row * FR_WS + (kk / F32_CHUNK) * FR_CS + kk % F32_CHUNK), W + (size_t)gn * ldw, r * FR_ROUND + kk, K);
        }
    };
    auto load_x = [&](int r) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm + (size_t)(r % stages) * stage_f + FR_ROWS * FR_WS);
        for (int idx = tid; idx < M * (FR_ROUND / 4); idx += FR_THREADS) {
            const int row = idx / (FR_ROUND / 4), kk = (idx % (FR_ROUND / 4)) * 4;
            f32_cp_piece<VEC>(base + 4u * (row * FR_XS + (kk / F32_CHUNK) * FR_CS + kk % F32_CHUNK), A + (size_t)row * lda, r * FR_ROUND + kk, K);
        }
    };
    if (early) load_w(0);
    il_pdl_wait();
    il_pdl_launch_dependents();                   // (the kernel behind may ask for its own weights meanwhile)
    if (!early) load_w(0);
    load_x(0);
    f32_commit();
    if (rounds > 1) load_w(1), load_x(1);
    f32_commit();

    const int on = tid & 7, om = tid >> 3;        // the output this thread adds up (om < M)
    float tot = 0.f, first = 0.f;                 // first: the first share's sum, once it is done (rounds are 16 chunks, shares whole rounds)
    for (int r = 0; r < rounds; ++r) {
        f32_wait<1>();
        __syncthreads();
        const float* st = sm + (size_t)(r % stages) * stage_f;
        const float* w = st + n * FR_WS + c * FR_CS;
        const float* x = st + FR_ROWS * FR_WS + c * FR_CS;
        il_f2 acc[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[m] = 0ull;
#pragma unroll 4
        for (int k = 0; k < F32_CHUNK; k += 4) {
            const F32Pair wv = f32_ld4(w + k);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const F32Pair xv = f32_ld4(x + (m < M ? m : 0) * FR_XS + k);
                acc[m] = il_f2_fma(wv.lo, xv.lo, acc[m]);
                acc[m] = il_f2_fma(wv.hi, xv.hi, acc[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
            if (m < M) red[(m * FR_CHUNKS + c) * FR_ROWS + n] = f32_halves(acc[m]);
        __syncthreads();
        if (r + 2 < rounds) load_w(r + 2), load_x(r + 2);
        f32_commit();
        if (om < M) {
#pragma unroll
            for (int i = 0; i < FR_CHUNKS; ++i) tot = __fadd_rn(tot, red[(om * FR_CHUNKS + i) * FR_ROWS + on]);
        }
        if ((r + 1) * FR_CHUNKS == f32_share(K) && r + 1 < rounds) first = tot, tot = 0.f;
    }
    tot = __fadd_rn(first, tot);
    if constexpr (GLU) {
        const int n = min(n0 + (on & 3), N - 1);
        const float y = __fmaf_rn(alpha, tot, bias ? bias[on < 4 ? n : N + n] : 0.f), up = __shfl_down_sync(0xffffffffu, y, 4);
        if (om < M && on < 4 && n0 + on < N)
            C[(size_t)om * ldc + n0 + on] = act == IL_ACT_CLAMPED ? il_clamped_glu(y, up, limit, act_alpha)
                                            : act == IL_ACT_GELU_TANH ? il_gelu_tanh_mul(y, up) : y / (1.f + expf(-y)) * up;
    } else if (om < M && n0 + on < N) {
        C[(size_t)om * ldc + n0 + on] = __fmaf_rn(alpha, tot, bias ? bias[n0 + on] : 0.f);
    }
}

// ---- more rows: tiles of 32 WM x 32 WN, K dealt out to KG groups of warps ------------------------------------------------------
// Eight warps; a warp holds 32 x 32 outputs (a lane 8 x 4: rows l/8 + 4i, columns l%8 + 8j) of one group's chunks, fed by a ring
// of stages of 16 k for every group, 16-byte asynchronous copies, rows padded to 20 floats (a lane's loads run along k, where the
// packed multiply-adds want their pairs, and no two lanes of a phase share a bank group). With KG > 1 the groups' chunk sums meet in
// shared memory after every round of KG chunks and are added in the order of the chunks. The first share's sums wait for the second's
// in shared memory or, KG 1, where it has no room for them, in C (the same thread's elements, once over the whole of K). SPLIT: two blocks, a cluster, take a share each and the sums meet through their
// shared memory, where the tiles leave SMs idle or alone: 800 rows to 1,024
// columns, K = 4,096, 278 -> 225 us; 61 rows 51 -> 27; 300 rows to 2,048 columns, K = 2,048, 130 -> 115.
constexpr int FT_BK = 16, FT_RS = FT_BK + 4, FT_THREADS = 256;
template <int WM, int WN, int KG> struct FtShape {
    static_assert(WM * WN * KG == 8, "eight warps");
    static constexpr int BM = 32 * WM, BN = 32 * WN, STAGES = KG > 1 ? 3 : 4;
    static constexpr int STAGE = KG * (BM + BN) * FT_RS, RSR = BN + 8;
    static constexpr int SMEM = (STAGES * STAGE + (KG > 1 ? KG * BM * RSR : 0) + BM * BN) * 4;
    static constexpr int BLOCKS = 2 * SMEM <= 224 * 1024 ? 2 : 1;     // an SM's worth: two where both fit
};

__device__ __forceinline__ float f32_peer(uint32_t addr, uint32_t rank) {
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void f32_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// MODE 0: one share; 1: two, one after the other; 2: a cluster's.
template <int WM, int WN, int KG, int MODE, bool VEC>
__global__ void __launch_bounds__(FT_THREADS, FtShape<WM, WN, KG>::BLOCKS) gemm_f32_tile_kernel(const float* A, int lda, const float* __restrict__ W, int ldw,
                                                                   float* C, int ldc, const float* __restrict__ bias, float alpha,
                                                                   int M, int N, int K) {
    using S = FtShape<WM, WN, KG>;
    constexpr bool SPLIT = MODE == 2;
    constexpr int BM = S::BM, BN = S::BN, ST = S::STAGES, GROUP = (BM + BN) * FT_RS;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = warp / (WM * WN), wm = warp % (WM * WN) / WN, wn = warp % WN;
    const int lm = lane >> 3, ln = lane & 7;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    // (shares are whole rounds of KG chunks; a cluster's block z has share z)
    const int k0 = SPLIT ? (int)blockIdx.z * f32_share(K) * F32_CHUNK : 0, k_own = SPLIT && blockIdx.z == 0 ? f32_share(K) * F32_CHUNK : K - k0;
    const int steps = ((k_own + F32_CHUNK * KG - 1) / (F32_CHUNK * KG)) * (F32_CHUNK / FT_BK), share_steps = f32_share(K) / KG * (F32_CHUNK / FT_BK);

    auto load = [&](int s) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm + (size_t)(s % ST) * S::STAGE);
        const int k_round = k0 + (s / (F32_CHUNK / FT_BK)) * KG * F32_CHUNK + (s % (F32_CHUNK / FT_BK)) * FT_BK;
#pragma unroll
        for (int i = 0; i < KG * (BM + BN) * 4 / FT_THREADS; ++i) {
            const int idx = tid + i * FT_THREADS, gg = idx / ((BM + BN) * 4), rem = idx % ((BM + BN) * 4), row = rem >> 2, q = rem & 3;
            const float* src = row < BM ? A + (size_t)min(m0 + row, M - 1) * lda : W + (size_t)min(n0 + row - BM, N - 1) * ldw;
            f32_cp_piece<VEC>(base + 4u * (gg * GROUP + row * FT_RS + q * 4), src, k_round + gg * F32_CHUNK + q * 4, K);
        }
    };
    il_pdl_wait();
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < steps) load(s);
        f32_commit();
    }
    il_f2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    // The sums over chunks. KG 1: this lane's outputs, kept in shared memory (one column a thread) - they are touched once in 64
    // k, and 32 registers fewer let two blocks share an SM. Else outputs tid + 256 i of the tile, in registers.
    constexpr int OUT = BM * BN / FT_THREADS;
    float* red = sm + ST * S::STAGE;              // KG 1: [32][256]; else [KG][BM][RSR]
    float* first = red + KG * BM * S::RSR;        // KG > 1: this thread's sums of the first share
    float tot[KG > 1 ? OUT : 1];
#pragma unroll
    for (int i = 0; i < OUT; ++i) {
        if (KG > 1) tot[KG > 1 ? i : 0] = 0.f;
        else red[i * FT_THREADS + tid] = 0.f;
    }
    for (int s = 0; s < steps; ++s) {
        f32_wait<ST - 2>();
        __syncthreads();
        if (s + ST - 1 < steps) load(s + ST - 1);
        f32_commit();
        const float* st = sm + (size_t)(s % ST) * S::STAGE + g * GROUP;
        const float* ap = st + (wm * 32 + lm) * FT_RS;
        const float* bp = st + (BM + wn * 32 + ln) * FT_RS;
#pragma unroll
        for (int k = 0; k < FT_BK; k += 4) {
            F32Pair b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = f32_ld4(bp + 8 * j * FT_RS + k);
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                const F32Pair a0 = f32_ld4(ap + 4 * i * FT_RS + k), a1 = f32_ld4(ap + 4 * (i + 1) * FT_RS + k);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = il_f2_fma(a0.lo, b[j].lo, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i + 1][j] = il_f2_fma(a1.lo, b[j].lo, acc[i + 1][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = il_f2_fma(a0.hi, b[j].hi, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i + 1][j] = il_f2_fma(a1.hi, b[j].hi, acc[i + 1][j]);
            }
        }
        if (s % (F32_CHUNK / FT_BK) == F32_CHUNK / FT_BK - 1) {       // a chunk is done
            if (KG == 1) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float* t = red + (i * 4 + j) * FT_THREADS + tid;
                        *t = __fadd_rn(*t, f32_halves(acc[i][j]));
                        acc[i][j] = 0ull;
                    }
            } else {
                float* mine = red + ((size_t)g * BM + wm * 32 + lm) * S::RSR + wn * 32 + ln;
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        mine[4 * i * S::RSR + 8 * j] = f32_halves(acc[i][j]);
                        acc[i][j] = 0ull;
                    }
                __syncthreads();
#pragma unroll
                for (int gg = 0; gg < KG; ++gg)
#pragma unroll
                    for (int i = 0; i < OUT; ++i) {
                        const int e = tid + i * FT_THREADS;
                        tot[KG > 1 ? i : 0] = __fadd_rn(tot[KG > 1 ? i : 0], red[((size_t)gg * BM + e / BN) * S::RSR + e % BN]);
                    }
            }
        }
        if (MODE == 1 && s + 1 == share_steps && s + 1 < steps) {
#pragma unroll
            for (int i = 0; i < OUT; ++i) {
                if (KG > 1) {
                    first[i * FT_THREADS + tid] = tot[KG > 1 ? i : 0];
                    tot[KG > 1 ? i : 0] = 0.f;
                } else {
                    const int row = wm * 32 + lm + 4 * (i / 4), col = wn * 32 + ln + 8 * (i % 4);
                    if (m0 + row < M && n0 + col < N) C[(size_t)(m0 + row) * ldc + n0 + col] = red[i * FT_THREADS + tid];
                    red[i * FT_THREADS + tid] = 0.f;
                }
            }
        }
    }
    il_pdl_tail();
    float* mine = KG > 1 ? sm : red;              // SPLIT: this block's sums for the other to read
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(mine + tid);
    if (SPLIT) {
        f32_wait<0>();
        __syncthreads();                          // (the stages are read)
        if (KG > 1) {
#pragma unroll
            for (int i = 0; i < OUT; ++i) mine[i * FT_THREADS + tid] = tot[KG > 1 ? i : 0];
        }
        f32_cluster_sync();
    }
    const bool second = MODE == 1 && steps > share_steps;
#pragma unroll
    for (int i = 0; i < OUT; ++i) {
        if (SPLIT && (i & 1) != (int)blockIdx.z) continue;     // block z stores every second of a thread's outputs
        const int e = tid + i * FT_THREADS;
        const int row = KG == 1 ? wm * 32 + lm + 4 * (i / 4) : e / BN, col = KG == 1 ? wn * 32 + ln + 8 * (i % 4) : e % BN;
        const int gm = m0 + row, gn = n0 + col;
        float v = KG > 1 ? tot[KG > 1 ? i : 0] : red[i * FT_THREADS + tid];
        if (SPLIT) {
            const float other = f32_peer(at + 4u * i * FT_THREADS, blockIdx.z ^ 1);
            v = blockIdx.z ? __fadd_rn(other, v) : __fadd_rn(v, other);
        }
        if (gm < M && gn < N) {
            float* c = C + (size_t)gm * ldc + gn;
            if (second) v = __fadd_rn(KG > 1 ? first[i * FT_THREADS + tid] : *c, v);
            *c = __fmaf_rn(alpha, v, bias ? bias[gn] : 0.f);
        }
    }
    if (SPLIT) f32_cluster_sync();                // (no block leaves while its sums are read)
}

struct F32Args {
    const float *A, *W, *bias;
    float* C;
    int lda, ldw, ldc, M, N, K, early, act;
    float alpha, limit, act_alpha;
    cudaStream_t stream;
};

// Dynamic shared memory beyond 48 KB is asked for once per device and kernel.
static cudaError_t f32_allow_smem(const void* kernel, int bytes, bool* done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (!done[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e == cudaSuccess) done[dev] = true;
    }
    return e;
}

template <int MT, bool VEC, bool GLU> static cudaError_t f32_launch_rows_as(const F32Args& a) {
    static bool done[64];
    const int stages = a.K > FR_ROUND ? 2 : 1;
    cudaError_t e = f32_allow_smem((const void*)gemm_f32_rows_kernel<MT, VEC, GLU>, fr_smem_floats(MT, 2) * 4, done);
    if (e != cudaSuccess) return e;
    constexpr int ROWS = GLU ? FR_ROWS / 2 : FR_ROWS;
    return il_launch(gemm_f32_rows_kernel<MT, VEC, GLU>, dim3((a.N + ROWS - 1) / ROWS), dim3(FR_THREADS), (size_t)fr_smem_floats(a.M, stages) * 4,
                     a.stream, a.A, a.lda, a.W, a.ldw, a.C, a.ldc, a.bias, a.alpha, a.M, a.N, a.K, stages, a.early, a.act, a.limit, a.act_alpha);
}
template <int MT, bool VEC> static cudaError_t f32_launch_rows(const F32Args& a) {
    return a.act ? f32_launch_rows_as<MT, VEC, true>(a) : f32_launch_rows_as<MT, VEC, false>(a);
}

template <int WM, int WN, int KG, int MODE, bool VEC> static cudaError_t f32_launch_tile_as(const F32Args& a) {
    using S = FtShape<WM, WN, KG>;
    static bool done[64];
    const auto kernel = gemm_f32_tile_kernel<WM, WN, KG, MODE, VEC>;
    constexpr bool SPLIT = MODE == 2;
    cudaError_t e = f32_allow_smem((const void*)kernel, S::SMEM, done);
    if (e != cudaSuccess) return e;
    const dim3 grid((a.N + S::BN - 1) / S::BN, (a.M + S::BM - 1) / S::BM, SPLIT ? 2 : 1);
    if (!SPLIT) return il_launch(kernel, grid, dim3(FT_THREADS), (size_t)S::SMEM, a.stream, a.A, a.lda, a.W, a.ldw, a.C, a.ldc, a.bias, a.alpha, a.M, a.N, a.K);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = a.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 2;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = il_pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, a.A, a.lda, a.W, a.ldw, a.C, a.ldc, a.bias, a.alpha, a.M, a.N, a.K);
}
template <int WM, int WN, int KG, bool VEC> static cudaError_t f32_launch_tile(const F32Args& a, bool split) {
    if (split) return f32_launch_tile_as<WM, WN, KG, 2, VEC>(a);
    return a.K > f32_share(a.K) * F32_CHUNK ? f32_launch_tile_as<WM, WN, KG, 1, VEC>(a) : f32_launch_tile_as<WM, WN, KG, 0, VEC>(a);
}

template <bool VEC> static cudaError_t f32_dispatch(const F32Args& a) {
    if (a.M <= 16)
        return a.M == 1 ? f32_launch_rows<1, VEC>(a) : a.M == 2 ? f32_launch_rows<2, VEC>(a) : a.M <= 4 ? f32_launch_rows<4, VEC>(a)
             : a.M <= 8 ? f32_launch_rows<8, VEC>(a) : f32_launch_rows<16, VEC>(a);
    // The tile, and whether K is cut, by what a wave of blocks was measured to take (us for K = 1,024 on a B200): one block on an SM, two on an SM.
    //   128 x 64: 78, 138    64 x 64 (K in 2): 50, 74    64 x 32 (K in 4): 25, 49    32 x 32 (K in 8): 14, 28
    // Large tiles do more work a byte, small ones give more SMs work: 61 rows to 1,024 columns 78 / 42 / 25 / 14 us, 2,048 rows to
    // 8,192 columns 908 / 954 / 1,309 / 1,425 us (37.9 TFLOP/s; one accumulator a product and plain loads took 389 us and 1.7 ms).
    // Cut, there are twice the blocks of half the time and some 5 us a wave for their ends; more than two waves whole are as good.
    const int share = f32_share(a.K) * F32_CHUNK;
    const float whole = (float)a.K / 1024.f, part = (float)share / 1024.f;
    static constexpr int BM[4] = {32, 64, 64, 128}, BN[4] = {32, 32, 64, 64};
    static constexpr float ONE[4] = {14.f, 25.f, 50.f, 78.f}, TWO[4] = {28.f, 49.f, 74.f, 138.f};
    int best = -1;
    float best_us = 0.f;
    for (int cut = 0; cut < (a.K > share ? 2 : 1); ++cut)
        for (int i = 0; i < 4; ++i) {
            const long long tiles = (long long)((a.M + BM[i] - 1) / BM[i]) * ((a.N + BN[i] - 1) / BN[i]), blocks = tiles << cut, rest = blocks % 296;
            if ((cut && tiles > 2 * 296) || (a.M + BM[i] - 1) / BM[i] > 65535) continue;     // (millions of rows: the taller tiles, a grid has 65,535 rows)
            const float waves = (float)(blocks / 296) * TWO[i] + (rest == 0 ? 0.f : rest <= 148 ? ONE[i] : TWO[i]);
            const float us = cut ? waves * part + 5.f * (float)((blocks + 295) / 296) : waves * whole;
            if (best < 0 || us < best_us) best = cut * 4 + i, best_us = us;
        }
    if (best < 0) return cudaErrorInvalidConfiguration;
    const bool split = best >= 4;
    switch (best & 3) {
        case 0: return f32_launch_tile<1, 1, 8, VEC>(a, split);
        case 1: return f32_launch_tile<2, 1, 4, VEC>(a, split);
        case 2: return f32_launch_tile<2, 2, 2, VEC>(a, split);
        default: return f32_launch_tile<4, 2, 1, VEC>(a, split);
    }
}

// act: 0, or the gate of a gated product (M <= 16): W is [2N, K], gate rows, then up rows, bias [2N].
// w_static: W was written long before (a model's weights), not by the kernel in front of this one in the stream.
IL_EXPORT int il_gemm_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc, const float* bias,
                          float alpha, int M, int N, int K, int act, float limit, float act_alpha, int w_static, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return IL_OK;
    if (K <= 0 || lda < K || ldw < K || ldc < N) return IL_BAD_ARG;
    if (act && (M > 16 || act < IL_ACT_SILU || act > IL_ACT_CLAMPED)) return IL_UNSUPPORTED;
    const F32Args a{A, W, bias, C, lda, ldw, ldc, M, N, K, w_static, act, alpha, limit, act_alpha, stream};
    const bool vec = !(lda & 3) && !(ldw & 3) && !((uintptr_t)A & 15) && !((uintptr_t)W & 15);
    const cudaError_t e = vec ? f32_dispatch<true>(a) : f32_dispatch<false>(a);
    if (e != cudaSuccess) return 1000 + (int)e;
    IL_LAUNCH_CHECK();
    return IL_OK;
}
