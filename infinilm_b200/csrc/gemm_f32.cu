// 32-bit matrix product on the bfloat16 tensor cores, with the error of 32-bit multiply-adds:
//   C[M,N] = alpha * A[M,K] * W[N,K]^T (+ bias[N])
// A and W are float32, row-major with K contiguous (the layout of activations and of checkpoint weights); nothing is stored in
// fewer bits. Each operand is taken apart on its way to the tensor cores, 2^23 x = h + m + l with h, m, l the bfloat16 nearest to 2^23 x,
// to what h leaves and to what m leaves: 24 bits, exactly 2^23 x for every finite x below 2^105, the smallest ones too (the last bit of a
// float32 is 2^-149 or more, that of l then 2^-126, the least bfloat16 that is not subnormal; without the factor, numbers below 2^-102
// lost bits, which a large number on the other side made visible). Products of two
// bfloat16 are exact in the tensor core; of the nine, three are below 2^-26 of the first and are left out.
//
// One order of summation for every kernel and shape, so that a row's result is bit-identical whatever else is in the batch:
//   - of a chunk of 64 k: the h h products of its first 32 k and of its last 32 k, two tensor-core instructions each from zero
//     (the tensor core cuts a sum off at 24 bits, towards zero, after each instruction: short sums keep that small), and the small
//     products, twenty instructions in a third accumulator (their cuts are 2^-8 of the others); (first + last) + small in float32;
//   - of a share, a half to an eighth of K's chunks (f32_shares): the chunks in order; of K: the shares in order.
// mma.sync and tcgen05.mma give the same bits for the same operands (512 x 128 x 48 sums of 24 instructions, five
// distributions: all equal); the tests compare the two kernels below row by row.
// Error against float64, norm of the difference over norm of the result, here and in 32-bit multiply-adds in chunks of 64 (the
// kernel before), K = 1,024 and 4,096: normal operands 0.79e-7 (1.31e-7) and 0.96e-7 (1.53e-7); normal times 2^-12 .. 2^12
// 0.98e-7 (1.10e-7) and 1.12e-7 (1.35e-7); all positive 0.55e-7 (0.61e-7) and 0.59e-7 (0.65e-7). With the h h products of a whole
// chunk in one accumulator: 1.03e-7, 1.36e-7 and 0.88e-7 at K = 1,024.
//
// A sum that is not finite may owe that to the pieces (an infinity has no remainder) or to the factor 2^46 (sums of 2^82 and more): it is
// computed again with 32-bit multiply-adds, in the same chunks (f32_plain).
//
// Up to 16 rows the kernel is bound by the bytes of W and by the instructions that take it apart (gemm_f32_rows_kernel,
// mma.sync on fragments that come straight from memory); beyond, by those instructions and by shared memory, where the pieces are written
// and read by the tensor core (gemm_f32_tile_kernel, tcgen05).
#include "tcgen05.cuh"

constexpr int F32_CHUNK = 64;
__host__ __device__ constexpr int f32_chunks(int K) { return (K + F32_CHUNK - 1) / F32_CHUNK; }
__host__ __device__ constexpr int f32_shares(int K) { return K <= 256 ? 1 : K <= 512 ? 2 : K <= 1024 ? 4 : 8; }
__host__ __device__ constexpr int f32_share_chunks(int K) { return (f32_chunks(K) + f32_shares(K) - 1) / f32_shares(K); }

// Two numbers taken apart, the pieces of a in the low halves: three conversions, two packed subtractions and four to widen. (Rounding
// by Veltkamp's splitting, or in the bit pattern, takes the conversions' place with more instructions: 2,048 x 8,192 x 1,024 in 540 and
// 740 us where the conversions took 370.)
__device__ __forceinline__ uint32_t f32_pack(float a, float b) {
    uint32_t v;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(v) : "f"(b), "f"(a));
    return v;
}
__device__ __forceinline__ il_f2 f32_less(il_f2 x, uint32_t p) {      // x minus the two bfloat16 of p
    il_f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(x), "l"(il_f2_make(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u))));
    return d;
}
constexpr float F32_SCALE = 0x1p23f, F32_UNSCALE = 0x1p-46f;          // of an operand; of a sum
// (FUSED: the same pieces, the factor once more in the first subtraction instead of a scaled pair held for it - for the kernel that is short of registers,
// 16 rows to 73,448 columns of K = 1,024: 111 us, 116 without; elsewhere it costs up to 2 %.)
template <bool FUSED = false>
__device__ __forceinline__ void f32_split(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    il_f2 r;
    if (FUSED) {
        h = f32_pack(a * F32_SCALE, b * F32_SCALE);
        r = il_f2_fma(il_f2_make(a, b), il_f2_dup(F32_SCALE), il_f2_make(__uint_as_float((h << 16) ^ 0x80000000u), __uint_as_float((h & 0xffff0000u) ^ 0x80000000u)));
    } else {
        r = il_f2_mul(il_f2_make(a, b), il_f2_dup(F32_SCALE));
        il_f2_get(r, a, b);
        h = f32_pack(a, b);
        r = f32_less(r, h);
    }
    il_f2_get(r, a, b);
    m = f32_pack(a, b);
    r = f32_less(r, m);
    il_f2_get(r, a, b);
    l = f32_pack(a, b);
}
__device__ __forceinline__ bool f32_suspect(float v) { return !(fabsf(v) < INFINITY); }
// The sum by multiply-adds: even and odd k apart, chunk by chunk.
__device__ __noinline__ float f32_plain(const float* a, const float* w, int K) {
    float sum = 0.f;
    for (int c = 0; c < K; c += F32_CHUNK) {
        float even = 0.f, odd = 0.f;
        const int end = min(K, c + F32_CHUNK);
        int k = c;
        for (; k + 1 < end; k += 2) even = __fmaf_rn(a[k], w[k], even), odd = __fmaf_rn(a[k + 1], w[k + 1], odd);
        if (k < end) even = __fmaf_rn(a[k], w[k], even);
        sum = __fadd_rn(sum, __fadd_rn(even, odd));
    }
    return sum;
}
// Four floats row[k .. k+3], zeros past K. VEC: row + k is 16-byte aligned.
__device__ __forceinline__ float4 f32_ld4(const float* p) {
    float4 v;
    asm volatile("ld.global.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
template <bool VEC>
__device__ __forceinline__ float4 f32_ld(const float* row, int k, int K) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (VEC && k + 4 <= K) {
        v = f32_ld4(row + k);
    } else {
        if (k < K) v.x = row[k];
        if (k + 1 < K) v.y = row[k + 1];
        if (k + 2 < K) v.z = row[k + 2];
        if (k + 3 < K) v.w = row[k + 3];
    }
    return v;
}
__device__ __forceinline__ void f32_put(float* p, uint32_t rank, float v) {     // to the same place of another block of the cluster
    uint32_t at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(at), "f"(v) : "memory");
}
__device__ __forceinline__ float4 f32_peer4(uint32_t addr, uint32_t rank) {
    uint32_t at;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

// ---- up to 16 rows: W streamed once -------------------------------------------------------------------------------------
// A block owns tiles of 16 rows of W (the A operand of m16n8k16; lane l holds k 4 (l % 4) .. + 3 of every 16 for rows l / 4 and
// l / 4 + 8, one 16-byte load each; the rows of A, the B operand, in the same order: up to 4 rows are taken apart once a block into shared
// memory (once for all its tiles where K has up to two rounds), more by every warp as it goes, which has fewer instructions then). K is taken in rounds of 8
// chunks, a chunk a warp; a warp has the weights of two rounds in registers or on their way, across tiles, the first two asked
// for before the wait for the kernel in front where the caller says that W is no kernel's output (`early`). Where the tiles are
// few, the shares go to the blocks of a cluster.
// Measured, weights not in cache, us (the kernel of multiply-adds before): one row, 2 x 4,096 gated columns of K = 1,024 9.6 (10.5), 73,448
// columns 58.8 (71; 5.1 TB/s), 1,024 columns of K = 4,096 6.6 (6.0), of K = 1,024 3.3 (2.3); 8 rows to 73,448 columns 64 (87), K = 4,096 7.1 (9.9); 16 rows
// 14.4 (22.8), 111 (156), K = 1,024 3.9 (5.2). 371 instructions a warp for 4 KB of W (counted by the profiler) bound the small ones. Without the factor 2^23:
// 9.5, 56.5, 6.4, 3.1; 63.6, 6.8; 13.7, 100, 3.6.
constexpr int FR_WARPS = 8, FR_THREADS = FR_WARPS * 32, FR_TILE = 16, FR_ROUND = FR_WARPS * F32_CHUNK;
// shared memory: a round's chunk sums; the shares' sums; two rounds of A's pieces, [16 k][piece][lane] 8 bytes
constexpr int FR_X = FR_ROUND / 16 * 3 * 256;
__host__ __device__ constexpr int fr_smem(int NT, bool STAGE, int rounds) { return (FR_WARPS + 8) * FR_TILE * NT * 8 * 4 + (!STAGE ? 0 : rounds > 1 ? 2 * FR_X : FR_X); }

__device__ __forceinline__ void f32_mma(float (&d)[4], const uint32_t (&a)[4], uint2 b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}

// NT: groups of 8 rows of A; STAGE: taken apart in shared memory. GLU: W holds N gate rows and then N up rows; a tile's 16 rows are 8 gate rows and the 8 up rows that go with
// them, and the output is act(gate) * up as the SwiGLU kernel computes it from the two products (one launch less between a step's products).
template <int NT, bool STAGE, bool VEC, bool GLU>
__global__ void __launch_bounds__(FR_THREADS, 2) gemm_f32_rows_kernel(const float* A, int lda, const float* W, int ldw,
                                                                      float* C, int ldc, const float* bias, float alpha,
                                                                      int M, int N, int K, int tiles, int cluster, int early, int act, float limit, float act_alpha) {
    constexpr int OUT = FR_TILE * NT * 8;         // outputs of a tile: [row of W, of the first eight][which eight][row of A]; thread e adds up output e
    extern __shared__ __align__(16) unsigned char fr_sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int rank = blockIdx.x % cluster, first = blockIdx.x / cluster, stride = gridDim.x / cluster;
    const int share_chunks = f32_share_chunks(K), own_shares = f32_shares(K) / cluster;
    const int c_lo = rank * own_shares * share_chunks, c_hi = min(f32_chunks(K), c_lo + own_shares * share_chunks);
    const int rounds = max(1, (c_hi - c_lo + FR_WARPS - 1) / FR_WARPS), mine = first < tiles ? (tiles - first + stride - 1) / stride : 0;
    const int total = mine * rounds;
    float* red = reinterpret_cast<float*>(fr_sm); // a round's chunk sums
    float* part = red + FR_WARPS * OUT;           // the shares' sums
    unsigned char* x_sm = fr_sm + (FR_WARPS + 8) * OUT * 4;

    // round i of this block: tile first + (i / rounds) * stride, chunk c_lo + (i % rounds) * 8 + warp
    float4 w[2][8];
    int ld_tile = first, ld_round = 0;
    auto load_w = [&](float4 (&v)[8]) {
        const int c = c_lo + ld_round * FR_WARPS + warp;
        const int n0 = ld_tile * (GLU ? FR_TILE / 2 : FR_TILE);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int n = GLU ? (half ? N : 0) + min(n0 + g, N - 1) : min(n0 + g + 8 * half, N - 1);     // rows past the end are computed and dropped
            const float* row = W + (size_t)n * ldw;
            if (VEC && c < c_hi && (c + 1) * F32_CHUNK <= K) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) v[half * 4 + kk] = f32_ld4(row + c * F32_CHUNK + kk * 16 + t * 4);
            } else {
                const int k_end = c < c_hi ? K : 0;               // (a chunk past the end: zeros)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) v[half * 4 + kk] = f32_ld<VEC>(row, c * F32_CHUNK + kk * 16 + t * 4, k_end);
            }
        }
        if (++ld_round == rounds) ld_round = 0, ld_tile += stride;
    };
    if (early) {
        if (0 < total) load_w(w[0]);
        if (1 < total) load_w(w[1]);
    }
    if (cluster > 1) il_cluster_arrive();        // (waited for before the first access to another block's memory)
    il_pdl_wait();
    il_pdl_launch_dependents();                   // (the kernel behind may ask for its own weights meanwhile)
    if (!early) {
        if (0 < total) load_w(w[0]);
        if (1 < total) load_w(w[1]);
    }
    // (columns of the product whose rows of A are not there come out as anything and are dropped)
    auto stage_x = [&](int r) {
        uint2* to = reinterpret_cast<uint2*>(x_sm + (r & 1) * FR_X);
        const int k0 = (c_lo + r * FR_WARPS) * F32_CHUNK, k_end = min(K, c_hi * F32_CHUNK);
        for (int i = tid; i < M * (FR_ROUND / 4); i += FR_THREADS) {
            const int m = i / (FR_ROUND / 4), q = i % (FR_ROUND / 4);
            const float* row = A + (size_t)m * lda;
            const float4 v = VEC && k0 + q * 4 + 4 <= k_end ? *reinterpret_cast<const float4*>(row + k0 + q * 4) : f32_ld<false>(row, k0 + q * 4, k_end);
            uint2 h, m1, l;
            f32_split(v.x, v.y, h.x, m1.x, l.x);
            f32_split(v.z, v.w, h.y, m1.y, l.y);
            uint2* at = to + (q >> 2) * 3 * 32 + m * 4 + (q & 3);
            at[0] = h, at[32] = m1, at[64] = l;
        }
    };
    if (STAGE) {
        if (total > 0) stage_x(0);
        if (total > 0 && rounds > 1) stage_x(1);
        __syncthreads();
    }
    const float* xrow[NT];                        // (rows past the end are the last one: computed and dropped)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) xrow[nt] = A + (size_t)min(g + 8 * nt, M - 1) * lda;

    int tile = first, r = 0, cs = 0, share = 0;   // cs: chunks of the running share so far
    float cur = 0.f;
    auto round = [&](float4 (&v)[8], int i) {
        const uint2* xs = reinterpret_cast<const uint2*>(x_sm + (r & 1) * FR_X) + warp * 4 * 3 * 32 + lane;
        const int c = c_lo + r * FR_WARPS + warp, k0 = c * F32_CHUNK + t * 4;
        const bool whole = VEC && c < c_hi && (c + 1) * F32_CHUNK <= K;
        float4 x[NT];
        auto load_x = [&](int kk) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
                x[nt] = whole ? *reinterpret_cast<const float4*>(xrow[nt] + k0 + kk * 16) : f32_ld<false>(xrow[nt], k0 + kk * 16, c < c_hi ? K : 0);
        };
        if (!STAGE) load_x(0);
        float s[NT][4], e[NT][4], d[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) e[nt][0] = e[nt][1] = e[nt][2] = e[nt][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            uint2 xh[NT], xm[NT], xl[NT];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                if (STAGE) {
                    xh[nt] = xs[kk * 96], xm[nt] = xs[kk * 96 + 32], xl[nt] = xs[kk * 96 + 64];
                } else {
                    f32_split<NT == 2>(x[nt].x, x[nt].y, xh[nt].x, xm[nt].x, xl[nt].x);
                    f32_split<NT == 2>(x[nt].z, x[nt].w, xh[nt].y, xm[nt].y, xl[nt].y);
                }
            }
            if (!STAGE && kk < 3) load_x(kk + 1);
            uint32_t h[4], m[4], l[4];
            f32_split<NT == 2>(v[kk].x, v[kk].y, h[0], m[0], l[0]);
            f32_split<NT == 2>(v[4 + kk].x, v[4 + kk].y, h[1], m[1], l[1]);
            f32_split<NT == 2>(v[kk].z, v[kk].w, h[2], m[2], l[2]);
            f32_split<NT == 2>(v[4 + kk].z, v[4 + kk].w, h[3], m[3], l[3]);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                f32_mma(e[nt], l, xh[nt]);
                f32_mma(e[nt], h, xl[nt]);
                f32_mma(e[nt], m, xm[nt]);
                f32_mma(e[nt], m, xh[nt]);
                f32_mma(e[nt], h, xm[nt]);
                if (!(kk & 1)) d[nt][0] = d[nt][1] = d[nt][2] = d[nt][3] = 0.f;
                f32_mma(d[nt], h, xh[nt]);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (kk & 1) s[nt][j] = kk == 1 ? d[nt][j] : __fadd_rn(s[nt][j], d[nt][j]);
            }
        }
        if (i + 2 < total) load_w(v);
        if (i > 0) __syncthreads();               // (the round before is added up)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int half = 0; half < 2; ++half)
                *reinterpret_cast<float2*>(red + warp * OUT + (g * 2 + half) * (NT * 8) + nt * 8 + t * 2) =
                    make_float2(__fadd_rn(s[nt][2 * half], e[nt][2 * half]), __fadd_rn(s[nt][2 * half + 1], e[nt][2 * half + 1]));
        __syncthreads();
        if (tid < OUT) {
            const int live = min(FR_WARPS, c_hi - c_lo - r * FR_WARPS);
            float in[FR_WARPS];
#pragma unroll
            for (int c = 0; c < FR_WARPS; ++c) in[c] = red[c * OUT + tid];
            if (share_chunks == FR_WARPS && live == FR_WARPS) {       // a round is a share
#pragma unroll
                for (int c = 1; c < FR_WARPS; ++c) in[0] = __fadd_rn(in[0], in[c]);
                part[share++ * OUT + tid] = in[0];
            } else if (2 * share_chunks == FR_WARPS && live == FR_WARPS) {      // two
                part[share++ * OUT + tid] = __fadd_rn(__fadd_rn(__fadd_rn(in[0], in[1]), in[2]), in[3]);
                part[share++ * OUT + tid] = __fadd_rn(__fadd_rn(__fadd_rn(in[4], in[5]), in[6]), in[7]);
            } else {
#pragma unroll
                for (int c = 0; c < FR_WARPS; ++c)
                    if (c < live) {
                        cur = cs == 0 ? in[c] : __fadd_rn(cur, in[c]);
                        if (++cs == share_chunks) part[share * OUT + tid] = cur, cs = 0, ++share;
                    }
            }
        }
        if (STAGE && r + 2 < rounds) stage_x(r + 2);       // (up to two rounds: x stays)
        ++r;
    };
    for (int i = 0; i < total; ++i) {
        if (i & 1) round(w[1], i); else round(w[0], i);
        if (r < rounds) continue;
        // ---- the tile is done ----
        if (tid < OUT && cs) part[share * OUT + tid] = cur, ++share;      // (a last share of fewer chunks)
        const int half = tid / (NT * 8) & 1, row = tid / (NT * 16), m = tid % (NT * 8);
        float v = 0.f;
        if (cluster > 1) {                        // (one tile a cluster)
            il_cluster_wait();
            if (rank > 0 && tid < OUT)
                for (int sh = 0; sh < share; ++sh) f32_put(part + (rank * own_shares + sh) * OUT + tid, 0, part[sh * OUT + tid]);
            il_cluster_sync();
        }
        if (rank == 0 && tid < OUT) {
            const int all = (f32_chunks(K) + share_chunks - 1) / share_chunks;
            v = part[tid];
            for (int sh = 1; sh < all; ++sh) v = __fadd_rn(v, part[sh * OUT + tid]);
        }
        if (rank == 0 && tid < OUT) {
            if (GLU) {
                const int n = tile * (FR_TILE / 2) + row, nc = min(n, N - 1) + half * N;
                v = m < M && f32_suspect(v) ? f32_plain(A + (size_t)m * lda, W + (size_t)nc * ldw, K) : v * F32_UNSCALE;
                const float y = __fmaf_rn(alpha, v, bias ? bias[nc] : 0.f), up = __shfl_down_sync(0xffffffffu, y, NT * 8);
                if (m < M && !half && n < N)
                    C[(size_t)m * ldc + n] = act == IL_ACT_CLAMPED ? il_clamped_glu(y, up, limit, act_alpha)
                                             : act == IL_ACT_GELU_TANH ? il_gelu_tanh_mul(y, up) : y / (1.f + expf(-y)) * up;
            } else {
                const int n = tile * FR_TILE + row + 8 * half;
                if (m < M && n < N) {
                    v = f32_suspect(v) ? f32_plain(A + (size_t)m * lda, W + (size_t)n * ldw, K) : v * F32_UNSCALE;
                    C[(size_t)m * ldc + n] = __fmaf_rn(alpha, v, bias ? bias[n] : 0.f);
                }
            }
        }
        tile += stride, r = 0, cs = 0, share = 0;
        if (STAGE && rounds > 2 && i + 1 < total) {       // x again from its beginning (every warp is past its last round)
            stage_x(0);
            stage_x(1);
            __syncthreads();
        }
    }
}

// ---- more rows: tiles of 128 rows of W x 64 of A, on tcgen05 ------------------------------------------------------------------
// Warps 8-15 bring a chunk of both operands to registers (a chunk ahead), take it apart and write three pieces of each to a ring
// of stages, K-major with the 128-byte swizzle; two threads issue the products, of even and of odd chunks, each with three
// accumulators of its own; warps 0-7 add these up, a running share in registers and, over several shares, the total in tensor memory. Blocks are persistent and
// take tiles b, b + G, ..: the next tile's chunks are taken apart while this one's sums are written. SPLIT: a cluster takes a
// tile, each block a share or two, and the shares meet in shared memory.
// Counters (2,048 rows to 8,192 columns of K = 1,024; a chunk takes 2,600 clocks under the profiler): 6,230 warp instructions a chunk keep the issue slots
// busy for 60 %, mostly those that take operands apart; L1 and shared memory 55 % (of a chunk the 24 products read 144 KB and the pieces are 72 KB written),
// the tensor pipe 30 %. Larger tiles would take less apart a product, but their sums have no room: 128 x 64 in three accumulators twice and a total are 448 of 512 columns.
// Measured, us (multiply-adds before; without the factor 2^23): 627 rows to 1,024 columns of K = 4,096 87.6 (226; 85.4); 2,048 rows to 8,192 columns of
// K = 1,024 317 (911; 318: 108 against 38 TFLOP/s); 61 rows to 1,024 columns of K = 1,024 10.6 (13.6; 10.5), of K = 4,096 17.8 (27.3; 17.7).
constexpr int FT_BM = 128, FT_BN = 64, FT_STAGES = 3, FT_A = FT_BM * 128, FT_B = FT_BN * 128, FT_STAGE = 3 * (FT_A + FT_B);
constexpr int FT_ACC_WARPS = 8, FT_CONV_WARPS = 8, FT_THREADS = (FT_ACC_WARPS + FT_CONV_WARPS + 2) * 32;
constexpr int FT_ROWS = 2 * FT_CONV_WARPS, FT_WU = FT_BM / FT_ROWS, FT_XU = FT_BN / FT_ROWS;       // rows at a time; pieces of a row a thread, of W and of A
constexpr int FT_SMEM = 1024 + FT_STAGES * FT_STAGE;
constexpr int FT_COLS = 3 * FT_BN, FT_COL_TOT = 2 * FT_COLS;   // tensor memory of a chunk: h h of 32 k, of the other 32, the small products; two chunks; the total
constexpr unsigned FT_SPIN = 1u << 24;

// Eight columns of this thread's lane.
__device__ __forceinline__ void f32_columns(uint32_t (&r)[8], uint32_t taddr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}

// SHARES 0: a block a tile; else K's number of shares, which the blocks of a cluster take one or two each.
template <int SHARES, bool VEC>
__global__ void __launch_bounds__(FT_THREADS, 1) gemm_f32_tile_kernel(const float* A, int lda, const float* W, int ldw,
                                                                      float* C, int ldc, const float* bias, float alpha,
                                                                      int M, int N, int K, int m_tiles, int units, int own, int early, int* status) {
    constexpr bool SPLIT = SHARES > 0;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t bars[2 * FT_STAGES + 4];
    const uint32_t full0 = t5_smem(bars), empty0 = full0 + FT_STAGES * 8, done0 = empty0 + FT_STAGES * 8, free0 = done0 + 16;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int chunks = f32_chunks(K), share_chunks = f32_share_chunks(K), cluster = SPLIT ? SHARES / own : 1;
    const int rank = SPLIT ? blockIdx.x % cluster : 0, first = blockIdx.x / cluster, stride = gridDim.x / cluster;
    const int c_lo = SPLIT ? min(chunks, rank * own * share_chunks) : 0, c_hi = SPLIT ? min(chunks, c_lo + own * share_chunks) : chunks;

    if (tid == 0) {
        for (int s = 0; s < FT_STAGES; ++s) {
            t5_mbar_init(full0 + s * 8, FT_CONV_WARPS);
            t5_mbar_init(empty0 + s * 8, 1);
        }
        for (int b = 0; b < 2; ++b) {             // even chunks, odd chunks
            t5_mbar_init(done0 + b * 8, 1);
            t5_mbar_init(free0 + b * 8, FT_ACC_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) t5_alloc(&tmem_slot, 512);
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp >= FT_ACC_WARPS && warp < FT_ACC_WARPS + FT_CONV_WARPS) {
        // ---------------- operands: memory -> pieces ----------------
        // thread: 4 k of rows r0 + FT_ROWS i of W, then of A (half a warp reads 256 bytes of a row and writes 128 of each piece)
        const int ct = tid - FT_ACC_WARPS * 32, r0 = ct >> 4, q = ct & 15;
        float4 v[FT_WU + FT_XU];
        int u = first, c = c_lo;                  // what is asked for next
        const float *wp = nullptr, *ap = nullptr;
        int w_last = 0, a_last = 0;
        auto tile_of = [&]() {
            const int nt = u / m_tiles, mt = u - nt * m_tiles;
            wp = W + (size_t)(nt * FT_BM) * ldw + q * 4, w_last = min(FT_BM, N - nt * FT_BM) - 1;
            ap = A + (size_t)(mt * FT_BN) * lda + q * 4, a_last = min(FT_BN, M - mt * FT_BN) - 1;
        };
        auto load = [&](int i0, int i1) {         // (rows past the end are the last one: computed and dropped)
            const int k = c * F32_CHUNK;
            if (VEC && k + F32_CHUNK <= K) {
#pragma unroll
                for (int i = 0; i < FT_WU + FT_XU; ++i)
                    if (i >= i0 && i < i1)
                        v[i] = *reinterpret_cast<const float4*>((i < FT_WU ? wp + (size_t)(unsigned)(min(r0 + FT_ROWS * i, w_last) * ldw)
                                                                           : ap + (size_t)(unsigned)(min(r0 + FT_ROWS * (i - FT_WU), a_last) * lda)) + k);
            } else {
#pragma unroll
                for (int i = 0; i < FT_WU + FT_XU; ++i)
                    if (i >= i0 && i < i1)
                        v[i] = f32_ld<false>((i < FT_WU ? wp + (size_t)min(r0 + FT_ROWS * i, w_last) * ldw
                                                        : ap + (size_t)min(r0 + FT_ROWS * (i - FT_WU), a_last) * lda) - q * 4, k + q * 4, K);
            }
        };
        const uint32_t at = (uint32_t)(r0 * 128 + (((q >> 1) ^ (r0 & 7)) << 4) + (q & 1) * 8);
        bool any = u < units && c < c_hi;
        if (any) tile_of();
        if (any && early) load(0, FT_WU);
        il_pdl_wait();
        if (any && !early) load(0, FT_WU);
        if (any) load(FT_WU, FT_WU + FT_XU);
        int stage = 0;
        uint32_t phase = 0;
        while (any) {
            if (!t5_mbar_wait(empty0 + stage * 8, phase ^ 1, FT_SPIN)) {
                if (lane == 0) atomicExch(status, 71);
                break;
            }
            unsigned char* st = smem + stage * FT_STAGE + at;
            if (++c == c_hi) {
                c = c_lo, u += stride;
                any = u < units;
                if (any) tile_of();
            }
#pragma unroll
            for (int i0 = 0; i0 < FT_WU + FT_XU; i0 += 2) {
                uint2 h[2], m[2], l[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    f32_split(v[i0 + i].x, v[i0 + i].y, h[i].x, m[i].x, l[i].x);
                    f32_split(v[i0 + i].z, v[i0 + i].w, h[i].y, m[i].y, l[i].y);
                }
                if (any) load(i0, i0 + 2);
                const uint32_t piece = i0 < FT_WU ? FT_A : FT_B;
                unsigned char* to = st + (i0 < FT_WU ? i0 * (FT_ROWS * 128u) : 3u * FT_A + (i0 - FT_WU) * (FT_ROWS * 128u));
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    *reinterpret_cast<uint2*>(to + i * (FT_ROWS * 128)) = h[i];
                    *reinterpret_cast<uint2*>(to + i * (FT_ROWS * 128) + piece) = m[i];
                    *reinterpret_cast<uint2*>(to + i * (FT_ROWS * 128) + 2 * piece) = l[i];
                }
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) t5_mbar_arrive(full0 + stage * 8);
            if (++stage == FT_STAGES) stage = 0, phase ^= 1;
        }
    } else if (warp >= FT_ACC_WARPS + FT_CONV_WARPS) {
        // ---------------- tensor-core issue ----------------
        il_pdl_wait();
        const uint32_t role = warp - FT_ACC_WARPS - FT_CONV_WARPS;        // even chunks, odd chunks
        if (lane == 0 && c_lo < c_hi && first < units) {
            const uint32_t idesc = t5_idesc(FT_BM, FT_BN, false), d = tmem + role * FT_COLS;
            const uint32_t total = (uint32_t)((units - first + stride - 1) / stride) * (uint32_t)(c_hi - c_lo);
            int stage = role;
            uint32_t phase = 0;
            for (uint32_t n = role; n < total; n += 2) {          // n: the block's chunks one after the other
                if (n >= 2 && !t5_mbar_wait(free0 + role * 8, ((n >> 1) - 1) & 1, FT_SPIN)) { atomicExch(status, 72); break; }
                if (!t5_mbar_wait(full0 + stage * 8, phase, FT_SPIN)) { atomicExch(status, 73); break; }
                t5_fence_after();
                const uint32_t sa = t5_smem(smem + stage * FT_STAGE);
                const uint64_t ah = t5_desc(sa, 16, 1024), bh = t5_desc(sa + 3 * FT_A, 16, 1024);
                const uint64_t am = ah + (FT_A >> 4), al = am + (FT_A >> 4), bm = bh + (FT_B >> 4), bl = bm + (FT_B >> 4);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {                  // 32 bytes further along K inside the swizzle span
                    t5_mma_ss(d + 2 * FT_BN, al + kk * 2, bh + kk * 2, idesc, kk > 0);
                    t5_mma_ss(d + 2 * FT_BN, ah + kk * 2, bl + kk * 2, idesc, 1);
                    t5_mma_ss(d + 2 * FT_BN, am + kk * 2, bm + kk * 2, idesc, 1);
                    t5_mma_ss(d + 2 * FT_BN, am + kk * 2, bh + kk * 2, idesc, 1);
                    t5_mma_ss(d + 2 * FT_BN, ah + kk * 2, bm + kk * 2, idesc, 1);
                    t5_mma_ss(d + (kk >> 1) * FT_BN, ah + kk * 2, bh + kk * 2, idesc, kk & 1);
                }
                t5_commit(empty0 + stage * 8);
                t5_commit(done0 + role * 8);
                stage += 2;
                if (stage >= FT_STAGES) stage -= FT_STAGES, phase ^= 1;
            }
        }
        __syncwarp();
    } else {
        // ---------------- sums: this warp's lanes 32 (warp % 4) .. of tensor memory, half of the columns ----------------
        il_pdl_wait();                            // these warps write the output
        const int q = warp & 3, col = (warp >> 2) * 32, row = q * 32 + lane;
        const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + col;
        uint32_t n = 0;
        bool ok = true;
        for (int u = first; u < units && ok; u += stride) {
            float share[32];
            int cs = 0, share_no = 0;
            for (int c = c_lo; c < c_hi; ++c, ++n) {
                if (!t5_mbar_wait(done0 + (n & 1) * 8, (n >> 1) & 1, FT_SPIN)) { ok = false; break; }
                t5_fence_after();
                const uint32_t at = base + (n & 1) * FT_COLS;
#pragma unroll
                for (int i0 = 0; i0 < 32; i0 += 8) {
                    uint32_t x[8], y[8], z[8];
                    f32_columns(x, at + i0);
                    f32_columns(y, at + FT_BN + i0);
                    f32_columns(z, at + 2 * FT_BN + i0);
                    t5_wait_ld();
                    if (i0 == 24) {
                        t5_fence_before();
                        __syncwarp();
                        if (lane == 0) t5_mbar_arrive(free0 + (n & 1) * 8);
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float s = __fadd_rn(__fadd_rn(__uint_as_float(x[i]), __uint_as_float(y[i])), __uint_as_float(z[i]));
                        share[i0 + i] = cs == 0 ? s : __fadd_rn(share[i0 + i], s);
                    }
                }
                if (++cs == share_chunks || c + 1 == c_hi) {
                    if (!SPLIT && share_no > 0) {
#pragma unroll
                        for (int i0 = 0; i0 < 32; i0 += 8) {
                            uint32_t x[8];
                            f32_columns(x, base + FT_COL_TOT + i0);
                            t5_wait_ld();
#pragma unroll
                            for (int i = 0; i < 8; ++i) share[i0 + i] = __fadd_rn(__uint_as_float(x[i]), share[i0 + i]);
                        }
                    }
                    if (c + 1 < c_hi) {           // (SPLIT: the first of two)
                        t5_st32(base + FT_COL_TOT, reinterpret_cast<uint32_t*>(share));
                        t5_wait_st();
                    }
                    cs = 0, ++share_no;
                }
            }
            if (!ok) break;
            if (SPLIT) {
                float* out = reinterpret_cast<float*>(smem) + col * FT_BM + row;      // [share][64][128]; (every product has read its stage)
                if (share_no == 2) {
#pragma unroll
                    for (int i0 = 0; i0 < 32; i0 += 8) {
                        uint32_t x[8];
                        f32_columns(x, base + FT_COL_TOT + i0);
                        t5_wait_ld();
#pragma unroll
                        for (int i = 0; i < 8; ++i) out[(i0 + i) * FT_BM] = __uint_as_float(x[i]);
                    }
                    out += FT_BN * FT_BM;
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) out[i * FT_BM] = c_lo < c_hi ? share[i] : 0.f;
            } else {
                const int nt = u / m_tiles, m0 = (u - nt * m_tiles) * FT_BN + col, gn = nt * FT_BM + row;
                const int rows = gn < N ? min(32, M - m0) : 0;
                const float b = bias && gn < N ? bias[gn] : 0.f;
                float* to = C + (size_t)m0 * ldc + gn;
                uint32_t again = 0;
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (i < rows) {
                        again |= f32_suspect(share[i]) ? 1u << i : 0u;
                        to[(size_t)(unsigned)(i * ldc)] = __fmaf_rn(alpha, share[i] * F32_UNSCALE, b);
                    }
                for (; again; again &= again - 1) {
                    const int i = __ffs(again) - 1;
                    to[(size_t)i * ldc] = __fmaf_rn(alpha, f32_plain(A + (size_t)(m0 + i) * lda, W + (size_t)gn * ldw, K), b);
                }
            }
        }
        if (!ok && lane == 0) atomicExch(status, 75);
    }
    il_pdl_tail();
    if (SPLIT) {
        il_cluster_sync();
        // block `rank` finishes 64 / cluster columns: the shares in order
        const int cols = FT_BN / cluster, live = (chunks + share_chunks - 1) / share_chunks;
        const int nt = first / m_tiles, mt = first - nt * m_tiles;
        const uint32_t from = t5_smem(smem);
        for (int e = tid; e < cols * (FT_BM / 4); e += FT_THREADS) {          // four rows of W each, every share asked for at once
            const int cc = rank * cols + e / (FT_BM / 4), row = e % (FT_BM / 4) * 4, gm = mt * FT_BN + cc, gn = nt * FT_BM + row;
            if (gm >= M || gn >= N) continue;
            float4 p[SPLIT ? SHARES : 1];
#pragma unroll
            for (int sh = 0; sh < SHARES; ++sh)
                p[sh] = f32_peer4(from + 4u * (uint32_t)(((own == 2 ? sh & 1 : 0) * FT_BN + cc) * FT_BM + row), sh < live ? sh / own : 0);
            float v[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
            for (int sh = 1; sh < SHARES; ++sh)
                if (sh < live) v[0] = __fadd_rn(v[0], p[sh].x), v[1] = __fadd_rn(v[1], p[sh].y), v[2] = __fadd_rn(v[2], p[sh].z), v[3] = __fadd_rn(v[3], p[sh].w);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (gn + i < N) {
                    v[i] = f32_suspect(v[i]) ? f32_plain(A + (size_t)gm * lda, W + (size_t)(gn + i) * ldw, K) : v[i] * F32_UNSCALE;
                    C[(size_t)gm * ldc + gn + i] = __fmaf_rn(alpha, v[i], bias ? bias[gn + i] : 0.f);
                }
        }
        il_cluster_sync();                       // (no block leaves while its sums are read)
    }
    t5_fence_before();
    __syncthreads();
    if (warp == 0) {
        t5_fence_after();
        t5_dealloc(tmem, 512);
    }
}

struct F32Args {
    const float *A, *W, *bias;
    float* C;
    int lda, ldw, ldc, M, N, K, early, act;
    float alpha, limit, act_alpha;
    int* status;
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
static int f32_sm_count() {
    static int n[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!n[dev] && (cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n[dev] <= 0)) n[dev] = 148;
    return n[dev];
}

template <typename... KArgs, typename... Args>
static cudaError_t f32_launch(void (*kernel)(KArgs...), int grid, int threads, int smem, int cluster, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (il_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster, attr[n].val.clusterDim.y = 1, attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

template <int NT, bool STAGE, bool VEC, bool GLU> static cudaError_t f32_rows_as(const F32Args& a) {
    static bool done[64];
    const auto kernel = gemm_f32_rows_kernel<NT, STAGE, VEC, GLU>;
    cudaError_t e = f32_allow_smem((const void*)kernel, fr_smem(NT, STAGE, 2), done);
    if (e != cudaSuccess) return e;
    constexpr int ROWS = GLU ? FR_TILE / 2 : FR_TILE;
    const int tiles = (a.N + ROWS - 1) / ROWS, n_sm = f32_sm_count(), shares = f32_shares(a.K);
    // Blocks a tile: up to two an SM; with up to 4 rows, two rounds of K each (one row to 1,024 columns of K = 1,024: 3.2 us, 3.5 in
    // clusters of two), with more a round (8 rows 3.8 and 3.5, 16 rows 4.9 and 3.8).
    int cluster = 1;
    while (cluster < shares && tiles * cluster * 2 <= 2 * n_sm && f32_chunks(a.K) > (a.M <= 4 ? 2 : 1) * FR_WARPS * cluster) cluster *= 2;
    const int clusters = 2 * n_sm / cluster, rounds = (f32_shares(a.K) / cluster * f32_share_chunks(a.K) + FR_WARPS - 1) / FR_WARPS;
    return f32_launch(kernel, (tiles < clusters ? tiles : clusters) * cluster, FR_THREADS, fr_smem(NT, STAGE, rounds), cluster, a.stream, a.A, a.lda, a.W, a.ldw, a.C, a.ldc,
                      a.bias, a.alpha, a.M, a.N, a.K, tiles, cluster, a.early, a.act, a.limit, a.act_alpha);
}

template <bool VEC, bool GLU> static cudaError_t f32_rows(const F32Args& a) {
    return a.M <= 4 ? f32_rows_as<1, true, VEC, GLU>(a) : a.M <= 8 ? f32_rows_as<1, false, VEC, GLU>(a) : f32_rows_as<2, false, VEC, GLU>(a);
}

template <int SHARES, bool VEC> static cudaError_t f32_tiles(const F32Args& a, int m_tiles, int units, int own) {
    static bool done[64];
    const auto kernel = gemm_f32_tile_kernel<SHARES, VEC>;
    cudaError_t e = f32_allow_smem((const void*)kernel, FT_SMEM, done);
    if (e != cudaSuccess) return e;
    const int n_sm = f32_sm_count(), cluster = SHARES ? SHARES / own : 1, grid = SHARES ? units * cluster : units < n_sm ? units : n_sm;
    return f32_launch(kernel, grid, FT_THREADS, FT_SMEM, cluster, a.stream, a.A, a.lda, a.W, a.ldw, a.C, a.ldc, a.bias, a.alpha, a.M, a.N, a.K,
                      m_tiles, units, own, a.early, a.status);
}

template <bool VEC> static cudaError_t f32_dispatch(const F32Args& a) {
    if (a.M <= 16) return a.act ? f32_rows<VEC, true>(a) : f32_rows<VEC, false>(a);
    const long long mt = ((long long)a.M + FT_BN - 1) / FT_BN, units = mt * ((a.N + FT_BM - 1) / FT_BM);
    if (units > 0x3fffffff) return cudaErrorInvalidConfiguration;
    // Blocks a tile, by what was measured in us: a chunk 1.2, a wave's beginning and end 4, a cluster's exchange 2; clusters of large blocks
    // reach some 136 SMs. 61 rows to 1,024 columns, K = 1,024: 28 us whole, 20 in clusters of two, 10.3 of four.
    const int n_sm = f32_sm_count(), shares = f32_shares(a.K);
    float best = (float)((units + n_sm - 1) / n_sm) * f32_chunks(a.K) * 1.2f + 4.f;
    int own = 0;
    for (int o = 2; o >= 1; --o) {
        if (shares / o < 2 || units * shares / o > 4096) continue;
        const int slots = n_sm - 12 > 8 ? n_sm - 12 : 8;
        const float us = (float)((units * (shares / o) + slots - 1) / slots) * (o * f32_share_chunks(a.K) * 1.2f + 6.f);
        if (us < best) best = us, own = o;
    }
    if (!own) return f32_tiles<0, VEC>(a, (int)mt, (int)units, 1);
    return shares == 2 ? f32_tiles<2, VEC>(a, (int)mt, (int)units, own) : shares == 4 ? f32_tiles<4, VEC>(a, (int)mt, (int)units, own)
                                                                                      : f32_tiles<8, VEC>(a, (int)mt, (int)units, own);
}

// act: 0, or the gate of a gated product (M <= 16): W is [2N, K], gate rows, then up rows, bias [2N].
// w_static: W was written long before (a model's weights), not by the kernel in front of this one in the stream.
// status: a device word that a wait that ran out sets.
IL_EXPORT int il_gemm_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc, const float* bias,
                          float alpha, int M, int N, int K, int act, float limit, float act_alpha, int w_static, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return IL_OK;
    if (K <= 0 || lda < K || ldw < K || ldc < N || !status) return IL_BAD_ARG;
    if (act && (M > 16 || act < IL_ACT_SILU || act > IL_ACT_CLAMPED)) return IL_UNSUPPORTED;
    const F32Args a{A, W, bias, C, lda, ldw, ldc, M, N, K, w_static, act, alpha, limit, act_alpha, status, stream};
    const bool vec = !(lda & 3) && !(ldw & 3) && !((uintptr_t)A & 15) && !((uintptr_t)W & 15);
    const cudaError_t e = vec ? f32_dispatch<true>(a) : f32_dispatch<false>(a);
    if (e != cudaSuccess) return 1000 + (int)e;
    IL_LAUNCH_CHECK();
    return IL_OK;
}
