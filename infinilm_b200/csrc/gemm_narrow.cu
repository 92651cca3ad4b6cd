// Decode products of 17 to 48 rows on a narrow model, with what follows the projection in a decoder layer done in the epilogue:
//   gated   out[M,N] = act(alpha * x . Wg^T + bg) * (alpha * x . Wu^T + bu),  W = [Wg; Wu], K <= 1,024
//   rope    the q/k/v projection, q and k rotated, k and v written to the paged cache, K <= 1,024
//   resid   resid += bscale * bf16(alpha * x . W^T + b), xw = resid * norm weight, sums of the residual's squares, K <= 1,024
//           (in steps of 64, or up to 32 rows: K <= 4,096)
// Two forms: on tcgen05 with K over a cluster (gemm_narrow_tc5.cuh), which more rows and the long product take (gc_ok has the times), and
// the one below.
// They do for these rows what the fused forms of the weight-streaming kernels do for up to 16, and take the same unfinished
// norms (the activations times a weight, to be divided by the rms that `GnNormIn` gives).
//
// At these sizes a matrix is 2 to 17 MB, a few microseconds of memory, and what a kernel built for throughput pays at its ends
// (tensor maps, barriers, tensor memory) and the norm and rotation kernels between them were most of a decode step. So: every
// weight a block needs is on its way to registers before the wait for the kernel in front (ordinary launch where the caller does
// not vouch that W is a weight); the activations come to shared memory once a block, in slabs of 512 columns by asynchronous
// copies; a warp multiplies one tile of 16 weight rows (mma.sync m16n8k16, W as the A operand, f32 sums) with all rows of x
// over its share of K; the shares meet in shared memory and are added in order. A block is TILES tiles x KG shares of K.
// A 24-layer model 1,024 wide, 40 requests arriving and leaving: 71.8 ms of steps before, 66.2 with these; its layer's products of 17 rows
// (gate+up / o / down, by themselves) 7.7 / 3.8 / 9.1 us before, 6.4 / 3.0 / 7.8 now, and two norms and a rotation less. With the
// activations read from L2 by every tile of weights instead of staged once a block the steps took 69.4; with the long product's K cut
// over a cluster of two blocks 71.5. With the tcgen05 form, which takes 40 rows' long product from the library too, 60.1.
#include "common.cuh"

constexpr int GN_SLAB = 512, GN_STAGES = 3, GN_MAX_ROWS = 48, GN_MAX_K = 4096;
constexpr int GN_ROW = GN_SLAB * 2 + 64;          // bytes of a staged row: 4 16-byte pieces more than a multiple of 8, so that the lanes of a
                                                  // load phase (two rows, four pieces) hit eight different bank groups
enum { GN_GLU = 0, GN_ROPE = 1, GN_RESID = 2 };

struct GnNormIn {
    const float* partial;                         // [M][n_partial] sums of squares (n_partial <= 64), or null: the activations are normalised
    int n_partial;
    float inv_h, eps;
};
struct GnRope {
    const int *tok_pos, *tok_entry, *block_table;
    int bt_stride;
    __nv_bfloat16* cache;                         // [page][2][nkv][page_size][hd], or null
    int page_size, nh, nkv, hd, rot;
    const float* inv_freq;
    float mscale;
};
struct GnArgs {
    const __nv_bfloat16 *x, *W;
    __nv_bfloat16* out;                           // gated, rope: the output; resid: xw
    const float* bias;
    int ldx, ldw, ldo, M, N, K;                   // N: output columns
    float alpha;
    GnNormIn ni;
    int act;                                      // gated
    float act_limit, act_alpha;
    GnRope rp;                                    // rope
    float *resid, *sumsq;                         // resid
    float bscale;
    const void* norm_w;
    int norm_w_kind;
};

#include "gemm_narrow_tc5.cuh"

__device__ __forceinline__ void gn_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__host__ __device__ constexpr int gn_smem(int NT, int TILES, int KG, int slabs) {
    const int ring = (slabs < GN_STAGES ? slabs : GN_STAGES) * NT * 8 * GN_ROW, part = KG * TILES * 16 * (NT * 8 + 1) * 4;
    return ring > part ? ring : part;
}

// NT: groups of 8 activation rows; SLABS: slabs of K at most. Slab s of K is blocks of 32 columns 16 s ..; share kg takes blocks kg, kg + KG, ..
template <int MODE, int NT, int TILES, int KG, int SLABS>
__global__ void __launch_bounds__(TILES * KG * 32, 1) gemm_narrow_kernel(const GnArgs p) {
    constexpr int WARPS = TILES * KG, THREADS = WARPS * 32, PER = 16 / KG, ROWS = NT * 8, PS = ROWS + 1;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ float rstd_s[ROWS];
    __shared__ float cs[MODE == GN_ROPE ? ROWS : 1][8], sn[MODE == GN_ROPE ? ROWS : 1][8];
    __shared__ long long slot[MODE == GN_ROPE ? ROWS : 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const int tile = warp % TILES, kg = warp / TILES;
    const int M = p.M, N = p.N, K = p.K;
    const int n_slabs = (K + GN_SLAB - 1) / GN_SLAB;
    // the two weight rows of this lane: row r of the tile's first eight and of its second eight
    int n_lo, step;                               // output column (weight row) of the tile's row 0; row 8 + i is n_lo + step + i
    bool rotated = false;
    int j = 0, d0 = 0;
    if (MODE == GN_GLU) {
        n_lo = (blockIdx.x * TILES + tile) * 8, step = N;
    } else if (MODE == GN_ROPE) {
        const int tiles_per_head = p.rp.hd >> 4;
        j = blockIdx.x / tiles_per_head;          // head (q, then k, then v) and tile in it; a rotated tile's halves are rot / 2 apart
        const int tl = blockIdx.x - j * tiles_per_head;
        rotated = j < p.rp.nh + p.rp.nkv && tl < (p.rp.rot >> 4);
        d0 = rotated ? tl * 8 : (j < p.rp.nh + p.rp.nkv ? p.rp.rot + (tl - (p.rp.rot >> 4)) * 16 : tl * 16);
        step = rotated ? p.rp.rot >> 1 : 8;
        n_lo = j * p.rp.hd + d0;
    } else {
        n_lo = (blockIdx.x * TILES + tile) * 16, step = 8;
    }
    const int n_w = MODE == GN_GLU ? 2 * N : N;   // weight rows
    const int row0 = MODE == GN_GLU ? min(n_lo + r, N - 1) : min(n_lo + r, n_w - 1);
    const int row1 = MODE == GN_GLU ? N + row0 : min(n_lo + step + r, n_w - 1);      // rows past the end are computed and dropped
    const __nv_bfloat16* w0 = p.W + (size_t)row0 * p.ldw;
    const __nv_bfloat16* w1 = p.W + (size_t)row1 * p.ldw;
    uint4 a[SLABS * PER][2];
#pragma unroll
    for (int i = 0; i < SLABS * PER; ++i) {
        const int k = ((i / PER) * 16 + (i % PER) * KG + kg) * 32 + c * 8;
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        a[i][0] = a[i][1] = zero;
        if (k < K) {
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(a[i][0].x), "=r"(a[i][0].y), "=r"(a[i][0].z), "=r"(a[i][0].w) : "l"(w0 + k));
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(a[i][1].x), "=r"(a[i][1].y), "=r"(a[i][1].z), "=r"(a[i][1].w) : "l"(w1 + k));
        }
    }
    if (MODE == GN_ROPE) {                        // positions, slots and angles come with the step's descriptors
        for (int i = tid; i < ROWS * 8; i += THREADS) {
            const int m = i >> 3, nl = i & 7;
            float sv = 0.f, cv = 1.f;
            if (rotated && m < M) {
                sincosf((float)p.rp.tok_pos[m] * p.rp.inv_freq[d0 + nl], &sv, &cv);
                sv *= p.rp.mscale;
                cv *= p.rp.mscale;
            }
            sn[m][nl] = sv, cs[m][nl] = cv;
        }
        for (int m = tid; m < ROWS; m += THREADS) {
            long long off = -1;
            if (m < M && p.rp.cache && j >= p.rp.nh) {
                const int pos = p.rp.tok_pos[m];
                const int page = p.rp.block_table[(size_t)p.rp.tok_entry[m] * p.rp.bt_stride + pos / p.rp.page_size];
                if (page >= 0) off = ((long long)page * 2 * p.rp.nkv * p.rp.page_size + pos % p.rp.page_size) * p.rp.hd;
            }
            slot[m] = off;
        }
    }
    il_pdl_wait();
    il_pdl_launch_dependents();

    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    auto load = [&](int s) {                      // slab s of x: rows of 512 columns, zeros past K and past M
        const uint32_t dst = sbase + (uint32_t)(s % GN_STAGES) * (ROWS * GN_ROW);
        for (int i = tid; i < ROWS * (GN_SLAB / 8); i += THREADS) {
            const int m = i / (GN_SLAB / 8), k = s * GN_SLAB + (i % (GN_SLAB / 8)) * 8;
            const bool in = m < M && k < K;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + m * GN_ROW + (i % (GN_SLAB / 8)) * 16),
                         "l"(p.x + (size_t)(in ? m : 0) * p.ldx + (in ? k : 0)), "r"(in ? 16 : 0));
        }
    };
#pragma unroll
    for (int s = 0; s < GN_STAGES; ++s) {
        if (s < SLABS && s < n_slabs) load(s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    if (MODE != GN_RESID) {                       // the rows' 1 / rms, where the activations came without it
#pragma unroll
        for (int i = 0; i < (ROWS + WARPS - 1) / WARPS; ++i) {
            const int m = warp + i * WARPS;
            float s = 0.f;
            if (p.ni.partial && m < M) {
                const float* q = p.ni.partial + (size_t)m * p.ni.n_partial;
                s = (lane < p.ni.n_partial ? q[lane] : 0.f) + (lane + 32 < p.ni.n_partial ? q[lane + 32] : 0.f);
            }
            s = il_warp_sum(s);
            if (lane == 0 && m < ROWS) rstd_s[m] = p.ni.partial ? rsqrtf(s * p.ni.inv_h + p.ni.eps) : 1.f;
        }
    }
    // what the epilogue of the resid form adds to, asked for now: thread t has column t % 16 of rows t / 16, + THREADS / 16, ..
    constexpr int E_STEP = THREADS / (16 * TILES), E_PER = (ROWS + E_STEP - 1) / E_STEP;
    const int e_n = blockIdx.x * TILES * 16 + tid % (16 * TILES), e_m = tid / (16 * TILES);
    float e_resid[MODE == GN_RESID ? E_PER : 1], e_w = 0.f, e_bias = 0.f;
    if (MODE == GN_RESID) {
#pragma unroll
        for (int i = 0; i < E_PER; ++i) e_resid[i] = e_m + i * E_STEP < M && e_n < N ? p.resid[(size_t)(e_m + i * E_STEP) * N + e_n] : 0.f;
        if (e_n < N) e_w = il_load_any(p.norm_w, p.norm_w_kind, e_n), e_bias = p.bias ? p.bias[e_n] : 0.f;
    }

    float acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[t][q] = 0.f;
#pragma unroll
    for (int s = 0; s < SLABS; ++s) {
        if (s < n_slabs) {                        // (uniform over the block)
            asm volatile("cp.async.wait_group %0;\n" ::"n"(GN_STAGES - 1) : "memory");
            __syncthreads();
            const unsigned char* xs = sm + (size_t)(s % GN_STAGES) * (ROWS * GN_ROW) + r * GN_ROW + c * 16;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const uint4 a0 = a[s * PER + i][0], a1 = a[s * PER + i][1];
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const uint4 b = *reinterpret_cast<const uint4*>(xs + t * 8 * GN_ROW + (i * KG + kg) * 64);
                    gn_mma(acc[t], a0.x, a1.x, a0.y, a1.y, b.x, b.y);
                    gn_mma(acc[t], a0.z, a1.z, a0.w, a1.w, b.z, b.w);
                }
            }
            if (SLABS > GN_STAGES) {
                __syncthreads();                  // everyone has read the stage
                if (s + GN_STAGES < n_slabs) load(s + GN_STAGES);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();                              // x is read: its place takes the shares' sums, [share][tile][16 weight rows][rows of x]
    float* part = reinterpret_cast<float*>(sm);
    {
        float* mine = part + (size_t)(kg * TILES + tile) * 16 * PS + r * PS + c * 2;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            mine[t * 8] = acc[t][0], mine[t * 8 + 1] = acc[t][1];
            mine[8 * PS + t * 8] = acc[t][2], mine[8 * PS + t * 8 + 1] = acc[t][3];
        }
    }
    __syncthreads();
    const auto sum = [&](int tl, int row, int m) {
        float s = 0.f;
#pragma unroll
        for (int g = 0; g < KG; ++g) s += part[((size_t)(g * TILES + tl) * 16 + row) * PS + m];
        return s;
    };
    if constexpr (MODE == GN_GLU) {
        for (int idx = tid; idx < TILES * 8 * ROWS; idx += THREADS) {
            const int nl = idx % (TILES * 8), m = idx / (TILES * 8), n = blockIdx.x * TILES * 8 + nl;     // consecutive threads: consecutive columns
            if (m >= M || n >= N) continue;
            const float an = __fmul_rn(p.alpha, rstd_s[m]);
            const float y = __fmaf_rn(an, sum(nl >> 3, nl & 7, m), p.bias ? p.bias[n] : 0.f);
            const float u = __fmaf_rn(an, sum(nl >> 3, (nl & 7) + 8, m), p.bias ? p.bias[N + n] : 0.f);
            p.out[(size_t)m * p.ldo + n] = __float2bfloat16_rn(p.act == IL_ACT_CLAMPED ? il_clamped_glu_fast(y, u, p.act_limit, p.act_alpha)
                                                               : p.act == IL_ACT_GELU_TANH ? il_gelu_tanh_mul_fast(y, u) : il_silu_mul_fast(y, u));
        }
    } else if constexpr (MODE == GN_ROPE) {
        const bool to_cache = j >= p.rp.nh;
        const int kv = j >= p.rp.nh + p.rp.nkv ? 1 : 0, g = j - p.rp.nh - kv * p.rp.nkv;            // for k and v heads
        const size_t head_off = ((size_t)kv * p.rp.nkv + (to_cache ? g : 0)) * p.rp.page_size * p.rp.hd;
        for (int idx = tid; idx < ROWS * 8; idx += THREADS) {
            const int nl = idx & 7, m = idx >> 3;
            if (m >= M) continue;
            const int n1 = n_lo + nl, n2 = n1 + step;
            // rounded as the product alone would store them, then rotated
            const float an = p.alpha * rstd_s[m];
            const float y1 = __bfloat162float(__float2bfloat16_rn(an * sum(0, nl, m) + (p.bias ? p.bias[n1] : 0.f)));
            const float y2 = __bfloat162float(__float2bfloat16_rn(an * sum(0, nl + 8, m) + (p.bias ? p.bias[n2] : 0.f)));
            const float cv = cs[m][nl], sv = sn[m][nl];
            const __nv_bfloat16 lo = __float2bfloat16_rn(rotated ? y1 * cv - y2 * sv : y1);
            const __nv_bfloat16 hi = __float2bfloat16_rn(rotated ? y2 * cv + y1 * sv : y2);
            p.out[(size_t)m * p.ldo + n1] = lo;
            p.out[(size_t)m * p.ldo + n2] = hi;
            if (to_cache && slot[m] >= 0) {
                __nv_bfloat16* dst = p.rp.cache + (size_t)slot[m] + head_off + (d0 + nl);
                dst[0] = lo;
                dst[step] = hi;
            }
        }
    } else {
        const int nl = tid % (16 * TILES);
#pragma unroll
        for (int i = 0; i < E_PER; ++i) {
            const int m = e_m + i * E_STEP;
            const bool live = m < M && e_n < N;
            float h = 0.f;
            if (live) {
                const float y = __bfloat162float(__float2bfloat16_rn(p.alpha * sum(nl >> 4, nl & 15, m) + e_bias));
                h = e_resid[i] + p.bscale * y;
                p.resid[(size_t)m * N + e_n] = h;
                p.out[(size_t)m * N + e_n] = __float2bfloat16_rn(h * e_w);
            }
            float sq = h * h;                     // 16 consecutive lanes share a row and a block of 16 columns
            sq += __shfl_xor_sync(0xffffffffu, sq, 8);
            sq += __shfl_xor_sync(0xffffffffu, sq, 4);
            sq += __shfl_xor_sync(0xffffffffu, sq, 2);
            sq += __shfl_xor_sync(0xffffffffu, sq, 1);
            if ((nl & 15) == 0 && live) p.sumsq[(size_t)m * ((N + 15) / 16) + (e_n >> 4)] = sq;
        }
    }
}

template <int MODE, int NT, int TILES, int KG, int SLABS>
static int gn_launch(const GnArgs& a, int blocks, bool w_static, cudaStream_t stream) {
    constexpr int smem = gn_smem(NT, TILES, KG, SLABS);
    static_assert(smem <= 220 * 1024, "shared memory of a block");
    const auto kernel = gemm_narrow_kernel<MODE, NT, TILES, KG, SLABS>;
    static bool done[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && (dev < 0 || dev >= 64 || !done[dev])) {
        e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
    }
    if (e == cudaSuccess) e = il_launch_as(w_static, kernel, dim3(blocks), dim3(TILES * KG * 32), (size_t)smem, stream, a);
    if (e != cudaSuccess) return 1000 + (int)e;
    IL_LAUNCH_CHECK();
    return IL_OK;
}
template <int MODE, int TILES, int KG, int SLABS>
static int gn_rows(const GnArgs& a, int blocks, bool w_static, cudaStream_t stream) {
    if (a.M <= 24) return gn_launch<MODE, 3, TILES, KG, SLABS>(a, blocks, w_static, stream);
    if (a.M <= 32) return gn_launch<MODE, 4, TILES, KG, SLABS>(a, blocks, w_static, stream);
    if constexpr (SLABS > 2) return IL_UNSUPPORTED;       // (the long product into the residual ends at 32 rows)
    else return a.M <= 40 ? gn_launch<MODE, 5, TILES, KG, SLABS>(a, blocks, w_static, stream) : gn_launch<MODE, 6, TILES, KG, SLABS>(a, blocks, w_static, stream);
}
static bool gn_bad(const GnArgs& a) {
    return a.M > GN_MAX_ROWS || a.K <= 0 || (a.K & 7) || (a.ldx & 7) || (a.ldw & 7) || a.ldx < a.K || a.ldw < a.K || ((uintptr_t)a.x & 15) ||
           ((uintptr_t)a.W & 15) || (a.ni.partial && (a.ni.n_partial <= 0 || a.ni.n_partial > 64));
}

// cluster: blocks a tile of the tcgen05 form (0: whether and how many is chosen here; negative: the mma.sync form). From which number of rows
// the tcgen05 form is taken: us at 17 / 32 / 40 / 48 rows, mma.sync and tcgen05, 1,024 wide with 4,096 in the feed-forward, replayed in a row:
//   gated 6.5, 7.6, 8.4, 9.5 and 6.9, 6.6, 7.6, 7.5; rotated 3.9, 4.5, 5.2, 6.5 and 4.3, 4.4, 4.6, 4.6;
//   into the residual K = 1,024 3.0, 3.4, 3.9, 5.0 and 4.0, 4.2, 4.6, 4.6; K = 4,096 7.8, 8.6, -, - and 5.9, 6.1, 6.2, 6.4.
static bool gc_ok(const GnArgs& a, int cluster, const int* status, int rows_from) {
    return cluster >= 0 && status && a.K % 64 == 0 && (cluster > 0 || a.M >= rows_from);
}

// Up to 48 rows (made for 17 and more), K <= 1,024. W [2N, K]: gate rows, then up rows; bias [2N] or null; act: 1 SiLU, 2 the tanh form of
// GELU, 3 the clamped gate. norm_partial: see GnNormIn. w_static: W was written long before, not by the kernel in front of this one.
IL_EXPORT int il_gemm_narrow_glu(const void* x, int ldx, const void* W, int ldw, void* out, int ldo, const float* bias, float alpha, int M, int N, int K,
                                 int act, float act_limit, float act_alpha, const float* norm_partial, int n_partial, int norm_h, float norm_eps,
                                 int w_static, int cluster, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return IL_OK;
    GnArgs a = {};
    a.x = (const __nv_bfloat16*)x, a.W = (const __nv_bfloat16*)W, a.out = (__nv_bfloat16*)out, a.bias = bias;
    a.ldx = ldx, a.ldw = ldw, a.ldo = ldo, a.M = M, a.N = N, a.K = K, a.alpha = alpha, a.act = act, a.act_limit = act_limit, a.act_alpha = act_alpha;
    a.ni = GnNormIn{norm_partial, n_partial, norm_partial ? 1.f / (float)norm_h : 0.f, norm_eps};
    if (gn_bad(a) || K > 2 * GN_SLAB || ldo < N || act < 1 || act > 3 || (norm_partial && norm_h <= 0)) return IL_UNSUPPORTED;
    if (gc_ok(a, cluster, status, 25)) {
        const int tiles = (N + 63) / 64;
        return gc_rows<GN_GLU, 2>(a, 2 * N, tiles, cluster > 0 ? cluster : gc_cluster(tiles, K), w_static != 0, status, stream);
    }
    return gn_rows<GN_GLU, 4, 4, 2>(a, (N + 31) / 32, w_static != 0, stream);
}

IL_EXPORT int il_gemm_narrow_rope(const void* x, int ldx, const void* W, int ldw, void* out, int ldo, const float* bias, float alpha, int M, int K,
                                  const int* tok_pos, const int* tok_entry, const int* block_table, int bt_stride, void* cache, int page_size, int nh,
                                  int nkv, int hd, int rot, const float* inv_freq, float mscale, const float* norm_partial, int n_partial, int norm_h,
                                  float norm_eps, int w_static, int cluster, int* status, cudaStream_t stream) {
    if (M <= 0) return IL_OK;
    GnArgs a = {};
    a.x = (const __nv_bfloat16*)x, a.W = (const __nv_bfloat16*)W, a.out = (__nv_bfloat16*)out, a.bias = bias;
    a.ldx = ldx, a.ldw = ldw, a.ldo = ldo, a.M = M, a.N = (nh + 2 * nkv) * hd, a.K = K, a.alpha = alpha;
    a.ni = GnNormIn{norm_partial, n_partial, norm_partial ? 1.f / (float)norm_h : 0.f, norm_eps};
    a.rp = GnRope{tok_pos, tok_entry, block_table, bt_stride, (__nv_bfloat16*)cache, page_size, nh, nkv, hd, rot, inv_freq, mscale};
    if (gn_bad(a) || K > 2 * GN_SLAB || ldo < a.N || (norm_partial && norm_h <= 0)) return IL_UNSUPPORTED;
    if (nh <= 0 || nkv <= 0 || hd <= 0 || (hd & 15) || rot < 0 || rot > hd || (rot & 15) || page_size <= 0) return IL_UNSUPPORTED;
    if (rot > 0 && !inv_freq) return IL_BAD_ARG;
    if (gc_ok(a, cluster, status, 33) && rot == hd && (hd == 64 || hd == 128)) {
        const int tiles = nh + 2 * nkv, c = cluster > 0 ? cluster : gc_cluster(tiles, K);
        return hd == 64 ? gc_rows<GN_ROPE, 1>(a, a.N, tiles, c, w_static != 0, status, stream) : gc_rows<GN_ROPE, 2>(a, a.N, tiles, c, w_static != 0, status, stream);
    }
    return gn_rows<GN_ROPE, 1, 8, 2>(a, a.N / 16, w_static != 0, stream);
}

// N = width of the residual stream (a multiple of nothing: the last block may be ragged); sumsq [M][ceil(N / 16)]. K <= 1,024, or
// K in steps of 64 or up to 32 rows, K <= 4,096.
IL_EXPORT int il_gemm_narrow_resid(const void* x, int ldx, const void* W, int ldw, const float* bias, float alpha, int M, int N, int K, float* resid,
                                   float bscale, const void* norm_w, int norm_w_kind, void* xw, float* sumsq, int w_static, int cluster, int* status,
                                   cudaStream_t stream) {
    if (M <= 0 || N <= 0) return IL_OK;
    GnArgs a = {};
    a.x = (const __nv_bfloat16*)x, a.W = (const __nv_bfloat16*)W, a.out = (__nv_bfloat16*)xw, a.bias = bias;
    a.ldx = ldx, a.ldw = ldw, a.ldo = N, a.M = M, a.N = N, a.K = K, a.alpha = alpha;
    a.resid = resid, a.sumsq = sumsq, a.bscale = bscale, a.norm_w = norm_w, a.norm_w_kind = norm_w_kind;
    if (gn_bad(a) || K > GN_MAX_K || !resid || !norm_w || !xw || !sumsq) return IL_UNSUPPORTED;
    if (norm_w_kind != IL_F32 && norm_w_kind != IL_BF16) return IL_BAD_ARG;
    if (gc_ok(a, cluster, status, K > 2 * GN_SLAB ? 1 : 41)) {
        const int tiles = (N + 63) / 64;
        return gc_rows<GN_RESID, 1>(a, N, tiles, cluster > 0 ? cluster : gc_cluster(tiles, K), w_static != 0, status, stream);
    }
    const int blocks = (N + 15) / 16;
    if (K <= 2 * GN_SLAB) return gn_rows<GN_RESID, 1, 8, 2>(a, blocks, w_static != 0, stream);
    return gn_rows<GN_RESID, 1, 16, GN_MAX_K / GN_SLAB>(a, blocks, w_static != 0, stream);
}
