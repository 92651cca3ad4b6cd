// The same products as gemm_narrow.cu on tcgen05, for K in steps of 64: tiles of 64 rows of W (one operand, or two that belong together:
// gate and up rows, the halves of a rotated head of 128), K cut over the blocks of a cluster, what follows the projection in the epilogue.
//
// A block multiplies its tile with all rows of x over its share of K: one thread asks for weights and activations by TMA tensor copies
// (128-byte swizzle), 128 k a stage, the weights before the dependent-launch wait; two threads issue tcgen05.mma with M = 64, an
// accumulator each (one operand: the blocks of 64 k in turn); the accumulators go to shared memory, and every block of the cluster
// finishes some of the rows of x: the shares are added in the order of K through the cluster's shared memory.
// At these sizes nothing is a rate (17 MB of weights, 2.6 us): the time is the trip of the activations to the block after the wait
// and the ends. So every block brings in only the columns of x that its share of K needs, and nothing stands between a stage's
// arrival and its products.
#pragma once
#include "tcgen05.cuh"

constexpr int GC_BK = 128, GC_MAX_STAGES = 8, GC_THREADS = 256;
constexpr int GC_RING = 108 * 1024;               // two blocks an SM: the next product's weights are on their way while this one ends (4,096 columns into the
                                                  // residual, 48 rows, clusters of 8: 11.9 us with a ring of 112 KB, 6.4 so)
constexpr unsigned GC_SPIN = 1u << 24;

struct GcCut {
    int cluster, chunks, per_rank, stages;        // blocks a tile; chunks of 128 k, and a block's; stages of the ring
    int* status;
};

__device__ __forceinline__ void gc_tma(uint32_t dst, const CUtensorMap* map, int row, int kb, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(row), "r"(kb) : "memory");
}
__device__ __forceinline__ void gc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ float4 gc_peer(uint32_t addr, uint32_t rank) {
    uint32_t at;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

// OPS: operands of 64 weight rows; NB: rows of x, a multiple of 16.
template <int MODE, int OPS, int NB>
__global__ void __launch_bounds__(GC_THREADS, 1) gemm_narrow_tc5_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                        const GnArgs p, const GcCut cut) {
    constexpr int W_BYTES = OPS * 64 * GC_BK * 2, STAGE = W_BYTES + NB * GC_BK * 2, ROWS = OPS * 64, PAIRS = 32 * OPS;
    extern __shared__ __align__(1024) unsigned char gc_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gc_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * GC_MAX_STAGES + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ float rstd_s[NB];
    __shared__ float cs[MODE == GN_ROPE ? NB * PAIRS : 1], sn[MODE == GN_ROPE ? NB * PAIRS : 1];
    __shared__ long long slot[MODE == GN_ROPE ? NB : 1];
    const uint32_t full0 = t5_smem(bars), empty0 = full0 + GC_MAX_STAGES * 8, tfull = empty0 + GC_MAX_STAGES * 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x % cut.cluster, tile = blockIdx.x / cut.cluster;
    const int M = p.M, N = p.N;
    const int c_lo = min(cut.chunks, rank * cut.per_rank), n_my = min(cut.chunks, c_lo + cut.per_rank) - c_lo;
    const int n0 = tile * (MODE == GN_GLU ? 64 : ROWS), n1 = MODE == GN_GLU ? N + n0 : n0 + 64;
    const int per = (NB + cut.cluster - 1) / cut.cluster, m_lo = rank * per, m_hi = min(M, m_lo + per);       // the rows of x that this block finishes

    if (tid == 0) {
        for (int s = 0; s < GC_MAX_STAGES; ++s) {
            t5_mbar_init(full0 + s * 8, 1);
            t5_mbar_init(empty0 + s * 8, 2);      // both issuers
        }
        t5_mbar_init(tfull, 2);
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_x) : "memory");        // (its first copy stands behind the wait)
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        const int n = min(n_my, cut.stages);
        for (int i = 0; i < n; ++i) {
            const uint32_t dst = t5_smem(smem + i * STAGE), bar = full0 + i * 8;
            t5_mbar_expect_tx(bar, STAGE);
            gc_tma(dst, &map_w, n0, (c_lo + i) * 2, bar);
            if (OPS == 2) gc_tma(dst + 64 * GC_BK * 2, &map_w, n1, (c_lo + i) * 2, bar);
        }
    }
    if (warp == 3) t5_alloc(&tmem_slot, 128);
    if (MODE == GN_ROPE && warp >= 4) {           // positions, slots and angles come with the step's descriptors
        const bool rotated = tile < p.rp.nh + p.rp.nkv;
        for (int i = tid - 128; i < per * PAIRS; i += 128) {
            const int m = m_lo + i / PAIRS;
            float sv = 0.f, cv = 1.f;
            if (rotated && m < M) {
                sincosf((float)p.rp.tok_pos[m] * p.rp.inv_freq[i % PAIRS], &sv, &cv);
                sv *= p.rp.mscale;
                cv *= p.rp.mscale;
            }
            sn[i] = sv, cs[i] = cv;
        }
        for (int i = tid - 128; i < per; i += 128) {
            const int m = m_lo + i;
            long long off = -1;
            if (m < M && p.rp.cache && tile >= p.rp.nh) {
                const int pos = p.rp.tok_pos[m];
                const int page = p.rp.block_table[(size_t)p.rp.tok_entry[m] * p.rp.bt_stride + pos / p.rp.page_size];
                if (page >= 0) off = ((long long)page * 2 * p.rp.nkv * p.rp.page_size + pos % p.rp.page_size) * p.rp.hd;
            }
            slot[i] = off;
        }
    }
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    const uint32_t tmem = tmem_slot;
    il_pdl_wait();
    il_pdl_launch_dependents();

    constexpr int E_PER = (NB * 16 + GC_THREADS - 1) / GC_THREADS;      // the epilogue's turns: four rows of the tile each
    float e_resid[MODE == GN_RESID ? E_PER : 1][4];
    if (warp == 0) {
        if (lane == 0) {
            const int n = min(n_my, cut.stages);
            for (int i = 0; i < n; ++i) gc_tma(t5_smem(smem + i * STAGE) + W_BYTES, &map_x, 0, (c_lo + i) * 2, full0 + i * 8);
            int stage = 0;
            uint32_t phase = 0;
            for (int i = n; i < n_my; ++i) {
                if (!t5_mbar_wait(empty0 + stage * 8, phase, GC_SPIN)) { atomicExch(cut.status, 81); break; }
                const uint32_t dst = t5_smem(smem + stage * STAGE), bar = full0 + stage * 8;
                t5_mbar_expect_tx(bar, STAGE);
                gc_tma(dst, &map_w, n0, (c_lo + i) * 2, bar);
                if (OPS == 2) gc_tma(dst + 64 * GC_BK * 2, &map_w, n1, (c_lo + i) * 2, bar);
                gc_tma(dst + W_BYTES, &map_x, 0, (c_lo + i) * 2, bar);
                if (++stage == cut.stages) stage = 0, phase ^= 1;
            }
        }
        __syncwarp();
    } else if (warp <= 2) {
        if (lane == 0 && n_my > 0) {
            const int me = warp - 1;
            const uint32_t idesc = t5_idesc(64, NB, false), d = tmem + me * NB;
            int stage = 0;
            uint32_t phase = 0;
            for (int i = 0; i < n_my; ++i) {
                if (!t5_mbar_wait(full0 + stage * 8, phase, GC_SPIN)) { atomicExch(cut.status, 82); break; }
                t5_fence_after();
                const uint32_t sa = t5_smem(smem + stage * STAGE);
#pragma unroll
                for (int kb = 0; kb < 2; ++kb) {
                    if (OPS == 1 && kb != me) continue;           // one operand: a block of 64 k each
                    const uint64_t a = t5_desc(sa + (OPS == 2 ? me * 2 + kb : kb) * 64 * 128, 16, 1024);
                    const uint64_t b = t5_desc(sa + W_BYTES + kb * NB * 128, 16, 1024);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) t5_mma_ss(d, a + kk * 2, b + kk * 2, idesc, i > 0 || kk > 0 || (OPS == 2 && kb > 0));
                }
                t5_commit(empty0 + stage * 8);
                if (++stage == cut.stages) stage = 0, phase ^= 1;
            }
            t5_commit(tfull);
        }
        __syncwarp();
    }
    if (MODE != GN_RESID && warp >= 3) {          // the rows' 1 / rms, where the activations came without it
        for (int i = warp - 3; i < per; i += 5) {
            const int m = m_lo + i;
            float s = 0.f;
            if (p.ni.partial && m < M) {
                const float* q = p.ni.partial + (size_t)m * p.ni.n_partial;
                s = (lane < p.ni.n_partial ? q[lane] : 0.f) + (lane + 32 < p.ni.n_partial ? q[lane + 32] : 0.f);
            }
            s = il_warp_sum(s);
            if (lane == 0) rstd_s[i] = p.ni.partial ? rsqrtf(s * p.ni.inv_h + p.ni.eps) : 1.f;
        }
    }
    if (MODE == GN_RESID) {                       // what the epilogue adds to, asked for now
#pragma unroll
        for (int e = 0; e < E_PER; ++e) {
            const int idx = tid + e * GC_THREADS, m = m_lo + (idx >> 4), n = n0 + (idx & 15) * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i) e_resid[e][i] = m < m_hi && n + i < N ? p.resid[(size_t)m * N + n + i] : 0.f;
        }
    }
    // accumulators to shared memory, [row of x][row of the tile]; their rows 16 q .. lie in the first 16 lanes of quarter q
    float* part = reinterpret_cast<float*>(smem);
    if (warp >= 4) {
        const int q = warp & 3;
        const bool any = n_my > 0;
        if (any && !t5_mbar_wait(tfull, 0, GC_SPIN) && lane == 0) atomicExch(cut.status, 83);
        t5_fence_after();
#pragma unroll
        for (int op = 0; op < OPS; ++op)
#pragma unroll
            for (int j0 = 0; j0 < NB; j0 += 16) {
                uint32_t a[16], b[16];
                gc_ld16(tmem + ((uint32_t)(q * 32) << 16) + op * NB + j0, a);
                if (OPS == 1) gc_ld16(tmem + ((uint32_t)(q * 32) << 16) + NB + j0, b);
                t5_wait_ld();
                if (lane < 16) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float v = OPS == 1 ? __uint_as_float(a[j]) + __uint_as_float(b[j]) : __uint_as_float(a[j]);
                        part[(j0 + j) * ROWS + op * 64 + q * 16 + lane] = any ? v : 0.f;
                    }
                }
            }
        t5_fence_before();
    }
    if (cut.cluster > 1) il_cluster_sync();
    else __syncthreads();
    const uint32_t part_at = t5_smem(part);
    const auto sum = [&](int m, int row, float (&s)[4]) {         // four rows of the tile: the shares of K in their order
        const uint32_t at = part_at + 4u * (uint32_t)(m * ROWS + row);
        float4 v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (r < cut.cluster) v[r] = cut.cluster > 1 ? gc_peer(at, r) : *reinterpret_cast<const float4*>(part + m * ROWS + row);
        s[0] = v[0].x, s[1] = v[0].y, s[2] = v[0].z, s[3] = v[0].w;
#pragma unroll
        for (int r = 1; r < 8; ++r)
            if (r < cut.cluster) s[0] += v[r].x, s[1] += v[r].y, s[2] += v[r].z, s[3] += v[r].w;
    };
    const auto store = [&](__nv_bfloat16* to, const float (&y)[4], int n) {       // up to n columns
        if (n >= 4 && !((uintptr_t)to & 7)) {
            __nv_bfloat162 q[2] = {__floats2bfloat162_rn(y[0], y[1]), __floats2bfloat162_rn(y[2], y[3])};
            *reinterpret_cast<uint2*>(to) = *reinterpret_cast<const uint2*>(q);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < n) to[i] = __float2bfloat16_rn(y[i]);
        }
    };
    if constexpr (MODE == GN_GLU) {
        for (int idx = tid; idx < per * 16; idx += GC_THREADS) {
            const int row = (idx & 15) * 4, m = m_lo + (idx >> 4), n = n0 + row;
            if (m >= m_hi || n >= N) continue;
            const float an = __fmul_rn(p.alpha, rstd_s[idx >> 4]);
            float g[4], u[4], o[4];
            sum(m, row, g);
            sum(m, 64 + row, u);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c = min(n + i, N - 1);
                const float y = __fmaf_rn(an, g[i], p.bias ? p.bias[c] : 0.f), z = __fmaf_rn(an, u[i], p.bias ? p.bias[N + c] : 0.f);
                o[i] = p.act == IL_ACT_CLAMPED ? il_clamped_glu_fast(y, z, p.act_limit, p.act_alpha)
                       : p.act == IL_ACT_GELU_TANH ? il_gelu_tanh_mul_fast(y, z) : il_silu_mul_fast(y, z);
            }
            store(p.out + (size_t)m * p.ldo + n, o, N - n);
        }
    } else if constexpr (MODE == GN_ROPE) {
        const int j = tile;                       // head: q, then k, then v
        const bool rotated = j < p.rp.nh + p.rp.nkv, to_cache = j >= p.rp.nh;
        const int kv = j >= p.rp.nh + p.rp.nkv ? 1 : 0, g = j - p.rp.nh - kv * p.rp.nkv;            // for k and v heads
        const size_t head_off = ((size_t)kv * p.rp.nkv + (to_cache ? g : 0)) * p.rp.page_size * p.rp.hd;
        for (int idx = tid; idx < per * (PAIRS / 4); idx += GC_THREADS) {
            const int d = idx % (PAIRS / 4) * 4, i = idx / (PAIRS / 4), m = m_lo + i;
            if (m >= m_hi) continue;
            const float an = p.alpha * rstd_s[i];
            float a[4], b[4], lo[4], hi[4];
            sum(m, d, a);
            sum(m, d + PAIRS, b);
#pragma unroll
            for (int k = 0; k < 4; ++k) {         // rounded as the product alone would store them, then rotated
                const float y1 = __bfloat162float(__float2bfloat16_rn(an * a[k] + (p.bias ? p.bias[n0 + d + k] : 0.f)));
                const float y2 = __bfloat162float(__float2bfloat16_rn(an * b[k] + (p.bias ? p.bias[n0 + d + PAIRS + k] : 0.f)));
                const float cv = cs[i * PAIRS + d + k], sv = sn[i * PAIRS + d + k];
                lo[k] = rotated ? y1 * cv - y2 * sv : y1;
                hi[k] = rotated ? y2 * cv + y1 * sv : y2;
            }
            store(p.out + (size_t)m * p.ldo + n0 + d, lo, 4);
            store(p.out + (size_t)m * p.ldo + n0 + d + PAIRS, hi, 4);
            if (to_cache && slot[i] >= 0) {
                __nv_bfloat16* dst = p.rp.cache + (size_t)slot[i] + head_off + d;
                store(dst, lo, 4);
                store(dst + PAIRS, hi, 4);
            }
        }
    } else {
#pragma unroll
        for (int e = 0; e < E_PER; ++e) {
            if (e * GC_THREADS >= per * 16) break;                // (uniform)
            const int idx = tid + e * GC_THREADS, row = (idx & 15) * 4, m = m_lo + (idx >> 4), n = n0 + row;
            const bool live = m < m_hi && n < N;
            float sq = 0.f;
            if (live) {
                float s[4], h[4], o[4];
                sum(m, row, s);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = min(n + i, N - 1);
                    const float y = __bfloat162float(__float2bfloat16_rn(p.alpha * s[i] + (p.bias ? p.bias[c] : 0.f)));
                    h[i] = e_resid[e][i] + p.bscale * y;
                    o[i] = h[i] * il_load_any(p.norm_w, p.norm_w_kind, c);
                    if (n + i < N) p.resid[(size_t)m * N + n + i] = h[i], sq += h[i] * h[i];
                }
                store(p.out + (size_t)m * N + n, o, N - n);
            }
            sq += __shfl_xor_sync(0xffffffffu, sq, 1);            // four consecutive lanes share a row and a block of 16 columns
            sq += __shfl_xor_sync(0xffffffffu, sq, 2);
            if ((row & 15) == 0 && live) p.sumsq[(size_t)m * ((N + 15) / 16) + (n >> 4)] = sq;
        }
    }
    if (cut.cluster > 1) il_cluster_sync();       // (no block leaves while its sums are read)
    else __syncthreads();
    if (warp == 3) {
        t5_fence_after();
        t5_dealloc(tmem, 128);
    }
}

typedef CUresult (*gc_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static gc_encode_fn gc_encoder() {
    static gc_encode_fn fn = nullptr;
    if (!fn) {
        void* q = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) == cudaSuccess && r == cudaDriverEntryPointSuccess) fn = (gc_encode_fn)q;
    }
    return fn;
}
// A [rows x K] bfloat16 matrix as [K / 64][rows][64], read in boxes of [2][box_rows][64]: two blocks of K, each a tile with the 128-byte swizzle.
static int gc_map(CUtensorMap* map, const void* base, int rows, int K, int ld, int box_rows) {
    gc_encode_fn enc = gc_encoder();
    if (!enc) return IL_UNSUPPORTED;
    cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(K / 64)}, strides[2] = {(cuuint64_t)ld * 2, 128};
    cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 2}, estr[3] = {1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 2000 + (int)r;
}

template <int MODE, int OPS, int NB>
static int gc_launch(const GnArgs& a, int w_rows, int tiles, int cluster, bool w_static, int* status, cudaStream_t stream) {
    constexpr int STAGE = OPS * 64 * GC_BK * 2 + NB * GC_BK * 2, PART = NB * OPS * 64 * 4;
    const auto kernel = gemm_narrow_tc5_kernel<MODE, OPS, NB>;
    static bool done[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && (dev < 0 || dev >= 64 || !done[dev])) {
        e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 1024 + GC_RING);
        if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
    }
    if (e != cudaSuccess) return 1000 + (int)e;
    GcCut cut;
    cut.cluster = cluster, cut.status = status;
    cut.chunks = (a.K + GC_BK - 1) / GC_BK, cut.per_rank = (cut.chunks + cluster - 1) / cluster;
    cut.stages = GC_RING / STAGE;
    if (cut.stages > cut.per_rank) cut.stages = cut.per_rank;
    if (cut.stages > GC_MAX_STAGES) cut.stages = GC_MAX_STAGES;
    const int ring = cut.stages * STAGE, smem = 1024 + (ring > PART ? ring : PART);
    CUtensorMap map_w, map_x;
    int rc = gc_map(&map_w, a.W, w_rows, a.K, a.ldw, 64);
    if (!rc) rc = gc_map(&map_x, a.x, a.M, a.K, a.ldx, NB);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * cluster);
    cfg.blockDim = dim3(GC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (w_static && il_pdl_enabled()) {           // (the weights are asked for before the wait)
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
    e = cudaLaunchKernelEx(&cfg, kernel, map_w, map_x, a, cut);
    return e == cudaSuccess ? IL_OK : 1000 + (int)e;
}
// Blocks a tile: as many as there are SMs for, with two chunks of K or more each (us, 40 rows, in clusters of 2 / 4 / 8: 1,280 rotated
// columns of K = 1,024 5.1 / 4.6 / 5.0, 1,024 into the residual 5.5 / 4.6 / 5.1, of K = 4,096 9.9 / 7.1 / 6.2; 4,096 gated 7.6 / 7.4 / 12.6).
static int gc_cluster(int tiles, int K) {
    int c = 1;
    while (c < 8 && tiles * c * 2 <= 148 && (K + GC_BK - 1) / GC_BK >= c * 4) c *= 2;
    return c;
}
template <int MODE, int OPS>
static int gc_rows(const GnArgs& a, int w_rows, int tiles, int cluster, bool w_static, int* status, cudaStream_t stream) {
    return a.M <= 32 ? gc_launch<MODE, OPS, 32>(a, w_rows, tiles, cluster, w_static, status, stream)
                     : gc_launch<MODE, OPS, 48>(a, w_rows, tiles, cluster, w_static, status, stream);
}
