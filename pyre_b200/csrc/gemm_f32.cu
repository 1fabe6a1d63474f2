// True 32-bit matrix product for the float32 path:  C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]).
//
// IEEE fp32 multiply-add on the CUDA cores, no tensor-core or TF32 mode anywhere.  W has
// the layout of a linear layer's weight ([out, in], in-dim contiguous, pyre/model.py:84-87
// via nn.Linear).  Every output element is summed in three levels:
//   * a run is 32 consecutive k; its even and its odd k are two chains part = fma(a[k], w[k], part), ascending, and the
//     run's sum is even + odd (a float4 of each operand then is two fma.rn.f32x2, without a move);
//   * chain c of eight adds the sums of the runs c, c + 8, c + 16, ... in ascending order;
//   * the eight chains are added in ascending order.
// The rounding error grows with 16 + K / 256 + 8 terms instead of K.  The grouping depends on k alone, whatever kernel
// or tile shape computes it: a row's result is bit-identical for any M and any batch composition.  The chains are
// what the kernels divide among threads (few rows) or CTAs (few tiles) without changing a bit.
//
// Two kernels, the same arithmetic in each:
//   * many rows: 64 x 64 tiles, one CTA per tile or a cluster of eight, one per chain;
//   * up to 32 rows (decode): a weight stream, 16 output features per CTA, the chains in different threads.
// Both bring their operands to shared memory by cp.async, 16 bytes at a time (VEC) where the rows of both operands are 16-byte
// aligned and K is a multiple of 4, else 4 bytes at a time.  Measured with rows of 3,585 floats (M x N; a plain tile kernel
// with scalar loads through registers, 128 x 128 or 64 x 128 outputs / 4-byte copies): 4 x 18944: 631 and 1417 / 87 us, 32 x 18944: 716
// and 1494 / 253 us, 509 x 18944: 8598 and 13395 / 2294 us; with rows of a multiple of four: 3385 us for 509 x 37888 x 3584.
#include "common.cuh"

namespace {
constexpr int RUN = 32, CHAINS = 8;       // the grouping of the sums, see above

typedef unsigned long long f32x2;         // two floats in one 64-bit register: the even k below, the odd k above

__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float run_sum(f32x2 p) {      // even + odd
    return __uint_as_float((uint32_t)p) + __uint_as_float((uint32_t)(p >> 32));
}
// a 16-byte copy into shared memory, or 16 bytes of zeros
__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
// a 4-byte copy, or 4 bytes of zeros
__device__ __forceinline__ void copy4(float* dst, const float* src, bool live) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = live ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
}  // namespace

// ---------------------------------------------------------------------------
// Many rows.  Bound by the FMA pipe's operands: out of registers alone, fma.rn.f32x2 reaches 49 TFLOP/s on this chip where no
// operand stays from one instruction to the next and 58 to 63 where one does (the register file's ports; scalar fmaf 61).  A thread owns 8 x 4
// outputs as even-odd pairs, four k cost it 12 reads of 16 bytes from shared memory and 64 fma.rn.f32x2.  128 threads on a
// 64 x 64 tile and 168 registers put three CTAs on an SM, whose barriers and first loads hide behind one another; operands
// arrive by cp.async, 16 k at a time and two steps ahead, in rows of 20 floats (reads of 16 bytes by eight neighbouring
// threads cover all banks).  Measured (M x N x K): 509 x 37888 x 3584: 3905 -> 3386 us (35 -> 41 TFLOP/s); 509 x 3584 x
// 18944: 2565 -> 1997 us; 40 x 3584 x 18944: 2505 -> 310 us (the tiles were 128 x 128, a CTA each, 8 x 8 outputs per
// thread).  8 x 8 outputs per thread here (255 registers): 3713 us for the first, scalar fmaf in their place 3597 us.
//
// PARTS == 1: a CTA walks the chains one after the other (runs c, c + 8, ...) and keeps the sum of the finished ones
// in shared memory.  PARTS == 8: the CTAs of a cluster take a chain each and add them up through distributed shared memory.
// ---------------------------------------------------------------------------
constexpr int TILE = 64, TILE_STAGES = 3;

template <int PARTS, bool VEC>
__global__ void __launch_bounds__(128, 3)
sgemm_nt_tiles_kernel(const float* A, long long lda, const float* W, long long ldw,
                      float* C, long long ldc, const float* bias, int M, int N, int K, int tiles_m) {
    constexpr int BM = TILE, BN = TILE, TN = BN / 16, BK = 16, PITCH = BK + 4, STAGES = TILE_STAGES, STAGE = (BM + BN) * PITCH;
    static_assert(PARTS == 1 || PARTS == CHAINS, "all chains in one CTA, or one in each");
    extern __shared__ __align__(16) float tiles[];      // STAGES x STAGE, then total: BM x BN
    float* const total = tiles + STAGES * STAGE;
    pdl_trigger();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int rank = PARTS > 1 ? blockIdx.x % PARTS : 0, tile = blockIdx.x / PARTS;
    // the tiles of one block of weight rows follow one another: their weights come out of the L2 cache
    const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * BN;
    const int n_runs = (K + RUN - 1) / RUN;
    // copies: per step 128 rows of 16 k; a thread fetches pieces of P floats, piece lq of the rows lr, lr + STEP, ... of both operands
    constexpr int P = VEC ? 4 : 1, PIECES = BK / P, STEP = 128 / PIECES;
    const int lr = tid / PIECES, lq = tid % PIECES;
    int f_chain = rank, f_run = rank, f_half = 0, f_stage = 0;      // where the next fetch stands
    auto copy = [](float* dst, const float* src, bool live) {
        if constexpr (VEC) copy16(dst, src, live);
        else copy4(dst, src, live);
    };
    auto fetch = [&]() {
        if (f_run < n_runs) {
            const int gk = f_run * RUN + f_half * BK + P * lq;
            const bool in_k = gk < K;
            float* dst = tiles + f_stage * STAGE + lr * PITCH + P * lq;
            // rows outside the matrices are not stored: whatever their sums are
#pragma unroll
            for (int h = 0; h < BM; h += STEP) {
                const int gm = m0 + lr + h;
                if (gm < M) copy(dst + h * PITCH, in_k ? A + (size_t)gm * lda + gk : A, in_k);
            }
#pragma unroll
            for (int h = 0; h < BN; h += STEP) {
                const int gn = n0 + lr + h;
                if (gn < N) copy(dst + (BM + h) * PITCH, in_k ? W + (size_t)gn * ldw + gk : W, in_k);
            }
            f_half ^= 1;
            if (f_half == 0) {
                f_run += CHAINS;
                if (PARTS == 1 && f_run >= n_runs && f_chain + 1 < CHAINS) f_run = ++f_chain;
            }
        }
        f_stage = f_stage == STAGES - 1 ? 0 : f_stage + 1;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    pdl_wait();
    for (int s = 0; s < STAGES - 1; ++s) fetch();
    float acc[8][TN];
    int stage = 0;
#pragma unroll 1
    for (int chain = rank; chain < (PARTS == 1 ? CHAINS : rank + 1); ++chain) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll 1
        for (int run = chain; run < n_runs; run += CHAINS) {
            f32x2 part[8][TN];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) part[i][j] = 0ull;
#pragma unroll 1
            for (int half = 0; half < RUN / BK; ++half) {
                asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
                __syncthreads();      // this step has landed for every thread; the stage filled below was read a step ago
                fetch();
                const float* as = tiles + stage * STAGE + ty * PITCH;
                const float* ws = tiles + stage * STAGE + (BM + tx) * PITCH;
                stage = stage == STAGES - 1 ? 0 : stage + 1;
#pragma unroll
                for (int q = 0; q < BK / 4; ++q) {
                    ulonglong2 w[TN];
#pragma unroll
                    for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + 16 * j * PITCH + 4 * q);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + 8 * i * PITCH + 4 * q);
#pragma unroll
                        for (int j = 0; j < TN; ++j) {
                            fma2(part[i][j], a.x, w[j].x);
                            fma2(part[i][j], a.y, w[j].y);
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] += run_sum(part[i][j]);
        }
        if constexpr (PARTS == 1) {
            // the finished chains' sum: this thread's own sums
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float4* t = reinterpret_cast<float4*>(total) + i * 128 + tid;
                float4 v = chain == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : *t;
                v.x += acc[i][0]; v.y += acc[i][1]; v.z += acc[i][2]; v.w += acc[i][3];
                *t = v;
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if constexpr (PARTS == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int gm = m0 + ty + 8 * i;
            if (gm >= M) continue;
            const float4 v = reinterpret_cast<const float4*>(total)[i * 128 + tid];
            const float out[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int gn = n0 + tx + 16 * j;
                if (gn < N) C[(size_t)gm * ldc + gn] = bias ? out[j] + bias[gn] : out[j];
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) total[(ty + 8 * i) * BN + tx + 16 * j] = acc[i][j];
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        // eight rows of the tile per CTA, four neighbouring columns at a time; the chains in ascending order
        for (int e = tid; e < (BM / PARTS) * (BN / 4); e += 128) {
            const int row = rank * (BM / PARTS) + e / (BN / 4), col = 4 * (e % (BN / 4));
            const uint32_t mine = (uint32_t)__cvta_generic_to_shared(total + row * BN + col);
            float out[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < PARTS; ++c) {
                uint32_t at;
                float4 v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine), "r"(c));
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
                out[0] += v.x; out[1] += v.y; out[2] += v.z; out[3] += v.w;
            }
            const int gm = m0 + row;
            if (gm >= M) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int gn = n0 + col + j;
                if (gn < N) C[(size_t)gm * ldc + gn] = bias ? out[j] + bias[gn] : out[j];
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");     // no CTA leaves while another reads its tile
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// ---------------------------------------------------------------------------
// Few rows: bound by reading the weights.  A CTA owns 16 output features; a stage is 256 k (a run of each chain: 1 KB
// of every weight row and of every row of A) in a ring of cp.async copies, 16 KB of weights each, so that even a
// product of few features has some 50 KB in flight on every SM.  A thread owns one chain of F features x MR rows.  Shared
// memory is what comes next after the memory: runs are 36 floats apart and rows 292, so that eight
// neighbouring threads (features of one run) and the runs of a warp fall on different banks.  Measured (M x N x K, weights
// read at): 4 x 37888 x 3584: 226 -> 119 us (4.6 TB/s); 4 x 3584 x 18944: 185 -> 70 us (3.9 TB/s); 8 x 3584 x 18944: 184 -> 97 us;
// 12 x 3584 x 18944: 723 -> 138 us; 32 x 3584 x 18944: 441 -> 213 us (a stage was one run of 32 k, a CTA's threads all walked it).
// ---------------------------------------------------------------------------
// SHORT: K fits into one stage.  A CTA then takes one of `row_tiles` tiles of MT rows (their weights are read once more from the L2
// cache, which is less than what a CTA loses on rows it walks one after another), and runs past K are neither copied nor multiplied.
template <int MR, int F, int GROUPS, int STAGES, bool VEC, bool SHORT>
__global__ void __launch_bounds__(CHAINS * 16 / F * GROUPS)
sgemm_nt_stream_kernel(const float* A, long long lda, const float* W, long long ldw,
                       float* C, long long ldc, const float* bias, int M, int N, int K, int row_tiles) {
    constexpr int FN = 16, FT = FN / F, MT = MR * GROUPS, THREADS = CHAINS * FT * GROUPS;
    constexpr int RUN_PITCH = RUN + 4, ROW = CHAINS * RUN_PITCH + 4, KS = RUN * CHAINS;
    constexpr int STAGE = (FN + MT) * ROW, STEP = THREADS / 64;
    static_assert(CHAINS * MT * FN <= STAGE * STAGES && THREADS % 64 == 0 && FN % STEP == 0 && KS % THREADS == 0, "copies and the last sum fit");
    extern __shared__ __align__(16) float ring[];
    pdl_trigger();
    const int tid = threadIdx.x;
    const int ft = tid % FT, chain = tid / FT % CHAINS, group = tid / (FT * CHAINS);
    const int n0 = (SHORT ? blockIdx.x / row_tiles : blockIdx.x) * FN;
    if (SHORT) {
        const int m0 = blockIdx.x % row_tiles * MT;
        A += (size_t)m0 * lda;
        C += (size_t)m0 * ldc;
        M -= m0;
    }
    const int n_steps = (K + KS - 1) / KS;
    // copies: VEC: a thread fetches quad cq of the rows cr, cr + STEP, ...; else a warp 32 neighbouring floats of a row
    const int cq = tid & 63, cr = tid >> 6;
    float* const to = ring + (cq >> 3) * RUN_PITCH + (cq & 7) * 4;
    // row r of `live` ones, on row `at` of the stage; rows outside the matrices are not stored: whatever their sums are
    auto load_scalars = [&](const float* from, long long ld, int rows, int live, int at, int t, int st) {
#pragma unroll 1
        for (int r = 0; r < min(rows, live); ++r) {
            float* dst = ring + st * STAGE + (at + r) * ROW;
            const float* src = from + (size_t)r * ld;
#pragma unroll
            for (int k = tid; k < KS; k += THREADS) {
                const int gk = t * KS + k;
                if (SHORT && gk - k % RUN >= K) continue;      // a run past the end
                copy4(dst + (k / RUN) * RUN_PITCH + k % RUN, gk < K ? src + gk : src, gk < K);
            }
        }
    };
    auto load_w = [&](int t, int st) {
        const int gk = t * KS + 4 * cq;
        const bool live = gk < K;
        if (t >= n_steps) return;
        if constexpr (VEC) {
            if (SHORT && gk - 4 * (cq & 7) >= K) return;      // a run past the end
#pragma unroll
            for (int r = cr; r < FN; r += STEP)
                if (n0 + r < N) copy16(to + st * STAGE + r * ROW, live ? W + (size_t)(n0 + r) * ldw + gk : W, live);
        } else load_scalars(W + (size_t)n0 * ldw, ldw, FN, N - n0, 0, t, st);
    };
    auto load_a = [&](int t, int st) {
        const int gk = t * KS + 4 * cq;
        const bool live = gk < K;
        if (t >= n_steps) return;
        if constexpr (VEC) {
            if (SHORT && gk - 4 * (cq & 7) >= K) return;
            for (int r = cr; r < MT; r += STEP)
                if (r < M) copy16(to + st * STAGE + (FN + r) * ROW, live ? A + (size_t)r * lda + gk : A, live);
        } else load_scalars(A, lda, MT, M, FN, t, st);
    };
    // the weights depend on no earlier kernel: their first stages are on their way before the wait
    for (int s = 0; s < STAGES - 1; ++s) load_w(s, s);
    pdl_wait();
    for (int s = 0; s < STAGES - 1; ++s) {
        load_a(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[MR][F];
#pragma unroll
    for (int i = 0; i < MR; ++i)
#pragma unroll
        for (int j = 0; j < F; ++j) acc[i][j] = 0.f;
    int st = 0, fill = STAGES - 1;
    for (int t = 0; t < n_steps; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();      // this stage has landed for every thread; the stage refilled below was read a step ago
        load_w(t + STAGES - 1, fill);
        load_a(t + STAGES - 1, fill);
        fill = fill == STAGES - 1 ? 0 : fill + 1;
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* ws = ring + st * STAGE + ft * ROW + chain * RUN_PITCH;
        const float* as = ring + st * STAGE + (FN + group * MR) * ROW + chain * RUN_PITCH;
        st = st == STAGES - 1 ? 0 : st + 1;
        if (SHORT && chain * RUN >= K) continue;
        f32x2 part[MR][F];
#pragma unroll
        for (int i = 0; i < MR; ++i)
#pragma unroll
            for (int j = 0; j < F; ++j) part[i][j] = 0ull;
#pragma unroll
        for (int q = 0; q < RUN / 4; ++q) {
            ulonglong2 w[F];
#pragma unroll
            for (int j = 0; j < F; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + j * FT * ROW + 4 * q);
#pragma unroll
            for (int i = 0; i < MR; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + i * ROW + 4 * q);
#pragma unroll
                for (int j = 0; j < F; ++j) {
                    fma2(part[i][j], a.x, w[j].x);
                    fma2(part[i][j], a.y, w[j].y);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < MR; ++i)
#pragma unroll
            for (int j = 0; j < F; ++j) acc[i][j] += run_sum(part[i][j]);
    }
    // the chains in ascending order, through the ring's memory
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MR; ++i)
#pragma unroll
        for (int j = 0; j < F; ++j) ring[(chain * MT + group * MR + i) * FN + ft + j * FT] = acc[i][j];
    __syncthreads();
    for (int e = tid; e < MT * FN; e += THREADS) {
        const int m = e / FN, n = n0 + e % FN;
        if (m >= M || n >= N) continue;
        float out = 0.f;
#pragma unroll
        for (int c = 0; c < CHAINS; ++c) out += ring[c * MT * FN + e];
        C[(size_t)m * ldc + n] = bias ? out + bias[n] : out;
    }
}

template <int MR, int F, int GROUPS, int STAGES, bool VEC, bool SHORT = false>
static int launch_stream(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc,
                         const float* bias, int M, int N, int K, cudaStream_t stream) {
    constexpr int BYTES = STAGES * (16 + MR * GROUPS) * (CHAINS * (RUN + 4) + 4) * 4;
    static_assert(BYTES <= 232448, "the ring does not fit into shared memory");
    static bool configured_on[PYRE_MAX_DEVICES] = {};      // the attribute is per device
    bool& configured = configured_on[pyre_current_device()];
    auto kernel = sgemm_nt_stream_kernel<MR, F, GROUPS, STAGES, VEC, SHORT>;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BYTES);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int row_tiles = SHORT ? ceil_div(M, MR * GROUPS) : 1;
    return (int)pyre_launch(kernel, dim3(ceil_div(N, 16) * row_tiles), dim3(CHAINS * 16 / F * GROUPS), (size_t)BYTES, stream,
                            A, lda, W, ldw, C, ldc, bias, M, N, K, row_tiles);
}

template <int PARTS, bool VEC>
static int launch_tiles_as(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc,
                           const float* bias, int M, int N, int K, cudaStream_t stream) {
    constexpr int BYTES = (TILE_STAGES * 2 * TILE * 20 + TILE * TILE) * 4;
    static bool configured_on[PYRE_MAX_DEVICES] = {};      // the attribute is per device
    bool& configured = configured_on[pyre_current_device()];
    auto kernel = sgemm_nt_tiles_kernel<PARTS, VEC>;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BYTES);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int tiles_m = ceil_div(M, TILE);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((long long)tiles_m * ceil_div(N, TILE) * PARTS));
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = PARTS;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = pyre_pdl_enabled() ? attr : attr + 1;
    cfg.numAttrs = (pyre_pdl_enabled() ? 1 : 0) + (PARTS > 1 ? 1 : 0);
    return (int)cudaLaunchKernelEx(&cfg, kernel, A, lda, W, ldw, C, ldc, bias, M, N, K, tiles_m);
}

template <bool VEC>
static int launch_tiles(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc,
                        const float* bias, int M, int N, int K, cudaStream_t stream) {
    const long long tiles = (long long)ceil_div(M, TILE) * ceil_div(N, TILE);
    const int sms = pyre_sm_count();
    // A CTA per chain where whole tiles would leave the SMs unevenly loaded (the busiest has ceil(tiles / SMs) of them) and
    // a chain is long enough (four runs) to pay for the cluster's meeting
    const long long busiest = (tiles + sms - 1) / sms;
    if (K >= 4 * RUN * CHAINS && busiest * sms * 10 > tiles * 11)
        return launch_tiles_as<CHAINS, VEC>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
    return launch_tiles_as<1, VEC>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
}

template <bool VEC>
static int launch_product(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc,
                          const float* bias, int M, int N, int K, cudaStream_t stream) {
    // up to a stage's K: tiles of 4 or 8 rows (M x N x K, tiles of 16 or 32 rows and four times the shared memory /
    // so: 8 x 64 x 64: 1.89 / 1.72 us, 16 x 512 x 64: 2.57 / 1.89, 32 x 512 x 64: 3.26 / 1.89, 32 x 64 x 176: 3.05 / 1.89)
    if (K <= RUN * CHAINS && M <= 4) return launch_stream<4, 1, 1, 2, VEC, true>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
    if (K <= RUN * CHAINS && M <= 32) return launch_stream<8, 1, 1, 2, VEC, true>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
    if (M <= 4) return launch_stream<4, 1, 1, 4, VEC>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
    if (M <= 8) return launch_stream<8, 1, 1, 4, VEC>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
    if (M <= 16) return launch_stream<8, 2, 2, 3, VEC>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
    if (M <= 32) return launch_stream<8, 2, 4, 2, VEC>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
    return launch_tiles<VEC>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
}

PYRE_API int pyre_sgemm_nt(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc,
                           const float* bias, int M, int N, int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K < 0) return PYRE_ERR_BAD_ARG;
    // 16-byte copies need aligned rows in both operands
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && !((uintptr_t)A & 15) && !((uintptr_t)W & 15);
    const int rc = vec ? launch_product<true>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream)
                       : launch_product<false>(A, lda, W, ldw, C, ldc, bias, M, N, K, stream);
    if (rc) return rc;
    PYRE_LAUNCH_CHECK();
    return 0;
}
