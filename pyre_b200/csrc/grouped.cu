// Products with one weight matrix per GROUP, and the small kernels of a routed feed-forward around them.
//
//   out[dst(p), g-th slice] = x[src(p), g-th slice] . w[g]^T        w[g] is [N, K] (a linear layer's layout)
//
// Two ways to say which rows belong to a group:
//   * every group takes all M rows (a product per HEAD: x and out hold the heads side by side in a row, each
//     group reads its own K columns and writes its own N columns);
//   * the rows are sorted by group, group g owning the sorted places offsets[g] .. offsets[g + 1] (a product per
//     EXPERT of a routed feed-forward: `src` gathers a place's input row, `dst` says where its result goes).
//
// One CTA computes a tile of a group's result.  float32: 64 x 64, FFMA, one chain per output element over k in
// ascending order, so a row's result does not depend on which other rows share its tile or its launch.
// bfloat16 operands: on the tensor cores with fp32 accumulators, by the rows per group on average: up to 16 of them tiles of
// 16 rows x 64 features, below 96 (or with K below 64) tiles of 64 x 64, both by mma.sync m16n8k16 (a weight stream), else 128 x 128 by
// tcgen05.mma.  The two instructions add the products of a k step in different orders: a bfloat16 row's last bits depend on which
// kernel takes its launch.
// `dtype`: type of x and w (0 = float32, 1 = bfloat16); `out_f32`: the result stays fp32, else it is rounded to dtype.
#include "common.cuh"

struct GroupedArgs {
    const void* x;
    long long x_row_stride, x_group_stride;   // in elements
    const void* w;
    long long w_group_stride;                 // in elements; rows of w[g] are K apart
    void* out;
    long long out_row_stride, out_group_stride;
    const int* offsets;   // [G + 1] sorted places per group, or null: every group takes rows 0 .. M - 1
    const int* src;       // [places] input row of a sorted place, or null: the place itself
    const int* dst;       // [places] output row of a sorted place, or null: the place itself
    int M, N, K, G;
    int out_f32;
};

constexpr int GB_M = 64, GB_N = 64, GB_K = 16;

// Which (group, first place, places) a CTA works on; false: nothing to do.
template <int TILE_M = 64>
__device__ __forceinline__ bool grouped_tile(const GroupedArgs& a, int& g, int& first, int& count) {
    constexpr int GB_M = TILE_M;
    if (!a.offsets) {
        g = blockIdx.z;
        first = blockIdx.x * GB_M;
        count = min(GB_M, a.M - first);
        return count > 0;
    }
    __shared__ int found[3];
    if (threadIdx.x < 32) {
        // a lane per group, 32 groups at a time: the tiles before a group by a scan over the lanes (one thread that walked
        // the groups waited for a load per group: some 8 us of a decode step's product at 32 groups)
        const int lane = threadIdx.x;
        int before = 0;
        if (lane == 0) found[0] = -1;
        __syncwarp();
        for (int g0 = 0; g0 < a.G; g0 += 32) {
            const int gg = g0 + lane;
            const int lo = gg < a.G ? a.offsets[gg] : 0, n = gg < a.G ? a.offsets[gg + 1] - lo : 0;
            const int tiles = (n + GB_M - 1) / GB_M;
            int upto = tiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const int tile = (int)blockIdx.x - before - (upto - tiles);       // within this lane's group
            if (tile >= 0 && tile < tiles) {
                found[0] = gg;
                found[1] = lo + tile * GB_M;
                found[2] = min(GB_M, n - tile * GB_M);
            }
            before += __shfl_sync(0xffffffffu, upto, 31);
            if (before > (int)blockIdx.x) break;
        }
    }
    __syncthreads();
    g = found[0];
    first = found[1];
    count = found[2];
    return g >= 0;
}

template <typename T>
__global__ void __launch_bounds__(256) grouped_linear_kernel(GroupedArgs a) {
    __shared__ float xs[GB_K][GB_M + 4];
    __shared__ float ws[GB_K][GB_N + 4];
    __shared__ int src_row[GB_M], dst_row[GB_M];
    pdl_trigger();
    pdl_wait();
    int g, first, count;
    if (!grouped_tile(a, g, first, count)) return;
    const int n0 = blockIdx.y * GB_N;
    if (threadIdx.x < GB_M) {
        const int p = first + threadIdx.x;
        const bool live = (int)threadIdx.x < count;
        src_row[threadIdx.x] = live ? (a.src ? a.src[p] : p) : -1;
        dst_row[threadIdx.x] = live ? (a.dst ? a.dst[p] : p) : -1;
    }
    __syncthreads();
    const T* x = (const T*)a.x + (size_t)g * a.x_group_stride;
    const T* w = (const T*)a.w + (size_t)g * a.w_group_stride;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    // loads: 64 rows x 16 k per operand = 1024 elements, four per thread: row = idx / 16, k = idx % 16
    for (int k0 = 0; k0 < a.K; k0 += GB_K) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int idx = threadIdx.x + u * 256;
            const int r = idx >> 4, k = idx & 15;
            const int sr = src_row[r];
            xs[k][r] = (sr >= 0 && k0 + k < a.K) ? to_f32<T>(x[(size_t)sr * a.x_row_stride + k0 + k]) : 0.f;
            ws[k][r] = (n0 + r < a.N && k0 + k < a.K) ? to_f32<T>(w[(size_t)(n0 + r) * a.K + k0 + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GB_K; ++k) {
            float xv[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) xv[i] = xs[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int dr = dst_row[ty * 4 + i];
        if (dr < 0) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= a.N) continue;
            const size_t at = (size_t)dr * a.out_row_stride + (size_t)g * a.out_group_stride + n;
            if (a.out_f32) ((float*)a.out)[at] = acc[i][j];
            else ((T*)a.out)[at] = from_f32<T>(acc[i][j]);
        }
    }
}

// ---------------------------------------------------------------------------
// bfloat16, groups of few rows: tiles of 64 features by mma.sync, bound by reading the weights (a decoded token's experts have a row
// or two each).  K in steps of 64 through a ring filled by cp.async, so that a CTA has up to 40 KB of weights in
// flight; each of the four warps owns 16 output features and as many 16-row pieces as the
// tile has rows, so that two rows do not cost the multiplications of 64.  Needs K % 8 == 0 and 16-byte aligned rows of x and w.
// Measured inside a decode step of 4 tokens (16 places of 32 experts, 2048 x 2048 and 2048 x 1024 weights), 64-row tiles one step
// ahead through registers / the ring with 64 rows: 95 / 28 us and 50 / 16 us; 64 tokens: 111 / 70 us.
// ROWS: the height of a tile.  Groups of few rows take tiles of 16 rows, whose ring holds little but weights; a group with more rows
// takes more tiles, whose weights then come out of the L2 cache.  32 experts of 2048 x 2048, top 4, captured launches one after the
// other, 64 rows of four stages / 16 rows of six / of four: 4 tokens 27.4 / 21.6 / 23.5 us, 8: 49.7 / 39.5 / 45.6, 32: 72.3 / 57.2 /
// 50.5, 128: 76.4 / 70.6 / 64.6.  The lines were drawn there; against the kernels with registers in 300 other cases (8 to 256 experts of
// 64 x 64 to 14336 x 4096, 1 to 2,240 tokens, top 2 and 4, also with all rows in four of the experts) no one got slower.
// ---------------------------------------------------------------------------
constexpr int GT_K = 64, GT_LD = GT_K + 8;   // padded rows: 144 bytes, conflict-free for ldmatrix
template <int ROWS, int STAGES> struct GtRing {
    static constexpr int STAGE = (ROWS + GB_N) * GT_LD, SMEM = STAGES * STAGE * 2;
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// a 16-byte copy into shared memory, or 16 bytes of zeros
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool live) {
    const int bytes = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Two neighbouring results of a row: one store where the row allows it.
__device__ __forceinline__ void store_pair(const GroupedArgs& a, size_t at, int n, float v0, float v1) {
    if (a.out_f32) {
        float* o = (float*)a.out + at;
        if (n + 1 < a.N && ((uintptr_t)o & 7) == 0) *reinterpret_cast<float2*>(o) = make_float2(v0, v1);
        else {
            if (n < a.N) o[0] = v0;
            if (n + 1 < a.N) o[1] = v1;
        }
    } else {
        __nv_bfloat16* o = (__nv_bfloat16*)a.out + at;
        if (n + 1 < a.N && ((uintptr_t)o & 3) == 0) *reinterpret_cast<__nv_bfloat162*>(o) = __floats2bfloat162_rn(v0, v1);
        else {
            if (n < a.N) o[0] = __float2bfloat16_rn(v0);
            if (n + 1 < a.N) o[1] = __float2bfloat16_rn(v1);
        }
    }
}

template <int ROWS, int GT_STAGES>
__global__ void __launch_bounds__(128, 3) grouped_linear_mma_kernel(GroupedArgs a) {
    constexpr int GT_STAGE = GtRing<ROWS, GT_STAGES>::STAGE;
    extern __shared__ __align__(16) __nv_bfloat16 g_ring[];      // [stages][ROWS rows of x, 64 rows of w][GT_LD]
    __shared__ int src_row[ROWS], dst_row[ROWS];
    pdl_trigger();
    const int n0 = blockIdx.y * GB_N;
    const int n_steps = (a.K + GT_K - 1) / GT_K;
    const int lr = threadIdx.x >> 3, lk = (threadIdx.x & 7) * 8;        // copies: rows lr, lr + 16, ..., eight threads to a row
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(g_ring);
    auto load_w = [&](const __nv_bfloat16* w, int s) {
        if (s >= n_steps) return;
        const uint32_t to = ring + ((s % GT_STAGES) * GT_STAGE + ROWS * GT_LD) * 2;
        const int k = s * GT_K + lk;
        const bool in_k = k < a.K;
#pragma unroll
        for (int r = lr; r < GB_N; r += 16)      // features past the end are not stored: whatever their sums are
            if (n0 + r < a.N) copy16(to + (r * GT_LD + lk) * 2, in_k ? w + (size_t)(n0 + r) * a.K + k : w, in_k);
    };
    int g = 0, first = 0, count = 0;
    if (!a.offsets) {      // the weights are known before the kernels before this one finish
        g = blockIdx.z;
        const __nv_bfloat16* w = (const __nv_bfloat16*)a.w + (size_t)g * a.w_group_stride;
        for (int s = 0; s < GT_STAGES - 1; ++s) load_w(w, s);
    }
    pdl_wait();
    if (!grouped_tile<ROWS>(a, g, first, count)) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    if (threadIdx.x < ROWS) {
        const int p = first + threadIdx.x;
        const bool live = (int)threadIdx.x < count;
        src_row[threadIdx.x] = live ? (a.src ? a.src[p] : p) : -1;
        dst_row[threadIdx.x] = live ? (a.dst ? a.dst[p] : p) : -1;
    }
    __syncthreads();
    const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + (size_t)g * a.x_group_stride;
    const __nv_bfloat16* w = (const __nv_bfloat16*)a.w + (size_t)g * a.w_group_stride;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m_tiles = (count + 15) / 16;
    auto load_x = [&](int s) {
        if (s >= n_steps) return;
        const uint32_t to = ring + (s % GT_STAGES) * GT_STAGE * 2;
        const int k = s * GT_K + lk;
        const bool in_k = k < a.K;
        for (int r = lr; r < count; r += 16)
            copy16(to + (r * GT_LD + lk) * 2, in_k ? x + (size_t)src_row[r] * a.x_row_stride + k : x, in_k);
    };
    for (int s = 0; s < GT_STAGES - 1; ++s) {
        if (a.offsets) load_w(w, s);
        load_x(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[ROWS / 16][2][4];
#pragma unroll
    for (int i = 0; i < ROWS / 16; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    for (int s = 0; s < n_steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GT_STAGES - 2) : "memory");
        __syncthreads();      // this step has landed for every thread; the stage filled below was read a step ago
        load_w(w, s + GT_STAGES - 1);
        load_x(s + GT_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const __nv_bfloat16* xs = g_ring + (s % GT_STAGES) * GT_STAGE;
        const __nv_bfloat16* ws = xs + (ROWS + warp * 16) * GT_LD;
#pragma unroll
        for (int kk = 0; kk < GT_K; kk += 16) {
            uint32_t bf[4];      // 16 n-rows: two 8-wide n tiles, both k halves
            ldmatrix_x4(bf, ws + ((lane & 7) + ((lane >> 4) << 3)) * GT_LD + kk + ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int i = 0; i < ROWS / 16; ++i) {
                if (i < m_tiles) {
                    uint32_t af[4];
                    ldmatrix_x4(af, xs + (i * 16 + (lane & 15)) * GT_LD + kk + (lane >> 4) * 8);
                    mma_bf16(acc[i][0], af, bf[0], bf[1]);
                    mma_bf16(acc[i][1], af, bf[2], bf[3]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < ROWS / 16; ++i)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int dr = dst_row[i * 16 + (lane >> 2) + half * 8];
            if (dr < 0) continue;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int n = n0 + warp * 16 + j * 8 + (lane & 3) * 2;
                store_pair(a, (size_t)dr * a.out_row_stride + (size_t)g * a.out_group_stride + n, n, acc[i][j][half * 2], acc[i][j][half * 2 + 1]);
            }
        }
}

// ---------------------------------------------------------------------------
// The same product for groups of many rows, on the 5th-generation tensor cores: 128 rows x 128 features per CTA, fp32
// accumulators in tensor memory, K in steps of 64 through a ring of three 32 KB stages; two CTAs fit on an SM, so that one
// drains its result while the other multiplies.
//   warps 0..3 : bring the rows of x (gathered) and of w into the ring by cp.async, 128-byte rows with the 128-byte swizzle
//                (16-byte piece c of row r lies at c ^ (r & 7)), and tell the MMA thread when a stage has landed; then the
//                epilogue, a row per thread.  (TMA would need a tensor map per launch and cannot gather rows cheaper.)
//   warp 4     : allocates tensor memory; one thread issues tcgen05.mma (M = 128, N = 128, four of K = 16 per stage).
// Bound by what an SM can load: 32 KB per 128 x 128 x 64 products.  Measured: 2,240 tokens, top 4 of
// 32 experts, 2048 x 2048: 336 -> 126 us (559 TFLOP/s), 2048 x 1024: 195 -> 72 us (mma.sync before); handing a stage over two
// copies later instead of one costs 155 us, six stages and one CTA per SM 208 us.  2,240 tokens x 16 heads of 256 x 128: 29 -> 14 us.
// Every wait on an mbarrier is bounded; if one runs out, the error flag is raised, nothing is stored, and the tensor
// memory is freed.
// ---------------------------------------------------------------------------
constexpr int GL_M = 128, GL_N = 128, GL_K = 64, GL_STAGES = 3, GL_THREADS = 160;
constexpr int GL_AHEAD = 1;      // a stage is handed over once the next one's copies are on their way
constexpr int GL_STAGE = (GL_M + GL_N) * GL_K * 2;                 // bytes
constexpr int GL_BARS = GL_STAGES * GL_STAGE;                      // full[], empty[], accumulator full
constexpr int GL_SMEM = GL_BARS + (2 * GL_STAGES + 1) * 8 + 1024;  // and what brings the ring to a 1024-byte boundary
constexpr int GL_ERR_TIMEOUT = 2;

__device__ __forceinline__ bool gl_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool gl_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err_flag) {
    if (gl_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t it = 1;; ++it) {
        if (gl_try_wait(bar, parity)) return true;
        if ((it & 63) == 0) {
            if (*abort_flag) return false;
            if (clock64() - t0 > PYRE_WAIT_CYCLES) break;
        }
    }
    *abort_flag = 1;
    if (err_flag) atomicExch(err_flag, GL_ERR_TIMEOUT);
    return false;
}
// K-major operand of 128-byte rows with the 128-byte swizzle: stride byte offset 1024 (eight rows), version 1, layout type 2
__device__ __forceinline__ uint64_t gl_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__global__ void __launch_bounds__(GL_THREADS, 2) grouped_linear_tc_kernel(GroupedArgs a, int* err_flag) {
    extern __shared__ uint8_t gl_raw[];
    __shared__ int src_row[GL_M], dst_row[GL_M];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    const uint32_t base = ((uint32_t)__cvta_generic_to_shared(gl_raw) + 1023u) & ~1023u;
    const uint32_t bar_full = base + GL_BARS, bar_empty = bar_full + 8 * GL_STAGES, bar_acc = bar_empty + 8 * GL_STAGES;
    volatile int* abort_flag = &abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_wait();
    int g, first, count;
    if (!grouped_tile<GL_M>(a, g, first, count)) return;      // the whole CTA, before anything is set up
    const int n0 = blockIdx.y * GL_N;
    if (threadIdx.x < GL_M) {
        const int p = first + threadIdx.x;
        const bool live = (int)threadIdx.x < count;
        src_row[threadIdx.x] = live ? (a.src ? a.src[p] : p) : -1;
        dst_row[threadIdx.x] = live ? (a.dst ? a.dst[p] : p) : -1;
    }
    if (threadIdx.x == 0) {
        abort_word = 0;
        for (int s = 0; s < GL_STAGES; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar_full + 8 * s), "r"(128) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar_empty + 8 * s), "r"(1) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar_acc), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&tmem_slot)), "r"(GL_N) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *(volatile uint32_t*)&tmem_slot;
    pdl_trigger();      // only now: a later kernel's CTA must not find tensor memory that this one has yet to take
    const int n_steps = (a.K + GL_K - 1) / GL_K;

    if (warp < 4) {
        const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + (size_t)g * a.x_group_stride;
        const __nv_bfloat16* w = (const __nv_bfloat16*)a.w + (size_t)g * a.w_group_stride;
        const int lr = threadIdx.x >> 3, piece = threadIdx.x & 7;       // rows lr, lr + 16, ..., eight threads to a row
        // where this thread's pieces come from: worked out once, the issue of copies is what bounds the loaders
        constexpr int PER = GL_M / 16;
        const __nv_bfloat16* xp[PER];
        const __nv_bfloat16* wp[PER];
        uint32_t x_live = 0, w_live = 0;      // rows and features past the end are not stored: whatever their sums are
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int r = lr + 16 * i;
            x_live |= (uint32_t)(r < count) << i;
            w_live |= (uint32_t)(n0 + r < a.N) << i;
            xp[i] = x + (size_t)max(src_row[r], 0) * a.x_row_stride + piece * 8;
            wp[i] = w + (size_t)min(n0 + r, a.N - 1) * a.K + piece * 8;
        }
        const uint32_t at0 = lr * 128 + ((piece ^ (lr & 7)) << 4);      // rows 16 apart lie 2048 bytes apart, swizzled alike
        bool alive = true;
        for (int s = 0; s < n_steps + GL_AHEAD && alive; ++s) {
            if (s < n_steps) {
                const int st = s % GL_STAGES;
                if (s >= GL_STAGES) alive = gl_wait(bar_empty + 8 * st, (s / GL_STAGES - 1) & 1, abort_flag, err_flag);
                if (!alive) break;
                const uint32_t xs = base + st * GL_STAGE, ws = xs + GL_M * GL_K * 2;
                const int k = s * GL_K;
                const bool in_k = k + piece * 8 < a.K;
                const int from = in_k ? k : 0;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    if (x_live >> i & 1) copy16(xs + at0 + i * 2048, xp[i] + from, in_k);
                    if (w_live >> i & 1) copy16(ws + at0 + i * 2048, wp[i] + from, in_k);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (s >= GL_AHEAD) {
                asm volatile("cp.async.wait_group %0;" ::"n"(GL_AHEAD) : "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // what this thread brought, for the tensor core
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_full + 8 * ((s - GL_AHEAD) % GL_STAGES)) : "memory");
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        // ---- epilogue: the thread's row
        alive = alive && gl_wait(bar_acc, 0, abort_flag, err_flag) && !*abort_flag;
        alive = __all_sync(0xffffffffu, alive);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int dr = dst_row[threadIdx.x];
        const size_t at = (size_t)(dr < 0 ? 0 : dr) * a.out_row_stride + (size_t)g * a.out_group_stride + n0;
        const int esize = a.out_f32 ? 4 : 2;
        const bool wide = (((uintptr_t)a.out + at * esize) & 31) == 0;
        if (alive) {
#pragma unroll 1
            for (int c = 0; c < GL_N; c += 16) {
                uint32_t r[16];
                __syncwarp();
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                    : "r"(tmem + c + ((uint32_t)(warp * 32) << 16)) : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (dr < 0 || n0 + c >= a.N) continue;
                if (wide && n0 + c + 16 <= a.N) {      // 32 bytes per request: whole sectors
                    if (a.out_f32) {
                        float* o = (float*)a.out + at + c;
#pragma unroll
                        for (int h = 0; h < 16; h += 8)
                            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + h), "r"(r[h]), "r"(r[h + 1]), "r"(r[h + 2]),
                                         "r"(r[h + 3]), "r"(r[h + 4]), "r"(r[h + 5]), "r"(r[h + 6]), "r"(r[h + 7]) : "memory");
                    } else {
                        uint32_t p[8];
#pragma unroll
                        for (int h = 0; h < 8; ++h) {
                            const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(r[2 * h]), __uint_as_float(r[2 * h + 1]));
                            p[h] = *reinterpret_cast<const uint32_t*>(&v);
                        }
                        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"((__nv_bfloat16*)a.out + at + c), "r"(p[0]), "r"(p[1]),
                                     "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]) : "memory");
                    }
                } else {
#pragma unroll
                    for (int h = 0; h < 16; ++h) {
                        if (n0 + c + h >= a.N) continue;
                        if (a.out_f32) ((float*)a.out)[at + c + h] = __uint_as_float(r[h]);
                        else ((__nv_bfloat16*)a.out)[at + c + h] = __float2bfloat16_rn(__uint_as_float(r[h]));
                    }
                }
            }
        }
    } else if (lane == 0) {
        // D fp32 (bit 4), A and B bf16 (bits 7, 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(GL_N >> 3) << 17) | ((uint32_t)(GL_M >> 4) << 24);
        for (int s = 0; s < n_steps; ++s) {
            const int st = s % GL_STAGES;
            if (!gl_wait(bar_full + 8 * st, (s / GL_STAGES) & 1, abort_flag, err_flag)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t da = gl_desc(base + st * GL_STAGE), db = gl_desc(base + st * GL_STAGE + GL_M * GL_K * 2);
#pragma unroll
            for (int k = 0; k < GL_K / 16; ++k)      // 16 bf16 = 32 bytes = 2 descriptor units along K
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    ::"r"(tmem), "l"(da + 2 * k), "l"(db + 2 * k), "r"(idesc), "r"((s > 0 || k > 0) ? 1u : 0u) : "memory");
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_empty + 8 * st) : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_acc) : "memory");      // also when it gave up
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 4) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(GL_N) : "memory");
    }
}

// A kernel with more dynamic shared memory than the default allows (the attribute is per device).
template <typename K>
static int allow_smem(K kernel, int bytes, bool (&done)[PYRE_MAX_DEVICES]) {
    bool& configured = done[pyre_current_device()];
    if (configured) return 0;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) configured = true;
    return (int)e;
}

// places: an upper bound of the sorted places (the host does not know the groups' sizes); with offsets == null it is unused
PYRE_API int pyre_grouped_linear(const void* x, long long x_row_stride, long long x_group_stride, const void* w,
                                 long long w_group_stride, void* out, long long out_row_stride, long long out_group_stride,
                                 const int* offsets, const int* src, const int* dst, int M, int N, int K, int G, int places,
                                 int out_f32, int dtype, int use_mma, int* err_flag, cudaStream_t stream) {
    if (N <= 0 || K <= 0 || G <= 0) return PYRE_ERR_BAD_ARG;
    GroupedArgs a{x, x_row_stride, x_group_stride, w, w_group_stride, out, out_row_stride, out_group_stride,
                  offsets, src, dst, M, N, K, G, out_f32};
    if ((offsets ? places : M) <= 0) return 0;
    auto tiles_of = [&](int rows, int features) {
        return offsets ? dim3(ceil_div(places, rows) + G, ceil_div(N, features), 1) : dim3(ceil_div(M, rows), ceil_div(N, features), G);
    };
    const dim3 grid = tiles_of(GB_M, GB_N);
    if (dtype == PYRE_BF16 && use_mma) {
        if (K % 8 || x_row_stride % 8 || x_group_stride % 8 || w_group_stride % 8 || (((uintptr_t)x | (uintptr_t)w) & 15))
            return PYRE_ERR_UNSUPPORTED;
        // by the rows per group on average: about a hundred or more (a prompt portion's heads or experts), tcgen05 on tiles of 128;
        // up to 16, tiles of 16 rows, with the deeper ring where nearly every group has one tile of a row or two (the figures
        // stand with the kernels)
        const long long rows_per_group = offsets ? (long long)places / G : M;
        auto small = [&](auto kernel, int rows, int smem, bool (&done)[PYRE_MAX_DEVICES]) {
            if (const int rc = allow_smem(kernel, smem, done)) return rc;
            return (int)pyre_launch(kernel, tiles_of(rows, GB_N), dim3(128), (size_t)smem, stream, a);
        };
        static bool done_tc[PYRE_MAX_DEVICES] = {}, done_64[PYRE_MAX_DEVICES] = {}, done_16[PYRE_MAX_DEVICES] = {}, done_16d[PYRE_MAX_DEVICES] = {};
        int rc;
        if (rows_per_group >= 96 && K >= GL_K) {      // a K below one step: setting up tensor memory costs more than it saves (2,240 rows of 4 heads, 32 x 24: 3.6 us by it, 3.3 without)
            rc = allow_smem(grouped_linear_tc_kernel, GL_SMEM, done_tc);
            if (!rc) rc = (int)pyre_launch(grouped_linear_tc_kernel, tiles_of(GL_M, GL_N), dim3(GL_THREADS), (size_t)GL_SMEM, stream, a, err_flag);
        } else if (rows_per_group > 16) rc = small(grouped_linear_mma_kernel<64, 4>, 64, GtRing<64, 4>::SMEM, done_64);
        else if (rows_per_group > 2) rc = small(grouped_linear_mma_kernel<16, 4>, 16, GtRing<16, 4>::SMEM, done_16);
        else rc = small(grouped_linear_mma_kernel<16, 6>, 16, GtRing<16, 6>::SMEM, done_16d);
        if (rc) return rc;
    } else if (dtype == PYRE_BF16) pyre_launch(grouped_linear_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, a);
    else if (dtype == PYRE_F32) pyre_launch(grouped_linear_kernel<float>, grid, dim3(256), 0, stream, a);
    else return PYRE_ERR_BAD_ARG;
    PYRE_LAUNCH_CHECK();
    return 0;
}

// ---------------------------------------------------------------------------
// The router of a routed feed-forward.  Per token: logits z = W h over all `n_out` router outputs in fp32 (W fp32
// [n_out, H]; h in the activation dtype), scores s = softmax(z), choice scores s + correction; the `top` outputs
// with the largest choice scores are chosen (the lowest index wins a tie), and each chosen output's weight is its
// plain score s times `scale` (not renormalised).  `sigmoid` != 0: the scores are s = sigmoid(z), each output by itself,
// instead of the softmax.  `bias` (fp32 [n_out] or null) is added to the logits before anything else.  `renorm` != 0: the
// chosen outputs' weights are divided by their sum + renorm_eps (with softmax scores: the softmax over the chosen logits alone).
// `groups` > 1: the outputs form so many equal groups of neighbours; a group's score is the sum of its two largest choice
// scores (of its one, if it has only one), and only outputs of the `keep` groups with the largest scores (the lowest index
// wins a tie) can be chosen.
// One block per token, one warp per output in turn.
//   idx_out [T, top] int32, weight_out [T, top] fp32
// ---------------------------------------------------------------------------
template <typename T>
__global__ void route_kernel(const T* h, const float* w, const float* correction, const float* bias, int* idx_out,
                             float* weight_out, int H, int n_out, int top, float scale, int sigmoid, int renorm, float renorm_eps,
                             int groups, int keep) {
    extern __shared__ float z_smem[];   // [n_out] logits, then scores; [n_out] choice scores; [groups] group scores
    pdl_trigger();
    // four blocks ask for the router's rows (a few hundred KB) while they wait; with the loads of a row unrolled by eight:
    // 18.8 -> 15.6 us a launch on average (34 outputs of 2,048 columns, steps of 4 tokens and one prompt)
    if (blockIdx.x < 4) {
        prefetch_floats(w, n_out * H, blockIdx.x * blockDim.x + threadIdx.x, 4 * blockDim.x);
        if (blockIdx.x == 0) prefetch_floats(correction, n_out, threadIdx.x, blockDim.x);
    }
    pdl_wait();
    const int t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const T* hr = h + (size_t)t * H;
    float* z = z_smem;
    float* choice = z_smem + n_out;
    // which columns a lane adds depends on H and the pointers' alignment only, never on the batch
    const bool vec = H % 128 == 0 && (((uintptr_t)hr | (uintptr_t)w) & 15) == 0;
    for (int e = warp; e < n_out; e += warps) {
        const float* wr = w + (size_t)e * H;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        if (vec) {
#pragma unroll 8
            for (int i = lane * 4; i < H; i += 128) {
                const Vec<T, 4> hv = load_vec<T, 4>(hr + i);
                const Vec<float, 4> wv = load_vec<float, 4>(wr + i);
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[k] = fmaf(to_f32<T>(hv.v[k]), wv.v[k], acc[k]);
            }
        } else {
            for (int i = lane; i < H; i += 32) acc[0] = fmaf(to_f32<T>(hr[i]), wr[i], acc[0]);
        }
        const float sum = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
        if (lane == 0) z[e] = bias ? __fadd_rn(sum, bias[e]) : sum;
    }
    __syncthreads();
    if (warp == 0) {
        float sum = 1.f;
        if (sigmoid) {
            for (int e = lane; e < n_out; e += 32) z[e] = 1.0f / (1.0f + expf(-z[e]));
        } else {
            float mx = -INFINITY;
            for (int e = lane; e < n_out; e += 32) mx = fmaxf(mx, z[e]);
            mx = warp_max(mx);
            sum = 0.f;
            for (int e = lane; e < n_out; e += 32) {
                const float p = expf(z[e] - mx);
                z[e] = p;
                sum += p;
            }
            sum = warp_sum(sum);
        }
        __syncwarp();
        for (int e = lane; e < n_out; e += 32) {
            const float s = sigmoid ? z[e] : z[e] / sum;
            z[e] = s;
            choice[e] = s + (correction ? correction[e] : 0.f);
        }
        __syncwarp();
        if (groups > 1) {
            const int size = n_out / groups;
            float* gs = choice + n_out;
            for (int g = lane; g < groups; g += 32) {
                float first = -INFINITY, second = -INFINITY;
                for (int e = g * size; e < (g + 1) * size; ++e) {
                    const float c = choice[e];
                    if (c > first) { second = first; first = c; }
                    else if (c > second) second = c;
                }
                gs[g] = size > 1 ? first + second : first;
            }
            __syncwarp();
            for (int g = lane; g < groups; g += 32) {      // a group stays if fewer than `keep` groups come before it
                int before = 0;
                for (int o = 0; o < groups; ++o) before += (gs[o] > gs[g] || (gs[o] == gs[g] && o < g)) ? 1 : 0;
                if (before >= keep)
                    for (int e = g * size; e < (g + 1) * size; ++e) choice[e] = -INFINITY;
            }
            __syncwarp();
        }
        for (int k = 0; k < top; ++k) {
            float best = -INFINITY;
            int at = 0x7fffffff;
            for (int e = lane; e < n_out; e += 32) {
                const float c = choice[e];
                if (c > best) { best = c; at = e; }      // ascending e within a lane: the lowest index of equals stays
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oa = __shfl_xor_sync(0xffffffffu, at, o);
                if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
            }
            if (at >= n_out) at = 0;      // scores that are no numbers choose nothing
            if (lane == 0) {
                idx_out[(size_t)t * top + k] = at;
                weight_out[(size_t)t * top + k] = z[at] * scale;
                choice[at] = -INFINITY;
            }
            __syncwarp();
        }
        if (renorm && lane == 0) {
            float total = 0.f;
            for (int k = 0; k < top; ++k) total += weight_out[(size_t)t * top + k];
            for (int k = 0; k < top; ++k) weight_out[(size_t)t * top + k] = weight_out[(size_t)t * top + k] / (total + renorm_eps);
        }
    }
}

PYRE_API int pyre_route(const void* h, const float* w, const float* correction, const float* bias, int* idx_out, float* weight_out,
                        int n_tokens, int H, int n_out, int top, float scale, int sigmoid, int renorm, float renorm_eps, int groups,
                        int keep, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (H <= 0 || n_out <= 0 || top <= 0 || top > n_out) return PYRE_ERR_BAD_ARG;
    if (groups < 0 || (groups > 1 && (n_out % groups || keep <= 0 || top > (long long)keep * (n_out / groups)))) return PYRE_ERR_BAD_ARG;
    const size_t smem = ((size_t)2 * n_out + max(groups, 0)) * sizeof(float);
    if (smem > 48 * 1024) return PYRE_ERR_UNSUPPORTED;
    const int threads = n_tokens >= 512 ? 256 : 1024;      // few tokens: more warps per token's outputs
    if (dtype == PYRE_BF16)
        pyre_launch(route_kernel<__nv_bfloat16>, dim3(n_tokens), dim3(threads), smem, stream, (const __nv_bfloat16*)h, w, correction,
                    bias, idx_out, weight_out, H, n_out, top, scale, sigmoid, renorm, renorm_eps, groups, keep);
    else if (dtype == PYRE_F32)
        pyre_launch(route_kernel<float>, dim3(n_tokens), dim3(threads), smem, stream, (const float*)h, w, correction, bias, idx_out,
                    weight_out, H, n_out, top, scale, sigmoid, renorm, renorm_eps, groups, keep);
    else return PYRE_ERR_BAD_ARG;
    PYRE_LAUNCH_CHECK();
    return 0;
}

// ---------------------------------------------------------------------------
// Sorting the (token, choice) pairs by expert.  idx [pairs] holds each pair's chosen output; outputs from
// `n_experts` on have no weights (their result is the input itself) and get no place.
//   offsets [n_experts + 1]   first sorted place of every expert
//   place_of [pairs]          the pair's sorted place, or -1
//   src [pairs]               for a sorted place, the token whose row it reads (pair / top)
// One block; the places inside an expert's range are handed out by atomic counters (any order: a place's result
// does not depend on its neighbours).
// ---------------------------------------------------------------------------
__global__ void group_pairs_kernel(const int* idx, int n_pairs, int top, int n_experts, int* offsets, int* place_of, int* src) {
    extern __shared__ int counts[];   // [n_experts] counts, then cursors
    pdl_trigger();
    pdl_wait();
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) counts[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int e = idx[p];
        if (e >= 0 && e < n_experts) atomicAdd(&counts[e], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int e = 0; e < n_experts; ++e) {
            const int n = counts[e];
            offsets[e] = run;
            counts[e] = run;
            run += n;
        }
        offsets[n_experts] = run;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int e = idx[p];
        int place = -1;
        if (e >= 0 && e < n_experts) {
            place = atomicAdd(&counts[e], 1);
            src[place] = p / top;
        }
        place_of[p] = place;
    }
}

PYRE_API int pyre_group_pairs(const int* idx, int n_pairs, int top, int n_experts, int* offsets, int* place_of, int* src,
                              cudaStream_t stream) {
    if (n_experts <= 0 || top <= 0) return PYRE_ERR_BAD_ARG;
    if ((size_t)n_experts * sizeof(int) > 48 * 1024) return PYRE_ERR_UNSUPPORTED;
    pyre_launch(group_pairs_kernel, dim3(1), dim3(1024), (size_t)n_experts * sizeof(int), stream, idx, n_pairs, top, n_experts,
                offsets, place_of, src);
    PYRE_LAUNCH_CHECK();
    return 0;
}

// ---------------------------------------------------------------------------
// out[t] = sum_k weight[t, k] * (y[place_of[t, k]]  or, for an output without weights,  h[t]), k ascending, fp32.
//   y [places, H] fp32 results of the experts' last product; h [T, H] the feed-forward's input
// ---------------------------------------------------------------------------
template <typename T>
__global__ void combine_pairs_kernel(const float* y, const T* h, const int* place_of, const float* weight, float* out,
                                     size_t total, int H, int top) {
    pdl_trigger();
    pdl_wait();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x; at < total; at += stride) {
        const size_t t = at / H;
        const int i = (int)(at - t * H);
        float acc = 0.f;
        for (int k = 0; k < top; ++k) {
            const int place = place_of[t * top + k];
            const float v = place >= 0 ? y[(size_t)place * H + i] : to_f32<T>(h[at]);
            acc = fmaf(weight[t * top + k], v, acc);
        }
        out[at] = acc;
    }
}

PYRE_API int pyre_combine_pairs(const float* y, const void* h, const int* place_of, const float* weight, float* out,
                                int n_tokens, int H, int top, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0 || H <= 0) return 0;
    const size_t total = (size_t)n_tokens * H;
    const int blocks = (int)min((long long)pyre_sm_count() * 8, ceil_div_ll((long long)total, 256));
    if (dtype == PYRE_BF16)
        pyre_launch(combine_pairs_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, y, (const __nv_bfloat16*)h, place_of,
                    weight, out, total, H, top);
    else if (dtype == PYRE_F32)
        pyre_launch(combine_pairs_kernel<float>, dim3(blocks), dim3(256), 0, stream, y, (const float*)h, place_of, weight, out,
                    total, H, top);
    else return PYRE_ERR_BAD_ARG;
    PYRE_LAUNCH_CHECK();
    return 0;
}

// ---------------------------------------------------------------------------
// The experts' inputs of a routed feed-forward whose weights multiply what an expert READS:
//   out[place_of[t, k]] = T( weight[t, k] * h[t] )      for every pair with a place (place_of >= 0)
// out [places, H] in the order of the sorted places, so the products that follow read it without a gather.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void scale_to_places_kernel(const T* h, const int* place_of, const float* weight, T* out, size_t total, int H, int top) {
    pdl_trigger();
    pdl_wait();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x; at < total; at += stride) {
        const size_t pair = at / H;
        const int i = (int)(at - pair * H);
        const int place = place_of[pair];
        if (place >= 0) out[(size_t)place * H + i] = from_f32<T>(weight[pair] * to_f32<T>(h[(pair / top) * H + i]));
    }
}

PYRE_API int pyre_scale_to_places(const void* h, const int* place_of, const float* weight, void* out, int n_tokens, int H, int top,
                                  int dtype, cudaStream_t stream) {
    if (n_tokens <= 0 || H <= 0 || top <= 0) return 0;
    const size_t total = (size_t)n_tokens * top * H;
    const int blocks = (int)min((long long)pyre_sm_count() * 8, ceil_div_ll((long long)total, 256));
    if (dtype == PYRE_BF16)
        pyre_launch(scale_to_places_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, (const __nv_bfloat16*)h, place_of, weight, (__nv_bfloat16*)out, total, H, top);
    else if (dtype == PYRE_F32)
        pyre_launch(scale_to_places_kernel<float>, dim3(blocks), dim3(256), 0, stream, (const float*)h, place_of, weight, (float*)out, total, H, top);
    else return PYRE_ERR_BAD_ARG;
    PYRE_LAUNCH_CHECK();
    return 0;
}
