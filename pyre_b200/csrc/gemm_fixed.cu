// 32-bit matrix product in fixed point on the 5th-generation tensor cores:  C[M, N] = A[M, K] * W[N, K]^T, all float32.
//
// A row of either operand is taken as 31-bit integers on a power-of-two scale of its own, x = X 2^(E - 29) with E the
// exponent of the row's largest element (|X| <= 2^30), and X as four signed bytes, X = sum_p d_p 2^(8 (3 - p)).  Products of
// byte planes are summed by tcgen05.mma kind::i8 in 32-bit integers, exactly, planes i and j into the sum i + j; the sums
// 0 .. 4 (13 of the 16 products) make a 64-bit integer that is scaled and rounded to float.  An output is therefore
// off by the rounding to float, 2^-30 of the rows' largest elements per factor, and the products left out (some 2^-35 of the product of
// the two largest elements per term), where a chain of fused multiply-adds rounds with every term.
//
// A scale gives every element the bits that are left below the row's largest one.  That costs nothing where the large elements make the
// result, and everything where they meet small ones and the rest of the row makes it.  So:
//   * A token's elements of more than 2^OUTLIER_BITS times the mean magnitude (2 to the mean exponent of the elements that are not zero;
//     the mean is taken again without the ones found, until there are none) stay out of the integers as long as they are no more than
//     MAX_OUTLIERS: they are listed, and the epilogue adds their products with the float weights in double precision.
//   * A feature with an element of more than 2^WEIGHT_BITS times its mean magnitude has no scale; nor has a row with an infinity or a
//     NaN.  A weight with many such features should not come here (ops.linear_weight).
//   * The 128 outputs of a token in a tile are held against what the scales may have cost them (by the norms of the rows, see
//     `result_holds`).  If that is more than 2^-23 of their 2-norm, or if the token or a feature has no scale, the outputs are made again from
//     the float operands in double precision, after the CTA's last tile: nothing waits for them under a bounded wait.
// All are facts of the row and the weight alone, so that a row's result does not depend on what else is in the batch.
// Against 64 bits (2-norm of the error over 2-norm of the result, this / the sums of gemm_f32.cu): normal operands
// 2.5e-8 / 1.0e-7 (K = 512), 1.2e-7 (3,584), 1.8e-7 (18,944); 1 to 200 columns of A 16 to 1e25 times the others and those of W by as much
// less 2.5e-8 to 7.8e-8 / the same; log-normal activations up to e^(3 x) 2.5e-8 to 5.1e-8 / 0.9e-7 to 1.9e-7; where they come nearest, a share of 0.7 of A's
// columns a hundredth and the rest of W's, 1.0e-7 / 1.0e-7 (512), 1.1e-7 / 1.2e-7 (3,584).
// What it costs, us: ordinary and heavy-tailed rows nothing measurable from 64 rows on, 0.5 to 2.3 of 18 to 97 for 1 to 4 rows; per output and
// outlier 7 ps (509 x 37,888 x 3,584: 770, with four columns of outliers 1,310); outputs made again some 13 multiplications a cycle and SM (all of the same
// product: 20,400; one row in 64: 330 for 115).
//
// Integers add up in any order: a row's result has the same bits for any M, tile, split of K or order of arrival.
//
// Two kernels: the activations' exponents and byte planes (they are few), then the product.  The product's CTA (640 threads)
// owns 128 output features (the weights on the MMA's rows) and TN tokens, K in steps of 32:
//   warp 0, one thread  : TMA.  Weights as they are, 128 x 32 floats a step (128-byte swizzle), into one ring; the tokens' four
//                         byte planes, 128 k at a time, into another.
//   warps 4..19         : a thread owns a feature.  Groups of four warps take the steps in turn: 32 floats from shared memory,
//                         scaled, converted, transposed into byte planes (six instructions each) and stored to tensor
//                         memory, which is where the MMAs take their A operand from.  After the K loop the same threads
//                         put the five sums of their features together.
//   warp 1, one thread  : four MMAs a step, one per weight plane i, with the tokens' planes 0 .. 4 - i side by side as the N
//                         dimension: they add to the sums i .. 4, which lie side by side in the same order.
// Weights stay float32 in memory and are converted on the way, once per tile of tokens: with few tokens that hides behind the
// stream from memory, with many behind the MMAs.
#include "tensor_core.cuh"

namespace {
constexpr int ERR_TIMEOUT = 2;
constexpr int E_NONE = 1000;                   // of a row without a scale
constexpr int E_MIN = -98;                     // of a row of zeros (its scale is a normal float)
constexpr int OUTLIER_BITS = 7, WEIGHT_BITS = 6, MAX_OUTLIERS = 16;      // see above
constexpr int ROW_THREADS = 1024, ROW_WARPS = ROW_THREADS / 32;      // of the kernel in front
constexpr int FEATURES = 128, STEP = 32, BLOCK_K = 128;
constexpr int CONV_WARP0 = 4, GROUPS = 4, CONV_THREADS = GROUPS * 128, THREADS = CONV_WARP0 * 32 + CONV_THREADS;
constexpr int W_BYTES = FEATURES * STEP * 4;   // a step's weights
constexpr int A_STAGES = 6, A_COLS = 32;       // converted steps in tensor memory: 8 columns per plane

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err_flag) {
    return mbar_wait_or<ERR_TIMEOUT>(bar, parity, abort_flag, err_flag);
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// D (tensor memory, 32-bit integers) += A (tensor memory, signed bytes) * B (shared memory, signed bytes)
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}

// 2^e for e in [-126, 127]
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

// The exponent of a row from the largest |x| of its elements as bits (NaN above infinity above all numbers).
__device__ __forceinline__ int row_exponent(uint32_t abs_bits) {
    if (abs_bits >= 0x7f800000u) return E_NONE;
    if (abs_bits == 0) return E_MIN;
    const int e = (int)(abs_bits >> 23);
    return e ? e - 127 : 31 - __clz(abs_bits) - 149;
}
__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((e + 1023) << 20, 0); }
// x 2^(29 - E) as two factors: 29 - E reaches 178 for rows of the smallest numbers
struct RowScale {
    float s1, s2;
};
__device__ __forceinline__ RowScale row_scale(int E) {
    if (E >= E_NONE) return {0.f, 1.f};
    const int t = 29 - E;
    return {pow2f(min(t, 127)), t > 127 ? pow2f(t - 127) : 1.f};
}
// Four numbers already on their row's scale -> a word of four bytes for each plane.  Signed digits: adding 0x80 to the three lower bytes
// carries what they exceed 127 by, taking it off again byte by byte leaves digits in [-128, 127].
__device__ __forceinline__ void bytes_of(float x0, float x1, float x2, float x3, uint32_t& p0, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    const uint32_t y0 = (uint32_t)__float2int_rn(x0) + 0x808080u, y1 = (uint32_t)__float2int_rn(x1) + 0x808080u;
    const uint32_t y2 = (uint32_t)__float2int_rn(x2) + 0x808080u, y3 = (uint32_t)__float2int_rn(x3) + 0x808080u;
    const uint32_t a = __byte_perm(y0, y1, 0x5140), b = __byte_perm(y2, y3, 0x5140);      // bytes 0 and 1
    const uint32_t c = __byte_perm(y0, y1, 0x7362), d = __byte_perm(y2, y3, 0x7362);      // bytes 2 and 3
    p3 = __byte_perm(a, b, 0x5410) ^ 0x80808080u;
    p2 = __byte_perm(a, b, 0x7632) ^ 0x80808080u;
    p1 = __byte_perm(c, d, 0x5410) ^ 0x80808080u;
    p0 = __byte_perm(c, d, 0x7632);
}

// A token's word: its exponent in the lower half, the number of its outliers in the upper one.
__device__ __forceinline__ int exponent_of(int word) { return (short)word; }
__device__ __forceinline__ int outliers_of(int word) { return word >> 16; }

struct FixedParams {
    const float* A;
    const float* W;
    const int* w_exp;             // [N]
    const int* a_word;            // [M]
    const int2* outliers;         // [M][MAX_OUTLIERS]: k and the element's bits, by ascending k
    const float* w_norm;          // [N]: squares of the rows' 2-norms over those of their scales, 4^E
    const float* a_norm;          // [M][ROW_WARPS]: the same in parts (without outliers)
    float4* squares;              // [tiles][TN]: of the outputs over their scales, by quarters of the features (a CTA's last tile: in shared memory)
    float2* features;             // [items][4]: by quarters of the features, their norms and, as bits, how many have a scale (the sign: some have none)
    int* decided;                 // [items]: the item completed its tile (where K is split)
    unsigned long long* again;    // [items]: the tokens whose outputs are made from the float operands
    float* C;
    long long lda, ldw, ldc;
    int M, N, K;
    int tiles_m, tiles;           // tiles of tokens; of everything (tokens fastest: the tiles of a block of weights run together)
    int splits, steps_per_split;  // of K, in steps of 32 (a multiple of four per split)
    long long* partial;           // [splits][tiles][TN][128] where K is split
    int* counters;                // [tiles], zero
    int* err_flag;
};

// What a token's outliers add to an output, in the order of their list.
__device__ __forceinline__ double outlier_sum(const int2* list, int n, const float* w) {
    double sum = 0.;
#pragma unroll 1
    for (int i = 0; i < n; ++i) sum += (double)__int_as_float(list[i].y) * (double)w[list[i].x];
    return sum;
}

// Do a token's outputs in a tile, `squares` in all over 4^(Ea + Ew), have error enough to spare?  An element is off by 2^-29 / sqrt(12) of
// its row's scale (2-norm), so an output by that times the other row's norm, and by 6.9e-12 sqrt(K) for the byte products left out.  The bound is 2^-23 of
// the outputs' 2-norm, the size of the error that sums in 32 bits have; normal operands are off by 2^-28.  Rows of zeros have none.
__device__ __forceinline__ bool result_holds(float squares, float a_norm, float w_norms, int features, int K) {
    constexpr float SHARE = 70368744177664.f;      // 2^46
    return squares >= SHARE * (2.9e-19f * ((float)features * a_norm + w_norms) + 4.8e-23f * (float)features * (float)K) || a_norm == 0.f || w_norms == 0.f;
}

// A token's norm, or -1 if it has no scale.
__device__ __forceinline__ float token_norm(const FixedParams& p, int t) {
    const int word = p.a_word[t];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < ROW_WARPS; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(p.a_norm + (size_t)t * ROW_WARPS + i);
        sum += (v.x + v.y) + (v.z + v.w);
    }
    return exponent_of(word) < E_NONE ? sum : -1.f;
}

__device__ __forceinline__ void conv_barrier() { asm volatile("bar.sync 1, 512;" ::: "memory"); }      // of the converting warps

// Outputs from the float operands, by all converting warps once the rings' shared memory is free: products of one row per thread of a
// group (`mine`, if it has `some`) with n rows of the other operand, staged in shared memory, in double precision.  A group's threads take every
// fourth block of 32 k in ascending order; the groups' sums are added in order.  AHEAD elements of a thread's own row are asked for at once: with
// few rows opposite the chain of their latencies is the bound, with BATCH of them shared memory's reads.
constexpr int UNSCALED_BYTES = CONV_THREADS * 16 * 8;      // staged rows and, after them, the groups' sums: a batch of 16
template <int BATCH, int AHEAD>
__device__ __noinline__ void double_products(const float* mine, bool some, const float* others, long long ld, const volatile int* list, int n, int K,
                                             double* memory, float* out, long long out_ld) {
    const int t = threadIdx.x - CONV_WARP0 * 32, lane = t & 31, group = t / FEATURES, row = t % FEATURES;
    double* const stage = memory + (t >> 5) * (BATCH * 32);
    const bool vec = !((uintptr_t)mine & 15);
    double total[BATCH] = {};
    for (int k0 = group * 32; k0 < K; k0 += GROUPS * 32) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < BATCH; ++j) stage[j * 32 + lane] = j < n && k0 + lane < K ? others[(size_t)list[j] * ld + k0 + lane] : 0.f;
        __syncwarp();
#pragma unroll 1
        for (int k = 0; k < 32; k += AHEAD) {
            float v[AHEAD];
            if (some && vec && k0 + k + AHEAD <= K) {
#pragma unroll
                for (int i = 0; i < AHEAD; i += 4) *reinterpret_cast<float4*>(v + i) = *reinterpret_cast<const float4*>(mine + k0 + k + i);
            } else {
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) v[i] = some && k0 + k + i < K ? mine[k0 + k + i] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < AHEAD; i += 2) {
                const double a = v[i], b = v[i + 1];
#pragma unroll
                for (int j = 0; j < BATCH; ++j) {
                    const double2 x = *reinterpret_cast<const double2*>(stage + j * 32 + k + i);
                    total[j] = fma(b, x.y, fma(a, x.x, total[j]));
                }
            }
        }
    }
    conv_barrier();      // the sums take the place of the staged rows
#pragma unroll
    for (int j = 0; j < BATCH; ++j) memory[j * CONV_THREADS + t] = total[j];
    conv_barrier();
    if (some)
        for (int j = group; j < n; j += GROUPS) {
            const double* s = memory + j * CONV_THREADS + row;
            out[(size_t)list[j] * out_ld] = (float)(((s[0] + s[FEATURES]) + s[2 * FEATURES]) + s[3 * FEATURES]);
        }
    conv_barrier();
}
// ... of a tile: `again` are the tokens.
__device__ __noinline__ void unscaled_outputs(const FixedParams& p, uint8_t* smem, int f0, int t0, int tokens, unsigned long long again) {
    const int t = threadIdx.x - CONV_WARP0 * 32, row = t % FEATURES;
    double* const memory = reinterpret_cast<double*>(smem);
    volatile int* const list = reinterpret_cast<volatile int*>(smem + UNSCALED_BYTES);
    int* const count = reinterpret_cast<int*>(smem + UNSCALED_BYTES) + FEATURES;
    const bool token = row < tokens && again >> row & 1, feature = f0 + row < p.N && p.w_exp[f0 + row] >= E_NONE;
    // the tile's features by those tokens, then its other tokens by its features without a scale
    for (int phase = 0; phase < 2; ++phase) {
        conv_barrier();
        if (t == 0) *count = 0;
        conv_barrier();
        if (t < FEATURES && (phase ? feature : token)) list[atomicAdd(count, 1)] = row;
        conv_barrier();
        const int listed = *const_cast<volatile int*>(count);
        const bool some = phase ? row < tokens && !token : f0 + row < p.N;
        const float* const mine = phase ? p.A + (size_t)(t0 + row) * p.lda : p.W + (size_t)(f0 + row) * p.ldw;
        const float* const others = phase ? p.W + (size_t)f0 * p.ldw : p.A + (size_t)t0 * p.lda;
        const long long ld = phase ? p.ldw : p.lda, out_ld = phase ? 1 : p.ldc;
        float* const out = p.C + (phase ? (size_t)(t0 + row) * p.ldc + f0 : (size_t)t0 * p.ldc + f0 + row);
        for (int at = 0; at < listed;) {
            const int left = listed - at;
            if (left > 2) double_products<16, 8>(mine, some, others, ld, list + at, min(left, 16), p.K, memory, out, out_ld), at += 16;
            else double_products<2, 32>(mine, some, others, ld, list + at, left, p.K, memory, out, out_ld), at += 2;
        }
    }
}

template <int TN> struct Layout {
    // The groups of converting warps take a ring's steps in turn, and a wait by parity cannot tell a phase from the one two before it.  With a
    // multiple of GROUPS stages a stage is always the same group's, which has waited for its last phase itself; with nine, a load that came
    // late let the next group read the stage ahead of it.  (Tensor memory's A_STAGES: a group's wait at step - 4 has shown that the
    // MMAs of step - 4 - A_STAGES are done, so those of step - 2 A_STAGES are.)
    static constexpr int W_STAGES = TN <= 16 ? 12 : 8;
    static constexpr int B_BYTES = 4 * TN * BLOCK_K, B_STAGES = TN <= 16 ? 4 : 3;
    static constexpr int W_OFF = 0, B_OFF = W_STAGES * W_BYTES, BARS = B_OFF + B_STAGES * B_BYTES;
    static constexpr int N_BARS = 2 * W_STAGES + 2 * B_STAGES + 2 * A_STAGES + 2;
    static constexpr int CHECK = BARS + N_BARS * 8 + 32;      // of the last tile: squares [TN], the tokens' norms [TN], the features' [4]
    static constexpr int TOTAL = CHECK + 20 * TN + 32 + 1024;
    // an MMA of M = 128 takes N in sixteens: with eight tokens the third plane's product is one plane wider (its last sum is not read)
    static constexpr int SUMS = TN == 8 ? 6 : 5;
    static constexpr int A_COL0 = 512 - A_STAGES * A_COLS;
    static_assert(W_STAGES % GROUPS == 0 && A_STAGES >= GROUPS, "a stage belongs to one group; see above");
    static_assert(B_OFF >= UNSCALED_BYTES + (FEATURES + 1) * 4 && CHECK % 16 == 0, "unscaled_outputs' memory");
    static_assert(TOTAL <= 232448 && SUMS * TN <= A_COL0 && (TN == 8 || TN % 16 == 0), "fits");
};

template <int TN>
__global__ void __launch_bounds__(THREADS, 1)
fixed_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ FixedParams p) {
    using L = Layout<TN>;
    static_assert(CONV_THREADS == 512, "the named barrier's count");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t w_full = base + L::BARS, w_empty = w_full + 8 * L::W_STAGES;
    const uint32_t b_full = w_empty + 8 * L::W_STAGES, b_empty = b_full + 8 * L::B_STAGES;
    const uint32_t a_full = b_empty + 8 * L::B_STAGES, a_empty = a_full + 8 * A_STAGES;
    const uint32_t acc_full = a_empty + 8 * A_STAGES, acc_empty = acc_full + 8;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + L::BARS + L::N_BARS * 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + L::BARS + L::N_BARS * 8 + 8);
    volatile int* last_flag = reinterpret_cast<volatile int*>(gen + L::BARS + L::N_BARS * 8 + 16);
    volatile int* unscaled_flag = reinterpret_cast<volatile int*>(gen + L::BARS + L::N_BARS * 8 + 24);      // some outputs are to be made from the float operands
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int items = p.tiles * p.splits, total_steps = (p.K + STEP - 1) / STEP;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        *unscaled_flag = 0;
        for (int s = 0; s < L::W_STAGES; ++s) { mbar_init(w_full + 8 * s, 1); mbar_init(w_empty + 8 * s, 4); }
        for (int s = 0; s < L::B_STAGES; ++s) { mbar_init(b_full + 8 * s, 1); mbar_init(b_empty + 8 * s, 1); }
        for (int s = 0; s < A_STAGES; ++s) { mbar_init(a_full + 8 * s, 4); mbar_init(a_empty + 8 * s, 1); }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, CONV_THREADS / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();

    // an item: a tile and a share of its K
    auto range = [&](int item, int& tile, int& split, int& first, int& n) {
        tile = item % p.tiles;
        split = item / p.tiles;
        first = split * p.steps_per_split;
        n = max(0, min(p.steps_per_split, total_steps - first));
    };

    if (warp == 0) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_w)) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_b)) : "memory");
            bool waited = false, ok = true;
            int it = 0, bt = 0;      // steps and blocks of 128 k asked for so far
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
                int tile, split, first, n;
                range(item, tile, split, first, n);
                const int f0 = tile / p.tiles_m * FEATURES, t0 = tile % p.tiles_m * TN;
                auto weights = [&](int i, int at) {
                    const int s = at % L::W_STAGES;
                    if (!mbar_wait(w_empty + 8 * s, ((at / L::W_STAGES) & 1) ^ 1, abort_flag, p.err_flag)) return false;
                    mbar_expect_tx(w_full + 8 * s, W_BYTES);
                    tma_load_2d(base + L::W_OFF + s * W_BYTES, &map_w, w_full + 8 * s, (first + i) * STEP, f0);
                    return true;
                };
                int done = 0;
                if (!waited) {
                    // the weights depend on no earlier kernel
                    done = min(n, L::W_STAGES);
                    for (int i = 0; i < done; ++i) weights(i, i);
                    pdl_wait();
                    waited = true;
                }
                for (int i = 0; i < n && ok; ++i) {
                    if ((i & 3) == 0) {
                        const int s = bt % L::B_STAGES;
                        ok = mbar_wait(b_empty + 8 * s, ((bt / L::B_STAGES) & 1) ^ 1, abort_flag, p.err_flag);
                        if (!ok) break;
                        mbar_expect_tx(b_full + 8 * s, L::B_BYTES);
                        tma_load_3d(base + L::B_OFF + s * L::B_BYTES, &map_b, b_full + 8 * s, (first + i) * STEP, t0, 0);
                        ++bt;
                    }
                    if (i >= done) ok = weights(i, it + i);
                }
                it += n;
            }
            if (!waited) pdl_wait();
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // D 32-bit integers (2 at bit 4), A and B signed bytes (1 at bits 7 and 10), N >> 3 at bit 17, M >> 4 at bit 24
            constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(FEATURES >> 4) << 24);
            constexpr uint32_t n4 = (uint32_t)(4 * TN >> 3) << 17, n3 = (uint32_t)((TN == 8 ? 32 : 3 * TN) >> 3) << 17, n2 = (uint32_t)(2 * TN >> 3) << 17;
            int it = 0, bt = 0, j = 0;
            bool ok = true;
            pdl_wait();      // the tokens' planes come after it, and no bounded wait should have to last as long as the kernels before
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++j) {
                int tile, split, first, n;
                range(item, tile, split, first, n);
                ok = mbar_wait(acc_empty, j & 1, abort_flag, p.err_flag);
                if (!ok) { umma_commit(acc_full); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int i = 0; i < n; ++i, ++it) {
                    const int sb = bt % L::B_STAGES, sa = it % A_STAGES;
                    if ((i & 3) == 0) {
                        ok = mbar_wait(b_full + 8 * sb, (bt / L::B_STAGES) & 1, abort_flag, p.err_flag);
                        if (!ok) break;
                    }
                    ok = mbar_wait(a_full + 8 * sa, (it / A_STAGES) & 1, abort_flag, p.err_flag);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t db = umma_desc(base + L::B_OFF + sb * L::B_BYTES) + 2 * (i & 3);      // 32 bytes of k further
                    const uint32_t a = tmem + L::A_COL0 + sa * A_COLS;
                    umma_i8(tmem, a, db, idesc | n4, i > 0);                      // plane 0: sums 0 .. 3
                    umma_i8(tmem + TN, a + 8, db, idesc | n4, 1);                 // plane 1: sums 1 .. 4 (4 starts as zeros)
                    umma_i8(tmem + 2 * TN, a + 16, db, idesc | n3, 1);            // plane 2: sums 2 .. 4
                    umma_i8(tmem + 3 * TN, a + 24, db, idesc | n2, 1);            // plane 3: sums 3, 4
                    umma_commit(a_empty + 8 * sa);
                    if ((i & 3) == 3 || i == n - 1) {
                        umma_commit(b_empty + 8 * sb);
                        ++bt;
                    }
                }
                umma_commit(acc_full);      // also where a wait ran out
            }
        }
    } else if (warp >= CONV_WARP0) {
        const int group = (warp - CONV_WARP0) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        // the tile's columns that this group puts together (whole loads of eight: with few columns not every group has some)
        constexpr int COLS = (TN + 8 * GROUPS - 1) / (8 * GROUPS) * 8;
        const int col0 = group * COLS;
        const bool has_cols = col0 < TN;
        static_assert(TN % COLS == 0, "every group has all of its columns or none");
        const uint32_t zeros[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        auto clear_last_sum = [&]() {      // no first MMA overwrites the sum 4
            if (has_cols)
                for (int c = 0; c < COLS; c += 8) tmem_st8(tmem + lanes + 4 * TN + col0 + c, zeros);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty);
        };
        float4* const s_squares = reinterpret_cast<float4*>(gen + L::CHECK);
        float* const s_tokens = reinterpret_cast<float*>(s_squares + TN);
        float2* const s_features = reinterpret_cast<float2*>(s_tokens + TN);
        // Do a tile's results hold?
        auto check = [&](int item, bool last_tile) {
            const int tile = item % p.tiles, t0 = tile % p.tiles_m * TN;
            float2 part[4];      // (asked for before anything is used: one latency)
#pragma unroll
            for (int r = 0; r < 4; ++r) part[r] = (last_tile ? s_features : p.features + (size_t)item * 4)[r];
            float norm[(TN + 31) / 32];
            float4 square[(TN + 31) / 32];
#pragma unroll
            for (int c = 0; c < TN; c += 32) {
                norm[c / 32] = 0.f;
                if (c + lane < TN && t0 + c + lane < p.M) {
                    norm[c / 32] = last_tile ? s_tokens[c + lane] : token_norm(p, t0 + c + lane);
                    square[c / 32] = last_tile ? s_squares[c + lane] : p.squares[(size_t)tile * TN + c + lane];
                }
            }
            float w_norms = 0.f;
            int features = 0;
            bool odd = false;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                w_norms += part[r].x;
                features += __float_as_int(part[r].y) & 0x7fffffff;
                odd |= __float_as_int(part[r].y) < 0;
            }
            unsigned long long again = 0;
#pragma unroll
            for (int c = 0; c < TN; c += 32) {
                bool holds = true;
                if (c + lane < TN && t0 + c + lane < p.M) {
                    const float4 s = square[c / 32];
                    holds = norm[c / 32] >= 0.f && result_holds(((s.x + s.y) + s.z) + s.w, norm[c / 32], w_norms, features, p.K);
                }
                again |= (unsigned long long)__ballot_sync(0xffffffffu, !holds) << c;
            }
            if (lane == 0) {
                if (odd || again) *unscaled_flag = 1;
                p.again[item] = again;
            }
        };
        clear_last_sum();
        bool waited = false, ok = true;
        int it = 0, j = 0;
        for (int item = blockIdx.x; item < items; item += gridDim.x, ++j) {
            int tile, split, first, n;
            range(item, tile, split, first, n);
            const int f = tile / p.tiles_m * FEATURES + row, t0 = tile % p.tiles_m * TN;
            const bool last_tile = item + gridDim.x >= items;
            const int Ew = f < p.N ? p.w_exp[f] : E_MIN;
            const float w_norm = group == 0 && f < p.N ? p.w_norm[f] : 0.f;      // (from memory: asked for well ahead)
            const RowScale sc = row_scale(Ew);
            const bool tiny = __any_sync(0xffffffffu, sc.s2 != 1.f);
            for (int i = (group - it) & (GROUPS - 1); i < n && ok; i += GROUPS) {
                const int at = it + i, s = at % L::W_STAGES, sa = at % A_STAGES;
                ok = mbar_wait(w_full + 8 * s, (at / L::W_STAGES) & 1, abort_flag, p.err_flag);
                const uint32_t src = base + L::W_OFF + s * W_BYTES + row * 128;
                uint32_t pl[4][8];
                float4 v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[q].x), "=f"(v[q].y), "=f"(v[q].z), "=f"(v[q].w)
                                 : "r"(src + ((q ^ (row & 7)) << 4)) : "memory");
                if (tiny) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) { v[q].x *= sc.s2; v[q].y *= sc.s2; v[q].z *= sc.s2; v[q].w *= sc.s2; }
                }
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    bytes_of(v[q].x * sc.s1, v[q].y * sc.s1, v[q].z * sc.s1, v[q].w * sc.s1, pl[0][q], pl[1][q], pl[2][q], pl[3][q]);
                __syncwarp();
                if (lane == 0) mbar_arrive(w_empty + 8 * s);
                if (!waited && at >= A_STAGES) { pdl_wait(); waited = true; }      // from here on the MMAs have to run
                ok = mbar_wait(a_empty + 8 * sa, ((at / A_STAGES) & 1) ^ 1, abort_flag, p.err_flag) && ok;
                ok = __all_sync(0xffffffffu, ok);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int q = 0; q < 4; ++q) tmem_st8(tmem + lanes + L::A_COL0 + sa * A_COLS + 8 * q, pl[q]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(a_full + 8 * sa);
            }
            it += n;
            if (!waited) { pdl_wait(); waited = true; }
            // what the tile's check needs, while the MMAs finish
            if (group == 0) {
                const bool scaled = f < p.N && Ew < E_NONE;
                const float norm = warp_sum(scaled ? w_norm : 0.f);
                const int count = __popc(__ballot_sync(0xffffffffu, scaled)) | (__any_sync(0xffffffffu, f < p.N && !scaled) ? 0x80000000 : 0);
                if (lane == 0) (last_tile ? s_features : p.features + (size_t)item * 4)[quarter] = make_float2(norm, __int_as_float(count));
            } else if (group == 1 && last_tile && row < TN && t0 + row < p.M) s_tokens[row] = token_norm(p, t0 + row);
            ok = mbar_wait(acc_full, j & 1, abort_flag, p.err_flag) && ok && !*abort_flag;
            // all warps of the groups agree: they meet at a barrier below
            {
                uint32_t r;
                asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.and.pred q, 1, 512, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                             : "=r"(r) : "r"((uint32_t)ok) : "memory");
                ok = r != 0;
            }
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (last_tile)      // the tiles before it, a warp each, from those that may have no columns on
                for (int q = CONV_WARP0 + 4 * GROUPS - 1 - warp; q < j; q += 4 * GROUPS) {
                    const int earlier = (int)blockIdx.x + q * (int)gridDim.x;
                    if (p.splits == 1 || p.decided[earlier]) check(earlier, false);
                }
            // sum s stands for 2^(8 (6 - s)); a row's scale is 2^(E - 29): C = total 2^(16 - 58) 2^(Ea + Ew).  Returns the square of C over 2^(Ea + Ew)
            auto finish = [&](int t, int word, long long total) {
                const int Ea = exponent_of(word);
                if (t >= p.M || f >= p.N || Ea >= E_NONE || Ew >= E_NONE) return 0.f;
                double x = __ll2double_rn(total) * 0x1p-42;
                if (outliers_of(word)) x += outlier_sum(p.outliers + (size_t)t * MAX_OUTLIERS, outliers_of(word), p.W + (size_t)f * p.ldw) * pow2d(-Ea - Ew);
                p.C[(size_t)t * p.ldc + f] = (float)(x * pow2d(Ea + Ew));
                return (float)x * (float)x;
            };
            float* const squares = reinterpret_cast<float*>(last_tile ? s_squares : p.squares + (size_t)tile * TN);
            long long* const mine = p.partial + ((size_t)(split * p.tiles + tile) * TN) * FEATURES + row;
            if (has_cols) {
#pragma unroll 1
                for (int c = 0; c < COLS; c += 8) {
                    int s[5][8], word[8];
                    // (the words' memory goes on beyond the last token's)
                    *reinterpret_cast<int4*>(word) = *reinterpret_cast<const int4*>(p.a_word + t0 + col0 + c);
                    *reinterpret_cast<int4*>(word + 4) = *reinterpret_cast<const int4*>(p.a_word + t0 + col0 + c + 4);
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 5; ++q) tmem_ld8(tmem + lanes + q * TN + col0 + c, s[q]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const long long total = ((long long)s[0][e] << 32) + ((long long)s[1][e] << 24) + ((long long)s[2][e] << 16) +
                                                ((long long)s[3][e] << 8) + s[4][e];
                        if (p.splits == 1) v[e] = finish(t0 + col0 + c + e, word[e], total);
                        else if (t0 + col0 + c + e < p.M) mine[(size_t)(col0 + c + e) * FEATURES] = total;
                    }
                    if (p.splits == 1) {
                        // the warp's eight sums at once (the tree of warp_sum): half of them go to the other half of the lanes, ...
#pragma unroll
                        for (int half = 4, o = 16; half; half >>= 1, o >>= 1) {
                            const bool upper = lane & o;
#pragma unroll
                            for (int i = 0; i < half; ++i) {
                                const float sent = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + half], o);
                                v[i] = (upper ? v[i + half] : v[i]) + sent;
                            }
                        }
                        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
                        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
                        if ((lane & 3) == 0) squares[(col0 + c + (lane >> 2)) * 4 + quarter] = v[0];
                    }
                }
            }
            __syncwarp();
            clear_last_sum();
            if (p.splits > 1) {
                // whoever arrives last adds up the tile's shares
                __threadfence();
                conv_barrier();
                if (threadIdx.x == CONV_WARP0 * 32) p.decided[item] = *last_flag = atomicAdd(p.counters + tile, 1) == p.splits - 1;
                conv_barrier();
                if (*last_flag) {
                    __threadfence();
                    const int rows = min(TN, p.M - t0);
                    for (int c = group; c < rows; c += 4 * GROUPS) {      // four tokens' shares asked for at once
                        long long total[4] = {};
                        int word[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) word[q] = p.a_word[t0 + min(c + q * GROUPS, rows - 1)];
                        for (int z = 0; z < p.splits; ++z)
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                total[q] += __ldcg(p.partial + ((size_t)(z * p.tiles + tile) * TN + min(c + q * GROUPS, rows - 1)) * FEATURES + row);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int at = c + q * GROUPS;
                            if (at < rows) {
                                const float square = warp_sum(finish(t0 + at, word[q], total[q]));
                                if (lane == 0) squares[at * 4 + quarter] = square;
                            }
                        }
                    }
                }
                conv_barrier();      // the flag is read before the next item writes it
            }
        }
        if (!waited) pdl_wait();
        if (p.splits == 1 || !ok) conv_barrier();
        if (ok) {
            if (warp == CONV_WARP0 && (p.splits == 1 || *last_flag)) check(items - 1 - (items - 1 - (int)blockIdx.x) % (int)gridDim.x, true);
            conv_barrier();
            if (*unscaled_flag)
                for (int item = blockIdx.x; item < items; item += gridDim.x)
                    if (p.splits == 1 || p.decided[item]) {
                        const int tile = item % p.tiles, t0 = tile % p.tiles_m * TN;
                        unscaled_outputs(p, gen, tile / p.tiles_m * FEATURES, t0, min(TN, p.M - t0), p.again[item]);
                    }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// PLANES: a token's word, norm and outliers, and its other elements as four byte planes [4][rows][pitch]; else a feature's exponent and norm.  A block
// per row; what bounds it is the chain of its latencies, so a thread asks for HELD pieces of four elements at once and keeps them (what a
// longer row has beyond them is read again, out of the caches).
template <bool PLANES, bool VEC, int HELD>
__global__ void __launch_bounds__(ROW_THREADS, HELD == 1 ? 2 : 1)
fixed_rows_kernel(const float* A, long long lda, int K, int* words, float* norms, int2* outliers, uint8_t* planes, long long plane_stride, int pitch, int* counters, int n_counters) {
    __shared__ int4 s_stats[ROW_WARPS];
    __shared__ int2 s_list[MAX_OUTLIERS];
    __shared__ int s_count;
    if (PLANES) pdl_trigger();      // a weight's exponents: no product may start beside them (it reads them ahead of its own wait)
    pdl_wait();
    const int tid = threadIdx.x;
    const float* a = A + (size_t)blockIdx.x * lda;
    if (PLANES) {
        for (int i = blockIdx.x * ROW_THREADS + tid; i < n_counters; i += gridDim.x * ROW_THREADS) counters[i] = 0;
        if (tid == 0) s_count = 0;
    }
    auto piece = [&](int k) {      // the four elements from k on, zeros beyond the row
        if (VEC) return k < K ? *reinterpret_cast<const float4*>(a + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 v;
        v.x = k < K ? a[k] : 0.f;
        v.y = k + 1 < K ? a[k + 1] : 0.f;
        v.z = k + 2 < K ? a[k + 2] : 0.f;
        v.w = k + 3 < K ? a[k + 3] : 0.f;
        return v;
    };
    float4 held[HELD];
#pragma unroll
    for (int h = 0; h < HELD; ++h) held[h] = piece(4 * (tid + h * ROW_THREADS));
    auto magnitude = [](float x) { return __float_as_uint(x) & 0x7fffffffu; };
    uint32_t limit = 0xffffffffu;      // elements from here on have been listed
    int E, listed = 0;
    for (;;) {
        // of the others: the largest, the sum of their exponents, how many are not zero
        uint32_t most = 0, both = 0;      // the sum below the count: a warp has at most 1,280 elements
        auto look = [&](float x) {
            const uint32_t u = magnitude(x);
            most = max(most, u);
            both += (u >> 23) + (u ? 1u << 20 : 0u);
        };
        if (limit == 0xffffffffu) {
#pragma unroll
            for (int h = 0; h < HELD; ++h) { look(held[h].x); look(held[h].y); look(held[h].z); look(held[h].w); }
#pragma unroll 1
            for (int k = 4 * (tid + HELD * ROW_THREADS); k < K; k += 4 * ROW_THREADS) {
                const float4 v = piece(k);
                look(v.x); look(v.y); look(v.z); look(v.w);
            }
        } else
            for (int k = tid; k < K; k += ROW_THREADS)
                if (magnitude(a[k]) < limit) look(a[k]);
        most = __reduce_max_sync(0xffffffffu, most);
        both = __reduce_add_sync(0xffffffffu, both);
        int sum, n;
        if ((tid & 31) == 0) s_stats[tid >> 5] = make_int4((int)most, (int)(both & 0xfffff), (int)(both >> 20), 0);
        __syncthreads();
        const int4 others = s_stats[tid & 31];
        static_assert(ROW_WARPS == 32, "a lane for each warp's");
        most = __reduce_max_sync(0xffffffffu, (uint32_t)others.x);
        sum = __reduce_add_sync(0xffffffffu, others.y);
        n = __reduce_add_sync(0xffffffffu, others.z);
        E = row_exponent(most);
        if (E >= E_NONE || n == 0) break;
        if (((int)(most >> 23) - (PLANES ? OUTLIER_BITS : WEIGHT_BITS)) * n <= sum) break;      // no more than the mean exponent and so many bits
        if (!PLANES) {
            E = E_NONE;
            break;
        }
        const uint32_t from = (uint32_t)(sum / n + OUTLIER_BITS + 1) << 23;      // at most the exponent of `most`
        for (int k = tid; k < K; k += ROW_THREADS) {
            const float x = a[k];
            const uint32_t u = magnitude(x);
            if (u >= from && u < limit) {
                const int at = atomicAdd(&s_count, 1);
                if (at < MAX_OUTLIERS) s_list[at] = make_int2(k, __float_as_int(x));
            }
        }
        __syncthreads();
        if (s_count > MAX_OUTLIERS) break;      // too many: these stay in the integers
        listed = s_count;                       // (the next turn adds to it behind its own barrier)
        limit = from;
    }
    const RowScale sc = row_scale(E);
    const bool none = E >= E_NONE;
    float norm = 0.f;
    auto scaled = [&](float x) { return none || magnitude(x) >= limit ? 0.f : x * sc.s2 * sc.s1; };
    auto square = [&](float x) { norm = fmaf(x, x, norm); };      // in units of 2^58
    if constexpr (!PLANES) {
        auto take = [&](const float4& v) { square(scaled(v.x)); square(scaled(v.y)); square(scaled(v.z)); square(scaled(v.w)); };
#pragma unroll
        for (int h = 0; h < HELD; ++h) take(held[h]);
        for (int k = 4 * (tid + HELD * ROW_THREADS); k < K; k += 4 * ROW_THREADS) take(piece(k));
        norm = warp_sum(norm);
        __syncthreads();
        if ((tid & 31) == 0) s_stats[tid >> 5].x = __float_as_int(norm);
        __syncthreads();
        if (tid == 0) {
            for (int i = 1; i < ROW_WARPS; ++i) norm += __int_as_float(s_stats[i].x);
            norms[blockIdx.x] = norm * 0x1p-58f;
            words[blockIdx.x] = E;
        }
    } else {
        if (tid < 32) {
            const int n = none ? 0 : listed;
            if (tid == 0) words[blockIdx.x] = n << 16 | (E & 0xffff);
            if (tid < n) {
                const int2 mine = s_list[tid];
                int rank = 0;
                for (int i = 0; i < n; ++i) rank += s_list[i].x < mine.x;
                outliers[(size_t)blockIdx.x * MAX_OUTLIERS + rank] = mine;
            }
        }
        uint8_t* out = planes + (size_t)blockIdx.x * pitch;
        auto put = [&](int k, const float4& v) {
            uint32_t w[4];
            const float x = scaled(v.x), y = scaled(v.y), z = scaled(v.z), u = scaled(v.w);
            square(x); square(y); square(z); square(u);
            bytes_of(x, y, z, u, w[0], w[1], w[2], w[3]);
#pragma unroll
            for (int q = 0; q < 4; ++q) *reinterpret_cast<uint32_t*>(out + q * plane_stride + k) = w[q];
        };
#pragma unroll
        for (int h = 0; h < HELD; ++h) {
            const int k = 4 * (tid + h * ROW_THREADS);
            if (k < pitch) put(k, held[h]);
        }
#pragma unroll 1
        for (int k = 4 * (tid + HELD * ROW_THREADS); k < pitch; k += 4 * ROW_THREADS) put(k, piece(k));
        norm = warp_sum(norm);
        if ((tid & 31) == 0) norms[blockIdx.x * ROW_WARPS + (tid >> 5)] = norm * 0x1p-58f;      // whoever reads them adds them up: no barrier for it here
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

struct Plan {
    int tn, tiles_m, tiles, splits, steps_per_split;
    long long planes, words, norms, outliers, squares, features, again, decided, counters, partial, bytes;      // offsets into the workspace
    int pitch;
};
// Tokens per tile and shares of K by estimated cycles of the busiest SM.
Plan make_plan(int M, int N, int K, int sms, int force_tn, int force_splits) {
    Plan best = {};
    const int steps = (K + STEP - 1) / STEP, blocks_n = ceil_div(N, FEATURES);
    double best_cost = 0;
    const int widths[5] = {8, 16, 32, 48, 64};
    for (int wi = 0; wi < 5; ++wi) {
        const int tn = widths[wi];
        if (force_tn ? tn != force_tn : (tn < 64 && tn < M && M <= 64)) continue;      // up to 64 tokens: one tile
        const int tiles_m = ceil_div(M, tn);
        const long long tiles = (long long)tiles_m * blocks_n;
        const double step_cost = tn <= 16 ? 350 : tn <= 32 ? 360 : tn <= 48 ? 420 : 520;
        for (int sp = 1; sp <= 16; ++sp) {
            if (force_splits ? sp != force_splits : (sp > 1 && (steps / sp < 16 || tiles >= 2 * sms))) continue;
            const int per = (ceil_div(steps, sp) + 3) / 4 * 4;
            if ((sp - 1) * per >= steps || tiles * sp > 0x7fffffffll) continue;      // no empty share
            const double rounds = (double)((tiles * sp + sms - 1) / sms);
            const double cost = rounds * (per * step_cost + 1500 + 12.0 * tn) + (sp > 1 ? 2500 + 30.0 * tn * (1 + rounds) : 0);
            if (!best.tn || cost < best_cost) {
                best_cost = cost;
                best.tn = tn; best.tiles_m = tiles_m; best.tiles = (int)tiles; best.splits = sp; best.steps_per_split = per;
            }
        }
        if (!force_tn && M <= tn) break;
    }
    auto up = [](long long v) { return (v + 255) / 256 * 256; };
    best.pitch = (K + 15) / 16 * 16;
    best.planes = 0;
    best.words = up(4ll * M * best.pitch);
    best.norms = best.words + up(4ll * best.tiles_m * best.tn);      // the epilogue reads the words of whole tiles
    best.outliers = best.norms + up(4ll * ROW_WARPS * M);
    best.squares = best.outliers + up(8ll * MAX_OUTLIERS * M);
    best.features = best.squares + up(16ll * best.tiles * best.tn);
    best.again = best.features + up(32ll * best.tiles * best.splits);
    best.decided = best.again + up(8ll * best.tiles * best.splits);
    best.counters = best.decided + up(best.splits > 1 ? 4ll * best.tiles * best.splits : 0);
    best.partial = best.counters + up(best.splits > 1 ? 4ll * best.tiles : 0);
    best.bytes = best.partial + (best.splits > 1 ? 8ll * best.splits * best.tiles * best.tn * FEATURES : 0);
    return best;
}

template <int TN>
int launch(const CUtensorMap& mw, const CUtensorMap& mb, const FixedParams& p, cudaStream_t stream) {
    using L = Layout<TN>;
    static bool configured_on[PYRE_MAX_DEVICES] = {};      // the attribute is per device
    bool& configured = configured_on[pyre_current_device()];
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(fixed_gemm_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int items = p.tiles * p.splits, sms = pyre_sm_count();
    return (int)pyre_launch(fixed_gemm_kernel<TN>, dim3(items < sms ? items : sms), dim3(THREADS), (size_t)L::TOTAL, stream, mw, mb, p);
}

// Rows of up to 4,096 elements hold a piece a thread (two blocks fit on an SM), longer ones five.
template <bool PLANES>
cudaError_t launch_rows(bool vec, const float* a, long long lda, int rows, int K, int* words, float* norms, int2* outliers, uint8_t* planes, long long plane_stride, int pitch,
                        int* counters, int n_counters, cudaStream_t stream) {
    const bool brief = K <= 4 * ROW_THREADS;
    auto kernel = vec ? (brief ? fixed_rows_kernel<PLANES, true, 1> : fixed_rows_kernel<PLANES, true, 5>)
                      : (brief ? fixed_rows_kernel<PLANES, false, 1> : fixed_rows_kernel<PLANES, false, 5>);
    return pyre_launch(kernel, dim3(rows), dim3(ROW_THREADS), (size_t)0, stream, a, lda, K, words, norms, outliers, planes, plane_stride, pitch, counters, n_counters);
}
}  // namespace

// The sizes that `pyre_fixed_linear` takes: sums of at most 3 K 2^14 in 32 bits, TMA rows on 16-byte boundaries.
static bool fixed_ok(const void* w, long long ldw, int K) { return K > 0 && K <= 40960 && ldw % 4 == 0 && !((uintptr_t)w & 15); }

// The exponents of a weight's rows, 1000 for one without a scale, and the squares of their norms over their scales, worked out once.
PYRE_API int pyre_fixed_exponents(const float* w, long long ldw, int N, int K, int* exps, float* norms, cudaStream_t stream) {
    if (N <= 0) return 0;
    if (!fixed_ok(w, ldw, K)) return PYRE_ERR_UNSUPPORTED;
    const cudaError_t e = launch_rows<false>(K % 4 == 0, w, ldw, N, K, exps, norms, nullptr, nullptr, 0, 0, nullptr, 0, stream);
    if (e != cudaSuccess) return (int)e;
    PYRE_LAUNCH_CHECK();
    return 0;
}

// Bytes of scratch memory that a product of these sizes needs (256-byte aligned), or -1 (tn and splits: 0 = the plan's own).
PYRE_API long long pyre_fixed_workspace(int M, int N, int K, int tn, int splits) {
    if (M <= 0 || N <= 0) return 0;
    const Plan pl = make_plan(M, N, K, pyre_sm_count(), tn, splits);
    return pl.tn ? pl.bytes : -1;
}

PYRE_API int pyre_fixed_linear(const float* A, long long lda, const float* W, long long ldw, const int* w_exp, const float* w_norm, float* C, long long ldc,
                               int M, int N, int K, void* workspace, long long workspace_bytes, int tn, int splits, int* err_flag, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (!fixed_ok(W, ldw, K) || ((uintptr_t)workspace & 255)) return PYRE_ERR_UNSUPPORTED;
    const Plan pl = make_plan(M, N, K, pyre_sm_count(), tn, splits);
    if (!pl.tn || workspace_bytes < pl.bytes) return PYRE_ERR_BAD_ARG;
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return PYRE_ERR_UNSUPPORTED;
    uint8_t* ws = (uint8_t*)workspace;
    CUtensorMap mw, mb;
    {
        cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
        cuuint64_t strides[1] = {(cuuint64_t)ldw * 4};
        cuuint32_t box[2] = {STEP, FEATURES}, elem[2] = {1, 1};
        if (fn(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return PYRE_ERR_BAD_ARG;
    }
    {
        cuuint64_t dims[3] = {(cuuint64_t)pl.pitch, (cuuint64_t)M, 4};
        cuuint64_t strides[2] = {(cuuint64_t)pl.pitch, (cuuint64_t)pl.pitch * M};
        cuuint32_t box[3] = {BLOCK_K, (cuuint32_t)pl.tn, 4}, elem[3] = {1, 1, 1};
        if (fn(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, ws + pl.planes, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return PYRE_ERR_BAD_ARG;
    }
    const bool vec = K % 4 == 0 && lda % 4 == 0 && !((uintptr_t)A & 15);
    int* words = (int*)(ws + pl.words);
    float* norms = (float*)(ws + pl.norms);
    int2* outliers = (int2*)(ws + pl.outliers);
    int* counters = (int*)(ws + pl.counters);
    const cudaError_t e = launch_rows<true>(vec, A, lda, M, K, words, norms, outliers, ws + pl.planes, (long long)pl.pitch * M, pl.pitch, counters, pl.splits > 1 ? pl.tiles : 0, stream);
    if (e != cudaSuccess) return (int)e;
    FixedParams p = {A, W, w_exp, words, outliers, w_norm, norms, (float4*)(ws + pl.squares), (float2*)(ws + pl.features), (int*)(ws + pl.decided), (unsigned long long*)(ws + pl.again), C, lda, ldw, ldc, M, N, K, pl.tiles_m, pl.tiles, pl.splits, pl.steps_per_split,
                     (long long*)(ws + pl.partial), counters, err_flag};
    int rc;
    switch (pl.tn) {
        case 8: rc = launch<8>(mw, mb, p, stream); break;
        case 16: rc = launch<16>(mw, mb, p, stream); break;
        case 32: rc = launch<32>(mw, mb, p, stream); break;
        case 48: rc = launch<48>(mw, mb, p, stream); break;
        default: rc = launch<64>(mw, mb, p, stream); break;
    }
    if (rc) return rc;
    PYRE_LAUNCH_CHECK();
    return 0;
}
