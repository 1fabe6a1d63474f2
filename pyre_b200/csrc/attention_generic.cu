// Paged attention over the block table, any head size that is a multiple of 16, any
// page size, float32 or bfloat16 storage, fp32 arithmetic throughout.
//
// This is the exact kernel: it serves the whole 32-bit path and every head size the
// tensor-core kernels do not cover.  A CTA of eight warps owns up to R rows, a row being one
// (query token, query head): the query heads of one key/value head, of one token or of a few
// neighbouring ones.  The keys are cut into chunks of 32, aligned to multiples of 32 from position 0;
// warp w walks the chunks w, w + 8, ... for all rows at once, a row with an online softmax of its own
// (running maximum m, sum l and an fp32 accumulator), and the eight warps' results are merged in
// their order at the end.  Prompt portions and single decoded tokens are the same
// case: a query at absolute position p sees the cached keys lo..p, where
// lo = max(0, p - window + 1) with a window and 0 without (and, with a window, the first
// `keep_first` positions of the sequence, however far back); the keys of the current
// portion were written to the pages before this kernel runs.
//
// What bounds it: a few decoded tokens, the latency of a warp's chain of chunks (hence eight warps on a row); prompts,
// the reads of keys and queries beside the multiplications (hence the rows that share a key: one load of it serves all of them).
// Measured (float32, 28 query heads, 4 key/value heads, size 128): four decoded tokens after some 1,000 keys 357 -> 75 us, a
// prompt of 509 tokens 576 -> 256 us (before, a warp walked all keys of one row alone).
//
// The arithmetic of a row depends on nothing but its own keys: which warp takes a chunk is
// decided by the chunk's place in the sequence, a chunk or key that a row does not see leaves the row alone, and every
// sum has a fixed order, so the result is bit-identical however the tokens were cut into steps, whatever else is
// in the batch, whichever rows share a CTA and wherever the pages lie.
//
// Formula: pyre/model.py:104-124 (scores = (q k^T) * scale, causal mask, fp32 softmax,
// probs v) and pyre/kernels/paged_attn.py:43-71 (online softmax over the block table);
// query head h reads key/value head h / (nh / nkv) (pyre/model.py:66-72).
#include "common.cuh"

constexpr int AG_WARPS = 8;

typedef unsigned long long f32x2;     // two floats in one 64-bit register

__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    return (f32x2)__float_as_uint(lo) | ((f32x2)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float lo2(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }

// R rows of NI * 128 dims at most (a lane holds the dims 4 lane + 128 i .. + 3).  Rows are (token of the group, head of
// the group), token first: `tpg` tokens of `hpg` heads, hpg * tpg <= R; blockIdx.y is the head group: kv head, and which
// of its `hgroups` groups of query heads.
// DEEP: a few CTAs only (decoded tokens), each alone on its SM: a warp's chain of memory latencies is what counts, so it asks
// for eight pieces of a key row and sixteen value rows at a time instead of two and four, with twice the registers.
template <typename T, int R, int NI, bool DEEP>
__global__ void __launch_bounds__(AG_WARPS * 32, DEEP ? 1 : 2) paged_attention_generic_kernel(
    const T* q,             // [n_tokens, nh, hd]
    const T* cache,         // one layer: [page][2][nkv][page_size][hd]
    T* out,                 // [n_tokens, nh * hd]
    const int* block_table, // [n_seqs, bt_stride] logical page -> physical page (or -1)
    int bt_stride,
    const int* seq_of_token,  // [n_tokens]
    const int* positions,     // [n_tokens]
    int n_tokens, int nh, int nkv, int hd, int page_size, int window, int keep_first, float scale, float sink, const float* head_sinks, long long n_pages, int* err_flag,
    int hpg, int hgroups, int tpg) {
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                                // [R][hd]
    float* ps = qs + R * hd;                         // [warps][32 keys][R] probabilities of a chunk, -1: the row does not see the key
    float* merged = ps + AG_WARPS * 32 * R;          // [warps][R][hd]
    __shared__ float m_s[AG_WARPS][R], l_s[AG_WARPS][R];
    __shared__ int row_seq[R], row_pos[R], row_lo[R];
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_rep = nh / nkv, kvh = blockIdx.y / hgroups;
    const int first_head = (blockIdx.y - kvh * hgroups) * hpg;                 // within the kv head's query heads
    const int heads = min(hpg, n_rep - first_head);
    const int t0 = blockIdx.x * tpg, rows = min(tpg, n_tokens - t0) * hpg;
    auto row_token = [&](int r) { return t0 + r / hpg; };
    auto row_head = [&](int r) { return kvh * n_rep + first_head + r % hpg; };
    if (threadIdx.x < R) {
        const int r = threadIdx.x;
        const bool live = r < rows && r % hpg < heads;
        const int pos = live ? positions[row_token(r)] : -1;
        row_seq[r] = r < rows ? seq_of_token[row_token(r)] : -1;
        row_pos[r] = pos;                                                      // negative: sees no key
        row_lo[r] = !live ? -1 : (pos >= 0 && window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    }
    for (int e = threadIdx.x; e < R * hd; e += AG_WARPS * 32) {
        const int r = e / hd, d = e - r * hd;
        qs[e] = (r < rows && r % hpg < heads) ? to_f32<T>(q[((size_t)row_token(r) * nh + row_head(r)) * hd + d]) : 0.f;
    }
    __syncthreads();

    constexpr int U = DEEP ? 16 / NI : 4;      // value rows fetched together
    const int keep = window > 0 ? keep_first : 0;
    float acc[R][4 * NI], m[R], l[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int i = 0; i < 4 * NI; ++i) acc[r][i] = 0.f;
    }
    float* my_ps = ps + warp * 32 * R;
    // the first chunk from c on that is this warp's
    auto mine = [&](int c) { return c + 32 * ((warp - (c >> 5)) & (AG_WARPS - 1)); };
    for (int r0 = 0; r0 < rows;) {      // the rows of one sequence after those of another
        const int seq = row_seq[r0];
        int r1 = r0, pos = -1, lo = 0x7fffffff;
        for (; r1 < rows && row_seq[r1] == seq; ++r1) {
            pos = max(pos, row_pos[r1]);
            if (row_pos[r1] >= 0) lo = min(lo, row_lo[r1]);
        }
        if (pos < 0) {      // no row of this piece sees a key
            r0 = r1;
            continue;
        }
        const int* table = block_table + (size_t)seq * bt_stride;
        const int lo_chunk = (lo / 32) * 32;
        // the chunks of the kept first keys (if any), then those of the window
        for (int c = mine(keep > 0 ? 0 : lo_chunk); c <= pos; c += 32 * AG_WARPS) {
            if (c >= keep && c < lo_chunk) {
                c = mine(lo_chunk);
                if (c > pos) break;
            }
            const int j = c + lane;
            const bool seen = (j >= lo || j < keep) && j <= pos;      // by at least one row
            int vrow = 0;      // row index of this key's value vector, in units of hd elements
            const T* kp = cache;
            if (seen) {
                const int page = pyre_checked_page(table[j / page_size], n_pages, err_flag);
                const int off = j % page_size;
                kp = cache + (((size_t)(page * 2) * nkv + kvh) * page_size + off) * hd;
                vrow = (int)(((size_t)(page * 2 + 1) * nkv + kvh) * page_size + off);
            }
            // four interleaved chains (dims e, e + 4 of every 8), added as a tree: shorter sums round less
            f32x2 dot[R][2];
#pragma unroll
            for (int r = 0; r < R; ++r) dot[r][0] = dot[r][1] = 0ull;
#pragma unroll (DEEP ? 8 : 2)
            for (int d = 0; d < hd; d += 8) {
                const Vec<T, 8> kv = load_vec<T, 8>(kp + d);      // a key that no row sees: the pool's first row, whose score is not used
                f32x2 k2[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) k2[e] = pack2(to_f32<T>(kv.v[2 * e]), to_f32<T>(kv.v[2 * e + 1]));
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const ulonglong2 q0 = *reinterpret_cast<const ulonglong2*>(qs + r * hd + d), q1 = *reinterpret_cast<const ulonglong2*>(qs + r * hd + d + 4);
                    fma2(dot[r][0], q0.x, k2[0]);
                    fma2(dot[r][1], q0.y, k2[1]);
                    fma2(dot[r][0], q1.x, k2[2]);
                    fma2(dot[r][1], q1.y, k2[3]);
                }
            }
            // every row of the CTA sees the same keys of this chunk: no row needs to be asked key by key below
            bool alike = r0 == 0 && r1 == rows;
            if (alike && tpg > 1) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    alike = alike && (row_lo[r] < 0 || (c + 31 <= row_pos[r] && (c >= row_lo[r] || c + 32 <= keep)));
            }
            float alpha[R];
            __syncwarp();      // every lane has read the probabilities of the chunk before
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int rp = row_pos[r], rl = row_lo[r];
                float p = alike ? 0.f : -1.f;
                alpha[r] = 1.f;
                if (r >= r0 && r < r1 && c <= rp && (c + 31 >= rl || c < keep)) {      // the same for the whole warp
                    const bool valid = (j >= rl || j < keep) && j <= rp;
                    const float score = valid ? ((lo2(dot[r][0]) + hi2(dot[r][0])) + (lo2(dot[r][1]) + hi2(dot[r][1]))) * scale : -INFINITY;
                    const float m_new = fmaxf(m[r], warp_max(score));
                    const float ref = m_new == -INFINITY ? 0.f : m_new;      // no score above minus infinity so far: every term is zero
                    const float e = valid ? expf(score - ref) : 0.f;
                    alpha[r] = expf(m[r] - ref);      // m = -inf at the start: exp(-inf) = 0
                    l[r] = l[r] * alpha[r] + warp_sum(e);
                    m[r] = m_new;
                    if (valid) p = e;
                }
                my_ps[lane * R + r] = p;
            }
            __syncwarp();
            // this chunk's share of the output, summed on its own and then added to the older keys'; the value rows of some
            // keys are fetched together, then added in the order of the keys
            float part[R][4 * NI];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int i = 0; i < 4 * NI; ++i) part[r][i] = 0.f;
            const unsigned some = __ballot_sync(0xffffffffu, seen);
            const int n_keys = min(32, pos - c + 1);
#pragma unroll 1
            for (int j0 = 0; j0 < n_keys; j0 += U) {
                float val[U][4 * NI];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const T* vp = cache + (size_t)__shfl_sync(0xffffffffu, vrow, (j0 + u) & 31) * hd;
#pragma unroll
                    for (int i = 0; i < NI; ++i) {
                        const int d = 4 * lane + 128 * i;
                        const Vec<T, 4> v = load_vec<T, 4>(vp + (d < hd ? d : 0));
#pragma unroll
                        for (int e = 0; e < 4; ++e) val[u][4 * i + e] = to_f32<T>(v.v[e]);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (!(some >> ((j0 + u) & 31) & 1)) {      // no row sees it: nothing is added, whatever its value holds
#pragma unroll
                        for (int i = 0; i < 4 * NI; ++i) val[u][i] = 0.f;
                    }
#pragma unroll
                    for (int r4 = 0; r4 < R; r4 += 4) {
                        const float4 p4 = *reinterpret_cast<const float4*>(my_ps + ((j0 + u) & 31) * R + r4);
                        const float pj[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (alike || !(pj[e] < 0.f)) {
#pragma unroll
                                for (int i = 0; i < 4 * NI; ++i) part[r4 + e][i] = fmaf(pj[e], val[u][i], part[r4 + e][i]);
                            }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int i = 0; i < 4 * NI; ++i) acc[r][i] = fmaf(acc[r][i], alpha[r], part[r][i]);
        }
        r0 = r1;
    }
    // the warps' results, merged in their order
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (lane == 0) {
            m_s[warp][r] = m[r];
            l_s[warp][r] = l[r];
        }
#pragma unroll
        for (int i = 0; i < NI; ++i)
            if (4 * lane + 128 * i < hd)
                *reinterpret_cast<float4*>(merged + (warp * R + r) * hd + 4 * lane + 128 * i) =
                    make_float4(acc[r][4 * i], acc[r][4 * i + 1], acc[r][4 * i + 2], acc[r][4 * i + 3]);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < R * hd; e += AG_WARPS * 32) {
        const int r = e / hd;
        if (row_lo[r] < 0) continue;      // a row that is not there
        float top = m_s[0][r];
#pragma unroll
        for (int w = 1; w < AG_WARPS; ++w) top = fmaxf(top, m_s[w][r]);
        float sum = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < AG_WARPS; ++w) {
            const float f = m_s[w][r] == -INFINITY ? 0.f : expf(m_s[w][r] - top);      // a warp without a chunk: nothing
            sum = fmaf(merged[w * R * hd + e], f, sum);
            den = fmaf(l_s[w][r], f, den);
        }
        // a sink: one more term exp(sink - m) in the denominator, with no value (sink = -inf: none, the term is 0);
        // head_sinks: a score per query head instead of the one for all
        const float inv_l = 1.0f / (den + expf((head_sinks ? head_sinks[row_head(r)] : sink) - top));
        out[((size_t)row_token(r) * nh + row_head(r)) * hd + (e - r * hd)] = from_f32<T>(sum * inv_l);
    }
}

template <typename T, int R, int NI>
static int launch_generic(const void* q, const void* cache, void* out, const int* block_table, int bt_stride, const int* seq_of_token,
                          const int* positions, int n_tokens, int nh, int nkv, int hd, int page_size, int window, int keep_first,
                          float scale, float sink, const float* head_sinks, long long n_pages, int* err_flag, int n_seqs, cudaStream_t stream) {
    const int n_rep = nh / nkv, hgroups = ceil_div(n_rep, R), hpg = ceil_div(n_rep, hgroups);
    // several tokens in a CTA where a kv head's query heads leave room: tokens of a prompt share their keys.  Not when every
    // token is a sequence of its own (they would be walked one after the other), nor while one token each does not fill the SMs twice.
    int tpg = R / hpg;
    if (n_tokens <= n_seqs || (long long)n_tokens * nkv * hgroups < 2ll * pyre_sm_count()) tpg = 1;
    const size_t smem = ((size_t)R * hd + AG_WARPS * 32 * R + (size_t)AG_WARPS * R * hd) * sizeof(float);
    static_assert((R * NI * 128 + AG_WARPS * 32 * R + AG_WARPS * R * NI * 128) * 4 <= 47 * 1024, "fits without an attribute");
    const dim3 grid(ceil_div(n_tokens, tpg), nkv * hgroups);
    const auto kernel = (long long)grid.x * grid.y <= pyre_sm_count() ? paged_attention_generic_kernel<T, R, NI, true> : paged_attention_generic_kernel<T, R, NI, false>;
    return (int)pyre_launch(kernel, grid, dim3(AG_WARPS * 32), smem, stream,
                            (const T*)q, (const T*)cache, (T*)out, block_table, bt_stride, seq_of_token, positions,
                            n_tokens, nh, nkv, hd, page_size, window, keep_first, scale, sink, head_sinks, n_pages, err_flag, hpg, hgroups, tpg);
}

PYRE_API int pyre_paged_attention_generic(const void* q, const void* cache, void* out, const int* block_table,
                                          int bt_stride, const int* seq_of_token, const int* positions,
                                          int n_tokens, int nh, int nkv, int hd, int page_size, int window,
                                          int keep_first, float scale, float sink, const float* head_sinks, int dtype, long long n_pages,
                                          int* err_flag, int n_seqs, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (hd % 8 || hd > 256 || hd <= 0 || nkv <= 0 || nh % nkv || page_size <= 0 || keep_first < 0) return PYRE_ERR_BAD_ARG;
#define GO(T, R, NI) launch_generic<T, R, NI>(q, cache, out, block_table, bt_stride, seq_of_token, positions, n_tokens, nh, nkv, hd, page_size, \
                                              window, keep_first, scale, sink, head_sinks, n_pages, err_flag, n_seqs, stream)
    int rc;
    if (dtype == PYRE_F32) rc = hd <= 128 ? GO(float, 8, 1) : GO(float, 4, 2);
    else if (dtype == PYRE_BF16) rc = hd <= 128 ? GO(__nv_bfloat16, 8, 1) : GO(__nv_bfloat16, 4, 2);
    else return PYRE_ERR_BAD_ARG;
#undef GO
    if (rc) return rc;
    PYRE_LAUNCH_CHECK();
    return 0;
}
