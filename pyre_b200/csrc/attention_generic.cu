// Paged attention over the block table, any head size that is a multiple of 16, any
// page size, float32 or bfloat16 storage, fp32 arithmetic throughout.
//
// This is the exact kernel: it serves the whole 32-bit path and every head size the
// tensor-core kernels do not cover.  Eight warps share a group of one to eight rows, a row being one
// (query token, query head): query heads of one key/value head, of one token or of a few
// neighbouring ones.  The keys are cut into chunks of 32, aligned to multiples of 32 from position 0;
// warp w walks the chunks w, w + 8, ... (chain w) for all rows at once, a row with an online softmax of its own
// (running maximum m, sum l and an fp32 accumulator), and the eight chains' results are merged in
// their order at the end.  Prompt portions and single decoded tokens are the same
// case: a query at absolute position p sees the cached keys lo..p, where
// lo = max(0, p - window + 1) with a window and 0 without (and, with a window, the first
// `keep_first` positions of the sequence, however far back); the keys of the current
// portion were written to the pages before this kernel runs.
//
// What bounds it: a few decoded tokens, the latency of a warp's chain of chunks (hence eight warps on a row); prompts,
// the reads of keys and queries beside the multiplications (hence the rows that share a key: one load of it serves all of them).
// How many rows share, and the figures: launch_generic_rows.
//
// The arithmetic of a row depends on nothing but its own keys: which warp takes a chunk is
// decided by the chunk's place in the sequence, a chunk or key that a row does not see leaves the row alone, and every
// sum has a fixed order, so the result is bit-identical however the tokens were cut into steps, whatever else is
// in the batch, whichever rows share a group or a CTA and wherever the pages lie.
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
// the group), token first: `tpg` tokens of `hpg` heads, hpg * tpg <= R; blockIdx.y (and .z) is the head group: kv head, and which
// of its `hgroups` groups of query heads.  Warp w takes chain w of the rows' chunks.
// SHORT: tables of at most 256 keys, so that a chain is one chunk and most chains of short rows are empty.  A CTA then owns `per_cta` groups
// of rows; as many warps share a group as its longest row has chunks, and the groups that do not fit follow in passes.
// DEEP: a few CTAs only (decoded tokens), each alone on its SM: a warp's chain of memory latencies is what counts, so it asks
// for eight pieces of a key row and sixteen value rows at a time, with twice the registers.
template <typename T, int R, int NI, bool DEEP, bool SHORT>
__global__ void __launch_bounds__(AG_WARPS * 32, DEEP ? 1 : R * NI <= 2 ? 3 : 2) paged_attention_generic_kernel(
    const T* q,             // [n_tokens, nh, hd]
    const T* cache,         // one layer: [page][2][nkv][page_size][hd]
    T* out,                 // [n_tokens, nh * hd]
    const int* block_table, // [n_seqs, bt_stride] logical page -> physical page (or -1)
    int bt_stride,
    const int* seq_of_token,  // [n_tokens]
    const int* positions,     // [n_tokens]
    int n_tokens, int nh, int nkv, int hd, int page_size, int window, int keep_first, float scale, float sink, const float* head_sinks, long long n_pages, int* err_flag,
    int hpg, int hgroups, int tpg, int per_cta) {
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, groups = SHORT ? per_cta : 1;
    float* const qs_all = smem;                                            // [groups][R][hd]
    float* const my_ps = smem + groups * R * hd + warp * 32 * R;           // [warps][32 keys][R] probabilities of a chunk, -1: the row does not see the key
    float* const merged_all = smem + groups * R * hd + AG_WARPS * 32 * R;  // [warps][R][hd]
    __shared__ float m_all[AG_WARPS * R], l_all[AG_WARPS * R], f_all[AG_WARPS * R], inv_all[AG_WARPS * R];
    __shared__ int seq_all[AG_WARPS * R], pos_all[AG_WARPS * R], lo_all[AG_WARPS * R], last_pos;
    pdl_trigger();
    pdl_wait();
    const int head_group = blockIdx.y + gridDim.y * blockIdx.z;                // a grid's second dimension ends at 65,535
    if (head_group >= nkv * hgroups) return;                                   // the whole CTA
    const int n_rep = nh / nkv, kvh = head_group / hgroups;
    const int first_head = (head_group - kvh * hgroups) * hpg;                 // within the kv head's query heads
    const int heads = min(hpg, n_rep - first_head);
    const int t_cta = blockIdx.x * groups * tpg;
    // row r of group g: its token, or -1 where there is no such row
    auto token_of = [&](int g, int r) {
        const int t = r / hpg;
        return t < tpg && t_cta + g * tpg + t < n_tokens ? t_cta + g * tpg + t : -1;
    };
    auto head_of = [&](int r) { return kvh * n_rep + first_head + r % hpg; };
    static_assert(!SHORT || AG_WARPS * R <= 32, "the rows' positions are looked at by one warp");
    if (threadIdx.x < (SHORT ? 32 : R)) {
        const int g = threadIdx.x / R, r = threadIdx.x - g * R, t = g < groups ? token_of(g, r) : -1;
        const bool live = t >= 0 && r % hpg < heads;
        const int pos = live ? positions[t] : -1;
        if (g < groups) {
            seq_all[threadIdx.x] = t >= 0 ? seq_of_token[t] : -1;
            pos_all[threadIdx.x] = pos;                                        // negative: sees no key
            lo_all[threadIdx.x] = !live ? -1 : (pos >= 0 && window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
        }
        if (SHORT) {
            const int top = __reduce_max_sync(0xffffffffu, pos);
            if (threadIdx.x == 0) last_pos = top;
        }
    }
    for (int e = threadIdx.x; e < groups * R * hd; e += AG_WARPS * 32) {
        const int gr = e / hd, d = e - gr * hd, g = gr / R, r = gr - g * R, t = token_of(g, r);
        qs_all[e] = (t >= 0 && r % hpg < heads) ? to_f32<T>(q[((size_t)t * nh + head_of(r)) * hd + d]) : 0.f;
    }
    __syncthreads();
    int gw = AG_WARPS;      // warps that share a group
    if (SHORT) gw = max(last_pos < 32 ? 1 : last_pos < 64 ? 2 : last_pos < 128 ? 4 : 8, AG_WARPS / groups);
    const int slot = warp / gw, chain = warp - slot * gw, gt = chain * 32 + lane, threads = gw * 32;
    float* const m_s = m_all + slot * gw * R;                              // [gw][R]
    float* const l_s = l_all + slot * gw * R;
    float* const f_s = f_all + slot * gw * R;
    float* const inv_s = inv_all + slot * R;
    float* const merged = merged_all + slot * gw * R * hd;                 // [gw][R][hd]
    auto sync_group = [&]() {      // the warps of a group; each group has a barrier of its own
        if (!SHORT) __syncthreads();
        else if (gw == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(threads) : "memory");
    };

    constexpr int U = DEEP ? 16 / NI : R <= 2 ? 8 / NI : 4;      // value rows fetched together
    constexpr int PV = R < 4 ? R : 4;          // probabilities read together
    const int keep = window > 0 ? keep_first : 0;
    for (int group = slot; group < groups; group += AG_WARPS / gw) {
        const float* qs = qs_all + group * R * hd;
        const int* row_seq = seq_all + group * R;
        const int* row_pos = pos_all + group * R;
        const int* row_lo = lo_all + group * R;
        const int rows = max(0, min(tpg, n_tokens - (t_cta + group * tpg))) * hpg;
        float acc[R][4 * NI], m[R], l[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            m[r] = -INFINITY;
            l[r] = 0.f;
#pragma unroll
            for (int i = 0; i < 4 * NI; ++i) acc[r][i] = 0.f;
        }
        // the first chunk from c on that is this warp's
        auto mine = [&](int c) { return c + 32 * ((chain - (c >> 5)) & (AG_WARPS - 1)); };
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
#pragma unroll (DEEP ? 8 : R <= 2 ? 4 : 2)
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
                // every row of the group sees the same keys of this chunk: no row needs to be asked key by key below
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
                        for (int r4 = 0; r4 < R; r4 += PV) {
                            const Vec<float, PV> pj = load_vec<float, PV>(my_ps + ((j0 + u) & 31) * R + r4);
#pragma unroll
                            for (int e = 0; e < PV; ++e)
                                if (alike || !(pj.v[e] < 0.f)) {
#pragma unroll
                                    for (int i = 0; i < 4 * NI; ++i) part[r4 + e][i] = fmaf(pj.v[e], val[u][i], part[r4 + e][i]);
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
        // the chains' results, merged in their order
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (lane == 0) {
                m_s[chain * R + r] = m[r];
                l_s[chain * R + r] = l[r];
            }
#pragma unroll
            for (int i = 0; i < NI; ++i)
                if (4 * lane + 128 * i < hd)
                    *reinterpret_cast<float4*>(merged + (chain * R + r) * hd + 4 * lane + 128 * i) =
                        make_float4(acc[r][4 * i], acc[r][4 * i + 1], acc[r][4 * i + 2], acc[r][4 * i + 3]);
        }
        sync_group();
        if (gt < R && row_lo[gt] >= 0) {      // a thread per row: what the chains count for, and the denominator
            const int r = gt;
            float top = -INFINITY, den = 0.f;
            for (int w = 0; w < gw; ++w) top = fmaxf(top, m_s[w * R + r]);
            for (int w = 0; w < gw; ++w) {
                const float f = m_s[w * R + r] == -INFINITY ? 0.f : expf(m_s[w * R + r] - top);      // a chain without a chunk: nothing
                f_s[w * R + r] = f;
                den = fmaf(l_s[w * R + r], f, den);
            }
            // a sink: one more term exp(sink - m) in the denominator, with no value (sink = -inf: none, the term is 0);
            // head_sinks: a score per query head instead of the one for all
            inv_s[r] = 1.0f / (den + expf((head_sinks ? head_sinks[head_of(r)] : sink) - top));
        }
        sync_group();
        for (int e = gt; e < R * hd; e += threads) {
            const int r = e / hd;
            if (row_lo[r] < 0) continue;      // a row that is not there
            float sum = 0.f;
            for (int w = 0; w < gw; ++w) sum = fmaf(merged[w * R * hd + e], f_s[w * R + r], sum);
            out[((size_t)token_of(group, r) * nh + head_of(r)) * hd + (e - r * hd)] = from_f32<T>(sum * inv_s[r]);
        }
        if (SHORT) sync_group();      // the next pass writes where this one reads
    }
}

struct GenericArgs {
    const void *q, *cache;
    void* out;
    const int* block_table;
    int bt_stride;
    const int *seq_of_token, *positions;
    int n_tokens, nh, nkv, hd, page_size, window, keep_first;
    float scale, sink;
    const float* head_sinks;
    long long n_pages;
    int* err_flag;
    cudaStream_t stream;
};

// How rows share CTAs: query heads per group, their groups per kv head, tokens per group, groups per CTA.
struct GenericPlan {
    int hpg, hgroups, tpg, per_cta;
};

// groups of a CTA at most: what 48 KB of shared memory hold
constexpr int most_per_cta(int R, int NI) { return R * NI <= 4 ? AG_WARPS : 2; }

template <typename T, int R, int NI, bool DEEP, bool SHORT>
static int launch_generic_as(const GenericArgs& a, const GenericPlan& p) {
    const size_t smem = ((size_t)p.per_cta * R * a.hd + AG_WARPS * 32 * R + (size_t)AG_WARPS * R * a.hd) * sizeof(float);
    static_assert(((SHORT ? AG_WARPS + most_per_cta(R, NI) : AG_WARPS + 1) * R * NI * 128 + AG_WARPS * 32 * R) * 4 <= 46 * 1024, "fits without an attribute");
    const int head_groups = a.nkv * p.hgroups, across = min(head_groups, 32768);
    const dim3 grid(ceil_div(ceil_div(a.n_tokens, p.tpg), p.per_cta), across, ceil_div(head_groups, across));
    return (int)pyre_launch(paged_attention_generic_kernel<T, R, NI, DEEP, SHORT>, grid, dim3(AG_WARPS * 32), smem, a.stream,
                            (const T*)a.q, (const T*)a.cache, (T*)a.out, a.block_table, a.bt_stride, a.seq_of_token, a.positions,
                            a.n_tokens, a.nh, a.nkv, a.hd, a.page_size, a.window, a.keep_first, a.scale, a.sink, a.head_sinks, a.n_pages, a.err_flag,
                            p.hpg, p.hgroups, p.tpg, p.per_cta);
}

template <typename T, int R, int NI>
static int launch_generic(const GenericArgs& a, GenericPlan p, bool is_short) {
    const long long sms = pyre_sm_count(), groups = (long long)ceil_div(a.n_tokens, p.tpg) * a.nkv * p.hgroups;
    if constexpr (R <= 4) {
        // short tables: several groups in a CTA while that leaves three CTAs for two SMs.  Fewer groups than that keep a CTA each, whose
        // idle warps cost nothing there
        while (is_short && p.per_cta < most_per_cta(R, NI) && groups * 2 >= sms * 3 * (p.per_cta * 2)) p.per_cta *= 2;
        if (p.per_cta > 1) return launch_generic_as<T, R, NI, false, true>(a, p);
    }
    return groups <= sms ? launch_generic_as<T, R, NI, true, false>(a, p) : launch_generic_as<T, R, NI, false, false>(a, p);
}

// The most rows whose groups still fill the SMs: 1.5 groups of eight per SM, 0.6 of four or two (few groups are bound by the
// chain of a warp's latencies, which more rows make longer); more than half of a group's rows have to be live.  Tables of a chunk or two: at most two
// rows, of up to eight chunks: at most four.  Tokens share a group only where the sequences (at most `n_seqs`) bring four groups each on
// average: rows of different sequences are walked one after the other.  Measured with float32 storage (us: a warp per row / eight warps
// and always eight rows / by this rule): 32 query heads on 32 of 128, 64 decoded tokens after some 1,600 keys 1040 / 1253 / 597, after 20 keys 15 / 106 /
// 18, 16 after 1,200 beside a portion of 200 679 / 1268 / 467; 28 on 4, four after 400 keys 116 / 34 / 17, 64 after 1,600 819 / 226 / 228,
// one after 20 7.7 / 14.3 / 5.9, a prompt of 509 571 / 256 / 254; 40 on 8, six prompts of 100 201 / 300 / 208.
template <typename T, int NI>
static int launch_generic_rows(const GenericArgs& a, int n_seqs, int bt_width) {
    const int n_rep = a.nh / a.nkv;
    const long long sms = pyre_sm_count(), most_keys = (long long)bt_width * a.page_size;
    const bool is_short = most_keys <= 32 * AG_WARPS;
    GenericPlan p{1, n_rep, 1, 1};
    int R = most_keys <= 64 ? 2 : is_short || NI > 1 ? 4 : 8;
    for (; R > 1; R /= 2) {
        p.hgroups = ceil_div(n_rep, R);
        p.hpg = ceil_div(n_rep, p.hgroups);
        p.tpg = R / p.hpg;
        while (p.tpg > 1 && a.n_tokens < 4ll * p.tpg * n_seqs) p.tpg /= 2;
        const long long groups = (long long)ceil_div(a.n_tokens, p.tpg) * a.nkv * p.hgroups;
        if (p.hpg * p.tpg > R / 2 && groups * 10 >= sms * (R == 8 ? 15 : 6)) break;
    }
    if constexpr (NI == 1) {
        if (R == 8) return launch_generic<T, 8, NI>(a, p, false);
    }
    if (R == 4) return launch_generic<T, 4, NI>(a, p, is_short);
    if (R == 2) return launch_generic<T, 2, NI>(a, p, is_short);
    p.hgroups = n_rep;
    p.hpg = p.tpg = 1;
    return launch_generic<T, 1, NI>(a, p, is_short);
}

PYRE_API int pyre_paged_attention_generic(const void* q, const void* cache, void* out, const int* block_table,
                                          int bt_stride, const int* seq_of_token, const int* positions,
                                          int n_tokens, int nh, int nkv, int hd, int page_size, int window,
                                          int keep_first, float scale, float sink, const float* head_sinks, int dtype, long long n_pages,
                                          int* err_flag, int n_seqs, int bt_width, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (hd % 8 || hd > 256 || hd <= 0 || nkv <= 0 || nh % nkv || page_size <= 0 || keep_first < 0) return PYRE_ERR_BAD_ARG;
    const GenericArgs a{q, cache, out, block_table, bt_stride, seq_of_token, positions, n_tokens, nh, nkv, hd, page_size, window, keep_first,
                        scale, sink, head_sinks, n_pages, err_flag, stream};
    int rc;
    if (dtype == PYRE_F32) rc = hd <= 128 ? launch_generic_rows<float, 1>(a, n_seqs, bt_width) : launch_generic_rows<float, 2>(a, n_seqs, bt_width);
    else if (dtype == PYRE_BF16) rc = hd <= 128 ? launch_generic_rows<__nv_bfloat16, 1>(a, n_seqs, bt_width) : launch_generic_rows<__nv_bfloat16, 2>(a, n_seqs, bt_width);
    else return PYRE_ERR_BAD_ARG;
    if (rc) return rc;
    PYRE_LAUNCH_CHECK();
    return 0;
}
