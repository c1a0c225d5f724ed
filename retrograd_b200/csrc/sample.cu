// On-device sampling for the step's output rows.
//
// A row of 128 256 logits read a dozen times by one block took 2.1 ms for 30 rows and 5.6 ms for 320 (top_k 20): the
// passes were serial, and most of them only looked for values that top_k had removed long before. Rows are now cut
// into chunks of 4096 logits that separate blocks read ONCE (sample_chunk_kernel: maximum, sum of exponentials, and the
// chunk's candidates for the largest `need` values), and one block per row finishes from the chunks' results
// (sample_kernel, row_from_chunks). The general passes remain for rows the chunks cannot serve: grammar masks, forced
// tokens, a nucleus over the whole vocabulary, a top_k whose candidates would not fit (sample_candidates_fit), rows whose
// ties overflow a candidate list, and rows with a NaN, an infinite maximum or a negative zero among their candidates.
//
// What is reproduced from the reference's CPU oracle
// (crates/retrograd-ffi/runtime/src/retro_gen_core.cpp:41-51,103-225,718-875,2942-2985):
//   - logprob = logit - max - log(sum exp(logit - max)), the sum taken in double;
//   - top logprobs ordered by (logit desc, id asc);
//   - probabilities p_i = exp((l_i - max) / T) in double; nucleus = highest-probability tokens
//     whose mass first reaches top_p * total; v2 order bias -> penalties -> top_k -> min_p ->
//     temperature -> top_p -> draw.
// What differs by design: the uniform draw comes from a counter-based generator (Philox4x32-10
// keyed by the request seed, counter = the request's draw index) instead of std::mt19937, and
// the cumulative draw walks the kept tokens in id order. Greedy rows (top_k == 1, or a nucleus
// that holds a single token) pick the arg-max with the lowest id on ties and are exact.
// Every reduction has a fixed order, so a (seed, draw index, logits) triple always yields the
// same token.

#include "kernels.cuh"

#include <cfloat>

namespace rb200 {

namespace {

constexpr int kThreads = kSampleRowThreads;
constexpr uint32_t kFlagV2 = 1u, kFlagWantLogprob = 2u, kFlagGreedyFast = 4u, kFlagChunked = kSampleFlagChunked;

constexpr int kChunk = kSampleChunk, kChunkThreads = kSampleChunkThreads;
constexpr int kChunkCands = kSampleChunkCands, kRowCands = kSampleRowCands;
constexpr int kListMax = 256;                   // values at or above the row's need-th largest (ties included)

struct ChunkStat {
    double sum;      // sum of exp(l - max) over the chunk's raw logits, fixed order
    double tsum;     // sum of exp((e - emax) / T) over its edited logits; only for rows without top_k
    float max;
    int32_t arg;     // lowest id holding the maximum
    float emax;      // maximum of the edited logits
    int32_t earg;
    int32_t count;   // candidates found (more than kChunkCands: the list is incomplete)
    int32_t pad[3];
};
static_assert(sizeof(ChunkStat) == 48, "ChunkStat layout");

struct Cand {
    float v;
    int32_t id;
};

struct Shared {
    double dwarp[32];
    float fwarp[32];
    int32_t iwarp[32];
    unsigned long long hist[256];
    double dval;
    float fval;
    int32_t ival;
    int32_t ival2;
    uint32_t uval;
    unsigned long long ullval;
    unsigned long long ullval2;
};

// Integers in the order of the floats; a positive NaN comes above them all. The bits are moved out by hand: as a plain cast the
// compiler may set the sign bit with a float negation, which gives NaNs other bits (they then ranked with the negative zero).
__device__ __forceinline__ uint32_t order_key(float f) {
    uint32_t u;
    asm("mov.b32 %0, %1;" : "=r"(u) : "f"(f));
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ void philox4x32(uint32_t k0, uint32_t k1, uint32_t (&c)[4]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c[0];
        const uint64_t p1 = (uint64_t)0xCD9E8D57u * c[2];
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c[1] ^ k0;
        const uint32_t n1 = (uint32_t)p1;
        const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c[3] ^ k1;
        const uint32_t n3 = (uint32_t)p0;
        c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
}

__device__ double philox_uniform(uint32_t seed, uint32_t draw_lo, uint32_t draw_hi) {
    uint32_t c[4] = {draw_lo, draw_hi, 0u, 0u};
    philox4x32(seed, 0x5EEDB200u, c);
    const uint64_t bits = (((uint64_t)c[0] << 32) | c[1]) >> 11;
    return (double)bits * (1.0 / 9007199254740992.0);
}

// (value desc, id asc) arg-max over the block. Result broadcast to every thread.
__device__ void block_argmax(Shared & sh, float v, int32_t id, float & out_v, int32_t & out_id) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int32_t oi = __shfl_xor_sync(0xffffffffu, id, o);
        if (ov > v || (ov == v && oi < id)) { v = ov; id = oi; }
    }
    __syncthreads();
    if (lane == 0) { sh.fwarp[wid] = v; sh.iwarp[wid] = id; }
    __syncthreads();
    if (wid == 0) {
        v = sh.fwarp[lane];
        id = sh.iwarp[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int32_t oi = __shfl_xor_sync(0xffffffffu, id, o);
            if (ov > v || (ov == v && oi < id)) { v = ov; id = oi; }
        }
        if (lane == 0) { sh.fval = v; sh.ival = id; }
    }
    __syncthreads();
    out_v = sh.fval;
    out_id = sh.ival;
}

// Fixed-order sum of doubles over the block, broadcast.
__device__ double block_sum(Shared & sh, double v) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sh.dwarp[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = sh.dwarp[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) sh.dval = v;
    }
    __syncthreads();
    return sh.dval;
}

// Exclusive prefix over threads in thread order; *total receives the block sum.
__device__ double block_exclusive_scan(Shared & sh, double v, double * total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    __syncthreads();
    if (lane == 31) sh.dwarp[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        double w = sh.dwarp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        sh.dwarp[lane] = w;
    }
    __syncthreads();
    const double pre = (wid ? sh.dwarp[wid - 1] : 0.0) + inc - v;
    if (total) *total = sh.dwarp[31];
    return pre;
}

__device__ int32_t block_exclusive_scan_int(Shared & sh, int32_t v, int32_t * total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    __syncthreads();
    if (lane == 31) sh.iwarp[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int32_t w = sh.iwarp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        sh.iwarp[lane] = w;
    }
    __syncthreads();
    const int32_t pre = (wid ? sh.iwarp[wid - 1] : 0) + inc - v;
    if (total) *total = sh.iwarp[31];
    return pre;
}

// Radix select over the descending order of logits. `by_mass`: weights are fixed-point
// probabilities and the walk stops when the accumulated weight reaches `target`; otherwise
// weights are 1 (a count). Returns the key of the last kept value in *thr_key, and the weight
// accumulated by strictly greater keys in *above.
__device__ void radix_select(Shared & sh, const float * __restrict__ l, int V, bool by_mass, float tmax, double inv_t,
                             unsigned long long target, uint32_t * thr_key, unsigned long long * above) {
    uint32_t prefix = 0;
    unsigned long long acc_above = 0;
    for (int digit = 3; digit >= 0; --digit) {
        __syncthreads();
        for (int b = threadIdx.x; b < 256; b += blockDim.x) sh.hist[b] = 0ull;
        __syncthreads();
        const int shift = digit * 8;
        for (int i = threadIdx.x; i < V; i += blockDim.x) {
            const float v = l[i];
            const uint32_t key = order_key(v);
            if (digit == 3 || (key >> (shift + 8)) == prefix) {
                unsigned long long w = 1ull;
                if (by_mass) w = (unsigned long long)(exp(((double)v - (double)tmax) * inv_t) * 1099511627776.0);
                if (w) atomicAdd(&sh.hist[(key >> shift) & 255u], w);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long acc = acc_above;
            int pick = 0;
            for (int b = 255; b >= 0; --b) {
                if (acc + sh.hist[b] >= target) { pick = b; break; }
                acc += sh.hist[b];
            }
            sh.ullval = acc;
            sh.uval = (prefix << 8) | (uint32_t)pick;
        }
        __syncthreads();
        prefix = sh.uval;
        acc_above = sh.ullval;
    }
    *thr_key = prefix;
    *above = acc_above;
}

__device__ __forceinline__ float edited(float v, const LogitEdit & ed) {
    float t = v + ed.bias;
    if (ed.repeat != 1.0f) t = t <= 0.0f ? t * ed.repeat : t / ed.repeat;
    return t - ed.subtract;
}

// Rows of the chunked paths by their options: the values that matter are the edited ones for v2 rows.
__device__ __forceinline__ bool truncates(const SampleDesc & d, int V) { return (d.flags & kFlagV2) && d.top_k > 0 && d.top_k < V; }
__device__ __forceinline__ int needed(const SampleDesc & d, int V, int top_stride) {
    return truncates(d, V) ? d.top_k : (int)min(d.n_top, (uint32_t)min(top_stride, V));
}

// One chunk of one row, read once into registers (16 values per thread). Bound by the double-precision exponentials
// of the log-sum (one per logit), not by memory: 257 rows of 201 088 logits take 130 us, 1.6 TB/s.
// Candidates: with `need` values wanted of the whole row, the need-th largest of the 256 per-thread maxima is a lower
// bound of the chunk's need-th largest value; everything at or above it goes to the list (a few more than `need`).
// CHUNKED: the step has rows that are served from candidate lists. A step of greedy rows alone takes the form without them,
// whose smaller register and shared-memory need lets more blocks hide the exponentials' latency.
template <bool CHUNKED>
__global__ void __launch_bounds__(kChunkThreads) sample_chunk_kernel(const float * __restrict__ raw_logits, int V, const SampleDesc * __restrict__ descs,
                                                                     const LogitEdit * __restrict__ edits, ChunkStat * __restrict__ stats,
                                                                     Cand * __restrict__ cands, int n_chunks, int top_stride) {
    const int row = blockIdx.y, chunk = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const SampleDesc d = descs[row];
    if (!(d.flags & (CHUNKED ? kFlagGreedyFast | kFlagChunked : kFlagGreedyFast))) return;
    constexpr int PER = kChunk / kChunkThreads;
    __shared__ float s_max[kChunkThreads / 32];
    __shared__ int32_t s_arg[kChunkThreads / 32];
    __shared__ double s_sum[kChunkThreads / 32];
    const float * l = raw_logits + (size_t)row * V;
    const int base = chunk * kChunk;
    float v[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = base + j * kChunkThreads + tid;
        v[j] = i < V ? l[i] : -INFINITY;
    }
    auto block_max = [&](float & m, int32_t & a) {
        m = -INFINITY;
        a = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (v[j] > m) { m = v[j]; a = base + j * kChunkThreads + tid; }       // ascending ids: the first maximum wins
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float om = __shfl_xor_sync(0xffffffffu, m, o);
            const int32_t oa = __shfl_xor_sync(0xffffffffu, a, o);
            if (om > m || (om == m && oa < a)) { m = om; a = oa; }
        }
        __syncthreads();
        if (lane == 0) { s_max[wid] = m; s_arg[wid] = a; }
        __syncthreads();
        m = s_max[0];
        a = s_arg[0];
#pragma unroll
        for (int w = 1; w < kChunkThreads / 32; ++w)
            if (s_max[w] > m || (s_max[w] == m && s_arg[w] < a)) { m = s_max[w]; a = s_arg[w]; }
    };
    auto block_exp_sum = [&](float m, double inv_t) {       // the sum, in thread 0
        double part = 0.0;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int i = base + j * kChunkThreads + tid;
            if (i < V) part += exp(((double)v[j] - (double)m) * inv_t);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        __syncthreads();
        if (lane == 0) s_sum[wid] = part;
        __syncthreads();
        double sum = 0.0;
        if (tid == 0) {
#pragma unroll
            for (int w = 0; w < kChunkThreads / 32; ++w) sum += s_sum[w];
        }
        return sum;
    };
    ChunkStat st;
    block_max(st.max, st.arg);
    st.sum = block_exp_sum(st.max, 1.0);
    st.emax = st.max;
    st.earg = st.arg;
    st.tsum = st.sum;
    st.count = 0;
    st.pad[0] = st.pad[1] = st.pad[2] = 0;
    if (CHUNKED && (d.flags & kFlagChunked)) {
        __shared__ float s_val[CHUNKED ? kChunk : 1];
        __shared__ int s_count;
        const uint32_t n_edits = (d.flags & kFlagV2) ? d.edit_end - d.edit_begin : 0u;
        if (n_edits) {
#pragma unroll
            for (int j = 0; j < PER; ++j) s_val[j * kChunkThreads + tid] = v[j];
            __syncthreads();
            for (uint32_t e = tid; e < n_edits; e += kChunkThreads) {       // one edit per distinct id
                const LogitEdit ed = edits[d.edit_begin + e];
                const int at = ed.id - base;
                if (at >= 0 && at < kChunk && ed.id < V) s_val[at] = edited(s_val[at], ed);
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < PER; ++j) v[j] = s_val[j * kChunkThreads + tid];
            block_max(st.emax, st.earg);
        }
        const double inv_t = 1.0 / (double)d.temperature;
        if (!truncates(d, V) && (n_edits || inv_t != 1.0)) st.tsum = block_exp_sum(st.emax, inv_t);
        const int need = needed(d, V, top_stride);
        if (need > 0) {
            uint32_t mine = 0;
#pragma unroll
            for (int j = 0; j < PER; ++j) mine = max(mine, order_key(v[j]));
            uint32_t bound = 0;        // the need-th largest of the threads' maxima, bit by bit
            for (int bit = 31; bit >= 0; --bit) {
                const uint32_t t = bound | (1u << bit);
                if (__syncthreads_count(mine >= t) >= need) bound = t;
            }
            if (bound == order_key(0.f)) bound = order_key(-0.f);       // equal values are handed on together
            if (tid == 0) s_count = 0;
            __syncthreads();
            Cand * list = cands + ((size_t)row * n_chunks + chunk) * kChunkCands;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int i = base + j * kChunkThreads + tid;
                if (i < V && order_key(v[j]) >= bound) {
                    const int at = atomicAdd(&s_count, 1);       // (the order in the list does not matter)
                    if (at < kChunkCands) list[at] = Cand{v[j], i};
                }
            }
            __syncthreads();
            st.count = s_count;
        }
    }
    if (tid == 0) stats[(size_t)row * n_chunks + chunk] = st;
}

// What row_from_chunks works with besides Shared.
struct RowShared {
    float cv[kRowCands];            // the row's candidates; later the drawn chunk's edited logits
    int32_t cid[kRowCands];
    float sv[kListMax];             // the kept values, largest first (ties: lowest id first)
    int32_t sid[kListMax];
    double p[kListMax];
    float lv[kListMax];             // the list before it is ordered
    int32_t lid[kListMax];
    int32_t by_id[kListMax];        // kept entries in id order
    int32_t offset[kThreads];       // first candidate of each chunk
    double total, rtotal, mass, prefix;
    float rmax, tmax, token_logit;
    int32_t rarg, targ, n_keep, token, chunk, n_list;
};

// The last step of a row whose chunks hold everything it needs; false when they do not (more ties than the lists take, a
// NaN, an infinite maximum, a negative zero among the candidates): the caller then runs the general passes. Follows the general kernel's rules line by line (the comments there).
__device__ bool row_from_chunks(Shared & sh, RowShared & rs, const float * __restrict__ raw, int V, const SampleDesc & d, const LogitEdit * __restrict__ edits,
                                const ChunkStat * __restrict__ st, const Cand * __restrict__ cands, int n_chunks, SampleOut * __restrict__ out,
                                int32_t * __restrict__ top_ids, float * __restrict__ top_lps, int top_stride) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool v2 = (d.flags & kFlagV2) != 0, cut = truncates(d, V);
    const int need = needed(d, V, top_stride);
    const double inv_t = 1.0 / (double)d.temperature;
    // ---- the row's statistics from its chunks'
    if (wid == 0) {
        float m = -INFINITY, em = -INFINITY;
        int32_t a = 0x7fffffff, ea = 0x7fffffff;
        for (int c = lane; c < n_chunks; c += 32) {
            if (st[c].max > m || (st[c].max == m && st[c].arg < a)) { m = st[c].max; a = st[c].arg; }
            if (st[c].emax > em || (st[c].emax == em && st[c].earg < ea)) { em = st[c].emax; ea = st[c].earg; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float om = __shfl_xor_sync(0xffffffffu, m, o), oem = __shfl_xor_sync(0xffffffffu, em, o);
            const int32_t oa = __shfl_xor_sync(0xffffffffu, a, o), oea = __shfl_xor_sync(0xffffffffu, ea, o);
            if (om > m || (om == m && oa < a)) { m = om; a = oa; }
            if (oem > em || (oem == em && oea < ea)) { em = oem; ea = oea; }
        }
        double total = 0.0, ttotal = 0.0;
        for (int c = lane; c < n_chunks; c += 32) {
            total += st[c].sum * exp((double)st[c].max - (double)m);
            if (!cut) ttotal += st[c].tsum * exp(((double)st[c].emax - (double)em) * inv_t);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            total += __shfl_xor_sync(0xffffffffu, total, o);
            ttotal += __shfl_xor_sync(0xffffffffu, ttotal, o);
        }
        if (lane == 0) { rs.rmax = m; rs.rarg = a; rs.tmax = em; rs.targ = ea; rs.rtotal = total; rs.total = ttotal; }
    }
    __syncthreads();
    // a NaN or an infinite maximum (of the raw row, or by its edits) makes a sum a NaN: the general passes have their rules for those
    if (!(rs.rtotal < INFINITY) || !(fabsf(rs.tmax) < INFINITY) || (!cut && !(rs.total < INFINITY))) return false;
    // ---- the largest `need` values, exactly
    int n_list = 0;
    if (need > 0) {
        int32_t n_cand;
        int32_t mine = 0;
        bool over = false, unordered = false;
        if (tid < n_chunks) { mine = st[tid].count; over = mine > kChunkCands; }
        const int32_t first = block_exclusive_scan_int(sh, mine, &n_cand);
        rs.offset[tid] = first;
        if (__syncthreads_or(over) || n_cand > kRowCands) return false;
        for (int c = wid; c < n_chunks; c += kThreads / 32) {
            const int n = st[c].count, at = rs.offset[c];
            for (int i = lane; i < n; i += 32) {
                const Cand e = cands[(size_t)c * kChunkCands + i];
                rs.cv[at + i] = e.v;
                rs.cid[at + i] = e.id;
                // the selection below goes by order_key, the order of the list by value: they differ for a NaN (edits can make one of
                // a finite row) and for the two zeros
                unordered = unordered || e.v != e.v || __float_as_uint(e.v) == 0x80000000u;
            }
        }
        if (__syncthreads_or(unordered)) return false;
        uint32_t key[kRowCands / kThreads];
        const int slots = (n_cand + kThreads - 1) / kThreads;
#pragma unroll
        for (int m = 0; m < kRowCands / kThreads; ++m) {
            const int i = m * kThreads + tid;
            key[m] = i < n_cand ? order_key(rs.cv[i]) : 0u;        // (no float has key 0)
        }
        auto count_from = [&](uint32_t t) {
            int n = 0;
#pragma unroll
            for (int m = 0; m < kRowCands / kThreads; ++m)
                if (m < slots) n += __syncthreads_count(key[m] >= t);
            return n;
        };
        uint32_t thr = 0;
        if (n_cand > need) {
            for (int bit = 31; bit >= 0; --bit) {
                const uint32_t t = thr | (1u << bit);
                if (count_from(t) >= need) thr = t;
            }
        }
        thr = max(thr, 1u);
        n_list = count_from(thr);
        if (n_list > kListMax) return false;
        if (tid == 0) rs.n_list = 0;
        __syncthreads();
#pragma unroll
        for (int m = 0; m < kRowCands / kThreads; ++m) {
            if (m < slots && key[m] >= thr) {
                const int at = atomicAdd(&rs.n_list, 1);
                rs.lv[at] = rs.cv[m * kThreads + tid];
                rs.lid[at] = rs.cid[m * kThreads + tid];
            }
        }
        __syncthreads();
        if (tid < n_list) {
            const float v = rs.lv[tid];
            const int32_t id = rs.lid[tid];
            int rank = 0;
            for (int i = 0; i < n_list; ++i) rank += rs.lv[i] > v || (rs.lv[i] == v && rs.lid[i] < id);
            rs.sv[rank] = v;
            rs.sid[rank] = id;
        }
        n_list = min(n_list, need);        // ties beyond the need-th value: the lowest ids stay
    }
    __syncthreads();
    const float rmax = rs.rmax;
    const double rlog = log(rs.rtotal);
    float tmax = rs.tmax;
    int32_t token;
    double kept;
    bool single;
    int n_keep = n_list;
    if (cut) {
        // ---- top_k, min_p, temperature and top_p on the kept list
        tmax = rs.sv[0];
        if (d.min_p > 0.0f) {
            const float thr = tmax + logf(d.min_p);
            n_keep = __syncthreads_count(tid < n_list && rs.sv[min(tid, kListMax - 1)] >= thr);
        }
        if (tid < n_keep) rs.p[tid] = exp(((double)rs.sv[tid] - (double)tmax) * inv_t);
        __syncthreads();
        const double total = block_sum(sh, tid < n_keep ? rs.p[tid] : 0.0);
        single = d.top_k == 1 || (double)d.top_p * total <= 1.0;
        if (!single && d.top_p < 1.0f) {
            const unsigned long long w = tid < n_keep ? (unsigned long long)(rs.p[tid] * 1099511627776.0) : 0ull;
            const double total_fixed = block_sum(sh, (double)w);
            unsigned long long target = (unsigned long long)((double)d.top_p * total_fixed);
            if (target < 1ull) target = 1ull;
            if (tid == 0) {
                unsigned long long above = 0;
                int keep = n_keep;
                for (int i = 0; i < n_keep;) {
                    int j = i + 1;
                    while (j < n_keep && rs.sv[j] == rs.sv[i]) ++j;
                    const unsigned long long one = (unsigned long long)(rs.p[i] * 1099511627776.0);
                    if (above + one * (unsigned long long)(j - i) >= target) {
                        const unsigned long long lack = target > above ? target - above : 1ull;
                        const unsigned long long ties = one ? (lack + one - 1) / one : 1ull;
                        keep = i + (int)min((unsigned long long)(j - i), max(ties, 1ull));
                        break;
                    }
                    above += one * (unsigned long long)(j - i);
                    i = j;
                }
                rs.n_keep = keep;
            }
            __syncthreads();
            n_keep = rs.n_keep;
        }
        if (single) {
            token = rs.sid[0];
            kept = 1.0;
        } else {
            if (tid < n_keep) {
                const int32_t id = rs.sid[tid];
                int rank = 0;
                for (int i = 0; i < n_keep; ++i) rank += rs.sid[i] < id;
                rs.by_id[rank] = tid;
            }
            __syncthreads();
            if (tid == 0) {
                double mass = 0.0;
                for (int i = 0; i < n_keep; ++i) mass += rs.p[rs.by_id[i]];
                const double draw = philox_uniform(d.seed, d.draw_lo, d.draw_hi) * mass;
                double acc = 0.0;
                int32_t pick = -1;
                for (int i = 0; i < n_keep; ++i) {
                    const double p = rs.p[rs.by_id[i]];
                    if (p <= 0.0) continue;
                    acc += p;
                    pick = rs.sid[rs.by_id[i]];
                    if (draw < acc) break;
                }
                rs.mass = mass;
                rs.token = pick;
            }
            __syncthreads();
            token = rs.token;
            kept = rs.mass;
        }
    } else {
        // ---- no truncation: the chunk the draw falls into, then the token within it
        single = (double)d.top_p * rs.total <= 1.0;
        kept = single ? 1.0 : rs.total;
        token = rs.targ;
        if (!single) {
            if (tid == 0) {
                const double draw = philox_uniform(d.seed, d.draw_lo, d.draw_hi) * rs.total;
                double acc = 0.0;
                int pick = -1;
                double before = 0.0;
                for (int c = 0; c < n_chunks; ++c) {
                    const double mass = st[c].tsum * exp(((double)st[c].emax - (double)tmax) * inv_t);
                    if (!(mass > 0.0)) continue;
                    pick = c;
                    before = acc;
                    acc += mass;
                    if (draw < acc) break;
                }
                rs.chunk = max(pick, 0);
                rs.prefix = before;
                rs.mass = draw;
                rs.token = -1;
            }
            __syncthreads();
            const int base = rs.chunk * kChunk;
            for (int i = tid; i < kChunk; i += kThreads) rs.cv[i] = base + i < V ? raw[base + i] : -INFINITY;
            __syncthreads();
            if (v2) {
                for (uint32_t e = d.edit_begin + tid; e < d.edit_end; e += kThreads) {
                    const LogitEdit ed = edits[e];
                    const int at = ed.id - base;
                    if (at >= 0 && at < kChunk && ed.id < V) rs.cv[at] = edited(rs.cv[at], ed);
                }
            }
            __syncthreads();
            constexpr int PER = kChunk / kThreads;
            double p[PER], mine = 0.0;
            int32_t my_last = -1;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                p[j] = base + tid * PER + j < V ? exp(((double)rs.cv[tid * PER + j] - (double)tmax) * inv_t) : 0.0;
                if (p[j] > 0.0) { mine += p[j]; my_last = base + tid * PER + j; }
            }
            const double before = rs.prefix + block_exclusive_scan(sh, mine, nullptr);
            const double draw = rs.mass;
            if (mine > 0.0 && draw >= before && draw < before + mine) {
                double acc = before;
                int32_t pick = -1;
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    acc += p[j];
                    if (pick < 0 && p[j] > 0.0 && draw < acc) pick = base + tid * PER + j;
                }
                rs.token = pick < 0 ? my_last : pick;
            }
            __syncthreads();
            if (rs.token < 0) {
                // rounding left the draw past the last boundary (or between two threads' sums): the chunk's last token
                float dummy;
                int32_t last;
                block_argmax(sh, (float)my_last, -my_last, dummy, last);
                token = (int32_t)dummy;
            } else {
                token = rs.token;
            }
        }
    }
    // ---- outputs
    const uint32_t n_top = min(d.n_top, (uint32_t)min(top_stride, V));
    if (n_top > 0 && !v2) {
        if ((uint32_t)tid < n_top) {
            top_ids[tid] = rs.sid[tid];
            top_lps[tid] = (float)((double)rs.sv[tid] - (double)rmax - rlog);
        }
    } else if (n_top > 0) {
        const uint32_t shown = single ? 1u : min(n_top, (uint32_t)n_keep);
        if ((uint32_t)tid < shown) {
            top_ids[tid] = single ? token : rs.sid[tid];
            top_lps[tid] = (float)log(exp(((double)(single ? tmax : rs.sv[tid]) - (double)tmax) * inv_t) / kept);
        }
        if (tid == 0) {
            // everything else was truncated away: ids in ascending order, probability zero
            int32_t id = 0;
            for (uint32_t j = shown; j < n_top; ++j, ++id) {
                for (bool taken = true; taken;) {
                    taken = false;
                    for (uint32_t i = 0; i < shown; ++i) taken = taken || (single ? token : rs.sid[i]) == id;
                    if (taken) ++id;
                }
                top_ids[j] = id;
                top_lps[j] = (float)log(exp(-INFINITY * inv_t) / kept);
            }
        }
    }
    if (token < 0 || token >= V) token = 0;      // a row of NaNs has no arg-max: stay inside the row
    const bool want_logprob = v2 && (d.flags & kFlagWantLogprob);
    if (want_logprob) {
        // the whole block looks for the token's edit: a long history has as many edits as distinct tokens
        if (tid == 0) rs.token_logit = raw[token];
        __syncthreads();
        for (uint32_t e = d.edit_begin + tid; e < d.edit_end; e += kThreads)
            if (edits[e].id == token) rs.token_logit = edited(raw[token], edits[e]);
        __syncthreads();
    }
    if (tid == 0) {
        SampleOut o;
        o.token = token;
        o.logprob = (float)((double)raw[token] - (double)rmax - rlog);
        o.sampled_logprob = want_logprob ? (float)log(exp(((double)rs.token_logit - (double)tmax) * inv_t) / kept) : 0.f;
        o.n_top = n_top;
        *out = o;
    }
    return true;
}

__global__ void __launch_bounds__(kThreads) sample_kernel(const float * __restrict__ raw_logits, float * __restrict__ work_logits, int V,
                                                          const SampleDesc * __restrict__ descs, const LogitEdit * __restrict__ edits,
                                                          const uint32_t * __restrict__ masks, const ChunkStat * __restrict__ stats,
                                                          const Cand * __restrict__ cands, int n_chunks, SampleOut * __restrict__ outs,
                                                          int32_t * __restrict__ top_ids, float * __restrict__ top_lps, int top_stride) {
    __shared__ Shared sh;
    extern __shared__ __align__(16) unsigned char row_shared[];
    const int row = blockIdx.x;
    const SampleDesc d = descs[row];
    if (d.flags & kFlagGreedyFast) return;      // served by greedy_finish_kernel
    const bool v2 = (d.flags & kFlagV2) != 0;
    const float * raw = raw_logits + (size_t)row * V;
    const int tid = threadIdx.x;
    if ((d.flags & kFlagChunked) &&
        row_from_chunks(sh, *reinterpret_cast<RowShared *>(row_shared), raw, V, d, edits, stats + (size_t)row * n_chunks,
                        cands + (size_t)row * n_chunks * kChunkCands, n_chunks, outs + row, top_ids + (size_t)row * top_stride,
                        top_lps + (size_t)row * top_stride, top_stride))
        return;
    // ---- the general passes: v2 rows transform a private copy of their row; v1 rows only read the raw one
    float * l = v2 ? work_logits + (size_t)row * V : const_cast<float *>(raw);
    __syncthreads();

    // ---- temperature-1 statistics of the raw row; the copy is written on the way (the barriers of the arg-max publish it). Eight
    // loads are in flight before the first store: one at a time, a row of 128 256 logits took 18 us longer.
    float rmax = -INFINITY;
    int32_t rarg = 0x7fffffff;
    if (v2) {
        float * __restrict__ work = work_logits + (size_t)row * V;
        for (int i0 = tid; i0 < V; i0 += 8 * kThreads) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = i0 + j * kThreads < V ? raw[i0 + j * kThreads] : -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int i = i0 + j * kThreads;
                if (i < V) work[i] = v[j];
                if (v[j] > rmax) { rmax = v[j]; rarg = i; }
            }
        }
    } else {
        for (int i = tid; i < V; i += kThreads) {
            const float v = l[i];
            if (v > rmax) { rmax = v; rarg = i; }
        }
    }
    block_argmax(sh, rmax, rarg, rmax, rarg);
    double part = 0.0;
    for (int i = tid; i < V; i += kThreads) part += exp((double)l[i] - (double)rmax);
    const double rlog = log(block_sum(sh, part));

    // ---- raw top logprobs (v1 rows report the temperature-1 policy)
    const uint32_t n_top = min(d.n_top, (uint32_t)min(top_stride, V));
    if (!v2 && n_top > 0) {
        float pv = INFINITY;
        int32_t pid = -1;
        for (uint32_t j = 0; j < n_top; ++j) {
            float bv = -INFINITY;
            int32_t bi = 0x7fffffff;
            for (int i = tid; i < V; i += kThreads) {
                const float v = l[i];
                const bool after = v < pv || (v == pv && i > pid);
                if (after && (v > bv || (v == bv && i < bi))) { bv = v; bi = i; }
            }
            block_argmax(sh, bv, bi, bv, bi);
            if (tid == 0) {
                top_ids[(size_t)row * top_stride + j] = bi;
                top_lps[(size_t)row * top_stride + j] = (float)((double)bv - (double)rmax - rlog);
            }
            pv = bv;
            pid = bi;
        }
    }

    // ---- v2 transformations, on the row's working copy
    const uint32_t n_edits = d.edit_end - d.edit_begin;
    __syncthreads();
    if (v2) {
        // logit_bias and penalties: one merged edit per distinct id
        for (uint32_t e = tid; e < n_edits; e += kThreads) {
            const LogitEdit ed = edits[d.edit_begin + e];
            l[ed.id] = edited(l[ed.id], ed);
        }
        __syncthreads();
        // grammar mask: one bit per token, tokens the grammar cannot continue with drop out here
        if (d.pad[0] != 0 && masks) {
            const uint32_t * bits = masks + (d.pad[0] - 1);
            for (int i = tid; i < V; i += kThreads)
                if (!((bits[i >> 5] >> (i & 31)) & 1u)) l[i] = -INFINITY;
            __syncthreads();
        }
        // top_k (count based, ties keep the lowest ids)
        if (d.top_k > 0 && d.top_k < V) {
            uint32_t thr;
            unsigned long long above;
            radix_select(sh, l, V, false, 0.f, 0.0, (unsigned long long)d.top_k, &thr, &above);
            const int32_t ties_keep = d.top_k - (int32_t)above;
            const int chunk = (V + kThreads - 1) / kThreads;
            const int c0 = min(V, tid * chunk), c1 = min(V, c0 + chunk);
            int32_t my_ties = 0;
            for (int i = c0; i < c1; ++i) my_ties += order_key(l[i]) == thr;
            int32_t rank = block_exclusive_scan_int(sh, my_ties, nullptr);
            for (int i = c0; i < c1; ++i) {
                const uint32_t key = order_key(l[i]);
                if (key < thr) {
                    l[i] = -INFINITY;
                } else if (key == thr) {
                    if (rank >= ties_keep) l[i] = -INFINITY;
                    ++rank;
                }
            }
            __syncthreads();
        }
        if (d.min_p > 0.0f) {
            float mv = -INFINITY;
            int32_t mi = 0;
            for (int i = tid; i < V; i += kThreads) mv = fmaxf(mv, l[i]);
            block_argmax(sh, mv, 0, mv, mi);
            const float thr = mv + logf(d.min_p);
            for (int i = tid; i < V; i += kThreads) if (l[i] < thr) l[i] = -INFINITY;
            __syncthreads();
        }
    }

    // ---- sampling distribution
    float tmax = rmax;
    int32_t targ = rarg;
    if (v2) {
        tmax = -INFINITY;
        targ = 0x7fffffff;
        for (int i = tid; i < V; i += kThreads) {
            const float v = l[i];
            if (v > tmax) { tmax = v; targ = i; }
        }
        block_argmax(sh, tmax, targ, tmax, targ);
    }
    const double inv_t = 1.0 / (double)d.temperature;
    part = 0.0;
    for (int i = tid; i < V; i += kThreads) part += exp(((double)l[i] - (double)tmax) * inv_t);
    const double total = block_sum(sh, part);

    int32_t token;
    double kept = total;
    uint32_t thr = 0;
    int32_t ties_keep = 0x7fffffff;
    const bool single = (v2 && d.top_k == 1) || (double)d.top_p * total <= 1.0;
    const bool nucleus = !single && d.top_p < 1.0f;
    if (nucleus) {
        // fixed-point masses make the selection independent of the order atomics land in
        double fp = 0.0;
        for (int i = tid; i < V; i += kThreads)
            fp += (double)(unsigned long long)(exp(((double)l[i] - (double)tmax) * inv_t) * 1099511627776.0);
        const double total_fixed = block_sum(sh, fp);
        unsigned long long target = (unsigned long long)((double)d.top_p * total_fixed);
        if (target < 1ull) target = 1ull;
        unsigned long long above;
        radix_select(sh, l, V, true, tmax, inv_t, target, &thr, &above);
        // weight of one token at the threshold
        float thr_val;
        {
            const uint32_t u = (thr & 0x80000000u) ? (thr & 0x7fffffffu) : ~thr;
            thr_val = __uint_as_float(u);
        }
        const unsigned long long w = (unsigned long long)(exp(((double)thr_val - (double)tmax) * inv_t) * 1099511627776.0);
        const unsigned long long need = target > above ? target - above : 1ull;
        ties_keep = w ? (int32_t)min((unsigned long long)0x7fffffff, (need + w - 1) / w) : 1;
        if (ties_keep < 1) ties_keep = 1;
    }

    if (single) {
        token = targ;
        kept = 1.0;   // exp(0) of the arg-max: the mass of a one-token nucleus
    } else {
        const int chunk = (V + kThreads - 1) / kThreads;
        const int c0 = min(V, tid * chunk), c1 = min(V, c0 + chunk);
        int32_t rank = 0;
        if (nucleus) {
            int32_t my_ties = 0;
            for (int i = c0; i < c1; ++i) my_ties += order_key(l[i]) == thr;
            rank = block_exclusive_scan_int(sh, my_ties, nullptr);
        }
        const int32_t rank0 = rank;
        double mine = 0.0;
        int32_t my_last = -1;
        for (int i = c0; i < c1; ++i) {
            const float v = l[i];
            bool keep = true;
            if (nucleus) {
                const uint32_t key = order_key(v);
                keep = key > thr || (key == thr && rank < ties_keep);
                if (key == thr) ++rank;
            }
            if (keep) {
                const double p = exp(((double)v - (double)tmax) * inv_t);
                if (p > 0.0) { mine += p; my_last = i; }
            } else if (v2) {
                l[i] = -INFINITY;   // v2 reports under the truncated distribution
            }
        }
        double kept_total;
        const double base = block_exclusive_scan(sh, mine, &kept_total);
        kept = kept_total;
        const double draw = philox_uniform(d.seed, d.draw_lo, d.draw_hi) * kept;
        if (tid == 0) { sh.ival2 = -1; }
        __syncthreads();
        if (mine > 0.0 && draw >= base && draw < base + mine) {
            double acc = base;
            int32_t pick = my_last;
            rank = rank0;
            for (int i = c0; i < c1; ++i) {
                const float v = l[i];
                bool keep = true;
                if (nucleus && !v2) {
                    const uint32_t key = order_key(v);
                    keep = key > thr || (key == thr && rank < ties_keep);
                    if (key == thr) ++rank;
                }
                if (!keep) continue;
                const double p = exp(((double)v - (double)tmax) * inv_t);
                if (p <= 0.0) continue;
                acc += p;
                if (draw < acc) { pick = i; break; }
            }
            sh.ival2 = pick;
        }
        __syncthreads();
        if (sh.ival2 < 0) {
            // rounding left the draw past the last boundary: the last kept token
            float dummy;
            int32_t last;
            block_argmax(sh, (float)my_last, -my_last, dummy, last);
            token = (int32_t)dummy;
        } else {
            token = sh.ival2;
        }
    }

    // ---- outputs
    __syncthreads();
    // A row whose reasoning budget is forcing reports the forced token in place of the drawn one (the draw still
    // happened: the request's counter moves as in the reference, which samples first and replaces afterwards).
    const int32_t drawn = token;
    const bool forced = d.pad[1] != 0;
    if (forced) token = (int32_t)d.pad[1] - 1;
    if (v2 && n_top > 0) {
        // post-transformation top-k: by probability desc (= transformed logit desc), id asc
        float pv = INFINITY;
        int32_t pid = -1;
        for (uint32_t j = 0; j < n_top; ++j) {
            float bv = -INFINITY;
            int32_t bi = 0x7fffffff;
            for (int i = tid; i < V; i += kThreads) {
                float v = l[i];
                if (single && i != drawn) v = -INFINITY;
                const bool after = v < pv || (v == pv && i > pid);
                if (after && (v > bv || (v == bv && i < bi))) { bv = v; bi = i; }
            }
            block_argmax(sh, bv, bi, bv, bi);
            if (tid == 0) {
                top_ids[(size_t)row * top_stride + j] = bi;
                top_lps[(size_t)row * top_stride + j] = (float)log(exp(((double)bv - (double)tmax) * inv_t) / kept);
            }
            pv = bv;
            pid = bi;
        }
    }
    if (token < 0 || token >= V) token = 0;      // a row of NaNs has no arg-max: stay inside the row
    if (tid == 0) {
        SampleOut o;
        o.token = token;
        o.logprob = (float)((double)raw[token] - (double)rmax - rlog);
        o.sampled_logprob = 0.f;
        if (v2 && (d.flags & kFlagWantLogprob)) {
            // (a one-token nucleus gives every other token, a forced one included, probability zero)
            o.sampled_logprob = single && token != drawn ? -INFINITY : (float)log(exp(((double)l[token] - (double)tmax) * inv_t) / kept);
        }
        o.n_top = n_top;
        outs[row] = o;
    }
}


// ---- greedy rows without logit edits (v2, top_k == 1): the token is the arg-max of the raw row and the only statistics
// needed are the row's maximum and its double-precision sum of exponentials. One warp per row merges the chunks'
// results (a single thread walking 32 chunks took 8.7 us, a dependent chain of loads and exponentials).
__global__ void greedy_finish_kernel(const float * __restrict__ raw_logits, int V, const SampleDesc * __restrict__ descs,
                                     const ChunkStat * __restrict__ stats, int n_chunks, SampleOut * __restrict__ outs,
                                     int32_t * __restrict__ top_ids, float * __restrict__ top_lps, int top_stride) {
    const int row = blockIdx.x;
    const SampleDesc d = descs[row];
    if (!(d.flags & kFlagGreedyFast)) return;
    const ChunkStat * st = stats + (size_t)row * n_chunks;
    const int lane = threadIdx.x;
    float rmax = -INFINITY;
    int32_t token = 0x7fffffff;
    for (int c = lane; c < n_chunks; c += 32)
        if (st[c].max > rmax || (st[c].max == rmax && st[c].arg < token)) { rmax = st[c].max; token = st[c].arg; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, rmax, o);
        const int32_t ot = __shfl_xor_sync(0xffffffffu, token, o);
        if (om > rmax || (om == rmax && ot < token)) { rmax = om; token = ot; }
    }
    double total = 0.0;
    for (int c = lane; c < n_chunks; c += 32) total += st[c].sum * exp((double)st[c].max - (double)rmax);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane != 0) return;
    const double rlog = log(total);
    if (token < 0 || token >= V) token = 0;      // a row of NaNs has no arg-max: stay inside the row
    const float * raw = raw_logits + (size_t)row * V;
    const double inv_t = 1.0 / (double)d.temperature;
    // the one-token nucleus: its post-transformation logprob is log(exp(0 / T) / 1)
    const float self_lp = (float)log(exp(((double)raw[token] - (double)rmax) * inv_t) / 1.0);
    const uint32_t n_top = min(d.n_top, (uint32_t)min(top_stride, V));
    int32_t next_id = 0;
    for (uint32_t j = 0; j < n_top; ++j) {
        if (j == 0) {
            top_ids[(size_t)row * top_stride] = token;
            top_lps[(size_t)row * top_stride] = self_lp;
        } else {
            // every other token was truncated away: ids in ascending order, probability zero
            if (next_id == token) ++next_id;
            top_ids[(size_t)row * top_stride + j] = next_id++;
            top_lps[(size_t)row * top_stride + j] = (float)log(exp(-INFINITY * inv_t) / 1.0);
        }
    }
    SampleOut o;
    o.token = token;
    o.logprob = (float)((double)raw[token] - (double)rmax - rlog);
    o.sampled_logprob = (d.flags & kFlagWantLogprob) ? self_lp : 0.f;
    o.n_top = n_top;
    outs[row] = o;
}

} // namespace

size_t sample_scratch_bytes(int n_vocab, int n_rows, bool candidates) {
    const size_t chunks = (size_t)n_rows * ((n_vocab + kChunk - 1) / kChunk);
    return chunks * (sizeof(ChunkStat) + (candidates ? kChunkCands * sizeof(Cand) : 0));
}

void launch_sample(const float * raw_logits, float * work_logits, int n_vocab, int n_rows, const SampleDesc * desc, const LogitEdit * edits,
                   const uint32_t * masks, SampleOut * out, int32_t * top_ids, float * top_logprobs, int top_stride, int n_greedy_fast, int n_chunked,
                   void * scratch, cudaStream_t stream) {
    if (n_rows <= 0) return;
    const int n_chunks = (n_vocab + kChunk - 1) / kChunk;
    ChunkStat * stats = static_cast<ChunkStat *>(scratch);
    Cand * cands = reinterpret_cast<Cand *>(stats + (size_t)n_rows * n_chunks);
    if (n_chunked > 0)
        sample_chunk_kernel<true><<<dim3(n_chunks, n_rows), kChunkThreads, 0, stream>>>(raw_logits, n_vocab, desc, edits, stats, cands, n_chunks, top_stride);
    else if (n_greedy_fast > 0)
        sample_chunk_kernel<false><<<dim3(n_chunks, n_rows), kChunkThreads, 0, stream>>>(raw_logits, n_vocab, desc, edits, stats, cands, n_chunks, top_stride);
    if (n_greedy_fast < n_rows) {
        static PerDeviceOnce configured;   // function attributes are per device
        if (configured.first()) cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RowShared));
        sample_kernel<<<n_rows, kThreads, n_chunked ? sizeof(RowShared) : 0, stream>>>(raw_logits, work_logits, n_vocab, desc, edits, masks, stats, cands,
                                                                                       n_chunks, out, top_ids, top_logprobs, top_stride);
    }
    if (n_greedy_fast > 0)
        greedy_finish_kernel<<<n_rows, 32, 0, stream>>>(raw_logits, n_vocab, desc, stats, n_chunks, out, top_ids, top_logprobs, top_stride);
}

} // namespace rb200
