// Fused PAM softmax and logsumexp over the last dimension, forward and backward.
//
// The reference builds both from primitives (epfml/pam pam/pam_ops.py:305-342): x*log2(e) by PAM,
// a shift by floor(max) of the WHOLE tensor, the piecewise affine exp2, an ordinary row sum and a
// PAM division (softmax) or log2 and a PAM division (logsumexp) — about ten launches each way.
// Here: one kernel finds the whole-tensor maximum of the scaled input (per-CTA maxima in scratch),
// and one row kernel does the rest with the row held in registers; every primitive goes through
// the same scalar functions as the elementwise kernels and rounds where the reference rounds.
// Traffic: 4 B/element for the maximum pass, then 8 B/element forward and 12 B/element backward.
//
// A row is owned by one warp (up to 1024 columns) or by a CTA of eight warps (up to 12288 columns,
// e.g. a 10000-word vocabulary).  -inf inputs (attention masks) get probability 0 as in the
// reference; NaN or +inf anywhere makes the shift, and with it every output, NaN as there.
#include <type_traits>

#include "common.cuh"
#include "pam_scalar.cuh"

namespace pamk {
namespace {

constexpr float kLog2e = 1.44269504088896340736f;   // float(math.log2(math.e)), pam_ops.py:309
constexpr float kLn2 = 0.693147180559945309417f;    // float(math.log(2.0)), cuda_bindings.py:232

// scaled input of one element: -inf stays -inf (the reference masks it back after the PAM)
__device__ __forceinline__ float scaled_of(float x, int32_t off) {
    return x == -INFINITY ? -INFINITY : mul(x, kLog2e, off);
}

// ---- whole-tensor maximum ------------------------------------------------------------------------
// NaN is sticky, as in torch.max.  One float per CTA is written to `partials`.
__device__ __forceinline__ float nan_max(float a, float b) { return (a != a || b != b) ? quiet_nan() : fmaxf(a, b); }

__global__ void __launch_bounds__(256) scaled_max_kernel(const float* __restrict__ x, int64_t n, int32_t off,
                                                         float* __restrict__ partials) {
    __shared__ float red[8];
    float m = -INFINITY;
    const int64_t stride = (int64_t)gridDim.x * 256;
    const bool vec = aligned16(x);
    if (vec) {
        const int64_t n4 = n >> 2;
        for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n4; i += stride) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(x) + i);
            m = nan_max(m, nan_max(nan_max(scaled_of(v.x, off), scaled_of(v.y, off)),
                                   nan_max(scaled_of(v.z, off), scaled_of(v.w, off))));
        }
        for (int64_t i = (n4 << 2) + (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += stride)
            m = nan_max(m, scaled_of(__ldg(x + i), off));
    } else {
        for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += stride)
            m = nan_max(m, scaled_of(__ldg(x + i), off));
    }
    // (not earlier: CTAs of the row pass would gather on the SMs that have room first, and keep their rows there)
    next_may_start();
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, d));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) m = nan_max(m, red[k]);
        partials[blockIdx.x] = m;
    }
}

// shift = floor(max over the per-CTA maxima), by all threads of the CTA: a warp alone would wait for 37 loads, one after the other
template <int THREADS>
__device__ __forceinline__ float load_shift(const float* partials, int count, float* scratch) {
    after_previous();
    float m = -INFINITY;
#pragma unroll 5
    for (int k = threadIdx.x; k < count; k += THREADS) m = nan_max(m, __ldcg(partials + k));
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, d));
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
    __syncthreads();
    m = scratch[0];
#pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) m = nan_max(m, scratch[w]);
    __syncthreads();                                          // (the sums of a row use the same words)
    return floorf(m);
}

// ---- values far inside the range rules' bounds ---------------------------------------------------
__host__ __device__ constexpr uint32_t exponent_bits(int e) { return (uint32_t)(127 + e) << 23; }
constexpr uint32_t kPlainLo = exponent_bits(-60), kPlainHi = exponent_bits(60), kPlainExp = exponent_bits(6);
constexpr uint32_t kNormalExp = 0x42fc0000u;      // 126: powers of two to less than this are normal numbers
// Below 2 * (hi - lo) where |x| lies in [lo, hi); what lies below wraps around.
__device__ __forceinline__ uint32_t above(float x, uint32_t lo) { return 2u * (uint32_t)f2i(x) - 2u * lo; }
constexpr int kMostE = 20;          // exponents of the exponentials that the short backward form takes
__device__ __forceinline__ int exponent_of(uint32_t magnitude) { return (int)(magnitude >> 23) - 127; }

// ---- rows in registers ---------------------------------------------------------------------------
struct RowArgs {
    const float* x;
    const float* g;          // backward: incoming gradient ([rows, len] softmax, [rows] logsumexp, one value for the losses)
    float* out;              // forward result or dx
    const float* partials;
    int partial_count;
    int64_t rows;
    int len;
    int32_t off;
    // loss kernels only
    const long long* target; // [rows] class index of every row
    const float* weight;     // optional per-class weights (cross-entropy gradient)
    long long ignore;        // rows whose target equals this contribute nothing (when has_ignore)
    int has_ignore;
    float c0, c1, c2;        // cross-entropy gradient: hot / cold target probability, row count (0 = no mean)
    float* aux;              // softmax forward: optional second output, the exponentials e (-0.0f where the
                             // input was -inf) for kSoftmaxBwdSaved, which takes them as x
    int post;                // softmax backward: multiply dx by post_scale (PAM product) before it is stored,
    float post_scale;        // the gradient of a PAM scaling of the scores by a constant (approx_bwd form)
};

// Thread t of a group of WARPS*32 threads holds NCH chunks of VEC consecutive columns: chunk q
// starts at column (q * WARPS*32 + t) * VEC.
template <int VEC, int NCH, int WARPS>
struct Row {
    float v[NCH * VEC];
    __device__ __forceinline__ static int col(int i, int t) { return ((i / VEC) * WARPS * 32 + t) * VEC + (i % VEC); }
    __device__ __forceinline__ void load(const float* p, int len, int t, float fill) {
#pragma unroll
        for (int q = 0; q < NCH; ++q) {
            const int c = (q * WARPS * 32 + t) * VEC;
            if (VEC == 4) {
                if (c < len) {
                    const float4 w = __ldg(reinterpret_cast<const float4*>(p + c));
                    v[q * 4] = w.x; v[q * 4 + 1] = w.y; v[q * 4 + 2] = w.z; v[q * 4 + 3] = w.w;
                } else {
                    v[q * 4] = v[q * 4 + 1] = v[q * 4 + 2] = v[q * 4 + 3] = fill;
                }
            } else {
                v[q] = c < len ? __ldg(p + c) : fill;
            }
        }
    }
    __device__ __forceinline__ void store(float* p, int len, int t) const {
#pragma unroll
        for (int q = 0; q < NCH; ++q) {
            const int c = (q * WARPS * 32 + t) * VEC;
            if (c < len) {
                if (VEC == 4) *reinterpret_cast<float4*>(p + c) = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
                else p[c] = v[q];
            }
        }
    }
};

// Sum over the group: per-thread running sum (done by the caller), butterfly over the lanes, then
// (WARPS > 1) the warp sums in warp order through shared memory.
template <int WARPS>
__device__ __forceinline__ float group_sum(float s, float* scratch) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s = fadd(s, __shfl_xor_sync(0xffffffffu, s, d));
    if (WARPS == 1) return s;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = s;
    __syncthreads();
    float t = scratch[0];
#pragma unroll
    for (int k = 1; k < WARPS; ++k) t = fadd(t, scratch[k]);
    return t;
}

// kLossFwd / kLossBwd: label-smoothed negative log-likelihood straight from the logits (log-softmax,
// gather and row sum of fairseq's label_smoothed_nll_loss fused into the logsumexp row pass).
// kCeBwd: the gradient of pam_opt.cross_entropy (softmax - target distribution, PAM-scaled).
// kSoftmaxBwdSaved: the approximate softmax backward from the exponentials the forward pass saved
// (RowArgs::aux) instead of the input: no maximum pass and no exp2 chain.
enum Op { kSoftmaxFwd, kSoftmaxBwd, kLseFwd, kLseBwd, kLossFwd, kLossBwd, kCeBwd, kSoftmaxBwdSaved };

template <int OP, bool APPROX, int VEC, int NCH, int WARPS>
// (the backward pass from the saved exponentials on the widest one-warp layouts: capped at 128 registers for
// four CTAs per SM instead of three at 146, measured 12 % faster; a cap of 96 registers spills)
__global__ void __launch_bounds__(WARPS == 1 ? 128 : WARPS * 32, (OP == kSoftmaxBwdSaved && WARPS == 1 && VEC * NCH >= 24) ? 4 : 0)
row_kernel(const RowArgs a) {
    __shared__ float scratch[8];
    constexpr int kRowsPerCta = WARPS == 1 ? 4 : 1;
    const int t = WARPS == 1 ? (threadIdx.x & 31) : threadIdx.x;
    const int sub = WARPS == 1 ? (threadIdx.x >> 5) : 0;
    using R = Row<VEC, NCH, WARPS>;
    // Short rows: the next row is on its way to registers while this one is worked on (a row is one chain of loads, two sums over the warp
    // and a divisor, and 32 warps per SM alone leave half of the issue slots empty).
    constexpr bool kAhead = WARPS == 1 && NCH * VEC <= 8 && (OP == kSoftmaxFwd || OP == kSoftmaxBwdSaved);
    const int64_t step = (int64_t)gridDim.x * kRowsPerCta;
    R ahead, ahead_g;
    if constexpr (kAhead) {                                    // (not written by the maximum pass, which may still run)
        const int64_t row = (int64_t)blockIdx.x * kRowsPerCta + sub;
        if (row < a.rows) {
            ahead.load(a.x + row * a.len, a.len, t, OP == kSoftmaxFwd ? -INFINITY : -0.0f);
            if (OP == kSoftmaxBwdSaved) ahead_g.load(a.g + row * a.len, a.len, t, 0.0f);
        }
    }
    const float shift = OP == kSoftmaxBwdSaved ? 0.0f : load_shift<WARPS == 1 ? 128 : WARPS * 32>(a.partials, a.partial_count, scratch);
    const float lb2 = log2f(2.0f);
    const int32_t off = a.off;
    // Rows whose values lie far inside the range rules' bounds, by a look at them all, skip the rules: a product or quotient is
    // one integer add instead of six instructions, chains of them without another operation between are one.  Zeros among the gradients
    // (attention dropout, targets that do not count) have a form of their own.  Without the look -> rows that skip the rules / with 10 %
    // zeros / that never do (us, forward with the maximum pass):
    //   37824 rows of 197   forward 32.6 -> 24.0 / 31.8 / 31.8    backward 28.6 -> 16.5 / 20.2 / 26.8
    //   8192 of 512                 17.3 -> 14.9 / 16.0 / 19.3             12.6 ->  8.3 / 10.1 / 13.0
    //   4096 of 1024                19.0 -> 16.2 / 17.2 / 23.1             14.4 ->  8.7 / 10.7 / 16.1
    // What is left is memory (13.7 us backward for the first) and the sums.
    constexpr bool kPlain = WARPS == 1 && (OP == kSoftmaxFwd || OP == kSoftmaxBwdSaved);
    // (an offset beyond an eighth of an exponent, or a post scale far from one, could carry results out of those bounds)
    const bool plain_call = off > -(1 << 20) && off < (1 << 20) && lb2 == 1.0f && (!a.post || (fabsf(a.post_scale) >= 0x1p-8f && fabsf(a.post_scale) <= 0x1p8f));
    // (after a row that failed the next three go without the look: it costs a fifth of a row)
    constexpr int kWithout = 3;
    int without = plain_call ? 0 : INT32_MAX;
    // masked entries count as an input whose exponent is -1 or -2
    const int32_t by_log2e = isub(f2i(kLog2e), kBias - off);
    const float stand_in = i2f(isub(f2i(shift == 1.0f ? -1.0f : fadd(shift, -1.0f)), by_log2e));
    for (int64_t row = (int64_t)blockIdx.x * kRowsPerCta + sub; row < a.rows; row += step) {
        R x, e, g;
        if constexpr (kAhead) {
            if (OP == kSoftmaxFwd) x = ahead;
            else { e = ahead; g = ahead_g; }
            if (row + step < a.rows) {
                ahead.load(a.x + (row + step) * a.len, a.len, t, OP == kSoftmaxFwd ? -INFINITY : -0.0f);
                if (OP == kSoftmaxBwdSaved) ahead_g.load(a.g + (row + step) * a.len, a.len, t, 0.0f);
            }
        } else if constexpr (OP == kSoftmaxBwdSaved) {
            // the saved exponentials; -0.0f marks a masked entry (and the padding) and acts as +0 in every
            // step below: flushed products and quotients are +0, and x + (-0) = x
            e.load(a.x + row * a.len, a.len, t, -0.0f);
            const int64_t next = row + (int64_t)gridDim.x * kRowsPerCta;
            if (next < a.rows) {                               // (this kernel waits on its loads: 12 warps per SM)
                prefetch_row_l2(a.x + next * a.len, a.len, t, WARPS * 32);
                prefetch_row_l2(a.g + next * a.len, a.len, t, WARPS * 32);
            }
        } else {
            x.load(a.x + row * a.len, a.len, t, -INFINITY);   // padding behaves like a masked entry
        }
        // forward kernels: this group's next row towards the L2 while the current one is computed (measured
        // on 1024-long rows: forward 169 -> 156 us per 2^26 elements; the backward kernels, which hold three
        // rows in registers at 12 warps per SM, lose a little with it)
        if (!kAhead && (OP == kSoftmaxFwd || OP == kLseFwd || OP == kLossFwd)) {
            const int64_t next = row + (int64_t)gridDim.x * kRowsPerCta;
            if (next < a.rows) prefetch_row_l2(a.x + next * a.len, a.len, t, WARPS * 32);
        }
        float part = 0.0f;
        bool plain = false, near = false;                      // every value of this row is far inside the rules' bounds (see kPlain), and every quotient
        if (kPlain && OP == kSoftmaxFwd && without > 0) --without;
        else if (kPlain && OP == kSoftmaxFwd) {
            uint32_t far_x = 0u, far_y = 0u;
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i) {
                const bool masked = x.v[i] == -INFINITY;
                const float xi = masked ? stand_in : x.v[i];
                const float y = i2f(iadd(f2i(fadd(i2f(iadd(f2i(xi), by_log2e)), -shift)), off));
                far_x = max(far_x, above(xi, kPlainLo));
                far_y = max(far_y, above(y, kPlainLo));
                const float fl = floorf(y);
                const float big = fmul(fadd(1.0f, fadd(y, -fl)), i2f((int32_t)(((uint32_t)(int32_t)fl << 23) + (uint32_t)kBias)));
                e.v[i] = masked ? 0.0f : big;
                part = fadd(part, e.v[i]);                     // (padding adds +0)
            }
            plain = near = __all_sync(0xffffffffu, far_x < 2u * (kPlainHi - kPlainLo) && far_y < 2u * (kPlainExp - kPlainLo));
            if (NCH * VEC > 8 && !plain) {
                // What also passes (looked at in long rows, where the first look costs a tenth and more): zeros, whose scaled pattern is a subnormal one and vanishes beside a shift that is not zero (with a shift of
                // zero it fails as y), and exponentials down to the least normal number, whose quotients need the rule.
                far_x = 0u;
#pragma unroll
                for (int i = 0; i < NCH * VEC; ++i) far_x = max(far_x, x.v[i] == 0.0f || x.v[i] == -INFINITY ? 0u : above(x.v[i], kPlainLo));
                plain = __all_sync(0xffffffffu, far_x < 2u * (kPlainHi - kPlainLo) && far_y < 2u * (kNormalExp - kPlainLo));
            }
            if (!plain) {
                part = 0.0f;
                without = kWithout;
            }
        }
        if constexpr (OP == kSoftmaxBwdSaved) {
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i)
                if (R::col(i, t) < a.len) part = fadd(part, e.v[i]);
        } else if (!plain)
#pragma unroll
        for (int i = 0; i < NCH * VEC; ++i) {
            const bool masked = x.v[i] == -INFINITY;
            const float adj = fadd(scaled_of(x.v[i], off), -shift);
            // (forward kernels and the exact backward measured faster with the compact form, the
            // approximate backward kernels with the inlined one)
            constexpr bool kCompact = OP == kSoftmaxFwd || OP == kLseFwd || OP == kLossFwd || (OP == kSoftmaxBwd && !APPROX);
            const float big = kCompact ? exp2_compact(mul(adj, lb2, off)) : exp_base(adj, lb2, off);
            e.v[i] = (OP == kSoftmaxFwd || OP == kSoftmaxBwd || OP == kCeBwd) && masked ? 0.0f : big;
            if (R::col(i, t) < a.len) part = fadd(part, e.v[i]);
        }
        const float total = group_sum<WARPS>(part, scratch);

        if (OP == kSoftmaxFwd) {
            if (a.aux) {                                       // e for the backward pass, masked entries as -0.0f
                R keep;
#pragma unroll
                for (int i = 0; i < NCH * VEC; ++i) keep.v[i] = x.v[i] == -INFINITY ? -0.0f : e.v[i];
                keep.store(a.aux + row * a.len, a.len, t);
            }
            if (kPlain && plain && near && total > 0x1p-40f && total < 0x1p40f) {
                // (exponentials between 2^-64 and 2^64: their quotients pass)
                const int32_t sub = isub(f2i(total), kBias - off);
#pragma unroll
                for (int i = 0; i < NCH * VEC; ++i) e.v[i] = e.v[i] == 0.0f ? 0.0f : i2f(isub(f2i(e.v[i]), sub));
            } else {
                const Divisor by_total = make_divisor(total, off);
#pragma unroll
                for (int i = 0; i < NCH * VEC; ++i) e.v[i] = div_by(e.v[i], by_total);
            }
            e.store(a.out + row * a.len, a.len, t);
        } else if (OP == kCeBwd) {
            // pam/pam_opt.py:27-51: (softmax(x) - target distribution), PAM-scaled by the class weight,
            // the row count (reduction = mean) and the incoming gradient
            const Divisor by_total = make_divisor(total, off);
            const long long tgt = a.target[row];
            const bool ignored = a.has_ignore && tgt == a.ignore;
            const int hot = ignored ? 0 : (int)tgt;                      // ignored rows use class 0, then times 0
            const float wt = a.weight ? __ldg(a.weight + hot) : 0.0f;
            const Divisor by_rows = make_divisor(a.c2, off);
            const float gout = __ldg(a.g);
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i) {
                const int col = R::col(i, t);
                float d = fadd(div_by(e.v[i], by_total), -(col == hot ? a.c0 : a.c1));
                if (a.weight) d = mul(d, wt, off);
                if (a.has_ignore) d = fmul(d, ignored ? 0.0f : 1.0f);
                if (a.c2 > 0.0f) d = div_by(d, by_rows);
                e.v[i] = mul(d, gout, off);
            }
            e.store(a.out + row * a.len, a.len, t);
        } else if (OP == kLossFwd) {
            // lprobs = x - logsumexp(x); nll = -lprobs[target]; smooth = -(row sum of lprobs)
            const float lse = div(fadd(shift, log_base(total, lb2, 0)), kLog2e, off);
            const long long tgt = a.target[row];
            const bool ignored = a.has_ignore && tgt == a.ignore;
            float neg_sum = 0.0f, picked = 0.0f;
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i) {
                const int col = R::col(i, t);
                const float neg_lp = fadd(lse, -x.v[i]);                  // -(x - lse), exactly
                if (col < a.len) neg_sum = fadd(neg_sum, neg_lp);
                if (col == (int)tgt) picked = neg_lp;
            }
            const float smooth = group_sum<WARPS>(neg_sum, scratch);
            const float nll = group_sum<WARPS>(picked, scratch);          // one thread holds it, the others add +0
            if (t == 0) {
                a.out[row * 3] = lse;
                a.out[row * 3 + 1] = ignored ? 0.0f : nll;
                a.out[row * 3 + 2] = ignored ? 0.0f : smooth;
            }
        } else if (OP == kLossBwd) {
            // d lprobs = -(d smooth) - (d nll at the target); d lse = -(row sum of d lprobs); then the
            // logsumexp gradient chain, and x receives both contributions
            const long long tgt = a.target[row];
            const bool ignored = a.has_ignore && tgt == a.ignore;
            const float d_nll = __ldg(a.g), d_smooth = __ldg(a.g + 1);
            const float d_all = ignored ? 0.0f : -d_smooth, d_hot = ignored ? 0.0f : fadd(-d_nll, -d_smooth);
            float part_d = 0.0f;
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i) {
                const int col = R::col(i, t);
                if (col < a.len) part_d = fadd(part_d, col == (int)tgt ? d_hot : d_all);
            }
            const float gr = -group_sum<WARPS>(part_d, scratch);
            const float u = fadd(shift, log_base(total, lb2, 0));
            const float recip = div(1.0f, kLog2e, off);
            const float d_u = APPROX ? mul(recip, gr, off) : mul_bwd(u, recip, gr, 0);
            const float d_total = log_base_bwd(total, d_u, lb2, 0);
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i) {
                const int col = R::col(i, t);
                const float adj = fadd(scaled_of(x.v[i], off), -shift);
                const float d_adj = APPROX ? mul(mul(e.v[i], kLn2, off), d_total, off)
                                           : exp_base_bwd(adj, d_total, lb2, off);
                const float via_lse = APPROX ? mul(d_adj, kLog2e, off) : mul_bwd(x.v[i], kLog2e, d_adj, off);
                e.v[i] = fadd(col == (int)tgt ? d_hot : d_all, via_lse);
            }
            e.store(a.out + row * a.len, a.len, t);
        } else if (OP == kLseFwd) {
            // log2 of the row sum runs with offset 0 whatever the call's offset (pam_ops.py:341)
            const float res = div(fadd(shift, log_base(total, lb2, 0)), kLog2e, off);
            if (t == 0) a.out[row] = res;
        } else if (OP == kSoftmaxBwd || OP == kSoftmaxBwdSaved) {
            if (!kAhead) g.load(a.g + row * a.len, a.len, t, 0.0f);
            if (kPlain && OP == kSoftmaxBwdSaved && without > 0) --without;
            else if (kPlain && OP == kSoftmaxBwdSaved) {
                // The magnitudes of the row's exponentials and gradients: with these bounds no product or quotient below leaves the
                // pass range, so that each is a sum of patterns, and chains of them one sum.
                uint32_t least_e = ~0u, most_e = 0u, least_g = ~0u, most_g = 0u;
#pragma unroll
                for (int i = 0; i < NCH * VEC; ++i) {
                    const uint32_t be = (uint32_t)f2i(e.v[i]), bg = (uint32_t)f2i(g.v[i]) & 0x7fffffffu;
                    const bool masked = e.v[i] == 0.0f;         // (an entry that counts for nothing, like the padding; an exponential that underflowed)
                    least_e = min(least_e, masked ? ~0u : be); most_e = max(most_e, masked ? 0u : be);
                    least_g = min(least_g, masked ? ~0u : bg); most_g = max(most_g, bg);       // (a masked entry's inf or NaN counts)
                }
                least_e = __reduce_min_sync(0xffffffffu, least_e); most_e = __reduce_max_sync(0xffffffffu, most_e);
                least_g = __reduce_min_sync(0xffffffffu, least_g); most_g = __reduce_max_sync(0xffffffffu, most_g);
                const bool zeros = least_g == 0u;
                if (zeros) {                                    // the least of the others
                    least_g = ~0u;
#pragma unroll
                    for (int i = 0; i < NCH * VEC; ++i) {
                        const uint32_t bg = (uint32_t)f2i(g.v[i]) & 0x7fffffffu;
                        least_g = min(least_g, e.v[i] == 0.0f || bg == 0u ? ~0u : bg);
                    }
                    least_g = __reduce_min_sync(0xffffffffu, least_g);
                }
                const int e0 = exponent_of(least_e), e1 = exponent_of(most_e), g0 = exponent_of(least_g), g1 = exponent_of(most_g);
                const int t0 = exponent_of((uint32_t)f2i(total));          // (a negative total has a huge one)
                // the exponents of e / total, e / total / total, their product with g, and g / total, with one to spare for each step;
                // e * (g / total + d_total) is looked at below, by a sum of patterns that a second factor of zero (or a subnormal one) only brings
                // below kProductLo where e < 2^22 (the forward pass saves none above 4)
                const bool ok = e0 >= -60 && e1 <= kMostE && g0 >= -60 && g1 <= 60 && t0 >= -40 && t0 <= 40 &&
                                min(e0 - t0, e0 - 2 * t0) >= -100 && max(e1 - t0, e1 - 2 * t0) <= 100 && e0 - 2 * t0 + g0 >= -108 && e1 - 2 * t0 + g1 <= 108;
                // with_zeros: gradients of zero, and second factors of zero, whose products flush to +0
                auto short_form = [&](auto with_zeros) {
                    constexpr bool kZeros = decltype(with_zeros)::value;
                    const int32_t sub = isub(f2i(total), kBias - off);
                    const int32_t by_den = isub(isub(isub(0, sub), sub), kBias - off), by_recip = isub(isub(kBias, sub), kBias - off);
                    float dsum = 0.0f;
                    R d;
#pragma unroll
                    for (int i = 0; i < NCH * VEC; ++i) {
                        const bool masked = e.v[i] == 0.0f, zero = kZeros && g.v[i] == 0.0f;
                        const float dden = -i2f(iadd3(f2i(e.v[i]), f2i(g.v[i]), by_den));
                        dsum = fadd(dsum, masked || zero ? -0.0f : dden);
                        d.v[i] = zero ? 0.0f : i2f(iadd(f2i(g.v[i]), by_recip));
                    }
                    const float d_total = group_sum<WARPS>(dsum, scratch);
                    // ((e * ln 2) * d) * log2 e (* post): the constants of the four products in one
                    const int32_t by_one = kBias - off, by_all = iadd(isub(isub(isub(iadd(f2i(kLn2), f2i(kLog2e)), by_one), by_one), by_one), a.post ? isub(f2i(a.post_scale), by_one) : 0);
                    constexpr uint32_t kProductLo = 2u * (uint32_t)kBias - (104u << 23), kProductSpan = 204u << 23;   // e * d in [2^-104, 2^100)
                    static_assert(exponent_bits(kMostE + 1) + (1u << 23) < kProductLo, "no e and subnormal d reach the bound");
                    uint32_t far = 0u;
#pragma unroll
                    for (int i = 0; i < NCH * VEC; ++i) {
                        d.v[i] = fadd(d.v[i], d_total);
                        const bool flushed = e.v[i] == 0.0f || (kZeros && d.v[i] == 0.0f);
                        const uint32_t sum = (uint32_t)f2i(e.v[i]) + ((uint32_t)f2i(d.v[i]) & 0x7fffffffu);
                        far = max(far, flushed ? 0u : sum - kProductLo);
                    }
                    if (!__all_sync(0xffffffffu, far < kProductSpan)) return false;
#pragma unroll
                    for (int i = 0; i < NCH * VEC; ++i) {
                        const bool flushed = e.v[i] == 0.0f || (kZeros && d.v[i] == 0.0f);
                        d.v[i] = flushed ? 0.0f : i2f(iadd3(f2i(e.v[i]), f2i(d.v[i]), by_all));
                    }
                    d.store(a.out + row * a.len, a.len, t);
                    return true;
                };
                if (ok && (zeros ? short_form(std::true_type{}) : short_form(std::false_type{}))) continue;      // (the same for a warp)
                without = kWithout;
            }
            const Divisor by_total = make_divisor(total, off);
            const float recip = div_by(1.0f, by_total);
            float dsum = 0.0f;
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i) {
                const float dden = APPROX ? -mul(div_by(div_by(e.v[i], by_total), by_total), g.v[i], off)
                                          : div_bwd(e.v[i], total, g.v[i], off);
                if (R::col(i, t) < a.len) dsum = fadd(dsum, dden);
                g.v[i] = APPROX ? mul(recip, g.v[i], off) : mul_bwd(e.v[i], recip, g.v[i], 0);
            }
            const float d_total = group_sum<WARPS>(dsum, scratch);
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i) {
                const bool masked = OP == kSoftmaxBwdSaved ? f2i(e.v[i]) == (int32_t)0x80000000 : x.v[i] == -INFINITY;
                const float adj = OP == kSoftmaxBwdSaved ? 0.0f : fadd(scaled_of(x.v[i], off), -shift);
                const float d_big = masked ? 0.0f : fadd(g.v[i], d_total);
                const float d_adj = APPROX ? mul(mul(e.v[i], kLn2, off), d_big, off)
                                           : exp_base_bwd(adj, d_big, lb2, off);
                const float d_s = masked ? 0.0f : d_adj;
                g.v[i] = APPROX ? mul(d_s, kLog2e, off) : mul_bwd(x.v[i], kLog2e, d_s, off);
                if (a.post) g.v[i] = mul(g.v[i], a.post_scale, off);
            }
            g.store(a.out + row * a.len, a.len, t);
        } else {
            const float gr = __ldg(a.g + row);
            const float u = fadd(shift, log_base(total, lb2, 0));
            const float recip = div(1.0f, kLog2e, off);
            const float d_u = APPROX ? mul(recip, gr, off) : mul_bwd(u, recip, gr, 0);
            const float d_total = log_base_bwd(total, d_u, lb2, 0);
#pragma unroll
            for (int i = 0; i < NCH * VEC; ++i) {
                const float adj = fadd(scaled_of(x.v[i], off), -shift);
                const float d_adj = APPROX ? mul(mul(e.v[i], kLn2, off), d_total, off)
                                           : exp_base_bwd(adj, d_total, lb2, off);
                e.v[i] = APPROX ? mul(d_adj, kLog2e, off) : mul_bwd(x.v[i], kLog2e, d_adj, off);
            }
            e.store(a.out + row * a.len, a.len, t);
        }
    }
}

constexpr int kMaxLen = 12288;

template <int OP, bool APPROX>
int launch_rows(const RowArgs& a, cudaStream_t st) {
    const bool vec = (a.len & 3) == 0 && aligned16(a.x) && (OP == kLseFwd || OP == kLossFwd || aligned16(a.out)) &&
                     ((OP != kSoftmaxBwd && OP != kSoftmaxBwdSaved) || aligned16(a.g)) && (a.aux == nullptr || aligned16(a.aux));
    const int64_t sms = sm_count();
    // Behind the maximum pass where there is one (2 us: 591 rows of 197 8.2 -> 6.5, 37824 26.7 -> 24.6).  Not the recomputing backward passes of
    // several rows per warp, which are long enough for an uneven start to cost more: 65536 rows of 197 91 -> 96.
    constexpr bool kForward = OP == kSoftmaxFwd || OP == kLseFwd || OP == kLossFwd;
    const bool behind = OP != kSoftmaxBwdSaved;
#define PAMK_ROWS(V, N, W)                                                                              \
    do {                                                                                                \
        const int64_t per = (W) == 1 ? 4 : 1;                                                           \
        const int64_t want = (a.rows + per - 1) / per, cap = sms * ((W) == 1 ? 8 : 4);                  \
        const dim3 grid((unsigned)(want < cap ? want : cap));                                            \
        if (behind && (kForward || want <= cap)) return launch_behind(row_kernel<OP, APPROX, V, N, W>, grid, (W) == 1 ? 128 : (W) * 32, st, a); \
        row_kernel<OP, APPROX, V, N, W><<<grid, (W) == 1 ? 128 : (W) * 32, 0, st>>>(a);                  \
        return check_launch();                                                                          \
    } while (0)
    // (the number of chunks per thread only sets how many register slots a row may fill: a shorter layout
    // for a shorter row leaves fewer idle slots and changes no sum, every thread adds its columns in the
    // same order either way)
    if (vec) {
        if (a.len <= 128) PAMK_ROWS(4, 1, 1);
        if (a.len <= 256) PAMK_ROWS(4, 2, 1);
        if (a.len <= 512) PAMK_ROWS(4, 4, 1);
        if (a.len <= 768) PAMK_ROWS(4, 6, 1);
        if (a.len <= 1024) PAMK_ROWS(4, 8, 1);
        if (a.len <= 4096) PAMK_ROWS(4, 4, 8);
        if (a.len <= kMaxLen) PAMK_ROWS(4, 12, 8);
    } else {
        if (a.len <= 64) PAMK_ROWS(1, 2, 1);
        if (a.len <= 128) PAMK_ROWS(1, 4, 1);
        if (a.len <= 224) PAMK_ROWS(1, 7, 1);
        if (a.len <= 256) PAMK_ROWS(1, 8, 1);
        if (a.len <= 1024) PAMK_ROWS(1, 32, 1);
        if (a.len <= kMaxLen) PAMK_ROWS(1, 48, 8);
    }
#undef PAMK_ROWS
    return PAMK_ERR_SIZE;
}

int max_grid(int64_t n) {
    const int64_t want = (n + 4 * 256 - 1) / (4 * 256);
    const int64_t cap = (int64_t)sm_count() * 8;
    return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

int run_rows(int op, bool approx, RowArgs a, int64_t len, float offset, void* workspace, size_t workspace_bytes, void* stream) {
    const int64_t rows = a.rows;
    if (rows < 0 || len <= 0) return PAMK_ERR_ARG;
    if (len > kMaxLen) return PAMK_ERR_SIZE;
    if (rows == 0) return PAMK_OK;
    if (!a.x || !a.out || ((op == kSoftmaxBwd || op == kSoftmaxBwdSaved || op == kLseBwd || op == kCeBwd || op == kLossBwd) && !a.g))
        return PAMK_ERR_ARG;
    if ((op == kLossFwd || op == kLossBwd || op == kCeBwd) && !a.target) return PAMK_ERR_ARG;
    const int64_t n = rows * len;
    const int grid = max_grid(n);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int32_t off = offset_bits(offset);
    if (op == kSoftmaxBwdSaved) {                     // works from the saved exponentials: no maximum pass
        a.len = (int)len;
        a.off = off;
        return launch_rows<kSoftmaxBwdSaved, true>(a, st);
    }
    if (!workspace || workspace_bytes < (size_t)grid * sizeof(float) || (reinterpret_cast<uintptr_t>(workspace) & 15u))
        return PAMK_ERR_WORKSPACE;
    float* partials = static_cast<float*>(workspace);
    scaled_max_kernel<<<grid, 256, 0, st>>>(a.x, n, off, partials);
    int rc = check_launch();
    if (rc != PAMK_OK) return rc;
    a.partials = partials;
    a.partial_count = grid;
    a.len = (int)len;
    a.off = off;
    switch (op) {
        case kSoftmaxFwd: return launch_rows<kSoftmaxFwd, false>(a, st);
        case kLseFwd: return launch_rows<kLseFwd, false>(a, st);
        case kLossFwd: return launch_rows<kLossFwd, false>(a, st);
        case kCeBwd: return launch_rows<kCeBwd, false>(a, st);
        case kSoftmaxBwd: return approx ? launch_rows<kSoftmaxBwd, true>(a, st) : launch_rows<kSoftmaxBwd, false>(a, st);
        case kLossBwd: return approx ? launch_rows<kLossBwd, true>(a, st) : launch_rows<kLossBwd, false>(a, st);
        default: return approx ? launch_rows<kLseBwd, true>(a, st) : launch_rows<kLseBwd, false>(a, st);
    }
}

RowArgs plain_rows(const float* x, const float* g, float* out, int64_t rows) {
    RowArgs a{};
    a.x = x; a.g = g; a.out = out; a.rows = rows;
    return a;
}

}  // namespace
}  // namespace pamk

using namespace pamk;

extern "C" {

int pamk_softmax_max_len(void) { return kMaxLen; }

size_t pamk_softmax_workspace_bytes(int64_t rows, int64_t len) {
    if (rows <= 0 || len <= 0) return 0;
    return (size_t)max_grid(rows * len) * sizeof(float);
}

int pamk_softmax_fwd(const float* x, float* y, int64_t rows, int64_t len, float offset,
                     void* workspace, size_t workspace_bytes, void* stream) {
    return run_rows(kSoftmaxFwd, false, plain_rows(x, nullptr, y, rows), len, offset, workspace, workspace_bytes, stream);
}

int pamk_softmax_bwd(const float* x, const float* dy, float* dx, int64_t rows, int64_t len, float offset,
                     int approx_bwd, void* workspace, size_t workspace_bytes, void* stream) {
    return run_rows(kSoftmaxBwd, approx_bwd != 0, plain_rows(x, dy, dx, rows), len, offset, workspace, workspace_bytes, stream);
}

int pamk_softmax_fwd_save(const float* x, float* y, float* e, int64_t rows, int64_t len, float offset,
                          void* workspace, size_t workspace_bytes, void* stream) {
    if (!e) return PAMK_ERR_ARG;
    RowArgs a = plain_rows(x, nullptr, y, rows);
    a.aux = e;
    return run_rows(kSoftmaxFwd, false, a, len, offset, workspace, workspace_bytes, stream);
}

int pamk_softmax_bwd_saved(const float* e, const float* dy, float* dx, int64_t rows, int64_t len, float offset,
                           int has_post_scale, float post_scale, void* stream) {
    RowArgs a = plain_rows(e, dy, dx, rows);
    a.post = has_post_scale != 0;
    a.post_scale = post_scale;
    return run_rows(kSoftmaxBwdSaved, true, a, len, offset, nullptr, 0, stream);
}

int pamk_softmax_bwd_scaled(const float* x, const float* dy, float* dx, int64_t rows, int64_t len, float offset,
                            int approx_bwd, float post_scale, void* workspace, size_t workspace_bytes, void* stream) {
    RowArgs a = plain_rows(x, dy, dx, rows);
    a.post = 1; a.post_scale = post_scale;
    return run_rows(kSoftmaxBwd, approx_bwd != 0, a, len, offset, workspace, workspace_bytes, stream);
}

int pamk_logsumexp_fwd(const float* x, float* y, int64_t rows, int64_t len, float offset,
                       void* workspace, size_t workspace_bytes, void* stream) {
    return run_rows(kLseFwd, false, plain_rows(x, nullptr, y, rows), len, offset, workspace, workspace_bytes, stream);
}

int pamk_logsumexp_bwd(const float* x, const float* dy, float* dx, int64_t rows, int64_t len, float offset,
                       int approx_bwd, void* workspace, size_t workspace_bytes, void* stream) {
    return run_rows(kLseBwd, approx_bwd != 0, plain_rows(x, dy, dx, rows), len, offset, workspace, workspace_bytes, stream);
}

int pamk_ls_loss_fwd(const float* logits, const long long* target, float* rows_out, int64_t rows, int64_t len,
                     int has_ignore, long long ignore_index, float offset,
                     void* workspace, size_t workspace_bytes, void* stream) {
    RowArgs a = plain_rows(logits, nullptr, rows_out, rows);
    a.target = target; a.has_ignore = has_ignore; a.ignore = ignore_index;
    return run_rows(kLossFwd, false, a, len, offset, workspace, workspace_bytes, stream);
}

int pamk_ls_loss_bwd(const float* logits, const long long* target, const float* grads, float* dlogits,
                     int64_t rows, int64_t len, int has_ignore, long long ignore_index, float offset, int approx_bwd,
                     void* workspace, size_t workspace_bytes, void* stream) {
    RowArgs a = plain_rows(logits, grads, dlogits, rows);
    a.target = target; a.has_ignore = has_ignore; a.ignore = ignore_index;
    return run_rows(kLossBwd, approx_bwd != 0, a, len, offset, workspace, workspace_bytes, stream);
}

int pamk_cross_entropy_bwd(const float* logits, const long long* target, const float* class_weight, const float* grad_out,
                           float* dlogits, int64_t rows, int64_t len, float hot_prob, float cold_prob, float mean_rows,
                           int has_ignore, long long ignore_index, float offset,
                           void* workspace, size_t workspace_bytes, void* stream) {
    RowArgs a = plain_rows(logits, grad_out, dlogits, rows);
    a.target = target; a.weight = class_weight; a.has_ignore = has_ignore; a.ignore = ignore_index;
    a.c0 = hot_prob; a.c1 = cold_prob; a.c2 = mean_rows;
    return run_rows(kCeBwd, false, a, len, offset, workspace, workspace_bytes, stream);
}

}
