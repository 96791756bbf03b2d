// Fused PAM Adam update.
//
// The reference (epfml/pam submodules/fairseq/fairseq/optim/adam.py:226-252) updates every parameter
// tensor with about a dozen elementwise launches plus host-to-device copies of each scalar:
//     m  = pam(m, b1) + pam(g, 1-b1)
//     v  = pam(v, b2);  v += pam(pam(g, g), 1-b2)
//     den = pow(v, 0.5) + eps              pow(a, .5) = (a == 0) ? 0 : exp2_op(pam(log2_op(a), .5))
//     p -= pam(p, wd*lr)                   (only when weight decay is on)
//     p -= pam(pad(m, den), step_size)
// with ordinary fp32 adds/subtractions between the PAM primitives.  Here the whole rule is one pass
// per element (read p, g, m, v; write p, m, v: 28 bytes per parameter, the algorithmic minimum)
// and one launch covers a table of tensors.  Each primitive is evaluated by the same scalar
// function as the elementwise kernels and every intermediate is rounded to fp32 exactly where the
// reference materialises a tensor, so p, m and v come out bit-identical to the reference's.
#include "common.cuh"
#include "pam_scalar.cuh"

namespace pamk {
namespace {

constexpr int kTensorsPerLaunch = 256;     // (an 11 KB kernel argument: within the 32 KB that sm_70 and later take)
constexpr int kThreads = 256;
constexpr int kPerBlock = kThreads * 4;

struct AdamTable {
    float* p[kTensorsPerLaunch];
    const float* g[kTensorsPerLaunch];
    float* m[kTensorsPerLaunch];
    float* v[kTensorsPerLaunch];
    int64_t n[kTensorsPerLaunch];
    // blocks [first[k], first[k + 1]) of the launch's one-dimensional grid belong to tensor k, so that a
    // table that mixes an embedding matrix with bias vectors launches no block without work
    unsigned first[kTensorsPerLaunch + 1];
    int used;
};

struct AdamScalars {
    float b1, one_minus_b1, b2, one_minus_b2, eps, decay, step_size;
    int32_t off;
    int plain;                                     // the scalars allow adam_plain (see there)
};

__device__ __forceinline__ void adam_one(float& p, float g, float& m, float& v, const AdamScalars& s, float lb2) {
    const float m1 = fadd(mul(m, s.b1, s.off), mul(g, s.one_minus_b1, s.off));
    const float v1 = fadd(mul(v, s.b2, s.off), mul(mul(g, g, s.off), s.one_minus_b2, s.off));
    const float root = v1 == 0.0f ? 0.0f
                                  : exp_base(mul(log_base(v1, lb2, s.off), 0.5f, s.off), lb2, s.off);
    const float den = fadd(root, s.eps);
    float q = p;
    if (s.decay != 0.0f) q = fadd(q, -mul(q, s.decay, s.off));
    q = fadd(q, -mul(div(m1, den, s.off), s.step_size, s.off));
    p = q;
    m = m1;
    v = v1;
}

// True if the magnitude's exponent field lies in [LO, HI).
template <uint32_t LO, uint32_t HI>
__device__ __forceinline__ bool field_in(int32_t bits) {
    const uint32_t b = (uint32_t)bits;
    return b + b - 2u * (LO << 23) < 2u * ((HI - LO) << 23);
}

// Whether the rule without its range rules (below) may be tried on these.
__device__ __forceinline__ bool ordinary(float g, float m, float v) {
    return field_in<66, 188>(f2i(g)) && field_in<27, 227>(f2i(m)) && field_in<27, 227>(f2i(v));
}

// The rule without its range rules, for values of ordinary magnitude; false (and nothing changed) where one of
// them might apply after all.  A primitive is one integer add: a product of factors in [2^-61, 2^61), or of one in
// [2^-100, 2^100) and a scalar in [2^-20, 2^20], passes the range rule, and so does such a quotient.  floor(log2f(x))
// is the exponent of x unless the mantissa lies so close to either end that log2f might round across
// the power of two (it is off by a few ulp, at most 2^-15 for exponents up to 128; the ends taken are 2^-11 wide): there it is
// called.  (Sent to the full rule instead, the one in a hundred values of a run with steady gradients that lies there made a third of the
// warps pay for both: 6+6 transformer 287 us after 3000 steps.)
__device__ __forceinline__ bool adam_plain(float& p, float g, float& m, float& v, const AdamScalars& s) {
    const int32_t gb = f2i(g), mb = f2i(m), vb = f2i(v), bias = kBias - s.off;
    const int32_t gg = isub(iadd(gb, gb), bias);
    const float m1 = fadd(i2f(iadd(mb, isub(f2i(s.b1), bias))), i2f(iadd(gb, isub(f2i(s.one_minus_b1), bias))));
    const float v1 = fadd(i2f(iadd(vb, isub(f2i(s.b2), bias))), i2f(iadd(gg, isub(f2i(s.one_minus_b2), bias))));
    const int32_t v1b = f2i(v1), mant = v1b & kMant;
    float x = fadd((float)((v1b >> 23) - 127), fadd(i2f(mant | kBias), -1.0f));              // log2(v1)
    if ((uint32_t)(mant - 0x1000) >= 0x7fe000u) {                                             // (log2's own form, see pam_scalar.cuh)
        const float e = floorf(log2f(v1));
        const int32_t ei = (int32_t)e;
        x = fadd(e, fmul(fadd(v1, -i2f((ei + 127) << 23)), i2f((127 - ei) << 23)));
    }
    // div by log2f(2) = 1, the product with 0.5, the product with log2f(2): one shift of the pattern
    const float h = i2f(iadd(f2i(x), s.off - 0x00800000));
    const float fl = floorf(h);
    const float root = fmul(fadd(1.0f, fadd(h, -fl)), i2f(((int32_t)fl + 127) << 23));
    const float den = fadd(root, s.eps);
    const int32_t d = iadd(isub(f2i(m1), f2i(den)), bias);
    // (v1 is positive: its field is read without the sign's bit; log2(v1) near 0 would be flushed)
    const bool ok = field_in<27, 227>(gg) && (uint32_t)(v1b - (27 << 23)) < (uint32_t)(200 << 23) &&
                    fabsf(x) > 0x1p-20f &&
                    field_in<66, 188>(f2i(m1)) && field_in<66, 188>(f2i(den)) && field_in<66, 188>(d);
    if (!ok) return false;
    if (s.decay != 0.0f) p = fadd(p, -mul(p, s.decay, s.off));
    p = fadd(p, -i2f(iadd(d, isub(f2i(s.step_size), bias))));
    m = m1;
    v = v1;
    return true;
}

// One element of each thread in `mask`, by one rule for all of them; the few whose values in between turn out not to be
// ordinary take the full rule after the short one.
__device__ __forceinline__ void adam_any(float& p, float g, float& m, float& v, const AdamScalars& s, float lb2, unsigned mask) {
    bool done = s.plain && __all_sync(mask, ordinary(g, m, v));
    if (done) done = adam_plain(p, g, m, v, s);
    if (!done) adam_one(p, g, m, v, s, lb2);
}

__device__ __forceinline__ void four_elements(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                                              const AdamScalars& s, float lb2, unsigned mask) {
    float4 p4 = *reinterpret_cast<const float4*>(p);
    const float4 g4 = __ldg(reinterpret_cast<const float4*>(g));
    float4 m4 = *reinterpret_cast<const float4*>(m);
    float4 v4 = *reinterpret_cast<const float4*>(v);
    adam_any(p4.x, g4.x, m4.x, v4.x, s, lb2, mask);
    adam_any(p4.y, g4.y, m4.y, v4.y, s, lb2, mask);
    adam_any(p4.z, g4.z, m4.z, v4.z, s, lb2, mask);
    adam_any(p4.w, g4.w, m4.w, v4.w, s, lb2, mask);
    *reinterpret_cast<float4*>(p) = p4;
    *reinterpret_cast<float4*>(m) = m4;
    *reinterpret_cast<float4*>(v) = v4;
}

// Four elements per thread, in at most 48 registers for five CTAs per SM: bound by DRAM with the short rule (the 254 tensors of a 6+6 transformer,
// 42 million parameters, 189 us; one tensor of 2^25 145), by its instructions with the full one, five or six per primitive and more
// for the division and log2f that only classify (2^25 elements with 30 % zeros among the gradients 210 us).  Eight elements per
// thread took 198, 152 and 257 us, and 6.8 us instead of 4.1 for 30000 elements with zeros: twice the code, fewer warps.
// The 32 elements that a warp works on at a time take one of the two together, by a vote on the inputs: where each
// thread chose for itself, zeros among the gradients (rows of an embedding that no token met, units behind
// a ReLU) made the warp run both (2^25 elements, one zero in ten: 365 us, with the vote 201 to 207).
__global__ void __launch_bounds__(kThreads, 5) adam_kernel(const AdamTable t, const AdamScalars s) {
    int which = 0, hi = t.used;                    // largest k with first[k] <= blockIdx.x (the same for the whole CTA)
    while (hi - which > 1) {
        const int mid = (which + hi) >> 1;
        if (blockIdx.x >= t.first[mid]) which = mid; else hi = mid;
    }
    const int64_t n = t.n[which];
    const int64_t base = (int64_t)(blockIdx.x - t.first[which]) * kPerBlock;
    if (base >= n) return;
    float* __restrict__ p = t.p[which];
    const float* __restrict__ g = t.g[which];
    float* __restrict__ m = t.m[which];
    float* __restrict__ v = t.v[which];
    const float lb2 = log2f(2.0f);
    const bool vec = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) |
                       reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 15u) == 0;
    const int64_t i = base + threadIdx.x * 4;
    // (whole blocks of aligned tensors: no look at the tensor's end)
    if (vec && base + kPerBlock <= n) {
        four_elements(p + i, g + i, m + i, v + i, s, lb2, 0xffffffffu);
        return;
    }
    const bool four = vec && i + 3 < n;
    const unsigned fours = __ballot_sync(0xffffffffu, four);          // (every thread of the CTA is here)
    if (four) {
        four_elements(p + i, g + i, m + i, v + i, s, lb2, fours);
    } else {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            const bool on = i + c < n;
            const unsigned ons = __ballot_sync(~fours, on);
            if (on) {
                float pp = p[i + c], mm = m[i + c], vv = v[i + c];
                const float gg = g[i + c];
                adam_any(pp, gg, mm, vv, s, lb2, ons);
                p[i + c] = pp;
                m[i + c] = mm;
                v[i + c] = vv;
            }
        }
    }
}

}  // namespace
}  // namespace pamk

using namespace pamk;

extern "C" {

int pamk_adam_step(float* const* p, const float* const* g, float* const* m, float* const* v,
                   const int64_t* n, int count,
                   float beta1, float one_minus_beta1, float beta2, float one_minus_beta2,
                   float eps, float decay, float step_size, float offset, void* stream) {
    if (count < 0) return PAMK_ERR_ARG;
    if (count == 0) return PAMK_OK;
    if (!p || !g || !m || !v || !n) return PAMK_ERR_ARG;
    AdamScalars s{beta1, one_minus_beta1, beta2, one_minus_beta2, eps, decay, step_size, offset_bits(offset), 1};
    for (float c : {beta1, one_minus_beta1, beta2, one_minus_beta2, step_size})
        if (!(c >= 0x1p-20f && c <= 0x1p20f)) s.plain = 0;
    if (s.off < -0x00200000 || s.off > 0x00200000) s.plain = 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int k = 0; k < count;) {
        AdamTable t{};
        int used = 0;
        int64_t blocks = 0;
        for (; k < count && used < kTensorsPerLaunch; ++k) {     // k carries on where the last table ended
            if (n[k] < 0) return PAMK_ERR_ARG;
            if (n[k] == 0) continue;
            if (!p[k] || !g[k] || !m[k] || !v[k]) return PAMK_ERR_ARG;
            const int64_t mine = (n[k] + kPerBlock - 1) / kPerBlock;
            if (blocks + mine > 0x7fffffff) {                    // this tensor starts the next table
                if (used == 0) return PAMK_ERR_SIZE;
                break;
            }
            t.p[used] = p[k]; t.g[used] = g[k]; t.m[used] = m[k]; t.v[used] = v[k]; t.n[used] = n[k];
            t.first[used] = (unsigned)blocks;
            blocks += mine;
            ++used;
        }
        if (used == 0) continue;
        t.first[used] = (unsigned)blocks;
        t.used = used;
        adam_kernel<<<(unsigned)blocks, kThreads, 0, st>>>(t, s);
        const int rc = check_launch();
        if (rc != PAMK_OK) return rc;
    }
    return PAMK_OK;
}

}
