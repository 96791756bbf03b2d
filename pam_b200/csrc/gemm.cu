// PAM matrix products for sm_100a.
//
//   C[z][i][j] = sum_k MUL(A[z][i][k], B[z][k][j])
//
// A PAM product is an integer add of the two fp32 bit patterns (minus the exponent bias), so the
// contraction cannot run on the tensor pipes; this is a CUDA-core kernel bounded by instruction
// issue.  The algorithmic cost per multiply-accumulate is one INT32 add and one FP32 add, and the
// kernel is organised so that the common case issues little more than those two:
//
//   * 8x8 register micro-tile per thread, 128x128 (256 threads) or 64x64 (64 threads) output
//     tile per CTA chosen per problem so that the tiles spread evenly over the 148 SMs: the
//     operand fetch is four 128-bit shared-memory loads per 64 products;
//   * operands are staged global -> registers -> shared one K-slab (16) ahead of the arithmetic
//     (double-buffered shared memory, one barrier per slab); while they pass through registers
//     the A side is pre-biased (bits - (0x3f800000 - offset)) so that the product is a single
//     add, both sides are laid out [k][row] whatever their layout in global memory (the four
//     row-/column-major combinations of the reference become two loader variants per side), and
//     every element's exponent is tested against the safe band;
//   * the reference's per-product range rule (flush below 1e-37, NaN above 1e37 or for
//     inf/NaN; epfml/pam pam/cuda_kernels.cu:24-37) is hoisted.  A slab whose elements all have their
//     exponent in a band that keeps every product in range runs the two-instruction loop.  In any other
//     slab the choice is made per k line, on the large tile per warp too: products that all pass are summed as they
//     are, products that all flush are left out, and only what is left evaluates the true product.  Either way every
//     product equals the reference's bit for bit;
//   * each output is summed by one thread, strictly in k order, from +0.0f — the same order as
//     the reference's kernel (cuda_kernels.cu:608-629), so without split-K the sums are
//     bit-identical too.
//
// Products that are large in both dimensions run on operands packed by a pass over them (gemm_packed.cuh), small ones in ranges of K
// in one launch (ranges_kernel).
// The same skeleton serves true-multiply products (standard_matmul) and the exact-gradient
// product (pam_matmul_bwd_kernel, cuda_kernels.cu:729-832).
#include <algorithm>
#include <array>
#include <type_traits>

#include "common.cuh"
#include "pam_scalar.cuh"

namespace pamk {
namespace {

enum Mode { kPam = 0, kStd = 1, kBwdL = 2, kBwdR = 3 };

// One matrix operand: element (r, k) of batch z lives at p[(z / inner)*sb + z*sb2 + r*sr + k*sk], where r
// is the non-contracted index (row of A / column of B) and `inner` (GemmParams) is the size of the inner
// batch dimension (1 for a plain batch: the heads of an attention product otherwise).  run() derives
// this form from the caller's (outer stride, inner stride): sb = outer - inner * inner_stride,
// sb2 = inner_stride; with inner = 1, sb = 0 and sb2 = the batch stride.
struct MatArg {
    const float* p;
    int64_t sb, sr, sk;
    int64_t sb2;
};

struct GemmParams {
    MatArg A, B;
    const float* D;           // exact-gradient product only: the operand the slope depends on
    int64_t sDb, sDm, sDn;
    float* C;                 // output, or [split][batch][M][N] partials when splits > 1
    int64_t ldc, sCb, sCb2;   // output row stride and batch strides (outer, inner); columns are contiguous
    int64_t sCsplit;          // distance between the partials of two K ranges
    const float* bias;        // optional [N]: added (ordinary fp32 add) to every output row after its sum
    int post;                 // multiply every finished sum by post_scale (PAM product) before it is stored
    float post_scale;
    int inner;                // size of the inner batch dimension (>= 1)
    unsigned inner_magic;     // floor(2^32 / inner) + 1 (0 when inner = 1): z / inner = umulhi(z, inner_magic)
    int M, N, K, batch;
    int splits, k_chunk;      // K is cut into `splits` ranges of k_chunk (a multiple of the slab)
    int32_t bias_sub;         // 0x3f800000 - offset_bits
    int32_t off;              // offset_bits
    int32_t one, least;       // 1 and INT32_MIN, as values that the compiler does not know (see sum_on_alu)
};

// Tile shapes.  Every thread owns an 8x8 register micro-tile unless said otherwise.
//   128x128x16, 256 threads, 2 CTAs/SM: least staging overhead, for large outputs;
//   64x64x8,     64 threads, 8 CTAs/SM: four times as many CTAs, for outputs that would leave a
//                                       large tile grid with a ragged last wave (e.g. 12608 x 192).
template <int BM_, int BN_, int BK_, int CPS_, int MT_ = 8, int MR_ = MT_>
struct Tile {
    // every thread owns an MR x MT micro-tile (8, or 4 for the tile meant for very small outputs; MR below MT leaves
    // the last row slots of every thread empty)
    static constexpr int BM = BM_, BN = BN_, BK = BK_, MT = MT_, MR = MR_, kCtasPerSm = CPS_;
    static constexpr int kRows = BM_ / MT_ * MR_;      // rows of the output that a tile covers
    static constexpr int kThreads = (BM_ / MT_) * (BN_ / MT_);
    static constexpr int TX = BN_ / MT_;
    // float4 tasks per thread when staging one operand slab
    static constexpr int kTasksA = BM_ * BK_ / 4 / kThreads, kTasksB = BN_ * BK_ / 4 / kThreads;
    // rows that one warp of the K-contiguous loader covers
    static constexpr int kRowsPerWarp = 32 / (BK_ / 4);
};
using TileLarge = Tile<128, 128, 16, 2>;
// 112x128x16: the large tile with seven rows per thread, for products of few large tiles per SM whose number then
// fits the SMs better (4096 rows x 1024: 256 tiles of 128 rows leave 40 of the 148 SMs with one tile where the others have two, 296
// tiles of 112 none; one CTA of this size already runs an SM at 95 % of what two do).  Row slot 7 of every thread is staged
// with a copy of a neighbouring row and takes no part in the sums.  4096x1024x512 174.5 -> 153.4 us, 8192x512x512 the same.
// Products that the plan cuts along K keep their ranges on it: 4096x512x512 in two ranges is 256 tiles of 128 rows on 296 slots, and
// exactly 296 of 112, 92.2 -> 84.0 us (1 % special values 187.7 -> 166.0).  (Unsplit it ran 83.5 us, but the order of the sums would
// depend on whether the operands' layout and alignment allow this tile.)
using TileLarge7 = Tile<128, 128, 16, 2, 8, 7>;
using TileSmall = Tile<64, 64, 8, 8>;
// 56x64x8: the 64x64 tile with seven rows per thread, for unsplit products whose rows fill tiles of 56 better (attention over 197 tokens:
// four tiles of 56 pad 14 % of the rows, of 64 30 %).  192 products 197x64x197 69.7 -> 57.4 us, with A contiguous along its rows 75.4 -> 59.4,
// 500 products 100x100x64 43.5 -> 40.1 (small7_better).
using TileSmall7 = Tile<64, 64, 8, 8, 8, 7>;
// 32x32x16 with a 4x4 micro-tile, 64 threads: batched products whose matrices are a fraction of a
// 64x64 tile (attention over 32 tokens) would otherwise spend three quarters of their adds on
// rows and columns that do not exist.  A launch of few such CTAs is a chain of slabs, each as long as a
// load from L2, so slabs of 16 run it in half the steps of 8
// (197x576x192: 10.8 -> 9.0 us, 3 products 197x64x197: 17.0 -> 13.9 us, 192 products 197x197x64: 80 -> 70 us).
// Slabs of 8 stay for launches that fill the SMs and whose K ends in the first half of a slab of 16, where the
// zero-filled rest would be work (192 products 197x64x197: 70 us against 78).
using TileTinyFine = Tile<32, 32, 8, 12, 4>;
using TileTiny = Tile<32, 32, 16, 12, 4>;

// Shared-memory layout of a slab: [k][row], rows of R floats padded by four.  The padding spreads
// the transposing stores of a K-contiguous operand (a warp writes kRowsPerWarp rows x BK/4
// k-groups) over the banks, and keeps every fragment address a constant offset from one base so
// that the arithmetic loops carry no address computation (an XOR swizzle measured the same speed
// with more instructions and a few spilled registers).
__host__ __device__ constexpr int row_stride(int R) { return R + 4; }

// Row of the tile that is staged in row slot `slot`: a thread's slots are ty * 4 + (0..3) and R / 2 + ty * 4 + (0..3), of
// which the last MT - MR are empty.  Identity for MR = MT.
template <class T, int R>
__host__ __device__ constexpr int slot_row(int slot) {
    constexpr int kSecond = T::MR - 4;                 // rows of a thread's second group of slots
    if (T::MR == T::MT || slot < R / 2) return slot;
    const int in = slot - R / 2;
    return R / 2 + in / 4 * kSecond + (in % 4 < kSecond ? in % 4 : kSecond - 1);
}

// ---- loaders: global -> registers ---------------------------------------------------------------
// (Plain loads: the compiler may move loads of constant memory, __ldg, in front of the wait for the kernel before, see after_previous.)
// A slab is R rows x BK k, staged as float4 "tasks"; thread t takes tasks t, t + kThreads, ...
//   KC (operand contiguous along k: row-major A, or B given as W[N,K]):
//       task id -> row id / (BK/4), k-group id % (BK/4): a warp reads kRowsPerWarp rows x 4*BK bytes;
//   otherwise (contiguous along the row index): task id -> k = id / (R/4), four rows (id % (R/4))*4:
//       a warp reads 512 contiguous bytes of one k.
// Rows beyond the matrix are clamped to the last valid row (their products land in outputs that
// are never stored); k beyond the range reads as 0.0f, which the range rule turns into +0.  This is the scalar form of the 32x32x16 tile, whose
// launches are chains of slabs: all addresses follow from k0, no slab waits for the last one's.
template <class T, int R, int NT, bool KC>
__device__ __forceinline__ void load_slab(float (&r)[NT * 4], const MatArg& m, const float* base,
                                          int row0, int rows, int k0, int k_end, int tid) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const int id = tid + t * T::kThreads;
        if (KC) {
            int row = row0 + id / (T::BK / 4);
            row = row < rows ? row : rows - 1;
            const int k = k0 + (id % (T::BK / 4)) * 4;
            const float* src = base + (int64_t)row * m.sr + k;
#pragma unroll
            for (int c = 0; c < 4; ++c) r[t * 4 + c] = k + c < k_end ? src[c] : 0.0f;
        } else {
            const int k = k0 + id / (R / 4);
            const int c0 = row0 + (id % (R / 4)) * 4;
            const bool on = k < k_end;
            const float* src = base + (int64_t)k * m.sk;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = c0 + c < rows ? c0 + c : rows - 1;
                r[t * 4 + c] = on ? src[col] : 0.0f;
            }
        }
    }
}

// The scalar form of the other tiles: one pointer per task that walks along K, and where the operand is contiguous along its rows the four
// clamped rows.  192 products 64x197x197 on 32x32x8 tiles 75.8 -> 69.6 us, 3001x1501x777 275 -> 265; on the 32x32x16 tile it is
// slower (12 products 197x64x197 14.4 -> 16.4).
template <class T, int R, int NT, bool KC>
struct ScalarWalker {
    const float* ptr[NT];
    int rows_of[KC ? 1 : NT][4];
    int64_t step;

    template <bool MAPPED>
    __device__ __forceinline__ void init(const MatArg& m, const float* base, int row0, int rows, int k_begin, int tid) {
        step = KC ? (int64_t)T::BK : (int64_t)T::BK * m.sk;
        auto row_at = [&](int slot) {
            const int row = row0 + (MAPPED ? slot_row<T, R>(slot) : slot);
            return row < rows ? row : rows - 1;
        };
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int id = tid + t * T::kThreads;
            if (KC) {
                ptr[t] = base + (int64_t)row_at(id / (T::BK / 4)) * m.sr + k_begin + (id % (T::BK / 4)) * 4;
            } else {
                ptr[t] = base + (int64_t)(k_begin + id / (R / 4)) * m.sk;
#pragma unroll
                for (int c = 0; c < 4; ++c) rows_of[KC ? 0 : t][c] = row_at((id % (R / 4)) * 4 + c);
            }
        }
    }

    __device__ __forceinline__ void load(float (&r)[NT * 4], int k0, int k_end, int tid) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int id = tid + t * T::kThreads;
            const int k = KC ? k0 + (id % (T::BK / 4)) * 4 : k0 + id / (R / 4);
#pragma unroll
            for (int c = 0; c < 4; ++c) r[t * 4 + c] = (KC ? k + c : k) < k_end ? ptr[t][KC ? c : rows_of[KC ? 0 : t][c]] : 0.0f;
            ptr[t] += step;
        }
    }
};

// Vectorised loads keep one pointer per task that walks along K, so the per-slab work is the load,
// the range predicate and one pointer increment; the row clamp and the 64-bit address arithmetic
// are done once per kernel.
template <class T, int R, int NT, bool KC>
struct SlabWalker {
    const float* ptr[NT];
    int64_t step;                                    // elements to advance per slab

    template <bool MAPPED>
    __device__ __forceinline__ void init(const MatArg& m, const float* base, int row0, int rows, int k_begin, int tid) {
        static_assert(KC || !MAPPED, "four consecutive rows have to lie in four consecutive slots");
        step = KC ? (int64_t)T::BK : (int64_t)T::BK * m.sk;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int id = tid + t * T::kThreads;
            if (KC) {
                int row = row0 + (MAPPED ? slot_row<T, R>(id / (T::BK / 4)) : id / (T::BK / 4));
                row = row < rows ? row : rows - 1;
                ptr[t] = base + (int64_t)row * m.sr + k_begin + (id % (T::BK / 4)) * 4;
            } else {
                const int c0 = row0 + (id % (R / 4)) * 4;
                ptr[t] = base + (int64_t)(k_begin + id / (R / 4)) * m.sk + (c0 < rows ? c0 : rows - 4);
            }
        }
    }

    __device__ __forceinline__ void load(float (&r)[NT * 4], int k0, int k_end, int tid) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int id = tid + t * T::kThreads;
            const int k = KC ? k0 + (id % (T::BK / 4)) * 4 : k0 + id / (R / 4);
            const float4 v = k < k_end ? *reinterpret_cast<const float4*>(ptr[t]) : make_float4(0.f, 0.f, 0.f, 0.f);
            r[t * 4] = v.x; r[t * 4 + 1] = v.y; r[t * 4 + 2] = v.z; r[t * 4 + 3] = v.w;
            ptr[t] += step;
        }
    }
};

// ---- registers -> shared, laid out [k][row] -----------------------------------------------------
template <class T, int R, int NT, bool KC>
__device__ __forceinline__ void store_slab(float* s, const float (&r)[NT * 4], int tid) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const int id = tid + t * T::kThreads;
        if (KC) {
            const int row = id / (T::BK / 4), kg = (id % (T::BK / 4)) * 4;
#pragma unroll
            for (int c = 0; c < 4; ++c) s[(kg + c) * row_stride(R) + row] = r[t * 4 + c];
        } else {
            const int k = id / (R / 4), c0 = (id % (R / 4)) * 4;
            *reinterpret_cast<float4*>(s + k * row_stride(R) + c0) = make_float4(r[t * 4], r[t * 4 + 1], r[t * 4 + 2], r[t * 4 + 3]);
        }
    }
}

// ---- which loop a slab, and each of its k lines, may run ---------------------------------------------
// Products of normal finite numbers satisfy 2^(ea+eb-254) <= |a*b| <= 2^(ea+eb-252) (ea, eb the
// biased exponents), so if both factors have their exponent field in the band [66, 187] the product
// lies in [2^-122, 2^122], inside the reference's pass range (1e-37, 1e37), and the range rule
// (cuda_kernels.cu:24-37) returns the integer sum.  The band test is one three-input add and one
// unsigned max per element: 2 * bits drops the sign, minus twice the band's lower bound makes "below"
// wrap around to huge values.
//   * A slab whose elements are all in the band runs the two-instruction loop.  Otherwise the staging threads that hold
//     out-of-band elements record for which k lines, and of what sort they are.
//   * Zeros alone, in most lines (an operand that went through a ReLU): a zero's products are left out of the sums by a
//     predicate or a weight.
//   * Anything else, large tile, where it pays (class_of): the lines with out-of-band elements are looked through once and every
//     warp takes, for each line, the cheapest loop that its own rows and columns allow (kind_of).
//   * Anything else: a line without out-of-band elements costs two instructions per product, any other evaluates the true fp32
//     product.  It can skip the overflow test when the largest
//     magnitudes of its two operand lines cannot multiply beyond 1e37 and neither holds an inf / NaN
//     (|a * b| rounded grows with |a| and |b|, so the two maxima bound every product of the line):
//     four instructions per product, "flush or add".  Only the remaining lines apply the full rule.  (On the smaller tiles a look
//     costs more than it saves: 12608x768x192 with 1 % specials 304 -> 475 us.)
constexpr uint32_t kBandLo = 66u << 23, kBandHi = 188u << 23;  // smallest magnitude in the band, smallest above it
constexpr uint32_t kBandLo2 = 2u * kBandLo, kBandHi2 = 2u * kBandHi;
constexpr uint32_t kBandSpan2 = kBandHi2 - kBandLo2;           // in band iff 2*bits - kBandLo2 < span

template <int N>
__device__ __forceinline__ uint32_t band_excess(const float (&r)[N], uint32_t vmax) {
#pragma unroll
    for (int c = 0; c < N; ++c) {
        const uint32_t b = (uint32_t)f2i(r[c]);
        vmax = max(vmax, b + b - kBandLo2);
    }
    return vmax;
}

// Position of element c of staging task `id` inside the slab: its k line.
template <class T, int R, bool KC>
__device__ __forceinline__ int slab_line(int id, int c) {
    return KC ? (id % (T::BK / 4)) * 4 + c : id / (R / 4);
}

// A slab's word: bit k for a k line that holds an out-of-band element, which operand such elements are in, and whether any is
// not zero, or above the band.
enum Word : unsigned { kInA = 1u << 16, kInB = 1u << 17, kNonZero = 1u << 18, kAbove = 1u << 19 };

// The k lines of this thread's staged elements that are out of the band; `bits` collects the magnitudes of those elements, `top` the
// largest magnitude (twice the pattern, both).  No branch per element: with one, few such elements in a slab cost
// more than many, 4096^3 with 2 % specials 1.5 %.
template <class T, int R, int NT, bool KC>
__device__ __forceinline__ unsigned dirty_lines(const float (&r)[NT * 4], int tid, uint32_t& bits, uint32_t& top) {
    unsigned lines = 0;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t b = (uint32_t)f2i(r[t * 4 + c]);
            const uint32_t m2 = b + b;
            const bool off = m2 - kBandLo2 >= kBandSpan2;
            lines |= off ? 1u << slab_line<T, R, KC>(tid + t * T::kThreads, c) : 0u;
            bits |= off ? m2 : 0u;
            top = max(top, m2);
        }
    return lines;
}

// ---- the large tile's look through a dirty slab ------------------------------------------------------------------------
// What does the range rule do to the products of an out-of-band element with its line's partners that are not above the band?
// The rounded product |a * b| grows with both factors, so the largest such partner and the smallest
// partner inside the band answer that exactly:
//   kMasked  every product flushes to +0 (zeros; small values against partners of ordinary size)
//   kSmall   below the band, and every product with a partner inside the band passes
//   kGreat   above the band, finite, and every product with a partner not above the band stays below the pass bound
//            (with a partner inside the band it does not flush either: 2^61 * 2^-61 = 1)
//   kOdd     anything else: inf, NaN, values whose products do not all behave alike
// Only products of two out-of-band elements are left to sort out: two masked ones flush (each has the other among its
// partners), and so do a masked and a small one; any other such pair among a warp's rows and columns, and anything odd,
// sends the line to the loop that forms the true product of every pair.
// When the look is taken.  A slab without it takes the loops of the smaller tiles: "flush or add" for every dirty line, the full
// rule for those that can overflow.  (Figures: 4096^3, with a look in every dirty slab -> now.)
//   * Not for one or two dirty lines (one in a slab with elements above the band): the look costs about 40 % of a clean slab, a
//     dirty line 8 % (0.01 % zeros 5130 -> 5010 us).
//   * Not while it finds too much to check.  A checked line takes the full rule (a second loop here, for lines that cannot overflow,
//     cost 2 % specials 24 %: the loops compete for the instruction cache), and warps with many of them keep the others waiting.
//     Each look weighs 2 * (lines to check, of 16 in each of 8 warps) against 3 * (dirty lines) - 4, or against 200 in a slab
//     with elements above the band, where a slab without the look has to search for overflows; the sum forgets
//     a quarter with each look, and above kAgainst the next slabs of the tile go without (one slab's count is too coarse:
//     where looks and slabs without alternate among the tiles of an SM, both are slower).
//     One operand around the flush bound 16700 -> 9560 us (with "flush or add" alone 10490), 3 % values below the
//     band 13410 -> 9530 (10530), 10 % specials 16920 -> 15830 (16300); 1 % specials keep their looks: 9880 (10650).
enum Class { kMasked = 1, kSmall = 2, kGreat = 4, kOdd = 8 };
enum LineKind { kPlain = 0, kRowsOff = 1, kColsOff = 2, kBothOff = 3, kChecked = 4, kNothing = 5 };

constexpr int kFewBelow = 2, kFewAbove = 1, kCheckedAbove = 200, kAgainst = 16, kSlabsWithout = 64;

__device__ __forceinline__ unsigned class_of(uint32_t magnitude, float smallest, float largest) {
    const float m = i2f((int32_t)magnitude);
    if (magnitude >= kBandHi) return fmul(m, largest) <= i2f(kPassBits) ? kGreat : kOdd;      // (not <=: inf and NaN)
    if (fmul(m, largest) <= i2f(kFlushBits)) return kMasked;
    return fmul(m, smallest) > i2f(kFlushBits) ? kSmall : kOdd;
}

// The loop for a line whose rows / columns of one warp hold elements of these classes; `flushes`: the line's largest
// magnitudes that are not above the band flush each other.
__device__ __forceinline__ unsigned kind_of(unsigned rows, unsigned cols, bool flushes) {
    const unsigned both = rows | cols;
    if ((both & kOdd) || ((rows & kGreat) && cols) || ((cols & kGreat) && rows) || (rows & cols & kSmall)) return kChecked;
    if (flushes && !(both & kGreat)) return kNothing;
    return (rows & kMasked ? kRowsOff : 0u) | (cols & kMasked ? kColsOff : 0u);
}

// ---- two sums in one instruction ----------------------------------------------------------------------------------
// acc0 += p0, acc1 += p1 and acc0 = p0 * w0 + acc0, acc1 = p1 * w1 + acc1, each with the one rounding of its scalar form.
// The packed add does not double the adds per cycle (register-only: 16.7 T pairs of one integer and one packed half against
// 16.3 T), but it halves the adds that the scheduler has to issue: clean loops 4096^3 4848 -> 4562 us, 4096x512x512 (two K ranges)
// 98.4 -> 94.4; the 64x64 and 32x32 tiles, which issue more beside the adds, gain 0 to 5 %.  In a rolled loop (the lines of dirty
// slabs) it is slower than the scalar one, 11.6 against 16.4 T.
// The exact-gradient products, which take three instructions per product, gain 3 to 10 % (12608x192x768 211 -> 200 us).
__device__ __forceinline__ void add_pair(float& acc0, float& acc1, int p0, int p1) {
    asm("{ .reg .b64 s, t;\n mov.b64 s, {%0, %1};\n mov.b64 t, {%2, %3};\n add.rn.f32x2 s, s, t;\n mov.b64 {%0, %1}, s; }"
        : "+f"(acc0), "+f"(acc1) : "r"(p0), "r"(p1));
}
__device__ __forceinline__ void fma_pair(float& acc0, float& acc1, int p0, int p1, float w0, float w1) {
    asm("{ .reg .b64 s, t, w;\n mov.b64 s, {%0, %1};\n mov.b64 t, {%2, %3};\n mov.b64 w, {%4, %5};\n"
        " fma.rn.f32x2 s, t, w, s;\n mov.b64 {%0, %1}, s; }"
        : "+f"(acc0), "+f"(acc1) : "r"(p0), "r"(p1), "f"(w0), "f"(w1));
}

// ---- which pipe an integer add runs on -------------------------------------------------------------------------------
// An SM partition dispatches one 32-lane instruction per cycle (a packed one counts twice) to three pipes of 16 lanes:
// integer / logic, and two for floating point, of which the first also takes integer multiply-adds.  Per pair of products
// the packed add occupies both floating-point pipes, so of the two integer adds three quarters belong on the integer pipe.
// Left to choose, the compiler forms so many as multiply-adds that the first floating-point pipe becomes the bound
// (4096^3: busy 84 %, the integer pipe 48 %, dispatch 93 %).  Here the source chooses: the larger of
// x + y and INT32_MIN is one instruction of the integer pipe, x * 1 + y one of the floating-point pipe, and both are
// x + y for all values.  (A constant bound or factor would be folded away.  A three-operand add is slower, 4096^3 4950
// to 5240 us: one more register read.)
// Products (i, j) of a thread's micro-tile that multiply_add_product names go to the floating-point pipe, 26 % of 64: 4096^3
// 4555 -> 4387 us, 12608x768x192 139.3 -> 131.5, 4096x512x512 96.3 -> 92.2.  The share and the places were found by trial:
// 0 % 4735, 19 % 4497, 25 % 4367 to 4550 by place, 31 % 4372, 38 % 4430, 50 % 4582.
__device__ __forceinline__ int sum_on_alu(int x, int y, int least) { return __viaddmax_s32(x, y, least); }
__device__ __forceinline__ int sum_on_fma(int x, int y, int one) {
    int d;
    asm("mad.lo.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(one), "r"(y));
    return d;
}
__host__ __device__ constexpr bool multiply_add_product(int i, int j) { return j == 3 || j == 5 || (i == 7 && j == 1); }
// The exact-gradient products mask every sum on the integer pipe, which leaves more of the sums to the other: 81 %.
// 12608x192x768 198 -> 182 us, 768x192x12608 209 -> 195, 2048x2048x1024 474 -> 446 (75 % 185 / 195 / 455, 88 % 185 / 197 / 450, all
// 195 / 208 / 469).
__host__ __device__ constexpr bool multiply_add_slope(int i, int j) { return (i + j) % 4 != 0 || i % 4 == 2; }
template <bool (*ON)(int, int)>
constexpr int products_on_fma() {
    int n = 0;
    for (int i = 0; i < 64; ++i) n += ON(i / 8, i % 8);
    return n;
}
static_assert(products_on_fma<multiply_add_product>() == 17 && products_on_fma<multiply_add_slope>() == 52, "the shares stated above, of 64");

// ---- eight sums at once, or none of them ----------------------------------------------------------------------------
// c += p where x is not zero (either sign of it), and where pattern x is not `zero`: one compare for eight adds.  Written as conditions
// around each add, the compiler makes branches of them once the products' adds are no longer plain ones.
#define PAMK_EIGHT(c0, c1, c2, c3, c4, c5, c6, c7) "+f"(c0), "+f"(c1), "+f"(c2), "+f"(c3), "+f"(c4), "+f"(c5), "+f"(c6), "+f"(c7)
#define PAMK_PRODUCTS "f"(i2f(q[0])), "f"(i2f(q[1])), "f"(i2f(q[2])), "f"(i2f(q[3])), "f"(i2f(q[4])), "f"(i2f(q[5])), "f"(i2f(q[6])), "f"(i2f(q[7]))
#define PAMK_ADD_EIGHT                                                                                            \
    "@on add.rn.f32 %0, %0, %8;\n @on add.rn.f32 %1, %1, %9;\n @on add.rn.f32 %2, %2, %10;\n @on add.rn.f32 %3, %3, %11;\n"   \
    "@on add.rn.f32 %4, %4, %12;\n @on add.rn.f32 %5, %5, %13;\n @on add.rn.f32 %6, %6, %14;\n @on add.rn.f32 %7, %7, %15; }"
#define PAMK_WEIGHTS_EIGHT "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3]), "f"(w[4]), "f"(w[5]), "f"(w[6]), "f"(w[7])
#define PAMK_FMA_EIGHT                                                                                                                     \
    "@on fma.rn.f32 %0, %8, %16, %0;\n @on fma.rn.f32 %1, %9, %17, %1;\n @on fma.rn.f32 %2, %10, %18, %2;\n @on fma.rn.f32 %3, %11, %19, %3;\n" \
    "@on fma.rn.f32 %4, %12, %20, %4;\n @on fma.rn.f32 %5, %13, %21, %5;\n @on fma.rn.f32 %6, %14, %22, %6;\n @on fma.rn.f32 %7, %15, %23, %7; }"
template <int MR, int MT>
__device__ __forceinline__ void add_column_unless_zero(int x, float (&acc)[MR][MT], int j, const int (&q)[8]) {
    float spare = 0.0f;
    float& last = MR == 8 ? acc[7 % MR][j] : spare;
    asm("{ .reg .pred on;\n setp.neu.f32 on, %16, 0f00000000;\n" PAMK_ADD_EIGHT
        : PAMK_EIGHT(acc[0][j], acc[1][j], acc[2][j], acc[3][j], acc[4 % MR][j], acc[5 % MR][j], acc[6 % MR][j], last)
        : PAMK_PRODUCTS, "f"(i2f(x)));
}
// the same where `off` is zero
template <int MR, int MT>
__device__ __forceinline__ void add_column_unless(unsigned off, float (&acc)[MR][MT], int j, const int (&q)[8]) {
    float spare = 0.0f;
    float& last = MR == 8 ? acc[7 % MR][j] : spare;
    asm("{ .reg .pred on;\n setp.eq.s32 on, %16, 0;\n" PAMK_ADD_EIGHT
        : PAMK_EIGHT(acc[0][j], acc[1][j], acc[2][j], acc[3][j], acc[4 % MR][j], acc[5 % MR][j], acc[6 % MR][j], last)
        : PAMK_PRODUCTS, "r"(off));
}
template <int MT>
__device__ __forceinline__ void add_row_unless(unsigned off, float (&acc)[MT], const int (&q)[8]) {
    asm("{ .reg .pred on;\n setp.eq.s32 on, %16, 0;\n" PAMK_ADD_EIGHT
        : PAMK_EIGHT(acc[0], acc[1], acc[2], acc[3], acc[4 % MT], acc[5 % MT], acc[6 % MT], acc[7 % MT])
        : PAMK_PRODUCTS, "r"(off));
}
template <int MT>
__device__ __forceinline__ void add_row_unless_zero(int x, int zero, float (&acc)[MT], const int (&q)[8]) {
    asm("{ .reg .pred on;\n setp.ne.s32 on, %16, %17;\n" PAMK_ADD_EIGHT
        : PAMK_EIGHT(acc[0], acc[1], acc[2], acc[3], acc[4 % MT], acc[5 % MT], acc[6 % MT], acc[7 % MT])
        : PAMK_PRODUCTS, "r"(x), "r"(zero));
}
// c = fma(p, w, c) where x is not zero
template <int MR, int MT>
__device__ __forceinline__ void fma_column_unless_zero(int x, float (&acc)[MR][MT], int j, const int (&q)[8], const float (&w)[8]) {
    float spare = 0.0f;
    float& last = MR == 8 ? acc[7 % MR][j] : spare;
    asm("{ .reg .pred on;\n setp.neu.f32 on, %24, 0f00000000;\n" PAMK_FMA_EIGHT
        : PAMK_EIGHT(acc[0][j], acc[1][j], acc[2][j], acc[3][j], acc[4 % MR][j], acc[5 % MR][j], acc[6 % MR][j], last)
        : PAMK_PRODUCTS, PAMK_WEIGHTS_EIGHT, "f"(i2f(x)));
}
template <int MR, int MT>
__device__ __forceinline__ void fma_column_unless(unsigned off, float (&acc)[MR][MT], int j, const int (&q)[8], const float (&w)[8]) {
    float spare = 0.0f;
    float& last = MR == 8 ? acc[7 % MR][j] : spare;
    asm("{ .reg .pred on;\n setp.eq.s32 on, %24, 0;\n" PAMK_FMA_EIGHT
        : PAMK_EIGHT(acc[0][j], acc[1][j], acc[2][j], acc[3][j], acc[4 % MR][j], acc[5 % MR][j], acc[6 % MR][j], last)
        : PAMK_PRODUCTS, PAMK_WEIGHTS_EIGHT, "r"(off));
}
#undef PAMK_FMA_EIGHT
#undef PAMK_WEIGHTS_EIGHT
#undef PAMK_ADD_EIGHT
#undef PAMK_PRODUCTS
#undef PAMK_EIGHT

template <int MODE, class T, bool A_KC, bool B_KC, bool VEC>
__global__ void __launch_bounds__(T::kThreads, MODE == kPam || MODE == kStd ? T::kCtasPerSm : T::kCtasPerSm / 2)
gemm_kernel(const GemmParams p) {
    constexpr int BM = T::BM, BN = T::BN, BK = T::BK, MT = T::MT, MR = T::MR;
    static_assert(MR == MT || (MODE == kPam && (A_KC || !VEC)), "fewer rows per thread: no 128-bit loads along A's rows");
    constexpr bool kLook = MODE == kPam && BM == 128;      // dirty slabs are looked through (see class_of)
    // (the variant with both operands contiguous along their row index spills registers at 8)
    constexpr int kFastUnroll = (!A_KC && !B_KC) || 8 > BK ? BK : 8;
    __shared__ __align__(16) float As[2][BK * row_stride(BM)];
    __shared__ __align__(16) float Bs[2][BK * row_stride(BN)];
    __shared__ __align__(16) float weights[MODE == kPam && MT == 4 ? BK * row_stride(BM) : 1];   // of the side that holds zeros (32x32 tile)
    __shared__ unsigned lines[3];   // per slab (Word)
    __shared__ int look_from, against;    // looks: from which slab on, and what speaks against them (see class_of)
    __shared__ unsigned overflow_lines;   // bit k = some product of k line may leave the pass range
    // looked-through slabs: per line and thread row / column a bit for each masked element, per warp and line the LineKind
    __shared__ unsigned char rows_off[kLook ? BK : 1][16], cols_off[kLook ? BK : 1][16], line_kinds[kLook ? 8 : 1][BK];

    const int tid = threadIdx.x;
    // a warp is 4 x 8 threads: the fewer rows and columns it has, the fewer of their lines hold out-of-band elements
    const int tx = T::TX == 16 ? (tid >> 5 & 1) * 8 + (tid & 7) : tid % T::TX;
    const int ty = T::TX == 16 ? (tid >> 6) * 4 + (tid >> 3 & 3) : tid / T::TX;
    const int m0 = blockIdx.y * T::kRows, n0 = blockIdx.x * BN;
    const int z = blockIdx.z / p.splits, sp = blockIdx.z - z * p.splits;
    const int k_begin = sp * p.k_chunk;
    const int k_end = min(p.K, k_begin + p.k_chunk);
    const int slabs = (k_end - k_begin + BK - 1) / BK;

    // batch z = outer * inner + (index in the inner dimension); outer = z / inner by a multiply-high with
    // the reciprocal prepared on the host (exact for z < 65536, the grid limit); the strides arrive
    // rearranged so that the offset is outer * sb + z * sb2
    const unsigned zo = __umulhi((unsigned)z, p.inner_magic);
    const float* Ab = p.A.p + (int64_t)zo * p.A.sb + (int64_t)z * p.A.sb2;
    const float* Bb = p.B.p + (int64_t)zo * p.B.sb + (int64_t)z * p.B.sb2;

    float acc[MR][MT];
#pragma unroll
    for (int i = 0; i < MR; ++i)
#pragma unroll
        for (int j = 0; j < MT; ++j) acc[i][j] = 0.0f;

    after_previous();
    // exact-gradient product: per-output constant (mantissa of D + offset) that the slope adds to
    // the other operand's bits (pam_scalar.cuh mul_slope).
    int32_t dm[MODE >= kBwdL ? MR : 1][MODE >= kBwdL ? MT : 1];
    if constexpr (MODE >= kBwdL) {
        const float* Db = p.D + (int64_t)z * p.sDb;
#pragma unroll
        for (int i = 0; i < MR; ++i) {
            int row = m0 + ty * 4 + (i & 3) + (i >> 2) * (BM / 2);
            row = row < p.M ? row : p.M - 1;
#pragma unroll
            for (int j = 0; j < MT; ++j) {
                int col = n0 + tx * 4 + (j & 3) + (j >> 2) * (BN / 2);
                col = col < p.N ? col : p.N - 1;
                dm[i][j] = iadd(kMant & f2i(Db[(int64_t)row * p.sDm + (int64_t)col * p.sDn]), p.off);
            }
        }
    }

    if (MODE == kPam && tid < 3) lines[tid] = 0;
    if (kLook && tid == 0) look_from = against = 0;

    float ra[T::kTasksA * 4], rb[T::kTasksB * 4];
    // (not the scalar form of the 32x32x16 tile, nor of the 32x32x8 tile with both operands along K: 200 products 151x150x150 98.6 -> 100.3 us)
    constexpr bool kWalks = VEC || T::MT == 8 || (T::BK == 8 && !(A_KC && B_KC));
    std::conditional_t<VEC, SlabWalker<T, BM, T::kTasksA, A_KC>, ScalarWalker<T, BM, T::kTasksA, A_KC>> walk_a;
    std::conditional_t<VEC, SlabWalker<T, BN, T::kTasksB, B_KC>, ScalarWalker<T, BN, T::kTasksB, B_KC>> walk_b;
    if constexpr (kWalks) {
        walk_a.template init<T::MR != T::MT>(p.A, Ab, m0, p.M, k_begin, tid);
        walk_b.template init<false>(p.B, Bb, n0, p.N, k_begin, tid);
    }
    auto stage_load = [&](int k0) {
        if constexpr (kWalks) {
            walk_a.load(ra, k0, k_end, tid);
            walk_b.load(rb, k0, k_end, tid);
        } else {
            load_slab<T, BM, T::kTasksA, A_KC>(ra, p.A, Ab, m0, p.M, k0, k_end, tid);
            load_slab<T, BN, T::kTasksB, B_KC>(rb, p.B, Bb, n0, p.N, k0, k_end, tid);
        }
    };
    auto stage_store = [&](int buf, int slot) {
        if (MODE == kPam) {
            // clean warps (the common case) pay the band test and one vote; only a warp that holds
            // an out-of-band element locates it and reports its k line to the slab's word
            const bool out = band_excess(rb, band_excess(ra, 0u)) >= kBandSpan2;
            if (__any_sync(0xffffffffu, out)) {
                unsigned f = 0;
                if (out) {
                    uint32_t bits = 0, top = 0;
                    const unsigned in_a = dirty_lines<T, BM, T::kTasksA, A_KC>(ra, tid, bits, top);
                    const unsigned in_b = dirty_lines<T, BN, T::kTasksB, B_KC>(rb, tid, bits, top);
                    f = in_a | in_b | (in_a ? (unsigned)kInA : 0u) | (in_b ? (unsigned)kInB : 0u) | (bits ? (unsigned)kNonZero : 0u) |
                        (top >= kBandHi2 ? (unsigned)kAbove : 0u);
                    if (MT == 8) {                     // one pattern for A's zeros, of either sign: the loops for zeros look for it
#pragma unroll
                        for (int c = 0; c < T::kTasksA * 4; ++c) ra[c] = fadd(ra[c], 0.0f);
                    }
                }
                if constexpr (MT == 4) {
                    // (the 32x32 tile's launches are chains of slabs: atomics of two warps cost less than the wait for a reduction)
                    if (f) atomicOr(&lines[slot], f);
                } else {
                    f = __reduce_or_sync(0xffffffffu, f);
                    if ((tid & 31) == 0) atomicOr(&lines[slot], f);
                }
            }
            // the A side is pre-biased (bits - (0x3f800000 - offset)) so that a product is a two-input add
#pragma unroll
            for (int c = 0; c < T::kTasksA * 4; ++c) ra[c] = i2f(isub(f2i(ra[c]), p.bias_sub));
        }
        store_slab<T, BM, T::kTasksA, A_KC>(As[buf], ra, tid);
        store_slab<T, BN, T::kTasksB, B_KC>(Bs[buf], rb, tid);
    };

    if (slabs > 0) stage_load(k_begin);
    __syncthreads();               // flag words initialised
    if (slabs > 0) stage_store(0, 0);
    __syncthreads();

    // One slab.  (Written as a lambda called from the loop below: in this form the compiler's register
    // allocation of the 128x128 kernels needs no spills, which the same statements placed directly in
    // the loop body do.)
    auto slab_iteration = [&](int s) {
        const int buf = s & 1;
        const bool more = s + 1 < slabs;
        if (more) stage_load(k_begin + (s + 1) * BK);
        unsigned dirty = 0;
        if (MODE == kPam) {
            dirty = lines[s % 3];
            // the word two slabs ahead was last read before the previous barrier: reset it now
            if (tid == 0) lines[(s + 2) % 3] = 0;
        }
        const float* as = As[buf];
        const float* bs = Bs[buf];

#define PAMK_FRAGMENTS(kk)                                                                              \
        const int4 a0 = *reinterpret_cast<const int4*>(as + (kk) * row_stride(BM) + ty * 4);           \
        const int4 a1 = MT == 8 ? *reinterpret_cast<const int4*>(as + (kk) * row_stride(BM) + ty * 4 + BM / 2) : a0; \
        const int4 b0 = *reinterpret_cast<const int4*>(bs + (kk) * row_stride(BN) + tx * 4);           \
        const int4 b1 = MT == 8 ? *reinterpret_cast<const int4*>(bs + (kk) * row_stride(BN) + tx * 4 + BN / 2) : b0; \
        const int a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};                              \
        const int b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};

#define PAMK_WEIGHTS(kk, at)                                                                            \
        const float4 w4 = *reinterpret_cast<const float4*>(weights + (kk) * row_stride(BM) + (at) * 4); \
        const float w[4] = {w4.x, w4.y, w4.z, w4.w};

        if (MODE == kPam && dirty == 0) {
#pragma unroll kFastUnroll
            for (int kk = 0; kk < BK; ++kk) {
                PAMK_FRAGMENTS(kk)
#pragma unroll
                for (int i = 0; i < MR; ++i)
#pragma unroll
                    for (int j = 0; j < MT; j += 2) {
                        if constexpr (MT == 8 || VEC) {
                            auto product = [&](int c) {
                                return multiply_add_product(i, c) ? sum_on_fma(a[i], b[c], p.one) : sum_on_alu(a[i], b[c], p.least);
                            };
                            add_pair(acc[i][j], acc[i][j + 1], product(j), product(j + 1));
                        } else {                                        // (the pairs made the 32x32 tile's scalar-load kernels spill)
                            acc[i][j] = fadd(acc[i][j], i2f(iadd(a[i], b[j])));
                            acc[i][j + 1] = fadd(acc[i][j + 1], i2f(iadd(a[i], b[j + 1])));
                        }
                    }
            }
        } else if constexpr (MODE == kPam) {
            constexpr unsigned all_lines = (1u << BK) - 1u;
            const unsigned any = dirty & all_lines;
            const bool mostly = __popc(any) * 4 >= BK * 3;              // most lines are dirty
            // One line by the plain sum, by "flush or add", or by the full rule.
            auto plain_line = [&](int kk) {
                PAMK_FRAGMENTS(kk)
#pragma unroll
                for (int i = 0; i < MR; ++i)
#pragma unroll
                    for (int j = 0; j < MT; ++j) acc[i][j] = fadd(acc[i][j], i2f(iadd(a[i], b[j])));
            };
            auto checked_line = [&](int kk, auto full_rule) {
                PAMK_FRAGMENTS(kk)
                float araw[MR];                                         // a[] holds pre-biased patterns; the rule needs the values
#pragma unroll
                for (int i = 0; i < MR; ++i) araw[i] = i2f(iadd(a[i], p.bias_sub));
#pragma unroll
                for (int i = 0; i < MR; ++i)
#pragma unroll
                    for (int j = 0; j < MT; ++j) {
                        const float mag = fabsf(fmul(araw[i], i2f(b[j])));
                        if constexpr (decltype(full_rule)::value) {
                            const float prod = mag <= i2f(kPassBits) ? i2f(iadd(a[i], b[j])) : quiet_nan();
                            if (!(mag <= i2f(kFlushBits))) acc[i][j] = fadd(acc[i][j], prod);
                        } else {
                            if (mag > i2f(kFlushBits)) acc[i][j] = fadd(acc[i][j], i2f(iadd(a[i], b[j])));
                        }
                    }
            };
            int kk = 0;
            auto run_end = [&](unsigned mask) { return min(BK, kk + __ffs((int)(~mask >> kk)) - 1); };
            if (MT == 8 && !(dirty & kNonZero) && mostly) {
                // Zeros, and everything else in the band: a zero's products are left out by a predicate.
                // 4096^3 with one operand half zeros 5500 us (clean: 4387), both 7070 (a condition around each add: 5840 and 7420, of
                // which a compare per row or column, and for A's rows the removal of the bias, took 16 instructions a line).
                if constexpr (MT == 8) {
                if (!(dirty & kInA)) {
#pragma unroll 1
                    for (; kk < BK; ++kk) {
                        PAMK_FRAGMENTS(kk)
#pragma unroll
                        for (int j = 0; j < MT; ++j) {
                            int q[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) q[i] = iadd(a[i], b[j]);
                            add_column_unless_zero(b[j], acc, j, q);
                        }
                    }
                } else if (!(dirty & kInB)) {
#pragma unroll 1
                    for (; kk < BK; ++kk) {
                        PAMK_FRAGMENTS(kk)
#pragma unroll
                        for (int i = 0; i < MR; ++i) {
                            int q[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) q[j] = iadd(a[i], b[j]);
                            add_row_unless_zero(a[i], -p.bias_sub, acc[i], q);
                        }
                    }
                } else {
                    // rows by a weight: a zero's products (made finite) get weight 0 in a fused multiply-add, which leaves a sum alone
                    // (it is never -0)
#pragma unroll 1
                    for (; kk < BK; ++kk) {
                        PAMK_FRAGMENTS(kk)
                        float w[8];
                        int ai[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const bool zero = a[i] == -p.bias_sub;
                            w[i] = zero ? 0.0f : 1.0f;
                            ai[i] = zero ? 0 : a[i];
                        }
#pragma unroll
                        for (int j = 0; j < MT; ++j) {
                            int q[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) q[i] = iadd(ai[i], b[j]);
                            fma_column_unless_zero(b[j], acc, j, q, w);
                        }
                    }
                }
                }
            } else if (kLook && __popc(any) > (dirty & kAbove ? kFewAbove : kFewBelow) && s >= look_from) {
                // (the same for all threads: look_from is read after the barrier that ends a slab and written after the one below)
                if constexpr (kLook) {
                // sixteen threads look through one line, the two groups of four elements of either side that thread row / column
                // `at` works on each
                static_assert(!kLook || (BK == 16 && T::kThreads == 256 && BN == 128 && MT == 8), "a warp looks through two lines");
                const int lane = tid & 31, warp = tid >> 5, line = tid >> 4, at = tid & 15;
                bool vote = false;
                if (any >> (2 * warp) & 3u) {                       // (the same for a warp)
                    uint32_t ma[8], mb[8];
                    // the smallest magnitude in the band and the largest that is not above it, as offsets in which what does not count
                    // wraps around to the losing end
                    uint32_t lo_a = ~0u, hi_a = 0u, lo_b = ~0u, hi_b = 0u;
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int4 va = *reinterpret_cast<const int4*>(as + line * row_stride(BM) + q * (BM / 2) + at * 4);
                        const int4 vb = *reinterpret_cast<const int4*>(bs + line * row_stride(BN) + q * (BN / 2) + at * 4);
                        const int ea[4] = {va.x, va.y, va.z, va.w}, eb[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint32_t xa = (uint32_t)iadd(ea[c], p.bias_sub) & 0x7fffffffu, xb = (uint32_t)eb[c] & 0x7fffffffu;
                            ma[q * 4 + c] = xa;
                            mb[q * 4 + c] = xb;
                            lo_a = min(lo_a, xa - kBandLo); hi_a = max(hi_a, xa - kBandHi);
                            lo_b = min(lo_b, xb - kBandLo); hi_b = max(hi_b, xb - kBandHi);
                        }
                    }
#pragma unroll
                    for (int d = 1; d < 16; d <<= 1) {
                        lo_a = min(lo_a, __shfl_xor_sync(0xffffffffu, lo_a, d)); hi_a = max(hi_a, __shfl_xor_sync(0xffffffffu, hi_a, d));
                        lo_b = min(lo_b, __shfl_xor_sync(0xffffffffu, lo_b, d)); hi_b = max(hi_b, __shfl_xor_sync(0xffffffffu, hi_b, d));
                    }
                    auto smallest = [](uint32_t lo) { return lo < kBandHi - kBandLo ? i2f((int32_t)(lo + kBandLo)) : INFINITY; };
                    auto largest = [](uint32_t hi) { return hi >= 0u - kBandHi ? i2f((int32_t)(hi + kBandHi)) : 0.0f; };   // +0: all above
                    const float small_a = smallest(lo_a), large_a = largest(hi_a), small_b = smallest(lo_b), large_b = largest(hi_b);
                    const bool flushes = fmul(large_a, large_b) <= i2f(kFlushBits);
                    unsigned off_a = 0, off_b = 0, classes = 0;          // masked elements; classes of the rows, and of the columns from bit 8 on
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        if (ma[c] - kBandLo >= kBandHi - kBandLo) {
                            const unsigned k = class_of(ma[c], small_b, large_b);
                            off_a |= (k & kMasked) << c;
                            classes |= k;
                        }
                        if (mb[c] - kBandLo >= kBandHi - kBandLo) {
                            const unsigned k = class_of(mb[c], small_a, large_a);
                            off_b |= (k & kMasked) << c;
                            classes |= k << 8;
                        }
                    }
                    rows_off[line][at] = (unsigned char)off_a;
                    cols_off[line][at] = (unsigned char)off_b;
                    // of the four thread rows, and the eight thread columns, of a warp
                    classes |= __shfl_xor_sync(0xffffffffu, classes, 1);
                    classes |= __shfl_xor_sync(0xffffffffu, classes, 2);
                    const unsigned rows = classes & 15u, cols = (classes | __shfl_xor_sync(0xffffffffu, classes, 4)) >> 8;
                    const unsigned other = __shfl_xor_sync(0xffffffffu, cols, 8);
                    const unsigned kind = kind_of(rows, cols, flushes), other_kind = kind_of(rows, other, flushes);
                    if (at % 4 == 0) {
                        line_kinds[at / 4 * 2 + at / 8][line] = (unsigned char)kind;
                        line_kinds[at / 4 * 2 + (at / 8 ^ 1)][line] = (unsigned char)other_kind;
                    }
                    vote = at % 4 == 0 ? kind == kChecked : (at % 4 == 1 && other_kind == kChecked);    // (four threads hold the same)
                } else if (at < 8) {
                    line_kinds[at][line] = kPlain;
                }
                const int votes = __syncthreads_count(vote);        // lines to be checked, of eight warps
                if (tid == 0) {
                    against += 2 * votes - (dirty & kAbove ? kCheckedAbove : 3 * __popc(any) - 4) - against / 4;
                    if (against > kAgainst) look_from = s + kSlabsWithout;
                }
                // This warp's lines, in runs of one kind, each kind with a loop of its own with one copy of its body (with three
                // bodies side by side in one loop the schedule cost 12 %).  Lane k holds the kind of line k: a mask per kind, kept in
                // registers, was 3 % faster with 0.1 % specials and 12 to 32 % slower with 1.5 to 3 %.
                const unsigned mine = line_kinds[warp][lane % BK];
                while (kk < BK) {
                    const unsigned kind = __shfl_sync(0xffffffffu, mine, kk);
                    const int end = run_end(__ballot_sync(0xffffffffu, mine == kind) & all_lines);
                    if (kind == kPlain) {
#pragma unroll 1
                        for (; kk < end; ++kk) plain_line(kk);
                    } else if (kind == kColsOff) {
#pragma unroll 1
                        for (; kk < end; ++kk) {
                            PAMK_FRAGMENTS(kk)
                            const unsigned off = cols_off[kk][tx];
#pragma unroll
                            for (int i = 0; i < MR; ++i)
#pragma unroll
                                for (int j = 0; j < MT; ++j)
                                    if (!(off & (1u << j))) acc[i][j] = fadd(acc[i][j], i2f(iadd(a[i], b[j])));
                        }
                    } else if (kind == kRowsOff) {
#pragma unroll 1
                        for (; kk < end; ++kk) {
                            PAMK_FRAGMENTS(kk)
                            const unsigned off = rows_off[kk][ty];
#pragma unroll
                            for (int j = 0; j < MT; ++j)
#pragma unroll
                                for (int i = 0; i < MR; ++i)
                                    if (!(off & (1u << i))) acc[i][j] = fadd(acc[i][j], i2f(iadd(a[i], b[j])));
                        }
                    } else if (kind == kChecked) {
#pragma unroll 1
                        for (; kk < end; ++kk) checked_line(kk, std::true_type{});
                    } else if (kind == kBothOff) {                      // rows by weights, as above
#pragma unroll 1
                        for (; kk < end; ++kk) {
                            PAMK_FRAGMENTS(kk)
                            const unsigned off = cols_off[kk][tx], rows = rows_off[kk][ty];
#pragma unroll
                            for (int i = 0; i < MR; ++i) {
                                const float w = rows & (1u << i) ? 0.0f : 1.0f;
                                const int ai = rows & (1u << i) ? 0 : a[i];
#pragma unroll
                                for (int j = 0; j < MT; ++j)
                                    if (!(off & (1u << j))) acc[i][j] = __fmaf_rn(i2f(iadd(ai, b[j])), w, acc[i][j]);
                            }
                        }
                    }
                    kk = end;                                           // (kNothing: there is nothing to add)
                }
                }
            } else if (MT == 4 && !(dirty & kNonZero) && mostly) {
                // Zeros on the 32x32 tile, whose launches are chains of slabs: a pass over one
                // side's slab replaces each zero by a value that makes the product in-band and writes a weight beside
                // it, 0 for a zero and 1 for anything else; the sum then is acc = fma(product, weight, acc), which
                // is the plain sum for weight 1 and leaves acc alone for weight 0 (the products are finite, and a
                // sum is never -0).
                const bool side_b = !(dirty & kInA);
                float* side = side_b ? Bs[buf] : As[buf];
                // (the stand-in makes the product the other operand's own pattern, whatever the offset)
                const int zero_bits = side_b ? 0 : -p.bias_sub, stand_in = side_b ? p.bias_sub : 0;
                static_assert(BM == BN, "one loop serves both sides");
#pragma unroll
                for (int t = 0; t < T::kTasksA; ++t) {
                    const int id = tid + t * T::kThreads;
                    const int at = id / (BM / 4) * row_stride(BM) + id % (BM / 4) * 4;
                    int4 v = *reinterpret_cast<const int4*>(side + at);
                    float4 w;
                    w.x = 2u * (uint32_t)isub(v.x, zero_bits) == 0 ? 0.0f : 1.0f; v.x = 2u * (uint32_t)isub(v.x, zero_bits) == 0 ? stand_in : v.x;
                    w.y = 2u * (uint32_t)isub(v.y, zero_bits) == 0 ? 0.0f : 1.0f; v.y = 2u * (uint32_t)isub(v.y, zero_bits) == 0 ? stand_in : v.y;
                    w.z = 2u * (uint32_t)isub(v.z, zero_bits) == 0 ? 0.0f : 1.0f; v.z = 2u * (uint32_t)isub(v.z, zero_bits) == 0 ? stand_in : v.z;
                    w.w = 2u * (uint32_t)isub(v.w, zero_bits) == 0 ? 0.0f : 1.0f; v.w = 2u * (uint32_t)isub(v.w, zero_bits) == 0 ? stand_in : v.w;
                    *reinterpret_cast<int4*>(side + at) = v;
                    *reinterpret_cast<float4*>(weights + at) = w;
                }
                __syncthreads();
                if ((dirty & (kInA | kInB)) == (kInA | kInB)) {
                    // (weights for A's zeros, a predicate for B's)
#pragma unroll 1
                    for (; kk < BK; ++kk) {
                        PAMK_FRAGMENTS(kk)
                        PAMK_WEIGHTS(kk, ty)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const bool on = 2u * (uint32_t)b[j] != 0;
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (on) acc[i % MR][j] = __fmaf_rn(i2f(iadd(a[i], b[j])), w[i], acc[i % MR][j]);
                        }
                    }
                } else if (!side_b) {
#pragma unroll 1
                    for (; kk < BK; ++kk) {
                        PAMK_FRAGMENTS(kk)
                        PAMK_WEIGHTS(kk, ty)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) acc[i % MR][j] = __fmaf_rn(i2f(iadd(a[i], b[j])), w[i], acc[i % MR][j]);
                    }
                } else {
#pragma unroll 1
                    for (; kk < BK; ++kk) {
                        PAMK_FRAGMENTS(kk)
                        PAMK_WEIGHTS(kk, tx)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) acc[i % MR][j] = __fmaf_rn(i2f(iadd(a[i], b[j])), w[j], acc[i % MR][j]);
                    }
                }
            } else {
                // lines of a slab that holds an element above the band: can a product leave the pass range?
                unsigned full = 0;
                if (dirty & kAbove) {                               // (uniform: read from shared memory after a barrier)
                    constexpr int kLanes = T::kThreads / BK;        // threads that share one k line
                    const int line = tid / kLanes, lane = tid % kLanes;
                    if (tid == 0) overflow_lines = 0;
                    __syncthreads();
                    // (every thread takes part, whatever its line: the shuffles below name all 32 lanes)
                    uint32_t hi_a = 0, hi_b = 0;                    // magnitudes compare like their bit patterns; inf / NaN are largest
                    for (int q = lane; q < BM; q += kLanes) {
                        hi_a = max(hi_a, (uint32_t)iadd(f2i(as[line * row_stride(BM) + q]), p.bias_sub) & 0x7fffffffu);
                        hi_b = max(hi_b, (uint32_t)f2i(bs[line * row_stride(BN) + q]) & 0x7fffffffu);
                    }
#pragma unroll
                    for (int d = 1; d < kLanes; d <<= 1) {
                        hi_a = max(hi_a, __shfl_xor_sync(0xffffffffu, hi_a, d));
                        hi_b = max(hi_b, __shfl_xor_sync(0xffffffffu, hi_b, d));
                    }
                    // (an inf or NaN maximum makes the product inf or NaN: not <= the pass bound)
                    if (lane == 0 && !(fmul(i2f((int32_t)hi_a), i2f((int32_t)hi_b)) <= i2f(kPassBits))) atomicOr(&overflow_lines, 1u << line);
                    __syncthreads();
                    full = overflow_lines;
                }
                // Most lines dirty, none can overflow (e.g. gradients of which most lie below the band): "flush or add" for the
                // whole slab, which is exact for clean lines too.  The 64x64 tile runs it in the loop for runs below: with a copy
                // of its own, 512 instructions, its dirty slabs wait for instructions (2235x183x1152 with 1 % specials 148 -> 109 us).
                const bool flush_all = mostly && full == 0;
                if (MT == 4 && flush_all) {
#pragma unroll 4
                    for (int k = 0; k < BK; ++k) checked_line(k, std::false_type{});
                } else {
                    const unsigned flush = flush_all ? all_lines : any & ~full;
                    while (kk < BK) {
                        const unsigned here = 1u << kk;
                        if (full & here) {
                            checked_line(kk, std::true_type{});
                            ++kk;
                        } else if (flush & here) {
                            const int end = run_end(flush);
#pragma unroll 1
                            for (; kk < end; ++kk) checked_line(kk, std::false_type{});
                        } else {
                            const unsigned others = any >> kk;
                            const int end = others ? kk + __ffs((int)others) - 1 : BK;
#pragma unroll 1
                            for (; kk < end; ++kk) plain_line(kk);
                        }
                    }
                }
            }
        } else if constexpr (MODE != kPam) {
#pragma unroll 2
            for (int kk = 0; kk < BK; ++kk) {
                PAMK_FRAGMENTS(kk)
                if constexpr (MODE == kStd) {
#pragma unroll
                    for (int i = 0; i < MR; ++i)
#pragma unroll
                        for (int j = 0; j < MT; ++j) acc[i][j] = __fmaf_rn(i2f(a[i]), i2f(b[j]), acc[i][j]);
                } else {
                    // acc += delta * 2^slope, slope from the non-delta operand and D
#pragma unroll
                    for (int i = 0; i < MR; ++i)
#pragma unroll
                        for (int j = 0; j < MT; j += 2) {
                            auto slope = [&](int c) {
                                const int of = MODE == kBwdL ? b[c] : a[i];
                                return kSignExp & (multiply_add_slope(i, c) ? sum_on_fma(of, dm[i][c], p.one) : sum_on_alu(of, dm[i][c], p.least));
                            };
                            fma_pair(acc[i][j], acc[i][j + 1], slope(j), slope(j + 1), i2f(MODE == kBwdL ? a[i] : b[j]),
                                     i2f(MODE == kBwdL ? a[i] : b[j + 1]));
                        }
                }
            }
        }
#undef PAMK_FRAGMENTS
#undef PAMK_WEIGHTS

        if (more) stage_store(buf ^ 1, (s + 1) % 3);
        __syncthreads();
    };
    for (int s = 0; s < slabs; ++s) slab_iteration(s);

    next_may_start();                                           // (the reduction pass)
    // ---- epilogue ----------------------------------------------------------------------------
    float* Cz = p.C + (int64_t)sp * p.sCsplit + (int64_t)__umulhi((unsigned)z, p.inner_magic) * p.sCb + (int64_t)z * p.sCb2;
    const bool vec_out = ((p.N | p.ldc | p.sCb | p.sCb2 | p.sCsplit) & 3) == 0 && aligned16(p.C);
    const bool post = p.post != 0 && p.splits == 1;             // (with split-K the reduction pass applies it)
    const bool add_bias = p.bias != nullptr && p.splits == 1;   // (with split-K the reduction pass adds it)
    if constexpr (MODE != kPam) {
        // The reference walks K in zero-filled tiles of 32 (cuda_kernels.cu:526-571, 608-629): when K
        // is not a multiple of 32 it also adds products of zeros, which turns a sum of -0 into +0.
        // (A PAM sum is never -0: flushed products are +0.)
        // In the exact-gradient kernel a padded term is pam_bwd(D, 0, 0) = 0 * slope(D, 0)
        // (cuda_kernels.cu:49-57, 795-809): with an offset below one and a small mantissa of D the
        // slope's bit pattern is -inf and the term is NaN.
        if (p.K & 31) {
#pragma unroll
            for (int i = 0; i < MR; ++i)
#pragma unroll
                for (int j = 0; j < MT; ++j) {
                    if constexpr (MODE == kStd) acc[i][j] = fadd(acc[i][j], 0.0f);
                    else acc[i][j] = __fmaf_rn(0.0f, i2f(kSignExp & dm[i][j]), acc[i][j]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < MR; ++i) {
        const int row = m0 + slot_row<T, BM>(ty * 4 + (i & 3) + (i >> 2) * (BM / 2));
        if (row >= p.M) continue;
        float* crow = Cz + (int64_t)row * p.ldc;
#pragma unroll
        for (int h = 0; h < MT / 4; ++h) {
            const int col = n0 + tx * 4 + h * (BN / 2);
            if (add_bias) {                            // the bias row is re-read per output row (it stays in L1)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (col + j < p.N) acc[i][h * 4 + j] = fadd(acc[i][h * 4 + j], p.bias[col + j]);
            }
            if (post) {
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][h * 4 + j] = mul(acc[i][h * 4 + j], p.post_scale, p.off);
            }
            if (vec_out) {
                if (col < p.N)
                    *reinterpret_cast<float4*>(crow + col) =
                        make_float4(acc[i][h * 4], acc[i][h * 4 + 1], acc[i][h * 4 + 2], acc[i][h * 4 + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (col + j < p.N) crow[col + j] = acc[i][h * 4 + j];
            }
        }
    }
}

#include "gemm_packed.cuh"

// Where the finished sums of a split-K product go: a plain [batch][M][N] array, or the strided output
// of the call (row stride and two batch strides).
struct OutArg {
    float* C;
    int64_t ldc, sCb, sCb2;
    int M, N, inner;
    int contiguous;
};

// Adds the split-K partials in split order: C = ((P0 + P1) + P2) + ... (+ bias[column] last; then the
// PAM product with post_scale, if asked for).  W consecutive outputs per thread, 4 or 1 (see the launch).  The
// partials of a launch sit in L2 and the pass, which is set up behind the product (512x512x1024 32.8 -> 29.6 us, 4096x512x512 83.3 -> 80.0), is bound by its loads: by their bytes for large outputs, where
// four at a time are faster (2048x2048 of 4 ranges 20.2 -> 12.0 us, 512x512 of 16 4.3 -> 3.7 us), by their latency
// for small ones, which need every thread.
template <int W>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* part, const OutArg o,
                                                            int64_t count, int splits,
                                                            const float* __restrict__ bias, int post,
                                                            float post_scale, int32_t off) {
    struct Pack { float f[W]; };
    auto read = [&](int64_t at) {
        Pack v;
        if constexpr (W == 4) {
            const float4 q = __ldcg(reinterpret_cast<const float4*>(part + at));
            v.f[0] = q.x; v.f[1] = q.y; v.f[2] = q.z; v.f[3] = q.w;
        } else {
            v.f[0] = __ldcg(part + at);
        }
        return v;
    };
    after_previous();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x * W;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * W; i < count; i += stride) {
        Pack v = read(i);
        for (int s = 1; s < splits; ++s) {
            const Pack u = read((int64_t)s * count + i);
#pragma unroll
            for (int c = 0; c < W; ++c) v.f[c] = fadd(v.f[c], u.f[c]);
        }
        const int64_t r = bias != nullptr || !o.contiguous ? i / o.N : 0;
        const int col = (int)(i - r * o.N);
        if (bias != nullptr) {
#pragma unroll
            for (int c = 0; c < W; ++c) v.f[c] = fadd(v.f[c], __ldg(bias + col + c));
        }
        if (post) {
#pragma unroll
            for (int c = 0; c < W; ++c) v.f[c] = mul(v.f[c], post_scale, off);
        }
        float* to = o.C + i;
        if (!o.contiguous) {
            const int64_t z = r / o.M;
            const int row = (int)(r - z * o.M);
            const int64_t zo = z / o.inner;
            to = o.C + zo * o.sCb + (z - zo * o.inner) * o.sCb2 + (int64_t)row * o.ldc + col;
        }
        if constexpr (W == 4) *reinterpret_cast<float4*>(to) = make_float4(v.f[0], v.f[1], v.f[2], v.f[3]);
        else *to = v.f[0];
    }
}

// ---- small products in ranges of K, in one launch ---------------------------------------------------------------------------
// The 32x32 tile's products in ranges are latencies: a launch that forms the partials, one that adds them, and the host's
// work for both.  Here one CTA forms all partials of a 16x16 tile, half a warp per range, and adds them from shared
// memory: same ranges, same order, same bits.  A call of 32x512x512 through the operators 11.6 and 8.8 us, most of it the host; kernel
// times, two launches and one:
//                               clean          half zeros in A   0.1 / 1 % specials
//   32x512x512 in 16 ranges     6.8 and 5.4    7.3 and 6.8        8.1 / 9.5 and 6.7 / 8.9
//   8x1024x512                  6.8 and 5.3    8.3 and 6.7        7.4 / 8.8 and 5.9 / 7.5
//   100x300x700 in 15           9.3 and 7.4   11.5 and 9.3       10.7 / 14.0 and 9.5 / 12.1
// Bound by latencies: the launch, two loads from the L2, the sum of the partials.  (A cluster of eight CTAs per tile with the partials in
// distributed shared memory: 6.9 us for the first.)
struct TileRange : Tile<16, 16, 16, 1, 4> {};
struct RangeShared {                                          // of one range
    union {
        struct { float a[TileRange::BK * row_stride(16)], b[TileRange::BK * row_stride(16)]; };
        float partial[16 * 16];
    };
};
constexpr int kMaxRanges = 16;                                // 256 threads: two CTAs per SM, 40 KB of shared memory each

// Whether a product planned as ranges on the 32x32 tile takes this form: no more ranges than above (197x192x768 in 24 ranges 9.3 us in two
// launches, 13.3 in one; 32x512x1024 in 32 7.8 and 9.2), at most three slabs each, which half a warp goes through one after the
// other, and no more warps than the SMs hold: 12 of 160 registers, 16 where the ranges are short.  Beyond that, clean operands, two
// launches and one: 12 products 17x1000x512 in 3 ranges of 11 slabs 24.6 and 42.8 us, 100x64x700 in 11 (18 warps) 12.9 and 20.0,
// 50x64x700 in 15 (16 warps, 3 slabs) 9.5 and 13.3.  At the edge: 100x512x512 in 16 (16 warps) 8.8 and 8.6, 4 products 16x1000x512 in 11 (12)
// 11.8 and 8.9.  Three slabs of a few tiles take longer by themselves (17x32x700 6.2 and 7.1), but less than the second launch
// costs the host.
int range_warps_per_sm(int64_t batch, int64_t M, int64_t N, int splits) {
    const int64_t ctas = batch * ((M + 15) / 16) * ((N + 15) / 16), per_sm = (ctas + sm_count() - 1) / sm_count();
    return (int)std::min<int64_t>(per_sm * ((splits + 1) / 2), 1 << 20);
}
constexpr int kWarpsOfAny = 12;                               // what the registers of every layout's kernel allow (see its launch bounds)

bool ranges_in_one_launch(int64_t batch, int64_t M, int64_t N, int64_t K, int splits) {
    if (splits <= 1 || splits > kMaxRanges || batch > 65535 || M > (int64_t)65535 * 16) return false;
    const int64_t slabs = (K + TileRange::BK - 1) / TileRange::BK, per_range = (slabs + splits - 1) / splits;
    return per_range <= 3 && range_warps_per_sm(batch, M, N, splits) <= (per_range < 3 ? 16 : kWarpsOfAny);
}

template <bool A_KC, bool B_KC, bool VEC, int PER_SM = 1>
__global__ void __launch_bounds__(PER_SM > 1 ? 16 * kMaxRanges : 32 * kWarpsOfAny, PER_SM) ranges_kernel(const GemmParams p) {
    using T = TileRange;
    constexpr int BK = T::BK;
    static_assert(T::kThreads == 16 && T::kTasksA == 4, "half a warp per range");
    extern __shared__ __align__(16) unsigned char range_bytes[];
    RangeShared* ranges = reinterpret_cast<RangeShared*>(range_bytes);
    const int range = threadIdx.x / 16, tid = threadIdx.x % 16, z = blockIdx.z;
    const unsigned half = 0xffffu << (threadIdx.x & 16);
    const int m0 = blockIdx.y * 16, n0 = blockIdx.x * 16, tx = tid % 4, ty = tid / 4;
    RangeShared& sh = ranges[range];
    const unsigned zo = __umulhi((unsigned)z, p.inner_magic);
    const float* Ab = p.A.p + (int64_t)zo * p.A.sb + (int64_t)z * p.A.sb2;
    const float* Bb = p.B.p + (int64_t)zo * p.B.sb + (int64_t)z * p.B.sb2;
    const int k_begin = range * p.k_chunk, k_end = min(p.K, k_begin + p.k_chunk);
    float acc[4][4] = {};
    // two slabs on their way: a range is seldom longer, and each wait is one for the L2
    float ra[2][T::kTasksA * 4], rb[2][T::kTasksB * 4];
    SlabWalker<T, 16, T::kTasksA, A_KC> walk_a;
    SlabWalker<T, 16, T::kTasksB, B_KC> walk_b;
    if constexpr (VEC) {
        walk_a.template init<false>(p.A, Ab, m0, p.M, k_begin, tid);
        walk_b.template init<false>(p.B, Bb, n0, p.N, k_begin, tid);
    }
    auto load = [&](float (&a)[T::kTasksA * 4], float (&b)[T::kTasksB * 4], int k0) {
        if (k0 >= k_end) return;
        if constexpr (VEC) {
            walk_a.load(a, k0, k_end, tid);
            walk_b.load(b, k0, k_end, tid);
        } else {
            load_slab<T, 16, T::kTasksA, A_KC>(a, p.A, Ab, m0, p.M, k0, k_end, tid);
            load_slab<T, 16, T::kTasksB, B_KC>(b, p.B, Bb, n0, p.N, k0, k_end, tid);
        }
    };
    // (the two ranges of a warp take the same loops, where both have a slab left: apart they would run one after the other)
    const int other_begin = (range ^ 1) * p.k_chunk, other_end = (range ^ 1) < p.splits ? min(p.K, other_begin + p.k_chunk) : other_begin;
    auto slab = [&](float (&a_in)[T::kTasksA * 4], float (&b_in)[T::kTasksB * 4], int k0) {
        if (k0 >= k_end) return;
        const unsigned both = k0 - k_begin + other_begin < other_end ? 0xffffffffu : half;
        const bool out = band_excess(b_in, band_excess(a_in, 0u)) >= kBandSpan2;
        // The lines with out-of-band elements and of what sort these are, as the slab's word of gemm_kernel: by the threads that hold
        // them, or, where registers are short, by a thread per line after the slab is stored.
        const bool dirty = __any_sync(both, out);
        unsigned f = 0;
        if (dirty) {
            if constexpr (PER_SM == 1) {
                uint32_t bits = 0, top = 0;
                f = dirty_lines<T, 16, T::kTasksA, A_KC>(a_in, tid, bits, top) | dirty_lines<T, 16, T::kTasksB, B_KC>(b_in, tid, bits, top);
                f |= (bits ? (unsigned)kNonZero : 0u) | (top >= kBandHi2 ? (unsigned)kAbove : 0u);
                f = __reduce_or_sync(both, f);
            }
#pragma unroll
            for (int c = 0; c < T::kTasksA * 4; ++c) a_in[c] = fadd(a_in[c], 0.0f);          // (one pattern for A's zeros)
        }
#pragma unroll
        for (int c = 0; c < T::kTasksA * 4; ++c) a_in[c] = i2f(isub(f2i(a_in[c]), p.bias_sub));
        __syncwarp(half);                                     // the last slab has been read
        store_slab<T, 16, T::kTasksA, A_KC>(sh.a, a_in, tid);
        store_slab<T, 16, T::kTasksB, B_KC>(sh.b, b_in, tid);
        load(a_in, b_in, k0 + 2 * BK);
        __syncwarp(half);
        if (PER_SM > 1 && dirty) {
            uint32_t bits = 0, top = 0;
            bool off = false;
            auto see = [&](int x) {
                const uint32_t m2 = 2u * (uint32_t)x;
                if (m2 - kBandLo2 >= kBandSpan2) { off = true; bits |= m2; }
                top = max(top, m2);
            };
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {
                const int4 va = *reinterpret_cast<const int4*>(sh.a + tid * row_stride(16) + q * 4);
                const int4 vb = *reinterpret_cast<const int4*>(sh.b + tid * row_stride(16) + q * 4);
                see(iadd(va.x, p.bias_sub)); see(iadd(va.y, p.bias_sub)); see(iadd(va.z, p.bias_sub)); see(iadd(va.w, p.bias_sub));
                see(vb.x); see(vb.y); see(vb.z); see(vb.w);
            }
            f = __ballot_sync(both, off);
            f = (f | f >> 16) & 0xffffu;                      // (bits of absent threads are zero)
            if (__any_sync(both, bits != 0)) f |= kNonZero;
            if (__any_sync(both, top >= kBandHi2)) f |= kAbove;
        }
#define PAMK_RANGE_FRAGMENTS(kk)                                                                     \
        const int4 a4 = *reinterpret_cast<const int4*>(sh.a + (kk) * row_stride(16) + ty * 4);       \
        const int4 b4 = *reinterpret_cast<const int4*>(sh.b + (kk) * row_stride(16) + tx * 4);       \
        const int a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
        auto plain_line = [&](int kk) {
            PAMK_RANGE_FRAGMENTS(kk)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fadd(acc[i][j], i2f(iadd(a[i], b[j])));
        };
        auto checked_line = [&](int kk, auto full_rule) {
            PAMK_RANGE_FRAGMENTS(kk)
            float araw[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) araw[i] = i2f(iadd(a[i], p.bias_sub));
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float mag = fabsf(fmul(araw[i], i2f(b[j])));
                    if constexpr (decltype(full_rule)::value) {
                        const float prod = mag <= i2f(kPassBits) ? i2f(iadd(a[i], b[j])) : quiet_nan();
                        if (!(mag <= i2f(kFlushBits))) acc[i][j] = fadd(acc[i][j], prod);
                    } else {
                        if (mag > i2f(kFlushBits)) acc[i][j] = fadd(acc[i][j], i2f(iadd(a[i], b[j])));
                    }
                }
        };
        auto zeros_line = [&](int kk) {                       // rows by weights, columns by predicates, as in gemm_kernel
            PAMK_RANGE_FRAGMENTS(kk)
            float w[4];
            int ai[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool zero = a[i] == -p.bias_sub;
                w[i] = zero ? 0.0f : 1.0f;
                ai[i] = zero ? 0 : a[i];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool on = 2u * (uint32_t)b[j] != 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (on) acc[i][j] = __fmaf_rn(i2f(iadd(ai[i], b[j])), w[i], acc[i][j]);
            }
        };
        // Zeros alone: all lines by weights.  Anything else: a few dirty lines one by one, many with the whole slab.  (The full rule for
        // every line of a dirty slab: 32x512x512 with half zeros 9.4 us, 0.1 % specials 10.9.)
        if (f == 0) {
#pragma unroll 4
            for (int kk = 0; kk < BK; ++kk) plain_line(kk);
        } else if (!(f & kNonZero)) {
#pragma unroll 4
            for (int kk = 0; kk < BK; ++kk) zeros_line(kk);
        } else if (__popc(f & 0xffffu) > 5) {
            if (f & kAbove) {
#pragma unroll 2
                for (int kk = 0; kk < BK; ++kk) checked_line(kk, std::true_type{});
            } else {                                          // "flush or add", exact for clean lines too
#pragma unroll 2
                for (int kk = 0; kk < BK; ++kk) checked_line(kk, std::false_type{});
            }
        } else {
            int kk = 0;
            while (kk < BK) {
                const unsigned left = (f & 0xffffu) >> kk;
                const int end = left ? kk + __ffs((int)left) - 1 : BK;
#pragma unroll 1
                for (; kk < end; ++kk) plain_line(kk);
                if (kk == BK) break;
                if (f & kAbove) checked_line(kk, std::true_type{});
                else checked_line(kk, std::false_type{});
                ++kk;
            }
        }
#undef PAMK_RANGE_FRAGMENTS
    };
    load(ra[0], rb[0], k_begin);
    load(ra[1], rb[1], k_begin + BK);
    for (int k0 = k_begin; k0 < k_end; k0 += 2 * BK) {
        slab(ra[0], rb[0], k0);
        slab(ra[1], rb[1], k0 + BK);
    }
    __syncwarp(half);                                         // the partial takes the slab's place
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(sh.partial + (ty * 4 + i) * 16 + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();

    float* Cz = p.C + (int64_t)zo * p.sCb + (int64_t)z * p.sCb2;
    for (int o = threadIdx.x; o < 16 * 16; o += blockDim.x) {
        const int row = m0 + o / 16, col = n0 + o % 16;
        if (row >= p.M || col >= p.N) continue;
        float v = ranges[0].partial[o];
        for (int r = 1; r < p.splits; ++r) v = fadd(v, ranges[r].partial[o]);
        if (p.bias != nullptr) v = fadd(v, __ldg(p.bias + col));
        if (p.post) v = mul(v, p.post_scale, p.off);
        Cz[(int64_t)row * p.ldc + col] = v;
    }
}

template <bool VEC>
int dispatch_ranges(const GemmParams& p, bool a_kc, bool b_kc, cudaStream_t st) {
    const dim3 grid((unsigned)((p.N + 15) / 16), (unsigned)((p.M + 15) / 16), (unsigned)p.batch);
    auto kernel = a_kc ? (b_kc ? ranges_kernel<true, true, VEC> : ranges_kernel<true, false, VEC>)
                       : (b_kc ? ranges_kernel<false, true, VEC> : ranges_kernel<false, false, VEC>);
    // (linear layers: in 128 registers, two CTAs of 16 ranges share an SM, 100x512x512 9.7 -> 8.6 us; 32x512x512, which fits as it is, 5.4 -> 6.3)
    if constexpr (VEC) {
        if (a_kc && b_kc && range_warps_per_sm(p.batch, p.M, p.N, p.splits) > kWarpsOfAny) kernel = ranges_kernel<true, true, true, 2>;
    }
    const size_t shared = p.splits * sizeof(RangeShared);
    static_assert(kMaxRanges * sizeof(RangeShared) <= 48 * 1024, "what a launch may use unasked");
    kernel<<<grid, (unsigned)(16 * p.splits), shared, st>>>(p);
    return check_launch();
}

// Launches a product's kernel, behind the kernel before it (512x512x1024 29.8 -> 27.6 us with its reduction, 12608x768x192 131.2 -> 129.7) where
// some SM gets as many of its CTAs as it holds anyway.  A launch of fewer would gather on the SMs that have room first: the 591 tiles
// of a product of 12608x192 are four per SM when all are free.
template <class T>
int launch_tiles(void (*kernel)(const GemmParams), const GemmParams& p, dim3 grid, int ctas_per_sm, cudaStream_t st) {
    const int64_t ctas = (int64_t)grid.x * grid.y * grid.z, sms = sm_count();
    if ((ctas + sms - 1) / sms >= ctas_per_sm) return launch_behind(kernel, grid, T::kThreads, st, p);
    kernel<<<grid, T::kThreads, 0, st>>>(p);
    return check_launch();
}

template <int MODE, class T>
int dispatch(const GemmParams& p, bool a_kc, bool b_kc, bool vec, dim3 grid, cudaStream_t st) {
    constexpr int kPerSm = MODE == kPam || MODE == kStd ? T::kCtasPerSm : T::kCtasPerSm / 2;
#define PAMK_LAUNCH(AK, BKC, V) return launch_tiles<T>(gemm_kernel<MODE, T, AK, BKC, V>, p, grid, kPerSm, st)
    if (vec) {
        if (a_kc) { if (b_kc) PAMK_LAUNCH(true, true, true); else PAMK_LAUNCH(true, false, true); }
        else      { if (b_kc) PAMK_LAUNCH(false, true, true); else PAMK_LAUNCH(false, false, true); }
    } else {
        if (a_kc) { if (b_kc) PAMK_LAUNCH(true, true, false); else PAMK_LAUNCH(true, false, false); }
        else      { if (b_kc) PAMK_LAUNCH(false, true, false); else PAMK_LAUNCH(false, false, false); }
    }
#undef PAMK_LAUNCH
}

// (with fewer rows per thread there are no 128-bit loads along A's rows, and of the large tile only 128-bit loads)
template <class T>
int dispatch_rows(const GemmParams& p, bool b_kc, dim3 grid, cudaStream_t st) {
    if (b_kc) return launch_tiles<T>(gemm_kernel<kPam, T, true, true, true>, p, grid, T::kCtasPerSm, st);
    else return launch_tiles<T>(gemm_kernel<kPam, T, true, false, true>, p, grid, T::kCtasPerSm, st);
}

template <class T>
int dispatch_rows_scalar(const GemmParams& p, bool a_kc, bool b_kc, dim3 grid, cudaStream_t st) {
    if (a_kc && b_kc) return launch_tiles<T>(gemm_kernel<kPam, T, true, true, false>, p, grid, T::kCtasPerSm, st);
    else if (a_kc) return launch_tiles<T>(gemm_kernel<kPam, T, true, false, false>, p, grid, T::kCtasPerSm, st);
    else if (b_kc) return launch_tiles<T>(gemm_kernel<kPam, T, false, true, false>, p, grid, T::kCtasPerSm, st);
    else return launch_tiles<T>(gemm_kernel<kPam, T, false, false, false>, p, grid, T::kCtasPerSm, st);
}

// An operand can use 128-bit loads when its base and both non-unit strides keep every group of
// four elements 16-byte aligned and its contiguous extent is a multiple of four.
bool vectorisable(const MatArg& m, bool kc, int rows, int K) {
    if (!aligned16(m.p) || (m.sb & 3) || (m.sb2 & 3)) return false;   // (either form of the batch strides)
    return kc ? ((m.sr & 3) == 0 && (K & 3) == 0) : ((m.sk & 3) == 0 && (rows & 3) == 0);
}

// ---- planning: tile shape and split-K ---------------------------------------------------------------
// The kernel is issue-bound, so the time of a launch is (the largest number of tiles any SM ends up
// with) x (work per tile), inflated when an SM holds too few warps to keep its schedulers busy,
// which is also the state of the SMs that run the last, partly filled wave of a larger launch.
enum TileKind { kTileLarge = 0, kTileSmall = 1, kTileTiny = 2, kTileLarge7 = 3, kTileSmall7 = 4 };

struct Plan {
    int tile;        // TileKind
    int splits;
    double cost;
};

template <class T>
Plan plan_for(int mode, int64_t batch, int64_t M, int64_t N, int64_t K, int split_request) {
    // the exact-gradient kernels hold a second 8x8 block of per-output constants in registers, so
    // half as many of their CTAs fit on an SM
    const int ctas_per_sm = mode == kBwdL || mode == kBwdR ? T::kCtasPerSm / 2 : T::kCtasPerSm;
    const int64_t sms = sm_count();
    const int64_t tiles = batch * ((M + T::kRows - 1) / T::kRows) * ((N + T::BN - 1) / T::BN);
    const int64_t slabs = (K + T::BK - 1) / T::BK;
    const int64_t slots = sms * ctas_per_sm;
    // cost of cutting K into s ranges, in multiply-accumulates per SM at full issue rate
    auto cost_of = [&](int64_t s, int64_t* actual) {
        if (s > slabs) s = slabs;
        const int64_t chunk_slabs = (slabs + s - 1) / s;
        s = (slabs + chunk_slabs - 1) / chunk_slabs;         // drop ranges that would be empty
        *actual = s;
        // measured: 16 resident warps per SM saturate the issue slots, 14 reach about 86 % of that,
        // 8 about 74 %
        auto util = [](int64_t ctas) {
            const double warps = (double)ctas * (T::kThreads / 32);
            if (T::BM >= 128 && T::MR < T::MT && warps >= 8.0) return warps >= 16.0 ? 1.0 : 0.94;      // (one 256-thread CTA: 2.75 us a slab, two: 5.23)
            return warps >= 16.0 ? 1.0 : (warps >= 8.0 ? 0.58 + 0.02 * warps : warps / 10.8);
        };
        // the smaller the tile, the more bytes are staged (and fragments loaded) per MAC
        const double staging = T::BM >= 128 ? 1.0 : (T::BM >= 64 ? 1.06 : 1.25);
        // every CTA also pays a prologue (first loads exposed) and an epilogue worth about 16 k-steps
        const double per_cta = (double)T::kRows * T::BN * ((double)(chunk_slabs * T::BK) + 16.0);
        const int64_t ctas = tiles * s;
        // CTAs spread evenly over the SMs ...
        const int64_t per_sm = (ctas + sms - 1) / sms;
        double cost = (double)per_sm * per_cta / util(per_sm < ctas_per_sm ? per_sm : ctas_per_sm);
        // ... and CTAs that run as full waves over all slots plus a last, partly filled one whose SMs
        // hold few warps.  The hardware refills slots one by one, which lies between the two: a sweep
        // of tile x split over products of 1 to 9 waves fits 0.62 / 0.38 (a vocabulary-sized weight
        // gradient of 1.07 waves loses 24 % to its tail without a split).
        const int64_t full = ctas / slots, rest = (ctas - full * slots + sms - 1) / sms;
        if (full >= 1) {
            const double waves = (double)(full * ctas_per_sm) * per_cta / util(ctas_per_sm) + (rest ? (double)rest * per_cta / util(rest) : 0.0);
            cost = 0.62 * cost + 0.38 * waves;
        }
        return cost * staging + (s > 1 ? 1.1e6 : 0.0);        // the reduction pass and its launch (~12 us)
    };
    Plan pl;
    pl.tile = T::MR < T::MT ? (T::BM >= 128 ? kTileLarge7 : kTileSmall7) : (T::BM >= 128 ? kTileLarge : (T::BM >= 64 ? kTileSmall : kTileTiny));
    int64_t s = split_request > 0 ? split_request : 1, actual = 1;
    pl.cost = cost_of(s, &actual);
    pl.splits = (int)actual;
    if (split_request == 0 && tiles < 8 * slots && slabs * T::BK >= 64) {  // automatic: fill the SMs, shorten the tail
        int64_t limit = 8 * slots / tiles;                   // up to eight full waves of CTAs
        if (limit < 2) limit = 2;
        const int64_t per_range = T::BM >= 64 ? 4 : 2;       // keep at least four slabs per range, two of the 32x32 tile's
        if (limit > slabs / per_range) limit = slabs / per_range;
        if (limit > 64) limit = 64;
        // a fixed ladder plus the splits that fill exactly one and two waves
        const int64_t ladder[] = {2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, slots / tiles, 2 * slots / tiles};
        for (int64_t cand : ladder) {
            if (cand < 2 || cand > limit) continue;
            int64_t got = 1;
            const double c = cost_of(cand, &got);
            // a split has to promise 5 % before it replaces the unsplit product (which also keeps
            // the reference's summation order)
            if (c < (pl.splits == 1 ? 0.95 * pl.cost : pl.cost)) { pl.cost = c; pl.splits = (int)got; }
        }
    }
    return pl;
}

// Whether an unsplit launch of `ctas` 32x32 tiles takes slabs of 8 (see TileTinyFine).
bool fine_slabs(int64_t ctas, int64_t K) {
    const int64_t tail = K % TileTiny::BK;
    return ctas > 4 * (int64_t)sm_count() && tail > 0 && tail <= TileTinyFine::BK;
}

// 0: choose by cost; 1: always the large tile; 2: the 64x64 tile wherever it exists; 3: the 32x32
// tile wherever it exists (PAM products), else the 64x64 tile; 4: the large tile, with seven rows per thread wherever
// that exists.
int g_tile_policy = 0;

Plan search_plan(int mode, int64_t batch, int64_t M, int64_t N, int64_t K, int split_request) {
    const Plan large = plan_for<TileLarge>(mode, batch, M, N, K, split_request);
    if (mode == kStd || g_tile_policy == 1) return large;    // the true-multiply product uses the large tile
    if (g_tile_policy == 4) return large;
    const Plan small = plan_for<TileSmall>(mode, batch, M, N, K, split_request);
    if (g_tile_policy == 2 || g_tile_policy == 5 || (g_tile_policy == 3 && mode != kPam)) return small;
    Plan best = small.cost < large.cost ? small : large;
    // The 32x32 tile wins where the 64x64 tile pads much (192 x 197x197x64: 256x256 against 224x224
    // outputs) or leaves most SMs empty.  Its modelled cost has to be lower by a margin that sweeps of
    // tile x split fitted: 10 % for launches of at least two waves of 64x64 tiles, where only throughput
    // counts (120 products: median -12 %, worst +6 %), and for matrices no larger than one tile in a
    // dimension; 20 % for smaller launches, where the model overrates the tile (106 products with that
    // margin: median -22 %, one slower, by 0.3 %; of 34 with 10 to 20 %, 13 were slower).
    if (mode == kPam) {
        const int64_t small_tiles = batch * ((M + TileSmall::BM - 1) / TileSmall::BM) * ((N + TileSmall::BN - 1) / TileSmall::BN);
        const bool throughput_bound = small_tiles >= 2 * (int64_t)sm_count() * TileSmall::kCtasPerSm;
        const double margin = throughput_bound || M <= TileTiny::BM || N <= TileTiny::BN ? 0.9 : 0.8;
        Plan tiny = plan_for<TileTiny>(mode, batch, M, N, K, split_request);
        // (slabs of 8 are a form of the unsplit launch: planned with the work that they leave, 363 products 47x65x17 stay
        // on this tile; taken for two slabs of 16 each, they went to the 64x64 tile, 18.5 -> 26.8 us)
        if (split_request <= 1 && fine_slabs(batch * ((M + TileTiny::BM - 1) / TileTiny::BM) * ((N + TileTiny::BN - 1) / TileTiny::BN), K)) {
            const Plan fine = plan_for<TileTinyFine>(mode, batch, M, N, K, 1);
            if (fine.cost < tiny.cost) tiny = fine;
        }
        if (g_tile_policy == 3 || tiny.cost < margin * best.cost) best = tiny;
    }
    return best;
}

// A thread's last automatic search and its last one for a given split are kept, functions of their arguments alone: a caller asks for
// the split and then calls the product with it, and a layer that is called again and again does not pay for the searches (0.6
// and 0.3 us on one host) each time.
Plan make_plan(int mode, int64_t batch, int64_t M, int64_t N, int64_t K, int split_request) {
    struct Search {
        std::array<int64_t, 8> key;
        Plan plan;
    };
    thread_local Search kept[2]{};                           // (all zero: the key of no search, which has at least one SM)
    Search& last = kept[split_request != 0];
    const std::array<int64_t, 8> key{mode, batch, M, N, K, split_request, g_tile_policy, sm_count()};
    if (last.key != key) last = {key, search_plan(mode, batch, M, N, K, split_request)};
    return last.plan;
}

// Whether a plain PAM product planned as `pl` takes TileLarge7 where its operands allow that.  The ranges of K, and with them the order of
// the sums, follow from the shape alone, not from how the operands lie in memory: unsplit products stay unsplit, and ranges keep their
// number and their bounds (both tiles have slabs of 16).
bool seven_rows_better(const Plan& pl, int64_t M, int64_t N, int64_t K) {
    if (pl.splits > 1 || (g_tile_policy != 0 && g_tile_policy != 4)) return false;
    if (M > (int64_t)65535 * TileLarge7::kRows) return false;                          // (grid.y)
    return g_tile_policy == 4 || plan_for<TileLarge7>(kPam, 1, M, N, K, 1).cost < 0.95 * pl.cost;
}

bool seven_rows_better_in_ranges(const Plan& pl, int64_t M, int64_t N, int64_t K) {
    if (pl.splits == 1 || pl.tile != kTileLarge || (g_tile_policy != 0 && g_tile_policy != 4)) return false;
    if (M > (int64_t)65535 * TileLarge7::kRows) return false;
    const Plan seven = plan_for<TileLarge7>(kPam, 1, M, N, K, pl.splits);
    return seven.splits == pl.splits && (g_tile_policy == 4 || seven.cost < 0.95 * pl.cost);
}

// Whether an unsplit PAM product planned for the 64x64 or the 32x32 tile takes TileSmall7 (the sums of one range are the same on any tile).
// By the model: 5 % cheaper; with scalar loads up to 15 % dearer than the 32x32 tile, whose cost with those it does not know, as long as the
// tiles cover at most a fifth more outputs.  Measured against the other tile, clean operands (1 % special values): 64x64, 26 products
// modelled 0.88 x 0.83 to 0.98 (0.80 to 0.95), 0.97 x and more 1.02 and up; 32x32, scalar loads, up to 1.2 x the outputs 0.85 to 0.99 (0.91
// to 1.11), 237 products 146x146x128, 1.26 x, 1.03 to 1.05 (1.09 to 1.11), 394 products 329x90x32, 1.27 x, 1.01 to 1.05 (1.15 to 1.18), modelled
// 1.18 x and more 0.97 to 1.15.
bool small7_better(const Plan& pl, int64_t batch, int64_t M, int64_t N, int64_t K, bool a_kc, bool vec) {
    if (pl.splits > 1 || (pl.tile != kTileSmall && pl.tile != kTileTiny) || (vec && !a_kc) || K == 0) return false;
    if (M > (int64_t)65535 * TileSmall7::kRows) return false;                          // (grid.y)
    if (g_tile_policy != 0) return g_tile_policy == 5;
    const bool lenient = !vec && pl.tile == kTileTiny;
    auto padded = [&](int64_t rows, int64_t cols) { return (M + rows - 1) / rows * rows * ((N + cols - 1) / cols * cols); };
    if (lenient && 5 * padded(TileSmall7::kRows, TileSmall7::BN) > 6 * padded(TileTiny::BM, TileTiny::BN)) return false;
    return plan_for<TileSmall7>(kPam, batch, M, N, K, 1).cost < (lenient ? 1.15 : 0.95) * pl.cost;
}

// Whether a PAM product planned as `pl` runs on packed operands, given the scratch, and its rows per tile then (whatever the operands'
// layout: packing brings them into one).
bool runs_packed(const Plan& pl, int64_t batch, int64_t M, int64_t N, int64_t K, int* tile_rows) {
    if (pl.tile != kTileLarge || K == 0 || !packing_pays(batch, M, N, K)) return false;
    const bool seven = batch == 1 && (seven_rows_better(pl, M, N, K) || seven_rows_better_in_ranges(pl, M, N, K));
    *tile_rows = seven ? TileLarge7::kRows : TileLarge::kRows;
    return true;
}

// Bytes of the partials of a product, a multiple of 256.
size_t partial_bytes(int splits, int64_t count) { return splits > 1 ? ((size_t)splits * (size_t)count * sizeof(float) + 255) / 256 * 256 : 0; }

bool workspace_ok(const void* ws, size_t bytes, int splits, int64_t count) {
    return ws != nullptr && (reinterpret_cast<uintptr_t>(ws) & 255u) == 0 &&
           bytes >= (size_t)splits * (size_t)count * sizeof(float);
}

int run(int mode, GemmParams p, bool a_kc, bool b_kc, int split_k, void* workspace, size_t workspace_bytes,
        cudaStream_t st) {
    if (p.M == 0 || p.N == 0 || p.batch == 0) return PAMK_OK;
    const int64_t count = (int64_t)p.batch * p.M * p.N;
    if (p.K == 0 && p.bias == nullptr && p.ldc == 0) {
        const cudaError_t e = cudaMemsetAsync(p.C, 0, count * sizeof(float), st);
        return e == cudaSuccess ? PAMK_OK : record_cuda_error(e);
    }
    if (split_k < 0) return PAMK_ERR_ARG;
    const bool vec = vectorisable(p.A, a_kc, p.M, p.K) && vectorisable(p.B, b_kc, p.N, p.K);
    Plan pl = p.K == 0 ? Plan{kTileSmall, 1, 0.0} : make_plan(mode, p.batch, p.M, p.N, p.K, split_k);   // K = 0: rows of bias
    if (pl.splits > 1 && !workspace_ok(workspace, workspace_bytes, pl.splits, count)) {
        if (split_k != 0) return PAMK_ERR_WORKSPACE;         // an explicit split needs its scratch
        pl = make_plan(mode, p.batch, p.M, p.N, p.K, 1);     // automatic: fall back to no split
    }
    // the M tiles ride on grid.y (at most 65535): a very tall product planned with a small tile moves to
    // the 128x128 tile, which reaches 8.3 M rows
    if (pl.tile != kTileLarge && (p.M + (pl.tile == kTileTiny ? TileTiny::BM : TileSmall::BM) - 1) /
                                         (pl.tile == kTileTiny ? TileTiny::BM : TileSmall::BM) > 65535) {
        const int splits = pl.splits;
        pl = plan_for<TileLarge>(mode, p.batch, p.M, p.N, p.K, splits);
    }
    int tile_rows = 0;
    PackLayout layout{};
    bool packed = mode == kPam && workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0 &&
                  runs_packed(pl, p.batch, p.M, p.N, p.K, &tile_rows);
    if (packed) {
        layout = pack_layout(p.batch, p.M, p.N, p.K, tile_rows);
        packed = workspace_bytes >= partial_bytes(pl.splits, count) && workspace_bytes - partial_bytes(pl.splits, count) >= layout.bytes;
    }
    if (!packed && mode == kPam && p.batch == 1 && p.K > 0 && a_kc && vec &&
        (seven_rows_better(pl, p.M, p.N, p.K) || seven_rows_better_in_ranges(pl, p.M, p.N, p.K)))
        pl.tile = kTileLarge7;
    if (mode == kPam && small7_better(pl, p.batch, p.M, p.N, p.K, a_kc, vec)) pl.tile = kTileSmall7;
    const int bm = packed ? tile_rows : pl.tile == kTileSmall7 ? TileSmall7::kRows : pl.tile == kTileTiny ? TileTiny::BM : (pl.tile == kTileSmall ? TileSmall::BM : (pl.tile == kTileLarge7 ? TileLarge7::kRows : TileLarge::BM));
    const int bn = pl.tile == kTileTiny ? TileTiny::BN : (pl.tile == kTileSmall || pl.tile == kTileSmall7 ? TileSmall::BN : TileLarge::BN);
    const int64_t ctas = ((p.N + bn - 1) / bn) * (int64_t)((p.M + bm - 1) / bm) * p.batch * pl.splits;
    const bool fine = pl.tile == kTileTiny && pl.splits == 1 && fine_slabs(ctas, p.K);
    const int bk = fine ? TileTinyFine::BK : pl.tile == kTileTiny ? TileTiny::BK : (pl.tile == kTileSmall || pl.tile == kTileSmall7 ? TileSmall::BK : TileLarge::BK);
    if (p.inner < 1) p.inner = 1;
    p.one = 1;
    p.least = INT32_MIN;
    if (p.ldc == 0) {                                        // plain output: [batch][M][N]
        p.ldc = p.N;
        p.sCb = (int64_t)p.inner * p.M * p.N;
        p.sCb2 = (int64_t)p.M * p.N;
    }
    OutArg out{p.C, p.ldc, p.sCb, p.sCb2, p.M, p.N, p.inner,
               p.ldc == p.N && p.sCb2 == (int64_t)p.M * p.N && p.sCb == (int64_t)p.inner * p.M * p.N};
    const bool one_launch = mode == kPam && pl.tile == kTileTiny && ranges_in_one_launch(p.batch, p.M, p.N, p.K, pl.splits);
    if (pl.splits > 1 && !one_launch) {                      // partials: [split][batch][M][N] in the scratch
        p.C = static_cast<float*>(workspace);
        p.ldc = p.N;
        p.sCb = (int64_t)p.inner * p.M * p.N;
        p.sCb2 = (int64_t)p.M * p.N;
        p.sCsplit = count;
    }
    // batch strides into the kernel's form (see MatArg)
    auto kernel_form = [&](int64_t& outer, int64_t& inner_stride) {
        if (p.inner == 1) { inner_stride = outer; outer = 0; }
        else outer -= (int64_t)p.inner * inner_stride;
    };
    kernel_form(p.A.sb, p.A.sb2);
    kernel_form(p.B.sb, p.B.sb2);
    kernel_form(p.sCb, p.sCb2);
    p.inner_magic = p.inner == 1 ? 0u : (unsigned)((uint64_t(1) << 32) / (uint64_t)p.inner) + 1u;
    const int slabs_total = (p.K + bk - 1) / bk;
    p.splits = pl.splits;
    p.k_chunk = ((slabs_total + pl.splits - 1) / pl.splits) * bk;

    const int64_t gx = (p.N + bn - 1) / bn, gy = (p.M + bm - 1) / bm, gz = (int64_t)p.batch * pl.splits;
    if (gy > 65535 || gz > 65535) return PAMK_ERR_SIZE;
    const dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)gz);
    int rc;
    switch (mode) {
        case kPam:
            rc = one_launch              ? (vec ? dispatch_ranges<true>(p, a_kc, b_kc, st) : dispatch_ranges<false>(p, a_kc, b_kc, st))
                 : packed                ? run_packed(p, layout, a_kc, b_kc, vectorisable(p.A, a_kc, p.M, p.K), vectorisable(p.B, b_kc, p.N, p.K),
                                                      static_cast<unsigned char*>(workspace) + partial_bytes(pl.splits, count), st)
                 : fine                  ? dispatch<kPam, TileTinyFine>(p, a_kc, b_kc, vec, grid, st)
                 : pl.tile == kTileTiny  ? dispatch<kPam, TileTiny>(p, a_kc, b_kc, vec, grid, st)
                 : pl.tile == kTileSmall ? dispatch<kPam, TileSmall>(p, a_kc, b_kc, vec, grid, st)
                 : pl.tile == kTileLarge7 ? dispatch_rows<TileLarge7>(p, b_kc, grid, st)
                 : pl.tile == kTileSmall7 ? (vec ? dispatch_rows<TileSmall7>(p, b_kc, grid, st) : dispatch_rows_scalar<TileSmall7>(p, a_kc, b_kc, grid, st))
                                         : dispatch<kPam, TileLarge>(p, a_kc, b_kc, vec, grid, st);
            break;
        case kStd: rc = dispatch<kStd, TileLarge>(p, a_kc, b_kc, vec, grid, st); break;
        case kBwdL:
            rc = pl.tile == kTileSmall ? dispatch<kBwdL, TileSmall>(p, a_kc, b_kc, vec, grid, st)
                                       : dispatch<kBwdL, TileLarge>(p, a_kc, b_kc, vec, grid, st);
            break;
        default:
            rc = pl.tile == kTileSmall ? dispatch<kBwdR, TileSmall>(p, a_kc, b_kc, vec, grid, st)
                                       : dispatch<kBwdR, TileLarge>(p, a_kc, b_kc, vec, grid, st);
            break;
    }
    if (rc != PAMK_OK || pl.splits == 1 || one_launch) return rc;
    // Four outputs per thread where there are enough of them (400x512 of 20 ranges 3.8 us with one, 4.1 with four; 192x192
    // of 64 ranges 4.9 and 7.4; for more see the kernel) and where N and the output's strides keep a group of
    // four in one row and 16-byte aligned.  (The partials are 256-byte aligned; count = batch * M * N is then a
    // multiple of 4 too.)
    const bool wide = count >= 1536 * (int64_t)sm_count() && ((out.N | out.ldc | out.sCb | out.sCb2) & 3) == 0 && aligned16(out.C);
    const int threads = wide ? 128 : 256;
    const int64_t blocks = (count / (wide ? 4 : 1) + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * (2048 / threads);
    const auto reduce = wide ? splitk_reduce_kernel<4> : splitk_reduce_kernel<1>;
    return launch_behind(reduce, dim3((unsigned)(blocks < cap ? blocks : cap)), (unsigned)threads, st, static_cast<const float*>(workspace), out,
                         count, pl.splits, p.bias, p.post, p.post_scale, p.off);
}

// Validates one operand and reports whether it is contiguous along k.
int operand_layout(const float* ptr, int64_t s_row, int64_t s_k, int rows, int K, bool* kc) {
    if (ptr == nullptr) return PAMK_ERR_ARG;
    if (s_k == 1 || K == 1) { *kc = true; return PAMK_OK; }
    if (s_row == 1 || rows == 1) { *kc = false; return PAMK_OK; }
    return PAMK_ERR_LAYOUT;
}

bool dims_ok(int64_t batch, int64_t M, int64_t N, int64_t K) {
    const int64_t lim = 0x7fffffff - 256;
    return batch >= 0 && M >= 0 && N >= 0 && K >= 0 && batch <= lim && M <= lim && N <= lim && K <= lim;
}

// ---- allocation-free split-K --------------------------------------------------------------------
// Scratch for pamk_matmul_static_scratch: lives in the library image, so every GPU that loads the
// library holds these 32 MiB from load until exit, and no allocation is ever needed for it.
constexpr size_t kStaticScratchFloats = size_t(8) << 20;
static __device__ __align__(256) float g_splitk_scratch[kStaticScratchFloats];

// In host code `g_splitk_scratch` is only a handle for the symbol; the device address has to be
// asked for, per device, with that device current.
constexpr int kMaxDevices = 64;
float* g_scratch_addr[kMaxDevices] = {};

int static_scratch(float** out) {
    int dev = -1;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return record_cuda_error(err);
    if (dev < 0 || dev >= kMaxDevices) return PAMK_ERR_SIZE;
    if (g_scratch_addr[dev] == nullptr) {
        void* ptr = nullptr;
        err = cudaGetSymbolAddress(&ptr, g_splitk_scratch);
        if (err != cudaSuccess) return record_cuda_error(err);
        g_scratch_addr[dev] = static_cast<float*>(ptr);
    }
    *out = g_scratch_addr[dev];
    return PAMK_OK;
}

}  // namespace
}  // namespace pamk

using namespace pamk;

extern "C" {

size_t pamk_matmul_workspace_bytes(int64_t batch, int64_t M, int64_t N, int split_k) {
    if (split_k <= 1 || batch <= 0 || M <= 0 || N <= 0) return 0;
    return (size_t)split_k * (size_t)batch * (size_t)M * (size_t)N * sizeof(float);
}

size_t pamk_matmul_scratch_bytes(int64_t batch, int64_t M, int64_t N, int64_t K, int split_k) {
    if (batch <= 0 || M <= 0 || N <= 0 || K <= 0 || split_k < 0 || !dims_ok(batch, M, N, K)) return 0;
    const Plan pl = make_plan(kPam, batch, M, N, K, split_k);
    const size_t partials = partial_bytes(pl.splits, batch * M * N);
    int tile_rows = 0;
    return partials + (runs_packed(pl, batch, M, N, K, &tile_rows) ? pack_layout(batch, M, N, K, tile_rows).bytes : 0);
}

int pamk_test_set_packing_policy(int policy) {
    if (policy < 0 || policy > 2) return PAMK_ERR_ARG;
    g_packing_policy = policy;
    return PAMK_OK;
}

int pamk_test_expired_waits(unsigned* count) {
    if (count == nullptr) return PAMK_ERR_ARG;
    const cudaError_t e = cudaMemcpyFromSymbol(count, g_expired_waits, sizeof(unsigned));
    return e == cudaSuccess ? PAMK_OK : record_cuda_error(e);
}

int pamk_test_run_out(unsigned ms, unsigned* out, void* stream) {
    if (ms > 1000 || out == nullptr) return PAMK_ERR_ARG;
    run_out_kernel<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(ms, out);
    return check_launch();
}

int pamk_test_set_tile_policy(int policy) {
    if (policy < 0 || policy > 5) return PAMK_ERR_ARG;
    g_tile_policy = policy;
    return PAMK_OK;
}

int pamk_test_planned_tile(int64_t batch, int64_t M, int64_t N, int64_t K) {
    if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return PAMK_ERR_ARG;
    const int tile = make_plan(kPam, batch, M, N, K, 0).tile;
    return tile == kTileLarge ? 128 : (tile == kTileSmall ? 64 : 32);
}

int pamk_test_planned_rows(int64_t M, int64_t N, int64_t K, int split_k) {
    if (M <= 0 || N <= 0 || K <= 0 || split_k < 0 || !dims_ok(1, M, N, K)) return PAMK_ERR_ARG;
    const Plan pl = make_plan(kPam, 1, M, N, K, split_k);
    if (seven_rows_better(pl, M, N, K)) return TileLarge7::kRows;
    return pl.tile == kTileLarge ? TileLarge::BM : (pl.tile == kTileSmall ? TileSmall::BM : TileTiny::BM);
}

int pamk_test_split_rows(int64_t M, int64_t N, int64_t K, int split_k) {
    if (M <= 0 || N <= 0 || K <= 0 || split_k < 0 || !dims_ok(1, M, N, K)) return PAMK_ERR_ARG;
    const Plan pl = make_plan(kPam, 1, M, N, K, split_k);
    return seven_rows_better_in_ranges(pl, M, N, K) ? TileLarge7::kRows : pamk_test_planned_rows(M, N, K, split_k);
}

int pamk_test_small_rows(int64_t batch, int64_t M, int64_t N, int64_t K, int a_along_k, int wide_loads) {
    if (batch <= 0 || M <= 0 || N <= 0 || K <= 0 || !dims_ok(batch, M, N, K)) return PAMK_ERR_ARG;
    const Plan pl = make_plan(kPam, batch, M, N, K, 1);
    if (small7_better(pl, batch, M, N, K, a_along_k != 0, wide_loads != 0)) return TileSmall7::kRows;
    return pl.tile == kTileLarge ? TileLarge::BM : (pl.tile == kTileSmall ? TileSmall::BM : TileTiny::BM);
}

int pamk_matmul_auto_split(int64_t batch, int64_t M, int64_t N, int64_t K) {
    if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return 1;
    return make_plan(kPam, batch, M, N, K, 0).splits;
}

int pamk_matmul_bwd_auto_split(int64_t batch, int64_t M, int64_t N, int64_t K) {
    if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return 1;
    return make_plan(kBwdL, batch, M, N, K, 0).splits;
}

int pamk_matmul_bias(int mul_kind, const float* A, const float* B, const float* bias, float* C,
                     int64_t batch, int64_t M, int64_t N, int64_t K,
                     int64_t sAb, int64_t sAm, int64_t sAk,
                     int64_t sBb, int64_t sBk, int64_t sBn,
                     float offset, int split_k, void* workspace, size_t workspace_bytes, void* stream) {
    if (mul_kind != PAMK_MUL_PAM && mul_kind != PAMK_MUL_STANDARD) return PAMK_ERR_ARG;
    if (!dims_ok(batch, M, N, K)) return batch < 0 || M < 0 || N < 0 || K < 0 ? PAMK_ERR_ARG : PAMK_ERR_SIZE;
    if (split_k < 0) return PAMK_ERR_ARG;
    if (batch == 0 || M == 0 || N == 0) return PAMK_OK;
    if (C == nullptr) return PAMK_ERR_ARG;
    GemmParams p{};
    bool a_kc = true, b_kc = true;
    if (K > 0) {
        int rc = operand_layout(A, sAm, sAk, (int)M, (int)K, &a_kc);
        if (rc != PAMK_OK) return rc;
        rc = operand_layout(B, sBn, sBk, (int)N, (int)K, &b_kc);
        if (rc != PAMK_OK) return rc;
    }
    p.A = {A, sAb, sAm, sAk};
    p.B = {B, sBb, sBn, sBk};
    p.C = C;
    p.bias = bias;
    p.M = (int)M; p.N = (int)N; p.K = (int)K; p.batch = (int)batch;
    p.off = offset_bits(offset);
    p.bias_sub = isub(kBias, p.off);
    return run(mul_kind == PAMK_MUL_PAM ? kPam : kStd, p, a_kc, b_kc, split_k, workspace, workspace_bytes,
               static_cast<cudaStream_t>(stream));
}

int pamk_matmul(int mul_kind, const float* A, const float* B, float* C,
                int64_t batch, int64_t M, int64_t N, int64_t K,
                int64_t sAb, int64_t sAm, int64_t sAk,
                int64_t sBb, int64_t sBk, int64_t sBn,
                float offset, int split_k, void* workspace, size_t workspace_bytes, void* stream) {
    return pamk_matmul_bias(mul_kind, A, B, nullptr, C, batch, M, N, K, sAb, sAm, sAk, sBb, sBk, sBn, offset, split_k,
                            workspace, workspace_bytes, stream);
}

int pamk_matmul_strided(const float* A, const float* B, float* C,
                        int64_t batch_outer, int64_t batch_inner, int64_t M, int64_t N, int64_t K,
                        int64_t sAo, int64_t sAi, int64_t sAm, int64_t sAk,
                        int64_t sBo, int64_t sBi, int64_t sBk, int64_t sBn,
                        int64_t sCo, int64_t sCi, int64_t sCm,
                        float offset, int has_post_scale, float post_scale,
                        int split_k, void* workspace, size_t workspace_bytes, void* stream) {
    if (batch_outer < 0 || batch_inner < 0) return PAMK_ERR_ARG;
    if (batch_inner > 0 && batch_outer > (0x7fffffff - 256) / batch_inner) return PAMK_ERR_SIZE;
    const int64_t batch = batch_outer * batch_inner;
    if (!dims_ok(batch, M, N, K)) return M < 0 || N < 0 || K < 0 ? PAMK_ERR_ARG : PAMK_ERR_SIZE;
    if (split_k < 0) return PAMK_ERR_ARG;
    if (batch == 0 || M == 0 || N == 0) return PAMK_OK;
    if (C == nullptr || sCm < N) return PAMK_ERR_ARG;
    GemmParams p{};
    bool a_kc = true, b_kc = true;
    if (K > 0) {
        int rc = operand_layout(A, sAm, sAk, (int)M, (int)K, &a_kc);
        if (rc != PAMK_OK) return rc;
        rc = operand_layout(B, sBn, sBk, (int)N, (int)K, &b_kc);
        if (rc != PAMK_OK) return rc;
    }
    p.A = {A, sAo, sAm, sAk, sAi};
    p.B = {B, sBo, sBn, sBk, sBi};
    p.C = C;
    p.ldc = sCm; p.sCb = sCo; p.sCb2 = sCi;
    p.inner = (int)batch_inner;
    p.post = has_post_scale != 0;
    p.post_scale = post_scale;
    p.M = (int)M; p.N = (int)N; p.K = (int)K; p.batch = (int)batch;
    p.off = offset_bits(offset);
    p.bias_sub = isub(kBias, p.off);
    return run(kPam, p, a_kc, b_kc, split_k, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

size_t pamk_matmul_static_scratch_bytes(void) { return kStaticScratchFloats * sizeof(float); }

int pamk_matmul_static_scratch(const float* A, const float* B, float* C,
                               int64_t batch, int64_t M, int64_t N, int64_t K,
                               int64_t sAb, int64_t sAm, int64_t sAk,
                               int64_t sBb, int64_t sBk, int64_t sBn,
                               float offset, int split_k, void* stream) {
    if (!dims_ok(batch, M, N, K)) return batch < 0 || M < 0 || N < 0 || K < 0 ? PAMK_ERR_ARG : PAMK_ERR_SIZE;
    if (split_k < 1) return PAMK_ERR_ARG;
    if (batch == 0 || M == 0 || N == 0) return PAMK_OK;
    if (C == nullptr) return PAMK_ERR_ARG;
    // every partial sum must fit in the fixed array
    if ((double)split_k * (double)batch * (double)M * (double)N > (double)kStaticScratchFloats) return PAMK_ERR_SIZE;
    GemmParams p{};
    bool a_kc = true, b_kc = true;
    if (K > 0) {
        int rc = operand_layout(A, sAm, sAk, (int)M, (int)K, &a_kc);
        if (rc != PAMK_OK) return rc;
        rc = operand_layout(B, sBn, sBk, (int)N, (int)K, &b_kc);
        if (rc != PAMK_OK) return rc;
    }
    float* scratch = nullptr;
    const int rc = static_scratch(&scratch);
    if (rc != PAMK_OK) return rc;
    p.A = {A, sAb, sAm, sAk};
    p.B = {B, sBb, sBn, sBk};
    p.C = C;
    p.M = (int)M; p.N = (int)N; p.K = (int)K; p.batch = (int)batch;
    p.off = offset_bits(offset);
    p.bias_sub = isub(kBias, p.off);
    return run(kPam, p, a_kc, b_kc, split_k, scratch, kStaticScratchFloats * sizeof(float),
               static_cast<cudaStream_t>(stream));
}

int pamk_matmul_bwd(const float* L, const float* R, const float* D, float* out,
                    int64_t batch, int64_t M, int64_t N, int64_t K,
                    int64_t sLb, int64_t sLm, int64_t sLk,
                    int64_t sRb, int64_t sRk, int64_t sRn,
                    int64_t sDb, int64_t sDm, int64_t sDn,
                    int delta_l, float offset, int split_k, void* workspace, size_t workspace_bytes, void* stream) {
    if (!dims_ok(batch, M, N, K)) return batch < 0 || M < 0 || N < 0 || K < 0 ? PAMK_ERR_ARG : PAMK_ERR_SIZE;
    if (split_k < 0) return PAMK_ERR_ARG;
    if (batch == 0 || M == 0 || N == 0) return PAMK_OK;
    if (out == nullptr || D == nullptr) return PAMK_ERR_ARG;
    GemmParams p{};
    bool l_kc = true, r_kc = true;
    if (K > 0) {
        int rc = operand_layout(L, sLm, sLk, (int)M, (int)K, &l_kc);
        if (rc != PAMK_OK) return rc;
        rc = operand_layout(R, sRn, sRk, (int)N, (int)K, &r_kc);
        if (rc != PAMK_OK) return rc;
    }
    p.A = {L, sLb, sLm, sLk};
    p.B = {R, sRb, sRn, sRk};
    p.D = D; p.sDb = sDb; p.sDm = sDm; p.sDn = sDn;
    p.C = out;
    p.M = (int)M; p.N = (int)N; p.K = (int)K; p.batch = (int)batch;
    p.off = offset_bits(offset);
    p.bias_sub = isub(kBias, p.off);
    return run(delta_l ? kBwdL : kBwdR, p, l_kc, r_kc, split_k, workspace, workspace_bytes,
               static_cast<cudaStream_t>(stream));
}

}
