// The large PAM products on packed operands.  Included by gemm.cu, whose definitions (MatArg, the band, class_of, kind_of, the
// pipes of the integer adds) it uses.
//
// A large product stages every element of A once per tile column and every element of B once per tile row, 64 times each at
// 8192^3, and the kernel in gemm.cu transposes, biases and tests it each time (12 % of its instructions on clean
// operands), looks through it for what the range rule needs on others (40 % of a clean slab), and stops all warps of a
// CTA at a barrier per slab, so that the one with the most lines to check holds up the rest.  Here a pass over the
// operands does that work once (pack_kernel, and for blocks with out-of-band elements classify_kernel), and leaves
// them in blocks of 16 k by 128 rows that a CTA fetches with one bulk copy each into a ring in shared
// memory; warps move through the ring on their own, up to three slabs apart.
// The sums are those of gemm.cu bit for bit: one thread per output, strictly in k order, the same ranges of K.
//   4096^3 (us)   clean  0.1 % zeros  0.1 / 1 / 3 / 10 % specials  half zeros in A / in both
//   in place      4375   6842         6765 / 9783 / 12558 / 15106  5534 / 7178
//   packed        4231   5246         5233 / 6152 /  8952 / 13525  5264 / 6691
// of which the passes take 68 (and 41 more where blocks have to be classified).  What bounds it: dispatch, 98 % on clean operands
// (a packed add counts as two); on others the instructions beside the products and the lines to check.

// One block: 16 k lines of 128 row slots.  A's patterns carry the bias, see gemm.cu.
struct PackBlock {
    float data[16][128];
    unsigned char off[16][16];      // per line and thread row / column: a bit for each of its eight elements that is masked
    unsigned char cls[16][4];       // per line and four thread rows / columns: the classes of their out-of-band elements
    unsigned flags[4];              // [0]: whether the block holds any; off and cls are written only then
};
static_assert(sizeof(PackBlock) % 16 == 0, "the bulk copy's unit");

struct PackArg {
    MatArg m;                       // element (r, k) as in gemm.cu
    PackBlock* out;                 // [batch][tiles][slabs]
    unsigned* extremes;             // per batch and k: ~(smallest magnitude in the band), largest not above it; 0 where there is none
    int32_t sub;                    // taken from every pattern: A's bias, 0 for B
    int rows, K, inner;
    unsigned inner_magic;
    int tiles, tile_rows, slabs;    // tile_rows: 128, or 112 (see slot_row)
    int kc, vec;
};

constexpr int kPackSlabs = 4;       // slabs that one CTA packs: 128 rows of 64 k

__device__ __forceinline__ int packed_row(int slot, int tile_rows) {
    return tile_rows == 128 ? slot : slot_row<TileLarge7, 128>(slot);
}

// Both operands in one launch, A's CTAs first.  An operand contiguous along K is read 256 bytes of a row at a time and transposed
// in shared memory, any other is read as it is written, line by line.  Bound by memory: 4096^3 61 us for 273 MB, 4.5 TB/s.
__global__ void __launch_bounds__(256) pack_kernel(const PackArg A, const PackArg B, int groups, int a_ctas) {
    __shared__ __align__(16) float stage[16 * kPackSlabs][row_stride(128)];
    __shared__ unsigned flags[kPackSlabs];
    const bool is_b = (int)blockIdx.x >= a_ctas;
    const PackArg& p = is_b ? B : A;
    const int id = is_b ? blockIdx.x - a_ctas : blockIdx.x;
    const int group = id % groups, rest = id / groups;
    const int tile = rest % p.tiles, z = rest / p.tiles;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* base = p.m.p + (int64_t)__umulhi((unsigned)z, p.inner_magic) * p.m.sb + (int64_t)z * p.m.sb2;
    const int k0 = group * 16 * kPackSlabs, row0 = tile * p.tile_rows;
    if (tid < kPackSlabs) flags[tid] = 0;
    if (p.kc) {
        const int c = (lane & 15) * 4, k = k0 + c;           // 16 lanes read one row
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int slot = (r * 8 + warp) * 2 + (lane >> 4);
            const int row = min(row0 + packed_row(slot, p.tile_rows), p.rows - 1);     // (rows beyond the matrix: copies, never stored)
            const float* src = base + (int64_t)row * p.m.sr + k;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p.vec) {
                if (k < p.K) v = __ldg(reinterpret_cast<const float4*>(src));
            } else {
                if (k < p.K) v.x = __ldg(src);
                if (k + 1 < p.K) v.y = __ldg(src + 1);
                if (k + 2 < p.K) v.z = __ldg(src + 2);
                if (k + 3 < p.K) v.w = __ldg(src + 3);
            }
            stage[c][slot] = v.x; stage[c + 1][slot] = v.y; stage[c + 2][slot] = v.z; stage[c + 3][slot] = v.w;
        }
    }
    __syncthreads();
    PackBlock* blocks = p.out + ((int64_t)z * p.tiles + tile) * p.slabs;
#pragma unroll 4
    for (int q = 0; q < 2 * kPackSlabs; ++q) {               // a warp's eight lines lie in one slab
        const int line = warp * 8 + q, k = k0 + line;
        if (k >= p.slabs * 16) break;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.kc) {
            v = *reinterpret_cast<const float4*>(&stage[line][lane * 4]);
        } else if (k < p.K) {
            const float* src = base + (int64_t)k * p.m.sk;
            const int first = row0 + lane * 4;
            if (p.vec && p.tile_rows == 128) {
                v = __ldg(reinterpret_cast<const float4*>(src + (first < p.rows ? first : p.rows - 4)));
            } else {
                int row[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) row[c] = min(row0 + packed_row(lane * 4 + c, p.tile_rows), p.rows - 1);
                v = make_float4(__ldg(src + row[0]), __ldg(src + row[1]), __ldg(src + row[2]), __ldg(src + row[3]));
            }
        }
        const int bits[4] = {f2i(v.x), f2i(v.y), f2i(v.z), f2i(v.w)};
        if (k < p.K) {                                       // (lines beyond K are zeros that nothing reads)
            uint32_t low = 0, high = 0;
            bool out = false;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t m = (uint32_t)bits[c] & 0x7fffffffu;
                const bool in = m - kBandLo < kBandHi - kBandLo;
                out |= !in;
                if (in) low = max(low, ~m);
                if (m < kBandHi) high = max(high, m);
            }
            low = __reduce_max_sync(0xffffffffu, low);
            high = __reduce_max_sync(0xffffffffu, high);
            const bool any = __any_sync(0xffffffffu, out);
            if (lane == 0) {
                unsigned* e = p.extremes + ((int64_t)z * p.slabs * 16 + k) * 2;
                if (low) atomicMax(e, low);
                if (high) atomicMax(e + 1, high);
                if (any) flags[warp >> 1] = 1u;
            }
        }
        *reinterpret_cast<int4*>(&blocks[k >> 4].data[k & 15][lane * 4]) =
            make_int4(isub(bits[0], p.sub), isub(bits[1], p.sub), isub(bits[2], p.sub), isub(bits[3], p.sub));
    }
    __syncthreads();
    if (tid < kPackSlabs && group * kPackSlabs + tid < p.slabs)
        *reinterpret_cast<uint4*>(blocks[group * kPackSlabs + tid].flags) = make_uint4(flags[tid], 0, 0, 0);
}

// The classes of the out-of-band elements (class_of), against the extremes of the partner's whole line: gemm.cu's look, once per
// element.  Blocks without any are passed over, 256 flags at a time.
__global__ void __launch_bounds__(256) classify_kernel(const PackArg A, const PackArg B, int64_t a_blocks, int64_t blocks) {
    __shared__ unsigned todo[8];
    const int tid = threadIdx.x, line = tid >> 4, at = tid & 15;         // sixteen threads share a line
    for (int64_t first = blockIdx.x; first < blocks; first += (int64_t)gridDim.x * 256) {
        const int64_t mine = first + (int64_t)tid * gridDim.x;
        bool dirty = false;
        if (mine < blocks) dirty = (mine < a_blocks ? A.out[mine] : B.out[mine - a_blocks]).flags[0] != 0;
        const unsigned vote = __ballot_sync(0xffffffffu, dirty);
        __syncthreads();                                     // (the last round's words have been read)
        if ((tid & 31) == 0) todo[tid >> 5] = vote;
        __syncthreads();
        for (int w = 0; w < 8; ++w)
            for (unsigned left = todo[w]; left != 0; left &= left - 1) {
                const int64_t id = first + (int64_t)(w * 32 + __ffs((int)left) - 1) * gridDim.x;
                const bool is_b = id >= a_blocks;
                const PackArg& p = is_b ? B : A;
                const int64_t n = is_b ? id - a_blocks : id;
                PackBlock& block = p.out[n];
                const int slab = (int)(n % p.slabs);
                const int64_t z = n / p.slabs / p.tiles;
                const unsigned* e = (is_b ? A : B).extremes + ((z * p.slabs + slab) * 16 + line) * 2;
                const unsigned low = __ldg(e), high = __ldg(e + 1);
                const float smallest = low ? i2f((int32_t)~low) : INFINITY, largest = i2f((int32_t)high);   // +0: all above the band
                unsigned off = 0, classes = 0;
                if (slab * 16 + line < p.K) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int4 v = *reinterpret_cast<const int4*>(&block.data[line][q * 64 + at * 4]);
                        const int x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint32_t m = (uint32_t)iadd(x[c], p.sub) & 0x7fffffffu;
                            if (m - kBandLo >= kBandHi - kBandLo) {
                                const unsigned k = class_of(m, smallest, largest);
                                off |= (k & kMasked) << (q * 4 + c);
                                classes |= k;
                            }
                        }
                    }
                }
                block.off[line][at] = (unsigned char)off;
                classes |= __shfl_xor_sync(0xffffffffu, classes, 1);
                classes |= __shfl_xor_sync(0xffffffffu, classes, 2);
                if (at % 4 == 0) block.cls[line][at / 4] = (unsigned char)classes;
            }
    }
}

struct PackedParams {
    const PackBlock *A, *B;
    float* C;
    int64_t ldc, sCb, sCb2, sCsplit;   // as in GemmParams
    const float* bias;
    int post;
    float post_scale;
    unsigned inner_magic;
    int M, N, K, splits, chunk_slabs, slabs, a_tiles, b_tiles;
    int32_t bias_sub, off, one, least;
};

// ---- the ring ---------------------------------------------------------------------------------------------------
// Six stages of one block of A and one of B, requested three slabs ahead: the stage that slab s + 3 goes to was slab s - 3's, so a
// warp may run three slabs ahead of the slowest one.  Two CTAs of 102 KB share an SM.
constexpr int kStages = 6, kAhead = 3;

__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void barrier_init(uint64_t* b, unsigned arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_address(b)), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void barrier_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(shared_address(b)) : "memory");
}

// Waits that ran out: how many CTAs met one on this device.  The outputs of such a CTA's warps are NaN.
__device__ unsigned g_expired_waits;

constexpr unsigned kWaitMs = 2000;          // (a slab takes microseconds; less than the clock's word below holds)

// (the clock's low word goes round every four seconds)
__device__ __forceinline__ unsigned clock_ns() {
    unsigned t;
    asm volatile("mov.u32 %0, %globaltimer_lo;" : "=r"(t));
    return t;
}
__device__ __forceinline__ bool barrier_done(uint64_t* b, unsigned parity) {
    unsigned done;
    asm volatile("{ .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n selp.u32 %0, 1, 0, q; }"
                 : "=r"(done) : "r"(shared_address(b)), "r"(parity) : "memory");
    return done != 0;
}

// A wait ends when `ms` have passed since its first tries failed, or when another wait of the CTA has ended so (`gave_up`, in shared
// memory; null: regardless of others), and then returns false.  A try sleeps for a time that the hardware chooses, so tries alone
// are no bound.  The first wait of a CTA to run out adds one to `expired`.
__device__ __forceinline__ bool barrier_wait(uint64_t* b, unsigned parity, unsigned* gave_up, unsigned* expired, unsigned ms = kWaitMs) {
    unsigned start = 0;
    for (int i = 0; i < (1 << 30); ++i) {
        if (barrier_done(b, parity)) return true;
        if (i < 64) continue;
        if (i == 64) start = clock_ns();
        if (gave_up != nullptr && *(volatile unsigned*)gave_up != 0) return false;
        if (clock_ns() - start > ms * 1000000u) break;
    }
    if (gave_up != nullptr && atomicExch(gave_up, 1u) == 0) atomicAdd(expired, 1u);
    return false;
}

// One block of each operand into a stage.
__device__ __forceinline__ void request_slab(PackBlock* stage, const PackBlock* a, const PackBlock* b, uint64_t* full) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(full)), "r"((unsigned)(2 * sizeof(PackBlock))) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(shared_address(stage)), "l"(a), "r"((unsigned)sizeof(PackBlock)), "r"(shared_address(full)) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(shared_address(stage + 1)), "l"(b), "r"((unsigned)sizeof(PackBlock)), "r"(shared_address(full)) : "memory");
}

struct Ring {
    PackBlock stages[kStages][2];
    uint64_t full[kStages], empty[kStages];
    unsigned gave_up;
};

// Test: eight warps at barriers that nothing arrives at, the first with a limit of `ms`, the others with the usual one.  out: what each
// warp's wait returned, the milliseconds until all had, and how many were counted.
__global__ void __launch_bounds__(256) run_out_kernel(unsigned ms, unsigned* out) {
    __shared__ uint64_t never[8];
    __shared__ unsigned gave_up, expired;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        gave_up = expired = 0;
        for (int i = 0; i < 8; ++i) barrier_init(never + i, 1);
    }
    const unsigned start = clock_ns();
    __syncthreads();
    const bool arrived = __any_sync(0xffffffffu, barrier_wait(never + warp, 0, &gave_up, &expired, warp == 0 ? ms : kWaitMs));
    if ((threadIdx.x & 31) == 0) out[warp] = arrived;
    __syncthreads();
    if (threadIdx.x == 0) {
        out[8] = (clock_ns() - start) / 1000000u;
        out[9] = expired;
    }
}

// MR rows per thread: 8, or 7 for tiles of 112 rows.  A warp is 4 x 8 threads, as in gemm.cu.
template <int MR>
__global__ void __launch_bounds__(256, 2) packed_kernel(const PackedParams p) {
    extern __shared__ __align__(128) unsigned char shared_bytes[];
    Ring& ring = *reinterpret_cast<Ring*>(shared_bytes);
    constexpr int MT = 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
    const int z = blockIdx.z / p.splits, sp = blockIdx.z - z * p.splits;
    const int s_begin = sp * p.chunk_slabs;
    const int count = min(p.slabs, s_begin + p.chunk_slabs) - s_begin;
    const PackBlock* a_src = p.A + ((int64_t)z * p.a_tiles + blockIdx.y) * p.slabs + s_begin;
    const PackBlock* b_src = p.B + ((int64_t)z * p.b_tiles + blockIdx.x) * p.slabs + s_begin;
    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) {
            barrier_init(ring.full + i, 1);
            barrier_init(ring.empty + i, 8);
        }
        ring.gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int s = 0; s < kAhead && s < count; ++s) request_slab(ring.stages[s], a_src + s, b_src + s, ring.full + s);
    }
    __syncthreads();

    float acc[MR][MT];
#pragma unroll
    for (int i = 0; i < MR; ++i)
#pragma unroll
        for (int j = 0; j < MT; ++j) acc[i][j] = 0.0f;

#define PAMK_FRAGMENTS(kk)                                                        \
        const int4 a0 = *reinterpret_cast<const int4*>(as + (kk) * 128 + ty * 4);      \
        const int4 a1 = *reinterpret_cast<const int4*>(as + (kk) * 128 + ty * 4 + 64); \
        const int4 b0 = *reinterpret_cast<const int4*>(bs + (kk) * 128 + tx * 4);      \
        const int4 b1 = *reinterpret_cast<const int4*>(bs + (kk) * 128 + tx * 4 + 64); \
        const int a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};             \
        const int b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};

    int stage = 0, parity = 0;                               // of the slab that is summed
    int ahead = kAhead, ahead_parity = 0;                    // of the slab that is requested
    int requested = min(kAhead, count), landed = 0;
    bool ok = true;
    for (int s = 0; s < count; ++s) {
        if (tid == 0 && s + kAhead < count) {
            if (s + kAhead >= kStages) ok = barrier_wait(ring.empty + ahead, ahead_parity ^ 1, &ring.gave_up, &g_expired_waits);
            if (ok) {
                request_slab(ring.stages[ahead], a_src + s + kAhead, b_src + s + kAhead, ring.full + ahead);
                ++requested;
            }
        }
        if (++ahead == kStages) { ahead = 0; ahead_parity ^= 1; }
        __syncwarp();
        ok = __all_sync(0xffffffffu, ok && barrier_wait(ring.full + stage, parity, &ring.gave_up, &g_expired_waits));
        if (!ok) break;
        ++landed;
        const PackBlock &block_a = ring.stages[stage][0], &block_b = ring.stages[stage][1];
        const float* as = &block_a.data[0][0];
        const float* bs = &block_b.data[0][0];
        const int lines = min(16, p.K - (s_begin + s) * 16);
        const bool dirty = (block_a.flags[0] | block_b.flags[0]) != 0;
        if (!dirty && lines == 16) {
#pragma unroll 8
            for (int kk = 0; kk < 16; ++kk) {
                PAMK_FRAGMENTS(kk)
#pragma unroll
                for (int i = 0; i < MR; ++i)
#pragma unroll
                    for (int j = 0; j < MT; j += 2) {
                        auto product = [&](int c) {
                            return multiply_add_product(i, c) ? sum_on_fma(a[i], b[c], p.one) : sum_on_alu(a[i], b[c], p.least);
                        };
                        add_pair(acc[i][j], acc[i][j + 1], product(j), product(j + 1));
                    }
            }
        } else {
            // Each line by the cheapest loop that this warp's rows and columns allow, in runs of one kind; lane k holds the kind of
            // line k.  Lines without out-of-band elements go with the masked columns: a loop of their own would serve runs of one or two.
            unsigned kind = kPlain;
            if (dirty && lane < lines) {
                const unsigned rows = block_a.flags[0] ? block_a.cls[lane][warp >> 1] : 0u;
                const unsigned cols = block_b.flags[0] ? block_b.cls[lane][(warp & 1) * 2] | block_b.cls[lane][(warp & 1) * 2 + 1] : 0u;
                kind = kind_of(rows, cols, false);
            }
            const unsigned checked = __ballot_sync(0xffffffffu, kind == kChecked), both = __ballot_sync(0xffffffffu, kind == kBothOff);
            const unsigned rowed = __ballot_sync(0xffffffffu, kind == kRowsOff);
            const unsigned b_dirty = block_b.flags[0] ? 255u : 0u;
            int kk = 0;
            auto run_end = [&](unsigned mask) { return min(lines, kk + __ffs((int)(~mask >> kk)) - 1); };   // (masks: 16 bits)
            while (kk < lines) {
                const unsigned here = 1u << kk;
                if (checked & here) {
                    const int end = run_end(checked);
#pragma unroll 1
                    for (; kk < end; ++kk) {
                        PAMK_FRAGMENTS(kk)
                        float araw[MR];
#pragma unroll
                        for (int i = 0; i < MR; ++i) araw[i] = i2f(iadd(a[i], p.bias_sub));
#pragma unroll
                        for (int i = 0; i < MR; ++i)
#pragma unroll
                            for (int j = 0; j < MT; ++j) {
                                const float mag = fabsf(fmul(araw[i], i2f(b[j])));
                                const float prod = mag <= i2f(kPassBits) ? i2f(iadd(a[i], b[j])) : quiet_nan();
                                if (!(mag <= i2f(kFlushBits))) acc[i][j] = fadd(acc[i][j], prod);
                            }
                    }
                } else if (both & here) {                    // rows by weights, as in gemm.cu
                    const int end = run_end(both);
#pragma unroll 1
                    for (; kk < end; ++kk) {
                        PAMK_FRAGMENTS(kk)
                        const unsigned cols_off = block_b.off[kk][tx], rows_off = block_a.off[kk][ty];
                        float w[8];
                        int ai[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            w[i] = rows_off & (1u << i) ? 0.0f : 1.0f;
                            ai[i] = rows_off & (1u << i) ? 0 : a[i];
                        }
#pragma unroll
                        for (int j = 0; j < MT; ++j) {
                            int q[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) q[i] = iadd(ai[i], b[j]);
                            fma_column_unless(cols_off & (1u << j), acc, j, q, w);
                        }
                    }
                } else if (rowed & here) {
                    const int end = run_end(rowed);
#pragma unroll 1
                    for (; kk < end; ++kk) {
                        PAMK_FRAGMENTS(kk)
                        const unsigned rows_off = block_a.off[kk][ty];
#pragma unroll
                        for (int i = 0; i < MR; ++i) {
                            int q[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) q[j] = iadd(a[i], b[j]);
                            add_row_unless(rows_off & (1u << i), acc[i], q);
                        }
                    }
                } else {
                    const unsigned others = (checked | both | rowed) >> kk;
                    const int end = others ? kk + __ffs((int)others) - 1 : lines;
#pragma unroll 1
                    for (; kk < end; ++kk) {
                        PAMK_FRAGMENTS(kk)
                        const unsigned cols_off = block_b.off[kk][tx] & b_dirty;
#pragma unroll
                        for (int j = 0; j < MT; ++j) {
                            int q[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) q[i] = iadd(a[i], b[j]);
                            add_column_unless(cols_off & (1u << j), acc, j, q);
                        }
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) barrier_arrive(ring.empty + stage);
        if (++stage == kStages) { stage = 0; parity ^= 1; }
    }
#undef PAMK_FRAGMENTS
    if (!ok) {
        // no copy may be in flight when the CTA leaves (at most kAhead are; one that does not land in time is the last waited for)
        for (int s = landed; tid == 0 && s < requested; ++s)
            if (!barrier_wait(ring.full + s % kStages, (unsigned)(s / kStages) & 1u, nullptr, nullptr)) break;
#pragma unroll
        for (int i = 0; i < MR; ++i)
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[i][j] = quiet_nan();
    }

    next_may_start();                                           // (the reduction pass)
    const int m0 = blockIdx.y * (MR * 16), n0 = blockIdx.x * 128;
    float* Cz = p.C + (int64_t)sp * p.sCsplit + (int64_t)__umulhi((unsigned)z, p.inner_magic) * p.sCb + (int64_t)z * p.sCb2;
    const bool vec_out = ((p.N | p.ldc | p.sCb | p.sCb2 | p.sCsplit) & 3) == 0 && aligned16(p.C);
    const bool post = p.post != 0 && p.splits == 1, add_bias = p.bias != nullptr && p.splits == 1;   // (with ranges the reduction's)
#pragma unroll
    for (int i = 0; i < MR; ++i) {
        const int row = m0 + packed_row(ty * 4 + (i & 3) + (i >> 2) * 64, MR * 16);
        if (row >= p.M) continue;
        float* crow = Cz + (int64_t)row * p.ldc;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int col = n0 + tx * 4 + h * 64;
            if (add_bias) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (col + j < p.N) acc[i][h * 4 + j] = fadd(acc[i][h * 4 + j], __ldg(p.bias + col + j));
            }
            if (post) {
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][h * 4 + j] = mul(acc[i][h * 4 + j], p.post_scale, p.off);
            }
            if (vec_out) {
                if (col < p.N)
                    *reinterpret_cast<float4*>(crow + col) = make_float4(acc[i][h * 4], acc[i][h * 4 + 1], acc[i][h * 4 + 2], acc[i][h * 4 + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (col + j < p.N) crow[col + j] = acc[i][h * 4 + j];
            }
        }
    }
}

// ---- where the operands are packed, and the scratch that it takes --------------------------------------------------------------
// The line lies where clean operands break even: 1.76 us saved per 1e9 products, 1.83 us per million elements and 12 us for the passes, their launches
// and flags.  Below it the operands are used in place, also where they hold special values, which nothing knows beforehand.  Clean operands,
// in place with both contiguous along their rows / in the other layouts / packed: 8192x8192x4096 16780 / 17350 to 17400 / 16510, 4096^3 4237 / 4377 to
// 4399 / 4230, and right above the line, where the layout that has least to gain loses 1 %, 3000^3 1795 / 1858 to 1871 / 1816 (1 % specials in place a
// half slower than packed); below it 4096x4096x512 543 us in place, 578 packed, 2048^3 557 and 603, 3000x1500x2000 608 and 625; with 1 % specials
// 1500x1500x4096 1411 and 946.
int g_packing_policy = 0;            // tests: 0 by the rule, 1 wherever it exists, 2 nowhere

bool packing_pays(int64_t batch, int64_t M, int64_t N, int64_t K) {
    if (g_packing_policy != 0) return g_packing_policy == 1;
    const double saved = 1.76e-9 * (double)batch * (double)M * (double)N * (double)K;
    return saved > 1.83e-6 * (double)batch * (double)K * ((double)M + (double)N) + 12.0;
}

struct PackLayout {
    int tile_rows, a_tiles, b_tiles, slabs;
    int64_t a_blocks, b_blocks;
    size_t extremes;                 // bytes of one operand's
    size_t bytes;                    // the two operands' extremes, then A's blocks, then B's
};

PackLayout pack_layout(int64_t batch, int64_t M, int64_t N, int64_t K, int tile_rows) {
    PackLayout l{};
    l.tile_rows = tile_rows;
    l.a_tiles = (int)((M + tile_rows - 1) / tile_rows);
    l.b_tiles = (int)((N + 127) / 128);
    l.slabs = (int)((K + 15) / 16);
    l.a_blocks = batch * l.a_tiles * l.slabs;
    l.b_blocks = batch * l.b_tiles * l.slabs;
    l.extremes = ((size_t)batch * l.slabs * 16 * 2 * sizeof(unsigned) + 255) / 256 * 256;
    l.bytes = 2 * l.extremes + (size_t)(l.a_blocks + l.b_blocks) * sizeof(PackBlock);
    return l;
}

// Packs both operands and forms the product (or the partials of its ranges); `p` is in the kernel's form, `space` 256-byte aligned.
int run_packed(const GemmParams& p, const PackLayout& l, bool a_kc, bool b_kc, bool a_vec, bool b_vec, void* space, cudaStream_t st) {
    unsigned char* at = static_cast<unsigned char*>(space);
    cudaError_t e = cudaMemsetAsync(at, 0, 2 * l.extremes, st);
    if (e != cudaSuccess) return record_cuda_error(e);
    PackArg A{p.A, reinterpret_cast<PackBlock*>(at + 2 * l.extremes), reinterpret_cast<unsigned*>(at), p.bias_sub, p.M, p.K, p.inner,
              p.inner_magic, l.a_tiles, l.tile_rows, l.slabs, a_kc, a_vec};
    PackArg B{p.B, A.out + l.a_blocks, reinterpret_cast<unsigned*>(at + l.extremes), 0, p.N, p.K, p.inner,
              p.inner_magic, l.b_tiles, 128, l.slabs, b_kc, b_vec};
    const int groups = (l.slabs + kPackSlabs - 1) / kPackSlabs;
    const int64_t a_ctas = (int64_t)p.batch * groups * l.a_tiles, b_ctas = (int64_t)p.batch * groups * l.b_tiles;
    if (a_ctas + b_ctas > 0x7fffffff) return PAMK_ERR_SIZE;
    pack_kernel<<<(unsigned)(a_ctas + b_ctas), 256, 0, st>>>(A, B, groups, (int)a_ctas);
    int rc = check_launch();
    if (rc != PAMK_OK) return rc;
    const int64_t blocks = l.a_blocks + l.b_blocks, resident = (int64_t)sm_count() * 8;
    classify_kernel<<<(unsigned)(blocks < resident ? blocks : resident), 256, 0, st>>>(A, B, l.a_blocks, blocks);
    rc = check_launch();
    if (rc != PAMK_OK) return rc;
    const PackedParams g{A.out, B.out, p.C, p.ldc, p.sCb, p.sCb2, p.sCsplit, p.bias, p.post, p.post_scale, p.inner_magic,
                         p.M, p.N, p.K, p.splits, p.k_chunk / 16, l.slabs, l.a_tiles, l.b_tiles, p.bias_sub, p.off, p.one, p.least};
    const auto kernel = l.tile_rows == 128 ? packed_kernel<8> : packed_kernel<7>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Ring));   // (per device)
    if (e != cudaSuccess) return record_cuda_error(e);
    kernel<<<dim3((unsigned)l.b_tiles, (unsigned)l.a_tiles, (unsigned)(p.batch * p.splits)), 256, sizeof(Ring), st>>>(g);
    return check_launch();
}
