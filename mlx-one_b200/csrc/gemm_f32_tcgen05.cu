// 32-bit matrix product for many rows on the fifth-generation tensor cores:
// out[M, N] = a[M, K] * w[N, K]^T (+ bias[N]), operands and result in 32 bits.
//
// A 32-bit number is three bfloat16 numbers: x = h + m + l, each the nearest to what the ones before it leave, so
// that the 24 bits of x are all there (also those of the smallest x: operands are scaled by 2^16 ahead). Of the
// nine products of two such numbers eight are added up; l l is below 2^-34 of the product.
//
// The order of additions of an output is a function of K alone, whatever the number of rows, the tile's width and
// the number of blocks that share K:
//   leading   h h of 16 values: one instruction into an empty accumulator. (The tensor cores cut what an
//             addition leaves behind the 24th bit, towards zero. Products of 8-bit numbers mostly fit, so little is
//             lost here; with the other products in the same accumulator, and 32 values, twice to three times as much is.)
//   others    the seven products of 256 values and more in one accumulator: 2^-8 of the leading ones, and so are its cuts
//   section   two leading accumulators (32 values), added with ordinary rounding; a part's last one takes the others
//             with it
//   part      K's parts (of 256 values up to K = 2,048, eight parts beyond) add up their sections in ascending order
//   output    the parts, ascending, then the bias
// Error against 64 bits (2-norm) here / by the FMA kernels, normal inputs, K = 256 / 1,024 / 2,048 / 8,192: 6.6e-8 / 1.17e-7,
// 7.7e-8 / 1.24e-7, 8.7e-8 / 1.30e-7, 1.26e-7 / 1.58e-7; all products positive (absolute values of the same): 5.4e-8 / 5.8e-8,
// 4.9e-8 / 4.8e-8, 5.4e-8 / 5.3e-8, 6.0e-8 / 9.0e-8, of which the cuts are 1.6e-8 at every K (mean, towards zero).
// Products of one sign over many powers of two (exp(2 normal) on both sides) are where the cuts show:
// 1.3e-7 to 2.4e-7 against 0.7e-7 to 1.1e-7.
//
// Bound: eight bfloat16 products; in fact by the chain of a stage, below. Us here / by FMA tiles (with a cold
// L2): 2048 -> 16384 at 200 / 300 / 1,200 / 4,096 rows 183 / 467, 271 / 604, 798 / 1,936, 2,453 / 6,043; 8192 -> 2048 at the
// same 162 / 273, 306 / 454, 444 / 1,383, 1,319 / 3,846; 1024 -> 1024 20 / 24, 31 / 37, 48 / 102, 97 / 245. (With six
// products and all of them in one accumulator, whose errors were 40 % above the FMA kernels' where products
// have one sign: 656 and 364 us at 1,200 rows.)
//
// An output that does not come out as an ordinary number (infinities and NaN in the inputs, inputs of 2^112 and
// more and results of 2^95 and more, which the scale takes out of range; results below 2^-132) is computed again
// by a warp in 32-bit FMAs, in the order of gemm_f32.cu. That is slow: 2048 -> 16384 at 1,200 rows takes 803 us, 1,230
// with one infinity among the inputs (a row of outputs), 2,550 with 19 rows of 2^115, 85 ms where all results are tiny.
//
// Persistent blocks, one per SM, of 20 warps; tiles of 128 x BN outputs:
//   warp 0       one thread issues tcgen05.mma (M = 128, K = 16): the leading products, then, while those are
//                read, the others (warps 1-3 idle)
//   warps 4-11   add up the sections: a quarter of the accumulator's lanes, half of its columns each
//   warps 12-19  read the operands, 64 values of K a stage, cut them and write the three parts into
//                shared memory (128-byte swizzle); the next stage's values are asked for once a stage is handed
//                over (asked for between the cuts they made a stage a quarter longer; 16 warps that cut took longer
//                too: 813 against 765 us when each was otherwise the same)
// Reading each operand tile as it is and cutting it here costs less than a pass that cuts the weights
// first (134 MB in and 201 MB out for 2048 -> 16384) or keeping three more copies of them.
#include "common.cuh"
#include "float_pairs.cuh"

namespace {

constexpr int BM = 128, BK = 64, SECTION = 32, GROUP = 256;
constexpr int STAGES = 2, MOST_PARTS = 8;
constexpr int SUM_WARPS = 8, CUT_WARPS = 8, FIRST_SUM = 4, FIRST_CUT = FIRST_SUM + SUM_WARPS;
constexpr int THREADS = 32 * (FIRST_CUT + CUT_WARPS);
// registers a thread: 96 at the launch (640 x 96 = 61,440), of which the first four warps give up what the
// ones that add take: 128 x 48 + 256 x 120 + 256 x 96 = 61,440
constexpr int ISSUE_REGISTERS = 48, SUM_REGISTERS = 120, CUT_REGISTERS = 96;
// operands are scaled by 2^16 ahead of the cut, so results by 2^32; those outside of these sizes are
// computed again in FMAs
constexpr float SCALE = 65536.f, UNSCALE = 1.f / (65536.f * 65536.f);
constexpr float LARGEST = 3.0e38f, SMALLEST = 7.9e-31f;
constexpr int WAIT_LIMIT = 1 << 24;                            // polls before a wait gives up
constexpr int ERROR_WAIT = 9;

__device__ __forceinline__ uint32_t shared_address(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void barrier_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void barrier_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool barrier_wait(uint32_t bar, uint32_t parity, int* error_flag) {
    for (int i = 0; i < WAIT_LIMIT; ++i) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.b32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    atomicExch(error_flag, ERROR_WAIT);
    return false;
}
__device__ __forceinline__ void fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// D = A B + D (or A B alone)
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
// Consecutive 32-bit columns of this thread's lane of tensor memory
__device__ __forceinline__ void tmem_load(uint32_t address, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(address));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// ... of two places, under way side by side
__device__ __forceinline__ void tmem_load(uint32_t address, float (&v)[16], uint32_t other, float (&u)[16]) {
    uint32_t r[16], q[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]),
          "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]),
          "=&r"(r[14]), "=&r"(r[15]), "=&r"(q[0]), "=&r"(q[1]), "=&r"(q[2]), "=&r"(q[3]), "=&r"(q[4]),
          "=&r"(q[5]), "=&r"(q[6]), "=&r"(q[7]), "=&r"(q[8]), "=&r"(q[9]), "=&r"(q[10]), "=&r"(q[11]),
          "=&r"(q[12]), "=&r"(q[13]), "=&r"(q[14]), "=&r"(q[15])
        : "r"(address), "r"(other) : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) { v[i] = __uint_as_float(r[i]); u[i] = __uint_as_float(q[i]); }
}
__device__ __forceinline__ void tmem_store(uint32_t address, const float* f) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
        ::"f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]), "f"(f[4]), "f"(f[5]), "f"(f[6]), "f"(f[7]),
          "f"(f[8]), "f"(f[9]), "f"(f[10]), "f"(f[11]), "f"(f[12]), "f"(f[13]), "f"(f[14]), "f"(f[15]),
          "r"(address)
        : "memory");
}
// K-major operand tile, rows of 128 bytes, 128-byte swizzle in atoms of 8 rows.
__device__ __forceinline__ uint64_t operand_descriptor(uint32_t address) {
    return (uint64_t)((address & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 |
           (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// 32-bit accumulator, bfloat16 operands, both K-major
__host__ __device__ constexpr uint32_t instruction_descriptor(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Two 32-bit numbers -> their parts h, m, l (times 2^16) as pairs of bfloat16. (Everything but the
// roundings to bfloat16 is exact.)
__device__ __forceinline__ uint32_t nearest_pair(FloatPair x) {
    float lo, hi;
    unpair(x, lo, hi);
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(hi), "f"(lo));
    return p;
}
__device__ __forceinline__ FloatPair left_over(FloatPair x, uint32_t part) {
    const FloatPair known = pair_of(__uint_as_float(part << 16), __uint_as_float(part & 0xffff0000u));
    return fma_pair(known, pair_of(-1.f), x);
}
__device__ __forceinline__ void cut(float lo, float hi, uint32_t& h, uint32_t& m, uint32_t& l) {
    FloatPair x = mul_pair(pair_of(lo, hi), pair_of(SCALE));
    h = nearest_pair(x);
    x = left_over(x, h);
    m = nearest_pair(x);
    l = nearest_pair(left_over(x, m));
}

// (also true of NaN)
__device__ __forceinline__ bool needs_plain(float value) {
    const float size = fabsf(value);
    return !(size <= LARGEST) || (size < SMALLEST && size > 0.f);
}

// One output as gemm_f32.cu adds it up (strands of 32 values, sections of 256), by a warp: a strand a
// lane, four sections at a time. Not inlined: it is all but never called.
__device__ __noinline__ float plain_product(const float* a, const float* w, int k) {
    const int lane = threadIdx.x & 31;
    float total = 0.f;
    for (int first = 0; first < k; first += 4 * GROUP) {
        float strand = 0.f;
        for (int j = 0; j < 4; ++j) {
            const int at = first + (lane >> 3) * GROUP + 64 * j + 8 * (lane & 7);
            if (at < k)                                         // (K is a multiple of 8)
                for (int i = 0; i < 8; ++i) strand = fmaf(a[at + i], w[at + i], strand);
        }
        float section = 0.f;
        for (int i = 0; i < 8; ++i) section += __shfl_sync(0xffffffffu, strand, i, 8);
        for (int i = 0; i < 4; ++i)
            if (first + i * GROUP < k) total += __shfl_sync(0xffffffffu, section, 8 * i);
        if (total != total) break;                              // NaN stays
    }
    return total;
}

// A thread's columns of its row of the output (`left`: columns up to the output's end)
template <int COLUMNS>
__device__ __forceinline__ void store_row(float* to, const float (&value)[COLUMNS], int left, bool whole) {
#pragma unroll
    for (int c = 0; c < COLUMNS; c += 4) {
        if (whole) *reinterpret_cast<float4*>(to + c) = make_float4(value[c], value[c + 1], value[c + 2], value[c + 3]);
        else
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (c + i < left) to[c + i] = value[c + i];
    }
}

template <int BN>
__host__ __device__ constexpr int stage_bytes() { return 3 * (BM + BN) * BK * 2; }

// K's parts: at most eight, of whole groups of 256 values. Part p starts at group part_start(...).
__host__ __device__ constexpr int part_start(int groups, int parts, int p) { return (int)((long long)groups * p / parts); }

// Every output is the sum of its parts of K in ascending order, whoever adds them: one block, or the blocks of
// a cluster (`splits`), each of which has some of the parts.
template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_split_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw,
                      const float* __restrict__ bias, float* __restrict__ out, int ldo, int m, int n, int k,
                      int tiles_m, int total_tiles, int splits, int* __restrict__ error_flag) {
    constexpr int A_PART = BM * BK * 2, W_PART = BN * BK * 2, COLUMNS = BN / 2;
    // pieces of 8 values, a thread and stage
    constexpr int ROWS = CUT_WARPS * 4, PIECES = (BM + BN) / ROWS;
    static_assert(BM % ROWS == 0 && BN % ROWS == 0 && BK == 64 && COLUMNS % 16 == 0, "tile");
    // Tensor memory: the newest two products of the leading parts (for half of the tile's columns at a time
    // where there is no room for more), the sum of all others, and K's parts added up so far
    constexpr int TURNS = BN == 160 ? 2 : 1, LEADING = BN / TURNS, SECOND = (LEADING + 31) / 32 * 32;
    constexpr int OTHERS = 2 * SECOND, SUMS = OTHERS + BN;
    static_assert(SUMS + (BN == 64 ? MOST_PARTS / 2 : 1) * BN <= 512, "tensor memory");
    extern __shared__ unsigned char shared_raw[];
    // full, empty per stage; ready, drained of the leading products and of the others
    __shared__ __align__(8) unsigned long long barriers[2 * STAGES + 6];
    __shared__ uint32_t tmem_base_slot;
    const uint32_t tiles = (shared_address(shared_raw) + 1023u) & ~1023u;
    float* partial = reinterpret_cast<float*>(shared_raw + (tiles - shared_address(shared_raw)));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // this block's parts of K
    const int groups = (k + GROUP - 1) / GROUP, parts = min(groups, MOST_PARTS), rank = blockIdx.x % splits;
    const int part_first = part_start(parts, splits, rank), part_last = part_start(parts, splits, rank + 1);
    auto part_at = [&](int part) { return min(k, part_start(groups, parts, part) * GROUP); };
    const int k_begin = part_at(part_first), k_end = part_at(part_last);
    const int stages = (k_end - k_begin + BK - 1) / BK;
    const int first_tile = blockIdx.x / splits, tile_step = gridDim.x / splits;
    auto full = [&](int s) { return shared_address(&barriers[s]); };
    auto empty = [&](int s) { return shared_address(&barriers[STAGES + s]); };
    auto leading_ready = [&](int turn) { return shared_address(&barriers[2 * STAGES + turn]); };
    auto leading_drained = [&](int turn) { return shared_address(&barriers[2 * STAGES + 2 + turn]); };
    const uint32_t others_ready = shared_address(&barriers[2 * STAGES + 4]), others_drained = others_ready + 8;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            barrier_init(full(s), CUT_WARPS);
            barrier_init(empty(s), 1);
        }
        for (int turn = 0; turn < TURNS; ++turn) {
            barrier_init(leading_ready(turn), 1);
            barrier_init(leading_drained(turn), SUM_WARPS / TURNS);
        }
        barrier_init(others_ready, 1);
        barrier_init(others_drained, SUM_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(shared_address(&tmem_base_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;

    // Tiles that follow one another share their rows of w.
    if (warp < FIRST_SUM) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ISSUE_REGISTERS));
        if (warp == 0 && lane == 0) {
            constexpr uint32_t idesc = instruction_descriptor(BM, BN);
            constexpr uint32_t idesc_leading = instruction_descriptor(BM, LEADING);
            const uint32_t others = tmem_base + OTHERS;
            int step = 0, round = 0, sum = 0;                     // stages, sections, parts so far
            bool ok = true;
            for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step)
                for (int part = part_first; part < part_last && ok; ++part, ++sum) {
                    const int values = part_at(part + 1) - part_at(part);
                    for (int at = 0; at < values && ok; at += BK, ++step) {
                        const int s = step % STAGES;
                        ok = barrier_wait(full(s), (step / STAGES) & 1, error_flag);
                        if (!ok) break;
                        fence_after_sync();
                        const uint32_t stage = tiles + s * stage_bytes<BN>();
                        for (int half = 0; half < 2 && at + half * SECTION < values; ++half, ++round) {
                            // 16 values: 32 bytes, 2 address units
                            const uint64_t ah = operand_descriptor(stage) + 4 * half;
                            const uint64_t wh = operand_descriptor(stage + 3 * A_PART) + 4 * half;
                            const uint64_t am = ah + (A_PART >> 4), al = am + (A_PART >> 4);
                            const uint64_t wm = wh + (W_PART >> 4), wl = wm + (W_PART >> 4);
                            auto add_others = [&](int y) {
                                mma(others, al + y, wm + y, idesc, at > 0 || half > 0 || y > 0);
                                mma(others, am + y, wl + y, idesc, true);
                                mma(others, al + y, wh + y, idesc, true);
                                mma(others, am + y, wm + y, idesc, true);
                                mma(others, ah + y, wl + y, idesc, true);
                                mma(others, am + y, wh + y, idesc, true);
                                mma(others, ah + y, wm + y, idesc, true);
                            };
#pragma unroll
                            for (int turn = 0; turn < TURNS && ok; ++turn) {
                                // (the columns before these have been read)
                                ok = TURNS == 1 || turn == 0
                                    ? barrier_wait(leading_drained(TURNS - 1), (round & 1) ^ 1, error_flag)
                                    : barrier_wait(leading_drained(0), round & 1, error_flag);
                                if (!ok) break;
                                fence_after_sync();
                                const uint64_t rows = wh + turn * (LEADING * 128 >> 4);
                                mma(tmem_base, ah, rows, idesc_leading, false);
                                mma(tmem_base + SECOND, ah + 2, rows + 2, idesc_leading, false);
                                mma_commit(leading_ready(turn));
                                // (what follows runs while the leading products are read)
                                if (turn == 0 && at == 0 && half == 0) {
                                    ok = barrier_wait(others_drained, (sum & 1) ^ 1, error_flag);
                                    if (!ok) break;
                                    fence_after_sync();
                                }
                                // (whoever reads a part's last leading products reads the others with them)
                                const bool last = at + (half + 1) * SECTION >= values;
                                if (turn == 0) add_others(0);
                                if (turn == 0 ? TURNS == 1 || last : !last) add_others(2);
                                if (turn == 0 && last) mma_commit(others_ready);
                            }
                            if (!ok) break;
                        }
                        if (ok) mma_commit(empty(s));
                    }
                }
        }
        if (BN == 64 && splits > 1) {
            __syncwarp();
            cluster_barrier();
            cluster_barrier();
        }
    } else if (warp < FIRST_CUT) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SUM_REGISTERS));
        const int quarter = warp & 3, half = (warp - FIRST_SUM) >> 2;      // (a warp may only touch its own quarter)
        const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16) + half * COLUMNS;
        const int turn = TURNS == 2 ? half : 0;
        const uint32_t leading = lanes - turn * COLUMNS;
        const bool whole_rows = ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
        int round = 0, sums = 0;
        bool ok = true;
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            float sum[COLUMNS];
            for (int part = part_first; part < part_last && ok; ++part, ++sums) {
#pragma unroll
                for (int c = 0; c < COLUMNS; ++c) sum[c] = 0.f;
                const int sections = (part_at(part + 1) - part_at(part) + SECTION - 1) / SECTION;
                for (int section = 0; section < sections; ++section, ++round) {
                    // (the other products join the last section: a rounding less of the whole sum)
                    const bool last = section + 1 == sections;
                    ok = barrier_wait(leading_ready(turn), round & 1, error_flag);
                    if (ok && last) ok = barrier_wait(others_ready, sums & 1, error_flag);
                    if (!ok) break;
                    fence_after_sync();
#pragma unroll
                    for (int c = 0; c < COLUMNS; c += 16) {
                        float first[16], second[16];
                        tmem_load(leading + c, first, leading + SECOND + c, second);
#pragma unroll
                        for (int i = 0; i < 16; ++i) first[i] += second[i];
                        if (last) {
                            tmem_load(lanes + OTHERS + c, second);
#pragma unroll
                            for (int i = 0; i < 16; ++i) first[i] += second[i];
                        }
#pragma unroll
                        for (int i = 0; i < 16; ++i) sum[c + i] += first[i];
                    }
                    fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        barrier_arrive(leading_drained(turn));
                        if (last) barrier_arrive(others_drained);
                    }
                }
                if (!ok) break;
                // parts of a cluster's block stay apart, others are added up
                const bool apart = BN == 64 && splits > 1;
                if (!apart && part > part_first)
#pragma unroll
                    for (int c = 0; c < COLUMNS; c += 16) {
                        float old[16];
                        tmem_load(lanes + SUMS + c, old);
#pragma unroll
                        for (int i = 0; i < 16; ++i) sum[c + i] += old[i];
                    }
                if (part + 1 < part_last) {
                    const uint32_t slot = lanes + SUMS + (apart ? part - part_first : 0) * BN;
#pragma unroll
                    for (int c = 0; c < COLUMNS; c += 16) tmem_store(slot + c, sum + c);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                }
            }
            if (!ok) break;
            if (BN == 64 && splits > 1) {
                // (one tile a block, and all its products have been read: the stages' memory is free)
                float* to = partial + (quarter * 32 + lane) * (BN + 4) + half * COLUMNS;
#pragma unroll
                for (int c = 0; c < COLUMNS; c += 4)
                    *reinterpret_cast<float4*>(to + (part_last - 1 - part_first) * BM * (BN + 4) + c) =
                        make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
                for (int part = part_first; part + 1 < part_last; ++part)
#pragma unroll
                    for (int c = 0; c < COLUMNS; c += 16) {
                        float old[16];
                        tmem_load(lanes + SUMS + (part - part_first) * BN + c, old);
#pragma unroll
                        for (int i = 0; i < 16; i += 4)
                            *reinterpret_cast<float4*>(to + (part - part_first) * BM * (BN + 4) + c + i) =
                                make_float4(old[i], old[i + 1], old[i + 2], old[i + 3]);
                    }
                break;
            }
            const int row = (tile % tiles_m) * BM + quarter * 32 + lane;
            const int column0 = (tile / tiles_m) * BN + half * COLUMNS;
            uint32_t again[COLUMNS / 16];                          // outputs to be computed again, a bit each
#pragma unroll
            for (int c = 0; c < COLUMNS; c += 16) {
                again[c / 16] = 0;
                float value[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    if (needs_plain(sum[c + i]) && row < m && column0 + c + i < n) again[c / 16] |= 1u << i;
                    value[i] = sum[c + i] * UNSCALE;
                    if (bias != nullptr && column0 + c + i < n) value[i] += bias[column0 + c + i];
                }
                if (row < m)
                    store_row<16>(out + (size_t)row * ldo + column0 + c, value, n - column0 - c,
                                  whole_rows && column0 + c + 16 <= n);
            }
#pragma unroll
            for (int c = 0; c < COLUMNS; c += 16)
                for (uint32_t those = __ballot_sync(0xffffffffu, again[c / 16] != 0); those != 0; those &= those - 1) {
                    const int whose = __ffs(those) - 1, its_row = row - lane + whose;
                    for (uint32_t left = __shfl_sync(0xffffffffu, again[c / 16], whose); left != 0; left &= left - 1) {
                        const int column = column0 + c + __ffs(left) - 1;
                        const float value = plain_product(a + (size_t)its_row * lda, w + (size_t)column * ldw, k);
                        if (lane == whose) out[(size_t)row * ldo + column] = value + (bias != nullptr ? bias[column] : 0.f);
                    }
                }
            __syncwarp();
        }
        if (BN == 64 && splits > 1) {
            // Every block of the cluster adds up, in the order of the parts of K, an equal share of the rows.
            __syncwarp();
            cluster_barrier();
            const int rows = BM / splits, row0 = (first_tile % tiles_m) * BM, column0 = (first_tile / tiles_m) * BN;
            // (a whole number of turns: BM / 8 rows of BN / 4 pieces at least)
            for (int i = threadIdx.x - 32 * FIRST_SUM; i < rows * (BN / 4); i += 32 * SUM_WARPS) {
                const int r = rank * rows + i / (BN / 4), c = i % (BN / 4) * 4;
                const int row = row0 + r, column = column0 + c;
                float value[4] = {0.f, 0.f, 0.f, 0.f};
                for (int s = 0; s < splits; ++s)
                    for (int p = part_start(parts, splits, s); p < part_start(parts, splits, s + 1); ++p) {
                        uint32_t from;
                        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from)
                            : "r"(shared_address(partial + (p - part_start(parts, splits, s)) * BM * (BN + 4) +
                                                 r * (BN + 4) + c)), "r"(s));
                        float4 sum;
                        asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                                     : "=f"(sum.x), "=f"(sum.y), "=f"(sum.z), "=f"(sum.w) : "r"(from) : "memory");
                        value[0] = p == 0 ? sum.x : value[0] + sum.x;
                        value[1] = p == 0 ? sum.y : value[1] + sum.y;
                        value[2] = p == 0 ? sum.z : value[2] + sum.z;
                        value[3] = p == 0 ? sum.w : value[3] + sum.w;
                    }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool again = needs_plain(value[j]) && row < m && column + j < n;
                    value[j] *= UNSCALE;
                    for (uint32_t those = __ballot_sync(0xffffffffu, again); those != 0; those &= those - 1) {
                        const int whose = __ffs(those) - 1;
                        const float plain =
                            plain_product(a + (size_t)__shfl_sync(0xffffffffu, row, whose) * lda,
                                          w + (size_t)__shfl_sync(0xffffffffu, column + j, whose) * ldw, k);
                        if (lane == whose) value[j] = plain;
                    }
                    if (bias != nullptr && column + j < n) value[j] += bias[column + j];
                }
                if (row >= m) continue;
                float* to = out + (size_t)row * ldo + column;
                if (whole_rows && column + 4 <= n) {
                    *reinterpret_cast<float4*>(to) = make_float4(value[0], value[1], value[2], value[3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (column + j < n) to[j] = value[j];
                }
            }
            __syncwarp();
            cluster_barrier();                  // (nobody leaves while its sums are read)
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CUT_REGISTERS));
        // A thread takes pieces of 8 values: eight lanes side by side along K, so a warp reads 256
        // contiguous bytes of four rows and its 16-byte stores fall on all banks.
        const int tid = threadIdx.x - 32 * FIRST_CUT;
        const int row0 = tid >> 3, column = tid & 7;              // piece i: row row0 + ROWS i of [a; w]
        float4 lo[PIECES], hi[PIECES];
        auto fetch = [&](int i, int tile, int stage) {
            const int r = row0 + ROWS * i, kk = k_begin + stage * BK + column * 8;
            const bool of_a = ROWS * i < BM;                      // (known when compiling)
            const int row = of_a ? (tile % tiles_m) * BM + r : (tile / tiles_m) * BN + r - BM;
            lo[i] = hi[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (kk < k_end && row < (of_a ? m : n)) {
                const float4* from = reinterpret_cast<const float4*>(
                    (of_a ? a + (size_t)row * lda : w + (size_t)row * ldw) + kk);
                lo[i] = from[0];
                hi[i] = from[1];
            }
        };
        int step = 0;
        bool ok = true;
        if (first_tile < total_tiles)
#pragma unroll
            for (int i = 0; i < PIECES; ++i) fetch(i, first_tile, 0);
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            for (int stage = 0; stage < stages; ++stage, ++step) {
                const int s = step % STAGES;
                ok = barrier_wait(empty(s), ((step / STAGES) & 1) ^ 1, error_flag);
                if (!ok) break;
                const bool end = stage + 1 == stages;
                const int next_tile = end ? tile + tile_step : tile, next_stage = end ? 0 : stage + 1;
                unsigned char* base = shared_raw + (tiles - shared_address(shared_raw)) + s * stage_bytes<BN>();
#pragma unroll
                for (int i = 0; i < PIECES; ++i) {
                    const int r = row0 + ROWS * i;
                    uint4 h, mid, l;
                    cut(lo[i].x, lo[i].y, h.x, mid.x, l.x);
                    cut(lo[i].z, lo[i].w, h.y, mid.y, l.y);
                    cut(hi[i].x, hi[i].y, h.z, mid.z, l.z);
                    cut(hi[i].z, hi[i].w, h.w, mid.w, l.w);
                    const bool of_a = ROWS * i < BM;
                    const int part = of_a ? A_PART : W_PART;
                    unsigned char* to = base + (of_a ? r * 128 : 3 * A_PART + (r - BM) * 128) +
                                        ((column ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4*>(to) = h;
                    *reinterpret_cast<uint4*>(to + part) = mid;
                    *reinterpret_cast<uint4*>(to + 2 * part) = l;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) barrier_arrive(full(s));
                if (next_tile < total_tiles)
#pragma unroll
                    for (int i = 0; i < PIECES; ++i) fetch(i, next_tile, next_stage);
            }
        }
        // (the last stages' products report to nobody else, and a block must not be gone when they do)
        for (int last = max(0, step - STAGES); last < step && ok; ++last)
            ok = barrier_wait(empty(last % STAGES), (last / STAGES) & 1, error_flag);
        if (BN == 64 && splits > 1) {
            __syncwarp();
            cluster_barrier();
            cluster_barrier();
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        fence_after_sync();
        if (*reinterpret_cast<volatile int*>(error_flag) == ERROR_WAIT)
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);    // (products may still be under way)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
    }
}

int sm_count() {
    static const int count = [] {
        int device = 0, value = 148;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device);
        return value;
    }();
    return count;
}

template <int BN>
int launch(const float* a, int lda, const float* w, int ldw, const float* bias, float* out, int ldo, int m,
           int n, int k, int splits, int* error_flag, cudaStream_t stream) {
    constexpr int bytes = STAGES * stage_bytes<BN>() + 1024;
    static_assert(bytes + 128 <= 227 * 1024, "shared memory");
    const int tiles_m = ceil_div_host(m, BM);
    const long long total = (long long)tiles_m * ceil_div_host(n, BN);
    MLXONE_REQUIRE(total < (1ll << 30), "gemm_f32: too many tiles");
    auto kernel = gemm_f32_split_kernel<BN>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    MLXONE_REQUIRE(err == cudaSuccess, "gemm_f32: %s", cudaGetErrorString(err));
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(splits > 1 ? (int)total * splits : total < sm_count() ? (int)total : sm_count());
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = bytes;
    config.stream = stream;
    cudaLaunchAttribute cluster[1];
    cluster[0].id = cudaLaunchAttributeClusterDimension;
    cluster[0].val.clusterDim.x = splits;
    cluster[0].val.clusterDim.y = cluster[0].val.clusterDim.z = 1;
    config.attrs = cluster;
    config.numAttrs = splits > 1 ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, a, lda, w, ldw, bias, out, ldo, m, n, k, tiles_m, (int)total, splits,
                       error_flag);
    MLXONE_LAUNCH_CHECK("gemm_f32 (many rows)");
    return 0;
}

}  // namespace

// a: [m, k] with row stride lda, w: [n, k] with row stride ldw, both on 16-byte boundaries, k a multiple
// of 8, row strides of 4.
MLXONE_API int mlxone_gemm_f32_split(const float* a, int lda, const float* w, int ldw, const float* bias,
                                     float* out, int ldo, int m, int n, int k, int* error_flag,
                                     cudaStream_t stream) {
    if (m == 0 || n == 0) return 0;
    MLXONE_REQUIRE(m > 0 && n > 0 && k > 0 && k % 8 == 0, "gemm_f32_split: bad sizes m=%d n=%d k=%d", m, n, k);
    MLXONE_REQUIRE(lda >= k && ldw >= k && ldo >= n && lda % 4 == 0 && ldw % 4 == 0,
                   "gemm_f32_split: leading dimensions %d, %d, %d", lda, ldw, ldo);
    MLXONE_REQUIRE(((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0,
                   "gemm_f32_split: operands must be 16-byte aligned");
    // K in parts where tiles of 128 x 64 leave SMs idle: a cluster of blocks a tile. (Clusters of eight and
    // of four do not fill every group of SMs.)
    const long long tiles = (long long)ceil_div_host(m, BM) * ceil_div_host(n, 64);
    const int groups = ceil_div_host(k, GROUP);
    int splits = 1;
    if (groups >= 2 && tiles * 2 <= sm_count() - 4) splits = 2;
    if (groups >= 4 && tiles * 4 <= sm_count() - 16) splits = 4;
    if (groups >= 8 && tiles * 8 <= sm_count() - 36) splits = 8;
    // Otherwise what a tile width takes: rounds of tiles over the SMs times a stage's time, measured (2048 -> 16384,
    // 8192 -> 2048, 1024 -> 9216 and 2048 -> 6144 at 300 to 4,096 rows: 2.4 to 2.6, 2.4 to 2.9, 2.6 to 3.1, 3.5 to 4.2 us).
    const auto cost = [&](int bn, double stage) {
        return stage * ceil_div_host((long long)ceil_div_host(m, BM) * ceil_div_host(n, bn), sm_count());
    };
    const double c64 = cost(64, 2.45), c96 = cost(96, 2.6), c128 = cost(128, 2.8), c160 = cost(160, 3.8);
#define TILES(BN) return launch<BN>(a, lda, w, ldw, bias, out, ldo, m, n, k, splits, error_flag, stream)
    if (splits > 1) TILES(64);
    if (c160 < c128 && c160 < c96 && c160 < c64) TILES(160);
    if (c128 <= c96 && c128 <= c64) TILES(128);
    if (c96 < c64) TILES(96);
    TILES(64);
#undef TILES
}
