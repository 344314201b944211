// 32-bit matrix product for many rows on the fifth-generation tensor cores:
// out[M, N] = a[M, K] * w[N, K]^T (+ bias[N]), operands and result in 32 bits.
//
// A 32-bit number is three bfloat16 numbers: x = h + m 2^-8 + l 2^-16, each the nearest to what the
// ones before it leave, so that the 24 bits of x are all there (and, scaled like this, they stay there
// down to the smallest normal x). Of the nine products of two such numbers the six of the first three
// orders are added up; the others are below 2^-26 of the product, a quarter of a 32-bit rounding. The
// orders of a section of 32 values of K are added from the smallest to the largest in one accumulator,
// which the instruction scales by 2^-8 between them. The tensor cores cut what an addition leaves
// behind the 24th bit; so the accumulator is emptied every 32 values (two cuts of the largest order),
// sections are added up with ordinary rounding in registers, eight at a time, and the sums of 256 values
// in tensor memory. Error against 64 bits (2-norm, normal inputs) at K = 1,024 / 2,048 / 8,192: 9.0e-8 / 9.8e-8 /
// 1.33e-7; the FMA kernels' 1.24e-7 / 1.30e-7 / 1.58e-7. With all products positive the cuts, which go towards
// zero, add up: 6.9e-8 / 7.3e-8 / 7.7e-8 against 4.8e-8 / 5.3e-8 / 9.0e-8.
//
// Us here / by FMA tiles (with a cold L2): 2048 -> 16384 at 200 / 300 / 1,200 / 4,096 rows 177 / 472, 253 / 610,
// 656 / 1,933, 2,180 / 6,042; 8192 -> 2048 at the same 157 / 277, 290 / 456, 364 / 1,389, 1,130 / 3,851; 1024 -> 1024
// 17 / 27, 26 / 40, 48 / 104, 95 / 247. So every product of more rows than 130 is taken, the number up to
// which all 32-bit kernels add a row up in one order.
//
// An output that does not come out as an ordinary number (infinities and NaN in the inputs make
// parts that are none, values near the largest round up to infinity as bfloat16; results below 2^-100)
// is computed again by one thread in 32-bit FMAs, in the order of gemm_f32.cu.
//
// Persistent blocks, one per SM, of 20 warps; tiles of 128 x BN outputs:
//   warp 0       one thread issues tcgen05.mma (M = 128, N = BN, K = 16), twelve a section (warps 1-3 idle)
//   warps 4-11   add up the sections: a quarter of the accumulator's lanes, half of its columns each
//   warps 12-19  read the operands, 64 values of K a stage, cut them and write the three parts into
//                shared memory (128-byte swizzle); the next stage's values are asked for once a stage is handed
//                over (asked for between the cuts they made a stage a quarter longer; with 16 warps that
//                cut it took 4 % longer)
// Reading each operand tile as it is and cutting it here costs less than a pass that cuts the weights
// first (134 MB in and 201 MB out for 2048 -> 16384) or keeping three more copies of them.
#include "common.cuh"
#include "float_pairs.cuh"

namespace {

constexpr int BM = 128, BK = 64, SECTION = 32, GROUP = 8;      // GROUP sections: 256 values of K
constexpr int STAGES = 2, BUFFERS = 2;
constexpr int SUM_WARPS = 8, CUT_WARPS = 8, FIRST_SUM = 4, FIRST_CUT = FIRST_SUM + SUM_WARPS;
constexpr int THREADS = 32 * (FIRST_CUT + CUT_WARPS);
// registers a thread: 96 at the launch (640 x 96 = 61,440), of which the first four warps give up what the
// ones that add take: 128 x 40 + 256 x 120 + 256 x 96 = 60,416
constexpr int ISSUE_REGISTERS = 40, SUM_REGISTERS = 120, CUT_REGISTERS = 96;
// results outside of these sizes are computed again in FMAs
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
// D = A B + 2^-8 D
__device__ __forceinline__ void mma_next_order(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.eq.b32 p, 0, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 8;\n}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc) : "memory");
}
// 16 consecutive 32-bit columns of this thread's lane of tensor memory
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

// Two 32-bit numbers -> their parts: h, m 2^8, l 2^16 as pairs of bfloat16. (Everything but the
// roundings to bfloat16 is exact: x 256 - h 256 has no more bits than x.)
__device__ __forceinline__ uint32_t nearest_pair(float lo, float hi) {
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(hi), "f"(lo));
    return p;
}
__device__ __forceinline__ void left_over(float& lo, float& hi, uint32_t part) {
    const FloatPair up = pair_of(256.f), down = pair_of(-256.f);
    const FloatPair known = pair_of(__uint_as_float(part << 16), __uint_as_float(part & 0xffff0000u));
    unpair(fma_pair(known, down, mul_pair(pair_of(lo, hi), up)), lo, hi);
}
__device__ __forceinline__ void cut(float lo, float hi, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = nearest_pair(lo, hi);
    left_over(lo, hi, h);
    m = nearest_pair(lo, hi);
    left_over(lo, hi, m);
    l = nearest_pair(lo, hi);
}

// (also true of NaN)
__device__ __forceinline__ bool needs_plain(float value) {
    const float size = fabsf(value);
    return !(size <= LARGEST) || (size < SMALLEST && size > 0.f);
}

// One output as gemm_f32.cu adds it up (strands of 32 values, sections of 256). Not inlined: it is
// all but never called.
__device__ __noinline__ float plain_product(const float* a, const float* w, int k) {
    float total = 0.f;
    for (int section = 0; section < k; section += 256) {
        float sum = 0.f;
        for (int strand = 0; strand < 8; ++strand) {
            float acc = 0.f;
            for (int j = 0; j < 4; ++j) {
                const int at = section + 64 * j + 8 * strand;
                if (at < k)                                     // (K is a multiple of 8)
                    for (int i = 0; i < 8; ++i) acc = fmaf(a[at + i], w[at + i], acc);
            }
            sum += acc;
        }
        total += sum;
        if (total != total) break;                              // NaN stays
    }
    return total;
}

template <int BN>
__host__ __device__ constexpr int stage_bytes() { return 3 * (BM + BN) * BK * 2; }

template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_split_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw,
                      const float* __restrict__ bias, float* __restrict__ out, int ldo, int m, int n, int k,
                      int tiles_m, int total_tiles, int splits, int* __restrict__ error_flag) {
    constexpr int A_PART = BM * BK * 2, W_PART = BN * BK * 2, COLUMNS = BN / 2;
    // pieces of 8 values, a thread and stage (the last for half of the threads where BN is 96 or 160)
    constexpr int ROWS = CUT_WARPS * 4, PIECES = (BM + BN + ROWS - 1) / ROWS;
    static_assert(BM % ROWS == 0 && BK == 64 && COLUMNS % 16 == 0 && 3 * BN <= 512, "tile");
    extern __shared__ unsigned char shared_raw[];
    // full, empty per stage; ready, drained per accumulator
    __shared__ __align__(8) unsigned long long barriers[2 * STAGES + 2 * BUFFERS];
    __shared__ uint32_t tmem_base_slot;
    const uint32_t tiles = (shared_address(shared_raw) + 1023u) & ~1023u;
    float* partial = reinterpret_cast<float*>(shared_raw + (tiles - shared_address(shared_raw)));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // this block's part of K, in whole groups of 256 values
    const int groups = (k + GROUP * SECTION - 1) / (GROUP * SECTION), rank = blockIdx.x % splits;
    const int k_begin = (int)((long long)groups * rank / splits) * GROUP * SECTION;
    const int k_end = min(k, (int)((long long)groups * (rank + 1) / splits) * GROUP * SECTION);
    const int stages = (k_end - k_begin + BK - 1) / BK, sections = (k_end - k_begin + SECTION - 1) / SECTION;
    const int first_tile = blockIdx.x / splits, tile_step = gridDim.x / splits;
    auto full = [&](int s) { return shared_address(&barriers[s]); };
    auto empty = [&](int s) { return shared_address(&barriers[STAGES + s]); };
    auto ready = [&](int b) { return shared_address(&barriers[2 * STAGES + b]); };
    auto drained = [&](int b) { return shared_address(&barriers[2 * STAGES + BUFFERS + b]); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            barrier_init(full(s), CUT_WARPS);
            barrier_init(empty(s), 1);
        }
        for (int b = 0; b < BUFFERS; ++b) {
            barrier_init(ready(b), 1);
            barrier_init(drained(b), SUM_WARPS);
        }
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
            int step = 0, round = 0;
            bool ok = true;
            for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
                for (int stage = 0; stage < stages && ok; ++stage, ++step) {
                    const int s = step % STAGES;
                    ok = barrier_wait(full(s), (step / STAGES) & 1, error_flag);
                    if (!ok) break;
                    fence_after_sync();
                    const uint32_t at = tiles + s * stage_bytes<BN>();
                    const uint64_t ah = operand_descriptor(at), wh = operand_descriptor(at + 3 * A_PART);
                    const uint64_t am = ah + (A_PART >> 4), al = ah + (2 * A_PART >> 4);
                    const uint64_t wm = wh + (W_PART >> 4), wl = wh + (2 * W_PART >> 4);
                    for (int half = 0; half < 2 && 2 * stage + half < sections; ++half, ++round) {
                        const int b = round % BUFFERS;
                        ok = barrier_wait(drained(b), ((round / BUFFERS) & 1) ^ 1, error_flag);
                        if (!ok) break;
                        fence_after_sync();
                        const uint32_t d = tmem_base + b * BN;
                        const int x = 4 * half, y = x + 2;        // 16 values: 32 bytes, 2 address units
                        mma(d, al + x, wh + x, idesc, false);
                        mma(d, al + y, wh + y, idesc, true);
                        mma(d, am + x, wm + x, idesc, true);
                        mma(d, am + y, wm + y, idesc, true);
                        mma(d, ah + x, wl + x, idesc, true);
                        mma(d, ah + y, wl + y, idesc, true);
                        mma_next_order(d, am + x, wh + x, idesc);
                        mma(d, am + y, wh + y, idesc, true);
                        mma(d, ah + x, wm + x, idesc, true);
                        mma(d, ah + y, wm + y, idesc, true);
                        mma_next_order(d, ah + x, wh + x, idesc);
                        mma(d, ah + y, wh + y, idesc, true);
                        mma_commit(ready(b));
                    }
                    mma_commit(empty(s));
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
        const uint32_t totals = lanes + BUFFERS * BN;
        const bool whole_rows = ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
        int round = 0;
        bool ok = true;
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            float sum[COLUMNS];
            for (int first = 0; first < sections && ok; first += GROUP) {
#pragma unroll
                for (int c = 0; c < COLUMNS; ++c) sum[c] = 0.f;
                const int last = min(first + GROUP, sections);
                for (int section = first; section < last; ++section, ++round) {
                    const int b = round % BUFFERS;
                    ok = barrier_wait(ready(b), (round / BUFFERS) & 1, error_flag);
                    if (!ok) break;
                    fence_after_sync();
#pragma unroll
                    for (int c = 0; c < COLUMNS; c += 16) {
                        float part[16];
                        tmem_load(lanes + b * BN + c, part);
#pragma unroll
                        for (int i = 0; i < 16; ++i) sum[c + i] += part[i];
                    }
                    fence_before_sync();
                    __syncwarp();
                    if (lane == 0) barrier_arrive(drained(b));
                }
                if (first > 0)
#pragma unroll
                    for (int c = 0; c < COLUMNS; c += 16) {
                        float old[16];
                        tmem_load(totals + c, old);
#pragma unroll
                        for (int i = 0; i < 16; ++i) sum[c + i] += old[i];
                    }
                if (last < sections) {
#pragma unroll
                    for (int c = 0; c < COLUMNS; c += 16) tmem_store(totals + c, sum + c);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                }
            }
            if (!ok) break;
            if (BN == 64 && splits > 1) {
                // (one tile a block, and all its products have been read: the stages' memory is free)
                float4* to = reinterpret_cast<float4*>(partial + (quarter * 32 + lane) * (BN + 4) + half * COLUMNS);
#pragma unroll
                for (int c = 0; c < COLUMNS; c += 4)
                    to[c / 4] = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
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
                for (int i = 0; i < 16; ++i) value[i] = sum[c + i];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    if (needs_plain(value[i])) again[c / 16] |= 1u << i;
                    if (bias != nullptr && column0 + c + i < n) value[i] += bias[column0 + c + i];
                }
                float* to = out + (size_t)row * ldo + column0 + c;
                if (whole_rows && column0 + c + 16 <= n) {
                    if (row < m)
#pragma unroll
                        for (int i = 0; i < 16; i += 4)
                            *reinterpret_cast<float4*>(to + i) =
                                make_float4(value[i], value[i + 1], value[i + 2], value[i + 3]);
                } else if (row < m) {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (column0 + c + i < n) to[i] = value[i];
                }
            }
#pragma unroll
            for (int c = 0; c < COLUMNS; c += 16)
                for (uint32_t left = row < m ? again[c / 16] : 0; left != 0; left &= left - 1) {
                    const int column = column0 + c + __ffs(left) - 1;
                    if (column >= n) break;
                    const float value = plain_product(a + (size_t)row * lda, w + (size_t)column * ldw, k);
                    out[(size_t)row * ldo + column] = value + (bias != nullptr ? bias[column] : 0.f);
                }
            __syncwarp();
        }
        if (BN == 64 && splits > 1) {
            // Every block of the cluster adds up, in the order of the parts of K, an equal share of the rows.
            __syncwarp();
            cluster_barrier();
            const int rows = BM / splits, row0 = (first_tile % tiles_m) * BM, column0 = (first_tile / tiles_m) * BN;
            for (int i = threadIdx.x - 32 * FIRST_SUM; i < rows * (BN / 4); i += 32 * SUM_WARPS) {
                const int r = rank * rows + i / (BN / 4), c = i % (BN / 4) * 4;
                const int row = row0 + r, column = column0 + c;
                if (row >= m || column >= n) continue;
                float value[4] = {0.f, 0.f, 0.f, 0.f};
                for (int s = 0; s < splits; ++s) {
                    uint32_t from;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from)
                        : "r"(shared_address(partial + r * (BN + 4) + c)), "r"(s));
                    float4 part;
                    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                                 : "=f"(part.x), "=f"(part.y), "=f"(part.z), "=f"(part.w) : "r"(from) : "memory");
                    value[0] = s == 0 ? part.x : value[0] + part.x;
                    value[1] = s == 0 ? part.y : value[1] + part.y;
                    value[2] = s == 0 ? part.z : value[2] + part.z;
                    value[3] = s == 0 ? part.w : value[3] + part.w;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (column + j >= n) continue;
                    if (needs_plain(value[j]))
                        value[j] = plain_product(a + (size_t)row * lda, w + (size_t)(column + j) * ldw, k);
                    if (bias != nullptr) value[j] += bias[column + j];
                }
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
            if (kk < k_end && r < BM + BN && row < (of_a ? m : n)) {
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
                    if (r >= BM + BN) break;
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
    const int groups = ceil_div_host(k, GROUP * SECTION);
    int splits = 1;
    if (groups >= 2 && tiles * 2 <= sm_count() - 4) splits = 2;
    if (groups >= 4 && tiles * 4 <= sm_count() - 16) splits = 4;
    if (groups >= 8 && tiles * 8 <= sm_count() - 36) splits = 8;
    // Otherwise what a tile width takes: rounds of tiles over the SMs times what a tile moves.
    const auto cost = [&](int bn) {
        const long long tiles = (long long)ceil_div_host(m, BM) * ceil_div_host(n, bn);
        return (double)ceil_div_host(tiles, sm_count()) * (128 + bn);
    };
    const double c64 = cost(64), c96 = cost(96), c128 = cost(128), c160 = cost(160);
#define TILES(BN) return launch<BN>(a, lda, w, ldw, bias, out, ldo, m, n, k, splits, error_flag, stream)
    if (splits > 1) TILES(64);
    if (c160 < c128 && c160 < c96 && c160 < c64) TILES(160);
    if (c128 <= c96 && c128 <= c64) TILES(128);
    if (c96 < c64) TILES(96);
    TILES(64);
#undef TILES
}
