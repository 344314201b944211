// True 32-bit matrix product: out[M, N] = a[M, K] * w[N, K]^T (+ bias[N]).
//
// Plain FMA on CUDA cores, no tensor cores and no reduced-precision mode. A row's result does not
// depend on how many other rows the call has, on where its tile lies or on which of the kernels
// below computed it: every output is added up in the same order, a function of K alone. (Products of more
// than 130 rows that 16-byte loads can take are gemm_f32_tcgen05.cu's, whose order is a function of K alone too,
// but another: a row's last bits are not the same on both sides of that line.)
//
//   strand   one chain of up to 32 FMAs from zero: of a section of 256 values of K, strand l takes
//            the pieces of eight values at 64 j + 8 l, j = 0 .. 3, in ascending order
//   section  the sum of its eight strands, from zero, l ascending
//   output   the sum of the sections, from zero, ascending, then the bias
//
// (Shorter chains than one of K also leave a smaller rounding error.) The order is made for reading
// a row of w with eight lanes, 32 bytes each: a warp then reads 256 contiguous bytes of each of four
// rows, its lanes need nothing from one another inside a section, and a tile that walks a strand
// still fetches whole 32-byte sectors.
#include "common.cuh"
#include "float_pairs.cuh"

#include <algorithm>

namespace {

constexpr int SECTION = 256, STRANDS = 8, PIECE = 8, PIECES = SECTION / (STRANDS * PIECE);

__device__ __forceinline__ uint32_t shared_address(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------------------------ few rows: w streamed once
//
// Bound by reading w. Up to MR rows of a (1, 2, 4 or 8). A block of eight warps owns `row_groups`
// groups of 4 R rows of w; a warp takes one section of one group at a time: lane = (row of the group,
// strand), and the 32 values of w that a lane needs of each of its R rows are loads of 32 bytes, all
// under way at once. Up to two rows of a the next section's weights are under way meanwhile; with
// more, what a lane issues most are its reads of a, so it takes two rows of w for each instead. The
// rows of a lie in shared memory, `depth` sections at a time, pieces' first and second halves in
// planes of their own so that eight lanes' 16-byte reads fall on all banks. The first group's weights
// are asked for before the wait for the kernel before this one.
constexpr int SKINNY_WARPS = 8;

struct Eight { float v[8]; };

__device__ __forceinline__ Eight load_eight(const float* p) {
    Eight e;
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(e.v[0]), "=f"(e.v[1]), "=f"(e.v[2]), "=f"(e.v[3]), "=f"(e.v[4]), "=f"(e.v[5]),
                   "=f"(e.v[6]), "=f"(e.v[7])
                 : "l"(p));
    return e;
}

__host__ __device__ constexpr int skinny_rows(int mr) { return mr >= 4 ? 2 : 1; }     // R

template <int MR>
__global__ void __launch_bounds__(SKINNY_WARPS * 32, 2)
gemm_f32_skinny_kernel(const float* a, int lda, const float* __restrict__ w, int ldw,
                       const float* __restrict__ bias, float* out, int ldo, int m, int n, int k,
                       int row_groups, int warps_k, int depth) {
    // shared: rows of a [depth sections][MR][2 halves][pieces of four], strands' sums
    // [warps][32 lanes][R * MR + 1], sections' sums [rows of w][MR][sections]
    constexpr int R = skinny_rows(MR), GROUP = 4 * R, SUMS = R * MR + 1, BUFFERS = R == 1 ? 2 : 1;
    extern __shared__ __align__(16) float shared[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane >> 3, strand = lane & 7;
    const int sections = (k + SECTION - 1) / SECTION;
    const int wk = warp % warps_k, wg = warp / warps_k, groups_side = SKINNY_WARPS / warps_k;
    float* rows = shared;
    float* strands = rows + depth * MR * SECTION + warp * 32 * SUMS;
    float* sums = rows + depth * MR * SECTION + SKINNY_WARPS * 32 * SUMS;
    const int m0 = blockIdx.y * MR;
    const int row0 = blockIdx.x * row_groups * GROUP;

    // this warp's walk: sections wk, wk + warps_k, ...; of each, groups wg, wg + groups_side, ...
    Eight wv[BUFFERS][R][PIECES];
    int fetch_section = wk, fetch_group = wg;
    auto fetch = [&](Eight (&to)[R][PIECES]) {
#pragma unroll
        for (int x = 0; x < R; ++x) {
            const int row = row0 + fetch_group * GROUP + x * 4 + sub;
            const float* from = w + (size_t)row * ldw + fetch_section * SECTION + strand * PIECE;
#pragma unroll
            for (int j = 0; j < PIECES; ++j) {
                // (k is a multiple of 8 here, so a piece lies inside a row or outside it)
                const bool live = row < n && fetch_section * SECTION + j * 64 + strand * PIECE < k;
                if (live) to[x][j] = load_eight(from + j * 64);
                else
#pragma unroll
                    for (int i = 0; i < 8; ++i) to[x][j].v[i] = 0.f;
            }
        }
        fetch_group += groups_side;
        if (fetch_group >= row_groups) { fetch_group = wg; fetch_section += warps_k; }
    };
    auto compute = [&](const Eight (&wx)[R][PIECES], const float* mine, int section, int group) {
        float acc[R][MR];
#pragma unroll
        for (int x = 0; x < R; ++x)
#pragma unroll
            for (int r = 0; r < MR; ++r) acc[x][r] = 0.f;
#pragma unroll
        for (int j = 0; j < PIECES; ++j) {
#pragma unroll
            for (int r = 0; r < MR; ++r) {
                const float* at = mine + r * SECTION + (j * STRANDS + strand) * 4;
                const float4 p = *reinterpret_cast<const float4*>(at);
                const float4 q = *reinterpret_cast<const float4*>(at + SECTION / 2);
#pragma unroll
                for (int x = 0; x < R; ++x) {
                    acc[x][r] = fmaf(p.x, wx[x][j].v[0], acc[x][r]);
                    acc[x][r] = fmaf(p.y, wx[x][j].v[1], acc[x][r]);
                    acc[x][r] = fmaf(p.z, wx[x][j].v[2], acc[x][r]);
                    acc[x][r] = fmaf(p.w, wx[x][j].v[3], acc[x][r]);
                    acc[x][r] = fmaf(q.x, wx[x][j].v[4], acc[x][r]);
                    acc[x][r] = fmaf(q.y, wx[x][j].v[5], acc[x][r]);
                    acc[x][r] = fmaf(q.z, wx[x][j].v[6], acc[x][r]);
                    acc[x][r] = fmaf(q.w, wx[x][j].v[7], acc[x][r]);
                }
            }
        }
#pragma unroll
        for (int x = 0; x < R; ++x)
#pragma unroll
            for (int r = 0; r < MR; ++r) strands[lane * SUMS + x * MR + r] = acc[x][r];
        __syncwarp();
#pragma unroll
        for (int i = strand; i < R * MR; i += STRANDS) {
            float sum = 0.f;
#pragma unroll
            for (int l = 0; l < STRANDS; ++l) sum += strands[(sub * STRANDS + l) * SUMS + i];
            const int row = group * GROUP + i / MR * 4 + sub;
            sums[(row * MR + i % MR) * sections + section] = sum;
        }
        __syncwarp();
    };
    fetch(wv[0]);                     // (warps_k <= sections, groups_side <= row_groups)
    griddep_wait();
    griddep_launch();
    int parity = 0;
    for (int base = 0; base < sections; base += depth) {
        if (base > 0) __syncthreads();
        // rows of a for the sections base .. base + depth - 1
        const int here = min(depth, sections - base), pieces = here * MR * (SECTION / 4);
        for (int i = threadIdx.x; i < pieces; i += SKINNY_WARPS * 32) {
            const int at = i % (SECTION / 4), r = (i / (SECTION / 4)) % MR, s = i / (SECTION / 4) / MR;
            const int kk = (base + s) * SECTION + at * 4;
            const bool live = m0 + r < m && kk < k;
            const float* from = live ? a + (size_t)(m0 + r) * lda + kk : a;
            const uint32_t to = shared_address(rows + ((s * MR + r) * 2 + (at & 1)) * (SECTION / 2) +
                                               (at >> 1) * 4);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(from),
                         "r"(live ? 16 : 0));
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        for (int s = wk; s < here; s += warps_k) {
            const float* mine = rows + s * MR * SECTION;
            for (int group = wg; group < row_groups; group += groups_side) {
                if (BUFFERS == 2) {
                    if (parity == 0) {
                        if (fetch_section < sections) fetch(wv[BUFFERS - 1]);
                        compute(wv[0], mine, base + s, group);
                    } else {
                        if (fetch_section < sections) fetch(wv[0]);
                        compute(wv[BUFFERS - 1], mine, base + s, group);
                    }
                    parity ^= 1;
                } else {
                    compute(wv[0], mine, base + s, group);
                    if (fetch_section < sections) fetch(wv[0]);
                }
            }
        }
    }
    __syncthreads();
    // (neighbouring threads: neighbouring columns of a row of out)
    for (int i = threadIdx.x; i < row_groups * GROUP * MR; i += SKINNY_WARPS * 32) {
        const int row = i % (row_groups * GROUP), r = i / (row_groups * GROUP);
        float total = 0.f;
        for (int s = 0; s < sections; ++s) total += sums[(row * MR + r) * sections + s];
        if (row0 + row < n && m0 + r < m)
            out[(size_t)(m0 + r) * ldo + row0 + row] = total + (bias ? bias[row0 + row] : 0.f);
    }
}

// ------------------------------------------------------------------ tiles
//
// Bound by FMA issue: this chip issues an FMA of one value a lane every second cycle, and of two
// (fma.f32x2, each rounded as fmaf) at the same rate, so all sums are held as pairs of neighbouring
// columns. (The same tile with plain FMAs stood at 35 TFLOP/s whatever its shape.) A thread owns
// TM x TN outputs; G groups of threads share a tile, each takes every G-th section of K (so that a
// tile keeps an SM busy where there are few tiles), and the sections' sums meet in shared memory, in
// order. Within a group: stages of BK values of K (16: two pieces of a strand, 32: all four), K
// outermost in shared memory, double-buffered, the next stage's values under way in registers.
template <int BM, int BN, int TM, int TN, int G, int BK, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN) * G)
gemm_f32_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw,
                const float* __restrict__ bias, float* __restrict__ out, int ldo, int m, int n, int k,
                long long batch_a, long long batch_w, long long batch_out) {
    constexpr int TX = BN / TN, THREADS = (BM / TM) * TX, PAIRS = TM * TN / 2;
    constexpr int STAGE = BK * (BM + 4 + BN + 4), PER_STRAND = SECTION / STRANDS / BK;
    static_assert(TM % 4 == 0 && TN % 4 == 0 && THREADS % 32 == 0 && (BK == 16 || BK == 32), "tile shape");
    // (blockIdx.z: one of several products of the same shape whose operands lie a fixed number
    // of values apart)
    a += blockIdx.z * batch_a;
    w += blockIdx.z * batch_w;
    out += blockIdx.z * batch_out;
    extern __shared__ __align__(16) float shared[];
    const int group = threadIdx.x / THREADS, tid = threadIdx.x % THREADS;
    float* stages = shared + group * 2 * STAGE;
    float2* totals = reinterpret_cast<float2*>(shared + G * 2 * STAGE);       // [PAIRS][THREADS]
    float2* parts = totals + PAIRS * THREADS;                                 // G > 1: [G][PAIRS][THREADS]
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    const int ty = tid / TX, tx = tid % TX;
    const int sections = (k + SECTION - 1) / SECTION;
    // (stages of a strand; in K's last section those that lie behind K for every strand are left out:
    // they would add zeros)
    const auto stages_of = [&](int section) {
        return min(PER_STRAND, (k - section * SECTION + BK * STRANDS - 1) / (BK * STRANDS));
    };

    // Copies of a stage: 16-byte quarters q = 0 .. BK / 4 - 1 of each row; two lanes share a 32-byte
    // sector, 16 rows a half-warp, so that the transposed stores fall on different banks.
    constexpr int A_LOADS = BM * (BK / 4) / THREADS, W_LOADS = BN * (BK / 4) / THREADS;
    static_assert(BM * (BK / 4) % THREADS == 0 && BN * (BK / 4) % THREADS == 0 && BM % 16 == 0 && BN % 16 == 0,
                  "copies");
    float4 av[A_LOADS], wv[W_LOADS];
    auto one = [&](const float* base, int ld, int row, int limit, int kk) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < limit) {
            const float* p = base + (size_t)row * ld + kk;
            if (VEC) {
                if (kk < k) v = *reinterpret_cast<const float4*>(p);
            } else {
                if (kk + 0 < k) v.x = p[0];
                if (kk + 1 < k) v.y = p[1];
                if (kk + 2 < k) v.z = p[2];
                if (kk + 3 < k) v.w = p[3];
            }
        }
        return v;
    };
    // copy i of a thread: quarter and row of the tile (pairs of quarters, then rows, then pairs)
    auto place = [&](int i, int rows, int& q, int& r) {
        const int at = i * THREADS + tid;
        q = (at & 1) + 2 * ((at >> 1) / rows);
        r = (at >> 1) % rows;
    };
    auto fetch = [&](int section, int strand, int stage) {
        const int base = section * SECTION + strand * PIECE + stage * BK * STRANDS;
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) {
            int q, r;
            place(i, BM, q, r);
            av[i] = one(a, lda, row0 + r, m, base + (q >> 1) * 64 + (q & 1) * 4);
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) {
            int q, r;
            place(i, BN, q, r);
            wv[i] = one(w, ldw, col0 + r, n, base + (q >> 1) * 64 + (q & 1) * 4);
        }
    };
    auto store = [&](int buffer) {
        float* as = stages + buffer * STAGE;
        float* ws = as + BK * (BM + 4);
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) {
            int q, r;
            place(i, BM, q, r);
            float* to = as + 4 * q * (BM + 4) + r;
            to[0] = av[i].x; to[BM + 4] = av[i].y; to[2 * (BM + 4)] = av[i].z; to[3 * (BM + 4)] = av[i].w;
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) {
            int q, r;
            place(i, BN, q, r);
            float* to = ws + 4 * q * (BN + 4) + r;
            to[0] = wv[i].x; to[BN + 4] = wv[i].y; to[2 * (BN + 4)] = wv[i].z; to[3 * (BN + 4)] = wv[i].w;
        }
    };
    auto meet = [&]() {                            // this group's threads
        if (G == 1) __syncthreads();
        else if (THREADS == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(THREADS) : "memory");
    };
    // a thread's rows and columns: fours, BM / (TM / 4) and BN / (TN / 4) apart, so that the threads
    // of a warp read neighbouring fours
    const auto row_of = [&](int i) { return ty * 4 + (i & 3) + (i >> 2) * (BM * 4 / TM); };
    const auto col_of = [&](int j) { return tx * 4 + (j & 3) + (j >> 2) * (BN * 4 / TN); };

#pragma unroll
    for (int i = 0; i < PAIRS; ++i)
        if (G == 1 || i % G == group) totals[i * THREADS + tid] = make_float2(0.f, 0.f);
    int buffer = 0;
    const int rounds = (sections + G - 1) / G;
    if (group < sections) {
        fetch(group, 0, 0);
        store(0);
        meet();
    }
    for (int round = 0; round < rounds; ++round) {
        const int section = round * G + group;
        FloatPair sum[TM][TN / 2];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) sum[i][j] = 0;
        if (section < sections) {
            const int deep = stages_of(section);
            for (int strand = 0; strand < STRANDS; ++strand) {
                FloatPair acc[TM][TN / 2];
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;
                for (int stage = 0; stage < deep; ++stage) {
                    const bool last = stage + 1 == deep, end = last && strand + 1 == STRANDS;
                    const bool more = !end || section + G < sections;
                    if (more)
                        fetch(end ? section + G : section, end ? 0 : last ? strand + 1 : strand,
                              last ? 0 : stage + 1);
                    const float* as = stages + buffer * STAGE + ty * 4;
                    const float* ws = stages + buffer * STAGE + BK * (BM + 4) + tx * 4;
#pragma unroll
                    for (int kk = 0; kk < BK; ++kk) {
                        FloatPair x[TM], y[TN / 2];
#pragma unroll
                        for (int i = 0; i < TM; i += 4) {
                            const float4 v = *reinterpret_cast<const float4*>(as + kk * (BM + 4) + i * (BM / TM));
                            x[i] = pair_of(v.x); x[i + 1] = pair_of(v.y); x[i + 2] = pair_of(v.z); x[i + 3] = pair_of(v.w);
                        }
#pragma unroll
                        for (int j = 0; j < TN; j += 4) {
                            const ulonglong2 v =
                                *reinterpret_cast<const ulonglong2*>(ws + kk * (BN + 4) + j * (BN / TN));
                            y[j / 2] = v.x; y[j / 2 + 1] = v.y;
                        }
#pragma unroll
                        for (int i = 0; i < TM; ++i)
#pragma unroll
                            for (int j = 0; j < TN / 2; ++j) accumulate_pair(acc[i][j], x[i], y[j]);
                    }
                    buffer ^= 1;
                    if (more) store(buffer);
                    meet();
                }
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) accumulate_pair(sum[i][j], acc[i][j]);
            }
        }
        if (G == 1) {
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                float2 total = totals[i * THREADS + tid];
                float2 here;
                unpair(sum[i / (TN / 2)][i % (TN / 2)], here.x, here.y);
                total.x += here.x;
                total.y += here.y;
                totals[i * THREADS + tid] = total;
            }
        } else {
            if (round > 0) __syncthreads();        // the last round's parts have been read
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                float2 here;
                unpair(sum[i / (TN / 2)][i % (TN / 2)], here.x, here.y);
                parts[(group * PAIRS + i) * THREADS + tid] = here;
            }
            __syncthreads();
            const int here = min(G, sections - round * G);
            for (int i = group; i < PAIRS; i += G) {
                float2 total = totals[i * THREADS + tid];
                for (int g = 0; g < here; ++g) {
                    const float2 part = parts[(g * PAIRS + i) * THREADS + tid];
                    total.x += part.x;
                    total.y += part.y;
                }
                totals[i * THREADS + tid] = total;
            }
        }
    }
    for (int i = G > 1 ? group : 0; i < PAIRS; i += G) {
        const int r = row0 + row_of(i / (TN / 2)), c = col0 + col_of(i % (TN / 2) * 2);
        const float2 total = totals[i * THREADS + tid];
        if (r < m && c < n) out[(size_t)r * ldo + c] = total.x + (bias ? bias[c] : 0.f);
        if (r < m && c + 1 < n) out[(size_t)r * ldo + c + 1] = total.y + (bias ? bias[c + 1] : 0.f);
    }
}

template <int BM, int BN, int TM, int TN, int G, int BK>
int launch_tiles(const float* a, int lda, long long batch_a, const float* w, int ldw, long long batch_w,
                 const float* bias, float* out, int ldo, long long batch_out, int m, int n, int k,
                 int batch, bool vec, cudaStream_t stream) {
    constexpr int threads = (BM / TM) * (BN / TN);
    constexpr size_t bytes = sizeof(float) * ((size_t)G * 2 * BK * (BM + 4 + BN + 4) + BM * BN +
                                              (G > 1 ? (size_t)G * BM * BN : 0));
    static_assert(bytes <= 227 * 1024, "shared memory");
    const dim3 grid(ceil_div_host(n, BN), ceil_div_host(m, BM), batch);
    MLXONE_REQUIRE(grid.y <= 65535, "gemm_f32: too many rows (%d)", m);
    auto kernel = vec ? gemm_f32_kernel<BM, BN, TM, TN, G, BK, true>
                      : gemm_f32_kernel<BM, BN, TM, TN, G, BK, false>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    kernel<<<grid, threads * G, bytes, stream>>>(a, lda, w, ldw, bias, out, ldo, m, n, k, batch_a, batch_w,
                                                 batch_out);
    MLXONE_LAUNCH_CHECK("gemm_f32");
    return 0;
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

template <int MR>
int launch_skinny(const float* a, int lda, const float* w, int ldw, const float* bias, float* out, int ldo,
                  int m, int n, int k, cudaStream_t stream) {
    constexpr int GROUP = 4 * skinny_rows(MR);
    const int sections = ceil_div_host(k, SECTION);
    const int warps_k = sections >= 8 ? 8 : sections >= 4 ? 4 : sections >= 2 ? 2 : 1;
    const int side = SKINNY_WARPS / warps_k;
    // two blocks an SM; each brings the rows of a into shared memory once for all its rows of w
    const int groups = ceil_div_host(n, GROUP), slots = 2 * sm_count();
    int row_groups = ceil_div_host(groups, slots);
    row_groups = ceil_div_host(row_groups, side) * side;
    // ... up to 32 KB of them at a time (64 KB where eight rows meet eight warps along K)
    const int depth = std::max(warps_k, std::min(ceil_div_host(sections, warps_k) * warps_k,
                                                 32 / MR / warps_k * warps_k));
    const auto bytes = [&](int g) {
        return sizeof(float) * ((size_t)depth * MR * SECTION +
                                SKINNY_WARPS * 32 * (skinny_rows(MR) * MR + 1) +
                                (size_t)g * GROUP * MR * sections);
    };
    while (row_groups > side && bytes(row_groups) > 110 * 1024) row_groups -= side;
    MLXONE_REQUIRE(bytes(row_groups) <= 200 * 1024, "gemm_f32: rows of %d values are too long", k);
    auto kernel = gemm_f32_skinny_kernel<MR>;
    const size_t shared = bytes(row_groups);
    if (shared > 48 * 1024)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    const dim3 grid(ceil_div_host(groups, row_groups), ceil_div_host(m, MR));
    launch_kernel(kernel, grid, dim3(SKINNY_WARPS * 32), shared, stream, true, a, lda, w, ldw, bias, out, ldo,
                  m, n, k, row_groups, warps_k, depth);
    MLXONE_LAUNCH_CHECK("gemm_f32 (few rows)");
    return 0;
}

bool aligned(const void* p, int to) { return reinterpret_cast<uintptr_t>(p) % to == 0; }

// Which kernel. Up to 32 rows: w is what there is to read, and the streaming kernel reads it once per
// eight rows, later times from L2. Its time grows with every eight rows, the tiles' hardly does, so where the
// two meet depends on the matrix. Us streamed / by tiles (with a cold L2) at 9 to 16, 17 to 24 and 25 to 32
// rows: 1024 -> 1024 11 / 30, 13 / 30, 15 / 31; 8192 -> 2048 70 / 166, 96 / 177, 125 / 181; 1536 -> 4608 31 / 42,
// 42 / 43, 48 / 44; 2048 -> 16384 80 / 95, 111 / 98, 140 / 102; 2048 -> 65536 282 / 291, 408 / 308, 537 / 320. One
// line at 32 gains up to 150 us at the long narrow matrices and gives up to 217 away at the widest; a line
// at 16 for matrices of more than about 6,000 rows would have both and is not drawn. With 33 to 64 rows the
// streaming kernel would be behind at all but the smallest matrices. One kernel for all, tiles of 64 x 64 walking K four values a thread at a time,
// took 134 us a product at one row of the 0.35 B shapes and 376 us at 1,200 rows beside decodes of the
// 1.2 B ones. Now, us at 1 / 4 / 8 / 128 / 1,200 rows: 1024 -> 9216 (37.7 MB): 9.8 / 9.4 / 15 / 73 / 547;
// 2048 -> 16384 (134 MB): 25 / 30 / 43 / 222 / 1932 (42 TFLOP/s); 8192 -> 2048: 18 / 26 / 43 / 158 / 1381.
int gemm_f32(const float* a, int lda, long long batch_a, const float* w, int ldw, long long batch_w,
             const float* bias, float* out, int ldo, long long batch_out, int m, int n, int k, int batch,
             cudaStream_t stream) {
    const bool vec = k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && batch_a % 4 == 0 && batch_w % 4 == 0 &&
                     aligned(a, 16) && aligned(w, 16);
    if (batch == 1 && m <= 32 && vec && k % 8 == 0 && ldw % 8 == 0 && aligned(w, 32) && k <= 32768) {
#define ROWS(MR) return launch_skinny<MR>(a, lda, w, ldw, bias, out, ldo, m, n, k, stream)
        if (m == 1) ROWS(1);
        if (m == 2) ROWS(2);
        if (m <= 4) ROWS(4);
        ROWS(8);
#undef ROWS
    }
    // What a tile shape takes, in outputs that an SM works through one after the other: a launch lasts
    // for whole rounds of tiles over the SMs. (Four and eight groups pay for the meeting of their sums.)
    const int sections = ceil_div_host(k, SECTION);
    const auto cost = [&](int bm, int bn, double factor) {
        const long long tiles = (long long)ceil_div_host(m, bm) * ceil_div_host(n, bn) * batch;
        return (double)ceil_div_host(tiles, sm_count()) * bm * bn * factor;
    };
    const double large = cost(128, 128, 1.0), medium = cost(64, 64, sections >= 4 ? 1.1 : 2.2),
                 small = cost(32, 64, sections >= 8 ? 1.2 : sections >= 4 ? 1.6 : 3.2);
#define TILES(...)                                                                                     \
    return launch_tiles<__VA_ARGS__>(a, lda, batch_a, w, ldw, batch_w, bias, out, ldo, batch_out, m, n, k, \
                                     batch, vec, stream)
    if (large <= medium && large <= small) TILES(128, 128, 8, 8, 1, 32);
    if (medium <= small) TILES(64, 64, 8, 8, 4, 16);
    TILES(32, 64, 8, 8, 8, 16);
#undef TILES
}

}  // namespace

MLXONE_API int mlxone_gemm_f32(const float* a, int lda, const float* w, int ldw,
                               const float* bias, float* out, int ldo, int m, int n, int k,
                               cudaStream_t stream) {
    if (m == 0 || n == 0) return 0;
    MLXONE_REQUIRE(m > 0 && n > 0 && k > 0, "gemm_f32: bad sizes m=%d n=%d k=%d", m, n, k);
    MLXONE_REQUIRE(lda >= k && ldw >= k && ldo >= n, "gemm_f32: leading dimension too small");
    return gemm_f32(a, lda, 0, w, ldw, 0, bias, out, ldo, 0, m, n, k, 1, stream);
}

// `batch` products of one shape: product b reads a + b * batch_a and w + b * batch_w and writes
// out + b * batch_out (distances in values). A head-by-head product over rows that hold all
// heads side by side is this with batch_a = the head's width and lda = the row's.
MLXONE_API int mlxone_gemm_f32_batched(const float* a, int lda, long long batch_a, const float* w,
                                       int ldw, long long batch_w, float* out, int ldo,
                                       long long batch_out, int m, int n, int k, int batch,
                                       cudaStream_t stream) {
    if (m == 0 || n == 0 || batch == 0) return 0;
    MLXONE_REQUIRE(m > 0 && n > 0 && k > 0 && batch > 0 && batch <= 65535,
                   "gemm_f32_batched: bad sizes m=%d n=%d k=%d batch=%d", m, n, k, batch);
    MLXONE_REQUIRE(lda >= k && ldw >= k && ldo >= n, "gemm_f32_batched: leading dimension too small");
    return gemm_f32(a, lda, batch_a, w, ldw, batch_w, nullptr, out, ldo, batch_out, m, n, k, batch, stream);
}
