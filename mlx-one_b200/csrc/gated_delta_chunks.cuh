// The gated delta rule over long portions, 32 tokens at a time (keys of 128 values).
//
// With G_t = g_1 .. g_t and D(t, j) = g_(j+1) .. g_t over the tokens of a chunk and S the head's matrix
// before it, the recurrence S_t = g_t S_(t-1) + k_t u_t^T, u_t = beta_t (v_t - g_t S_(t-1)^T k_t) gives
//   r_t = v_t - G_t (S^T k_t)                   u = T diag(beta) r,  T = (1 + A)^-1,
//                                               A(t, j) = beta_t D(t, j) (k_t . k_j) for j < t
//   o_t = G_t (S^T q_t) + sum_(j <= t) D(t, j) (q_t . k_j) u_j
//   S'  = G_32 S + sum_j D(32, j) k_j u_j^T
// (Yang, Kautz, Hatamizadeh, "Gated Delta Networks", 2024: the chunkwise form.) What does not need S,
// the 32 x 32 matrices T diag(beta) and P T diag(beta) with P(t, j) = D(t, j) (q_t . k_j), is worked out for
// all chunks side by side; the walk over the chunks is then three products a chunk and five barriers
// instead of a chain of sums and shuffles per four tokens. All in 32-bit; decays are multiplied up and
// never divided, so a decay of zero is like any other. What is not finite in a token reaches itself and
// later tokens only: above the diagonals nothing is multiplied.
#pragma once

#include "delta_common.cuh"
#include "float_pairs.cuh"

namespace {

constexpr int DC = 32;                    // tokens of a chunk
constexpr int DC_KEY = 128;               // values of a key
constexpr int DC_COLUMNS = 16;            // columns of S of a block of the walk
constexpr int DC_PITCH = DC_KEY + 4, DC_SMALL = DC + 4;
constexpr int DC_THREADS = 256;
// what a chunk and head leave for the walk: T diag(beta), P T diag(beta), G_t, D(32, t)
constexpr int DC_VALUES = 2 * DC * DC + 2 * DC;

// Requests' chunks lie one behind another; every request may leave one place unused, and those of fewer than
// `chunk_from` tokens leave theirs. The first `lead` requests, of one token each, have none.
__host__ __device__ __forceinline__ int chunk_places(int tokens, int requests) { return tokens / DC + requests; }
__device__ __forceinline__ int first_chunk(int first_token, int request, int lead) {
    return (first_token - lead) / DC + request - lead;
}

// 16 bytes, or zeros
__device__ __forceinline__ void copy_or_zero_16(float* dst, const float* src, bool live) {
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(live ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ float4 quad_of(FloatPair a, FloatPair b) {
    float4 v;
    unpair(a, v.x, v.y);
    unpair(b, v.z, v.w);
    return v;
}

// ------------------------------------------------------------------ what does not need S
// One block of DC_THREADS threads per place of a chunk (x) and query/key head (y) (`shared`: DC_PREPARE_SHARED
// bytes). The products of the chunk's k and q with its k: a warp takes 16
// of the 128 values of a key, a lane 8 x 8 products (16 values read from shared memory for 64 FMAs:
// shared memory gives a thread's value for every four FMAs that an SM can do); then a warp per value
// head, lane = column: T by forward substitution in registers, P T behind it. (A and P of up to three
// heads lie where k and q lay, so that two blocks share an SM: room for eight of them beside k and q left
// one: 31 us for 2,048 tokens of 16 heads, 24 now.)
constexpr int DC_SOLVERS = 3;
constexpr size_t DC_PREPARE_SHARED = sizeof(float) * ((size_t)2 * DC * DC_PITCH + 8 * 2 * DC * DC);
static_assert(DC_SOLVERS * 2 * DC * DC_SMALL <= 2 * DC * DC_PITCH, "A and P fit where k and q were");

__device__ __forceinline__ void prepare_chunk(const float* q_in, const float* k_in, const float* coef,
                                              const int* request_start, float* chunks,
                                              const DeltaSizes& sizes, int requests, int lead,
                                              int chunk_from, float* shared) {
    float* kq = shared;                                      // [k of 32 tokens, q of 32][DC_PITCH]
    float* part = kq + 2 * DC * DC_PITCH;                    // [8][64][32]
    __shared__ int place[2];                                 // first token, tokens
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = blockIdx.y;
    const int H = sizes.heads, G = sizes.kv_heads, per_group = H / G;
    if (tid == 0) place[1] = 0;
    __syncthreads();
    for (int r = lead + tid; r < requests; r += DC_THREADS) {
        const int first = request_start[r], count = request_start[r + 1] - first;
        const int c = (int)blockIdx.x - first_chunk(first, r, lead);
        if (count >= chunk_from && c >= 0 && c * DC < count) {
            place[0] = first + c * DC;
            place[1] = min(DC, count - c * DC);
        }
    }
    __syncthreads();
    const int base = place[0], count = place[1];
    if (count == 0) return;
    for (int i = tid; i < 2 * DC * (DC_KEY / 4); i += DC_THREADS) {
        const int row = i / (DC_KEY / 4), e = i % (DC_KEY / 4) * 4, t = row % DC;
        const float* from = (row < DC ? k_in : q_in) + ((size_t)(base + min(t, count - 1)) * G + g) * DC_KEY + e;
        copy_or_zero_16(kq + row * DC_PITCH + e, from, t < count);
    }
    copy_commit();
    copy_wait_for<0>();
    __syncthreads();
    {
        const int rg = lane >> 2, cg = lane & 3;             // rows rg + 8 i, columns cg + 4 j
        float acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll 1
        for (int e = warp * 16; e < warp * 16 + 16; e += 4) {
            float4 x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                x[i] = *reinterpret_cast<const float4*>(kq + (rg + 8 * i) * DC_PITCH + e);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 y = *reinterpret_cast<const float4*>(kq + (cg + 4 * j) * DC_PITCH + e);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    acc[i][j] = fmaf(x[i].x, y.x, acc[i][j]);
                    acc[i][j] = fmaf(x[i].y, y.y, acc[i][j]);
                    acc[i][j] = fmaf(x[i].z, y.z, acc[i][j]);
                    acc[i][j] = fmaf(x[i].w, y.w, acc[i][j]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                part[(warp * 2 * DC + rg + 8 * i) * DC + ((cg + 4 * j) ^ rg)] = acc[i][j];
    }
    __syncthreads();
    // (in place: the first section becomes the sum; its columns stay exchanged by the row's low bits)
    for (int i = tid; i < 2 * DC * DC; i += DC_THREADS) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += part[w * 2 * DC * DC + i];
        part[i] = sum;
    }
    __syncthreads();
    if (warp >= DC_SOLVERS) return;
    float* a = kq + warp * 2 * DC * DC_SMALL;
    float* p = a + DC * DC_SMALL;
    for (int hh = warp; hh < per_group; hh += DC_SOLVERS) {
        const int h = g * per_group + hh;
        float gate = 1.f, beta = 0.f;                        // (behind the portion's end: changes nothing)
        if (lane < count) {
            gate = coef[((size_t)(base + lane) * H + h) * 2];
            beta = coef[((size_t)(base + lane) * H + h) * 2 + 1];
        }
        // lane j: D(t, j) down the rows
        float decay = 0.f, whole = 1.f, mine = 1.f;
        for (int t = 0; t < DC; ++t) {
            const float g_t = __shfl_sync(0xffffffffu, gate, t), beta_t = __shfl_sync(0xffffffffu, beta, t);
            decay = lane == t ? 1.f : decay * g_t;           // zero above the diagonal
            whole *= g_t;
            if (lane == t) mine = whole;
            const float kk = part[t * DC + (lane ^ (t & 7))], qk = part[(DC + t) * DC + (lane ^ (t & 7))];
            a[t * DC_SMALL + lane] = lane < t ? beta_t * decay * kk : 0.f;
            p[t * DC_SMALL + lane] = lane <= t ? decay * qk : 0.f;
        }
        __syncwarp();
        float* out = chunks + ((size_t)blockIdx.x * H + h) * DC_VALUES;
        float column[DC];                                    // T(., lane), then T diag(beta)
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            float sum = lane == t ? 1.f : 0.f;
#pragma unroll
            for (int j = 0; j < t; j += 4) {
                const float4 v = *reinterpret_cast<const float4*>(a + t * DC_SMALL + j);
                sum = fmaf(-v.x, column[j], sum);
                if (j + 1 < t) sum = fmaf(-v.y, column[j + 1], sum);
                if (j + 2 < t) sum = fmaf(-v.z, column[j + 2], sum);
                if (j + 3 < t) sum = fmaf(-v.w, column[j + 3], sum);
            }
            column[t] = sum;
        }
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            // (above the diagonal by selection: a later token's beta may be NaN)
            column[t] = lane <= t ? column[t] * beta : 0.f;
            out[t * DC + lane] = column[t];
        }
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j <= t; j += 4) {
                const float4 v = *reinterpret_cast<const float4*>(p + t * DC_SMALL + j);
                sum = fmaf(v.x, column[j], sum);
                if (j + 1 <= t) sum = fmaf(v.y, column[j + 1], sum);
                if (j + 2 <= t) sum = fmaf(v.z, column[j + 2], sum);
                if (j + 3 <= t) sum = fmaf(v.w, column[j + 3], sum);
            }
            out[(DC + t) * DC + lane] = sum;
        }
        out[2 * DC * DC + lane] = mine;
        out[2 * DC * DC + DC + lane] = decay;                // (after the last row: D(32, lane))
        __syncwarp();
    }
}

// ------------------------------------------------------------------ the walk
// Grid (tiles of 16 columns of S, heads + 1, requests behind the first `lead`), of which those of fewer than
// `chunk_from` tokens are the scan's; blocks with blockIdx.y == heads write the convolution's inputs into the ring. S lies in shared memory (and in the registers of the 128 threads
// that update it). [k; q] S and [T diag(beta); P T diag(beta)] r are products of 64 rows by 16 columns: a
// lane takes 8 x 4 outputs, a warp an eighth of the sum (16 values of a key, 4 tokens), and the eighths
// are added up in order. Bound by the chain of products, barriers and reads of shared memory of a chunk
// (2.6 us; 56 % of the SMs' shared memory reads, 40 % of their FMAs): tiles of 8 columns and twice the
// blocks were 5 to 10 % slower, for 4 heads too. While half the warps update S the other half asks for the
// chunk after next. 2,048 tokens of 16 heads: 170 us (530 by the scan of four tokens at a time).
constexpr int DC_BUFFERS = 3;
constexpr int DC_BUFFER = 2 * DC * DC_PITCH + DC * DC_COLUMNS + 2 * DC * DC_SMALL + 2 * DC;
constexpr size_t DC_WALK_SHARED =
    sizeof(float) * ((size_t)DC_BUFFERS * DC_BUFFER + DC_KEY * DC_COLUMNS + 8 * 2 * DC * DC_COLUMNS + 2 * DC * DC_COLUMNS);

// part[warp][64][16] = x[64 rows, 4 STEPS columns from e0] * y[4 STEPS rows, 16 columns]. LOWER: x is two
// matrices of 32 rows that are zero above the diagonal (`column`: where its first column here stands), and
// what stands there meets nothing of y.
template <int STEPS, bool LOWER = false>
__device__ __forceinline__ void chunk_product(const float* x, int pitch, const float* y, float* part,
                                              int column = 0) {
    const int lane = threadIdx.x & 31, rg = lane >> 2, cg = lane & 3;
    FloatPair acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0;
#pragma unroll
    for (int step = 0; step < STEPS; ++step) {
        ulonglong2 b[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            b[e] = *reinterpret_cast<const ulonglong2*>(y + (step * 4 + e) * DC_COLUMNS + cg * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(x + (rg + 8 * i) * pitch + step * 4);
            const float values[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (LOWER && column + step * 4 + e > (rg + 8 * i) % DC) continue;
                const FloatPair f = pair_of(values[e]);
                accumulate_pair(acc[i][0], f, b[e].x);
                accumulate_pair(acc[i][1], f, b[e].y);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(part + (rg + 8 * i) * DC_COLUMNS + cg * 4) = quad_of(acc[i][0], acc[i][1]);
}

template <typename T>
__global__ void __launch_bounds__(DC_THREADS)
delta_walk_kernel(const float* q_in, const float* k_in, const float* v_in, const float* chunks,
                  const T* __restrict__ projected, float* state, const int* __restrict__ slots,
                  const int* __restrict__ request_start, const int* __restrict__ history, float* out,
                  DeltaSizes sizes, int lead, int chunk_from, int write, int ld) {
    extern __shared__ __align__(16) float shared[];
    float* matrix_s = shared + DC_BUFFERS * DC_BUFFER;       // S [128][16]
    float* part = matrix_s + DC_KEY * DC_COLUMNS;            // [8][64][16]
    float* rest = part + 8 * 2 * DC * DC_COLUMNS;            // r [32][16]
    float* moved = rest + DC * DC_COLUMNS;                   // D(32, t) u_t [32][16]
    const int tid = threadIdx.x, warp = tid >> 5, r = lead + blockIdx.z;
    griddep_wait();
    const int first = request_start[r], last = request_start[r + 1];
    if (last - first < chunk_from) return;
    const int H = sizes.heads, G = sizes.kv_heads, V = sizes.value_dim;
    float* slot = state + (size_t)slots[r] * sizes.state();
    if ((int)blockIdx.y == H) {
        griddep_launch();
        if (!write) return;
        const int channels = sizes.channels(), taps = sizes.taps;
        const int n = last - first, kept = min(n, taps);
        float* ring = slot + sizes.matrices();
        for (int c = blockIdx.x * blockDim.x + tid; c < channels; c += gridDim.x * blockDim.x)
            for (int index = n - kept; index < n; ++index)
                ring[(size_t)((history[r] + index) % taps) * channels + c] =
                    to_float<T>(projected[(size_t)(first + index) * ld + c]);
        return;
    }
    const int h = blockIdx.y, g = h / (H / G), column0 = blockIdx.x * DC_COLUMNS;
    // the chunk's operands into its buffer, by `count_of` threads of which this is number `me`; a group of
    // copies even where there is no such chunk
    auto fetch = [&](int chunk, int me, int count_of) {
        if (first + chunk * DC >= last) { copy_commit(); return; }
        float* to = shared + chunk % DC_BUFFERS * DC_BUFFER;
        const int base = first + chunk * DC, count = min(DC, last - base);
        for (int i = me; i < 2 * DC * (DC_KEY / 4); i += count_of) {
            const int row = i / (DC_KEY / 4), e = i % (DC_KEY / 4) * 4, t = row % DC;
            copy_or_zero_16(to + row * DC_PITCH + e,
                            (row < DC ? k_in : q_in) + ((size_t)(base + min(t, count - 1)) * G + g) * DC_KEY + e,
                            t < count);
        }
        to += 2 * DC * DC_PITCH;
        if (me < DC * (DC_COLUMNS / 4)) {
            const int t = me / (DC_COLUMNS / 4), c = me % (DC_COLUMNS / 4) * 4;
            copy_or_zero_16(to + t * DC_COLUMNS + c,
                            v_in + ((size_t)(base + min(t, count - 1)) * H + h) * V + column0 + c, t < count);
        }
        to += DC * DC_COLUMNS;
        const float* from = chunks + ((size_t)(first_chunk(first, r, lead) + chunk) * H + h) * DC_VALUES;
        for (int i = me; i < 2 * DC * (DC / 4); i += count_of) {
            const int row = i / (DC / 4), e = i % (DC / 4) * 4;
            copy_or_zero_16(to + row * DC_SMALL + e, from + row * DC + e, true);
        }
        to += 2 * DC * DC_SMALL;
        if (me < 2 * DC / 4) copy_or_zero_16(to + me * 4, from + 2 * DC * DC + me * 4, true);
        copy_commit();
    };
    const int total = (last - first + DC - 1) / DC;
    fetch(0, tid, DC_THREADS);
    fetch(1, tid, DC_THREADS);
    // S: thread t < 128 keeps rows 4 (t / 4) .. + 3 of columns 4 (t % 4) .. + 3
    const int own_row = tid / 4 * 4, own_column = tid % 4 * 4;
    float* matrix = slot + (size_t)h * DC_KEY * V + column0;
    FloatPair S[4][2];
    if (tid < 128) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* from = matrix + (size_t)(own_row + i) * V + own_column;
            S[i][0] = pair_of(from[0], from[1]);
            S[i][1] = pair_of(from[2], from[3]);
            *reinterpret_cast<float4*>(matrix_s + (own_row + i) * DC_COLUMNS + own_column) =
                quad_of(S[i][0], S[i][1]);
        }
    }
    // sums of the eighths: thread t adds up four columns of row t / 4
    const int row = tid / 4;
    auto gather = [&]() {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const float4 v =
                *reinterpret_cast<const float4*>(part + (w * 2 * DC + row) * DC_COLUMNS + own_column);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        return sum;
    };
    for (int chunk = 0; chunk < total; ++chunk) {
        const float* kq = shared + chunk % DC_BUFFERS * DC_BUFFER;
        const float* vs = kq + 2 * DC * DC_PITCH;
        const float* small = vs + DC * DC_COLUMNS;
        const float* decays = small + 2 * DC * DC_SMALL;     // G_t, D(32, t)
        copy_wait_for<1>();                                  // (the chunk behind this one may be under way)
        __syncthreads();
        chunk_product<4>(kq + warp * 16, DC_PITCH, matrix_s + warp * 16 * DC_COLUMNS,
                         part + warp * 2 * DC * DC_COLUMNS);
        __syncthreads();
        float4 with_q = gather();                            // (rows of k: becomes r)
        const float before = decays[row % DC];
        bool finite = true;
        if (row < DC) {
            const float4 v = *reinterpret_cast<const float4*>(vs + row * DC_COLUMNS + own_column);
            const float4 r = make_float4(fmaf(-before, with_q.x, v.x), fmaf(-before, with_q.y, v.y),
                                         fmaf(-before, with_q.z, v.z), fmaf(-before, with_q.w, v.w));
            finite = isfinite(r.x) && isfinite(r.y) && isfinite(r.z) && isfinite(r.w);
            *reinterpret_cast<float4*>(rest + row * DC_COLUMNS + own_column) = r;
        }
        // (zero times an infinity or NaN of a later token would reach the tokens before it)
        if (__syncthreads_and(finite))
            chunk_product<1>(small + warp * 4, DC_SMALL, rest + warp * 4 * DC_COLUMNS,
                             part + warp * 2 * DC * DC_COLUMNS);
        else
            chunk_product<1, true>(small + warp * 4, DC_SMALL, rest + warp * 4 * DC_COLUMNS,
                                   part + warp * 2 * DC * DC_COLUMNS, warp * 4);
        __syncthreads();
        const float4 sum = gather();
        if (row < DC) {
            const float after = decays[DC + row];
            *reinterpret_cast<float4*>(moved + row * DC_COLUMNS + own_column) =
                make_float4(after * sum.x, after * sum.y, after * sum.z, after * sum.w);
        } else if (first + chunk * DC + row - DC < last) {
            float* to = out + ((size_t)(first + chunk * DC + row - DC) * H + h) * V + column0 + own_column;
            *reinterpret_cast<float4*>(to) =
                make_float4(fmaf(before, with_q.x, sum.x), fmaf(before, with_q.y, sum.y),
                            fmaf(before, with_q.z, sum.z), fmaf(before, with_q.w, sum.w));
        }
        __syncthreads();
        if (tid < 128) {
            // (half the warps, the other half asks for the chunk after next meanwhile)
            const FloatPair whole = pair_of(decays[DC - 1]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) S[i][j] = mul_pair(S[i][j], whole);
#pragma unroll 8
            for (int t = 0; t < DC; ++t) {
                const float4 k = *reinterpret_cast<const float4*>(kq + t * DC_PITCH + own_row);
                const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(moved + t * DC_COLUMNS + own_column);
                const FloatPair ks[4] = {pair_of(k.x), pair_of(k.y), pair_of(k.z), pair_of(k.w)};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    accumulate_pair(S[i][0], ks[i], u.x);
                    accumulate_pair(S[i][1], ks[i], u.y);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<float4*>(matrix_s + (own_row + i) * DC_COLUMNS + own_column) =
                    quad_of(S[i][0], S[i][1]);
            copy_commit();                                   // (groups are counted thread by thread)
        } else {
            fetch(chunk + 2, tid - 128, 128);
        }
    }
    griddep_launch();
    if (write && tid < 128) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 v = quad_of(S[i][0], S[i][1]);
            float* to = matrix + (size_t)(own_row + i) * V + own_column;
            to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w;
        }
    }
}

}  // namespace
