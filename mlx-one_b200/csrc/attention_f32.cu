// Paged grouped-query attention of the 32-bit engine: head sizes 32, 64 and 128, every earlier key
// visible, no sinks (the general kernel takes the rest).
//
// The query at position p reads the keys 0 .. p of its request. Keys are taken in units of 64,
// aligned to absolute positions: scores (one FMA chain over the head's values), the unit's maximum,
// weights, their sum and the weighted values (one FMA chain over the unit's keys); the units are then
// joined in ascending order by the online softmax. So the order of operations for a query depends
// only on its position, never on how the tokens were cut into steps or batched, nor on whether the
// units were computed by one block or by many.
//
// A block holds 8 * RPT rows, a row being one (token, query head), all of one key head, and reads
// each unit's keys and values once for all of them, 16 bytes a thread. RPT = 4 (32 rows: 8 tokens
// of 4 heads) for portions, RPT = 1 for single tokens. SPLIT: a block computes one unit, and a merge
// kernel joins them: taken where there would be too few blocks to keep the chip busy. (One warp per
// query and head, which reads every key for itself by a lane per key, 4-byte loads a head apart: 188
// us a launch for one token behind 140 keys, 760 us for four prompts of 300; now 8 and 110. With the
// rows looked up by every thread for itself and all loads behind the wait 12.5 and 130.)
#include "common.cuh"

namespace {

constexpr int UNIT = 64, THREADS = 128;

__device__ __forceinline__ uint32_t shared_address(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void copy16(float* to, const float* from, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(shared_address(to)), "l"(from),
                 "r"(live ? 16 : 0));
}
__device__ __forceinline__ float half_max(float v) {            // over 16 lanes
#pragma unroll
    for (int offset = 8; offset > 0; offset >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, offset));
    return v;
}
__device__ __forceinline__ float half_sum(float v) {
#pragma unroll
    for (int offset = 8; offset > 0; offset >>= 1) v += __shfl_xor_sync(0xffffffffu, v, offset);
    return v;
}

// Joins a unit (maximum, sum, and a value of its weighted sum) to what has been joined so far.
struct Joint {
    float keep, take, max;
    __device__ __forceinline__ Joint(float max_so_far, float unit_max) {
        max = fmaxf(max_so_far, unit_max);
        keep = expf(max_so_far - max);                          // 0 when nothing was joined yet
        take = expf(unit_max - max);
    }
    __device__ __forceinline__ float operator()(float so_far, float unit) const {
        return __fmaf_rn(unit, take, __fmul_rn(so_far, keep));
    }
};

template <int D, int RPT, bool SPLIT>
__global__ void __launch_bounds__(THREADS)
attention_f32_kernel(const float* q, const float* kv, const int* block_table, int table_width, int page_size,
                     long long kv_half, const int* positions, const int* token_request, float* out,
                     float* partial, int units, int first_token, int end_token, int tile_tokens, int heads,
                     int kv_heads, float scale, int* error_flag) {
    constexpr int ROWS = 8 * RPT, PAD = D + 4, DIMS = D / 16;
    extern __shared__ __align__(16) float shared[];
    float* keys = shared;                             // [UNIT][PAD]
    float* values = keys + UNIT * PAD;                // [UNIT][D]
    float* queries = values + UNIT * D;               // [ROWS][PAD]
    float* weights = queries + ROWS * PAD;            // [ROWS][UNIT + 1]
    __shared__ long long row_of[UNIT];                // where a key's row lies, -1: its position has no page
    const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;
    const int group = heads / kv_heads, kv_head = blockIdx.y;
    const int token0 = first_token + blockIdx.x * tile_tokens;
    const int tokens_here = min(tile_tokens, end_token - token0);

    // the rows of a unit's keys, looked up once; then keys low .. high - 1 of it, 16 bytes a thread
    auto look_up = [&](const int* table, int base, int last) {
        if (tid < UNIT) {
            const int key = base + tid;
            long long at = -1;
            if (key <= last) {
                const int block = key / page_size;
                const int page = block < table_width ? __ldcg(table + block) : -1;
                if (page < 0) atomicExch(error_flag, 3);
                else at = (((long long)page * kv_heads + kv_head) * page_size + key % page_size) * D;
            }
            row_of[tid] = at;
        }
        __syncthreads();
    };
    auto bring = [&](int low, int high) {
        for (int i = low * (D / 4) + tid; i < high * (D / 4); i += THREADS) {
            const int j = i / (D / 4), e = i % (D / 4) * 4;
            const long long at = row_of[j];
            const float* from = at >= 0 ? kv + at + e : kv;
            copy16(keys + j * PAD + e, from, at >= 0);
            copy16(values + j * D + e, at >= 0 ? from + kv_half : kv, at >= 0);
        }
    };
    // A single token's first unit: all keys but its own lie in the pages since earlier steps, so they are
    // asked for ahead of the wait for the kernel that writes that one (positions and tables are older still).
    bool ahead = false;
    if (RPT == 1) {
        const int last = __ldcg(positions + token0), base = SPLIT ? (int)blockIdx.z * UNIT : 0;
        ahead = base <= last;
        if (ahead) {
            look_up(block_table + (size_t)__ldcg(token_request + token0) * table_width, base, last);
            bring(0, min(last - base, UNIT));
        }
        griddep_wait();
        if (ahead) bring(min(last - base, UNIT), UNIT);
    } else {
        griddep_wait();
    }
    griddep_launch();

    // rows: row = (token of the tile) * group + head of the group
    const int rows = tokens_here * group;
    for (int i = tid; i < ROWS * D; i += THREADS) {
        const int row = i / D, e = i % D;
        queries[row * PAD + e] =
            row < rows ? __ldcg(q + ((size_t)(token0 + row / group) * heads + kv_head * group + row % group) * D +
                                e) * scale
                       : 0.f;
    }
    int position[RPT], request[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = ty * RPT + i;
        position[i] = row < rows ? __ldcg(positions + token0 + row / group) : -1;
        request[i] = row < rows ? __ldcg(token_request + token0 + row / group) : -1;
    }
    float max_so_far[RPT], sum[RPT], acc[RPT][DIMS];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        max_so_far[i] = -INFINITY;
        sum[i] = 0.f;
#pragma unroll
        for (int d = 0; d < DIMS; ++d) acc[i][d] = 0.f;
    }

    // the tile's tokens in runs of one request
    for (int run = 0; run < tokens_here;) {
        const int r = __ldcg(token_request + token0 + run);
        int run_end = run, last = -1;
        while (run_end < tokens_here && __ldcg(token_request + token0 + run_end) == r) {
            last = max(last, __ldcg(positions + token0 + run_end));
            ++run_end;
        }
        run = run_end;
        const int* table = block_table + (size_t)r * table_width;
        const int first_unit = SPLIT ? blockIdx.z : 0;
        const int end_unit = SPLIT ? min(first_unit + 1, last / UNIT + 1) : last / UNIT + 1;
        for (int unit = first_unit; unit < end_unit; ++unit) {
            const int base = unit * UNIT;
            if (!ahead || unit != first_unit) {
                __syncthreads();                      // the unit before has been read
                look_up(table, base, last);
                bring(0, UNIT);
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();

            float score[RPT][4];
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int c = 0; c < 4; ++c) score[i][c] = 0.f;
#pragma unroll 4
            for (int e = 0; e < D; e += 4) {
                float4 x[RPT];
#pragma unroll
                for (int i = 0; i < RPT; ++i)
                    x[i] = *reinterpret_cast<const float4*>(queries + (ty * RPT + i) * PAD + e);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 y = *reinterpret_cast<const float4*>(keys + (tx + 16 * c) * PAD + e);
#pragma unroll
                    for (int i = 0; i < RPT; ++i) {
                        score[i][c] = fmaf(x[i].x, y.x, score[i][c]);
                        score[i][c] = fmaf(x[i].y, y.y, score[i][c]);
                        score[i][c] = fmaf(x[i].z, y.z, score[i][c]);
                        score[i][c] = fmaf(x[i].w, y.w, score[i][c]);
                    }
                }
            }
            // (keys of this unit that a row sees: those below `seen`, on the request of this run; what a
            // row that sees none of them computes here is dropped)
            int seen[RPT];
            float unit_max[RPT], unit_sum[RPT];
            bool whole = true;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                seen[i] = request[i] == r ? min(max(position[i] - base + 1, 0), UNIT) : 0;
                whole = whole && (seen[i] == UNIT || seen[i] == 0);
                float most = -INFINITY;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int j = tx + 16 * c;
                    if (j >= seen[i] || row_of[j] < 0) score[i][c] = -INFINITY;
                    most = fmaxf(most, score[i][c]);
                }
                unit_max[i] = half_max(most);
                float total = 0.f;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int j = tx + 16 * c;
                    // (a maximum of nothing but NaN is -inf too: the weights stay NaN)
                    const bool live = j < seen[i] && row_of[j] >= 0;
                    const float weight =
                        live ? expf(score[i][c] - (unit_max[i] == -INFINITY ? 0.f : unit_max[i])) : 0.f;
                    weights[(ty * RPT + i) * (UNIT + 1) + j] = weight;
                    total += weight;
                }
                unit_sum[i] = half_sum(total);
            }
            __syncwarp();                             // (a row's weights are its own half-warp's)
            float mixed[RPT][DIMS];
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int d = 0; d < DIMS; ++d) mixed[i][d] = 0.f;
            auto add = [&](int j, bool all) {
                float v[DIMS];
                const float* from = values + j * D + tx * DIMS;
                if constexpr (DIMS % 4 == 0) {
#pragma unroll
                    for (int d = 0; d < DIMS; d += 4)
                        *reinterpret_cast<float4*>(v + d) = *reinterpret_cast<const float4*>(from + d);
                } else {
#pragma unroll
                    for (int d = 0; d < DIMS; d += 2)
                        *reinterpret_cast<float2*>(v + d) = *reinterpret_cast<const float2*>(from + d);
                }
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const float weight = weights[(ty * RPT + i) * (UNIT + 1) + j];
                    // (a key that a row does not see never meets its sum: its value may be infinite)
                    if (all || j < seen[i]) {
#pragma unroll
                        for (int d = 0; d < DIMS; ++d) mixed[i][d] = fmaf(weight, v[d], mixed[i][d]);
                    }
                }
            };
            if (whole) {
#pragma unroll 8
                for (int j = 0; j < UNIT; ++j) add(j, true);
            } else {
                const int some = min(UNIT, last - base + 1);
#pragma unroll 4
                for (int j = 0; j < some; ++j) add(j, false);
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                if (SPLIT) {
                    const int row = ty * RPT + i;
                    if (request[i] == r && position[i] >= base) {
                        const size_t item = (size_t)(token0 - first_token + row / group) * heads +
                                            kv_head * group + row % group;
                        float* to = partial + (item * units + unit) * (D + 4);
#pragma unroll
                        for (int d = 0; d < DIMS; ++d) to[tx * DIMS + d] = mixed[i][d];
                        if (tx == 0) { to[D] = unit_max[i]; to[D + 1] = unit_sum[i]; }
                    }
                } else if (seen[i] > 0 && fmaxf(max_so_far[i], unit_max[i]) != -INFINITY) {
                    const Joint join(max_so_far[i], unit_max[i]);
                    max_so_far[i] = join.max;
                    sum[i] = join(sum[i], unit_sum[i]);
#pragma unroll
                    for (int d = 0; d < DIMS; ++d) acc[i][d] = join(acc[i][d], mixed[i][d]);
                }
            }
        }
    }
    if (!SPLIT) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int row = ty * RPT + i;
            if (row >= rows) continue;
            float* to = out + ((size_t)(token0 + row / group) * heads + kv_head * group + row % group) * D;
            const float inverse = sum[i] > 0.f ? 1.f / sum[i] : 0.f;
#pragma unroll
            for (int d = 0; d < DIMS; ++d) to[tx * DIMS + d] = acc[i][d] * inverse;
        }
    }
}

// One block of D threads per (token, head). A position behind the units that were launched raises the
// error flag, as a key without a page does.
template <int D>
__global__ void __launch_bounds__(D) attention_f32_merge_kernel(const float* partial, const int* positions,
                                                                float* out, int units, int first_token,
                                                                int heads, int* error_flag) {
    griddep_wait();
    griddep_launch();
    const int item = blockIdx.x, d = threadIdx.x;
    const int seen = __ldcg(positions + first_token + item / heads) / UNIT + 1, count = min(seen, units);
    if (seen > units && d == 0) atomicExch(error_flag, 3);
    const float* from = partial + (size_t)item * units * (D + 4);
    float max_so_far = -INFINITY, sum = 0.f, acc = 0.f;
#pragma unroll 4
    for (int unit = 0; unit < count; ++unit, from += D + 4) {
        const float value = __ldcg(from + d), unit_max = __ldcg(from + D), unit_sum = __ldcg(from + D + 1);
        const Joint join(max_so_far, unit_max);
        if (join.max == -INFINITY) continue;
        max_so_far = join.max;
        sum = join(sum, unit_sum);
        acc = join(acc, value);
    }
    out[((size_t)first_token * heads + item) * D + d] = acc * (sum > 0.f ? 1.f / sum : 0.f);
}

struct Arguments {
    const float *q, *kv;
    const int* table;
    int table_width, page_size;
    long long kv_half;
    const int *positions, *token_request;
    float *out, *partial;
    int units, heads, kv_heads;
    float scale;
    int* error_flag;
    cudaStream_t stream;
};

template <int D, int RPT, bool SPLIT>
void launch(const Arguments& x, int first, int end, int tile_tokens) {
    constexpr int ROWS = 8 * RPT;
    constexpr size_t bytes = sizeof(float) * (UNIT * (D + 4) + UNIT * D + ROWS * (D + 4) + ROWS * (UNIT + 1));
    auto kernel = attention_f32_kernel<D, RPT, SPLIT>;
    if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    const dim3 grid(ceil_div_host(end - first, tile_tokens), x.kv_heads, SPLIT ? x.units : 1);
    launch_kernel(kernel, grid, dim3(THREADS), bytes, x.stream, true, x.q, x.kv, x.table, x.table_width,
                  x.page_size, x.kv_half, x.positions, x.token_request, x.out, x.partial, x.units, first, end,
                  tile_tokens, x.heads, x.kv_heads, x.scale, x.error_flag);
    if (SPLIT)
        launch_kernel(attention_f32_merge_kernel<D>, dim3((end - first) * x.heads), dim3(D), 0, x.stream, true,
                      x.partial, x.positions, x.out, x.units, first, x.heads, x.error_flag);
}

template <int D>
void launch_part(const Arguments& x, int first, int end, bool single, bool split) {
    const int group = x.heads / x.kv_heads;
    const int tile_tokens = single ? 1 : 32 / group;
    if (single && group <= 8) {
        if (split) launch<D, 1, true>(x, first, end, tile_tokens);
        else launch<D, 1, false>(x, first, end, tile_tokens);
    } else {
        if (split) launch<D, 4, true>(x, first, end, tile_tokens);
        else launch<D, 4, false>(x, first, end, tile_tokens);
    }
}

}  // namespace

MLXONE_API int mlxone_attention_f32_supports(int head_dim, int heads, int kv_heads) {
    return (head_dim == 32 || head_dim == 64 || head_dim == 128) && kv_heads > 0 && kv_heads <= 65535 &&
           heads % kv_heads == 0 && heads / kv_heads <= 32;
}

// The tokens first .. end - 1 of a step. `single`: each of them is its request's only one. `units`: 0,
// or an upper bound of the units of 64 keys that a token reads (one that reads more raises the error flag);
// then a block computes one unit and `partial` holds (end - first) * heads * units * (head_dim + 4) values.
MLXONE_API int mlxone_attention_f32(const float* q, const float* kv, const int* block_table, int table_width,
                                    int page_size, int pages, const int* positions, const int* token_request,
                                    float* out, float* partial, int first, int end, int single, int units,
                                    int heads, int kv_heads, int head_dim, float scale, int* error_flag,
                                    cudaStream_t stream) {
    if (end <= first) return 0;
    MLXONE_REQUIRE(first >= 0 && mlxone_attention_f32_supports(head_dim, heads, kv_heads),
                   "attention: %d heads over %d key heads of size %d", heads, kv_heads, head_dim);
    MLXONE_REQUIRE(page_size > 0 && pages > 0 && table_width > 0, "attention: bad page geometry");
    MLXONE_REQUIRE(units >= 0 && units <= 65535 && (units == 0 || partial != nullptr),
                   "attention: bad number of parts (%d)", units);
    MLXONE_REQUIRE((((uintptr_t)kv) & 15) == 0, "attention: pages must be aligned to 16 bytes");
    const Arguments x{q, kv, block_table, table_width, page_size,
                      (long long)pages * kv_heads * page_size * head_dim, positions, token_request, out,
                      partial, units, heads, kv_heads, scale, error_flag, stream};
    if (head_dim == 32) launch_part<32>(x, first, end, single != 0, units > 0);
    else if (head_dim == 64) launch_part<64>(x, first, end, single != 0, units > 0);
    else launch_part<128>(x, first, end, single != 0, units > 0);
    MLXONE_LAUNCH_CHECK("attention_f32");
    return 0;
}
