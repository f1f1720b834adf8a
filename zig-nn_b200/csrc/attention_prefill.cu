// Attention of a prompt's tokens over the f32 cache, in the arithmetic order of gqa_cached_attention / cached_attention
// (src/models/gemma3.zig:1062-1120, src/models/gpt2.zig:796-849): the same roundings as one row at a time through
// attention_scores_step_kernel and attention_softmax_v_step_kernel (ops.cu), so the results are the same bits.
//
// A CTA owns 16 (short prompts: 4) consecutive tokens of one head. Row at a time, every token read all of its keys and
// values through L2 and its scores went through memory; here a tile of 64 keys (or its values) comes into shared memory once
// for all of them, by cp.async one tile ahead, and the scores stay in shared memory from the dots to the weighted sum. What
// bounds it: the separate multiplies and adds of the prescribed order (no FMA, no tensor cores) and the shared-memory reads
// that feed them, which is why a lane holds up to 2 tokens x 2 keys in the dots and a thread up to 8 tokens of one dimension
// in the sum; for a prompt of a few dozen tokens the latency of one CTA's chains, which is why such a prompt is cut finer.
// Measured (B200, row-at-a-time kernels before, shares of a whole prompt): GPT-2, 900 tokens, 14.7 -> 8.4 ms; Gemma-3-1B, 600
// tokens, 23 -> 14 ms (with chunks of 512 in place of 128).
#include "zq_internal.h"

namespace zq {
namespace {

constexpr uint32_t kKeys = 64;  // keys per tile of the dots

__device__ __forceinline__ float exp_f32(float x) { return (float)exp((double)x); }

// quantize_row_q8 (src/gguf/simd_dot.zig:17-43) of the 32 values held one per lane of a warp.
__device__ __forceinline__ void quantize_block_warp(float v, size_t blk, uint32_t lane, int8_t* __restrict__ q,
                                                    float* __restrict__ scale, int32_t* __restrict__ sum) {
    float amax = fabsf(v);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, off));
    const float s = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
    const float inv = __fdiv_rn(1.0f, s);
    float r = roundf(__fmul_rn(v, inv));
    r = fminf(127.0f, fmaxf(-127.0f, r));
    const int qi = (int)r;
    int acc = qi;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, off);
    q[blk * 32 + lane] = (int8_t)qi;
    if (lane == 0) {
        scale[blk] = s;
        sum[blk] = acc;
    }
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

template <int HD, int ROWS>  // ROWS: tokens per CTA
struct PrefillShape {
    static constexpr uint32_t kThreads = ROWS == 16 && HD > 64 ? 512 : 256;
    static constexpr uint32_t kKeysLane = ROWS == 16 && kThreads == 256 ? 2 : 1;  // keys of a lane in the dots
    static constexpr uint32_t kRowsWarp = ROWS * kKeys / (kThreads * kKeysLane);  // and tokens
    static constexpr uint32_t kWarpsRow = kKeys / (32 * kKeysLane);               // warps that share these tokens
    static constexpr uint32_t kDims = HD < 128 ? HD : 128;      // dimensions of a key tile
    static constexpr uint32_t kParts = HD / kDims;              // key tiles per 64 keys
    static constexpr uint32_t kPitch = kDims + 4;               // 128-bit reads of 8 neighbouring keys cover all banks
    static constexpr uint32_t kTile = kKeys * kPitch;           // floats
    static constexpr uint32_t kValues = kKeys * kDims / HD;     // positions of a value tile, in the same room
    static constexpr uint32_t kPerThread = ROWS * HD / kThreads;  // tokens of one dimension per thread
    static_assert(kThreads / 32 / kWarpsRow * kRowsWarp == ROWS && kPerThread >= 1, "a warp's share of the dots");
};

struct PrefillArgs {
    const float* q;
    const float* kc;
    const float* vc;
    float* out;
    int8_t* oq;
    float* oscale;
    int32_t* osum;
    const uint32_t* state;  // [1]: position of token 0
    uint32_t n_head, group, kv_dim, rows, window, q_stride, pitch;  // pitch: floats of a score row
    int gpt2_tail;
};

template <int HD, int ROWS>
__global__ void __launch_bounds__(PrefillShape<HD, ROWS>::kThreads)
attention_prefill_kernel(PrefillArgs a) {
    using S = PrefillShape<HD, ROWS>;
    constexpr uint32_t kRows = ROWS, T = S::kThreads, RW = S::kRowsWarp, KL = S::kKeysLane;
    extern __shared__ __align__(16) float sm[];
    float* tile = sm;                             // two tiles
    float* qs = tile + 2 * S::kTile;              // [ROWS][HD]
    float* w = qs + kRows * HD;                   // [ROWS][pitch]: scores, then weights, of positions lo + ...
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t h = blockIdx.y, kvh = h / a.group;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t pos0 = a.state[1];
    const uint32_t t0 = (gridDim.x - 1 - blockIdx.x) * kRows;  // the longest rows first
    const uint32_t n = min(kRows, a.rows - t0);
    // token t0 + r attends to positions [first(r), last(r)); rows past the end repeat the last one
    auto last = [&](uint32_t r) { return pos0 + t0 + min(r, n - 1) + 1; };
    auto first = [&](uint32_t r) {
        const uint32_t e = last(r);
        return (a.window && e > a.window) ? e - a.window : 0u;
    };
    const uint32_t lo = first(0), hi = last(kRows - 1);
    const float* kbase = a.kc + (size_t)kvh * HD;
    const float* vbase = a.vc + (size_t)kvh * HD;

    for (uint32_t i = tid; i < kRows * (HD / 4); i += T) {
        const uint32_t r = min(i / (HD / 4), n - 1), c = i % (HD / 4);
        const float* from = a.q + (size_t)(t0 + r) * a.q_stride + (size_t)h * HD + c * 4;
        reinterpret_cast<float4*>(qs)[i] = *reinterpret_cast<const float4*>(from);
    }
    // ---- dots: 16 lane sums over the dimensions (dimension mod 16), added in order
    const uint32_t n_key_tiles = (hi - lo + kKeys - 1) / kKeys * S::kParts;
    auto fetch_keys = [&](uint32_t i) {
        if (i < n_key_tiles) {
            const uint32_t p0 = lo + i / S::kParts * kKeys, part = i % S::kParts;
            float* to = tile + (i & 1u) * S::kTile;
            for (uint32_t j = tid; j < kKeys * (S::kDims / 4); j += T) {
                const uint32_t k = j / (S::kDims / 4), c = j % (S::kDims / 4);
                const uint32_t p = min(p0 + k, hi - 1);  // keys past the end repeat the last one; nothing reads their scores
                cp_async16(to + k * S::kPitch + c * 4, kbase + (size_t)p * a.kv_dim + part * S::kDims + c * 4);
            }
        }
        cp_commit();
    };
    const uint32_t r0 = warp / S::kWarpsRow * RW, key0 = warp % S::kWarpsRow * 32 * KL + lane;
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)HD));
    float acc[RW][KL][16];
    fetch_keys(0);
#pragma unroll 1
    for (uint32_t i = 0; i < n_key_tiles; ++i) {
        fetch_keys(i + 1);
        cp_wait_1();
        __syncthreads();
        const uint32_t p0 = lo + i / S::kParts * kKeys, part = i % S::kParts;
        if (p0 < last(r0 + RW - 1) && p0 + kKeys > first(r0)) {
            if (part == 0) {
#pragma unroll
                for (uint32_t r = 0; r < RW; ++r)
#pragma unroll
                    for (uint32_t k = 0; k < KL; ++k)
#pragma unroll
                        for (int l = 0; l < 16; ++l) acc[r][k][l] = 0.0f;
            }
            const float* k0 = tile + (i & 1u) * S::kTile + key0 * S::kPitch;
            const float* q0 = qs + r0 * HD + part * S::kDims;
#pragma unroll 2
            for (uint32_t d = 0; d < S::kDims; d += 16) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float4 kv[KL], qv[RW];
#pragma unroll
                    for (uint32_t k = 0; k < KL; ++k)
                        kv[k] = *reinterpret_cast<const float4*>(k0 + k * 32 * S::kPitch + d + 4 * c);
#pragma unroll
                    for (uint32_t r = 0; r < RW; ++r) qv[r] = *reinterpret_cast<const float4*>(q0 + r * HD + d + 4 * c);
#pragma unroll
                    for (uint32_t r = 0; r < RW; ++r)
#pragma unroll
                        for (uint32_t k = 0; k < KL; ++k) {
                            float* s = acc[r][k] + 4 * c;
                            s[0] = __fadd_rn(s[0], __fmul_rn(qv[r].x, kv[k].x));
                            s[1] = __fadd_rn(s[1], __fmul_rn(qv[r].y, kv[k].y));
                            s[2] = __fadd_rn(s[2], __fmul_rn(qv[r].z, kv[k].z));
                            s[3] = __fadd_rn(s[3], __fmul_rn(qv[r].w, kv[k].w));
                        }
                }
            }
            if (part == S::kParts - 1) {
#pragma unroll
                for (uint32_t r = 0; r < RW; ++r)
#pragma unroll
                    for (uint32_t k = 0; k < KL; ++k) {
                        float s = acc[r][k][0];
#pragma unroll
                        for (int l = 1; l < 16; ++l) s = __fadd_rn(s, acc[r][k][l]);
                        w[(r0 + r) * a.pitch + (p0 - lo) + k * 32 + key0] = __fmul_rn(s, scale);
                    }
            }
        }
        __syncthreads();  // this tile is overwritten by the copies of the next round
    }

    // ---- values: the first tile is on its way during the softmax
    const uint32_t n_value_tiles = (hi - lo + S::kValues - 1) / S::kValues;
    auto fetch_values = [&](uint32_t i) {
        if (i < n_value_tiles) {
            float* to = tile + (i & 1u) * S::kTile;
            for (uint32_t j = tid; j < S::kValues * (HD / 4); j += T) {
                const uint32_t k = j / (HD / 4), c = j % (HD / 4);
                const uint32_t p = min(lo + i * S::kValues + k, hi - 1);
                cp_async16(to + k * HD + c * 4, vbase + (size_t)p * a.kv_dim + c * 4);
            }
        }
        cp_commit();
    };
    fetch_values(0);

    // ---- softmax, a warp per row: exponentials added one by one
#pragma unroll 1
    for (uint32_t r = warp; r < kRows; r += T / 32) {
        float* row = w + r * a.pitch + (first(r) - lo);
        const uint32_t len = last(r) - first(r), whole = a.gpt2_tail ? (len & ~15u) : len;
        float mx = -INFINITY;
        for (uint32_t p = lane; p < len; p += 32) mx = fmaxf(mx, row[p]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, off));
        for (uint32_t p = lane; p < len; p += 32) row[p] = exp_f32(__fsub_rn(row[p], mx));
        __syncwarp();
        float sum = 0.0f;  // the same chain in every lane
        uint32_t p = 0;
        for (; p + 16 <= len; p += 16) {
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = row[p + j];
#pragma unroll
            for (int j = 0; j < 16; ++j) sum = __fadd_rn(sum, v[j]);
        }
        for (; p < len; ++p) sum = __fadd_rn(sum, row[p]);
        __syncwarp();
        const float inv = __fdiv_rn(1.0f, sum);
        for (p = lane; p < len; p += 32) row[p] = p < whole ? __fmul_rn(row[p], inv) : __fdiv_rn(row[p], sum);
    }

    // ---- weighted sums, position by position
    const uint32_t d = tid % HD, g0 = tid / HD * S::kPerThread;
    float o[S::kPerThread];
#pragma unroll
    for (uint32_t j = 0; j < S::kPerThread; ++j) o[j] = 0.0f;
#pragma unroll 1
    for (uint32_t i = 0; i < n_value_tiles; ++i) {
        fetch_values(i + 1);
        cp_wait_1();
        __syncthreads();  // first round: the weights are complete as well
        const float* v = tile + (i & 1u) * S::kTile + d;
        const uint32_t p0 = lo + i * S::kValues;
        const float* wr = w + g0 * a.pitch + (p0 - lo);
        if (first(g0 + S::kPerThread - 1) <= p0 && p0 + S::kValues <= last(g0)) {
#pragma unroll 2
            for (uint32_t p = 0; p < S::kValues; p += 4) {
                const float v0 = v[p * HD], v1 = v[(p + 1) * HD], v2 = v[(p + 2) * HD], v3 = v[(p + 3) * HD];
#pragma unroll
                for (uint32_t j = 0; j < S::kPerThread; ++j) {
                    const float4 ww = *reinterpret_cast<const float4*>(wr + j * a.pitch + p);
                    o[j] = __fadd_rn(o[j], __fmul_rn(ww.x, v0));
                    o[j] = __fadd_rn(o[j], __fmul_rn(ww.y, v1));
                    o[j] = __fadd_rn(o[j], __fmul_rn(ww.z, v2));
                    o[j] = __fadd_rn(o[j], __fmul_rn(ww.w, v3));
                }
            }
        } else {  // a tile that some row sees in part: positions outside its window leave its sum as it is
            const uint32_t n_here = min((uint32_t)S::kValues, hi - p0);
#pragma unroll 1
            for (uint32_t p = 0; p < n_here; p += 4) {
                const float vv[4] = {v[p * HD], v[(p + 1) * HD], v[(p + 2) * HD], v[(p + 3) * HD]};
#pragma unroll
                for (uint32_t j = 0; j < S::kPerThread; ++j) {
                    const float4 ww = *reinterpret_cast<const float4*>(wr + j * a.pitch + p);
                    const float wv[4] = {ww.x, ww.y, ww.z, ww.w};
                    const uint32_t from = first(g0 + j) - p0, len = last(g0 + j) - first(g0 + j);  // `from` may wrap
#pragma unroll
                    for (uint32_t e = 0; e < 4; ++e) {
                        const float next = __fadd_rn(o[j], __fmul_rn(wv[e], vv[e]));
                        o[j] = p + e - from < len ? next : o[j];
                    }
                }
            }
        }
        __syncthreads();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (uint32_t j = 0; j < S::kPerThread; ++j) {
        if (g0 + j >= n) break;  // the same for a whole warp
        const size_t at = ((size_t)(t0 + g0 + j) * a.n_head + h) * HD + d;
        if (a.out) a.out[at] = o[j];
        if (a.oq) quantize_block_warp(o[j], at >> 5, lane, a.oq, a.oscale, a.osum);
    }
}

constexpr size_t kMostSmem = 227 * 1024;  // of a CTA

uint32_t pitch_of(uint32_t span) { return (span + kKeys - 1) / kKeys * kKeys + 4; }

template <int HD, int ROWS>
size_t prefill_smem(uint32_t pitch) {
    return (2 * (size_t)PrefillShape<HD, ROWS>::kTile + (size_t)ROWS * HD + (size_t)ROWS * pitch) * sizeof(float);
}

template <int HD, int ROWS>
int launch_rows(PrefillArgs a, uint32_t end, bool shared_split, cudaStream_t st) {
    const uint32_t span = a.window && end > a.window + ROWS ? a.window + ROWS : end;  // positions that a CTA may see
    a.pitch = pitch_of(span);
    const size_t smem = prefill_smem<HD, ROWS>(a.pitch);
    if (smem > kMostSmem) return ZQ_ERR_LIMIT;
    auto kern = attention_prefill_kernel<HD, ROWS>;
    // the most that any prompt asks for: the limit is the process's, and another thread may be about to launch a longer one
    ZQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem));
    ZQ_CUDA(launch_pdl_split(shared_split, kern, dim3((a.rows + ROWS - 1) / ROWS, a.n_head),
                             dim3(PrefillShape<HD, ROWS>::kThreads), smem, st, a));
    return ZQ_OK;
}

// Four tokens per CTA while sixteen would leave half of the GPU without one (head_dim 256, 40 tokens of 4 heads: 19.9 us
// with sixteen, 9.9 us with four).
template <int HD>
int launch_hd(const PrefillArgs& a, uint32_t end, bool shared_split, cudaStream_t st) {
    constexpr int kFew = HD >= 64 ? 4 : 16;
    if ((a.rows + 15) / 16 * a.n_head * 2 < (uint32_t)sm_count()) return launch_rows<HD, kFew>(a, end, shared_split, st);
    return launch_rows<HD, 16>(a, end, shared_split, st);
}

}  // namespace

bool attention_prefill_takes(uint32_t head_dim, uint32_t ctx) {
    const uint32_t pitch = pitch_of(ctx);
    switch (head_dim) {
        case 32: return prefill_smem<32, 16>(pitch) <= kMostSmem;
        case 64: return prefill_smem<64, 16>(pitch) <= kMostSmem;
        case 128: return prefill_smem<128, 16>(pitch) <= kMostSmem;
        case 256: return prefill_smem<256, 16>(pitch) <= kMostSmem;
        default: return false;
    }
}

int launch_attention_prefill(const float* q, const float* kc, const float* vc, float* out, int8_t* oq, float* oscale,
                             int32_t* osum, uint32_t n_head, uint32_t n_kv_head, uint32_t head_dim, const uint32_t* state,
                             uint32_t window, uint32_t end, int flags, uint32_t rows, uint32_t q_stride, cudaStream_t st,
                             bool shared_split) {
    if (rows == 0) return ZQ_OK;
    const uint32_t kv_dim = n_kv_head * head_dim;
    if (((uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc) & 15 || q_stride % 4 || n_head > 65535u) return ZQ_ERR_LIMIT;
    PrefillArgs a{q, kc, vc, out, oq, oscale, osum, state, n_head, n_head / n_kv_head, kv_dim, rows, window, q_stride, 0,
                  (flags & ZQ_ATTN_GPT2_SOFTMAX) ? 1 : 0};
    switch (head_dim) {
        case 32: return launch_hd<32>(a, end, shared_split, st);
        case 64: return launch_hd<64>(a, end, shared_split, st);
        case 128: return launch_hd<128>(a, end, shared_split, st);
        case 256: return launch_hd<256>(a, end, shared_split, st);
        default: return ZQ_ERR_LIMIT;
    }
}

}  // namespace zq
