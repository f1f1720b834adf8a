// Quantised weights times many f32 activation rows at f32 accuracy: the prompt of the GPT-2 engine and calls of more rows
// than the decode kernel's 16 (gemv_mma.cu) whose precision stays that of the CPU path.
//
// Arithmetic is the decode kernel's: integer weights (exact in fp16) times the fp16 parts hi and lo of an activation row
// brought under 2^14 by a power of two, products exact, 32-value block dots in f32, times the block's f32 scale in f32.
// Both parts go into one accumulator (lo first), so a block costs one multiply-add per output.
//
// What bounds it: mma.sync, 4 m16n8k16 per 16 x 8 outputs and block. tcgen05 is not taken because every block dot is
// scaled before it is added: with the scale folded into 19-bit weights the sum over all of K would stay inside the tensor
// core, whose accumulation is coarser than the f32 sum over blocks. The activations are split once per call into an image
// in fragment order (split_rows_kernel), so the loop loads them with 128-bit accesses free of bank conflicts; a warp owns
// 16 weight rows and unpacks a weight word once for all NT x 8 activation rows.
// What a CTA's step costs besides is its instructions: the chain's first MMA takes its zeros from registers that stay, and a thread
// finds its copies by one addition each (768 <- 3072 at 32 rows 12.8 -> 9.3 us, 1152 <- 6912 at 24 rows 24.2 -> 17.6; GPT-2 document of 900
// tokens 7.33 -> 7.22 ms).
// Measured (B200, graph-timed, split_rows included; passes of the decode kernel, this product): 3072 <- 768 at 48 rows 31, 7.3 us;
// 1152 <- 6912 at 48 rows 137, 26 us.
#include "zq_internal.h"

namespace zq {
namespace {

struct SplitEpilogue {
    const float* bias;
    const float* mul;
    const float* residual;
    int gelu;
};

__device__ __forceinline__ float gelu_tanh(float v) {
    const float cube = __fmul_rn(__fmul_rn(__fmul_rn(0.044715f, v), v), v);
    const float inner = __fmul_rn(0.7978845608f, __fadd_rn(v, cube));
    return __fmul_rn(__fmul_rn(0.5f, v), __fadd_rn(1.0f, (float)tanh((double)inner)));
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// ---- activation image -------------------------------------------------------------------------------
// frag[tile of 8 rows][block][part: hi, lo][lane = 4 * row + t] (uint4): elements 4t..4t+3 and 16+4t..16+4t+3 of the
// block as the B registers {b0, b1} of the two MMAs, K slots (2t, 2t+1, 2t+8, 2t+9) <- elements (0, 2, 1, 3).
// sums[tile][block][8]: f32 sums of the 32 values (q4_1). post[row]: factor that undoes the row's prescale.
// Rows >= M of the last tile and blocks >= nb are zero.
struct SplitImage {
    uint4* frag;
    float* sums;
    float* post;
};

__host__ __device__ inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

SplitImage split_image(void* workspace, const zq_weight* w, uint32_t m_rows) {
    const size_t tiles = (m_rows + 7) / 8;
    char* p = static_cast<char*>(workspace);
    SplitImage im;
    im.frag = reinterpret_cast<uint4*>(p);
    p += align256(tiles * w->nbp * 1024);
    im.sums = reinterpret_cast<float*>(p);
    p += align256(tiles * w->nbp * 32);
    im.post = reinterpret_cast<float*>(p);
    return im;
}

// One CTA per row.
__global__ void __launch_bounds__(128)
split_rows_kernel(const float* __restrict__ x, uint32_t M, uint32_t K, uint32_t nb, uint32_t nbp, SplitImage im) {
    __shared__ float red[4];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t m = blockIdx.x, tid = threadIdx.x;
    const bool real = m < M;
    const float4* row = reinterpret_cast<const float4*>(x + (size_t)(real ? m : 0) * K);
    float amax = 0.0f;
    if (real) {
        for (uint32_t i = tid; i < K / 4; i += 128) {
            const float4 v = row[i];
            amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, off));
    if ((tid & 31) == 0) red[tid >> 5] = amax;
    __syncthreads();
    amax = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    const int e = row_scale_exponent(amax);
    const float pre = ldexpf(1.0f, -e);
    if (tid == 0) im.post[m] = ldexpf(1.0f, e);
    const uint32_t tile = m >> 3, g = m & 7u;
    uint4* frag = im.frag + (size_t)tile * nbp * 64 + g * 4;
    for (uint32_t i = tid; i < nbp * 4; i += 128) {  // nbp * 4 is a multiple of 16: a block's four threads stay together
        const uint32_t blk = i >> 2, t = i & 3u;
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
        if (real && blk < nb) {
            a = row[blk * 8 + t];
            b = row[blk * 8 + 4 + t];
        }
        const float v[8] = {a.x * pre, a.y * pre, a.z * pre, a.w * pre, b.x * pre, b.y * pre, b.z * pre, b.w * pre};
        float s8 = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        const uint32_t mask = 0xFu << (tid & 28u);
        s8 += __shfl_xor_sync(mask, s8, 1);
        s8 += __shfl_xor_sync(mask, s8, 2);
        if (t == 0) im.sums[((size_t)tile * nbp + blk) * 8 + g] = s8;
        float hi[8], lo[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            hi[j] = __half2float(__float2half_rn(v[j]));
            lo[j] = v[j] - hi[j];  // exact in f32
        }
        frag[(size_t)blk * 64 + t] = make_uint4(pack_half2(hi[0], hi[2]), pack_half2(hi[1], hi[3]),
                                                pack_half2(hi[4], hi[6]), pack_half2(hi[5], hi[7]));
        frag[(size_t)blk * 64 + 32 + t] = make_uint4(pack_half2(lo[0], lo[2]), pack_half2(lo[1], lo[3]),
                                                     pack_half2(lo[4], lo[6]), pack_half2(lo[5], lo[7]));
    }
}

// ---- product ----------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The first of a chain: zeros from registers of the caller's, so that none are cleared for it.
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&zero)[4]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(zero[0]), "f"(zero[1]), "f"(zero[2]), "f"(zero[3]));
}
__device__ __forceinline__ void rotate(uint4& v) {
    v.x = v.y;
    v.y = v.z;
    v.z = v.w;
}
__device__ __forceinline__ uint32_t hsub2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// A quant word -> fp16 pairs (e0, e2), (e1, e3), exact: int8 values ...
__device__ __forceinline__ void unpack_q8(uint32_t q, uint32_t& p02, uint32_t& p13) {
    const uint32_t u = q ^ 0x80808080u;
    constexpr uint32_t kSub = 0x64806480u;  // 1024 + 128
    p02 = hsub2(__byte_perm(u, 0x64646464u, 0x4240), kSub);
    p13 = hsub2(__byte_perm(u, 0x64646464u, 0x4341), kSub);
}
// ... or the low and the high nibbles, minus 8 for q4_0.
template <bool MINUS8>
__device__ __forceinline__ void unpack_q4(uint32_t q, uint32_t& lo02, uint32_t& lo13, uint32_t& hi02, uint32_t& hi13) {
    constexpr uint32_t kSub = MINUS8 ? 0x64086408u : 0x64006400u;  // 1024 (+ 8)
    constexpr uint32_t k16th = 0x2C002C00u;                        // 1 / 16
    constexpr uint32_t kAdd = MINUS8 ? 0xD480D480u : 0xD400D400u;  // -64 (- 8)
    const uint32_t s = q >> 8;
    lo02 = hsub2((q & 0x000F000Fu) | 0x64006400u, kSub);
    lo13 = hsub2((s & 0x000F000Fu) | 0x64006400u, kSub);
    hi02 = hfma2((q & 0x00F000F0u) | 0x64006400u, k16th, kAdd);
    hi13 = hfma2((s & 0x00F000F0u) | 0x64006400u, k16th, kAdd);
}

// A CTA has WR x KS warps: WR x 16 weight rows, NT x 8 activation rows, and KS parts of K. A stage of the ring holds KS quads
// (4 blocks each): per quad the activations of NT tiles (4 KB each, q4_1: and their sums), and per warp the packed words and
// scales of its own quad and 16 rows, each lane's pieces in its own slots.
template <int TYPE, int WR, int KS, int NT>
struct SplitStage {
    static constexpr uint32_t kSums = TYPE == ZQ_TYPE_Q4_1 ? 128 : 0;
    static constexpr uint32_t kTile = 4096 + kSums;
    static constexpr uint32_t kAct = KS * NT * kTile;
    static constexpr uint32_t kWq = TYPE == ZQ_TYPE_Q8_0 ? 2048 : 1024;
    static constexpr uint32_t kWsHalf = TYPE == ZQ_TYPE_Q4_1 ? 512 : 256;
    static constexpr uint32_t kWTile = kWq + 2 * kWsHalf;
    static constexpr uint32_t kBytes = kAct + WR * KS * kWTile;
};

template <int TYPE, int WR, int KS, int NT, int D>
__global__ void __launch_bounds__(WR * KS * 32)
gemm_split_kernel(const uint8_t* __restrict__ qs, const uint8_t* __restrict__ sc, SplitImage im, float* __restrict__ y,
                  uint32_t N, uint32_t M, uint32_t nbp, uint32_t scp, SplitEpilogue ep) {
    constexpr bool Q8 = TYPE == ZQ_TYPE_Q8_0, Q41 = TYPE == ZQ_TYPE_Q4_1;
    constexpr uint32_t QB = Q8 ? 32 : 16, QUAD = 4 * QB, SB = Q41 ? 4 : 2, THREADS = WR * KS * 32;
    using S = SplitStage<TYPE, WR, KS, NT>;
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t smem32 = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t wr = warp % WR, ks = warp / WR;
    const uint32_t nq = nbp / 4, steps = (nq + KS - 1) / KS;
    const uint32_t n0 = blockIdx.x * (WR * 16) + wr * 16, tile0 = blockIdx.y * NT, tiles = (M + 7) / 8;
    const uint32_t nt = min((uint32_t)NT, tiles - tile0);  // tiles that exist

    const uint8_t* pw[2];
    const uint8_t* ps[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t row = min(n0 + h * 8 + g, N - 1);
        pw[h] = qs + (size_t)row * nbp * QB + 16 * t;
        ps[h] = sc + (size_t)row * scp * SB;
    }
    const uint32_t wslot = smem32 + S::kAct + warp * S::kWTile;
    static_assert(THREADS == 256, "a thread copies 16 bytes of a tile's quad");
    const uint4* px = im.frag + (size_t)tile0 * nbp * 64 + tid;

    auto issue_weights = [&](uint32_t stage, uint32_t step) {
        const uint32_t q = step * KS + ks;
        if (q >= nq) return;
        const uint32_t wb = wslot + stage * S::kBytes;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            cp_async16(wb + h * 512 + lane * 16, pw[h] + (size_t)q * QUAD);
            if (Q8) cp_async16(wb + 1024 + h * 512 + lane * 16, pw[h] + (size_t)q * QUAD + 64);
            if (Q41)
                cp_async16(wb + S::kWq + h * S::kWsHalf + lane * 16, ps[h] + (size_t)q * 16);
            else
                cp_async8(wb + S::kWq + h * S::kWsHalf + lane * 8, ps[h] + (size_t)q * 8);
        }
    };
    auto issue_acts = [&](uint32_t stage, uint32_t step) {
        const uint32_t base = smem32 + stage * S::kBytes;
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            const uint32_t q = step * KS + k;
            if (q >= nq) break;
#pragma unroll
            for (int j = 0; j < NT; ++j)
                if ((uint32_t)j < nt) cp_async16(base + (k * NT + j) * S::kTile + tid * 16, px + ((uint32_t)j * nbp + q * 4) * 64);
            if (Q41) {
                for (uint32_t i = tid; i < nt * 8; i += THREADS) {
                    const uint32_t j = i >> 3, o = i & 7u;
                    cp_async16(base + (k * NT + j) * S::kTile + 4096 + o * 16,
                               im.sums + ((size_t)(tile0 + j) * nbp + q * 4) * 8 + o * 4);
                }
            }
        }
    };

    // Sums in two levels, kFlush quads below and those above: the f32 chain over K stays as short as that of the
    // decode kernel, which cuts K into up to eight parts (in one level the error at 216 blocks was 1.6e-7 against 1.2e-7).
    constexpr uint32_t kFlush = 4;
    float acc[NT][4], sum[NT][4], zero[4];
    asm volatile("mov.b32 %0, 0; mov.b32 %1, 0; mov.b32 %2, 0; mov.b32 %3, 0;" : "=f"(zero[0]), "=f"(zero[1]), "=f"(zero[2]), "=f"(zero[3]));
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[j][c] = sum[j][c] = 0.0f;
    auto flush = [&] {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                sum[j][c] += acc[j][c];
                acc[j][c] = 0.0f;
            }
    };

    pdl_launch_dependents();
#pragma unroll 1
    for (uint32_t s = 0; s + 1 < (uint32_t)D; ++s)
        if (s < steps) issue_weights(s, s);  // no earlier kernel writes the weights
    pdl_wait();
#pragma unroll 1
    for (uint32_t s = 0; s + 1 < (uint32_t)D; ++s) {
        if (s < steps) issue_acts(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    uint32_t stage = 0, p_stage = D - 1;
#pragma unroll 1
    for (uint32_t s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");  // step s has landed
        __syncthreads();  // for every thread; and all are done with the stage that is filled next
        if (s + D - 1 < steps) {
            issue_weights(p_stage, s + D - 1);
            issue_acts(p_stage, s + D - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        p_stage = p_stage + 1 == (uint32_t)D ? 0 : p_stage + 1;

        if (s * KS + ks < nq) {
            const uint32_t act = smem32 + stage * S::kBytes + ks * NT * S::kTile, wb = wslot + stage * S::kBytes;
            uint4 wlo[2], whi[2], ws[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                wlo[h] = lds128(wb + h * 512 + lane * 16);
                if (Q8) whi[h] = lds128(wb + 1024 + h * 512 + lane * 16);
                if (Q41) {
                    ws[h] = lds128(wb + S::kWq + h * S::kWsHalf + lane * 16);
                } else {
                    const uint2 v = lds64(wb + S::kWq + h * S::kWsHalf + lane * 8);
                    ws[h].x = v.x;
                    ws[h].y = v.y;
                }
            }
#pragma unroll 1  // unrolled, the compiler unpacks all four blocks ahead and spills; the words rotate instead
            for (int b = 0; b < 4; ++b) {
                uint32_t aL[4], aH[4];
                float d[2], mn[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (Q8) {
                        unpack_q8(wlo[h].x, aL[h], aL[2 + h]);
                        unpack_q8(whi[h].x, aH[h], aH[2 + h]);
                        rotate(whi[h]);
                    } else {
                        unpack_q4<!Q41>(wlo[h].x, aL[h], aL[2 + h], aH[h], aH[2 + h]);
                    }
                    rotate(wlo[h]);
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&ws[h].x));
                    d[h] = f.x;
                    mn[h] = f.y;  // q4_1; otherwise the next block's scale
                    if (Q41) {
                        rotate(ws[h]);
                    } else {
                        ws[h].x = b & 1 ? ws[h].y : ws[h].x >> 16;
                    }
                }
                // One of the four MMAs after the other over all tiles: a tile's MMAs depend on one another (28 cycles each),
                // and taken tile by tile a warp waits out the latency of each.
                uint4 hi[NT], lo[NT];
                float p[NT][4];
#pragma unroll
                for (int j = 0; j < NT; ++j) {  // tiles past the last: what the stage happens to hold, stored nowhere
                    const uint32_t at = act + j * S::kTile + b * 1024 + lane * 16;
                    lo[j] = lds128(at + 512);
                    hi[j] = lds128(at);
                }
#pragma unroll
                for (int ph = 0; ph < 4; ++ph)
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        const uint4& v = ph < 2 ? lo[j] : hi[j];
                        if (ph == 0) mma_f16(p[j], aL, v.x, v.y, zero);
                        else mma_f16(p[j], ph & 1 ? aH : aL, ph & 1 ? v.z : v.x, ph & 1 ? v.w : v.y);
                    }
#pragma unroll
                for (int j = 0; j < NT; ++j) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[j][c] = fmaf(p[j][c], d[c >> 1], acc[j][c]);
                    if (Q41) {
                        const uint2 v = lds64(act + j * S::kTile + 4096 + b * 32 + t * 8);
                        const float xs[2] = {__uint_as_float(v.x), __uint_as_float(v.y)};
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[j][c] = fmaf(mn[c >> 1], xs[c & 1], acc[j][c]);
                    }
                }
            }
            if (s % kFlush == kFlush - 1) flush();
        }
        stage = stage + 1 == (uint32_t)D ? 0 : stage + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    flush();
    // sums of the K parts, in their order, through shared memory
    if (KS > 1) {
        float* red = reinterpret_cast<float*>(smem);  // [ks - 1][wr][NT * 4][32]
        if (ks > 0) {
            float* to = red + (size_t)((ks - 1) * WR + wr) * (NT * 4 * 32) + lane;
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) to[(j * 4 + c) * 32] = sum[j][c];
        }
        __syncthreads();
        if (ks > 0) return;
#pragma unroll
        for (int k = 1; k < KS; ++k) {
            const float* from = red + (size_t)((k - 1) * WR + wr) * (NT * 4 * 32) + lane;
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) sum[j][c] += from[(j * 4 + c) * 32];
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t n = n0 + h * 8 + g;
        if (n >= N) continue;
        const float bias = ep.bias ? ep.bias[n] : 0.0f;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint32_t m = (tile0 + j) * 8 + 2 * t + c;
                if (m >= M) continue;
                const size_t o = (size_t)m * N + n;
                float v = sum[j][h * 2 + c] * im.post[m];
                if (ep.bias) v = __fadd_rn(v, bias);
                if (ep.gelu) v = gelu_tanh(v);
                if (ep.mul) v = __fmul_rn(v, ep.mul[o]);
                if (ep.residual) v = __fadd_rn(ep.residual[o], v);
                y[o] = v;
            }
        }
    }
}

template <int TYPE, int WR, int KS, int NT, int D>
int launch_cfg(const zq_weight* w, const SplitImage& im, float* y, uint32_t M, const SplitEpilogue& ep, cudaStream_t st) {
    const dim3 grid((w->out_dim + WR * 16 - 1) / (WR * 16), (M + NT * 8 - 1) / (NT * 8));
    if (grid.y > 65535u) return ZQ_ERR_LIMIT;
    constexpr size_t ring = (size_t)D * SplitStage<TYPE, WR, KS, NT>::kBytes;
    constexpr size_t red = (size_t)(KS - 1) * WR * NT * 512;
    constexpr size_t smem = ring > red ? ring : red;
    static_assert(smem <= 227 * 1024, "a CTA's shared memory");
    auto kern = gemm_split_kernel<TYPE, WR, KS, NT, D>;
    ZQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    ZQ_CUDA(launch_pdl(kern, grid, dim3(WR * KS * 32), smem, st, w->qs, static_cast<const uint8_t*>(w->sc), im, y,
                       w->out_dim, M, w->nbp, w->scp, ep));
    return ZQ_OK;
}

// The tile whose CTAs run all at once and whose chain of steps (KS quads of K each) is the shortest, `start` and `step` in tenths of a
// microsecond: launch and sums of a CTA, conversions and MMAs of NT tiles and KS x NT x 4 KB of activations. Registers and rings
// leave one CTA per SM to the first eight; the last two run two, whose steps (`pair`) then share the SM. With none that fits, CTAs of the
// last but one take turns. (B200, us with the split, weights from HBM, the ten tiles in this order, the one taken in brackets:
// 768 <- 3072 4_0 at 48 rows [10.0], 12.8, 13.5, 16.5, 20.0, 25.1, 32.4, 53.9, 27.4, 33.4; 1152 <- 6912 8_0 at 48 rows 27.8, [25.5], 27.1, 30.7, 43.8,
// 50.7, 62.8, 107, 66.9, 75.9; 5003 <- 1184 4_1 at 24 rows 20.6, 16.3, 13.7, 16.6, [10.9], 13.1, 16.7, 26.6, 15.5, 18.4; 4096 <- 6144 4_0 at 32 rows
// 47.7, 42.4, 42.7, [30.1], 39.5, 48.6, 60.0, 106, 63.3, 71.5; 12000 <- 1152 4_0 at 24 rows 42.3, 30.1, 18.3, 22.6, 17.4, 21.5, 27.9, 23.0, [14.4], 16.7
// and at 32 rows 43.5, 30.8, 31.3, 23.5, 23.8, 22.0, 28.4, 23.3, 23.9, [17.1]. The tile taken is the best of the ten or within 17 % of it, 0.4 % in the mean,
// for 17 to 48 rows of 16 matrices. A GPT-2 document of 900 tokens: 7.12 ms with CTAs of the last but one in turns, 7.22 with the last.)
template <int TYPE>
int launch_type(const zq_weight* w, const SplitImage& im, float* y, uint32_t M, const SplitEpilogue& ep, cudaStream_t st) {
    struct Tile {
        uint32_t rows, cols, quads, start, step, pair;
    };
    constexpr int kInTurns = 8;
    constexpr Tile tiles[10] = {{16, 16, 8, 36, 20, 0}, {32, 16, 4, 33, 16, 0}, {32, 24, 4, 33, 17, 0}, {32, 32, 4, 40, 20, 0}, {64, 24, 2, 30, 15, 0},
                                {64, 32, 2, 34, 18, 0}, {64, 48, 2, 49, 23, 0}, {128, 48, 1, 52, 20, 0}, {64, 24, 2, 22, 23, 27}, {64, 32, 2, 24, 26, 31}};
    const uint32_t nq = w->nbp / 4;
    const uint64_t sms = (uint64_t)sm_count();
    int best = kInTurns;
    uint32_t least = ~0u;
    for (int i = 0; i < 10; ++i) {
        const Tile& t = tiles[i];
        const uint64_t ctas = (uint64_t)((w->out_dim + t.rows - 1) / t.rows) * ((M + t.cols - 1) / t.cols);
        if (ctas > (t.pair ? 2 : 1) * sms) continue;
        const uint32_t cost = t.start + (nq + t.quads - 1) / t.quads * (ctas > sms ? t.pair : t.step);
        if (cost < least) {
            least = cost;
            best = i;
        }
    }
    switch (best) {
        case 0: return launch_cfg<TYPE, 1, 8, 2, 2>(w, im, y, M, ep, st);
        case 1: return launch_cfg<TYPE, 2, 4, 2, 3>(w, im, y, M, ep, st);
        case 2: return launch_cfg<TYPE, 2, 4, 3, 3>(w, im, y, M, ep, st);
        case 3: return launch_cfg<TYPE, 2, 4, 4, 2>(w, im, y, M, ep, st);
        case 4: return launch_cfg<TYPE, 4, 2, 3, 4>(w, im, y, M, ep, st);
        case 5: return launch_cfg<TYPE, 4, 2, 4, 4>(w, im, y, M, ep, st);
        case 6: return launch_cfg<TYPE, 4, 2, 6, 3>(w, im, y, M, ep, st);
        case 7: return launch_cfg<TYPE, 8, 1, 6, 2>(w, im, y, M, ep, st);
        case 9: return launch_cfg<TYPE, 4, 2, 4, 2>(w, im, y, M, ep, st);
        default: return launch_cfg<TYPE, 4, 2, 3, 2>(w, im, y, M, ep, st);
    }
}

}  // namespace

// Up to 20 rows the calls of more weight rows than 32 per SM stay with the passes (unless K is so deep that a pass holds two rows, or
// the matrix so large that its passes take the ring): where a call needs a workspace is a line that callers have sized theirs by, and
// it was drawn when these calls took tiles of 32 x 32 in turns. With the tiles of now the product is ahead there too (B200, us in passes and
// split at 17 rows: 5760 <- 6144 4_0 84.5 and 39.2, 9472 <- 5120 4_1 60.5 and 40.3, 12000 <- 512 4_0 13.2 and 7.8), and closer to 64 bits with 4-bit
// weights (4_0 8.2e-7 in passes, 1.1e-7 split), though not with 8_0 of few columns (11000 <- 1152 0.95e-7 and 1.06e-7).
bool gemm_split_takes(const zq_weight* w, uint32_t m_rows) {
    if (m_rows < 17) return false;
    const bool ring = w->type != ZQ_TYPE_Q4_1 && (size_t)w->out_dim * w->nbp * w->qb >= ((size_t)64 << 20);
    return m_rows > 20 || (w->out_dim + 31) / 32 <= (uint32_t)sm_count() || w->in_dim >= 12288 || ring;
}

size_t gemm_split_workspace_bytes(const zq_weight* w, uint32_t m_rows) {
    const size_t tiles = (m_rows + 7) / 8;
    return align256(tiles * w->nbp * 1024) + align256(tiles * w->nbp * 32) + align256(tiles * 8 * sizeof(float));
}

int launch_gemm_split(const zq_weight* w, const float* x, float* y, uint32_t m_rows, const zq_epilogue* ep, void* workspace,
                      cudaStream_t st) {
    if (m_rows == 0) return ZQ_OK;
    if (((uintptr_t)x & 15) != 0 || ((uintptr_t)workspace & 255) != 0) return ZQ_ERR_BAD_ARG;
    const SplitImage im = split_image(workspace, w, m_rows);
    SplitEpilogue a{nullptr, nullptr, nullptr, 0};
    if (ep) a = SplitEpilogue{ep->d_bias, ep->d_mul, ep->d_residual, ep->gelu};
    ZQ_CUDA(launch_pdl(split_rows_kernel, dim3((m_rows + 7) / 8 * 8), dim3(128), 0, st, x, m_rows, w->in_dim, w->nb, w->nbp,
                       im));
    switch (w->type) {
        case ZQ_TYPE_Q4_0: return launch_type<ZQ_TYPE_Q4_0>(w, im, y, m_rows, a, st);
        case ZQ_TYPE_Q4_1: return launch_type<ZQ_TYPE_Q4_1>(w, im, y, m_rows, a, st);
        case ZQ_TYPE_Q8_0: return launch_type<ZQ_TYPE_Q8_0>(w, im, y, m_rows, a, st);
        default: return ZQ_ERR_UNSUPPORTED;
    }
}

}  // namespace zq
