// Exact integer GEMM for Q8-quantised activations and many activation rows (batched decode, prefill).
//
// Same arithmetic as the decode kernel in gemv_q8.cu and as zig-nn's CPU path
// (ThreadPool.matmul, src/gguf/thread_pool.zig:96-181 -> src/gguf/simd_dot.zig:71-152): per 32-block an
// exact int8 x int8 -> int32 dot, turned into the f32 term (d * s) * float(idot) [+ (m * s) * float(qsum)],
// and the terms of a row added in block order. Here the block dots of 16 weight rows x 8 activation rows
// come from one mma.sync.m16n8k32 (s8 x s8 -> s32, exact), the weights are read once per CTA's 8 to
// 64 activation rows instead of once per row, and each (weight row, activation row) pair keeps its running f32 sum in
// a register, so the result is bit-identical to running the decode kernel row by row.
//
// Tile: W warps x MT x 16 weight rows, NT x 8 activation rows per CTA; K advances by one quad of blocks
// (128 values). Everything a quad needs travels through a ring of D shared-memory stages filled with
// cp.async, D - 1 quads ahead of the multiplications: the quantised activations (128 bytes per row and their
// scales; 4_1: and sums) and, per warp, the packed weight words and scales of its rows. The small CTA shapes used
// for matrices with few rows have only a few warps per SM, so the depth of this ring - not occupancy - is what
// hides the memory latency there.
//
// What bounds it: issue slots and their latencies around the scaling. Per MMA tile of 16 x 8 that is four conversions and, two
// columns at a time (f32x2), two multiplies and an add for each of its pairs; 4_0 weights are centred before the product, so
// that no sum of activations is needed. Against one column at a time and sums subtracted behind the product (B200, us with the
// quantiser and weights from HBM, before and now): 14336 <- 4096 4_0 at 8, 64 and 140 rows 27.3, 92.2, 181 and 22.0, 50.3, 94.5; 262144 <-
// 1152 4_1 at 8 rows 87.0 and 65.1; 13824 <- 1152 8_0 at 16, 100 and 512 rows 14.2, 32.5, 91.1 and 9.5, 24.7, 84.8; 1152 <- 6912 8_0 at 512
// rows 112 and 67.6 (its shape, cheapest_shape). Two weight tiles per warp (MT) share the activation fragments, which costs registers:
// only shape 1 has them. (The same on tcgen05.mma.kind::i8, a block per MMA of K = 32 and the scaling behind tcgen05.ld, came to 76 and 54
// us for the two 512-row products, and was slower than this form at all smaller ones: about 8 cycles of an SM for a column of
// 128 weight rows and a block, where its three f32 operations need 3.)
// What a CTA takes besides its blocks counts for short rows: the copies' sources are 32-bit offsets from the CTA's first rows, and the
// sums leave by rows without the epilogue's questions where it has none (30000 <- 320 8_0 at 64 and 512 rows 16.2 and 80.0 us with 64-bit
// products per piece, 12.8 and 56.7 so).
#include "zq_internal.h"

namespace zq {
namespace {

struct QgEpilogue {
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

__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async4_zfill(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ __half lds_half(uint32_t addr) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return __ushort_as_half(v);
}
__device__ __forceinline__ unsigned long long lds_pair(uint32_t addr) {
    unsigned long long v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%10,%10,%10,%10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
// The same with the four zeros in registers of the caller's.
__device__ __forceinline__ void mma_s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const int (&zero)[4]) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%10,%11,%12,%13};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(zero[0]), "r"(zero[1]), "r"(zero[2]), "r"(zero[3]));
}
__device__ __forceinline__ uint32_t pick4(const uint4& v, int j) {
    return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
}

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

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// a + b. The assembler makes one fused operation of a packed multiply and the packed add behind it, although both say .rn (seen
// on this toolkit: a * b + c of two such instructions has the bits of fmaf); as a multiply-add whose factor `one` it cannot know to
// be 1, the sum keeps its own rounding.
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b, f32x2 one) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(b), "l"(one), "l"(a));
    return d;
}
// Nibbles n of a word as signed bytes n - 8.
__device__ __forceinline__ uint32_t centred(uint32_t n) {
    const uint32_t s = n ^ 0x08080808u;
    return s | ((s & 0x08080808u) * 0x1Eu);
}

// Bytes of one ring stage: activations of the CTA, then per warp the packed words (512 bytes per array of 16 bytes per lane)
// and the scales of its rows.
template <int TYPE, int W, int MT, int NT>
struct QgStage {
    static constexpr uint32_t kXq = 4 * NT * 8 * 32;   // 4 blocks x BM rows x 32 int8
    static constexpr uint32_t kSc = 4 * NT * 8 * 4;    // 4 blocks x BM rows x f32 (4_1: and the same for the sums)
    static constexpr uint32_t kAct = kXq + (TYPE == ZQ_TYPE_Q4_1 ? 2 : 1) * kSc;
    static constexpr uint32_t kWq = MT * (TYPE == ZQ_TYPE_Q8_0 ? 2048 : 1024);
    static constexpr uint32_t kRowScales = TYPE == ZQ_TYPE_Q4_1 ? 16 : 8;
    static constexpr uint32_t kWarp = kWq + MT * 16 * kRowScales;
    static constexpr uint32_t kBytes = (kAct + W * kWarp + 127u) & ~127u;
};

template <int TYPE, int W, int MT, int NT, int D>
__global__ void __launch_bounds__(W * 32)
gemm_q8_kernel(const uint8_t* __restrict__ qs, const uint8_t* __restrict__ sc, const int8_t* __restrict__ xq,
               const float* __restrict__ xscale, const int32_t* __restrict__ xqsum, float* __restrict__ y,
               uint32_t N, uint32_t K, uint32_t M, uint32_t nb, uint32_t scp, float one, QgEpilogue ep) {
    constexpr bool Q8 = TYPE == ZQ_TYPE_Q8_0;
    constexpr bool Q41 = TYPE == ZQ_TYPE_Q4_1;
    constexpr uint32_t QB = Q8 ? 32 : 16;
    constexpr uint32_t QUAD = 4 * QB;
    using S = QgStage<TYPE, W, MT, NT>;
    constexpr int QG_BN = W * MT * 16, QG_BM = NT * 8, T = W * 32;
    constexpr uint32_t QG_XQ_BYTES = S::kXq, QG_SC_BYTES = S::kSc, QG_STAGE = S::kBytes;
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t smem32 = (uint32_t)__cvta_generic_to_shared(smem);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t nbp = (nb + 3u) & ~3u, nq = nbp / 4;
    const uint32_t n0 = blockIdx.x * QG_BN + warp * (MT * 16), m0 = blockIdx.y * QG_BM;
    const uint32_t wring = smem32 + S::kAct + warp * S::kWarp;  // this warp's part of stage 0

    // Sources of this thread's copies of quad 0, as offsets from the first of the CTA's rows; a quad further they lie a constant number
    // of bytes on.
    // Weights: the words of its own rows g and g + 8 of each tile. 8_0: words 2t and 2t + 1 of the four blocks are 32 contiguous
    // bytes; 4-bit: word t, whose low nibbles are the block's word t and whose high ones its word 4 + t.
    // Scales: a lane per row of the warp. Activations: xq entries [blk][row][32 bytes], scales [blk][row], sums [blk][row]; rows
    // >= M and blocks >= nb are zero-filled (never used for output).
    uint32_t w_off[MT * 2];
#pragma unroll
    for (int r = 0; r < MT * 2; ++r) w_off[r] = (min(n0 + r * 8 + g, N - 1) - min(n0, N - 1)) * (nbp * QB);
    const uint8_t* w_src = qs + (size_t)min(n0, N - 1) * nbp * QB + 16 * t;
    const uint8_t* s_src = sc + (size_t)min(n0 + (uint32_t)lane % (MT * 16), N - 1) * scp * (Q41 ? 4 : 2);
    constexpr int XP = (8 * QG_BM + T - 1) / T, SP = (4 * QG_BM + T - 1) / T;  // pieces of a thread, T / 8 and T / 4 rows apart
    // a thread's pieces are of one block and half (T / 8 rows apart in the activations), of one block (T / 4 in the scales)
    const uint32_t xr = tid >> 3, xb = (tid >> 1) & 3u, xh = tid & 1u, sr = tid >> 2, sb = tid & 3u;
    const int8_t* x_src = xq + (size_t)m0 * K;
    const float* sc_src = xscale + (size_t)m0 * nb;
    const int32_t* qsum_src = xqsum + (size_t)m0 * nb;
    const uint32_t x_off = xr * K + (tid & 7u) * 16, s_off = sr * nb + sb, rows = M - m0;
    // 4-bit: the halves of rows with bit 2 set change places, or the fragment loads would meet in a bank
    static_assert(T % 64 == 0, "pieces of a thread lie a multiple of eight rows apart");
    const uint32_t x_to = ((xb * QG_BM + xr) * 2 + (Q8 ? xh : xh ^ ((xr >> 2) & 1u))) * 16, s_to = QG_XQ_BYTES + (sb * QG_BM + sr) * 4;
    auto issue = [&](uint32_t stage, uint32_t q) {
        const uint32_t base = smem32 + stage * QG_STAGE, left = nb - q * 4;  // blocks from this quad on
#pragma unroll
        for (int i = 0; i < XP; ++i) {
            if (8 * QG_BM % T == 0 || tid + i * T < 8 * QG_BM) {
                const bool ok = xr + i * (T / 8) < rows && xb < left;
                cp_async16_zfill(base + x_to + i * (T / 8) * 32, x_src + (ok ? x_off + i * (T / 8) * K + q * 128 : 0), ok ? 16u : 0u);
            }
        }
#pragma unroll
        for (int i = 0; i < SP; ++i) {
            if (4 * QG_BM % T == 0 || tid + i * T < 4 * QG_BM) {
                const bool ok = sr + i * (T / 4) < rows && sb < left;
                const uint32_t o = ok ? s_off + i * (T / 4) * nb + q * 4 : 0;
                cp_async4_zfill(base + s_to + i * (T / 4) * 4, sc_src + o, ok ? 4u : 0u);
                if (Q41) cp_async4_zfill(base + s_to + QG_SC_BYTES + i * (T / 4) * 4, qsum_src + o, ok ? 4u : 0u);
            }
        }
        const uint32_t wb = wring + stage * QG_STAGE;
#pragma unroll
        for (int r = 0; r < MT * 2; ++r) {
            const uint8_t* from = w_src + (w_off[r] + q * QUAD);
            if (Q8) {  // piece w of a row at w ^ (row & 1): the lanes of a fragment load meet in no bank
                const uint32_t to = wb + (r * 8 + g) * 128 + ((t ^ (g & 1)) << 4);
                cp_async16(to, from);
                cp_async16(to + 64, from + 64);
            } else {
                cp_async16(wb + r * 512 + lane * 16, from);
            }
        }
        if (MT == 2 || lane < 16) {
            const uint32_t to = wb + S::kWq + lane * S::kRowScales;
            if (Q41) cp_async16(to, s_src + q * 16);
            else cp_async8(to, s_src + q * 8);
        }
    };

    const f32x2 one2 = pack2(one, one);
    int zero[4];
    asm volatile("mov.b32 %0, 0; mov.b32 %1, 0; mov.b32 %2, 0; mov.b32 %3, 0;" : "=r"(zero[0]), "=r"(zero[1]), "=r"(zero[2]), "=r"(zero[3]));
    f32x2 run[MT][NT][2];  // [tile][column tile][row g, row g + 8]: columns 2t and 2t + 1
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) run[i][j][0] = run[i][j][1] = 0;

    // fragment addressing inside a stage: entry (blk, row = 8j + g). 8_0: words 2t and 2t + 1; 4-bit: t and 4 + t, halves swapped
    const uint32_t swap = ((uint32_t)g >> 2) & 1u;
    const uint32_t frag_lo = Q8 ? (uint32_t)lane * 8 : ((uint32_t)g * 2 + swap) * 16 + t * 4;
    const uint32_t frag_hi = ((uint32_t)g * 2 + (1u ^ swap)) * 16 + t * 4;

    // the quantised activations come from the kernel before this one
    pdl_launch_dependents();
    pdl_wait();

    // group number n holds quad n (an empty group when the row has no such quad)
#pragma unroll 1
    for (uint32_t i = 0; i + 1 < (uint32_t)D; ++i) {
        if (i < nq) issue(i, i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    uint32_t stage = 0, p_stage = D - 1;
#pragma unroll 1
    for (uint32_t q = 0; q < nq; ++q) {
        if (q + D - 1 < nq) issue(p_stage, q + D - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        p_stage = p_stage + 1 == (uint32_t)D ? 0 : p_stage + 1;
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");  // quad q has landed
        __syncthreads();

        const uint32_t base = smem32 + stage * QG_STAGE;
        const uint32_t wb = wring + stage * QG_STAGE;
        const uint32_t blocks = min(4u, nb - q * 4);  // row padding: no term is added for blocks that do not exist
        uint4 w[MT * 2][Q8 ? 2 : 1];
#pragma unroll
        for (int r = 0; r < MT * 2; ++r) {
            const uint32_t at = wb + (Q8 ? (r * 8 + g) * 128 + (((2 * t) ^ (g & 1)) << 4) : r * 512 + lane * 16);
            w[r][0] = lds128(at);
            if (Q8) w[r][Q8 ? 1 : 0] = lds128(at ^ 16u);
        }
#pragma unroll
        for (uint32_t b = 0; b < 4; ++b) {
            if (b >= blocks) break;
            uint32_t a[MT][4];
            f32x2 dd[MT * 2], mm[MT * 2];
#pragma unroll
            for (int r = 0; r < MT * 2; ++r) {
                uint32_t lo = pick4(w[r][0], b), hi = Q8 ? pick4(w[r][Q8 ? 1 : 0], b) : lo >> 4;
                if (!Q8) {
                    lo &= 0x0F0F0F0Fu;
                    hi &= 0x0F0F0F0Fu;
                }
                if (TYPE == ZQ_TYPE_Q4_0) {
                    lo = centred(lo);
                    hi = centred(hi);
                }
                a[r >> 1][r & 1] = lo;
                a[r >> 1][2 + (r & 1)] = hi;
                const uint32_t at = wb + S::kWq + (r * 8 + g) * S::kRowScales + b * (Q41 ? 4 : 2);
                if (Q41) {
                    const uint32_t u = lds32(at);
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u));
                    dd[r] = pack2(f.x, f.x);
                    mm[r] = pack2(f.y, f.y);
                } else {
                    const float f = __half2float(lds_half(at));
                    dd[r] = pack2(f, f);
                }
            }
            const uint32_t xb = base + b * (QG_BM * 32), sbase = base + QG_XQ_BYTES + b * (QG_BM * 4) + t * 8;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                uint2 xw;
                if (Q8) {
                    xw = lds64(xb + j * 256 + frag_lo);
                } else {
                    xw.x = lds32(xb + j * 256 + frag_lo);
                    xw.y = lds32(xb + j * 256 + frag_hi);
                }
                const f32x2 s = lds_pair(sbase + j * 32);  // scales of activation rows 8j + 2t and 8j + 2t + 1
                f32x2 qsum = 0;
                if (Q41) {
                    const uint2 u = lds64(sbase + j * 32 + QG_SC_BYTES);
                    qsum = pack2((float)(int)u.x, (float)(int)u.y);
                }
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    int d[4];
                    if (Q8) mma_s8(d, a[i], xw.x, xw.y, zero);
                    else mma_s8(d, a[i][0], a[i][1], a[i][2], a[i][3], xw.x, xw.y);
                    f32x2 t0 = mul2(mul2(dd[2 * i], s), pack2((float)d[0], (float)d[1]));
                    f32x2 t1 = mul2(mul2(dd[2 * i + 1], s), pack2((float)d[2], (float)d[3]));
                    if (Q41) {
                        t0 = add2(t0, mul2(mul2(mm[2 * i], s), qsum), one2);
                        t1 = add2(t1, mul2(mul2(mm[2 * i + 1], s), qsum), one2);
                    }
                    run[i][j][0] = add2(run[i][j][0], t0, one2);
                    run[i][j][1] = add2(run[i][j][1], t1, one2);
                }
            }
        }
        __syncthreads();  // this stage is overwritten by the copies issued in the next iteration
        stage = stage + 1 == (uint32_t)D ? 0 : stage + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    const bool plain = !ep.bias && !ep.gelu && !ep.mul && !ep.residual;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const uint32_t m = m0 + j * 8 + 2 * t + c;
            if (m >= M) continue;
            const size_t row = (size_t)m * N;
#pragma unroll
            for (int r = 0; r < MT * 2; ++r) {
                const uint32_t n = n0 + r * 8 + g;
                if (n >= N) continue;
                const f32x2 pair = run[r >> 1][j][r & 1];
                float v = __uint_as_float((uint32_t)(c ? pair >> 32 : pair));
                if (!plain) {
                    if (ep.bias) v = __fadd_rn(v, ep.bias[n]);
                    if (ep.gelu) v = gelu_tanh(v);
                    if (ep.mul) v = __fmul_rn(v, ep.mul[row + n]);
                    if (ep.residual) v = __fadd_rn(ep.residual[row + n], v);
                }
                y[row + n] = v;
            }
        }
}

// ---- the same for products that leave the GPU idle: K split over the warps of a CTA -------------------
// The terms of an output have to be added in block order, but they need not be computed in that order. A CTA owns 16
// activation rows x NTL * 8 weight rows; its eight warps take the quads of K in turn, compute the block terms (activations
// as the A operand of the MMA, weights as B) and leave them in shared memory, and one thread per output then adds them in
// order. Nothing waits for anything until all terms of a round are there, so a launch costs the latency of a few loads and
// one chain of nb adds, where the kernel above walks over all of K with one quad per step. What bounds it: that chain (4
// cycles a block) and the terms' way through shared memory; the products that fill the GPU stay with the kernel above,
// whose sums never leave their registers.
constexpr int kTermWarps = 8;

template <int TYPE>
struct TermQuad {         // what one lane needs of one quad of the activations
    uint32_t a[4][4];     // words t and 4 + t of rows g and g + 8
    float s[2][4];        // their scales
    int32_t qs[2][4];     // and sums (4-bit types)
};
template <int NTL>
struct TermWeights {      // and of the weights
    uint4 w[NTL][2];
    uint4 ws[NTL][2];
};

template <int TYPE, int NTL, bool WIDE>
__global__ void __launch_bounds__(kTermWarps * 32)
gemm_q8_terms_kernel(const uint8_t* __restrict__ qs, const uint8_t* __restrict__ sc, const int8_t* __restrict__ xq,
                     const float* __restrict__ xscale, const int32_t* __restrict__ xqsum, float* __restrict__ y,
                     uint32_t N, uint32_t K, uint32_t M, uint32_t nb, uint32_t scp, uint32_t round_blocks, QgEpilogue ep) {
    constexpr bool Q8 = TYPE == ZQ_TYPE_Q8_0, Q41 = TYPE == ZQ_TYPE_Q4_1;
    constexpr uint32_t QB = Q8 ? 32 : 16, SB = Q41 ? 4 : 2;
    constexpr uint32_t H = WIDE ? 2 : 1;                // WIDE: more than 8 activation rows
    constexpr uint32_t OUTS = 64 * H * NTL;             // outputs of the CTA
    extern __shared__ __align__(16) float terms[];      // [blocks of a round][NTL][row][8 weight rows]
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t nbp = (nb + 3u) & ~3u, n0 = blockIdx.x * (8 * NTL), m0 = blockIdx.y * 16;

    const uint8_t* pw[NTL];
    const uint8_t* ps[NTL][2];
#pragma unroll
    for (int i = 0; i < NTL; ++i) {
        pw[i] = qs + (size_t)min(n0 + i * 8 + g, N - 1) * nbp * QB + 16 * t;
        ps[i][0] = sc + (size_t)min(n0 + i * 8 + 2 * t, N - 1) * scp * SB;
        ps[i][1] = sc + (size_t)min(n0 + i * 8 + 2 * t + 1, N - 1) * scp * SB;
    }
    const uint32_t row_a = min(m0 + g, M - 1), row_b = min(m0 + g + 8, M - 1);
    pdl_launch_dependents();
    // the weight rows on their way into L2 while the kernel before this one still runs (the engines' quantisers, which let this one
    // start early; behind the quantiser of a single call, a plain launch, this begins when that has ended)
    if (tid < 8 * NTL && n0 + tid < N) {
        const uint8_t* row = qs + (size_t)(n0 + tid) * nbp * QB;
        for (uint32_t o = 0; o < nbp * QB; o += 16384) prefetch_l2_bulk(row + o, min(nbp * QB - o, 16384u));
    }
    pdl_wait();

    // U quads of a warp are requested before the first is multiplied (16 rows of 1152 <- 6912 through the
    // public call: 14.3 us with one quad ahead, 13.4 so)
    constexpr int U = WIDE ? (NTL == 1 ? 2 : 1) : (NTL == 1 ? 4 : 2);
    TermQuad<TYPE> xs[U];
    TermWeights<NTL> wts[U];
    auto load = [&](uint32_t q, TermQuad<TYPE>& x, TermWeights<NTL>& wt) {
        auto &w = wt.w, &ws = wt.ws;
#pragma unroll
        for (int i = 0; i < NTL; ++i) {
            w[i][0] = __ldg(reinterpret_cast<const uint4*>(pw[i] + (size_t)q * 4 * QB));
            if (Q8) w[i][1] = __ldg(reinterpret_cast<const uint4*>(pw[i] + (size_t)q * 4 * QB + 64));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (Q41) {
                    ws[i][h] = __ldg(reinterpret_cast<const uint4*>(ps[i][h]) + q);
                } else {
                    const uint2 v = __ldg(reinterpret_cast<const uint2*>(ps[i][h]) + q);
                    ws[i][h].x = v.x;
                    ws[i][h].y = v.y;
                }
            }
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint32_t blk = min(q * 4 + b, nb - 1);  // terms of blocks that do not exist are not stored
#pragma unroll
            for (uint32_t h = 0; h < H; ++h) {
                const uint32_t row = h ? row_b : row_a;
                const uint32_t* p = reinterpret_cast<const uint32_t*>(xq + (size_t)row * K + (size_t)blk * 32) + t;
                x.a[b][h] = p[0];
                x.a[b][2 + h] = p[4];
                x.s[h][b] = xscale[(size_t)row * nb + blk];
                if (!Q8) x.qs[h][b] = xqsum[(size_t)row * nb + blk];
            }
            if (!WIDE) x.a[b][1] = x.a[b][3] = 0;
        }
    };
    auto compute = [&](uint32_t q, uint32_t round0, const TermQuad<TYPE>& x, const TermWeights<NTL>& wt) {
        const auto &w = wt.w, &ws = wt.ws;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            if (q * 4 + b >= nb) break;
            float* to = terms + (size_t)(q * 4 + b - round0) * OUTS + g * 8 + 2 * t;
#pragma unroll
            for (int i = 0; i < NTL; ++i) {
                uint32_t b0, b1;
                if (Q8) {
                    b0 = pick4(w[i][0], b);
                    b1 = pick4(w[i][1], b);
                } else {
                    const uint32_t u = pick4(w[i][0], b);
                    b0 = u & 0x0F0F0F0Fu;
                    b1 = (u >> 4) & 0x0F0F0F0Fu;
                }
                int d[4];
                mma_s8(d, x.a[b][0], x.a[b][1], x.a[b][2], x.a[b][3], b0, b1);
                float dw[2], mw[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint32_t u = Q41 ? pick4(ws[i][c], b) : (b < 2 ? ws[i][c].x : ws[i][c].y);
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u));
                    dw[c] = !Q41 && (b & 1) ? f.y : f.x;
                    mw[c] = f.y;
                }
#pragma unroll
                for (uint32_t h = 0; h < H; ++h) {
                    float v[2];
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        int dot = d[h * 2 + c];
                        if (TYPE == ZQ_TYPE_Q4_0) dot -= 8 * x.qs[h][b];
                        v[c] = __fmul_rn(__fmul_rn(dw[c], x.s[h][b]), (float)dot);
                        if (Q41) v[c] = __fadd_rn(v[c], __fmul_rn(__fmul_rn(mw[c], x.s[h][b]), (float)x.qs[h][b]));
                    }
                    *reinterpret_cast<float2*>(to + (i * H + h) * 64) = make_float2(v[0], v[1]);
                }
            }
        }
    };

    float run = 0.0f;
#pragma unroll 1
    for (uint32_t r0 = 0; r0 < nb; r0 += round_blocks) {
        const uint32_t end = min(r0 + round_blocks, nb);
#pragma unroll 1
        for (uint32_t q = r0 / 4 + warp; q * 4 < end; q += kTermWarps * U) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if ((q + u * kTermWarps) * 4 < end) load(q + u * kTermWarps, xs[u], wts[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if ((q + u * kTermWarps) * 4 < end) compute(q + u * kTermWarps, r0, xs[u], wts[u]);
        }
        __syncthreads();
        if (tid < OUTS) {
            const float* from = terms + tid;
            uint32_t b = 0;
            const uint32_t n = end - r0;
            for (; b + 16 <= n; b += 16) {
                float v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) v[u] = from[(size_t)(b + u) * OUTS];
#pragma unroll
                for (int u = 0; u < 16; ++u) run = __fadd_rn(run, v[u]);
            }
            for (; b < n; ++b) run = __fadd_rn(run, from[(size_t)b * OUTS]);
        }
        __syncthreads();
    }
    if (tid < OUTS) {
        const uint32_t n = n0 + tid / (64 * H) * 8 + (tid & 7u), m = m0 + ((tid >> 3) & 7u) + (tid / 64 % H) * 8;
        if (n < N && m < M) {
            const size_t o = (size_t)m * N + n;
            float v = run;
            if (ep.bias) v = __fadd_rn(v, ep.bias[n]);
            if (ep.gelu) v = gelu_tanh(v);
            if (ep.mul) v = __fmul_rn(v, ep.mul[o]);
            if (ep.residual) v = __fadd_rn(ep.residual[o], v);
            y[o] = v;
        }
    }
}

// Shared memory that a grid asks for: `need`, or as much as leaves no SM room for more than its share of the CTAs.
// Under programmatic launches the CTAs of a grid are placed while those of the kernels before it still sit on the SMs, and
// small ones are then stacked on a few of them. (B200, prompts and steps of several sequences, ms without and with it, products
// of this file only: eight sequences of 4_1 weights 33.4 and 31.4, six of 4_0 17.2 and 15.6, four of 8_0 21.7 and 20.6; a prompt of 600
// tokens and 17 steps of 8_0 30.9 and 29.9. Alone: 1152 <- 6912 4_0 at 12 and 17 rows, 144 CTAs, 12.4 -> 11.7 and 16.7 -> 16.0 us.)
constexpr uint32_t kAlone = 115 * 1024;  // no second CTA finds as much
uint32_t spread_smem(uint64_t ctas, uint32_t need) {
    const uint64_t sms = (uint64_t)sm_count(), share = (ctas + sms - 1) / sms;
    const uint64_t spread = (227 * 1024 / (share + 1) + 128) & ~(uint64_t)127;
    return spread < need ? need : spread > kAlone ? kAlone : (uint32_t)spread;
}

constexpr uint32_t kMostGridY = 65535;

template <int TYPE, int NTL, bool WIDE>
int launch_terms(const zq_weight* w, const int8_t* xq, const float* xs, const int32_t* xsum, float* y, uint32_t M,
                 QgEpilogue ep, bool split, cudaStream_t st) {
    constexpr uint32_t kBlockBytes = (WIDE ? 128 : 64) * NTL * 4;
    constexpr uint32_t kMost = 112 * 1024 / kBlockBytes / 4 * 4;  // two CTAs share an SM
    const uint32_t rounds = (w->nb + kMost - 1) / kMost, per = ((w->nb + rounds - 1) / rounds + 3) / 4 * 4;
    const dim3 grid((w->out_dim + 8 * NTL - 1) / (8 * NTL), (M + 15) / 16);
    if (grid.y > kMostGridY) return ZQ_ERR_LIMIT;
    auto kern = gemm_q8_terms_kernel<TYPE, NTL, WIDE>;
    const uint32_t smem = spread_smem((uint64_t)grid.x * grid.y, per * kBlockBytes);
    // the most that any call asks for: the limit is the process's, and another thread may be about to launch a deeper matrix
    ZQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAlone));
    ZQ_CUDA(launch_pdl_split(split, kern, grid, dim3(kTermWarps * 32), smem, st, w->qs,
                       static_cast<const uint8_t*>(w->sc), xq, xs, xsum, y, w->out_dim, w->in_dim, M, w->nb, w->scp, per, ep));
    return ZQ_OK;
}

template <int TYPE, int W, int MT, int NT, int D>
int launch_cfg(const zq_weight* w, const int8_t* xq, const float* xs, const int32_t* xsum, float* y, uint32_t M,
               QgEpilogue ep, bool split, cudaStream_t st) {
    const dim3 grid((w->out_dim + W * MT * 16 - 1) / (W * MT * 16), (M + NT * 8 - 1) / (NT * 8));
    if (grid.y > kMostGridY) return ZQ_ERR_LIMIT;
    constexpr uint32_t kRing = D * QgStage<TYPE, W, MT, NT>::kBytes;
    static_assert(kRing <= kAlone, "ring");
    const uint32_t smem = spread_smem((uint64_t)grid.x * grid.y, kRing);
    auto kern = gemm_q8_kernel<TYPE, W, MT, NT, D>;
    // the most that any call asks for: the limit is the process's, and another thread may be about to launch a larger grid
    ZQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAlone));
    ZQ_CUDA(launch_pdl_split(split, kern, grid, dim3(W * 32), smem, st, w->qs,
                       static_cast<const uint8_t*>(w->sc), xq, xs, xsum, y, w->out_dim, w->in_dim, M, w->nb, w->scp, 1.0f, ep));
    return ZQ_OK;
}

// CTA shape: the one whose busiest SM is through first, by a count of nanoseconds. A CTA holds W * MT * NT MMA tiles. An SM that is full
// takes `tile` for one of them and a block of K, and `tile_start` for the start and the sums of each; no warp is through its own tiles
// before `block` for a block and `start`; of the two a geometric sum. The constants are a fit to 671 calls of 17 matrices (96 to 6912
// columns) at 2 to 1000 rows, in all five shapes, nudged where the choice was not the fastest: it is within 11 % of the fastest for each
// type, 0.3 to 0.7 % in the mean (the count of blocks alone, the same for all types, within 34 %, 1.5 to 5.1 % in the mean).
// Measured on a B200 with the quantiser, weights from HBM, us for shapes 0 to 4, the one taken in brackets: 30000 <- 320 8_0 at 333 rows 43.6, [41.9],
// 47.3, 55.8, 101; 30000 <- 640 4_1 at 333 rows 97.3, [74.1], 90.5, 93.6, 126; 3000 <- 512 4_0 at 24 rows 8.8, 6.8, 6.2, 4.9, [4.3]; 8000 <- 1152 4_1 at
// 200 rows 38.7, [28.0], 31.8, 31.4, 40.4; 1152 <- 6912 8_0 at 140 rows 94.5, 57.8, 43.3, [39.0], 41.9. A shape whose rows of CTAs are more than a
// grid has is left out; the first one, of the most columns, remains for the launch to refuse.
template <int TYPE>
int cheapest_shape(uint32_t n, uint32_t m, uint32_t nb, uint32_t sms) {
    struct Shape {
        uint32_t rows, cols, tiles;
        float tile, tile_start, block, start;
    };
    constexpr bool Q41 = TYPE == ZQ_TYPE_Q4_1, Q8 = TYPE == ZQ_TYPE_Q8_0;
    constexpr Shape shapes[5] = {
        Q41 ? Shape{128, 64, 64, 6.9f, 8, 222, 290} : Q8 ? Shape{128, 64, 64, 5.2f, 10, 263, 0} : Shape{128, 64, 64, 4.5f, 11, 154, 22},
        Q41 ? Shape{128, 32, 32, 6.1f, 6, 170, 65} : Q8 ? Shape{128, 32, 32, 5.5f, 13, 179, 0} : Shape{128, 32, 32, 4.8f, 9, 148, 0},
        Q41 ? Shape{64, 32, 16, 7.3f, 12, 161, 96} : Q8 ? Shape{64, 32, 16, 6.2f, 16, 146, 150} : Shape{64, 32, 16, 5.7f, 12, 144, 170},
        Q41 ? Shape{64, 16, 8, 7.5f, 20, 101, 78} : Q8 ? Shape{64, 16, 8, 7.7f, 27, 93, 190} : Shape{64, 16, 8, 7.3f, 19, 92, 122},
        Q41 ? Shape{64, 8, 4, 10.8f, 35, 86, 0} : Q8 ? Shape{64, 8, 4, 14.9f, 60, 77, 1} : Shape{64, 8, 4, 11.3f, 35, 90, 0}};
    int best = 0;
    float least = INFINITY;
    for (int i = 0; i < 5; ++i) {
        const Shape& s = shapes[i];
        if (i && (m - 1) / s.cols >= kMostGridY) continue;
        const uint64_t ctas = (uint64_t)((n + s.rows - 1) / s.rows) * ((m - 1) / s.cols + 1);
        const float full = (float)((ctas + sms - 1) / sms * s.tiles) * (s.tile * nb + s.tile_start), warp = s.block * nb + s.start;
        const float cost = full * full + warp * warp;
        if (cost < least) {
            least = cost;
            best = i;
        }
    }
    return best;
}

template <int TYPE>
int launch_one(const zq_weight* w, const int8_t* xq, const float* xs, const int32_t* xsum, float* y, uint32_t M,
               QgEpilogue ep, bool split, cudaStream_t st) {
    // Few tiles of 8 weight rows x 16 activation rows: K split over the warps. How many tiles it may be depends on K, whose
    // blocks are what the warps share (below 16 to 24 of them the kernel above is ahead), and on how many CTAs run at once: two
    // per SM, up to 8 rows with one weight tile or with 4_1 weights one. More pay where the kernel above pads an odd number of
    // 8-row tiles to an even one, or unpacks 4_1; fewer where it reads whole bytes, a ring of which is on its way from HBM
    // before the kernel ahead has ended. Two weight tiles per CTA once one would give more CTAs than run at once.
    // (B200, the kernel above and then this form. Graph-timed with the quantiser, us: 1152 <- 6912 8_0 at 8 rows 25.4 and 10.9,
    // 1152 <- 1024 at 16 rows 6.7 and 5.1, 4736 <- 1152 8_0 at 8 rows 7.5 and 6.2; left to the kernel above: 1536 <- 256 at 8
    // rows 4.3 and 5.8, 3072 <- 768 4_1 at 8 rows 6.4 and 6.8. Whole Gemma-3-1B steps, ms: 40 sequences of 8_0 2.59 and 2.29, of
    // 4_1 3.02 and 2.65; left to the kernel above: 32 sequences of 8_0 2.09 and 2.14, 48 of 8_0 2.31 and 2.43.)
    const uint64_t tiles = (uint64_t)((w->out_dim + 7) / 8) * ((M + 15) / 16), sms = (uint64_t)sm_count();
    const uint32_t nb = w->nb;
    constexpr bool Q41 = TYPE == ZQ_TYPE_Q4_1, Q8 = TYPE == ZQ_TYPE_Q8_0;
    if (M <= 8 && (tiles <= 2 * sms ? nb >= 16 : tiles <= 4 * sms && nb >= (Q41 ? 48 : 20)))
        return tiles <= sms ? launch_terms<TYPE, 1, false>(w, xq, xs, xsum, y, M, ep, split, st)
                            : launch_terms<TYPE, 2, false>(w, xq, xs, xsum, y, M, ep, split, st);
    const bool padded = (M + 7) / 8 & 1u;
    const uint64_t most = Q41 || padded ? 480 : Q8 && M > 16 ? 192 : 2 * sms;
    if (M > 8 && (tiles <= sms ? nb >= 16 : tiles <= most && nb >= 24))
        return tiles <= 192 ? launch_terms<TYPE, 1, true>(w, xq, xs, xsum, y, M, ep, split, st)
                            : launch_terms<TYPE, 2, true>(w, xq, xs, xsum, y, M, ep, split, st);
    switch (cheapest_shape<TYPE>(w->out_dim, M, nb, (uint32_t)sms)) {
        case 0: return launch_cfg<TYPE, 8, 1, 8, 3>(w, xq, xs, xsum, y, M, ep, split, st);
        case 1: return launch_cfg<TYPE, 4, 2, 4, 3>(w, xq, xs, xsum, y, M, ep, split, st);
        case 2: return launch_cfg<TYPE, 4, 1, 4, 3>(w, xq, xs, xsum, y, M, ep, split, st);
        case 3: return launch_cfg<TYPE, 4, 1, 2, 4>(w, xq, xs, xsum, y, M, ep, split, st);
        default: return launch_cfg<TYPE, 4, 1, 1, 6>(w, xq, xs, xsum, y, M, ep, split, st);
    }
}

}  // namespace

int launch_gemm_q8(const zq_weight* w, const int8_t* xq, const float* xscale, const int32_t* xsum, float* y,
                   uint32_t m_rows, const zq_epilogue* ep, cudaStream_t st, bool shared_split) {
    QgEpilogue a{nullptr, nullptr, nullptr, 0};
    if (ep) {
        a.bias = ep->d_bias;
        a.gelu = ep->gelu;
        a.mul = ep->d_mul;
        a.residual = ep->d_residual;
    }
    switch (w->type) {
        case ZQ_TYPE_Q4_0: return launch_one<ZQ_TYPE_Q4_0>(w, xq, xscale, xsum, y, m_rows, a, shared_split, st);
        case ZQ_TYPE_Q4_1: return launch_one<ZQ_TYPE_Q4_1>(w, xq, xscale, xsum, y, m_rows, a, shared_split, st);
        case ZQ_TYPE_Q8_0: return launch_one<ZQ_TYPE_Q8_0>(w, xq, xscale, xsum, y, m_rows, a, shared_split, st);
        default: return ZQ_ERR_UNSUPPORTED;
    }
}

}  // namespace zq
