// Linears over bf16 weights for few activation rows: one warp (or, for short deep matrices, the four warps of a
// CTA) per few weight rows, 16-byte weight loads one to four steps ahead of their use, the first of them ahead of the wait
// for the producing kernel. f32 activations take this path for any number of rows; many bf16 rows go to the
// tensor cores (gemm_bf16.cu).
#include "dense.h"

namespace zq {
namespace {

constexpr int kGemvWarps = 4;

struct GemvParams {
    const bf16* w;
    uint32_t kp;
    const void* x;
    uint32_t T;
    void* y;              // f32 outputs, or activation outputs of a GLU
    uint32_t y_stride;
    LinGroups groups;
    GluSpec glu;
    bool prefetch;        // ask L2 for the warp's whole rows while the producing kernel still runs
    // mixture of experts: blockIdx.y = pair (then the tokens of the shared expert)
    const int32_t* ids;
    const float* weights;  // of the pairs' inputs (null: 1)
    uint32_t top, n_pairs, rows_per_expert;
    bool x_by_pair;       // x row = pair (down projection) instead of token
    const bf16* w_shared;
    uint32_t kp_shared, rows_shared;
    const void* x_shared;  // x rows of the shared expert when x_by_pair
    uint32_t y_stride_shared;
    void* y_shared;
    GluSpec glu_shared;
};

// Sums and products of two neighbouring columns at once: half the instructions of scalar multiply-adds.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 pair_of(float lo, float hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float pair_sum(f32x2 a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
    return lo + hi;
}
// Eight consecutive activations as they lie in memory, and as four pairs.
template <typename TX>
struct XChunk;
template <>
struct XChunk<bf16> {
    uint4 v;
};
template <>
struct XChunk<float> {
    float4 a, b;
};
__device__ __forceinline__ void pairs(const uint4& u, f32x2 (&f)[4]) {
    f[0] = pair_of(bf16_lo(u.x), bf16_hi(u.x));
    f[1] = pair_of(bf16_lo(u.y), bf16_hi(u.y));
    f[2] = pair_of(bf16_lo(u.z), bf16_hi(u.z));
    f[3] = pair_of(bf16_lo(u.w), bf16_hi(u.w));
}
__device__ __forceinline__ void pairs(const XChunk<bf16>& x, f32x2 (&f)[4]) { pairs(x.v, f); }
__device__ __forceinline__ void pairs(const XChunk<float>& x, f32x2 (&f)[4]) {
    f[0] = pair_of(x.a.x, x.a.y);
    f[1] = pair_of(x.a.z, x.a.w);
    f[2] = pair_of(x.b.x, x.b.y);
    f[3] = pair_of(x.b.z, x.b.w);
}
// Sums of N values over a warp. While the count is even a lane keeps half of its values and hands the other half on (16
// values cost 16 exchanges in place of 80); it ends with the sums of the values from `result` on, as many as
// N's odd part.
template <int N, int OFF, int M>
__device__ __forceinline__ uint32_t warp_sums(float (&v)[M], uint32_t lane) {
    if constexpr (OFF == 0) {
        return 0;
    } else if constexpr (N % 2 == 0) {
        const bool upper = lane & OFF;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            const float give = upper ? v[i] : v[i + N / 2], keep = upper ? v[i + N / 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, OFF);
        }
        return (upper ? N / 2 : 0) + warp_sums<N / 2, OFF / 2>(v, lane);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xFFFFFFFFu, v[i], OFF);
        return warp_sums<N, OFF / 2>(v, lane);
    }
}

// TR activation rows x RW weight rows per warp; SK: the four warps share the rows and split K.
// Bound: for one row the latency of a step's chain of launches (a layer's matrices come from L2 ahead of their turn, the vocabulary's
// at 5.3 TB/s); for several rows the instructions on the activations, which every warp unpacks for itself. Hence pairs of columns per
// multiply-add, a reduction by halves, chunks requested again as soon as they are used, and a form for 3 and for 6 rows: at 6 rows of
// 768 a layer's matrix takes 2.6 us of a step's chain in place of 4.7, the 50304-row vocabulary 32 us in place of 39 (77 MB, 12 us at
// the memory's rate: short rows leave a warp three chunks and a reduction).
// GLU: RW counts features, each one gate and one up row.
// Chunks of a weight row that a lane holds ahead, and the CTAs that an SM has to hold (a bound on the registers), of a kernel for TR
// activation rows and NR weight rows per warp. More chunks hide the memory, more CTAs let a layer's grid run at once; past what the
// registers hold either one spills. The general rule is for the forms without a line of their own: as many CTAs as cost no spills (five for
// six rows of two weight rows, 28.8 and 43.9 us for 50304 <- 768 and <- 1152 against 30.1 and 45.2 with four; eight rows spill with five,
// 42.0 and 65.9 against 33.8 and 52.5 with four). A line of its own has each form that the rule made slower than the kernel of
// scalar multiply-adds ahead of it was, with the fastest choice of 1, 2, 4 chunks and 1, 3 to 6, 8, 9 CTAs that is not (B200, us, that kernel, the
// rule, the line): gated bf16, 9000 <- 1152, one row 9.2, 9.4, 8.3, two rows 10.9, 11.7, 10.0; bf16 50304 <- 1152, one row 20.9,
// 22.0, 20.6, two rows 25.4, 29.1, 23.8, eight rows 50.7, 52.5, 50.2; 1152 <- 6912, two rows 4.86, 5.54, 4.28; f32 2304 <- 768, one row
// 2.32, 2.50, 1.90, six rows 5.1, 5.9, 4.0, eight rows 5.2, 7.2, 5.1; f32 768 <- 3072, one, two and four rows 2.33, 2.70, 2.31, 3.25, 3.58, 3.26 and
// 4.75, 5.24, 4.80; f32 50304 <- 1152, one, two and four rows 21.1, 23.6, 20.9, 27.0, 30.5, 26.0 and 42.8, 44.9, 37.1. (One gated row with two
// chunks and six CTAs is faster alone, 6.4 in place of 7.1 for 6912 <- 1152, and in a step of Lenisun, 146.6 us of 148.3 for four layers, but not in
// one of Vepinex, 184.2 of 179.6 for six.)
struct GemvChoice {
    int ahead, ctas;
};
template <typename TX, int TR, int RW, bool SK, bool GLU, bool MOE>
constexpr GemvChoice gemv_choice() {
    constexpr bool F32 = sizeof(TX) == 4;
    constexpr int NR = GLU ? 2 * RW : RW;
    constexpr int ahead = TR == 1 ? (NR == 1 ? 4 : 2) : NR * TR > 16 ? 1 : NR * TR > 8 ? 2 : 4;
    if (MOE) return {ahead, 5};
    if (GLU) {
        if (TR == 1 && RW == 2) return F32 ? GemvChoice{4, 4} : GemvChoice{1, 8};
        if (TR == 2 && RW == 2) return {2, 4};
        if (TR == 2 && F32) return {2, 6};
        return {ahead, TR == 1 ? 6 : 1};
    }
    if (TR == 1) {
        if (RW == 2) return {2, 9};
        return F32 ? (SK ? GemvChoice{1, 8} : GemvChoice{1, 3}) : GemvChoice{ahead, 9};
    }
    if (TR == 2 && SK) return F32 ? GemvChoice{1, 8} : GemvChoice{2, 8};
    if (TR == 2 && RW == 2) return F32 ? GemvChoice{2, 6} : GemvChoice{1, 9};
    if (F32) {
        if (TR == 4 && RW == 2) return {2, 6};
        if (TR == 4 && SK) return {1, 1};
        if (TR >= 6 && RW == 1 && !SK) return {4, 4};
        return {ahead, 3};
    }
    if (TR == 8 && RW == 2) return {4, 3};
    return {ahead, RW == 2 && TR != 6 ? 4 : 5};
}
template <typename TX, int TR, int RW, bool SK, bool GLU, bool MOE>
struct GemvShape {
    static constexpr int ahead = gemv_choice<TX, TR, RW, SK, GLU, MOE>().ahead, ctas = gemv_choice<TX, TR, RW, SK, GLU, MOE>().ctas;
};
template <typename TX, int TR, int RW, bool SK, bool GLU, bool MOE>
__global__ void __launch_bounds__(kGemvWarps * 32, GemvShape<TX, TR, RW, SK, GLU, MOE>::ctas)
dense_gemv_kernel(const __grid_constant__ GemvParams p) {
    constexpr int NR = GLU ? 2 * RW : RW, P = RW * TR;
    __shared__ float red[SK ? kGemvWarps * NR * TR : 1];
    pdl_launch_dependents();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t j0 = (SK ? blockIdx.x : blockIdx.x * kGemvWarps + warp) * RW;
    const bf16* w = p.w;
    uint32_t kp = p.kp, rows, w_row0, x_row0, y_col = 0, t0 = 0, nt = TR, y_stride = p.y_stride;
    const TX* x = static_cast<const TX*>(p.x);
    void* yv = p.y;
    float in_scale = 1.0f;
    GluSpec glu = p.glu;
    uint32_t pair = 0, y_row0;
    bool waited = false;
    if (MOE) {
        pair = blockIdx.y;
        if (pair < p.n_pairs) {
            pdl_wait();
            waited = true;
            rows = p.rows_per_expert;
            w_row0 = (uint32_t)p.ids[pair] * (GLU ? 2 * rows : rows);
            x_row0 = p.x_by_pair ? pair : pair / p.top;
            if (GLU && p.weights) in_scale = p.weights[pair];
            y_row0 = pair;
        } else {
            const uint32_t t = pair - p.n_pairs;
            w = p.w_shared;
            kp = p.kp_shared;
            rows = p.rows_shared;
            w_row0 = 0;
            if (p.x_by_pair) x = static_cast<const TX*>(p.x_shared);
            x_row0 = t;
            y_row0 = t;
            yv = p.y_shared;
            y_stride = p.y_stride_shared;
            glu = p.glu_shared;
        }
    } else {
        const LinGroup g = p.groups.g[blockIdx.y];
        rows = g.rows;
        w_row0 = g.w_row;
        t0 = blockIdx.z * TR;
        nt = p.T - t0 < (uint32_t)TR ? p.T - t0 : TR;
        x_row0 = g.x_row + t0;
        y_row0 = t0;
        y_col = g.y_col;
    }
    if (j0 >= rows) return;  // uniform over the warp (over the CTA with SK)

    const uint4* wr[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const uint32_t j = min(j0 + (GLU ? r / 2 : r), rows - 1);
        const uint32_t row = w_row0 + (GLU ? glu_row(j, r & 1) : j);
        wr[r] = reinterpret_cast<const uint4*>(w + (size_t)row * kp);
    }
    if (!MOE && p.prefetch && lane < NR && (!SK || warp == 0)) {
        const uint32_t j = min(j0 + (GLU ? lane / 2 : lane), rows - 1);
        prefetch_l2_bulk(w + (size_t)(w_row0 + (GLU ? glu_row(j, lane & 1) : j)) * kp, kp * 2);
    }
    const XChunk<TX>* xr[TR];
#pragma unroll
    for (int t = 0; t < TR; ++t)
        xr[t] = reinterpret_cast<const XChunk<TX>*>(x + (size_t)(x_row0 + min((uint32_t)t, nt - 1)) * kp);

    const uint32_t n_chunks = kp / 8;  // 16 bytes of a weight row each
    constexpr uint32_t step = SK ? kGemvWarps * 32 : 32;
    uint32_t c = SK ? threadIdx.x : lane;
    f32x2 sums[NR][TR];  // of the even and of the odd columns
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int t = 0; t < TR; ++t) sums[r][t] = 0;

    // Chunks of a lane held ahead, of the weights and of the activations: a chunk's registers are loaded again as soon as it is used.
    constexpr int U = GemvShape<TX, TR, RW, SK, GLU, MOE>::ahead;
    constexpr int V = TR * sizeof(TX) <= 2 ? U : TR * sizeof(TX) <= 8 && U > 1 ? 2 : 1;
    uint4 wq[U][NR];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < NR; ++r)
            wq[u][r] = c + u * step < n_chunks ? __ldg(wr[r] + c + u * step) : make_uint4(0, 0, 0, 0);
    if (!waited) pdl_wait();
    XChunk<TX> xq[V][TR];
#pragma unroll
    for (int v = 0; v < V; ++v)
        if (c + v * step < n_chunks)
#pragma unroll
            for (int t = 0; t < TR; ++t) xq[v][t] = xr[t][c + v * step];
    for (; c < n_chunks; c += U * step) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t cc = c + u * step;
            if (cc >= n_chunks) break;
            f32x2 wf[NR][4];
#pragma unroll
            for (int r = 0; r < NR; ++r) pairs(wq[u][r], wf[r]);
            if (cc + U * step < n_chunks)
#pragma unroll
                for (int r = 0; r < NR; ++r) wq[u][r] = __ldg(wr[r] + cc + U * step);
            const bool more = cc + V * step < n_chunks;
#pragma unroll
            for (int t = 0; t < TR; ++t) {
                f32x2 xf[4];
                pairs(xq[u % V][t], xf);
                if (more) xq[u % V][t] = xr[t][cc + V * step];
#pragma unroll
                for (int r = 0; r < NR; ++r)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sums[r][t] = fma2(wf[r][e], xf[e], sums[r][t]);
            }
        }
    }
    float val[P], up[GLU ? P : 1];
#pragma unroll
    for (int i = 0; i < P; ++i) {
        val[i] = pair_sum(sums[GLU ? 2 * (i / TR) : i / TR][i % TR]);
        if (GLU) up[i % (GLU ? P : 1)] = pair_sum(sums[(2 * (i / TR) + 1) % NR][i % TR]);
    }
    const uint32_t first = warp_sums<P, 16>(val, lane);
    if (GLU) warp_sums<GLU ? P : 1, 16>(up, lane);
    auto write = [&](uint32_t i, float v, float u) {
        const uint32_t f = i / TR, t = i % TR;
        if (j0 + f >= rows || t >= nt) return;
        const size_t o = (size_t)(y_row0 + t) * y_stride + y_col + j0 + f;
        if (GLU)
            static_cast<TX*>(yv)[o] = to_act<TX>(glu_value(v * in_scale, u * in_scale, glu.kind, glu.limit));
        else
            static_cast<float*>(yv)[o] = v;
    };
    constexpr int KEPT = P / (P & -P), LANES = 32 / (P & -P);  // LANES neighbours have the same KEPT sums
    if (!SK) {
        if (lane % LANES == 0)
#pragma unroll
            for (int k = 0; k < KEPT; ++k) write(first + k, val[k], up[GLU ? k : 0]);
        return;
    }
    if (lane % LANES == 0)
#pragma unroll
        for (int k = 0; k < KEPT; ++k) {
            red[warp * NR * TR + first + k] = val[k];
            if (GLU) red[warp * NR * TR + P + first + k] = up[GLU ? k : 0];
        }
    __syncthreads();
    if (threadIdx.x >= P) return;
    const float* part = red + threadIdx.x;
    float v = part[0], u = GLU ? part[P] : 0.0f;
#pragma unroll
    for (int q = 1; q < kGemvWarps; ++q) {
        v += part[q * NR * TR];
        if (GLU) u += part[q * NR * TR + P];
    }
    write(threadIdx.x, v, u);
}

template <typename TX, int TR, bool GLU, bool MOE>
int gemv_shape(GemvParams p, uint32_t rows, uint32_t kp, uint32_t gy, uint32_t gz, cudaStream_t st) {
    p.prefetch = (uint64_t)rows * (GLU ? 2 : 1) * gy * kp * 2 <= (64u << 20);  // a part of L2 at most
    // Two rows (features) per warp when there are warps enough to fill the GPU that way, the K split when one row
    // per warp does not.
    const uint64_t per_sm = (uint64_t)sm_count() * 16;
    const uint64_t total = (uint64_t)rows * gy * gz;
    cudaError_t e;
    if (total >= 2 * per_sm) {
        e = launch_pdl(dense_gemv_kernel<TX, TR, 2, false, GLU, MOE>, dim3((rows + 2 * kGemvWarps - 1) / (2 * kGemvWarps), gy, gz),
                       dim3(kGemvWarps * 32), 0, st, p);
    } else if (total < per_sm && kp >= 1024) {
        e = launch_pdl(dense_gemv_kernel<TX, TR, 1, true, GLU, MOE>, dim3(rows, gy, gz), dim3(kGemvWarps * 32), 0, st, p);
    } else {
        e = launch_pdl(dense_gemv_kernel<TX, TR, 1, false, GLU, MOE>, dim3((rows + kGemvWarps - 1) / kGemvWarps, gy, gz),
                       dim3(kGemvWarps * 32), 0, st, p);
    }
    if (e != cudaSuccess) return cuda_fail(e);
    return ZQ_OK;
}

template <typename TX, bool GLU>
int gemv_rows(const GemvParams& p, uint32_t rows, uint32_t n_groups, cudaStream_t st) {
    if (p.T == 1) return gemv_shape<TX, 1, GLU, false>(p, rows, p.kp, n_groups, 1, st);
    if (p.T == 2) return gemv_shape<TX, 2, GLU, false>(p, rows, p.kp, n_groups, 1, st);
    if (p.T == 3) return gemv_shape<TX, 3, GLU, false>(p, rows, p.kp, n_groups, 1, st);
    if (p.T == 4) return gemv_shape<TX, 4, GLU, false>(p, rows, p.kp, n_groups, 1, st);
    if (p.T <= 6) return gemv_shape<TX, 6, GLU, false>(p, rows, p.kp, n_groups, 1, st);
    return gemv_shape<TX, 8, GLU, false>(p, rows, p.kp, n_groups, (p.T + 7) / 8, st);
}

}  // namespace

int launch_dense_linear(const DenseWeight& W, const LinGroups& G, const void* x, uint32_t x_rows, uint32_t T, float* y,
                        uint32_t y_stride, bool f32, cudaStream_t st, Addends* add, size_t y_floats) {
    if (add) *add = Addends{};
    if (T == 0) return ZQ_OK;
    if (!f32 && T >= kDenseGemmMinRows)
        return launch_gemm_bf16(W, G, static_cast<const bf16*>(x), x_rows, T, y, y_stride, nullptr, 0, nullptr, st, add,
                                y_floats);
    GemvParams p{};
    p.w = W.w;
    p.kp = W.kp;
    p.x = x;
    p.T = T;
    p.y = y;
    p.y_stride = y_stride;
    p.groups = G;
    uint32_t rows = 0;
    for (uint32_t i = 0; i < G.n; ++i) rows = rows > G.g[i].rows ? rows : G.g[i].rows;
    return f32 ? gemv_rows<float, false>(p, rows, G.n, st) : gemv_rows<bf16, false>(p, rows, G.n, st);
}

int launch_dense_glu(const DenseWeight& W, const void* x, uint32_t T, void* out, GluSpec glu, bool f32, cudaStream_t st) {
    if (T == 0) return ZQ_OK;
    const uint32_t ffp = W.rows / 2;
    if (!f32 && T >= kDenseGemmMinRows)
        return launch_gemm_bf16(W, one_group(W.rows), static_cast<const bf16*>(x), T, T, nullptr, 0, static_cast<bf16*>(out),
                                ffp, &glu, st);
    GemvParams p{};
    p.w = W.w;
    p.kp = W.kp;
    p.x = x;
    p.T = T;
    p.y = out;
    p.y_stride = ffp;
    p.groups = one_group(ffp);
    p.glu = glu;
    return f32 ? gemv_rows<float, true>(p, ffp, 1, st) : gemv_rows<bf16, true>(p, ffp, 1, st);
}

int launch_moe_pairs(const MoeWeights& M, const MoeRouting& R, const void* x, uint32_t T, void* hidden, float* parts,
                     bool f32, cudaStream_t st) {
    if (T == 0) return ZQ_OK;
    const uint32_t pairs = T * M.top, gy = pairs + (M.shared_ffp ? T : 0);
    if (gy > 65535) return ZQ_ERR_LIMIT;
    GemvParams p{};
    p.ids = R.ids;
    p.weights = M.scale_input ? R.weights : nullptr;
    p.top = M.top;
    p.n_pairs = pairs;
    // gate | up of every pair
    p.w = M.gate_up.w;
    p.kp = M.gate_up.kp;
    p.x = x;
    p.y = hidden;
    p.y_stride = M.ffp;
    p.rows_per_expert = M.ffp;
    p.glu = M.glu;
    p.glu_shared = M.shared_glu;
    p.w_shared = M.shared_gate_up.w;
    p.kp_shared = M.shared_gate_up.kp;
    p.rows_shared = M.shared_ffp;
    p.y_stride_shared = M.shared_ffp;
    void* hidden_shared = static_cast<char*>(hidden) + (size_t)pairs * M.ffp * act_bytes(f32);
    p.y_shared = hidden_shared;
    const uint32_t rows = M.ffp > M.shared_ffp ? M.ffp : M.shared_ffp;
    int rc = f32 ? gemv_shape<float, 1, true, true>(p, rows, p.kp, gy, 1, st)
                 : gemv_shape<bf16, 1, true, true>(p, rows, p.kp, gy, 1, st);
    if (rc != ZQ_OK) return rc;
    // down
    p.w = M.down.w;
    p.kp = M.down.kp;
    p.x = hidden;
    p.x_by_pair = true;
    p.x_shared = hidden_shared;
    p.y = parts;
    p.y_stride = M.width;
    p.rows_per_expert = M.width;
    p.w_shared = M.shared_down.w;
    p.kp_shared = M.shared_down.kp;
    p.rows_shared = M.width;
    p.y_shared = parts + (size_t)pairs * M.width;
    p.y_stride_shared = M.width;
    return f32 ? gemv_shape<float, 1, false, true>(p, M.width, p.kp, gy, 1, st)
               : gemv_shape<bf16, 1, false, true>(p, M.width, p.kp, gy, 1, st);
}

}  // namespace zq
