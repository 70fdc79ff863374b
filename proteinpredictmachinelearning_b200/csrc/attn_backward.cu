// Flash-attention backward (the reference's flash_attn_backward_cuda, src/cuda/FlashAttnKernel.cu:1524, same math as
// flash_attn_backward_cpu, src/ops/FlashAttn.cpp:144-216), exact fp32 on CUDA cores, without atomics:
//
//   P_ij = exp(S_ij - LSE_i),  D_i = sum_d dO_id O_id,  dP_ij = sum_d dO_id V_jd,  dS_ij = P_ij (dP_ij - D_i)
//   dQ_id = scale sum_j dS_ij K_jd     dK_jd = scale sum_i dS_ij Q_id     dV_jd = sum_i P_ij dO_id     dbias_ij = dS_ij
//
// Two kernels, each recomputing the scores of its tiles (nothing but the outputs is written, every output element is
// written exactly once, so no zero-fill pass and no atomic adds: the results do not depend on the launch order):
//   attn_bwd_dq_kernel   one CTA = 64 query rows of one (batch, head); walks the key tiles of 64; writes dQ and dbias
//   attn_bwd_dkv_kernel  one CTA = 64 key rows of one (batch, head); walks the query tiles of 64; writes dK and dV
// Per tile: scores and dP as register tiles over the channels, exp and dS in registers, dS (and P, one after the other through
// the same buffer) to shared memory as [partner][own row], then the result's register tile over the partners (attn_tile.cuh).  A
// causal row takes nothing from the partner rows beyond its diagonal, whatever values they hold.
//
// Bound: instruction issue (fp32 FMAs are half of it: 3 products in one kernel, 4 in the other; FMA pipe 45 % busy at two CTAs
// per SM).  64 x 8 x 256 x 32 with dbias 1535 -> 498 us (30 TFLOP/s over the seven products), head dim 8 613 -> 251 us, against
// 32-row tiles with a warp per 8 rows, whose lanes read one scalar from shared memory per FMA or two.  The next tile and this
// tile's bias are requested before the products (255 registers, two CTAs per SM): 573 us with three CTAs per SM that wait for
// them.  Sequences that fit one tile of 32 rows keep that form (attn_backward_short.cu, with both sides' times); above, the
// 64-row tiles are faster throughout, also where they are emptiest (256 x 8, 33 rows: 120 -> 74, 343 -> 138 and 641 -> 251 us for
// head dims 8, 32 and 64; 72 rows: 279 -> 249, 801 -> 495, 1434 -> 903).
// Layouts as the forward: Q, K, V, O, dO, dQ, dK, dV [B, h, L, d]; bias [B, h, L, L] with a batch stride (0: shared);
// dbias [B, h, L, L]; LSE [B, h, L].  d <= 64.
#include <cuda_runtime.h>
#include <math_constants.h>

#include "attn_tile.cuh"
#include "kernels.h"

namespace ppml_b200 {

namespace {

struct BwdParams {
    int B, H, L, d, causal;
    float scale;
    const float *Q, *K, *V, *bias, *O, *dO, *LSE;
    long long bias_batch_stride;
    float *dQ, *dK, *dV, *dbias;
    int vec_in;             // rows of Q, K, V, O, dO in 16-byte pieces
    int vec_out;            // rows of dQ, dK, dV
    int vec_bias;           // rows of bias; vec_dbias: rows of dbias
    int vec_dbias;
};

constexpr int kT = kAttnTile;

// D_i of the 64 query rows whose dO and O rows are in registers: a row lies in DP / 4 neighbouring lanes
template <int DP>
__device__ __forceinline__ void store_row_dots(const AttnRows<DP>& g, const AttnRows<DP>& o, float* Dr) {
#pragma unroll
    for (int it = 0; it < AttnRows<DP>::kN; ++it) {
        const float4 a = g.v[it], b = o.v[it];
        float D = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)));
#pragma unroll
        for (int off = 1; off < DP / 4; off <<= 1) D += __shfl_xor_sync(0xffffffffu, D, off);
        if (AttnRows<DP>::chan() == 0) Dr[AttnRows<DP>::row(it)] = D;
    }
}
// LSE of query row i0 + thread (threads of the first 64); rows past L: -inf, which masks them
__device__ __forceinline__ float row_lse(const BwdParams& p, int bh, int i0) {
    const int i = i0 + static_cast<int>(threadIdx.x);
    return (threadIdx.x < kT && i < p.L) ? p.LSE[static_cast<size_t>(bh) * p.L + i] : -CUDART_INF_F;
}

// rows [r0, r0 + 64) of a result from the groups' parts
template <int DP>
__device__ __forceinline__ void store_rows(float* dst, const float* red, int r0, int L, int d, float scale, bool vec) {
    for (int e = threadIdx.x; e < kT * DP / 4; e += kAttnThreads) {
        const int r = e / (DP / 4), c = (e % (DP / 4)) * 4;
        if (r0 + r >= L || c >= d) continue;
        const float4 s = AttnOut<DP>::sum(red, r, c);
        float* o = dst + static_cast<size_t>(r0 + r) * d + c;
        if (vec) *reinterpret_cast<float4*>(o) = make_float4(scale * s.x, scale * s.y, scale * s.z, scale * s.w);
        else {
            o[0] = scale * s.x;
            if (c + 1 < d) o[1] = scale * s.y;
            if (c + 2 < d) o[2] = scale * s.z;
            if (c + 3 < d) o[3] = scale * s.w;
        }
    }
}

// four neighbours of a row of [L] floats from column c on, zero past L
__device__ __forceinline__ float4 row4(const float* row, int c, int L, bool vec) {
    if (vec) return c < L ? attn_ld4(row + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < L) v.x = row[c];
    if (c + 1 < L) v.y = row[c + 1];
    if (c + 2 < L) v.z = row[c + 2];
    if (c + 3 < L) v.w = row[c + 3];
    return v;
}
__device__ __forceinline__ void put4(float* row, int c, int L, bool vec, const float (&v)[4]) {
    if (vec) { if (c < L) *reinterpret_cast<float4*>(row + c) = make_float4(v[0], v[1], v[2], v[3]); return; }
#pragma unroll
    for (int j = 0; j < 4; ++j) if (c + j < L) row[c + j] = v[j];
}

// ---- dQ and dbias -------------------------------------------------------------------------------------------------------
template <int DP> constexpr int dq_smem_floats() { return 5 * DP * kT + kT * kT + 2 * kT; }

template <int DP, bool CAUSAL>
__global__ void __launch_bounds__(kAttnThreads, 2) attn_bwd_dq_kernel(const BwdParams p) {
    extern __shared__ __align__(16) float sm[];
    float* Qt = sm;                                   // own rows, transposed
    float* dOt = Qt + DP * kT;
    float* Kt = dOt + DP * kT;                        // key tile, transposed
    float* Vt = Kt + DP * kT;
    float* Kr = Vt + DP * kT;                         // key tile, row by row
    float* probs = Kr + DP * kT;                      // dS [key][query]
    float* Dr = probs + kT * kT;
    float* Ls = Dr + kT;

    const int bh = blockIdx.y, i0 = blockIdx.x * kT;
    const int b = bh / p.H, hh = bh - b * p.H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int arow = (warp >> 1) * 32 + ((lane & 1) | ((lane >> 4) << 1)) * 4, bcol = (warp & 1) * 32 + ((lane >> 1) & 7) * 4;
    const size_t base = static_cast<size_t>(bh) * p.L * p.d;
    const float* bias = p.bias ? p.bias + static_cast<size_t>(b) * p.bias_batch_stride + static_cast<size_t>(hh) * p.L * p.L : nullptr;
    float* dbias = p.dbias ? p.dbias + static_cast<size_t>(bh) * p.L * p.L : nullptr;

    AttnRows<DP> rk, rv;                              // the next key tile on its way
    {
        AttnRows<DP> q, g, o;
        q.fetch(p.Q + base, p.d, i0, p.L, p.d, p.vec_in);
        g.fetch(p.dO + base, p.d, i0, p.L, p.d, p.vec_in);
        o.fetch(p.O + base, p.d, i0, p.L, p.d, p.vec_in);
        const float lse = row_lse(p, bh, i0);
        rk.fetch(p.K + base, p.d, 0, p.L, p.d, p.vec_in);
        rv.fetch(p.V + base, p.d, 0, p.L, p.d, p.vec_in);
        q.template store<true, false>(Qt, nullptr);
        g.template store<true, false>(dOt, nullptr);
        store_row_dots<DP>(g, o, Dr);
        if (threadIdx.x < kT) Ls[threadIdx.x] = lse;
    }

    const AttnOut<DP> out;
    float o[8][AttnOut<DP>::kCols];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int c = 0; c < AttnOut<DP>::kCols; ++c) o[i][c] = 0.0f;

    const int jend = CAUSAL ? min(p.L, i0 + kT) : p.L;           // keys past the last row's diagonal are masked for all
    for (int j0 = 0; j0 < jend; j0 += kT) {
        __syncthreads();                               // the tiles of the previous step are no longer read
        rk.template store<true, true>(Kt, Kr);
        rv.template store<true, false>(Vt, nullptr);
        const bool diag = CAUSAL && j0 == i0, fin = !diag || rk.finite();
        const int j = j0 + bcol;
        float4 bi[8];                                  // this tile's bias and the next tile's keys travel during the products
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int i = i0 + arow + (r < 4 ? r : 12 + r);
            bi[r] = (bias && i < p.L) ? row4(bias + static_cast<size_t>(i) * p.L, j, p.L, p.vec_bias) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (j0 + kT < jend) {
            rk.fetch(p.K + base, p.d, j0 + kT, p.L, p.d, p.vec_in);
            rv.fetch(p.V + base, p.d, j0 + kT, p.L, p.d, p.vec_in);
        }
        bool masked = false;                           // unseen K rows may not even be multiplied by zero
        if (diag) masked = __syncthreads_or(!fin);
        else __syncthreads();
        float s[8][4], dp[8][4];
        attn_scores<DP, 16>(Qt, Kt, arow, bcol, s);
        attn_scores<DP, 16>(dOt, Vt, arow, bcol, dp);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int rl = arow + (r < 4 ? r : 12 + r), i = i0 + rl;
            const float lse = Ls[rl], Di = Dr[rl];
            const float bj[4] = {bi[r].x, bi[r].y, bi[r].z, bi[r].w};
            const int keys = (lse > -CUDART_INF_F ? (CAUSAL ? min(i + 1, p.L) : p.L) : 0) - j;      // visible ones from column j on
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                s[r][u] = u < keys ? expf(s[r][u] * p.scale + bj[u] - lse) * (dp[r][u] - Di) : 0.0f;
            }
            if (dbias && i < p.L) put4(dbias + static_cast<size_t>(i) * p.L, j, p.L, p.vec_dbias, s[r]);
        }
        if (p.dQ) {
            attn_store_probs<16>(probs, arow, bcol, s);
            __syncthreads();
            if (masked) out.template mac_diag<false>(probs, Kr, o);
            else out.mac(probs, Kr, o);
        }
    }
    // keys past jend of a causal CTA: dbias stays 0 there
    if (dbias && CAUSAL) {
        const int j1 = ((jend + kT - 1) / kT) * kT;    // the walked tiles wrote up to here
        for (int r = warp; r < kT; r += 4)
            if (i0 + r < p.L) for (int j = j1 + lane; j < p.L; j += 32) dbias[static_cast<size_t>(i0 + r) * p.L + j] = 0.0f;
    }
    if (p.dQ) {
        __syncthreads();
        out.spill(probs, o);
        __syncthreads();
        store_rows<DP>(p.dQ + base, probs, i0, p.L, p.d, p.scale, p.vec_out);
    }
}

// ---- dK and dV ----------------------------------------------------------------------------------------------------------
template <int DP> constexpr int dkv_smem_floats() { return 6 * DP * kT + kT * kT + 2 * kT; }

template <int DP, bool CAUSAL>
__global__ void __launch_bounds__(kAttnThreads, 2) attn_bwd_dkv_kernel(const BwdParams p) {
    extern __shared__ __align__(16) float sm[];
    float* Kt = sm;                                   // own rows, transposed
    float* Vt = Kt + DP * kT;
    float* Qt = Vt + DP * kT;                         // query tile, transposed
    float* dOt = Qt + DP * kT;
    float* Qr = dOt + DP * kT;                        // query tile, row by row
    float* dOr = Qr + DP * kT;
    float* probs = dOr + DP * kT;                     // P, then dS [query][key]
    float* Dr = probs + kT * kT;
    float* Ls = Dr + kT;

    const int bh = blockIdx.y, j0 = blockIdx.x * kT;
    const int b = bh / p.H, hh = bh - b * p.H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int arow = (warp >> 1) * 32 + ((lane & 1) | ((lane >> 4) << 1)) * 4, bcol = (warp & 1) * 32 + ((lane >> 1) & 7) * 4;
    const size_t base = static_cast<size_t>(bh) * p.L * p.d;
    const float* bias = p.bias ? p.bias + static_cast<size_t>(b) * p.bias_batch_stride + static_cast<size_t>(hh) * p.L * p.L : nullptr;

    const int ibeg = CAUSAL ? j0 : 0;                  // query rows before the first key of the tile see none of it
    AttnRows<DP> rq, rg, ro;                           // the next query tile on its way: Q, dO, O and the LSE
    float rl;
    auto fetch_queries = [&](int i0) {
        rq.fetch(p.Q + base, p.d, i0, p.L, p.d, p.vec_in);
        rg.fetch(p.dO + base, p.d, i0, p.L, p.d, p.vec_in);
        ro.fetch(p.O + base, p.d, i0, p.L, p.d, p.vec_in);
        rl = row_lse(p, bh, i0);
    };
    {
        AttnRows<DP> k, v;
        k.fetch(p.K + base, p.d, j0, p.L, p.d, p.vec_in);
        v.fetch(p.V + base, p.d, j0, p.L, p.d, p.vec_in);
        fetch_queries(ibeg);
        k.template store<true, false>(Kt, nullptr);
        v.template store<true, false>(Vt, nullptr);
    }

    const AttnOut<DP> out;
    constexpr int NC = AttnOut<DP>::kCols;
    float ok[8][NC], ov[8][NC];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int c = 0; c < NC; ++c) { ok[i][c] = 0.0f; ov[i][c] = 0.0f; }

    for (int i0 = ibeg; i0 < p.L; i0 += kT) {
        __syncthreads();                               // the tiles of the previous step are no longer read
        rq.template store<true, true>(Qt, Qr);
        rg.template store<true, true>(dOt, dOr);
        store_row_dots<DP>(rg, ro, Dr);
        if (threadIdx.x < kT) Ls[threadIdx.x] = rl;
        const bool diag = CAUSAL && i0 == j0, fin = !diag || (rq.finite() && rg.finite());
        float4 bi[4][2];                               // this tile's bias and the next query tile travel during the products
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = i0 + bcol + u;
                bi[u][h] = (bias && i < p.L) ? row4(bias + static_cast<size_t>(i) * p.L, j0 + arow + 16 * h, p.L, p.vec_bias)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        if (i0 + kT < p.L) fetch_queries(i0 + kT);
        bool masked = false;                           // Q and dO rows that do not see a key may not even be multiplied by zero
        if (diag) masked = __syncthreads_or(!fin);
        else __syncthreads();
        float s[8][4], dp[8][4];
        attn_scores<DP, 16>(Kt, Qt, arow, bcol, s);    // [key][query]
        const float4 l4 = attn_ld4(Ls + bcol);
        const float lse[4] = {l4.x, l4.y, l4.z, l4.w};
        int keys[4];                                   // per query: its visible keys from this thread's first key row on
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + bcol + u;
            keys[u] = (lse[u] > -CUDART_INF_F ? (CAUSAL ? min(i + 1, p.L) : p.L) : 0) - (j0 + arow);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float bj[4] = {bi[u][h].x, bi[u][h].y, bi[u][h].z, bi[u][h].w};
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    s[4 * h + r][u] = 16 * h + r < keys[u] ? expf(s[4 * h + r][u] * p.scale + bj[r] - lse[u]) : 0.0f;
            }
        }
        attn_store_probs<16>(probs, arow, bcol, s);
        attn_scores<DP, 16>(Vt, dOt, arow, bcol, dp);
        const float4 d4 = attn_ld4(Dr + bcol);
        const float Di[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int u = 0; u < 4; ++u) s[r][u] = (r < 4 ? r : 12 + r) < keys[u] ? s[r][u] * (dp[r][u] - Di[u]) : 0.0f;
        __syncthreads();
        if (masked) out.template mac_diag<true>(probs, dOr, ov);
        else out.mac(probs, dOr, ov);
        __syncthreads();
        attn_store_probs<16>(probs, arow, bcol, s);
        __syncthreads();
        if (masked) out.template mac_diag<true>(probs, Qr, ok);
        else out.mac(probs, Qr, ok);
    }
    if (p.dK) {
        __syncthreads();
        out.spill(probs, ok);
        __syncthreads();
        store_rows<DP>(p.dK + base, probs, j0, p.L, p.d, p.scale, p.vec_out);
    }
    if (p.dV) {
        __syncthreads();
        out.spill(probs, ov);
        __syncthreads();
        store_rows<DP>(p.dV + base, probs, j0, p.L, p.d, 1.0f, p.vec_out);
    }
}

template <int DP, bool CAUSAL>
int launch_causal(const BwdParams& p, cudaStream_t st) {
    const dim3 grid((p.L + kT - 1) / kT, p.B * p.H);
    constexpr int dq_bytes = dq_smem_floats<DP>() * 4, dkv_bytes = dkv_smem_floats<DP>() * 4;
    static bool configured[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return ST_LAUNCH; }
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(attn_bwd_dq_kernel<DP, CAUSAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, dq_bytes) != cudaSuccess ||
            cudaFuncSetAttribute(attn_bwd_dkv_kernel<DP, CAUSAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, dkv_bytes) != cudaSuccess) {
            cudaGetLastError();
            return ST_LAUNCH;
        }
        configured[dev] = true;
    }
    if (p.dQ || p.dbias) {
        attn_bwd_dq_kernel<DP, CAUSAL><<<grid, kAttnThreads, dq_bytes, st>>>(p);
        if (cudaGetLastError() != cudaSuccess) return ST_LAUNCH;
    }
    if (p.dK || p.dV) {
        attn_bwd_dkv_kernel<DP, CAUSAL><<<grid, kAttnThreads, dkv_bytes, st>>>(p);
        if (cudaGetLastError() != cudaSuccess) return ST_LAUNCH;
    }
    return ST_OK;
}

// causal calls have instances of their own: what their tiles ask for cost the others 3 % (515 against 498 us at 64 x 8 x 256 x 32)
template <int DP>
int launch_dp(const BwdParams& p, cudaStream_t st) { return p.causal ? launch_causal<DP, true>(p, st) : launch_causal<DP, false>(p, st); }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

int launch_attn_backward(int B, int H, int L, int d, int causal, float scale, const float* Q, const float* K, const float* V,
                         const float* bias, long long bias_batch_stride, const float* O, const float* dO, const float* LSE,
                         float* dQ, float* dK, float* dV, float* dbias, cudaStream_t st) {
    if (d > 64 || static_cast<long long>(B) * H > 65535) return ST_UNSUPPORTED_PATH;
    if (L <= kAttnBackwardShortRows)
        return launch_attn_backward_short(B, H, L, d, causal, scale, Q, K, V, bias, bias_batch_stride, O, dO, LSE, dQ, dK, dV, dbias, st);
    BwdParams p;
    p.B = B; p.H = H; p.L = L; p.d = d; p.causal = causal; p.scale = scale;
    p.Q = Q; p.K = K; p.V = V; p.bias = bias; p.O = O; p.dO = dO; p.LSE = LSE; p.bias_batch_stride = bias_batch_stride;
    p.dQ = dQ; p.dK = dK; p.dV = dV; p.dbias = dbias;
    p.vec_in = d % 4 == 0 && aligned16(Q) && aligned16(K) && aligned16(V) && aligned16(O) && aligned16(dO);
    p.vec_out = d % 4 == 0 && aligned16(dQ) && aligned16(dK) && aligned16(dV);
    p.vec_bias = L % 4 == 0 && aligned16(bias) && bias_batch_stride % 4 == 0;
    p.vec_dbias = L % 4 == 0 && aligned16(dbias);
    if (d <= 8) return launch_dp<8>(p, st);
    if (d <= 16) return launch_dp<16>(p, st);
    if (d <= 32) return launch_dp<32>(p, st);
    return launch_dp<64>(p, st);
}

}  // namespace ppml_b200
