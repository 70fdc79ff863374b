// attn_exact.cu -- exact-fp32 attention forward for head dims 17 .. 64 (what the drop-in launchers run for head dim 32 by default),
// fp32 or 16-bit Q / K / V, any strides.  One CTA = 64 query rows of one (batch, head); the keys go by in tiles of 64.  Per tile: scores
// as 8 x 4 register tiles (a warp owns 16 rows, so the row maximum stays within 16 lanes), online softmax in registers, the
// probabilities to shared memory as [key][query], then the output's register tile over the keys (attn_tile.cuh).
//
// Arithmetic contract as attn_rowwarp_kernel: denominator l + eps, LSE = m + log(l + eps), a row without a visible key (or, with
// ft > 0, whose first ft scores are all -inf) gives O = 0, LSE = -inf.
//
// Bound: instruction issue, about half of it the FMAs of the two products.  256 x 8 x 256 x 32 with a shared bias 2375 -> 749 us, 51 x 8 x
// 51 x 32 32 -> 16 us back to back in a graph (33 -> 19 as calls) against attn_rowwarp_kernel (16 rows per CTA, one key per lane: a
// scalar shared-memory read and a shuffle for every few FMAs).
#include <cuda_runtime.h>
#include <math_constants.h>

#include "attn_tile.cuh"
#include "kernels.h"

namespace ppml_b200 {

namespace {

struct ExactAttn {
    int H, L, Lk, d, causal, ft;
    float scale, eps;
    long long bias_batch_stride;
    int vec_q, vec_k, vec_v, vec_bias, vec_o, vec_g;     // rows in whole groups of four elements
    AttnLayout lay;
};

template <int DP> constexpr int exact_smem_floats() { return 3 * DP * kAttnTile + kAttnTile * kAttnTile + kAttnTile; }

template <typename T, int DP, bool CAUSAL>
__global__ void __launch_bounds__(kAttnThreads, DP == 32 ? 3 : 2)
attn_exact_kernel(const T* __restrict__ Q, const T* __restrict__ K, const T* __restrict__ V, const float* __restrict__ bias,
                  float* __restrict__ O, float* __restrict__ LSE, const ExactAttn p) {
    extern __shared__ __align__(16) float sm[];
    constexpr int kT = kAttnTile;
    float* Qt = sm;                                   // query rows, transposed
    float* Kt = Qt + DP * kT;                         // key tile, transposed
    float* Vr = Kt + DP * kT;                         // key tile, row by row
    float* probs = Vr + DP * kT;                      // [key][query]
    float* rowf = probs + kT * kT;                    // per row: this tile's rescale factor; at the end 1 / (l + eps)
    const int i0 = blockIdx.x * kT, hh = blockIdx.y, b = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int arow = warp * 16 + (lane & 1) * 4, bcol = (lane >> 1) * 4;      // rows arow .. +3, arow + 8 .. +3
    const AttnLayout& lay = p.lay;
    const T* Kb = K + b * lay.k_b + hh * lay.k_h;
    const T* Vb = V + b * lay.v_b + hh * lay.v_h;
    const float* bh = bias ? bias + static_cast<size_t>(b) * p.bias_batch_stride + static_cast<size_t>(hh) * p.L * static_cast<size_t>(p.Lk) : nullptr;
    const int jend = CAUSAL ? min(min(i0 + kT, p.L), p.Lk) : p.Lk;            // keys needed by any row of this CTA

    AttnRows<DP> rk, rv;                              // the next key tile on its way
    {
        AttnRows<DP> q;
        q.fetch(Q + b * lay.q_b + hh * lay.q_h, lay.q_l, i0, p.L, p.d, p.vec_q);
        rk.fetch(Kb, lay.k_l, 0, p.Lk, p.d, p.vec_k);
        rv.fetch(Vb, lay.v_l, 0, p.Lk, p.d, p.vec_v);
        q.template store<true, false>(Qt, nullptr);
    }
    const AttnOut<DP> out;
    constexpr int NC = AttnOut<DP>::kCols;
    float o[8][NC], m[8], l[8];                       // l: this lane's share of the row sum
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m[i] = -CUDART_INF_F; l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; ++c) o[i][c] = 0.0f;
    }
    uint32_t seen = 0;                                // bit i: row i has a score above -inf among the first ft keys

    for (int j0 = 0; j0 < jend; j0 += kT) {
        __syncthreads();                              // the tiles of the previous step are no longer read
        rk.template store<true, false>(Kt, nullptr);
        rv.template store<false, true>(nullptr, Vr);
        const bool diag = CAUSAL && j0 == i0, fin = !diag || rv.finite();
        if (j0 + kT < jend) {
            rk.fetch(Kb, lay.k_l, j0 + kT, p.Lk, p.d, p.vec_k);
            rv.fetch(Vb, lay.v_l, j0 + kT, p.Lk, p.d, p.vec_v);
        }
        bool masked = false;                          // unseen V rows may not even be multiplied by zero
        if (diag) masked = __syncthreads_or(!fin);
        else __syncthreads();
        float s[8][4];
        attn_scores<DP, 8>(Qt, Kt, arow, bcol, s);
        const int j = j0 + bcol;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int i = i0 + arow + (r < 4 ? r : 4 + r);
            const int keys = (i < p.L ? (CAUSAL ? min(i + 1, p.Lk) : p.Lk) : 0) - j;       // visible ones from column j on
            float bj[4] = {0.f, 0.f, 0.f, 0.f};
            if (bh && keys > 0) {
                const float* br = bh + static_cast<size_t>(i) * p.Lk + j;
                if (p.vec_bias) { const float4 x = attn_ld4(br); bj[0] = x.x; bj[1] = x.y; bj[2] = x.z; bj[3] = x.w; }
                else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) if (u < keys) bj[u] = br[u];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) s[r][u] = u < keys ? (bh ? s[r][u] * p.scale + bj[u] : s[r][u] * p.scale) : -CUDART_INF_F;
            if (j0 < p.ft) {
#pragma unroll
                for (int u = 0; u < 4; ++u) if (j + u < p.ft && s[r][u] > -CUDART_INF_F) seen |= 1u << r;
            }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            float mt = fmaxf(fmaxf(s[r][0], s[r][1]), fmaxf(s[r][2], s[r][3]));
#pragma unroll
            for (int off = 2; off < 32; off <<= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, off));
            const float m_new = fmaxf(m[r], mt);
            const float alpha = (m[r] == -CUDART_INF_F) ? 0.0f : expf(m[r] - m_new);
            float lt = 0.0f;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                s[r][u] = (m_new == -CUDART_INF_F) ? 0.0f : expf(s[r][u] - m_new);
                lt += s[r][u];
            }
            l[r] = alpha * l[r] + lt;
            m[r] = m_new;
            if (lane < 2) rowf[arow + (r < 4 ? r : 4 + r)] = alpha;
        }
        attn_store_probs<8>(probs, arow, bcol, s);
        __syncthreads();
        if (j0 > 0) {
            float a[8];
            *reinterpret_cast<float4*>(a) = attn_ld4(rowf + out.row);
            *reinterpret_cast<float4*>(a + 4) = attn_ld4(rowf + out.row + AttnOut<DP>::kStep);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int c = 0; c < NC; ++c) o[i][c] *= a[i];
        }
        if (masked) out.template mac_diag<false>(probs, Vr, o);
        else out.mac(probs, Vr, o);
    }

    __syncthreads();                                  // probs and rowf are no longer read
    out.spill(probs, o);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        float lr = l[r];
        uint32_t sn = (seen >> r) & 1u;
#pragma unroll
        for (int off = 2; off < 32; off <<= 1) {
            lr += __shfl_xor_sync(0xffffffffu, lr, off);
            sn |= __shfl_xor_sync(0xffffffffu, sn, off);
        }
        if (p.ft > 0 && sn == 0) lr = 0.0f;           // the reference's first key tile is fully masked
        const int rl = arow + (r < 4 ? r : 4 + r), i = i0 + rl;
        if (lane < 2) {
            rowf[rl] = lr > 0.0f ? 1.0f / (lr + p.eps) : -1.0f;
            if (LSE && i < p.L) LSE[(static_cast<size_t>(b) * p.H + hh) * p.L + i] = lr > 0.0f ? m[r] + logf(lr + p.eps) : -CUDART_INF_F;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kT * DP / 4; e += kAttnThreads) {
        const int r = e / (DP / 4), c = (e % (DP / 4)) * 4, i = i0 + r;
        if (i >= p.L || c >= p.d) continue;
        const float4 a = AttnOut<DP>::sum(probs, r, c);
        const float inv = rowf[r];
        float v[4] = {a.x * inv, a.y * inv, a.z * inv, a.w * inv};
        if (inv < 0.0f) { v[0] = 0.0f; v[1] = 0.0f; v[2] = 0.0f; v[3] = 0.0f; }
        if (lay.gate && inv >= 0.0f) {
            const float* g = lay.gate + b * lay.g_b + hh * lay.g_h + static_cast<long long>(i) * lay.g_l + c;
            float gv[4];
            if (p.vec_g) *reinterpret_cast<float4*>(gv) = attn_ld4(g);
            else {
#pragma unroll
                for (int u = 0; u < 4; ++u) gv[u] = c + u < p.d ? g[u] : 0.0f;
            }
#pragma unroll 1
            for (int u = 0; u < 4; ++u) {             // one copy of the activations' code
                const float x = act_scalar(lay.act, gv[0]) * v[0];
                gv[0] = gv[1]; gv[1] = gv[2]; gv[2] = gv[3];
                v[0] = v[1]; v[1] = v[2]; v[2] = v[3]; v[3] = x;
            }
        }
        float* dst = O + b * lay.o_b + hh * lay.o_h + static_cast<long long>(i) * lay.o_l + c;
        if (p.vec_o) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        else {
#pragma unroll
            for (int u = 0; u < 4; ++u) if (c + u < p.d) dst[u] = v[u];
        }
    }
}

template <typename T, int DP, bool CAUSAL>
int launch_causal(const T* Q, const T* K, const T* V, const float* bias, float* O, float* LSE, int B, const ExactAttn& p, cudaStream_t st) {
    constexpr int bytes = exact_smem_floats<DP>() * 4;
    static bool configured[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return ST_LAUNCH; }
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(attn_exact_kernel<T, DP, CAUSAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
            cudaGetLastError();
            return ST_LAUNCH;
        }
        configured[dev] = true;
    }
    attn_exact_kernel<T, DP, CAUSAL><<<dim3((p.L + kAttnTile - 1) / kAttnTile, p.H, B), kAttnThreads, bytes, st>>>(Q, K, V, bias, O, LSE, p);
    return cudaGetLastError() == cudaSuccess ? ST_OK : ST_LAUNCH;
}

template <typename T, int DP>
int launch_typed(const T* Q, const T* K, const T* V, const float* bias, float* O, float* LSE, int B, const ExactAttn& p, cudaStream_t st) {
    return p.causal ? launch_causal<T, DP, true>(Q, K, V, bias, O, LSE, B, p, st) : launch_causal<T, DP, false>(Q, K, V, bias, O, LSE, B, p, st);
}

// rows that start on 4-element boundaries: base and every stride
bool rows_of_four(const void* base, size_t elem, int d, long long s_b, long long s_h, long long s_l) {
    return d % 4 == 0 && reinterpret_cast<uintptr_t>(base) % (4 * elem) == 0 && s_b % 4 == 0 && s_h % 4 == 0 && s_l % 4 == 0;
}

}  // namespace

int launch_attn_exact(const void* Q, const void* K, const void* V, int elem, const float* bias, float* O, float* LSE, int B, int H, int L,
                      int Lk, int d, int causal, float scale, float eps, long long bias_batch_stride, int ft, const AttnLayout& lay,
                      cudaStream_t st) {
    if (d <= 16 || d > 64) return ST_UNSUPPORTED_PATH;
    // scores computed with tiles of 64 x 64 against attn_rowwarp_kernel's 16 x 32: a short or just-too-long sequence leaves most of
    // the large tiles empty (10 x 8 x 70 x 32, 3.3 against 1.6 times the scores asked for: 22 us here, 19.5 there; 4 x 4 x 40,
    // 2.6 against 1.9: 12.3 here, 13.8 there)
    const long long here = static_cast<long long>((L + 63) / 64 * 64LL) * ((Lk + 63) / 64 * 64LL);
    const long long there = static_cast<long long>((L + 15) / 16 * 16LL) * ((Lk + 31) / 32 * 32LL);
    if (here > 2 * there) return ST_UNSUPPORTED_PATH;
    // at a ratio of 2 itself the head dims with an unrolled instance there (32, 64) still lose in two places:
    // one tile of 32 keys, as long as that kernel runs in one wave of 6 CTAs per SM (64 (batch, head)s of 128 rows and 32 keys, head dim
    // 32: 1.19 times its time here; 148 of them, two waves there, 0.67);
    // head dim 64, with two CTAs per SM here, when the second wave is less than half full (32 rows, 408 (batch, head)s: 1.17 times with
    // 64 keys, 1.09 with 256; 296 and 450 of them 0.66 to 0.78; 512 keys 0.76, K and V no longer staying in L2 there)
    if ((d == 32 || d == 64) && here == 2 * there) {
        const long long bh = static_cast<long long>(B) * H, sms = num_sms();
        const long long ctas = (L + 63) / 64 * bh, ctas_there = (L + 15) / 16 * bh;
        if (Lk <= 32 && ctas_there <= 6 * sms) return ST_UNSUPPORTED_PATH;
        if (d == 64 && Lk <= 256 && ctas > 2 * sms && ctas < 3 * sms) return ST_UNSUPPORTED_PATH;
    }
    ExactAttn p;
    p.H = H; p.L = L; p.Lk = Lk; p.d = d; p.causal = causal; p.ft = ft; p.scale = scale; p.eps = eps;
    p.bias_batch_stride = bias_batch_stride; p.lay = lay;
    const size_t es = elem == 0 ? 4 : 2;
    p.vec_q = rows_of_four(Q, es, d, lay.q_b, lay.q_h, lay.q_l);
    p.vec_k = rows_of_four(K, es, d, lay.k_b, lay.k_h, lay.k_l);
    p.vec_v = rows_of_four(V, es, d, lay.v_b, lay.v_h, lay.v_l);
    p.vec_o = rows_of_four(O, 4, d, lay.o_b, lay.o_h, lay.o_l);
    p.vec_g = lay.gate != nullptr && rows_of_four(lay.gate, 4, d, lay.g_b, lay.g_h, lay.g_l);
    p.vec_bias = rows_of_four(bias, 4, Lk, bias_batch_stride, 0, 0);
    auto go = [&](auto tag) {
        using T = decltype(tag);
        const T* q = static_cast<const T*>(Q);
        const T* k = static_cast<const T*>(K);
        const T* v = static_cast<const T*>(V);
        return d <= 32 ? launch_typed<T, 32>(q, k, v, bias, O, LSE, B, p, st) : launch_typed<T, 64>(q, k, v, bias, O, LSE, B, p, st);
    };
    if (elem == 0) return go(float{});
    return elem == 1 ? go(__nv_bfloat16{}) : go(__half{});
}

}  // namespace ppml_b200
