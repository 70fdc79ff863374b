// attn_tile.cuh -- building blocks of the exact-fp32 attention kernels (attn_exact.cu, attn_backward.cu): a CTA of four warps owns
// 64 rows of one (batch, head) and walks the partner rows in tiles of 64.  Two kinds of product, both packed fp32 FMAs on
// register tiles (a packed pair takes one issue slot and leaves the others to the shared-memory reads):
//   scores    [own row][partner] = sum over the channels; both operands transposed in shared memory, 8 x 4 outputs per thread
//   results   [own row][channel] += sum over the partners of a [partner][own row] tile (probabilities) times partner rows
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace ppml_b200 {

constexpr int kAttnTile = 64;          // own rows of a CTA = partner rows of a tile
constexpr int kAttnThreads = 128;

// Transposed operand tile [channel][64 rows], probability tile [partner][64 own rows]: the row index is XORed with a multiple of
// four (eight) that follows the other index, so that a warp's transposed stores spread over the banks and four consecutive rows
// stay one 16-byte read.
__device__ __forceinline__ int attn_swz_t(int c) { return ((c >> 2) & 7) << 2; }
__device__ __forceinline__ int attn_swz_p(int j) { return ((j >> 2) & 7) << 3; }

__device__ __forceinline__ float attn_f32(float v) { return v; }
__device__ __forceinline__ float attn_f32(__half v) { return __half2float(v); }
__device__ __forceinline__ float attn_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float4 attn_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <typename T> __device__ __forceinline__ float4 attn_ld4(const T* p) {      // 16-bit types: 8 bytes
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const T* h = reinterpret_cast<const T*>(&u);
    return make_float4(attn_f32(h[0]), attn_f32(h[1]), attn_f32(h[2]), attn_f32(h[3]));
}

// Rows [r0, r0 + 64) of a matrix with d channels and the given row stride, on their way from global memory (fetch) to shared
// memory (store: as a transposed tile `tr` and / or row by row `rm`, [64][DP]); rows past L and channels past d read as zero.
// vec: rows start on 4-element boundaries and d is a multiple of 4.
template <int DP>
struct AttnRows {
    static constexpr int kQ = DP / 4, kN = kAttnTile * kQ / kAttnThreads;
    float4 v[kN];

    static __device__ __forceinline__ int row(int it) { return (it * kAttnThreads + static_cast<int>(threadIdx.x)) / kQ; }
    static __device__ __forceinline__ int chan() { return (static_cast<int>(threadIdx.x) % kQ) * 4; }
    template <typename T>
    __device__ __forceinline__ void fetch(const T* src, long long stride, int r0, int L, int d, bool vec) {
        const int c = chan();
#pragma unroll
        for (int it = 0; it < kN; ++it) {
            const int r = r0 + row(it);
            v[it] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < L && c < d) {
                const T* p = src + r * stride + c;
                if (vec) v[it] = attn_ld4(p);
                else {
                    v[it].x = attn_f32(p[0]);
                    if (c + 1 < d) v[it].y = attn_f32(p[1]);
                    if (c + 2 < d) v[it].z = attn_f32(p[2]);
                    if (c + 3 < d) v[it].w = attn_f32(p[3]);
                }
            }
        }
    }
    // no infinity and no NaN among this thread's values
    __device__ __forceinline__ bool finite() const {
        float t = 0.0f;
#pragma unroll
        for (int it = 0; it < kN; ++it) t = fmaf(v[it].x, 0.0f, fmaf(v[it].y, 0.0f, fmaf(v[it].z, 0.0f, fmaf(v[it].w, 0.0f, t))));
        return t == 0.0f;
    }
    template <bool TR, bool RM>
    __device__ __forceinline__ void store(float* tr, float* rm) const {
        const int c = chan();
#pragma unroll
        for (int it = 0; it < kN; ++it) {
            const int r = row(it);
            if constexpr (TR) {
                float* t = tr + c * kAttnTile + (r ^ attn_swz_t(c));
                t[0] = v[it].x; t[kAttnTile] = v[it].y; t[2 * kAttnTile] = v[it].z; t[3 * kAttnTile] = v[it].w;
            }
            if constexpr (RM) *reinterpret_cast<float4*>(rm + r * DP + c) = v[it];
        }
    }
};

// acc[i][j] = sum_c at[c][own row i] * bt[c][partner j]; own rows arow .. +3 and arow + STEP .. +3, partners bcol .. +3
template <int DP, int STEP>
__device__ __forceinline__ void attn_scores(const float* at, const float* bt, int arow, int bcol, float (&acc)[8][4]) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll 8
    for (int c = 0; c < DP; ++c) {
        const int sw = attn_swz_t(c);
        float a[8], b[4];
        *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(at + c * kAttnTile + (arow ^ sw));
        *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(at + c * kAttnTile + ((arow + STEP) ^ sw));
        *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(bt + c * kAttnTile + (bcol ^ sw));
#pragma unroll
        for (int j = 0; j < 4; ++j) {                    // pairs of rows: only the four column values have to be doubled
            const uint64_t b2 = pack2(b[j], b[j]);
#pragma unroll
            for (int i = 0; i < 8; i += 2)
                unpack2(ffma2(pack2(a[i], a[i + 1]), b2, pack2(acc[i][j], acc[i + 1][j])), acc[i][j], acc[i + 1][j]);
        }
    }
}

// Where a thread's part of the result [64][DP] lies.  Narrow results would leave a thread too few outputs per shared-memory read,
// so the partners of a tile are shared among kGroups groups of warps, each with the whole result; sum() adds them.
template <int DP>
struct AttnOut {
    static constexpr int kCols = DP >= 16 ? 4 : 2;                               // columns per thread (rows: 8)
    static constexpr int kGroupWarps = DP == 64 ? 4 : (DP == 32 ? 2 : 1);
    static constexpr int kGroups = 4 / kGroupWarps;
    static constexpr int kPartners = kAttnTile / kGroups;
    static constexpr int kStep = DP >= 32 ? 16 : 32;                             // distance of the two groups of four rows
    int group, row, col;
    __device__ __forceinline__ AttnOut() {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        group = warp / kGroupWarps;
        if constexpr (DP >= 32) {                                                // a warp: 32 rows x 32 columns
            row = (warp & 1) * 32 + ((lane & 1) | ((lane >> 4) << 1)) * 4;
            col = ((warp % kGroupWarps) >> 1) * 32 + ((lane >> 1) & 7) * 4;
        } else {                                                                 // a warp: 64 rows x DP columns
            row = (lane >> 2) * 4;
            col = (lane & 3) * kCols;
        }
    }
    // o += sum over the group's partners of probs[partner][row] * rm[partner][col]
    __device__ __forceinline__ void mac(const float* probs, const float* rm, float (&o)[8][kCols]) const {
        const float* pj = probs + group * kPartners * kAttnTile;
        const float* vj = rm + group * kPartners * DP + col;
#pragma unroll 2
        for (int j4 = 0; j4 < kPartners / 4; ++j4, pj += 4 * kAttnTile, vj += 4 * DP) {
            const int sw = attn_swz_p(group * kPartners + j4 * 4);
            const float* p0 = pj + (row ^ sw);
            const float* p1 = pj + ((row + kStep) ^ sw);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float a[8], b[kCols];
                *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(p0 + u * kAttnTile);
                *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(p1 + u * kAttnTile);
                if constexpr (kCols == 4) *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(vj + u * DP);
                else *reinterpret_cast<float2*>(b) = *reinterpret_cast<const float2*>(vj + u * DP);
#pragma unroll
                for (int c = 0; c < kCols; ++c) {
                    const uint64_t b2 = pack2(b[c], b[c]);
#pragma unroll
                    for (int i = 0; i < 8; i += 2)
                        unpack2(ffma2(pack2(a[i], a[i + 1]), b2, pack2(o[i][c], o[i + 1][c])), o[i][c], o[i + 1][c]);
                }
            }
        }
    }
    // The same for a tile on the diagonal of a causal attention whose partner rows hold an infinity or a NaN: a partner enters only the
    // rows that see it (partner <= row, or with OWN_IS_KEY partner >= row).  For the others its probability is zero, which is enough
    // for finite values (the kernels ask while they store the tile; this form on every diagonal tile made 51 x 8 x 51 x 32 causal 48 us
    // instead of 40 backward).
    template <bool OWN_IS_KEY>
    __device__ __forceinline__ void mac_diag(const float* probs, const float* rm, float (&o)[8][kCols]) const {
#pragma unroll 1
        for (int j = group * kPartners; j < (group + 1) * kPartners; ++j) {
            const int sw = attn_swz_p(j);
            float a[8];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(probs + j * kAttnTile + (row ^ sw));
            *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(probs + j * kAttnTile + ((row + kStep) ^ sw));
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                const float b = rm[j * DP + col + c];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = row + (i < 4 ? i : kStep - 4 + i);
                    if (OWN_IS_KEY ? j >= r : j <= r) o[i][c] = fmaf(a[i], b, o[i][c]);
                }
            }
        }
    }
    // every group's part into red[group][64][DP] (at most 16 KB); the caller synchronizes and adds with sum()
    __device__ __forceinline__ void spill(float* red, const float (&o)[8][kCols]) const {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float* r = red + (group * kAttnTile + row + (i < 4 ? i : kStep - 4 + i)) * DP + col;
            if constexpr (kCols == 4) *reinterpret_cast<float4*>(r) = make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
            else *reinterpret_cast<float2*>(r) = make_float2(o[i][0], o[i][1]);
        }
    }
    static __device__ __forceinline__ float4 sum(const float* red, int r, int c) {
        float4 s = *reinterpret_cast<const float4*>(red + r * DP + c);
#pragma unroll
        for (int g = 1; g < kGroups; ++g) {
            const float4 x = *reinterpret_cast<const float4*>(red + (g * kAttnTile + r) * DP + c);
            s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
        }
        return s;
    }
};

// probs[partner bcol + j][own row] for a thread's 8 x 4 scores
template <int STEP>
__device__ __forceinline__ void attn_store_probs(float* probs, int arow, int bcol, const float (&s)[8][4]) {
    const int sw = attn_swz_p(bcol);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float* p = probs + (bcol + j) * kAttnTile;
        *reinterpret_cast<float4*>(p + (arow ^ sw)) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
        *reinterpret_cast<float4*>(p + ((arow + STEP) ^ sw)) = make_float4(s[4][j], s[5][j], s[6][j], s[7][j]);
    }
}

}  // namespace ppml_b200
