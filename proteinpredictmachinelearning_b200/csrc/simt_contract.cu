// simt_contract.cu -- exact-fp32 contraction on CUDA cores: every product the tensor-core paths do not take (unaligned K, inner
// batch > 1, tiny extents, broadcast planes) and every product the caller wants in plain fp32.
//
//   D[p][m][n] = epi( sum_k A[pa][m][k] * B[pb][n][k] )
//
// Each output element is one chain of fused multiply-adds with k ascending, the reference's order, so fp32 results agree with
// its CPU kernels to rounding and do not depend on which of the kernels below, or how many planes, a call runs.  Only out_prod may be
// asked for without that order, and then sums long contractions in parts (in_parts, below).
#include "kernels.h"

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace ppml_b200 {

namespace {

constexpr int kSlice = 16;             // contraction depth of one shared-memory stage

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <typename T> __device__ __forceinline__ float4 load4(const T* p) {         // 16-bit types: 8 bytes
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const T* h = reinterpret_cast<const T*>(&u);
    return make_float4(to_f32<T>(h[0]), to_f32<T>(h[1]), to_f32<T>(h[2]), to_f32<T>(h[3]));
}

// How four neighbouring elements of an operand are fetched: one vector load along k or along the row index (every such
// group aligned and entirely inside or outside the operand), or element by element with any strides.
enum class Fetch { VEC_K, VEC_ROW, ANY };

// Stage layout: [kSlice][ROWS] floats, the row index XORed with a multiple of four that depends on k, so that four consecutive
// rows stay together (they are read back with one 16-byte load) while a warp's stores spread over the banks.  A warp stores
// 8 rows x 4 groups of four k (VEC_K: no conflicts), 128 rows of one k (VEC_ROW: none), or 2 rows x 16 k (ANY: two-way).
template <Fetch F> __device__ __forceinline__ int stage_swizzle(int k) { return F == Fetch::ANY ? (k & 7) << 2 : ((k >> 2) & 3) << 3; }

// One operand's share of a stage, in registers between the global load and the shared store.  Every thread owns the same
// elements in every slice, so it keeps its pointers and steps them.  `slices`: distance to the thread's next slice.
template <typename T, Fetch F, int ROWS, int NT>
struct Loader {
    static constexpr int kGroups = ROWS * kSlice / 4 / NT;       // groups of four elements per thread
    static constexpr bool kAlongK = F == Fetch::VEC_K;
    float4 v[kGroups];
    const T* ptr[kGroups];
    long long step;
    int rows_left;                                               // rows of the operand from the tile's first row on

    static __device__ __forceinline__ int group_row(int tid, int g) {
        const int idx = tid + g * NT;
        return kAlongK ? idx / (kSlice / 4) : (idx % (ROWS / 4)) * 4;
    }
    static __device__ __forceinline__ int group_k(int tid, int g) {
        const int idx = tid + g * NT;
        return kAlongK ? (idx % (kSlice / 4)) * 4 : idx / (ROWS / 4);
    }
    __device__ __forceinline__ void init(const T* src, int tid, long long row0, long long rows, long long k0, long long s_row, long long s_k,
                                         long long slices = 1) {
        rows_left = static_cast<int>(min(rows - row0, static_cast<long long>(ROWS)));
        step = s_k * kSlice * slices;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) ptr[g] = src + (row0 + group_row(tid, g)) * s_row + (k0 + group_k(tid, g)) * s_k;
    }
    __device__ __forceinline__ void fetch(int tid, int k_left) { // the slice at the pointers, k_left of it inside the operand
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            v[g] = (group_row(tid, g) < rows_left && group_k(tid, g) < k_left) ? load4(ptr[g]) : make_float4(0.f, 0.f, 0.f, 0.f);
            ptr[g] += step;
        }
    }
    __device__ __forceinline__ void skip(long long elems) {
#pragma unroll
        for (int g = 0; g < kGroups; ++g) ptr[g] += elems;
    }
    __device__ __forceinline__ void store(int tid, float* stage) const {
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            const int r = group_row(tid, g), k = group_k(tid, g);
            float* c = stage + k * ROWS + (r ^ stage_swizzle<F>(k));
            if constexpr (kAlongK) { c[0] = v[g].x; c[ROWS] = v[g].y; c[2 * ROWS] = v[g].z; c[3 * ROWS] = v[g].w; }
            else *reinterpret_cast<float4*>(c) = v[g];
        }
    }
};

// Any strides: neighbouring threads take neighbouring elements along the shorter one, so that a warp's load covers as few lines
// as the operand allows (65536 tokens x 33 -> 256: 72 us with groups of four per thread here too, 65 us this way; bf16 operands 87 and 72).
template <typename T, int ROWS, int NT>
struct Loader<T, Fetch::ANY, ROWS, NT> {
    static constexpr int kElems = ROWS * kSlice / NT;
    static_assert(NT % kSlice == 0 && NT % ROWS == 0 && kElems * NT == ROWS * kSlice, "whole rows or whole k per round");
    float v[kElems];
    const T* ptr;
    long long step, delta;                                       // to the next slice; between this thread's elements of a slice
    int rows_left, r0, k0, dr, dk;

    __device__ __forceinline__ void init(const T* src, int tid, long long row0, long long rows, long long kb, long long s_row, long long s_k,
                                         long long slices = 1) {
        rows_left = static_cast<int>(min(rows - row0, static_cast<long long>(ROWS)));
        step = s_k * kSlice * slices;
        if (s_k <= s_row) { r0 = tid / kSlice; k0 = tid % kSlice; dr = NT / kSlice; dk = 0; delta = dr * s_row; }
        else { r0 = tid % ROWS; k0 = tid / ROWS; dr = 0; dk = NT / ROWS; delta = dk * s_k; }
        ptr = src + (row0 + r0) * s_row + (kb + k0) * s_k;
    }
    __device__ __forceinline__ void fetch(int, int k_left) {
#pragma unroll
        for (int i = 0; i < kElems; ++i) v[i] = (r0 + i * dr < rows_left && k0 + i * dk < k_left) ? to_f32<T>(ptr[i * delta]) : 0.0f;
        ptr += step;
    }
    __device__ __forceinline__ void skip(long long elems) { ptr += elems; }
    __device__ __forceinline__ void store(int, float* stage) const {
#pragma unroll
        for (int i = 0; i < kElems; ++i) {
            const int r = r0 + i * dr, k = k0 + i * dk;
            stage[k * ROWS + (r ^ stage_swizzle<Fetch::ANY>(k))] = v[i];
        }
    }
};

// One slice of a warp's 32 x 8 TN outputs: lane rows {arow .. +3, arow + 16 ..}, lane columns {bcol .. +3 (, bcol + 32 ..)}.  Per k
// two 16-byte reads of A (four distinct addresses in the warp) and TN / 4 of B (eight) feed 8 TN FMAs.  The FMAs are packed pairs
// of rows: a pair takes the FMA pipe as long as two scalar ones but one issue slot, which leaves slots for the reads
// (4096 x 4096 x 4096: 41 TFLOP/s with scalar FMAs, 52 packed; the same rounding either way).
template <Fetch F, int BM, int BN, int TN>
__device__ __forceinline__ void mac_slice(const float* as, const float* bs, int arow, int bcol, float (&acc)[8][TN]) {
#pragma unroll
    for (int kk = 0; kk < kSlice; ++kk) {
        const int sw = stage_swizzle<F>(kk);
        float a[8], b[TN];
        *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(as + kk * BM + (arow ^ sw));
        *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(as + kk * BM + ((arow + 16) ^ sw));
        *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(bs + kk * BN + (bcol ^ sw));
        if constexpr (TN == 8) *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(bs + kk * BN + ((bcol + 32) ^ sw));
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const uint64_t b2 = pack2(b[j], b[j]);
#pragma unroll
            for (int i = 0; i < 8; i += 2)
                unpack2(ffma2(pack2(a[i], a[i + 1]), b2, pack2(acc[i][j], acc[i + 1][j])), acc[i][j], acc[i + 1][j]);
        }
    }
}
// A warp's lanes in a 4 x 8 grid.  Neighbouring lanes share a column group: 1 to 3 % over rows of eight lanes.
__device__ __forceinline__ int lane_m(int lane) { return (lane & 1) | ((lane >> 4) << 1); }
__device__ __forceinline__ int lane_n(int lane) { return (lane >> 1) & 7; }
__device__ __forceinline__ int clip_slice(long long k_left) { return static_cast<int>(min(k_left, static_cast<long long>(kSlice))); }

template <typename T> struct PlanePtrs { const T* a; const T* b; float* c; };
template <typename T>
__device__ __forceinline__ PlanePtrs<T> plane_ptrs(const T* A, const T* B, float* C, const SimtContract& p, long long plane) {
    const long long i3 = plane / p.ne2, i2 = plane - i3 * p.ne2;
    return {A + (i2 / p.a_div2) * p.a_s2 + (i3 / p.a_div3) * p.a_s3, B + (i2 / p.b_div2) * p.b_s2 + (i3 / p.b_div3) * p.b_s3,
            C + i2 * p.c_s2 + i3 * p.c_s3};
}

// A CTA computes a (32 WM) x (8 TN WN) tile.  The next slice travels global -> registers while the current one is multiplied, then
// registers -> the other stage: one barrier per slice.
//
// Bound: fp32 FMA issue (74 TFLOP/s at 1965 MHz).  64 x 128 tiles with three CTAs per SM (168 registers) beat 128 x 128 with
// two (128 registers, spills): 190 against 204 us at 65536 x 256 x 256, 2.65 against 2.89 ms at 4096 x 4096 x 4096 (187 us, 46
// TFLOP/s, and 2.56 ms, 54, as it stands; 462 us with 64 x 64 tiles, 4 x 4 outputs per thread and unpipelined loads before).
template <typename T, Fetch F, int WM, int WN, int TN, bool FUSED>
__global__ void __launch_bounds__(WM * WN * 32, TN == 8 || F == Fetch::ANY ? 3 : 4)
simt_contract_kernel(const T* __restrict__ A, const T* __restrict__ B, float* __restrict__ C, const SimtContract p, int n_tiles) {
    constexpr int NT = WM * WN * 32, BM = WM * 32, BN = WN * 8 * TN;
    __shared__ __align__(16) float smem[2 * kSlice * (BM + BN)];
    float* const As = smem;                              // [2][kSlice][BM]
    float* const Bs = smem + 2 * kSlice * BM;            // [2][kSlice][BN]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int arow = (warp / WN) * 32 + lane_m(lane) * 4;
    const int bcol = (warp % WN) * (8 * TN) + lane_n(lane) * 4;
    const long long mt = blockIdx.x / n_tiles;
    const long long m0 = mt * BM, n0 = (static_cast<long long>(blockIdx.x) - mt * n_tiles) * BN;

    for (long long plane = blockIdx.z; plane < p.planes; plane += gridDim.z) {
        const PlanePtrs<T> pp = plane_ptrs(A, B, C, p, plane);
        float* Cp = pp.c;

        float acc[8][TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const long long n = n0 + bcol + (j < 4 ? j : 28 + j);
            const float seed = (p.bias_seed && p.bias != nullptr && n < p.N) ? p.bias[n] : 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i][j] = seed;
        }

        Loader<T, F, BM, NT> la;
        Loader<T, F, BN, NT> lb;
        la.init(pp.a, threadIdx.x, m0, p.M, 0, p.a_sm, p.a_sk);
        lb.init(pp.b, threadIdx.x, n0, p.N, 0, p.b_sn, p.b_sk);
        long long k_left = p.K;
        la.fetch(threadIdx.x, clip_slice(k_left));
        lb.fetch(threadIdx.x, clip_slice(k_left));
        la.store(threadIdx.x, As);
        lb.store(threadIdx.x, Bs);
        __syncthreads();
        int buf = 0;
        for (; k_left > 0; k_left -= kSlice, buf ^= 1) {
            const bool more = k_left > kSlice;
            if (more) {
                la.fetch(threadIdx.x, clip_slice(k_left - kSlice));
                lb.fetch(threadIdx.x, clip_slice(k_left - kSlice));
            }
            mac_slice<F, BM, BN, TN>(As + buf * (kSlice * BM), Bs + buf * (kSlice * BN), arow, bcol, acc);
            if (more) {
                la.store(threadIdx.x, As + (buf ^ 1) * (kSlice * BM));
                lb.store(threadIdx.x, Bs + (buf ^ 1) * (kSlice * BN));
            }
            __syncthreads();
        }

        // element (m, n) goes to row_off(m) + col_off(n), for the blocked outer-product-mean store too (extents below 2^32 there:
        // a 64-bit division per element was most of the time of a short contraction)
        auto row_off = [&](long long m) -> long long {
            if (p.opm_L > 0) {
                const uint32_t L = static_cast<uint32_t>(p.opm_L), d1 = static_cast<uint32_t>(m) / L, ii = static_cast<uint32_t>(m) - d1 * L;
                return (d1 * p.opm_D * p.opm_L + ii) * p.opm_L * p.opm_B;
            }
            return m * p.c_sm;
        };
        auto col_off = [&](long long n) -> long long {
            if (p.opm_L > 0) {
                const uint32_t L = static_cast<uint32_t>(p.opm_L), d2 = static_cast<uint32_t>(n) / L, jj = static_cast<uint32_t>(n) - d2 * L;
                return (d2 * p.opm_L * p.opm_L + jj) * p.opm_B;
            }
            return n * p.c_sn;
        };
        // what the fused neighbours read is requested before the first store (the compiler may not move a load across one): row by row,
        // a tile waited for memory eight times (with LayerNorm and gate 2601 x 33 x 100 16.3 -> 11.9 us, 408 x 128 x 128 19.4 -> 13.5,
        // 65536 x 128 x 128 134 -> 123)
        [[maybe_unused]] float mean[8], rstd[8];
        if constexpr (FUSED) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const long long m = m0 + arow + (i < 4 ? i : 12 + i);
                const bool in = p.ln_stats != nullptr && m < p.M;
                mean[i] = in ? p.ln_stats[2 * m] : 0.0f;
                rstd[i] = in ? p.ln_stats[2 * m + 1] : 1.0f;
            }
        }
#pragma unroll
        for (int jg = 0; jg < TN / 4; ++jg) {
            const long long n = n0 + bcol + 32 * jg;
            if (n >= p.N) continue;
            float bias[4] = {0.f, 0.f, 0.f, 0.f};
            if (!p.bias_seed && p.bias != nullptr) {
#pragma unroll
                for (int j = 0; j < 4; ++j) if (n + j < p.N) bias[j] = p.bias[n + j];
            }
            [[maybe_unused]] float lu[4] = {0.f, 0.f, 0.f, 0.f}, gate[8][4];
            if constexpr (FUSED) {
                if (p.ln_stats != nullptr) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) if (n + j < p.N) lu[j] = p.ln_u[n + j];
                }
                if (p.gate != nullptr) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long long m = m0 + arow + (i < 4 ? i : 12 + i);
                        const float* g = p.gate + m * p.c_sm + n * p.c_sn;       // row-major here
                        // 16-byte rows of C mean 16-byte rows of the gate: the entry point refuses the others
                        if (p.vec_c) *reinterpret_cast<float4*>(gate[i]) = m < p.M ? load4(g) : make_float4(0.f, 0.f, 0.f, 0.f);
                        else {
#pragma unroll
                            for (int j = 0; j < 4; ++j) gate[i][j] = (m < p.M && n + j < p.N) ? g[j * p.c_sn] : 0.0f;
                        }
                    }
                }
            }
            long long co[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) co[j] = col_off(n + j);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const long long m = m0 + arow + (i < 4 ? i : 12 + i);
                if (m >= p.M) continue;
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] = acc[i][4 * jg + j] * p.alpha;
                    if constexpr (FUSED) { if (p.ln_stats != nullptr) v[j] = fmaf(-mean[i], lu[j], v[j]) * rstd[i]; }
                    if (!p.bias_seed && p.bias != nullptr) v[j] += bias[j];
                    if (p.clamp) v[j] = (v[j] == v[j]) ? fminf(fmaxf(v[j], -1e4f), 1e4f) : 0.0f;
                }
                if constexpr (FUSED) {
                    if (p.act == 1 || p.act == 2) {                              // the gates of the model: four at a time
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[j] = p.act == 1 ? act_scalar(1, v[j]) : act_scalar(2, v[j]);
                    } else if (p.act != 0) {
#pragma unroll 1
                        for (int j = 0; j < 4; ++j) {                            // one copy of the others' code
                            const float x = act_scalar(p.act, v[0]);
                            v[0] = v[1]; v[1] = v[2]; v[2] = v[3]; v[3] = x;
                        }
                    }
                    if (p.gate != nullptr) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[j] *= gate[i][j];
                    }
                }
                const long long r0 = row_off(m);
                if (p.vec_c) {
                    *reinterpret_cast<float4*>(Cp + r0 + co[0]) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) if (n + j < p.N) Cp[r0 + co[j]] = v[j];
                }
            }
        }
    }
}

// The narrow form, for plain fp32 products with the row index contiguous in both operands, a long contraction and a small result
// (weight gradients: K = the tokens).  64 x 64 tiles would occupy a handful of SMs, and the contraction itself is not split: every
// output stays one ascending chain.  So the tiles are 32 x 16, two warps with 4 x 2 outputs per thread, and three slices are on
// their way through cp.async.
//
// Bound: with a CTA per SM the issue of its two warps and the restart after each slice's barrier (16 cycles per k: 10 instructions, of which 8
// FMAs); with several, shared-memory reads (24 bytes per thread and k: 12 cycles per k and CTA, broadcast or not).  128 x 256 over
// 2601 tokens 135 -> 24 us, 256 x 256 over 65536 4793 -> 553, 64 x 64 over 65536 3214 -> 526 (64 x 64 tiles of 256 threads before).
// 2 x 2 outputs per thread on four warps with slices of 32: 28 us and 640; one warp with a 16 x 16 tile: 26 and 613.
// The contraction in parts (below) takes 16 and 273 us for the first two.
constexpr int kNarrowSlice = 64, kNarrowDepth = 4, kNarrowM = 32, kNarrowN = 16, kNarrowThreads = 64;

__device__ __forceinline__ void cp_async(uint32_t dst, const float* src, bool in, std::integral_constant<int, 16>) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async(uint32_t dst, const float* src, bool in, std::integral_constant<int, 4>) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}

// A thread's copies of one operand [k][row] into the stages [kNarrowSlice][ROWS], VEC elements each, slice after slice; zeros outside
// the operand.
template <int ROWS, int VEC>
struct NarrowCopy {
    static constexpr int kPerRow = ROWS / VEC, kRound = kNarrowThreads / kPerRow;        // copies per k; k per round of the CTA
    static_assert(kNarrowThreads % kPerRow == 0 && kNarrowSlice % kRound == 0, "whole k per round");
    const float* ptr;
    const float* base;
    long long delta;
    int k, dst;
    bool in;
    __device__ __forceinline__ void init(const float* src, long long s_k, int rows_left) {
        const int r = (static_cast<int>(threadIdx.x) % kPerRow) * VEC;
        k = static_cast<int>(threadIdx.x) / kPerRow;
        in = r < rows_left;
        base = src;
        ptr = in ? src + k * s_k + r : src;
        delta = kRound * s_k;
        dst = k * ROWS + r;
    }
    __device__ __forceinline__ void fetch(float* stage, int k_left) {
        const uint32_t d = smem_u32(stage + dst);
#pragma unroll
        for (int i = 0; i < kNarrowSlice / kRound; ++i) {
            const bool ok = in && k + i * kRound < k_left;
            cp_async(d + i * kRound * ROWS * 4, ok ? ptr + i * delta : base, ok, std::integral_constant<int, 4 * VEC>());
        }
        ptr += in ? (kNarrowSlice / kRound) * delta : 0;
    }
};

template <int VEC>
__global__ void __launch_bounds__(kNarrowThreads, 4)
simt_contract_narrow_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, const SimtContract p, int n_tiles) {
    constexpr int BM = kNarrowM, BN = kNarrowN, kStage = kNarrowSlice * (BM + BN), kDepth = kNarrowDepth;
    __shared__ __align__(16) float stages[kDepth * kStage];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int arow = warp * 16 + (lane & 3) * 4, bcol = (lane >> 2) * 2;
    const int mt = blockIdx.x / n_tiles;
    const long long m0 = static_cast<long long>(mt) * BM, n0 = static_cast<long long>(blockIdx.x - mt * n_tiles) * BN;
    const int a_left = static_cast<int>(min(p.M - m0, static_cast<long long>(BM))), b_left = static_cast<int>(min(p.N - n0, static_cast<long long>(BN)));
    const int slices = static_cast<int>((p.K + kNarrowSlice - 1) / kNarrowSlice);

    for (long long plane = blockIdx.z; plane < p.planes; plane += gridDim.z) {
        const PlanePtrs<float> pp = plane_ptrs(A, B, C, p, plane);
        NarrowCopy<BM, VEC> ca;
        NarrowCopy<BN, VEC> cb;
        ca.init(pp.a + m0, p.a_sk, a_left);
        cb.init(pp.b + n0, p.b_sk, b_left);
        auto fetch = [&](int s) {
            if (s < slices) {
                float* st = stages + (s % kDepth) * kStage;
                const int k_left = static_cast<int>(min(p.K - static_cast<long long>(s) * kNarrowSlice, static_cast<long long>(kNarrowSlice)));
                ca.fetch(st, k_left);
                cb.fetch(st + kNarrowSlice * BM, k_left);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float acc[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) { acc[i][0] = 0.0f; acc[i][1] = 0.0f; }
        __syncthreads();                                 // the stages of the previous plane are no longer read
        for (int s = 0; s < kDepth - 1; ++s) fetch(s);
        for (int s = 0; s < slices; ++s) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 2) : "memory");
            __syncthreads();                             // slice s has arrived for everyone, slice s - 1 is no longer read
            fetch(s + kDepth - 1);
            const float* as = stages + (s % kDepth) * kStage + arow;
            const float* bs = stages + (s % kDepth) * kStage + kNarrowSlice * BM + bcol;
#pragma unroll
            for (int kk = 0; kk < kNarrowSlice; ++kk) {
                float a[4];
                *reinterpret_cast<float4*>(a) = load4(as + kk * BM);
                const float2 b = *reinterpret_cast<const float2*>(bs + kk * BN);
#pragma unroll
                for (int i = 0; i < 4; ++i) { acc[i][0] = fmaf(a[i], b.x, acc[i][0]); acc[i][1] = fmaf(a[i], b.y, acc[i][1]); }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (arow + i < a_left && bcol + j < b_left) pp.c[(m0 + arow + i) * p.c_sm + n0 + bcol + j] = acc[i][j] * p.alpha;
    }
}

// A contraction in parts, for out_prod with a long contraction and a small result where the caller does not ask for one chain: part w of W
// takes the slices of k w, w + W, ..., ascending, and the result is ((part 0 + part 1) + ...) in fp32.  W follows from M, N and K
// alone, so the bits do not depend on how many planes a call holds.  The shorter chains come closer to the 64-bit result than one
// (128 x 256 over 2601 tokens: 1.9e-7 against 9.1e-7).  Where the parts run:
//
// simt_contract_split_kernel: a CTA is two or four groups of four warps, a cluster up to 16 CTAs, a group takes one part of a 64 x 64 tile,
// with stages and a barrier of its own.  The partial tiles are left in shared memory and added piece by piece over the cluster (no
// atomics).
// Bound: FMA issue with 16 or more tiles; latency of a group's loads below that (one slice in flight per group), which is why
// the parts are many and short.  256 x 256 over 65536 tokens 4793 -> 273 us (one CTA per 64 x 64 tile before), 64 x 256 over
// 30000 1490 -> 63 us, 33 x 32 over 30000 1470 -> 73 us.
template <Fetch F, int kSplitGroups>
__global__ void __launch_bounds__(kSplitGroups * 128, 4 / kSplitGroups)
simt_contract_split_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, const SimtContract p, int n_tiles) {
    constexpr int BM = 64, BN = 64;
    static_assert(BM * BN == 2 * kSlice * (BM + BN), "a partial tile fills its group's stages");
    extern __shared__ __align__(16) float dyn[];
    cg::cluster_group cl = cg::this_cluster();
    const int splits = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
    const int grp = threadIdx.x >> 7, gtid = threadIdx.x & 127;
    float* const As = dyn + grp * (BM * BN);
    float* const Bs = As + 2 * kSlice * BM;
    const int warp = gtid >> 5, lane = gtid & 31;
    const int arow = (warp >> 1) * 32 + lane_m(lane) * 4, bcol = (warp & 1) * 32 + lane_n(lane) * 4;
    const int mt = blockIdx.x / n_tiles;
    const long long m0 = static_cast<long long>(mt) * BM, n0 = static_cast<long long>(blockIdx.x - mt * n_tiles) * BN;
    const PlanePtrs<float> pp = plane_ptrs(A, B, C, p, blockIdx.z / splits);

    const long long ways = static_cast<long long>(splits) * kSplitGroups;
    const long long kbeg = (rank * kSplitGroups + grp) * static_cast<long long>(kSlice), kstep = ways * kSlice;
    long long k_left = p.K - kbeg;                       // not positive: a group without a share
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory"); };
    Loader<float, F, BM, 128> la;
    Loader<float, F, BN, 128> lb;
    la.init(pp.a, gtid, m0, p.M, kbeg, p.a_sm, p.a_sk, ways);
    lb.init(pp.b, gtid, n0, p.N, kbeg, p.b_sn, p.b_sk, ways);
    la.fetch(gtid, clip_slice(k_left));
    lb.fetch(gtid, clip_slice(k_left));
    la.store(gtid, As);
    lb.store(gtid, Bs);
    group_sync();
    int buf = 0;
    for (; k_left > 0; k_left -= kstep, buf ^= 1) {
        const bool more = k_left > kstep;
        if (more) {
            la.fetch(gtid, clip_slice(k_left - kstep));
            lb.fetch(gtid, clip_slice(k_left - kstep));
        }
        mac_slice<F, BM, BN, 4>(As + buf * (kSlice * BM), Bs + buf * (kSlice * BN), arow, bcol, acc);
        if (more) {
            la.store(gtid, As + (buf ^ 1) * (kSlice * BM));
            lb.store(gtid, Bs + (buf ^ 1) * (kSlice * BN));
        }
        group_sync();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(As + (arow + (i < 4 ? i : 12 + i)) * BN + bcol) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    cl.sync();
    for (int e = rank * (kSplitGroups * 128) + static_cast<int>(threadIdx.x); e < BM * BN / 4; e += splits * (kSplitGroups * 128)) {
        const int r = e / (BN / 4), c = (e % (BN / 4)) * 4;
        if (m0 + r >= p.M || n0 + c >= p.N) continue;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int q = 0; q < splits; ++q) {
            const float* part = cl.map_shared_rank(dyn, q) + r * BN + c;
#pragma unroll
            for (int g = 0; g < kSplitGroups; ++g) {
                const float4 x = *reinterpret_cast<const float4*>(part + g * (BM * BN));
                s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
            }
        }
        float* dst = pp.c + (m0 + r) * p.c_sm + (n0 + c);
        const float o[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) if (n0 + c + j < p.N) dst[j] = o[j];
    }
    cl.sync();                                           // nobody leaves while a peer still reads
}

// The same parts one after the other in one CTA, where the planes bring enough tiles for the SMs: simt_contract_kernel's tiles and
// pipeline over the slices in the order of the parts, each part added to C by the threads that own its elements.
template <Fetch F, int TN>
__global__ void __launch_bounds__(128, TN == 8 || F == Fetch::ANY ? 3 : 4)
simt_contract_parts_kernel(const float* __restrict__ A, const float* __restrict__ B, float* C, const SimtContract p, int n_tiles, int parts) {
    constexpr int BM = 64, BN = 16 * TN;
    __shared__ __align__(16) float smem[2 * kSlice * (BM + BN)];
    float* const As = smem;
    float* const Bs = smem + 2 * kSlice * BM;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int arow = (warp >> 1) * 32 + lane_m(lane) * 4, bcol = (warp & 1) * (8 * TN) + lane_n(lane) * 4;
    const long long mt = blockIdx.x / n_tiles;
    const long long m0 = mt * BM, n0 = (static_cast<long long>(blockIdx.x) - mt * n_tiles) * BN;
    const int slices = static_cast<int>((p.K + kSlice - 1) / kSlice);

    for (long long plane = blockIdx.z; plane < p.planes; plane += gridDim.z) {
        const PlanePtrs<float> pp = plane_ptrs(A, B, C, p, plane);
        float acc[8][TN];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
        Loader<float, F, BM, 128> la;
        Loader<float, F, BN, 128> lb;
        la.init(pp.a, threadIdx.x, m0, p.M, 0, p.a_sm, p.a_sk, parts);
        lb.init(pp.b, threadIdx.x, n0, p.N, 0, p.b_sn, p.b_sk, parts);
        // fetches slice s and moves on to the next one of its part, or to the first of the next part
        auto fetch = [&](int s) {
            const int k_left = clip_slice(p.K - static_cast<long long>(s) * kSlice);
            la.fetch(threadIdx.x, k_left);
            lb.fetch(threadIdx.x, k_left);
            if (s + parts < slices) return s + parts;
            const int next = s % parts + 1;
            la.skip(static_cast<long long>(next - s - parts) * kSlice * p.a_sk);
            lb.skip(static_cast<long long>(next - s - parts) * kSlice * p.b_sk);
            return next;
        };
        int s = 0, ahead = fetch(0);
        la.store(threadIdx.x, As);
        lb.store(threadIdx.x, Bs);
        __syncthreads();
        for (int it = 0, buf = 0; it < slices; ++it, buf ^= 1) {
            const bool more = it + 1 < slices;
            const int now = s;
            if (more) { s = ahead; ahead = fetch(s); }
            mac_slice<F, BM, BN, TN>(As + buf * (kSlice * BM), Bs + buf * (kSlice * BN), arow, bcol, acc);
            if (now + parts >= slices) {                  // the last slice of its part
                const bool first = now % parts == 0;
#pragma unroll
                for (int jg = 0; jg < TN / 4; ++jg) {
                    const long long n = n0 + bcol + 32 * jg;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long long m = m0 + arow + (i < 4 ? i : 12 + i);
                        float* c = pp.c + m * p.c_sm + n;
                        float v[4] = {0.f, 0.f, 0.f, 0.f};
                        if (m < p.M && n < p.N) {
                            if (p.vec_c) {
                                if (!first) *reinterpret_cast<float4*>(v) = load4(c);
                                *reinterpret_cast<float4*>(c) = make_float4(v[0] + acc[i][4 * jg], v[1] + acc[i][4 * jg + 1], v[2] + acc[i][4 * jg + 2], v[3] + acc[i][4 * jg + 3]);
                            } else {
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    if (n + j < p.N) c[j] = (first ? 0.0f : c[j]) + acc[i][4 * jg + j];
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc[i][4 * jg + j] = 0.0f;
                    }
                }
            }
            if (more) {
                la.store(threadIdx.x, As + (buf ^ 1) * (kSlice * BM));
                lb.store(threadIdx.x, Bs + (buf ^ 1) * (kSlice * BN));
            }
            __syncthreads();
        }
    }
}

template <typename T, Fetch F, int WM, int WN, int TN, bool FUSED>
int launch_tile(const T* A, const T* B, float* C, const SimtContract& p, cudaStream_t st) {
    constexpr int BM = WM * 32, BN = WN * 8 * TN;
    const long long mt = (p.M + BM - 1) / BM, nt = (p.N + BN - 1) / BN;
    if (nt > 0x7fffffffLL || mt > 0x7fffffffLL / nt) return ST_BAD_ARGS;
    const unsigned planes = static_cast<unsigned>(p.planes < 32768 ? p.planes : 32768);
    simt_contract_kernel<T, F, WM, WN, TN, FUSED><<<dim3(static_cast<unsigned>(mt * nt), 1, planes), WM * WN * 32, 0, st>>>(A, B, C, p, static_cast<int>(nt));
    return cudaGetLastError() == cudaSuccess ? ST_OK : ST_LAUNCH;
}

// ---- the contraction in parts
// Clusters of each size that a B200 holds at once for two and for four groups (cudaOccupancyMaxActiveClusters, 148 SMs); constants, so that
// the number of parts follows from the extents alone.
constexpr int kSplitSms = 148;
constexpr int kResident2[17] = {0, 296, 148, 93, 71, 56, 45, 37, 33, 30, 26, 21, 21, 17, 14, 14, 14};
constexpr int kResident4[17] = {0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7};

// Groups per CTA and CTAs per cluster: clusters beyond what the GPU holds at once wait for a second wave, so the size is the one with
// the fewest slices one after the other for one plane, at three (four from 64 slices on) or more slices per part (with one, many planes
// waited for the sums: 32 of 128 x 128 over 408 45 us against 19 in one chain; 128 x 128 over 408 itself 7.6 us with three, 8.7 with four).  groups = 1, one chain: a result with a tile for more than half the SMs, or K
// below 24 slices, where the narrow form is faster (128 x 256 over 225 4.3 us against 5.8) and a chain is about as far from the 64-bit
// result as the forward product's; above, the chain falls behind in its error first (408: 6.0 us, in parts 7.7), then in time (1000 k).
struct SplitPlan { int groups, splits; long long rounds; };
inline long long split_waves(const int (&resident)[17], int splits, long long tiles) { return (tiles + resident[splits] - 1) / resident[splits]; }
inline void plan_split(SplitPlan& best, int groups, const int (&resident)[17], long long tiles, long long slices) {
    const long long least = slices < 64 ? 3 : 4;
    for (int s = 1; s <= 16 && least * s * groups <= slices; ++s) {
        const long long rounds = split_waves(resident, s, tiles) * ((slices + s * groups - 1) / (s * groups));
        if (rounds < best.rounds) best = {groups, s, rounds};
    }
}
SplitPlan plan_parts(const SimtContract& p) {
    const long long slices = (p.K + kSlice - 1) / kSlice;
    SplitPlan plan{1, 1, slices};
    if (!p.in_parts || slices < 24 || p.K > 0x7fffffffLL || p.M > 64LL * kSplitSms || p.N > 64LL * kSplitSms) return plan;
    const long long tiles = ((p.M + 63) / 64) * ((p.N + 63) / 64);
    if (2 * tiles > kSplitSms) return plan;
    plan_split(plan, 2, kResident2, tiles, slices);
    plan_split(plan, 4, kResident4, tiles, slices);
    return plan;
}

template <Fetch F, int G>
int launch_split(const float* A, const float* B, float* C, const SimtContract& p, int splits, cudaStream_t st) {
    constexpr int kSmem = G * 64 * 64 * static_cast<int>(sizeof(float));
    auto kern = simt_contract_split_kernel<F, G>;
    static bool configured[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return ST_LAUNCH; }
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            return ST_LAUNCH;
        }
        configured[dev] = true;
    }
    const int nt = static_cast<int>((p.N + 63) / 64);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    cfg.gridDim = dim3(static_cast<unsigned>((p.M + 63) / 64 * nt), 1, static_cast<unsigned>(p.planes * splits));
    cfg.blockDim = dim3(G * 128); cfg.dynamicSmemBytes = kSmem; cfg.stream = st;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1; at.val.clusterDim.y = 1; at.val.clusterDim.z = static_cast<unsigned>(splits);
    cfg.attrs = &at; cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, kern, A, B, C, p, nt) != cudaSuccess) { cudaGetLastError(); return ST_LAUNCH; }
    return ST_OK;
}

template <Fetch F, int TN>
int launch_parts(const float* A, const float* B, float* C, const SimtContract& p, int parts, cudaStream_t st) {
    const int mt = static_cast<int>((p.M + 63) / 64), nt = static_cast<int>((p.N + 16 * TN - 1) / (16 * TN));
    const unsigned planes = static_cast<unsigned>(p.planes < 32768 ? p.planes : 32768);
    simt_contract_parts_kernel<F, TN><<<dim3(static_cast<unsigned>(mt * nt), 1, planes), 128, 0, st>>>(A, B, C, p, nt, parts);
    return cudaGetLastError() == cudaSuccess ? ST_OK : ST_LAUNCH;
}

template <Fetch F>
int launch_in_parts(const float* A, const float* B, float* C, const SimtContract& p, const SplitPlan& plan, cudaStream_t st) {
    // times (ns): waves of clusters, each 1700 a slice of its groups, 120 a part for the sum and 2000 beside; or CTAs with all parts of
    // their tiles, 600 a slice and 1600 for adding a part (64 x 64 over 2601 tokens in 54 parts: 64 planes 152 us on clusters, 187 in one
    // CTA each; in 40 parts 80 on clusters)
    const long long sms = num_sms(), slices = (p.K + kSlice - 1) / kSlice;
    const int parts = plan.groups * plan.splits;
    const long long tiles = ((p.M + 63) / 64) * ((p.N + 63) / 64) * p.planes;
    const long long wave = 2000 + 120 * parts + 1700 * ((slices + parts - 1) / parts), serial = 600 * slices + 1600 * parts;
    const long long waves = split_waves(plan.groups == 2 ? kResident2 : kResident4, plan.splits, tiles);
    if (p.planes <= 16384 / plan.splits && waves * wave <= ((tiles + 2 * sms - 1) / (2 * sms)) * serial)
        return plan.groups == 2 ? launch_split<F, 2>(A, B, C, p, plan.splits, st) : launch_split<F, 4>(A, B, C, p, plan.splits, st);
    if constexpr (F != Fetch::ANY) {                      // tiles as for one chain, below
        if (p.N > 64 && ((p.M + 63) / 64) * ((p.N + 127) / 128) * p.planes >= 3 * sms) return launch_parts<F, 8>(A, B, C, p, parts, st);
    }
    return launch_parts<F, 4>(A, B, C, p, parts, st);
}

// at most half the SMs would have a 64 x 64 tile (so no extent of the launch below is large).  A CTA per SM takes 102 us for the 2601
// tokens of a 64 x 64 tile; 64 such tiles (8 planes of 128 x 256) take 60 narrow, and 128 would take twice that.
bool takes_narrow(const SimtContract& p) {
    const bool plain = p.bias == nullptr && !p.clamp && p.opm_L == 0 && p.ln_stats == nullptr && p.gate == nullptr && p.act == 0;
    return plain && p.a_sm == 1 && p.b_sn == 1 && p.c_sn == 1 && p.K >= 4 * kSlice && p.K <= 0x7fffffffLL &&
           p.M <= 64LL * num_sms() && p.N <= 64LL * num_sms() && p.planes <= num_sms() &&
           2 * ((p.M + 63) / 64) * ((p.N + 63) / 64) * p.planes <= num_sms();
}
template <int VEC>
int launch_narrow(const float* A, const float* B, float* C, const SimtContract& p, cudaStream_t st) {
    const int mt = static_cast<int>((p.M + kNarrowM - 1) / kNarrowM), nt = static_cast<int>((p.N + kNarrowN - 1) / kNarrowN);
    simt_contract_narrow_kernel<VEC><<<dim3(static_cast<unsigned>(mt * nt), 1, static_cast<unsigned>(p.planes)), kNarrowThreads, 0, st>>>(A, B, C, p, nt);
    return cudaGetLastError() == cudaSuccess ? ST_OK : ST_LAUNCH;
}

template <typename T, Fetch F>
int launch_fetch(const T* A, const T* B, float* C, const SimtContract& p, cudaStream_t st) {
    const bool fused = p.ln_stats != nullptr || p.gate != nullptr || p.act != 0;
    const int sms = num_sms();
    if (p.N <= 32)
        return fused ? launch_tile<T, F, 4, 1, 4, true>(A, B, C, p, st) : launch_tile<T, F, 4, 1, 4, false>(A, B, C, p, st);
    // 64 x 128 tiles where there are enough of them to fill the SMs three deep, 64 x 64 below
    const long long wide = ((p.M + 63) / 64) * ((p.N + 127) / 128) * p.planes;
    if constexpr (F != Fetch::ANY) {
        if (p.N > 64 && wide >= 3LL * sms)
            return fused ? launch_tile<T, F, 2, 2, 8, true>(A, B, C, p, st) : launch_tile<T, F, 2, 2, 8, false>(A, B, C, p, st);
    }
    return fused ? launch_tile<T, F, 2, 2, 4, true>(A, B, C, p, st) : launch_tile<T, F, 2, 2, 4, false>(A, B, C, p, st);
}

template <typename T>
int launch_typed(const T* A, const T* B, float* C, const SimtContract& p, cudaStream_t st) {
    // groups of four elements with one load each: aligned bases, strides and plane steps, extents in whole groups
    const size_t gb = 4 * sizeof(T);
    const bool base_ok = reinterpret_cast<uintptr_t>(A) % gb == 0 && reinterpret_cast<uintptr_t>(B) % gb == 0 &&
                         (p.ne2 == 1 || (p.a_s2 % 4 == 0 && p.b_s2 % 4 == 0)) &&
                         (p.planes == p.ne2 || (p.a_s3 % 4 == 0 && p.b_s3 % 4 == 0));
    if constexpr (std::is_same_v<T, float>) {
        const bool vec = base_ok && p.a_sm == 1 && p.b_sn == 1 && p.M % 4 == 0 && p.N % 4 == 0 && p.a_sk % 4 == 0 && p.b_sk % 4 == 0;
        const SplitPlan plan = plan_parts(p);
        if (plan.groups > 1)
            return vec ? launch_in_parts<Fetch::VEC_ROW>(A, B, C, p, plan, st) : launch_in_parts<Fetch::ANY>(A, B, C, p, plan, st);
        if (takes_narrow(p)) {
            return vec ? launch_narrow<4>(A, B, C, p, st) : launch_narrow<1>(A, B, C, p, st);
        }
    }
    if (base_ok && p.a_sk == 1 && p.b_sk == 1 && p.K % 4 == 0 && p.a_sm % 4 == 0 && p.b_sn % 4 == 0)
        return launch_fetch<T, Fetch::VEC_K>(A, B, C, p, st);
    if (base_ok && p.a_sm == 1 && p.b_sn == 1 && p.M % 4 == 0 && p.N % 4 == 0 && p.a_sk % 4 == 0 && p.b_sk % 4 == 0)
        return launch_fetch<T, Fetch::VEC_ROW>(A, B, C, p, st);
    return launch_fetch<T, Fetch::ANY>(A, B, C, p, st);
}

}  // namespace

int launch_simt_contract(const void* A, const void* B, float* C, const SimtContract& q, int elem /*0 f32,1 f16,2 bf16*/,
                         cudaStream_t st) {
    SimtContract p = q;
    if (p.M <= 0 || p.N <= 0 || p.planes <= 0 || (p.M + 63) / 64 > 65535) return ST_BAD_ARGS;
    if (p.opm_L > 0 && (p.M > 0xffffffffLL || p.N > 0xffffff00LL)) return ST_BAD_ARGS;
    if (p.b_div2 == 0) p.b_div2 = 1;
    if (p.b_div3 == 0) p.b_div3 = 1;
    if (p.c_sm == 1 && p.c_sn != 1 && p.bias == nullptr && p.opm_L == 0 && p.ln_stats == nullptr && p.gate == nullptr) {
        // the destination is contiguous along m: exchange the operands, so that it is contiguous along n
        SimtContract s = p;
        s.M = p.N; s.N = p.M; s.a_sm = p.b_sn; s.a_sk = p.b_sk; s.b_sn = p.a_sm; s.b_sk = p.a_sk; s.c_sm = p.c_sn; s.c_sn = p.c_sm;
        s.a_s2 = p.b_s2; s.a_s3 = p.b_s3; s.a_div2 = p.b_div2; s.a_div3 = p.b_div3;
        s.b_s2 = p.a_s2; s.b_s3 = p.a_s3; s.b_div2 = p.a_div2; s.b_div3 = p.a_div3;
        p = s;
        const void* t = A; A = B; B = t;
    }
    const bool c_al = (reinterpret_cast<uintptr_t>(C) & 15u) == 0 && p.N % 4 == 0 && (p.ne2 == 1 || p.c_s2 % 4 == 0) && (p.planes == p.ne2 || p.c_s3 % 4 == 0);
    p.in_parts = p.in_parts && p.c_sn == 1 && p.alpha == 1.0f && p.bias == nullptr && !p.clamp && p.opm_L == 0;
    p.vec_c = p.opm_L > 0 ? (c_al && p.opm_B == 1 && p.opm_L % 4 == 0) : (c_al && p.c_sn == 1 && p.c_sm % 4 == 0);
    if (elem == 0) return launch_typed<float>(static_cast<const float*>(A), static_cast<const float*>(B), C, p, st);
    if (elem == 1) return launch_typed<__half>(static_cast<const __half*>(A), static_cast<const __half*>(B), C, p, st);
    return launch_typed<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(A), static_cast<const __nv_bfloat16*>(B), C, p, st);
}

}  // namespace ppml_b200
