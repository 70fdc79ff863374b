// simt_contract.cu -- exact-fp32 contraction on CUDA cores: every product the tensor-core paths do not take (unaligned K, inner
// batch > 1, tiny extents, broadcast planes) and every product the caller wants in plain fp32.
//
//   D[p][m][n] = epi( sum_k A[pa][m][k] * B[pb][n][k] )
//
// Each output element is one chain of fused multiply-adds with k ascending, the reference's order (unless the contraction is
// split, see below), so fp32 results agree with its CPU kernels to rounding.
#include "kernels.h"

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <mutex>

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
#pragma unroll
        for (int jg = 0; jg < TN / 4; ++jg) {
            const long long n = n0 + bcol + 32 * jg;
            if (n >= p.N) continue;
            float bias[4] = {0.f, 0.f, 0.f, 0.f};
            if (!p.bias_seed && p.bias != nullptr) {
#pragma unroll
                for (int j = 0; j < 4; ++j) if (n + j < p.N) bias[j] = p.bias[n + j];
            }
            long long co[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) co[j] = col_off(n + j);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const long long m = m0 + arow + (i < 4 ? i : 12 + i);
                if (m >= p.M) continue;
                float v[4];
                float mean = 0.0f, rstd = 1.0f;
                if (FUSED && p.ln_stats != nullptr) { mean = p.ln_stats[2 * m]; rstd = p.ln_stats[2 * m + 1]; }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] = acc[i][4 * jg + j] * p.alpha;
                    if (FUSED && p.ln_stats != nullptr && n + j < p.N) v[j] = fmaf(-mean, p.ln_u[n + j], v[j]) * rstd;
                    if (!p.bias_seed && p.bias != nullptr) v[j] += bias[j];
                    if (p.clamp) v[j] = (v[j] == v[j]) ? fminf(fmaxf(v[j], -1e4f), 1e4f) : 0.0f;
                }
                const long long r0 = row_off(m);
                if constexpr (FUSED) {
#pragma unroll 1
                    for (int j = 0; j < 4; ++j) {
                        if (n + j >= p.N) break;
                        const long long off = r0 + (n + j) * p.c_sn;          // row-major here
                        float x = j == 0 ? v[0] : (j == 1 ? v[1] : (j == 2 ? v[2] : v[3]));
                        if (p.gate != nullptr) x = act_scalar(p.act, x) * p.gate[off];
                        else if (p.act != 0) x = act_scalar(p.act, x);
                        Cp[off] = x;
                    }
                } else if (p.vec_c) {
                    *reinterpret_cast<float4*>(Cp + r0 + co[0]) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) if (n + j < p.N) Cp[r0 + co[j]] = v[j];
                }
            }
        }
    }
}

// The split form, for plain products whose contraction is long and whose result is small (weight gradients: K = the tokens):
// a CTA is two or four groups of four warps, a cluster up to 16 CTAs, and the groups take the slices of k of one 64 x 64 tile in turn, with
// stages and a barrier of their own.  The partial tiles are left in shared memory and added piece by piece over the cluster in
// the order of the groups (no atomics: the result does not depend on timing).
//
// Bound: FMA issue with 16 or more tiles; latency of a group's loads below that (one slice in flight per group), which is why
// the ways are many and short.  256 x 256 over 65536 tokens 4850 -> 289 us (one CTA per 64 x 64 tile before), 64 x 256 over
// 30000 1490 -> 63 us, 33 x 32 over 30000 1470 -> 76 us.  A group's slices lie next to the other groups', not in a range of its
// own: all of them then move through the operands together.
template <typename T, Fetch F, int kSplitGroups>
__global__ void __launch_bounds__(kSplitGroups * 128, 4 / kSplitGroups)
simt_contract_split_kernel(const T* __restrict__ A, const T* __restrict__ B, float* __restrict__ C, const SimtContract p, int n_tiles) {
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
    const PlanePtrs<T> pp = plane_ptrs(A, B, C, p, blockIdx.z / splits);

    const long long ways = static_cast<long long>(splits) * kSplitGroups;
    const long long kbeg = (rank * kSplitGroups + grp) * static_cast<long long>(kSlice), kstep = ways * kSlice;
    long long k_left = p.K - kbeg;                       // not positive: a group without a share
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory"); };
    Loader<T, F, BM, 128> la;
    Loader<T, F, BN, 128> lb;
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
        const float o[4] = {s.x * p.alpha, s.y * p.alpha, s.z * p.alpha, s.w * p.alpha};
#pragma unroll
        for (int j = 0; j < 4; ++j) if (n0 + c + j < p.N) dst[j] = o[j];
    }
    cl.sync();                                           // nobody leaves while a peer still reads
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

// CTAs per cluster: clusters beyond what the GPU's processor clusters hold at once wait for a second wave, so the size is the one
// with the fewest slices one after the other (resident[S]: clusters of S that run together, 148 SMs: 74 of 2, 33 of 4, 15 of 8
// and 7 of 16 with four groups, 33 of 8 and 14 of 16 with two).
struct SplitPlan { int groups, splits; long long rounds; };
inline void plan_split(SplitPlan& best, int groups, const int (&resident)[17], long long tiles, long long slices) {
    for (int s = 1; s <= 16; ++s) {
        if (resident[s] <= 0 || static_cast<long long>(s - 1) * groups >= slices) break;
        const long long rounds = ((tiles + resident[s] - 1) / resident[s]) * ((slices + s * groups - 1) / (s * groups));
        if (rounds < best.rounds) best = {groups, s, rounds};
    }
}

template <typename T, Fetch F, int G>
struct SplitKernel {
    static constexpr int kThreads = G * 128, kSmem = G * 64 * 64 * static_cast<int>(sizeof(float));
    static void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at, dim3 grid, int splits, cudaStream_t st) {
        cfg.gridDim = grid; cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = kSmem; cfg.stream = st;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 1; at.val.clusterDim.y = 1; at.val.clusterDim.z = static_cast<unsigned>(splits);
        cfg.attrs = &at; cfg.numAttrs = 1;
    }
    // clusters of each size that are resident together on the current device, asked once per device; null on an error
    static const int (*resident(int dev))[17] {
        static int table[64][17];
        static std::once_flag once[64];
        static bool ok[64];
        std::call_once(once[dev], [&] {
            auto kern = simt_contract_split_kernel<T, F, G>;
            ok[dev] = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) == cudaSuccess &&
                      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
            for (int s = 1; ok[dev] && s <= 16; ++s) {
                cudaLaunchConfig_t cfg{};
                cudaLaunchAttribute at{};
                config(cfg, at, dim3(1, 1, static_cast<unsigned>(s)), s, nullptr);
                int n = 0;
                table[dev][s] = cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess ? n : 0;
            }
            cudaGetLastError();
        });
        return ok[dev] ? &table[dev] : nullptr;
    }
    static int launch(const T* A, const T* B, float* C, const SimtContract& p, int splits, cudaStream_t st) {
        const int nt = static_cast<int>((p.N + 63) / 64);
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        config(cfg, at, dim3(static_cast<unsigned>((p.M + 63) / 64 * nt), 1, static_cast<unsigned>(p.planes * splits)), splits, st);
        if (cudaLaunchKernelEx(&cfg, simt_contract_split_kernel<T, F, G>, A, B, C, p, nt) != cudaSuccess) { cudaGetLastError(); return ST_LAUNCH; }
        return ST_OK;
    }
};

// ST_UNSUPPORTED_PATH: not worth a split
template <typename T, Fetch F>
int launch_split(const T* A, const T* B, float* C, const SimtContract& p, long long tiles, cudaStream_t st) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return ST_UNSUPPORTED_PATH; }
    const auto* r2 = SplitKernel<T, F, 2>::resident(dev);
    const auto* r4 = SplitKernel<T, F, 4>::resident(dev);
    if (!r2 || !r4) return ST_UNSUPPORTED_PATH;
    const long long slices = (p.K + kSlice - 1) / kSlice;
    SplitPlan plan{1, 1, slices};
    plan_split(plan, 2, *r2, tiles, slices);
    plan_split(plan, 4, *r4, tiles, slices);
    if (plan.groups == 1) return ST_UNSUPPORTED_PATH;
    return plan.groups == 2 ? SplitKernel<T, F, 2>::launch(A, B, C, p, plan.splits, st) : SplitKernel<T, F, 4>::launch(A, B, C, p, plan.splits, st);
}

template <typename T, Fetch F>
int launch_fetch(const T* A, const T* B, float* C, const SimtContract& p, cudaStream_t st) {
    const bool fused = p.ln_stats != nullptr || p.gate != nullptr || p.act != 0;
    const int sms = num_sms();
    const long long small = ((p.M + 63) / 64) * ((p.N + 63) / 64) * p.planes;
    if (p.may_split && !fused && 2 * small <= sms && p.K >= 4 * kSlice) {      // at most half the SMs would have a tile
        const int rc = launch_split<T, F>(A, B, C, p, small, st);
        if (rc != ST_UNSUPPORTED_PATH) return rc;
    }
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
    p.vec_c = p.opm_L > 0 ? (c_al && p.opm_B == 1 && p.opm_L % 4 == 0) : (c_al && p.c_sn == 1 && p.c_sm % 4 == 0);
    p.may_split = p.may_split && p.c_sn == 1 && p.bias == nullptr && !p.clamp && p.opm_L == 0;
    if (elem == 0) return launch_typed<float>(static_cast<const float*>(A), static_cast<const float*>(B), C, p, st);
    if (elem == 1) return launch_typed<__half>(static_cast<const __half*>(A), static_cast<const __half*>(B), C, p, st);
    return launch_typed<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(A), static_cast<const __nv_bfloat16*>(B), C, p, st);
}

}  // namespace ppml_b200
