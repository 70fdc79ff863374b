// umma_gemm.cu -- host side of the tcgen05 contraction engine: eligibility checks, tensor maps,
// tile shape selection and the launch.
#include <climits>
#include <cstdlib>
#include "kernels.h"
#include "tma_host.h"
#include "umma_gemm.cuh"

namespace ppml_b200 {

int num_sms() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

namespace {

template <MmaKind KIND, int BN, Epi EPI, bool CONVERT, bool MNMAJOR = false>
int launch_one(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmParams p, cudaStream_t st) {
    auto kern = umma_gemm_kernel<KIND, BN, EPI, CONVERT, MNMAJOR>;
    constexpr int smem = gemm_smem_bytes<BN>();
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
            cudaGetLastError();
            return ST_LAUNCH;
        }
        configured[dev] = true;
    }
    p.n_tiles = (p.N + BN - 1) / BN;
    p.m_tiles = (p.M + 127) / 128;
    const long long total = static_cast<long long>(p.m_tiles) * p.n_tiles * p.batch;
    if (total <= 0 || total > 0x7fffffffLL) return ST_BAD_ARGS;
    const int grid = static_cast<int>(total < num_sms() ? total : num_sms());
    // equal row ranges per CTA instead of whole tiles dealt round robin, when the tiles do not divide evenly
    static const int flat_env = [] { const char* e = std::getenv("PPML_B200_GEMM_FLAT"); return e ? (e[0] != '0' ? 1 : 0) : 1; }();
    // (one column tile only: with several, a partial row tile costs every one of them and the round robin balances better;
    // measured at M = 65536: 36.5 -> 35.0 us at 256 x 256 tf32, 31.9 -> 31.3 at 128 x 256, but 57 -> 63 at 256 x 512)
    // (and short contractions only: at K = 1024 the partial tile costs more tensor and L2 time than the balance gains,
    // 75 -> 80 us at 65536 x 1024 x 256)
    p.flat_rows = (flat_env && p.batch == 1 && !MNMAJOR && EPI != Epi::OPM_BLOCKED && p.n_tiles == 1 && p.k_steps <= 8 &&
                   p.m_tiles > grid && p.m_tiles % grid != 0) ? 1 : 0;
    kern<<<grid, CONVERT ? 320 : 192, smem, st>>>(tmA, tmB, p);
    return cudaGetLastError() == cudaSuccess ? ST_OK : ST_LAUNCH;
}

template <MmaKind KIND, Epi EPI, bool CONVERT>
int launch_bn(int BN, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, cudaStream_t st) {
    switch (BN) {
        case 32: return launch_one<KIND, 32, EPI, CONVERT>(tmA, tmB, p, st);
        case 64: return launch_one<KIND, 64, EPI, CONVERT>(tmA, tmB, p, st);
        case 128: return launch_one<KIND, 128, EPI, CONVERT>(tmA, tmB, p, st);
        default: return launch_one<KIND, 256, EPI, CONVERT>(tmA, tmB, p, st);
    }
}

int launch_bn_mn(int BN, bool half, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, cudaStream_t st) {
    if (half) {
        switch (BN) {
            case 32: case 64: return launch_one<MmaKind::F16, 64, Epi::ROW_MAJOR, false, true>(tmA, tmB, p, st);
            case 128: return launch_one<MmaKind::F16, 128, Epi::ROW_MAJOR, false, true>(tmA, tmB, p, st);
            default: return launch_one<MmaKind::F16, 256, Epi::ROW_MAJOR, false, true>(tmA, tmB, p, st);
        }
    }
    switch (BN) {
        case 32: return launch_one<MmaKind::TF32, 32, Epi::ROW_MAJOR, false, true>(tmA, tmB, p, st);
        case 64: return launch_one<MmaKind::TF32, 64, Epi::ROW_MAJOR, false, true>(tmA, tmB, p, st);
        case 128: return launch_one<MmaKind::TF32, 128, Epi::ROW_MAJOR, false, true>(tmA, tmB, p, st);
        default: return launch_one<MmaKind::TF32, 256, Epi::ROW_MAJOR, false, true>(tmA, tmB, p, st);
    }
}

// ---- the contraction in parts (umma_gemm_split_kernel, umma_gemm_parts_kernel) -------------------------------------------
// Clusters of S CTAs of the split kernel that a B200 holds at once (one CTA per SM, 148 SMs; cudaOccupancyMaxActiveClusters), index S.
// Constants, so that the number of parts and with it the bits of a result follow from the extents alone.
constexpr int kSplitSms = 148;
constexpr int kSplitResident[17] = {0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7};
constexpr long long kStepNs = 340;             // one K step of a CTA

template <typename Kernel>
bool configure_once(Kernel kern, int smem, bool clusters, bool (&done)[64]) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return false; }
    if (done[dev]) return true;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        (clusters && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
        cudaGetLastError();
        return false;
    }
    return done[dev] = true;
}

template <int BN>
int launch_split(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmParams p, int box_a, int box_b, int parts, cudaStream_t st) {
    static bool done[64] = {false};
    auto kern = umma_gemm_split_kernel<BN>;
    if (!configure_once(kern, gemm_split_smem_bytes<BN>(), true, done)) return ST_LAUNCH;
    p.n_tiles = (p.N + BN - 1) / BN;
    p.m_tiles = (p.M + 127) / 128;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    cfg.gridDim = dim3(static_cast<unsigned>(p.m_tiles * p.n_tiles * p.batch), static_cast<unsigned>(parts));
    cfg.blockDim = dim3(192); cfg.dynamicSmemBytes = gemm_split_smem_bytes<BN>(); cfg.stream = st;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1; at.val.clusterDim.y = static_cast<unsigned>(parts); at.val.clusterDim.z = 1;
    cfg.attrs = &at; cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p, box_a, box_b) != cudaSuccess) { cudaGetLastError(); return ST_LAUNCH; }
    return ST_OK;
}

template <int BN>
int launch_parts(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmParams p, int box_a, int box_b, int parts, cudaStream_t st) {
    static bool done[64] = {false};
    auto kern = umma_gemm_parts_kernel<BN>;
    if (!configure_once(kern, gemm_parts_smem_bytes<BN>(), false, done)) return ST_LAUNCH;
    p.n_tiles = (p.N + BN - 1) / BN;
    p.m_tiles = (p.M + 127) / 128;
    const long long total = static_cast<long long>(p.m_tiles) * p.n_tiles * p.batch;
    if (total > 0x7fffffffLL - num_sms()) return ST_BAD_ARGS;
    const int grid = static_cast<int>(total < num_sms() ? total : num_sms());
    kern<<<grid, 64 + 32 * kPartsEpiWarps<BN>, gemm_parts_smem_bytes<BN>(), st>>>(tmA, tmB, p, parts, box_a, box_b);
    return cudaGetLastError() == cudaSuccess ? ST_OK : ST_LAUNCH;
}

// Time (ns) of `batch` results on clusters of S CTAs and tiles of BN columns: waves of clusters (what does not run together waits), each
// with its launch, the sum over the cluster and the K steps of a CTA.  Fitted to 32 x 32 .. 512 x 256 over 128 .. 16384 tokens at
// 1 .. 512 planes; the choice below was the faster form, or within 5 % of it, at all of them.
long long split_ns(const UmmaGemmArgs& a, int batch, int BN, int S, int k_steps) {
    if (BN > 32 && a.N <= BN / 2) return LLONG_MAX;
    const long long tiles = static_cast<long long>((a.M + 127) / 128) * ((a.N + BN - 1) / BN) * batch;
    return ((tiles + kSplitResident[S] - 1) / kSplitResident[S]) * (2900 + 27 * BN + kStepNs * ((k_steps + S - 1) / S));
}
// The same with all parts of a tile in one CTA: a part takes its K steps, or the time to add it to the sum where that is longer.
long long parts_ns(const UmmaGemmArgs& a, int BN, int parts, int k_steps) {
    const long long tiles = static_cast<long long>((a.M + 127) / 128) * ((a.N + BN - 1) / BN) * a.batch;
    const long long steps = kStepNs * ((k_steps + parts - 1) / parts), add = 390 + 4 * BN / 5;
    return 3600 + 14 * BN + ((tiles + kSplitSms - 1) / kSplitSms) * parts * (steps > add ? steps : add);
}

// Parts of the contraction, from M, N and K alone: the cluster size that is fastest for one result, at least two K steps per part (with
// one, a CTA that computes all parts waits for its sums: 512 planes of 256 x 256 over 408 tokens 107 us in 13 parts, 88 undivided).
// 1: more than half the SMs have a tile of the general kernel, or there are fewer than four K steps (256 x 256 over 256 tokens,
// eight of them: 11.7 -> 5.4 us; over 128: 9.4 -> 5.2).
int gemm_parts(const UmmaGemmArgs& a, int general_bn, int k_steps) {
    const long long tiles = static_cast<long long>((a.M + 127) / 128) * ((a.N + general_bn - 1) / general_bn);
    if (!a.may_split || k_steps < 4 || 2 * tiles > kSplitSms) return 1;
    long long best = LLONG_MAX;
    int parts = 1;
    for (int s = 2; s <= 16 && 2 * s <= k_steps; ++s)
        for (int BN : {32, 64, 128}) {
            const long long ns = split_ns(a, 1, BN, s, k_steps);
            if (ns < best) { best = ns; parts = s; }
        }
    return parts;
}

// Tile width of the split kernel for a whole call, or 0: all parts of a tile in one CTA.
int split_width(const UmmaGemmArgs& a, int general_bn, int k_steps, int parts) {
    long long best = parts_ns(a, general_bn, parts, k_steps);
    int width = 0;
    for (int BN : {32, 64, 128}) {
        const long long ns = split_ns(a, a.batch, BN, parts, k_steps);
        if (ns < best) { best = ns; width = BN; }
    }
    return width;
}

int pick_bn(int N) {
    if (N <= 32) return 32;
    if (N <= 64) return 64;
    if (N <= 128) return 128;
    return 256;
}

}  // namespace

int launch_umma_gemm(const UmmaGemmArgs& a, cudaStream_t st) {
    if (!a.A || !a.B || !a.C || a.M <= 0 || a.N <= 0 || a.K <= 0 || a.batch <= 0) return ST_BAD_ARGS;
    const int es = (a.elem == 0) ? 4 : 2;
    // TMA: 16-byte aligned bases and strides; otherwise the CUDA-core kernel takes the call
    if ((reinterpret_cast<uintptr_t>(a.A) & 15u) || (reinterpret_cast<uintptr_t>(a.B) & 15u)) return ST_UNSUPPORTED_PATH;
    if ((a.lda * es) % 16 || (a.ldb * es) % 16 || (a.a_batch * es) % 16 || (a.b_batch * es) % 16) return ST_UNSUPPORTED_PATH;
    if (a.batch > 1 && (a.a_batch == 0 || a.b_batch == 0)) return ST_UNSUPPORTED_PATH;
    int* err = device_error_ptr();
    if (!err) return ST_LAUNCH;

    const int BN = pick_bn(a.N);
    const int bk = 128 / es;
    if (a.mn_major) {
        // A[b][k][m], B[b][k][n] with the row index contiguous: fp32 operands become tf32 in the TMA unit and use
        // the 32-byte-chunk swizzle, 16-bit operands the ordinary 128-byte swizzle
        if (a.opm_L > 0) return ST_UNSUPPORTED_PATH;
        const bool half = a.elem != 0;
        const TmaType tt = !half ? TmaType::TF32 : (a.elem == 1 ? TmaType::F16 : TmaType::BF16);
        const uint32_t box = half ? 64 : 32;
        const uint64_t a_bs = (a.batch > 1) ? static_cast<uint64_t>(a.a_batch) * es : 0;
        const uint64_t b_bs = (a.batch > 1) ? static_cast<uint64_t>(a.b_batch) * es : 0;
        GemmParams p{};
        p.M = a.M; p.N = a.N; p.K = a.K; p.batch = a.batch;
        p.k_steps = (a.K + bk - 1) / bk;
        p.ab_fmt = (a.elem == 2) ? 1 : 0;
        p.C = a.C; p.ldc = a.ldc; p.c_batch = a.c_batch;
        p.bias = a.bias; p.alpha = a.alpha; p.clamp = a.clamp;
        p.err = err;
        p.vec_ok = ((reinterpret_cast<uintptr_t>(a.C) & 15u) == 0) && (a.ldc % 4 == 0) && (a.c_batch % 4 == 0) && (a.N % 4 == 0);
        const int parts = half ? 1 : gemm_parts(a, BN, p.k_steps);
        const int width = parts > 1 ? split_width(a, BN, p.k_steps, parts) : 0, bn = width ? width : BN;
        CUtensorMap tmA, tmB;
        // whole row blocks: an operand as [batch][row block][k][32], whose box holds all row blocks of a stage (one issuing thread
        // needs 60 to 80 ns per load: 256 x 256 over 65536 tokens 62 us with a box per row block)
        const int box_a = parts > 1 && a.M % 32 == 0 ? (a.M < 128 ? a.M / 32 : 4) : 0;
        const int box_b = parts > 1 && a.N % 32 == 0 ? (a.N < bn ? a.N : bn) / 32 : 0;
        auto map = [&](CUtensorMap* m, const void* base, int rows, long long pitch, uint64_t bs, int blocks) {
            const uint64_t pb = static_cast<uint64_t>(pitch) * es;
            return blocks ? make_tmap_4d(m, tt, base, 32, a.K, rows / 32, a.batch, pb, 128, bs, 32, 32, 2, blocks)
                          : make_tmap_3d(m, tt, base, rows, a.K, a.batch, pb, bs, box, box, half ? 1 : 2);
        };
        if (!map(&tmA, a.A, a.M, a.lda, a_bs, box_a) || !map(&tmB, a.B, a.N, a.ldb, b_bs, box_b)) return ST_UNSUPPORTED_PATH;
        if (parts > 1) {
            switch (width) {
                case 128: return launch_split<128>(tmA, tmB, p, box_a, box_b, parts, st);
                case 64: return launch_split<64>(tmA, tmB, p, box_a, box_b, parts, st);
                case 32: return launch_split<32>(tmA, tmB, p, box_a, box_b, parts, st);
            }
            switch (BN) {
                case 32: return launch_parts<32>(tmA, tmB, p, box_a, box_b, parts, st);
                case 64: return launch_parts<64>(tmA, tmB, p, box_a, box_b, parts, st);
                case 128: return launch_parts<128>(tmA, tmB, p, box_a, box_b, parts, st);
                default: return launch_parts<256>(tmA, tmB, p, box_a, box_b, parts, st);
            }
        }
        return launch_bn_mn(BN, half, tmA, tmB, p, st);
    }
    TmaType tt = (a.elem == 0) ? (a.tf32_mode == 1 ? TmaType::TF32 : TmaType::F32)
                               : (a.elem == 1 ? TmaType::F16 : TmaType::BF16);
    CUtensorMap tmA, tmB;
    const uint64_t a_bs = (a.batch > 1) ? static_cast<uint64_t>(a.a_batch) * es : 0;
    const uint64_t b_bs = (a.batch > 1) ? static_cast<uint64_t>(a.b_batch) * es : 0;
    if (!make_tmap_3d(&tmA, tt, a.A, a.K, a.M, a.batch, static_cast<uint64_t>(a.lda) * es, a_bs, bk, 128, true))
        return ST_UNSUPPORTED_PATH;
    if (!make_tmap_3d(&tmB, tt, a.B, a.K, a.N, a.batch, static_cast<uint64_t>(a.ldb) * es, b_bs, bk, BN, true))
        return ST_UNSUPPORTED_PATH;

    GemmParams p{};
    p.M = a.M; p.N = a.N; p.K = a.K; p.batch = a.batch;
    p.k_steps = (a.K + bk - 1) / bk;
    p.C = a.C; p.ldc = a.ldc; p.c_batch = a.c_batch;
    p.bias = a.bias; p.alpha = a.alpha; p.clamp = a.clamp;
    p.ln_stats = a.ln_stats; p.ln_u = a.ln_u; p.gate = a.gate; p.act = a.act;
    p.opm_D = a.opm_D; p.opm_L = a.opm_L;
    p.ab_fmt = (a.elem == 2) ? 1 : 0;
    p.err = err;
    const bool c_al = (reinterpret_cast<uintptr_t>(a.C) & 15u) == 0;
    if (a.opm_L > 0) p.vec_ok = c_al && (a.opm_L % 4 == 0);
    else p.vec_ok = c_al && (a.ldc % 4 == 0) && (a.c_batch % 4 == 0) && (a.N % 4 == 0);

    const bool opm = a.opm_L > 0;
    const bool fused = a.ln_stats != nullptr || a.gate != nullptr || a.act != 0;
    if (fused) {                                   // fp32 operands, row-major result only
        if (opm || a.elem != 0) return ST_UNSUPPORTED_PATH;
        return (a.tf32_mode == 0) ? launch_bn<MmaKind::TF32, Epi::ROW_MAJOR_FUSED, true>(BN, tmA, tmB, p, st)
                                  : launch_bn<MmaKind::TF32, Epi::ROW_MAJOR_FUSED, false>(BN, tmA, tmB, p, st);
    }
    if (a.elem == 0) {
        const bool conv = (a.tf32_mode == 0);
        if (opm) return conv ? launch_bn<MmaKind::TF32, Epi::OPM_BLOCKED, true>(BN, tmA, tmB, p, st)
                             : launch_bn<MmaKind::TF32, Epi::OPM_BLOCKED, false>(BN, tmA, tmB, p, st);
        return conv ? launch_bn<MmaKind::TF32, Epi::ROW_MAJOR, true>(BN, tmA, tmB, p, st)
                    : launch_bn<MmaKind::TF32, Epi::ROW_MAJOR, false>(BN, tmA, tmB, p, st);
    }
    if (opm) return launch_bn<MmaKind::F16, Epi::OPM_BLOCKED, false>(BN, tmA, tmB, p, st);
    return launch_bn<MmaKind::F16, Epi::ROW_MAJOR, false>(BN, tmA, tmB, p, st);
}

}  // namespace ppml_b200
