// K5: FP64 centring + top-k symmetric eigensolve on the GPU
// (src/kernels.rs:311-348 uses faer's dense self_adjoint_eigen on the CPU).
//
//   cov = (G - c c^T / n) / (n - 1)    (FP64, from the upper triangle of G)
//   total = trace(cov)
//   top-k eigenpairs, descending, clamped at 0, largest |loading| positive.
//
// d <= 160: cyclic Jacobi on the whole matrix in one CTA (matrix in shared
// memory, round-robin parallel ordering).
//
// d > 160: Chebyshev-filtered subspace iteration (Zhou & Saad 2007) with
// locking, on a block of p = k + 14 (rounded up to 16) vectors:
//  * a short Lanczos run brackets the spectrum;
//    the filter damps [lambda_min, a] with a = the smallest active Ritz
//    value, so eigenvalues far from zero (scaled single-cell data: a dense
//    bulk near 1) still separate quickly;
//  * converged leading Ritz pairs are locked; the filter then acts on the
//    remaining columns only, keeping the dynamic range among active columns
//    small (one dominant component no longer swamps the bulk edge);
//  * the filter degree follows the estimated gap: enough growth per outer
//    step for the weakest wanted value, bounded so the block stays well
//    conditioned for Cholesky QR;
//  * orthonormalisation is shifted Cholesky QR (Fukaya et al. 2020) built
//    from split-K FP64 GEMMs (this file; no library GEMM), Rayleigh-Ritz is a
//    cyclic Jacobi on the p x p projected matrix (k_rr, eig_block.cuh, for
//    p <= 64, else the one-CTA kernel of d <= 160).
// Stops when every wanted residual ||C v - theta v|| <= tol * theta_1.
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "eig_block.cuh"
#include "kernels.cuh"
#include "prof.cuh"

namespace crest {
namespace {

constexpr int kJacobiMax = 160;
constexpr int kJacobiSmemV = kBlkMax;  // V also kept in shared memory up to this size
constexpr int kLanczos = 32;  // steps of the spectrum-bounds run

// ------------------------------------------------------------ centring
// Matrices and blocks of the solver have ld = d rounded up to 16 rows, the
// extra rows and columns zero: every product then has aligned columns and
// whole tiles whatever d is, and zero rows of a block stay zero.
__global__ void k_centre(const double *__restrict__ G, const double *__restrict__ c, int64_t d, int64_t ld, double n,
                         double *__restrict__ C) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ld * ld) return;
    const int64_t i = idx / ld, j = idx % ld;
    if (i >= d || j >= d) {
        C[idx] = 0.0;
        return;
    }
    const int64_t a = i <= j ? i : j, b = i <= j ? j : i;
    C[idx] = __ddiv_rn(__dsub_rn(G[a * d + b], __ddiv_rn(__dmul_rn(c[a], c[b]), n)), __dsub_rn(n, 1.0));
}

// total = sum_i cov[i][i] in index order (src/kernels.rs:323): the diagonal
// is gathered 1024 entries at a time into shared memory by the whole block,
// then added up in order by one thread.
__global__ void __launch_bounds__(1024) k_trace(const double *__restrict__ C, int64_t d, int64_t ld, double *total) {
    __shared__ double diag[1024];
    double s = 0.0;
    for (int64_t i0 = 0; i0 < d; i0 += 1024) {
        const int64_t i = i0 + threadIdx.x;
        if (i < d) diag[threadIdx.x] = C[i * ld + i];
        __syncthreads();
        if (threadIdx.x == 0) {
            const int64_t n = d - i0 < 1024 ? d - i0 : 1024;
            for (int64_t j = 0; j < n; ++j) s = __dadd_rn(s, diag[j]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = s;
}

// ------------------------------------------------------------------ GEMM
// Column-major FP64 GEMM: O = alpha * op(A) B + beta * X + gamma * Y, with an
// optional split of K over gridDim.z (partials to ws, then k_gemm_reduce).
struct Gemm {
    int M, N, K;
    const double *A;
    int lda;
    int tA;
    const double *B;
    int ldb;
    double *O;
    int ldo;
    double alpha;
    const double *X;
    double beta;
    const double *Y;
    double gamma;
    int tB = 0;  // 1: B is given transposed (element (k, n) at B[n + k ldb])
    // 1: may start before the launch ahead of it has ended, reading A only
    // until then; nothing in flight may write A
    int overlap = 0;
};

// 128 x 64 output tile per CTA (128 threads, 8 x 8 outputs each: rows
// 8 tr .. 8 tr + 7, columns 8 tc .. 8 tc + 7), K in steps of 8 staged
// through double-buffered shared memory with the next step's loads in
// registers.  gridDim.z splits K: each slice writes its partial product to
// ws (summed in slice order by k_gemm_reduce, so results do not depend on
// scheduling); without a split the epilogue is applied here.
constexpr int kGM = 128, kGN = 64, kGK = 8;

__global__ void __launch_bounds__(128) k_gemm(Gemm g, int kchunk, double *ws) {
    __shared__ __align__(16) double As[2][kGK][kGM];
    __shared__ __align__(16) double Bs[2][kGK][kGN];
    const int m0 = blockIdx.x * kGM, n0 = blockIdx.y * kGN;
    const int kb = blockIdx.z * kchunk, ke = min(g.K, kb + kchunk);
    const int tid = threadIdx.x, tr = tid >> 3, tc = tid & 7;
    double acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0;
    double ra[8], rb[4];
    // element r of this thread's share: A (m, k) and B (k, n) of the K step at k0
    auto a_mk = [&](int r, int &mm, int &kk) {
        const int e = tid + 128 * r;
        if (!g.tA) {
            mm = e & (kGM - 1);
            kk = e >> 7;
        } else {
            kk = e & (kGK - 1);
            mm = e >> 3;
        }
    };
    auto b_kn = [&](int r, int &kk, int &nn) {
        const int e = tid + 128 * r;
        if (!g.tB) {
            kk = e & (kGK - 1);
            nn = e >> 3;
        } else {
            nn = e & (kGN - 1);
            kk = e >> 6;
        }
    };
    auto gload = [&](int k0) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            int mm, kk;
            a_mk(r, mm, kk);
            const int m = m0 + mm, k = k0 + kk;
            ra[r] = (m < g.M && k < ke) ? (g.tA ? g.A[k + (int64_t)m * g.lda] : g.A[m + (int64_t)k * g.lda]) : 0.0;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            int kk, nn;
            b_kn(r, kk, nn);
            const int n = n0 + nn, k = k0 + kk;
            rb[r] = (n < g.N && k < ke) ? (g.tB ? g.B[n + (int64_t)k * g.ldb] : g.B[k + (int64_t)n * g.ldb]) : 0.0;
        }
    };
    auto sstore = [&](int buf) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            int mm, kk;
            a_mk(r, mm, kk);
            As[buf][kk][mm] = ra[r];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            int kk, nn;
            b_kn(r, kk, nn);
            Bs[buf][kk][nn] = rb[r];
        }
    };
    int buf = 0;
    if (kb < ke) {
        gload(kb);
        sstore(0);
    }
    __syncthreads();
    for (int k0 = kb; k0 < ke; k0 += kGK) {
        const bool more = k0 + kGK < ke;
        if (more) gload(k0 + kGK);
#pragma unroll
        for (int kk = 0; kk < kGK; ++kk) {
            double a[8], b[8];
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                const double2 va = *reinterpret_cast<const double2 *>(&As[buf][kk][tr * 8 + i]);
                const double2 vb = *reinterpret_cast<const double2 *>(&Bs[buf][kk][tc * 8 + i]);
                a[i] = va.x;
                a[i + 1] = va.y;
                b[i] = vb.x;
                b[i + 1] = vb.y;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        if (more) sstore(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int m = m0 + tr * 8 + i, n = n0 + tc * 8 + j;
            if (m >= g.M || n >= g.N) continue;
            if (ws) {
                ws[((int64_t)blockIdx.z * g.N + n) * g.M + m] = acc[i][j];
                continue;
            }
            const int64_t o = m + (int64_t)n * g.ldo;
            double v = g.alpha * acc[i][j];
            if (g.X) v += g.beta * g.X[o];
            if (g.Y) v += g.gamma * g.Y[o];
            g.O[o] = v;
        }
}

__global__ void k_gemm_reduce(Gemm g, int ksplit, const double *__restrict__ ws) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)g.M * g.N) return;
    const int m = (int)(idx % g.M), n = (int)(idx / g.M);
    double s = 0.0;
    for (int z = 0; z < ksplit; ++z) s += ws[((int64_t)z * g.N + n) * g.M + m];
    const int64_t o = m + (int64_t)n * g.ldo;
    double v = g.alpha * s;
    if (g.X) v += g.beta * g.X[o];
    if (g.Y) v += g.gamma * g.Y[o];
    g.O[o] = v;
}

// Tall-skinny products O = alpha op(A) B + beta X + gamma Y with B (K x N,
// N <= 64) column-major and op(A) = A (M x K) or A^T (A given K x M), all
// column-major (the filter and Rayleigh-Ritz products C V and V^T W of the
// subspace iteration): FP64 tensor-core MMAs (m16n8k16).
//
// CTA tile 64 x 8 FN with FN = ceil(N / 8), so the padding of N is at most 7
// columns; four warps of 16 x 8 FN outputs each.  K in steps of 16 through a
// four-stage cp.async ring; shared-memory rows are padded so that each
// half-warp's 8-byte fragment loads fall in 16 distinct 8-byte slots (row
// strides of 68 and 20 doubles are 4 mod 16; op(A) = A^T is staged [m][k]
// like B).  K is split over gridDim.z = the cluster's z extent: every slice
// leaves its partial tile in its own shared memory, and after a cluster
// barrier slice r sums its share of all slices' partials in slice order
// (distributed shared memory), so results do not depend on scheduling.
//
// The 2000 x N x 2000 filter products are bound by the FP64 MMA rate (36.9
// TFLOP/s measured, 13.9 us at N = 64) plus about 8 us of launch, first loads
// and reduction: 24.7 us at N = 64, 16.5 at N = 32.  Eight warps of 16 x 32
// took 28.9; a second resident wave of 9 slices, 128-row tiles with one CTA
// per SM (only 15 clusters of 8 fit) and fewer slices are all slower.
// A launch with overlap set starts while the previous product drains and
// fetches its first tiles of A, which no kernel in flight writes.  The ring
// is padded to kTwoPerSm so that the early CTAs wait for a finished one's
// place: as third residents they crowd some SMs (35 us).
namespace dm {
constexpr int kBM = 64, kBK = 16, kST = 4, kThreads = 128;
constexpr int kAS = kBM + 4;  // A staging [k][m]: m stride
constexpr int kBS = kBK + 4;  // [n][k] (and A^T's [m][k]) staging: k stride
constexpr int kPS = kBM + 2;  // partial tile [n][m]: m stride
constexpr int kMaxSplit = 16;
constexpr size_t kTwoPerSm = 78 * 1024;
static_assert(kAS % 16 == 4 && kBS % 16 == 4, "fragment loads must not conflict");
static_assert(kBM * kBS >= kBK * kAS, "either A staging fits its stage");

template <int FN>
constexpr size_t smem_bytes() {
    const size_t ring = sizeof(double) * (size_t)kST * (kBM + 8 * FN) * kBS;
    static_assert((size_t)kST * (kBM + 8 * FN) * kBS >= (size_t)kPS * 8 * FN, "partial tile must fit the ring");
    return ring > kTwoPerSm ? ring : kTwoPerSm;
}

__device__ __forceinline__ void cp16(void *smem, const void *gmem, bool ok) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// a: rows ar, ar + 8 of columns ac, ac + 4, .. ac + 12 (row + 8 first); b: rows
// ac, ac + 4, .. of column ar; c: (ar, 2 ac), (ar, 2 ac + 1), then rows + 8
__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, "
        "{%4, %5, %6, %7, %8, %9, %10, %11}, {%12, %13, %14, %15}, {%0, %1, %2, %3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
          "d"(b[2]), "d"(b[3]));
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// generic address of the same shared-memory location in cluster CTA `rank`
__device__ __forceinline__ const double *cluster_ptr(const double *p, unsigned rank) {
    uint64_t r;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(reinterpret_cast<uint64_t>(p)), "r"(rank));
    return reinterpret_cast<const double *>(r);
}

template <int FN, bool TA>
__global__ void __launch_bounds__(kThreads, 2) k_gemm_dmma(Gemm g, int kchunk) {
    constexpr int BN = 8 * FN;
    extern __shared__ __align__(16) double sm[];
    double *As = sm, *Bs = sm + kST * kBM * kBS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.x * kBM;
    const int kb = blockIdx.z * kchunk, ke = min(g.K, kb + kchunk);
    const int ntiles = ke > kb ? (ke - kb + kBK - 1) / kBK : 0;

    // chunks of two doubles; this thread's place in a row of 8 (along k) or 32 (along m)
    const int lr = tid >> 3, lc = (tid & 7) * 2;
    auto load_a = [&](int t, int stage) {
        double *as = As + stage * kBM * kBS;
        if (TA) {
            const int k = kb + t * kBK + lc;
#pragma unroll
            for (int r = 0; r < kBM; r += kThreads / 8) {
                const int m = m0 + lr + r;
                const bool ok = m < g.M && k < ke;
                cp16(as + (lr + r) * kBS + lc, ok ? g.A + k + (int64_t)m * g.lda : g.A, ok);
            }
        } else {
            const int mm = (tid & 31) * 2, m = m0 + mm;
#pragma unroll
            for (int r = 0; r < kBK; r += kThreads / 32) {
                const int kk = (tid >> 5) + r, k = kb + t * kBK + kk;
                const bool ok = m < g.M && k < ke;
                cp16(as + kk * kAS + mm, ok ? g.A + m + (int64_t)k * g.lda : g.A, ok);
            }
        }
    };
    auto load_b = [&](int t, int stage) {
        double *bs = Bs + stage * BN * kBS;
        const int k = kb + t * kBK + lc;
#pragma unroll
        for (int r = 0; r < BN; r += kThreads / 8) {
            const int n = lr + r;
            if (n >= BN) break;
            const bool ok = n < g.N && k < ke;
            cp16(bs + n * kBS + lc, ok ? g.B + k + (int64_t)n * g.ldb : g.B, ok);
        }
    };

    double acc[FN][4];
#pragma unroll
    for (int j = 0; j < FN; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
    for (int s = 0; s < kST - 1; ++s)
        if (s < ntiles && g.overlap) load_a(s, s);
    asm volatile("griddepcontrol.wait;" ::: "memory");  // B, X and Y come from the launch before
#pragma unroll
    for (int s = 0; s < kST - 1; ++s) {
        if (s < ntiles) {
            if (!g.overlap) load_a(s, s);
            load_b(s, s);
        }
        cp_commit();  // the first group also covers every early load of A
    }
    const int ar = lane >> 2, ac = lane & 3;  // fragment row / column of this lane
    for (int t = 0; t < ntiles; ++t) {
        cp_wait<kST - 2>();
        __syncthreads();
        if (t + kST - 1 < ntiles) {
            load_a(t + kST - 1, (t + kST - 1) % kST);
            load_b(t + kST - 1, (t + kST - 1) % kST);
        }
        cp_commit();
        const double *as = As + (t % kST) * kBM * kBS + (TA ? (warp * 16 + ar) * kBS + ac : warp * 16 + ar + ac * kAS);
        const double *bs = Bs + (t % kST) * BN * kBS + ar * kBS + ac;
        double a[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            a[q] = TA ? as[8 * (q & 1) * kBS + 4 * (q >> 1)] : as[8 * (q & 1) + 4 * (q >> 1) * kAS];
#pragma unroll
        for (int j = 0; j < FN; ++j) {
            double b[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) b[q] = bs[j * 8 * kBS + 4 * q];
            dmma(acc[j], a, b);
        }
    }
    cp_wait<0>();

    auto out = [&](int m, int n, double v) {
        if (m >= g.M || n >= g.N) return;
        const int64_t o = m + (int64_t)n * g.ldo;
        double r = g.alpha * v;
        if (g.X) r += g.beta * g.X[o];
        if (g.Y) r += g.gamma * g.Y[o];
        g.O[o] = r;
    };
    const int ks = (int)gridDim.z;
    if (ks == 1) {
#pragma unroll
        for (int j = 0; j < FN; ++j)
#pragma unroll
            for (int h = 0; h < 4; ++h) out(m0 + warp * 16 + ar + 8 * (h >> 1), j * 8 + ac * 2 + (h & 1), acc[j][h]);
        return;
    }
    // partial tile [n][m] in this CTA's ring, then the cluster-wide split of its pairs of rows
    __syncthreads();
    double *part = sm;
#pragma unroll
    for (int j = 0; j < FN; ++j)
#pragma unroll
        for (int h = 0; h < 4; ++h) part[(j * 8 + ac * 2 + (h & 1)) * kPS + warp * 16 + ar + 8 * (h >> 1)] = acc[j][h];
    cluster_sync_all();
    const int pairs = kBM / 2 * BN, per = (pairs + ks - 1) / ks;
    const int e0 = (int)blockIdx.z * per, e1 = min(pairs, e0 + per);
    for (int e = e0 + tid; e < e1; e += kThreads) {
        const int n = e / (kBM / 2), m = e % (kBM / 2) * 2;
        double v0 = 0.0, v1 = 0.0;
        for (int z = 0; z < ks; ++z) {
            const double2 v = *reinterpret_cast<const double2 *>(cluster_ptr(part + n * kPS + m, (unsigned)z));
            v0 += v.x;
            v1 += v.y;
        }
        out(m0 + m, n, v0);
        out(m0 + m + 1, n, v1);
    }
    cluster_sync_all();  // no CTA leaves while another reads its partial
}
}  // namespace dm

struct GemmWs {
    DevBuf ws;
};

static bool dmma_enabled() {  // CREST_EIG_DMMA=0: CUDA-core kernel for every product
    static const bool on = [] {
        const char *e = getenv("CREST_EIG_DMMA");
        return !(e && e[0] == '0');
    }();
    return on;
}

static bool dmma_fits(const Gemm &g) {
    auto al = [](const void *p) { return ((uintptr_t)p & 15) == 0; };
    return !g.tB && g.N >= 1 && g.N <= 64 && g.M >= 1 && g.K >= dm::kBK && !(g.K & 1) && !(g.lda & 1) &&
           !(g.ldb & 1) && (g.tA || !(g.M & 1)) && al(g.A) && al(g.B);
}

template <int FN, bool TA>
static int launch_dmma(const Gemm &g, cudaStream_t st) {
    constexpr size_t smem = dm::smem_bytes<FN>();
    const void *fn = (const void *)dm::k_gemm_dmma<FN, TA>;
    CREST_TRY(ensure_smem_attr(fn, smem));
    static bool nonportable = [fn] {
        const bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        (void)cudaGetLastError();
        return ok;
    }();
    const int mt = (int)ceil_div(g.M, dm::kBM);
    // K split = the cluster's z extent: about two CTAs per SM, slices of at
    // least 64, a power of two up to 16 (8 without non-portable clusters)
    const int want = std::max(1, std::min((2 * device_sms()) / mt, g.K / (4 * dm::kBK)));
    int ks = 1;
    while (ks * 2 <= want && ks * 2 <= (nonportable ? dm::kMaxSplit : 8)) ks *= 2;
    auto launch = [&](int z) {
        const int kc = z > 1 ? (int)round_up(ceil_div(g.K, z), dm::kBK) : g.K;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(mt, 1, z);
        cfg.blockDim = dim3(dm::kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = z;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = g.overlap ? 2 : 1;
        return cudaLaunchKernelEx(&cfg, dm::k_gemm_dmma<FN, TA>, g, kc);
    };
    cudaError_t e = launch(ks);
    if (e != cudaSuccess && ks > 1) {  // a cluster shape that cannot be placed: a power of two up to 8
        (void)cudaGetLastError();
        int z = 1;
        while (z * 2 <= std::min(ks, 8)) z *= 2;
        e = launch(z);
    }
    CREST_CUDA_TRY(e);
    return CREST_OK;
}

template <bool TA>
static int gemm_dmma(const Gemm &g, cudaStream_t st) {
    switch ((g.N + 7) / 8) {
        case 1: return launch_dmma<1, TA>(g, st);
        case 2: return launch_dmma<2, TA>(g, st);
        case 3: return launch_dmma<3, TA>(g, st);
        case 4: return launch_dmma<4, TA>(g, st);
        case 5: return launch_dmma<5, TA>(g, st);
        case 6: return launch_dmma<6, TA>(g, st);
        case 7: return launch_dmma<7, TA>(g, st);
        default: return launch_dmma<8, TA>(g, st);
    }
}

int gemm(const Gemm &g, GemmWs &w, cudaStream_t st) {
    prof::Scope ps("eig_gemm_fp64", st);
    if (dmma_fits(g) && dmma_enabled()) return g.tA ? gemm_dmma<true>(g, st) : gemm_dmma<false>(g, st);
    const int mt = (int)ceil_div(g.M, kGM), nt = (int)ceil_div(g.N, kGN);
    int ksplit = 1;
    if (g.K > 0) {  // about one CTA per SM, slices of at least 64
        const int want = (int)ceil_div(device_sms(), mt * nt);
        ksplit = std::max(1, std::min(want, (int)ceil_div(g.K, 64)));
    }
    if (ksplit == 1) {
        k_gemm<<<dim3(mt, nt, 1), 128, 0, st>>>(g, std::max(g.K, 1), nullptr);
        CREST_CUDA_TRY(cudaGetLastError());
        return CREST_OK;
    }
    const int kchunk = (int)round_up(ceil_div(g.K, ksplit), kGK);
    ksplit = (int)ceil_div(g.K, kchunk);
    CREST_TRY(w.ws.ensure(sizeof(double) * (size_t)ksplit * g.M * g.N));
    k_gemm<<<dim3(mt, nt, ksplit), 128, 0, st>>>(g, kchunk, w.ws.as<double>());
    CREST_CUDA_TRY(cudaGetLastError());
    k_gemm_reduce<<<(unsigned)ceil_div((int64_t)g.M * g.N, 256), 256, 0, st>>>(g, ksplit, w.ws.as<double>());
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

// ---------------------------------------------------------------- Jacobi
// Cyclic Jacobi on a symmetric n_in x n_in column-major matrix (padded to an
// even n with a decoupled zero row/column).  Round-robin ordering: n/2
// disjoint pairs per round, n-1 rounds per sweep.  The rotation of pair
// (p, q) is P with P_pp = P_qq = c, P_pq = s, P_qp = -s (Rutishauser's
// formulas), chosen so that (P^T A P)_pq = 0.  The pairs of a round
// partition the indices, so A' = J^T A J splits into independent 2x2 blocks
// (rows of pair i, columns of pair j): each thread updates whole blocks,
// R_i^T M R_j, and one round costs two barriers.  A rotation is skipped when
// |A_pq| <= n u sqrt(|A_pp A_qq|), u = 2^-52 (or below 1e-18 ||A||_F): below
// that level a rotation only moves rounding noise around.  The solver stops
// after a sweep without rotations.  The rotations accumulate in V (shared
// memory when n <= 112, else the n x n global scratch Vwork).  The padding
// row/column never couples, so the leading n_in x n_in block of V holds the
// eigenvectors.  On exit: vals[i] = A_ii, Vout (n_in x n_in, col-major).
template <bool V_SMEM>
__global__ void __launch_bounds__(512) k_jacobi(const double *__restrict__ Ain, int n_in, int n, double *Vwork,
                                                 double *Vout, double *vals, int max_sweeps, int *sweeps_out) {
    extern __shared__ double S[];
    const int ld = n + 1;
    double *V = V_SMEM ? S + (size_t)n * ld : Vwork;
    __shared__ double cs_[kJacobiMax / 2], sn_[kJacobiMax / 2];
    __shared__ int pp_[kJacobiMax / 2], qq_[kJacobiMax / 2];
    __shared__ double red[32];
    __shared__ int rotated;
    __shared__ double floor_abs;
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int w = tid; w < n * n; w += nt) {
        const int r = w % n, c = w / n;
        S[r + c * ld] = (r < n_in && c < n_in) ? Ain[r + (int64_t)c * n_in] : 0.0;
        V[r + (int64_t)c * n] = (r == c) ? 1.0 : 0.0;
    }
    // ||A||_F (invariant under the rotations) for the absolute skip floor
    double ss = 0.0;
    for (int w = tid; w < n * n; w += nt) {
        const double v = S[(w % n) + (w / n) * ld];
        ss += v * v;
    }
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int i = 0; i < (nt >> 5); ++i) t += red[i];
        floor_abs = 1e-18 * sqrt(t);
        rotated = 0;
    }
    __syncthreads();
    const int half = n / 2;
    const double eps = (double)n * 0x1.0p-52, eps2 = eps * eps;
    int sweep = 0;
    for (; sweep < max_sweeps; ++sweep) {
        for (int r = 0; r < n - 1; ++r) {
            for (int i = tid; i < half; i += nt) {
                const int a = (i == 0) ? 0 : ((i - 1 + r) % (n - 1)) + 1;
                const int b = ((n - 2 - i + r) % (n - 1)) + 1;
                const int p = a < b ? a : b, q = a < b ? b : a;
                const double apq = S[p + q * ld], app = S[p + p * ld], aqq = S[q + q * ld];
                double c = 1.0, s = 0.0;
                if (fabs(apq) > floor_abs && apq * apq > eps2 * fabs(app * aqq)) {
                    // t = sign(tau) / (|tau| + sqrt(1 + tau^2)), tau = (aqq - app) / (2 apq),
                    // written with one square root and one division
                    const double dd = aqq - app, two = 2.0 * apq;
                    const double r = sqrt(fma(dd, dd, two * two));
                    const double t = (dd >= 0.0 ? two : -two) / (fabs(dd) + r);
                    c = rsqrt(fma(t, t, 1.0));
                    s = t * c;
                    rotated = 1;
                }
                cs_[i] = c;
                sn_[i] = s;
                pp_[i] = p;
                qq_[i] = q;
            }
            __syncthreads();
            // Warp w owns the row pairs bi = w, w + nw, ...; lane l owns the
            // column pairs bj = l, l + 32, ... and the rows j = l, l + 32, ...
            // of V, so every rotation parameter is read once into registers.
            {
                const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
                double cj[3], sj[3];
                int uj[3], vj[3];
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    const int bj = lane + 32 * t;
                    const bool in = bj < half;
                    cj[t] = in ? cs_[bj] : 1.0;
                    sj[t] = in ? sn_[bj] : 0.0;
                    uj[t] = in ? pp_[bj] : 0;
                    vj[t] = in ? qq_[bj] : 0;
                }
                for (int bi = wid; bi < half; bi += nw) {
                    const double ci = cs_[bi], si = sn_[bi];
                    const int p = pp_[bi], q = qq_[bi];
#pragma unroll
                    for (int t = 0; t < 3; ++t) {
                        const int bj = lane + 32 * t;
                        if (bj >= half || (si == 0.0 && sj[t] == 0.0)) continue;
                        const int u = uj[t], v = vj[t];
                        const double m00 = S[p + u * ld], m01 = S[p + v * ld];
                        const double m10 = S[q + u * ld], m11 = S[q + v * ld];
                        // rows: [c -s; s c] M
                        const double r00 = ci * m00 - si * m10, r01 = ci * m01 - si * m11;
                        const double r10 = si * m00 + ci * m10, r11 = si * m01 + ci * m11;
                        // columns: R [c s; -s c]
                        double n00 = cj[t] * r00 - sj[t] * r01, n01 = sj[t] * r00 + cj[t] * r01;
                        double n10 = cj[t] * r10 - sj[t] * r11, n11 = sj[t] * r10 + cj[t] * r11;
                        if (bi == bj) {  // the rotated pair itself: zero by construction
                            n01 = 0.0;
                            n10 = 0.0;
                        }
                        S[p + u * ld] = n00;
                        S[p + v * ld] = n01;
                        S[q + u * ld] = n10;
                        S[q + v * ld] = n11;
                    }
                    // V <- V J for the columns of pair bi
                    if (si != 0.0) {
                        for (int j = lane; j < n; j += 32) {
                            const double vx = V[j + (int64_t)p * n], vy = V[j + (int64_t)q * n];
                            V[j + (int64_t)p * n] = ci * vx - si * vy;
                            V[j + (int64_t)q * n] = si * vx + ci * vy;
                        }
                    }
                }
            }
            __syncthreads();
        }
        const bool any = rotated != 0;
        __syncthreads();
        if (tid == 0) rotated = 0;
        if (!any) break;
        __syncthreads();
    }
    __syncthreads();
    for (int i = tid; i < n; i += nt) vals[i] = S[i + i * ld];
    for (int w = tid; w < n_in * n_in; w += nt) Vout[w] = V[(w % n_in) + (int64_t)(w / n_in) * n];
    if (tid == 0 && sweeps_out) *sweeps_out = sweep;
}

// V: n_in x n_in eigenvectors (col-major); Vwork: (n_in+1)^2 doubles of
// global scratch, used when the rotations do not fit in shared memory.
// Threads of the Jacobi CTA (CREST_JACOBI_THREADS, a multiple of 32 in [64, 512]).
static int jacobi_threads() {
    const char *e = getenv("CREST_JACOBI_THREADS");
    int v = e ? atoi(e) : 512;
    v = (v / 32) * 32;
    return v < 64 ? 64 : (v > 512 ? 512 : v);
}

int jacobi(const double *A, int n_in, double *Vwork, double *V, double *vals, int *sweeps, cudaStream_t st,
           int max_sweeps = 40) {
    const int n = n_in + (n_in & 1);
    CREST_REQUIRE(n <= kJacobiMax, CREST_EINVAL, "Jacobi size %d exceeds %d", n, kJacobiMax);
    prof::Scope ps("eig_jacobi", st);
    const int nt = jacobi_threads();
    if (n <= kJacobiSmemV) {
        const size_t smem = sizeof(double) * ((size_t)n * (n + 1) + (size_t)n * n);
        CREST_TRY(ensure_smem_attr((const void *)k_jacobi<true>, (size_t)smem));
        k_jacobi<true><<<1, nt, smem, st>>>(A, n_in, n, nullptr, V, vals, max_sweeps, sweeps);
    } else {
        const size_t smem = sizeof(double) * (size_t)n * (size_t)(n + 1);
        CREST_TRY(ensure_smem_attr((const void *)k_jacobi<false>, (size_t)smem));
        k_jacobi<false><<<1, nt, smem, st>>>(A, n_in, n, Vwork, V, vals, max_sweeps, sweeps);
    }
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

// ------------------------------------------------- order + emit results
// perm = indices of the n_in leading Jacobi values sorted descending
// (ties: lower index first, NaN last); one thread per candidate.
__global__ void k_rank(const double *vals, int n_in, int *perm, double *sorted) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_in) return;
    const double v = vals[i];
    int r = 0;
    for (int j = 0; j < n_in; ++j)
        if (stands_before(vals[j], j, v, i)) ++r;
    perm[r] = i;
    sorted[r] = v;
}

// Column j of out (d x k row-major) = sign * col perm[j] of Vb (d x ldv
// col-major); vals[j] = max(sorted[j], 0).  sign makes the first entry of
// largest magnitude positive (sklearn svd_flip rule, src/kernels.rs:334-345).
__global__ void k_emit(const double *__restrict__ Vb, int64_t d, int64_t ldv, const int *perm,
                       const double *sorted, int64_t k, double *out_vals, double *out_vecs) {
    __shared__ double bv[32];
    __shared__ int bi[32];
    const int64_t j = blockIdx.x;
    const double *col = Vb + (int64_t)perm[j] * ldv;
    double best = -1.0;
    int besti = 0x7fffffff;
    for (int64_t r = threadIdx.x; r < d; r += blockDim.x) {
        const double a = fabs(col[r]);
        if (a > best) {  // rows visited in increasing order per thread
            best = a;
            besti = (int)r;
        }
    }
    for (int o = 16; o; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
        if (ob > best || (ob == best && oi < besti)) {
            best = ob;
            besti = oi;
        }
    }
    if ((threadIdx.x & 31) == 0) {
        bv[threadIdx.x >> 5] = best;
        bi[threadIdx.x >> 5] = besti;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = -1.0;
        int ib = 0x7fffffff;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w)
            if (bv[w] > b || (bv[w] == b && bi[w] < ib)) {
                b = bv[w];
                ib = bi[w];
            }
        bi[0] = ib;
        bv[0] = b;
        out_vals[j] = fmax(sorted[j], 0.0);
    }
    __syncthreads();
    const double sign = (bv[0] > 0.0 && col[bi[0]] < 0.0) ? -1.0 : 1.0;
    for (int64_t r = threadIdx.x; r < d; r += blockDim.x) out_vecs[r * k + j] = col[r] * sign;
}

// --------------------------------------------------------- block kernels
__device__ __forceinline__ uint64_t mix64(uint64_t x) {  // SplitMix64 finaliser (Steele et al. 2014)
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// Columns of d random values in (-1, 1), the rows past d zero.
__global__ void k_random_block(double *V, int64_t d, int64_t ld, int64_t p, uint64_t seed) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ld * p) return;
    const int64_t r = i % ld, c = i / ld;
    V[i] = r < d ? (double)(mix64(seed ^ (uint64_t)(c * d + r)) >> 11) * 0x1.0p-52 - 1.0 : 0.0;
}

// Block reduction helper (sum over the CTA), result valid in every thread.
__device__ double block_sum(double v, double *red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[w];
    return s;
}

// Classical Gram-Schmidt with one re-orthogonalisation pass, one CTA, on
// columns [j0, p) of a column-major d x p block (columns < j0 are already
// orthonormal).  A column whose norm collapses below 1e-10 of its starting
// norm is replaced by a deterministic random vector and processed again.
// Fallback orthonormalisation when Cholesky QR meets a rank-deficient block.
__global__ void __launch_bounds__(1024) k_cgs2(double *Q, int64_t d, int64_t ld, int j0, int p, uint64_t seed) {
    extern __shared__ double sh[];  // r[p] + red[32]
    double *rcoef = sh;
    double *red = sh + p;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    for (int j = j0; j < p; ++j) {
        double *y = Q + (int64_t)j * ld;
        for (int attempt = 0; attempt < 3; ++attempt) {
            double s = 0.0;
            for (int64_t r = tid; r < d; r += nt) s += y[r] * y[r];
            const double n0 = block_sum(s, red);
            for (int pass = 0; pass < 2; ++pass) {
                for (int i = wid; i < j; i += nw) {
                    const double *qi = Q + (int64_t)i * ld;
                    double t = 0.0;
                    for (int64_t r = lane; r < d; r += 32) t += qi[r] * y[r];
                    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                    if (lane == 0) rcoef[i] = t;
                }
                __syncthreads();
                for (int64_t r = tid; r < d; r += nt) {
                    double v = y[r];
                    for (int i = 0; i < j; ++i) v -= rcoef[i] * Q[(int64_t)i * ld + r];
                    y[r] = v;
                }
                __syncthreads();
            }
            s = 0.0;
            for (int64_t r = tid; r < d; r += nt) s += y[r] * y[r];
            const double n1 = block_sum(s, red);
            if (n1 > 1e-20 * n0 && n1 > 0.0) {
                const double inv = 1.0 / sqrt(n1);
                for (int64_t r = tid; r < d; r += nt) y[r] *= inv;
                __syncthreads();
                break;
            }
            for (int64_t r = tid; r < d; r += nt)
                y[r] = (double)(mix64(seed ^ ((uint64_t)(j * 7 + attempt + 1) << 40) ^ (uint64_t)r) >> 11) *
                           0x1.0p-52 -
                       1.0;
            __syncthreads();
        }
    }
}

// Blocks of more than 64 columns (k > 50): Cholesky QR factor for a block Y
// with Gram matrix B = Y^T Y (p x p).  The
// Gram matrix is first equilibrated, B' = D B D with D = diag(B)^-1/2 (column
// scaling leaves the span unchanged and removes the norm disparity a
// Chebyshev filter creates), shifted by shift_coef * ||B'||_2 (bounded by
// trace(B') = p), and factored B' = L L^T.  Rinv = D L^-T (upper triangular),
// so Y Rinv has orthonormal columns.  One CTA; L, L^-1 and a 16-row panel in
// shared memory.  Both the factorisation and the inverse go by 16 x 16
// blocks: the diagonal block by one warp, the panel and the trailing update
// by the whole block, three barriers per block column.  *fail = 1 (and
// Rinv = I, leaving Y unchanged) when a column is zero or a pivot is not
// positive.
constexpr int kCholNb = 16;

__global__ void __launch_bounds__(512) k_chol_inv(const double *__restrict__ B, int p, double shift_coef,
                                                  double *__restrict__ Rinv, int *fail) {
    extern __shared__ double sm[];
    double *L = sm;                     // p x p, col-major (lower triangle used)
    double *X = sm + (size_t)p * p;     // L^-1, col-major
    double *T = X + (size_t)p * p;      // kCholNb x p panel
    __shared__ double dsc[kJacobiMax];
    __shared__ int bad;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) bad = 0;
    __syncthreads();
    for (int i = tid; i < p; i += nt) {
        const double b = B[i + (int64_t)i * p];
        if (!(b > 0.0)) bad = 1;
        dsc[i] = b > 0.0 ? 1.0 / sqrt(b) : 1.0;
    }
    __syncthreads();
    const double shift = shift_coef * (double)p;
    for (int w = tid; w < p * p; w += nt) {
        const int r = w % p, c = w / p;
        L[w] = (r == c) ? 1.0 + shift : B[w] * dsc[r] * dsc[c];
        X[w] = 0.0;
    }
    __syncthreads();
    // ---- B' = L L^T, right-looking by block columns
    for (int k0 = 0; k0 < p; k0 += kCholNb) {
        const int kb = min(kCholNb, p - k0);
        if (wid == 0) {  // diagonal block, unblocked, lane i owns row k0 + i
            for (int j = 0; j < kb; ++j) {
                const int jj = k0 + j;
                double piv = L[jj + jj * p];
                if (!(piv > 0.0)) {
                    if (lane == 0) bad = 1;
                    piv = 1.0;
                }
                const double r = sqrt(piv);
                __syncwarp();
                if (lane == j) L[jj + jj * p] = r;
                if (lane > j && lane < kb) L[k0 + lane + jj * p] /= r;
                __syncwarp();
                if (lane > j && lane < kb) {
                    const int i = k0 + lane;
                    const double lij = L[i + jj * p];
                    for (int c = j + 1; c <= lane; ++c) L[i + (k0 + c) * p] -= lij * L[k0 + c + jj * p];
                }
                __syncwarp();
            }
        }
        __syncthreads();
        // panel below the diagonal block: L21 = A21 L11^-T, one row per thread
        for (int i = k0 + kb + tid; i < p; i += nt) {
            for (int j = 0; j < kb; ++j) {
                double v = L[i + (k0 + j) * p];
                for (int t = 0; t < j; ++t) v -= L[i + (k0 + t) * p] * L[k0 + j + (k0 + t) * p];
                L[i + (k0 + j) * p] = v / L[k0 + j + (k0 + j) * p];
            }
        }
        __syncthreads();
        // trailing lower triangle: A22 -= L21 L21^T
        const int r0 = k0 + kb, rem = p - r0;
        for (int w = tid; w < rem * rem; w += nt) {
            const int i = r0 + w % rem, j = r0 + w / rem;
            if (i < j) continue;
            double v = L[i + j * p];
            for (int t = 0; t < kb; ++t) v -= L[i + (k0 + t) * p] * L[j + (k0 + t) * p];
            L[i + j * p] = v;
        }
        __syncthreads();
    }
    // ---- X = L^-1 by block rows: X_II = L_II^-1, X_IC = -X_II sum_K L_IK X_KC
    for (int i0 = 0; i0 < p; i0 += kCholNb) {
        const int ib = min(kCholNb, p - i0);
        if (wid == 0 && lane < ib) {  // diagonal block, lane c owns column i0 + c
            const int c = lane;
            for (int i = c; i < ib; ++i) {
                double v = (i == c) ? 1.0 : 0.0;
                for (int t = c; t < i; ++t) v -= L[i0 + i + (i0 + t) * p] * X[i0 + t + (i0 + c) * p];
                X[i0 + i + (i0 + c) * p] = v / L[i0 + i + (i0 + i) * p];
            }
        }
        for (int w = tid; w < ib * i0; w += nt) {  // T[ii][c] = sum_{t=c}^{i0-1} L[i0+ii][t] X[t][c]
            const int ii = w % ib, c = w / ib;
            double v = 0.0;
            for (int t = c; t < i0; ++t) v += L[i0 + ii + t * p] * X[t + c * p];
            T[ii + c * kCholNb] = v;
        }
        __syncthreads();
        for (int w = tid; w < ib * i0; w += nt) {
            const int ii = w % ib, c = w / ib;
            double v = 0.0;
            for (int t = 0; t <= ii; ++t) v += X[i0 + ii + (i0 + t) * p] * T[t + c * kCholNb];
            X[i0 + ii + c * p] = -v;
        }
        __syncthreads();
    }
    // Rinv = D (L^-1)^T, or the identity (Y left as it is) when the factor failed
    for (int w = tid; w < p * p; w += nt) {
        const int r = w % p, c = w / p;
        Rinv[w] = bad ? (r == c ? 1.0 : 0.0) : dsc[r] * X[c + r * p];
    }
    if (tid == 0 && bad) atomicOr(fail, 1);
}

// r_i = || W_i - theta_i V_i || for the given columns.
__global__ void k_residual(const double *__restrict__ W, const double *__restrict__ V, const double *theta,
                           int64_t d, double *res) {
    __shared__ double red[32];
    const int i = blockIdx.x;
    const double th = theta[i];
    double s = 0.0;
    for (int64_t r = threadIdx.x; r < d; r += blockDim.x) {
        const double e = W[(int64_t)i * d + r] - th * V[(int64_t)i * d + r];
        s += e * e;
    }
    const double t = block_sum(s, red);
    if (threadIdx.x == 0) res[i] = sqrt(t);
}

// Permute the Ritz basis: dst[:, j] = src[:, perm[j]] for j < p.
__global__ void k_permute_cols(const double *src, double *dst, int64_t d, const int *perm, int p) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= d * p) return;
    const int64_t r = idx % d, j = idx / d;
    dst[idx] = src[(int64_t)perm[j] * d + r];
}

// Z[:, j] = (theta[j] - t) V[:, j] for j < nl (d x nl, col-major).
__global__ void k_scale_cols(const double *V, const double *theta, double t, int64_t d, int nl, double *Z) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= d * nl) return;
    Z[idx] = (theta[idx / d] - t) * V[idx];
}

// Symmetrise a p x p col-major matrix in place: H = (H + H^T)/2.
__global__ void k_symmetrise(double *H, int p) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= p * p) return;
    const int r = idx % p, c = idx / p;
    if (r < c) {
        const double v = 0.5 * (H[r + c * p] + H[c + r * p]);
        H[r + c * p] = v;
        H[c + r * p] = v;
    }
}

// y = C x for a symmetric d x d C (column-major; reads column i for y_i).
__global__ void k_symv(const double *__restrict__ C, int64_t d, int64_t ld, const double *__restrict__ x,
                       double *__restrict__ y) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= d) return;
    const double *col = C + i * ld;
    double s = 0.0;
    for (int64_t j = lane; j < d; j += 32) s += col[j] * x[j];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) y[i] = s;
}

// One Lanczos step after w = C v_j: alpha_j = v_j.w, w -= alpha v_j + beta v_{j-1},
// full re-orthogonalisation (twice) against V[:, 0..j], beta_j = |w|,
// v_{j+1} = w / beta_j.  One CTA; V is d x (kLanczos + 1) col-major.
__global__ void __launch_bounds__(1024) k_lanczos_step(double *V, int64_t d, int j, double *w, double *ab) {
    __shared__ double red[32];
    __shared__ double coef[kLanczos + 1];
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    const double *vj = V + (int64_t)j * d;
    double s = 0.0;
    for (int64_t r = tid; r < d; r += nt) s += vj[r] * w[r];
    const double alpha = block_sum(s, red);
    const double beta_prev = j > 0 ? ab[kLanczos + j - 1] : 0.0;
    for (int64_t r = tid; r < d; r += nt) {
        double v = w[r] - alpha * vj[r];
        if (j > 0) v -= beta_prev * V[(int64_t)(j - 1) * d + r];
        w[r] = v;
    }
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
        for (int i = wid; i <= j; i += nw) {
            const double *qi = V + (int64_t)i * d;
            double t = 0.0;
            for (int64_t r = lane; r < d; r += 32) t += qi[r] * w[r];
            for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) coef[i] = t;
        }
        __syncthreads();
        for (int64_t r = tid; r < d; r += nt) {
            double v = w[r];
            for (int i = 0; i <= j; ++i) v -= coef[i] * V[(int64_t)i * d + r];
            w[r] = v;
        }
        __syncthreads();
    }
    s = 0.0;
    for (int64_t r = tid; r < d; r += nt) s += w[r] * w[r];
    const double beta = sqrt(block_sum(s, red));
    double *vn = V + (int64_t)(j + 1) * d;
    const double inv = beta > 0.0 ? 1.0 / beta : 0.0;
    for (int64_t r = tid; r < d; r += nt) vn[r] = w[r] * inv;
    if (tid == 0) {
        ab[j] = alpha;
        ab[kLanczos + j] = beta;
    }
}

// All L Lanczos steps in one cooperative launch (one CTA per SM).  CTA b
// keeps rows [r0, r1) of C in shared memory as FP32 (the run only brackets
// the spectrum: FP32 products move the extreme Ritz values by ~1e-7
// relative, far inside the guard the filter interval keeps) and the whole
// current vector in FP64; the previous one is in registers, each thread
// holding the elements it updates, so that shared memory takes matrices of up
// to 2,764 rows on 148 SMs (2,638 with both vectors there; larger ones take a
// launch per step, 1.34 ms instead of 0.34 at 2,700 rows).  A step is one grid barrier: every
// CTA publishes its rows of C v_j, then each reads the whole product and
// forms alpha_j, v_{j+1} and beta_j for itself, in the same order everywhere.
// The basis is not re-orthogonalised: that lets copies of converged extreme
// values appear but leaves the extreme Ritz values and their residual bounds
// |beta_L s_L| valid (Paige 1976), which is all the filter asks for.  (With
// two Gram-Schmidt passes a step took three barriers and the exchange of
// every CTA's partial coefficients: 612 us for 32 steps at d = 2000 against
// 250.)  Each barrier wait is bounded (about one second of %globaltimer); on
// expiry the CTA raises *err and every later barrier is skipped, so the
// launch always ends.
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid barrier on counters that only grow (zeroed before the launch).  CTAs
// arrive on the counter of their group of 16 (one 128-byte line each, so
// arrivals do not all queue on one address); the last arrival of a group
// adds one to the top counter, and barrier number `phase` is passed once the
// top counter reaches phase x groups.
constexpr int kBarGroup = 16;

__device__ void grid_barrier(unsigned *bar, unsigned &phase, unsigned nblk, int *err) {
    __syncthreads();
    ++phase;
    if (threadIdx.x == 0) {
        volatile int *e = err;
        if (!*e) {
            const unsigned n_groups = (nblk + kBarGroup - 1) / kBarGroup, g = blockIdx.x / kBarGroup;
            const unsigned in_group = min((unsigned)kBarGroup, nblk - g * kBarGroup);
            unsigned *top = bar, *mine = bar + 32 * (1 + g);
            __threadfence();
            if (atomicAdd(mine, 1u) == phase * in_group - 1) atomicAdd(top, 1u);
            const unsigned target = phase * n_groups;
            const unsigned long long t0 = gtimer();
            unsigned spins = 0;
            for (;;) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(top) : "memory");
                if (v >= target) break;
                if (*e || ((++spins & 63u) == 0 && gtimer() - t0 > 1000000000ull)) {
                    atomicExch(err, 1);
                    break;
                }
            }
        }
        __threadfence();
    }
    __syncthreads();
}

struct LanczosArgs {
    const double *C;
    int64_t d, ld;
    int L;
    int rows;          // rows per CTA (the last CTAs may own fewer)
    const double *z0;  // the start vector (any length)
    double *w;         // 2 x d: C v_j, published each step, in turn
    double *ab;        // alpha [0, kLanczos), beta [kLanczos, 2 kLanczos)
    unsigned *bar;
    int *err;
};

constexpr int kLzThreads = 512, kLzHeld = 6;  // elements of the previous vector per thread, at most

size_t lanczos_smem(int64_t d, int rows) { return sizeof(float) * (size_t)rows * d + sizeof(double) * (size_t)d; }

__global__ void __launch_bounds__(kLzThreads) k_lanczos(LanczosArgs a) {
    extern __shared__ __align__(16) unsigned char lz_smem[];
    __shared__ double red[32];
    constexpr int nt = kLzThreads;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    const int64_t d = a.d;
    const int64_t r0 = min(d, (int64_t)blockIdx.x * a.rows), r1 = min(d, r0 + a.rows);
    const int R = (int)(r1 - r0);
    double *v = reinterpret_cast<double *>(lz_smem);  // v_j
    float *cs = reinterpret_cast<float *>(v + d);      // rows x d: owned rows of C
    double vp[kLzHeld];                                // v_{j-1}: elements tid, tid + nt, ..
    for (int rr = 0; rr < R; ++rr)
        for (int64_t e = tid; e < d; e += nt) cs[rr * d + e] = (float)a.C[(r0 + rr) * a.ld + e];
    double s = 0.0;
    for (int64_t e = tid; e < d; e += nt) {
        v[e] = a.z0[e];
        s += v[e] * v[e];
    }
#pragma unroll
    for (int i = 0; i < kLzHeld; ++i) vp[i] = 0.0;
    double nrm = sqrt(block_sum(s, red));
    for (int64_t e = tid; e < d; e += nt) v[e] *= nrm > 0.0 ? 1.0 / nrm : 0.0;
    double beta = 0.0;
    unsigned phase = 0;
    __syncthreads();
    for (int j = 0; j < a.L; ++j) {
        double *w = a.w + (j & 1) * d;  // step j - 1's readers have passed this step's barrier before it is reused
        for (int rr = wid; rr < R; rr += nw) {
            const float *row = cs + (size_t)rr * d;
            double t0 = 0.0, t1 = 0.0;
            int64_t i = lane;
            for (; i + 32 < d; i += 64) {
                t0 += (double)row[i] * v[i];
                t1 += (double)row[i + 32] * v[i + 32];
            }
            if (i < d) t0 += (double)row[i] * v[i];
            double t = t0 + t1;
            for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) w[r0 + rr] = t;
        }
        grid_barrier(a.bar, phase, gridDim.x, a.err);
        s = 0.0;
        for (int64_t e = tid; e < d; e += nt) s += v[e] * __ldcg(w + e);
        const double alpha = block_sum(s, red);
        s = 0.0;
#pragma unroll
        for (int i = 0; i < kLzHeld; ++i) {
            const int64_t e = tid + i * nt;
            if (e >= d) continue;
            const double z = __ldcg(w + e) - alpha * v[e] - beta * vp[i];
            vp[i] = z;
            s += z * z;
        }
        beta = sqrt(block_sum(s, red));
        const double inv = beta > 0.0 ? 1.0 / beta : 0.0;
#pragma unroll
        for (int i = 0; i < kLzHeld; ++i) {  // v_j and v_{j+1} change places
            const int64_t e = tid + i * nt;
            if (e >= d) continue;
            const double t = v[e];
            v[e] = vp[i] * inv;
            vp[i] = t;
        }
        if (blockIdx.x == 0 && tid == 0) {
            a.ab[j] = alpha;
            a.ab[kLanczos + j] = beta;
        }
        __syncthreads();
    }
}

// Extreme eigenvalues of the Lanczos tridiagonal (alpha, beta, L) with their
// residual bounds: bisection on the Sturm count, and the last component of
// the eigenvector from the recurrence run up from the last row, whose terms
// keep one sign at an extreme eigenvalue (it lies outside the spectrum of
// every trailing block).
struct Extremes {
    double lo, hi, res_lo, res_hi;
};
Extremes tridiag_extremes(const double *alpha, const double *beta, int L) {
    double scale = 0.0;
    for (int i = 0; i < L; ++i) scale = std::max(scale, fabs(alpha[i]) + fabs(beta[i]));
    for (int i = 0; i + 1 < L; ++i)  // an invariant subspace ends the run early
        if (!(beta[i] > 1e-14 * scale)) L = i + 1;
    const double tiny = std::max(1e-300, 1e-32 * scale);
    auto below = [&](double x) {  // eigenvalues < x
        int n = 0;
        double q = 1.0;
        for (int i = 0; i < L; ++i) {
            q = alpha[i] - x - (i ? beta[i - 1] * beta[i - 1] / q : 0.0);
            if (fabs(q) < tiny) q = -tiny;
            n += q < 0.0;
        }
        return n;
    };
    auto find = [&](int rank) {  // eigenvalue number `rank` from below
        double lo = -2.0 * scale, hi = 2.0 * scale;
        for (int it = 0; it < 80 && lo < hi; ++it) {
            const double mid = 0.5 * (lo + hi);
            if (mid == lo || mid == hi) break;
            (below(mid) > rank ? hi : lo) = mid;
        }
        return 0.5 * (lo + hi);
    };
    auto bound = [&](double th) {
        double x = 1.0, nx = 0.0, sum = 1.0;  // x_i and x_{i+1}, from the last row up
        for (int i = L - 1; i > 0; --i) {
            const double up = ((th - alpha[i]) * x - (i < L - 1 ? beta[i] * nx : 0.0)) / beta[i - 1];
            nx = x;
            x = up;
            sum += x * x;
            if (sum > 1e200) return 0.0;  // the last component is below any rounding
        }
        return fabs(beta[L - 1]) / sqrt(sum);
    };
    Extremes e;
    e.lo = find(0);
    e.hi = find(L - 1);
    e.res_lo = bound(e.lo);
    e.res_hi = bound(e.hi);
    return e;
}

struct EigWork {
    DevBuf C, V[2], W[2], Y, S, H, Q, rot, part, out, vals, sorted, perm, lz, lw, lbar, lab, fail;
    HostBuf h;
    GemmWs g;
};

// The cooperative Lanczos launch; CREST_ERUNTIME (nothing launched) when the
// device cannot hold one CTA per SM of it.
int lanczos_coop(EigWork &w, const double *C, int64_t d, int64_t ld, int L, cudaStream_t st) {
    static const bool off = [] {
        const char *e = getenv("CREST_EIG_COOP");
        return e && e[0] == '0';
    }();
    if (off) return CREST_ERUNTIME;
    const int nb = (int)std::min<int64_t>(device_sms(), std::max<int64_t>(1, d / 4));
    const int rows = (int)ceil_div(d, nb);
    const size_t smem = lanczos_smem(d, rows);
    if (d > kLzThreads * kLzHeld || smem > (size_t)kMaxSmem || ensure_smem_attr((const void *)k_lanczos, smem) != CREST_OK) {
        (void)cudaGetLastError();
        return CREST_ERUNTIME;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lanczos, kLzThreads, smem) != cudaSuccess || per_sm < 1) {
        (void)cudaGetLastError();
        return CREST_ERUNTIME;
    }
    // the top counter, then one 128-byte line per group of CTAs
    const size_t bar_bytes = sizeof(unsigned) * 32 * (1 + (size_t)ceil_div(nb, kBarGroup));
    CREST_TRY(w.lbar.ensure(bar_bytes));
    CREST_CUDA_TRY(cudaMemsetAsync(w.lbar.ptr, 0, bar_bytes, st));
    CREST_CUDA_TRY(cudaMemsetAsync(w.fail.ptr, 0, sizeof(int), st));
    LanczosArgs a{C, d, ld, L, rows, w.lz.as<double>(), w.lw.as<double>(), w.lab.as<double>(), w.lbar.as<unsigned>(),
                  w.fail.as<int>()};
    void *args[] = {&a};
    prof::Scope ps("eig_lanczos", st);
    if (cudaLaunchCooperativeKernel((const void *)k_lanczos, dim3(nb), dim3(kLzThreads), args, smem, st) != cudaSuccess) {
        (void)cudaGetLastError();
        return CREST_ERUNTIME;
    }
    return CREST_OK;
}

// The block of the solver: p columns of D rows (ld D), the locked ones first.
// cur holds it; other has the same locked columns, and its remaining columns
// are scratch, so a step that cannot work in place writes there and swaps.
struct Block {
    int D, p;
    double *cur, *other;
    void swap() { std::swap(cur, other); }
};

// One Cholesky-QR pass (Fukaya et al. 2020) on columns [j0, p) of b.cur,
// against its first j0 columns (orthonormal already) and among themselves,
// into b.other; a failed factor copies them unchanged.
int ortho_pass(EigWork &w, const Block &b, int j0, bool shifted, cudaStream_t st) {
    const int D = b.D, p = b.p, q = p - j0;
    const double *Ya = b.cur + (int64_t)j0 * D;
    double *To = b.other + (int64_t)j0 * D;
    double *S = w.S.as<double>(), *R = w.Q.as<double>();
    EigOut *out = w.out.as<EigOut>();
    // shift = 11 (d q + q (q + 1)) u ||B'||_2 on the first pass of the shifted form
    const double shift_coef = shifted ? 11.0 * ((double)D * q + (double)q * (q + 1)) * 0x1.0p-53 : 0.0;
    if (p <= kBlk) {
        CREST_TRY(gemm(Gemm{p, q, D, b.cur, D, 1, Ya, D, S, p, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st));
        {
            prof::Scope ps("eig_cholqr", st);
            k_ortho_coef<<<1, 256, 0, st>>>(S, p, j0, shift_coef, R, out);
        }
        CREST_CUDA_TRY(cudaGetLastError());
        return gemm(Gemm{D, q, p, b.cur, D, 0, R, p, To, D, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st);
    }
    double *Yw = w.Y.as<double>();
    CREST_CUDA_TRY(cudaMemcpyAsync(Yw, Ya, sizeof(double) * (size_t)D * q, cudaMemcpyDeviceToDevice, st));
    if (j0 > 0) {
        CREST_TRY(gemm(Gemm{j0, q, D, b.cur, D, 1, Yw, D, S, j0, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st));
        CREST_TRY(gemm(Gemm{D, q, j0, b.cur, D, 0, S, j0, Yw, D, -1.0, Yw, 1.0, nullptr, 0.0}, w.g, st));
    }
    CREST_TRY(gemm(Gemm{q, q, D, Yw, D, 1, Yw, D, S, q, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st));
    {
        prof::Scope ps("eig_cholqr", st);
        const size_t csmem = sizeof(double) * (2 * (size_t)q * q + (size_t)kCholNb * q);
        CREST_TRY(ensure_smem_attr((const void *)k_chol_inv, csmem));
        k_chol_inv<<<1, 512, csmem, st>>>(S, q, shift_coef, R, &out->fail);
    }
    CREST_CUDA_TRY(cudaGetLastError());
    return gemm(Gemm{D, q, q, Yw, D, 0, R, q, To, D, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st);
}

// Orthonormalise columns [j0, p) of b.cur: a pass (shifted for a filtered
// block, whose columns may be nearly dependent) and an unshifted one, which
// leaves them orthonormal to working precision unless its factor reports
// otherwise (out->fail; the caller reads it with the next Ritz values and
// calls repair()).  The wide form, whose factor does not report, takes a
// third pass after a shifted first one, through the scratch columns.
int orthonormalise(EigWork &w, Block &b, int j0, bool shifted, cudaStream_t st) {
    const int passes = shifted && b.p > kBlk ? 3 : 2;
    for (int pass = 0; pass < passes; ++pass) {
        CREST_TRY(ortho_pass(w, b, j0, shifted && pass == 0, st));
        b.swap();
    }
    return CREST_OK;
}

// After a reported failure: Gram-Schmidt with random replacements for a
// rank-deficient block (fail bit 0), else two more unshifted passes.
int repair(EigWork &w, Block &b, int64_t d, int j0, int fail, uint64_t seed, cudaStream_t st) {
    CREST_CUDA_TRY(cudaMemsetAsync(&w.out.as<EigOut>()->fail, 0, sizeof(int), st));
    if (!(fail & 1)) return orthonormalise(w, b, j0, false, st);
    prof::Scope ps("eig_cgs2", st);
    k_cgs2<<<1, 1024, sizeof(double) * (size_t)(b.p + 32), st>>>(b.cur, d, b.D, j0, b.p, seed);
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

// Rayleigh-Ritz on columns [j0, p): w = C v, H = v^T w, its rotations applied
// to both, Ritz pairs in descending order with their residuals in *out.
int rayleigh_ritz(EigWork &w, Block &v, Block &cv, const double *C, int j0, int max_sweeps, cudaStream_t st) {
    const int D = v.D, p = v.p, q = p - j0;
    double *Va = v.cur + (int64_t)j0 * D, *Wa = cv.cur + (int64_t)j0 * D;
    double *Vo = v.other + (int64_t)j0 * D, *Wo = cv.other + (int64_t)j0 * D;
    double *H = w.H.as<double>();
    EigOut *out = w.out.as<EigOut>();
    CREST_TRY(gemm(Gemm{D, q, D, C, D, 1, Va, D, Wa, D, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st));
    CREST_TRY(gemm(Gemm{q, q, D, Va, D, 1, Wa, D, H, q, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st));
    int *perm = w.perm.as<int>();
    if (p <= kBlk) {
        {
            prof::Scope ps("eig_jacobi", st);
            k_rr<<<1, kRrThreads, 0, st>>>(H, q, q, max_sweeps, w.rot.as<double2>(), out->theta + j0, perm, out);
        }
        CREST_CUDA_TRY(cudaGetLastError());
        prof::Scope ps("eig_rotate", st);
        k_apply_rot<<<(unsigned)(D / kRotRows), 256, 0, st>>>(Va, Wa, Vo, Wo, D, q, w.rot.as<double2>(),
                                                             out->theta + j0, perm, w.part.as<double>(), out->res + j0,
                                                             out);
        CREST_CUDA_TRY(cudaGetLastError());
    } else {
        double *Q = w.Q.as<double>(), *jvals = w.vals.as<double>();
        k_symmetrise<<<(unsigned)ceil_div(q * q, 256), 256, 0, st>>>(H, q);
        CREST_CUDA_TRY(cudaGetLastError());
        CREST_TRY(jacobi(H, q, w.Y.as<double>(), Q, jvals, nullptr, st, max_sweeps));
        k_rank<<<(unsigned)ceil_div(q, 128), 128, 0, st>>>(jvals, q, perm, out->theta + j0);
        k_permute_cols<<<(unsigned)ceil_div(q * q, 256), 256, 0, st>>>(Q, H, q, perm, q);
        CREST_CUDA_TRY(cudaGetLastError());
        CREST_TRY(gemm(Gemm{D, q, q, Va, D, 0, H, q, Vo, D, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st));
        CREST_TRY(gemm(Gemm{D, q, q, Wa, D, 0, H, q, Wo, D, 1.0, nullptr, 0.0, nullptr, 0.0}, w.g, st));
        k_residual<<<(unsigned)q, 256, 0, st>>>(Wo, Vo, out->theta + j0, D, out->res + j0);
        CREST_CUDA_TRY(cudaGetLastError());
    }
    v.swap();
    cv.swap();
    return CREST_OK;
}

}  // namespace

int eig_topk(const double *G, const double *colsum, int64_t d, int64_t n, int64_t k, double *out_vals,
             double *out_vecs, double *out_total, EigStats *stats, cudaStream_t st) {
    CREST_REQUIRE(d >= 1 && n >= 2, CREST_ERUNTIME, "need at least 2 cells and 1 gene");
    CREST_REQUIRE(k >= 0 && k <= d, CREST_EINVAL, "k=%lld must be in [0, d=%lld]", (long long)k, (long long)d);
    int dev = 0;
    CREST_CUDA_TRY(cudaGetDevice(&dev));
    CREST_REQUIRE(dev >= 0 && dev < 64, CREST_ERUNTIME, "device index %d out of range", dev);
    static thread_local EigWork ws[64];  // per host thread and device
    EigWork &w = ws[dev];
    const double nf = (double)n;
    const bool whole = d <= kJacobiMax;  // whole-matrix Jacobi: no padding
    const int64_t ld = whole ? d : round_up(d, kRotRows);
    CREST_TRY(w.C.ensure(sizeof(double) * (size_t)(ld * ld)));
    double *C = w.C.as<double>();
    {
        prof::Scope ps("eig_centre", st);
        k_centre<<<(unsigned)ceil_div(ld * ld, 256), 256, 0, st>>>(G, colsum, d, ld, nf, C);
    }
    CREST_CUDA_TRY(cudaGetLastError());
    k_trace<<<1, 1024, 0, st>>>(C, d, ld, out_total);
    CREST_CUDA_TRY(cudaGetLastError());
    if (stats) *stats = EigStats{0, 1, 0.0};
    if (k == 0) return CREST_OK;

    CREST_TRY(w.perm.ensure(sizeof(int) * 512));
    CREST_TRY(w.sorted.ensure(sizeof(double) * 512));
    CREST_TRY(w.vals.ensure(sizeof(double) * 512));
    CREST_TRY(w.fail.ensure(sizeof(int) * 4));
    int *perm = w.perm.as<int>();
    double *sorted = w.sorted.as<double>();
    double *jvals = w.vals.as<double>();

    if (whole) {
        const int nn = (int)(d + (d & 1));
        CREST_TRY(w.Q.ensure(sizeof(double) * (size_t)nn * nn));
        CREST_TRY(w.Y.ensure(sizeof(double) * (size_t)nn * nn));
        CREST_TRY(jacobi(C, (int)d, w.Y.as<double>(), w.Q.as<double>(), jvals, w.perm.as<int>() + 256, st));
        k_rank<<<(unsigned)ceil_div(d, 128), 128, 0, st>>>(jvals, (int)d, perm, sorted);
        CREST_CUDA_TRY(cudaGetLastError());
        k_emit<<<(unsigned)k, 256, 0, st>>>(w.Q.as<double>(), d, d, perm, sorted, k, out_vals, out_vecs);
        CREST_CUDA_TRY(cudaGetLastError());
        if (stats) {
            int sweeps = 0;
            CREST_CUDA_TRY(cudaMemcpyAsync(&sweeps, w.perm.as<int>() + 256, sizeof(int), cudaMemcpyDeviceToHost, st));
            CREST_CUDA_TRY(cudaStreamSynchronize(st));
            stats->iters = sweeps;
        }
        return CREST_OK;
    }

    int p = (int)round_up(k + 14, 16);
    if (p > kJacobiSmemV) p = kJacobiSmemV;
    if (p > d) p = (int)d;
    CREST_REQUIRE(k <= p - 8, CREST_EINVAL, "n_comps=%lld too large for the block eigensolver (max %d)",
                  (long long)k, kJacobiSmemV - 8);
    const int D = (int)ld;
    const size_t blk = sizeof(double) * (size_t)D * (size_t)p;
    for (int i = 0; i < 2; ++i) {
        CREST_TRY(w.V[i].ensure(blk));
        CREST_TRY(w.W[i].ensure(blk));
    }
    CREST_TRY(w.Y.ensure(blk));
    CREST_TRY(w.H.ensure(sizeof(double) * (size_t)p * p));
    CREST_TRY(w.Q.ensure(sizeof(double) * (size_t)p * p));
    CREST_TRY(w.S.ensure(sizeof(double) * (size_t)p * p));
    constexpr int kSweeps = 40;
    if (p <= kBlk) {
        CREST_TRY(w.rot.ensure(sizeof(double2) * (size_t)kSweeps * (kBlk - 1) * 32));
        CREST_TRY(w.part.ensure(sizeof(double) * (size_t)(D / kRotRows) * kBlk));
    }
    CREST_TRY(w.out.ensure(sizeof(EigOut)));
    CREST_TRY(w.h.ensure(sizeof(EigOut)));
    CREST_TRY(w.lz.ensure(sizeof(double) * (size_t)d * (kLanczos + 1)));
    CREST_TRY(w.lw.ensure(sizeof(double) * 2 * (size_t)d));
    CREST_TRY(w.lab.ensure(sizeof(double) * 2 * kLanczos));
    EigOut *out = w.out.as<EigOut>();
    const EigOut &ho = *w.h.as<EigOut>();
    CREST_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(EigOut), st));

    // ---- spectrum bounds by Lanczos
    double lam_lo, lam_hi;
    {
        double *LZ = w.lz.as<double>(), *lw = w.lw.as<double>(), *lab = w.lab.as<double>();
        k_random_block<<<(unsigned)ceil_div(d, 256), 256, 0, st>>>(LZ, d, d, 1, 0x452821e638d01377ull);
        CREST_CUDA_TRY(cudaGetLastError());
        const int L = (int)std::min<int64_t>(kLanczos, d - 1);
        CREST_CUDA_TRY(cudaMemsetAsync(w.fail.ptr, 0, sizeof(int), st));
        if (lanczos_coop(w, C, d, ld, L, st) != CREST_OK) {  // one launch per step, re-orthogonalised
            prof::Scope ps("eig_lanczos_steps", st);
            k_cgs2<<<1, 1024, sizeof(double) * 64, st>>>(LZ, d, d, 0, 1, 1);
            for (int j = 0; j < L; ++j) {
                k_symv<<<(unsigned)ceil_div(d * 32, 256), 256, 0, st>>>(C, d, ld, LZ + (int64_t)j * d, lw);
                k_lanczos_step<<<1, 1024, 0, st>>>(LZ, d, j, lw, lab);
            }
        }
        CREST_CUDA_TRY(cudaGetLastError());
        double hab[2 * kLanczos];
        int lz_err = 0;
        CREST_CUDA_TRY(cudaMemcpyAsync(hab, lab, sizeof hab, cudaMemcpyDeviceToHost, st));
        CREST_CUDA_TRY(cudaMemcpyAsync(&lz_err, w.fail.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
        CREST_CUDA_TRY(cudaStreamSynchronize(st));
        CREST_REQUIRE(!lz_err, CREST_ERUNTIME, "Lanczos grid barrier timed out");
        const Extremes ex = tridiag_extremes(hab, hab + kLanczos, L);
        lam_hi = ex.hi + ex.res_hi;
        // a guard below the smallest Ritz value: eigenvalues a little below
        // the damped interval only slow convergence, they cannot be chosen
        lam_lo = ex.lo - ex.res_lo - 1e-3 * (ex.hi - ex.lo);
        if (lam_lo < 0.0) lam_lo = 0.0 - 1e-12 * fabs(lam_hi);
    }
    Block v{D, p, w.V[0].as<double>(), w.V[1].as<double>()}, cv{D, p, w.W[0].as<double>(), w.W[1].as<double>()};
    k_random_block<<<(unsigned)ceil_div((int64_t)D * p, 256), 256, 0, st>>>(v.cur, d, D, p, 0x243f6a8885a308d3ull);
    CREST_CUDA_TRY(cudaGetLastError());
    if (!(lam_hi > 0.0)) {
        // zero covariance: every eigenvalue is 0; any orthonormal basis will do
        k_cgs2<<<1, 1024, sizeof(double) * (size_t)(p + 32), st>>>(v.cur, d, D, 0, p, 3);
        std::vector<int> hp(k);
        std::vector<double> hz(k, 0.0);
        for (int64_t i = 0; i < k; ++i) hp[i] = (int)i;
        CREST_CUDA_TRY(cudaMemcpyAsync(perm, hp.data(), sizeof(int) * k, cudaMemcpyHostToDevice, st));
        CREST_CUDA_TRY(cudaMemcpyAsync(sorted, hz.data(), sizeof(double) * k, cudaMemcpyHostToDevice, st));
        k_emit<<<(unsigned)k, 256, 0, st>>>(v.cur, d, D, perm, sorted, k, out_vals, out_vecs);
        CREST_CUDA_TRY(cudaGetLastError());
        CREST_CUDA_TRY(cudaStreamSynchronize(st));
        return CREST_OK;
    }

    // ---- start block
    CREST_TRY(orthonormalise(w, v, 0, false, st));

    const double tol = 1e-11;
    const int max_outer = 60;
    int locked = 0, it = 0;
    double res_max = INFINITY;
    bool converged = false;
    for (; it < max_outer; ++it) {
        // While the wanted residuals are far from converged the Ritz vectors
        // only have to span the block (the filter acts on the subspace), so
        // two sweeps stand in for the full diagonalisation; the Ritz values
        // (diagonal of the partly rotated H) only set the filter interval.
        CREST_TRY(rayleigh_ritz(w, v, cv, C, locked, res_max > 1e-5 ? 2 : kSweeps, st));
        CREST_CUDA_TRY(cudaMemcpyAsync(w.h.ptr, out, sizeof(EigOut), cudaMemcpyDeviceToHost, st));
        CREST_CUDA_TRY(cudaStreamSynchronize(st));
        if (ho.fail) {  // the block was not orthonormal: mend it and take the step again
            CREST_TRY(repair(w, v, d, locked, ho.fail, 1000 + it, st));
            continue;
        }
        const double *theta = ho.theta, *hres = ho.res;
        const double scale_ref = fmax(fabs(theta[0]), 1e-300);
        // lock the leading converged pairs (in order) and deflate them: their
        // eigenvalues move to lam_lo, the edge of every damped interval, so
        // the filter never amplifies what leaks back into the active block
        const int l0 = locked;
        while (locked < k && hres[locked] <= tol * scale_ref) ++locked;
        if (locked > l0 && locked < k) {
            const int nl = locked - l0;
            double *Vl = v.cur + (int64_t)l0 * D, *Z = w.Y.as<double>();
            CREST_CUDA_TRY(cudaMemcpyAsync(v.other + (int64_t)l0 * D, Vl, sizeof(double) * (size_t)D * nl,
                                           cudaMemcpyDeviceToDevice, st));
            k_scale_cols<<<(unsigned)ceil_div((int64_t)D * nl, 256), 256, 0, st>>>(Vl, out->theta + l0, lam_lo, D, nl, Z);
            CREST_CUDA_TRY(cudaGetLastError());
            Gemm g{D, D, nl, Z, D, 0, Vl, D, C, D, -1.0, C, 1.0, nullptr, 0.0};
            g.tB = 1;
            CREST_TRY(gemm(g, w.g, st));
        }
        res_max = 0.0;
        for (int i = 0; i < k; ++i) res_max = fmax(res_max, hres[i] / scale_ref);
        if (locked >= k) {
            converged = true;
            break;
        }
        if (it + 1 >= max_outer) break;
        // Chebyshev filter on the active columns, damping [lam_lo, a]
        const int qa = p - locked;
        const int64_t off = (int64_t)locked * D;
        const double a = theta[p - 1], top = theta[locked];
        const double e = 0.5 * (a + lam_lo), c = 0.5 * (a - lam_lo);
        if (!(c > 0.0) || !(top > a)) {
            // no usable interval: one power step
            CREST_CUDA_TRY(cudaMemcpyAsync(v.cur + off, cv.cur + off, sizeof(double) * (size_t)D * qa,
                                           cudaMemcpyDeviceToDevice, st));
        } else {
            // degree: growth 2e4 of the weakest wanted value over the damped
            // interval, capped so that no eigenvalue of the active operator
            // grows by more than 1e8 (the filtered block stays within reach of
            // shifted Cholesky QR).  Until a pair is locked the largest
            // eigenvalue is bounded by the Lanczos estimate, afterwards by the
            // leading active Ritz value plus its residual.
            double bound = top + hres[locked];
            if (locked == 0) bound = fmax(bound, lam_hi);
            const double xk = (theta[k - 1] - e) / c, xb = (bound - e) / c;
            const double gk = acosh(fmax(xk, 1.0 + 1e-12)), gb = acosh(fmax(xb, 1.0 + 1e-12));
            int m = (int)ceil(log(2e4) / fmax(gk, 1e-6));
            const int m_cap = (int)floor(log(1e8) / fmax(gb, 1e-6));
            m = std::max(2, std::min(m, std::min(m_cap, 60)));
            const double sigma1 = c / (top - e);
            double sigma = sigma1;
            // Y_1 = (sigma1 / c) (C - e) Y_0, C Y_0 at hand from the Ritz step, into the other buffer
            {
                prof::Scope ps("eig_gemm_fp64", st);
                const int64_t ne = (int64_t)D * qa;
                k_axpby<<<(unsigned)ceil_div(ne, 256), 256, 0, st>>>(cv.cur + off, v.cur + off, sigma1 / c,
                                                                     -sigma1 * e / c, ne, v.other + off);
            }
            CREST_CUDA_TRY(cudaGetLastError());
            v.swap();
            // Y_{j+1} = (2 s' / c) (C - e) Y_j - s s' Y_{j-1}, written over Y_{j-1}: the shift and the
            // older term are the product's epilogue
            for (int j = 2; j <= m; ++j) {
                const double sigma_next = 1.0 / (2.0 / sigma1 - sigma);
                double *Yj = v.cur + off, *Yo = v.other + off;
                Gemm g{D, qa, D, C, D, 1, Yj, D, Yo, D, 2.0 * sigma_next / c, Yo, -sigma * sigma_next, Yj,
                       -2.0 * sigma_next * e / c};
                g.overlap = 1;  // C is written before the k_axpby launch, which is ordered after it
                CREST_TRY(gemm(g, w.g, st));
                sigma = sigma_next;
                v.swap();
            }
        }
        CREST_TRY(orthonormalise(w, v, locked, true, st));
    }
    if (stats) *stats = EigStats{it + 1, converged ? 1 : 0, res_max};
    // columns 0..k-1 are the wanted Ritz vectors: locked ones (descending,
    // in locking order) then the active ones; order them by value once more
    k_rank<<<(unsigned)ceil_div(k, 128), 128, 0, st>>>(out->theta, (int)k, perm, jvals);
    CREST_CUDA_TRY(cudaGetLastError());
    k_emit<<<(unsigned)k, 256, 0, st>>>(v.cur, d, D, perm, jvals, k, out_vals, out_vecs);
    CREST_CUDA_TRY(cudaGetLastError());
    CREST_CUDA_TRY(cudaStreamSynchronize(st));
    return CREST_OK;
}

}  // namespace crest
