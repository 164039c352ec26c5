// Gram accumulation over the HVG columns (K3 densify + K4 SYRK).
//
// src/kernels.rs:221-309 accumulates G += S^T S sparsely on the CPU.  On the
// GPU each tile of up to m_cap cells is densified into a cell-major tile
// T[m_pad][d_pad] (one contiguous row of HVG genes per cell; the cells are
// the K dimension of the contraction) that stays L2-resident, and contracted
// as a dense SYRK over the upper-triangular block tiles of G:
//
//  * FP64: T = S, CUDA-core DMUL+DADD accumulating straight into G in cell
//    order, which reproduces the reference's f64 sums bit for bit (the extra
//    terms are exact zeros);
//  * FP32 (plain form): T = S + shift with shift = bias rounded to f32, i.e.
//    the dense scaled matrix Z (centred by construction) with its repeated
//    zero value stored exactly; FP32 register-tiled SYRK, folded into G in
//    FP64 with the exact correction S^T S = T^T T - shift c^T - c shift^T -
//    n shift shift^T;
//  * BF16X3 (product form): the same values split into bf16 hi/lo tiles,
//    contracted on the tcgen05 tensor cores (k_gram_tc.cu), same FP64 fold.
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "prof.cuh"
#include "rowwarp.cuh"

namespace crest {

int syrk_bf16x3_fold(const GramWork &w, int64_t m, const DevScale &t, double *gram, cudaStream_t st);

size_t gram_tile_bytes(int precision, int64_t d_pad, int64_t m_cap) {
    const size_t n = (size_t)d_pad * (size_t)m_cap;
    if (precision == CREST_GRAM_FP64) return n * 8;
    if (precision == CREST_GRAM_FP32) return n * 4;
    return n * 4;  // hi and lo bf16 tiles
}

// ----------------------------------------------------------------- shift
// Tile value of a zero entry for the centred forms: bias rounded to the tile
// precision (f32, or bf16 so that hi = shift and lo = 0), i.e. every repeated
// zero is stored exactly and the rounding error left in the tile is that of
// the stored entries only.  The epilogues correct with the same rounded value.
__global__ void k_tile_shift(int precision, const double *__restrict__ bias, int64_t d, int64_t d_pad,
                             double *__restrict__ shift) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= d_pad) return;
    double v = 0.0;
    if (bias && j < d) {
        v = bias[j];
        v = precision == CREST_GRAM_FP32 ? (double)__double2float_rn(v) : (double)__bfloat162float(__double2bfloat16(v));
    }
    shift[j] = v;
}

int launch_tile_shift(const GramWork &w, const DevScale &t, cudaStream_t st) {
    k_tile_shift<<<(unsigned)ceil_div(w.d_pad, 256), 256, 0, st>>>(w.precision, t.bias, w.d, w.d_pad, w.shift);
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

// ------------------------------------------------------------- HVG codes
// code[g] for a store gene id g < n_gene_map: -1 when the gene is dropped,
// sub_map[gene_map[g]] in [0, d) for an HVG column, d for another kept gene
// (it still counts towards the cell total).  One table lookup per entry
// then serves both the normalisation total and the HVG selection.  The
// same codes follow as int16 (when d < 2^15 - 1), zero-padded to a multiple
// of 8, for the kernels that copy the table to shared memory.
__global__ void k_hvg_code(const int32_t *__restrict__ gene_map, int64_t n_gene_map,
                           const int32_t *__restrict__ sub_map, int64_t n_vars, int64_t d, int32_t *__restrict__ code) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= round_up(n_gene_map, 8)) return;
    int32_t v = -1;
    if (g < n_gene_map) {
        const int32_t m = gene_map[g];
        if (m >= 0) v = (m < n_vars && sub_map[m] >= 0) ? sub_map[m] : (int32_t)d;
        code[g] = v;
    }
    if (d < 32767) const_cast<int16_t *>(codes16(code, n_gene_map))[g] = (int16_t)v;
}

size_t hvg_code_bytes(int64_t n_gene_map) {
    return 4 * (size_t)round_up(n_gene_map, 4) + 2 * (size_t)round_up(n_gene_map, 8);
}

int launch_hvg_code(const DevChunk &c, const int32_t *sub_map, int64_t n_vars, int64_t d, int32_t *code,
                    cudaStream_t st) {
    if (c.n_gene_map <= 0) return CREST_OK;
    k_hvg_code<<<(unsigned)ceil_div(round_up(c.n_gene_map, 8), 256), 256, 0, st>>>(c.gene_map, c.n_gene_map, sub_map,
                                                                                   n_vars, d, code);
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

// Shared-memory copy of the codes as int16 (d < 2^15 - 1) when it fits next
// to the kernel's other buffers; the global int32 table otherwise.
bool codes_in_smem(int64_t n_gene_map, int64_t d, size_t other_smem) {
    return d < 32767 && other_smem + 2 * (size_t)round_up(n_gene_map, 8) <= (size_t)kMaxSmem;
}

// ------------------------------------------------------------- densify
// Warp per cell row i of the tile (i < m_pad, padding rows included),
// written straight into the (L2-resident) tile.  Rows are handed out one at
// a time through a counter, since cells differ in length.  One read of the
// cell's entries (four per lane, 16-byte loads): lanes add up the kept
// values (the normalisation total) and queue the HVG entries (code, raw
// value), in entry order, in a per-warp shared-memory queue.  Then the row
// is filled with the zero-entry value of every gene -- the shift for kept
// cells, 0 for dropped / padding rows -- with 16-byte stores and, after a
// warp barrier that orders the two sets of stores, the queued entries are
// transformed and stored.  A cell with more than kQueue HVG entries, or
// whose total needs the in-order fold, reads its entries a second time
// (rare: such cells are the longest of a tile and would otherwise set its
// duration).  The colsum of S (FP32 / BF16X3) is privatised per block in
// shared memory.  Duplicate (cell, column) entries, which a dense tile cannot
// hold (the reference's pairwise loop adds v1^2 + v1 v2 + v2^2 for two
// entries of one gene), are detected: a cell whose HVG columns are not
// strictly increasing is searched for a repeated column (bit 1 of *status),
// or flagged as unchecked when it overflowed the queue (bit 2).
template <int MODE>  // 0 FP64 (T = S), 1 FP32 (T = S + shift), 2 BF16X3 (hi/lo of S + shift)
struct RowElem;
template <> struct RowElem<0> { using T = double; };
template <> struct RowElem<1> { using T = float; };
template <> struct RowElem<2> { using T = __nv_bfloat16; };

constexpr int kDensifyWarps = 32;
constexpr int kQueue = 512;

// Queued codes are int16 when the code table itself is (SMAP), else int32.
template <int MODE, bool SMAP>
static size_t densify_smem_fixed(int64_t d, int64_t d_pad) {
    using E = typename RowElem<MODE>::T;
    using Q = typename std::conditional<SMAP, int16_t, int32_t>::type;
    const size_t priv = MODE != 0 ? sizeof(double) * (size_t)round_up(d, 2) + sizeof(E) * (size_t)d_pad : 0;
    return priv + (size_t)kDensifyWarps * kQueue * (sizeof(Q) + sizeof(float));
}

template <int MODE, bool SMAP>
__global__ void __launch_bounds__(kDensifyWarps * 32, 1) k_densify(DevChunk c, const int32_t *__restrict__ code,
                                                                   DevScale t, const double *__restrict__ shift,
                                                                   int64_t d, int64_t d_pad, int64_t m_pad,
                                                                   void *tile, double *__restrict__ colsum,
                                                                   int64_t *n_kept, unsigned int *counter,
                                                                   int *status) {
    using E = typename RowElem<MODE>::T;
    using Q = typename std::conditional<SMAP, int16_t, int32_t>::type;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr bool priv = MODE != 0;
    // [colsum of S (f64)] [shift row (tile type)]   (MODE != 0)
    // [queue values (f32)] [queue codes (Q)] [codes (int16), SMAP]
    double *s_col = reinterpret_cast<double *>(smem);
    E *shift_row = reinterpret_cast<E *>(smem + (priv ? sizeof(double) * (size_t)round_up(d, 2) : 0));
    unsigned char *qbase = reinterpret_cast<unsigned char *>(shift_row) + (priv ? sizeof(E) * (size_t)d_pad : 0);
    float *q_x = reinterpret_cast<float *>(qbase) + (size_t)wid * kQueue;
    Q *q_code = reinterpret_cast<Q *>(qbase + sizeof(float) * (size_t)kDensifyWarps * kQueue) + (size_t)wid * kQueue;
    int16_t *s_code = reinterpret_cast<int16_t *>(qbase + (sizeof(Q) + sizeof(float)) * (size_t)kDensifyWarps * kQueue);
    if (priv) {
        for (int64_t j = threadIdx.x; j < d_pad; j += blockDim.x) shift_row[j] = (E)((shift && j < d) ? shift[j] : 0.0);
        for (int64_t j = threadIdx.x; j < d; j += blockDim.x) s_col[j] = 0.0;
    }
    if (SMAP) copy_codes16(code, c.n_gene_map, s_code);
    __syncthreads();
    auto lookup = [&](uint32_t g) -> int32_t { return SMAP ? (int32_t)s_code[g] : __ldg(code + g); };
    const int32_t dd = (int32_t)d;
    const int64_t nvec = d_pad * (int64_t)sizeof(E) / 16;
    E *hi_plane = reinterpret_cast<E *>(tile);
    E *lo_plane = hi_plane + (size_t)m_pad * d_pad;  // BF16X3 only
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const bool norm = c.target_sum > 0.0;
    int kept_count = 0;
    for (;;) {
        int64_t i = 0;
        if (lane == 0) i = atomicAdd(counter, 1u);
        i = __shfl_sync(kFull, i, 0);
        if (i >= m_pad) break;
        int64_t lo = 0, hi = 0, r = -1;
        if (i < c.n_spans) r = span_row(c, i, lo, hi);
        const bool kept = r >= 0;
        // one pass: total of the kept values and the queue of HVG entries
        double tsum = 0.0;
        bool ok = true, ovf = false, ordered = true;
        int nq = 0;
        int32_t carry = -1;
        if (kept) {
            for_entries_x4<true, kDensifyDepth>(c, lo, hi, lookup, [&](const int32_t (&m)[4], const float (&x)[4]) {
                bool hv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (m[u] >= 0 && norm) {
                        ok = ok && x[u] == rintf(x[u]) && fabsf(x[u]) < 16777216.0f;
                        tsum += (double)x[u];
                    }
                    hv[u] = m[u] >= 0 && m[u] < dd;
                }
                int cnt;
                int pos = nq + block_rank4(hv, cnt);
                if (cnt == 0) return;
                order_check4(hv, m, carry, ordered);
                if (nq + cnt > kQueue) {
                    ovf = true;
                    return;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (hv[u]) {
                        q_code[pos] = (Q)m[u];
                        q_x[pos] = x[u];
                        ++pos;
                    }
                nq += cnt;
            });
        }
        // fill the row with the zero-entry values
        E *row = hi_plane + (size_t)i * d_pad;
        {
            uint4 *dst = reinterpret_cast<uint4 *>(row);
            const uint4 *src = reinterpret_cast<const uint4 *>(shift_row);
            for (int64_t v = lane; v < nvec; v += 32) dst[v] = (priv && kept) ? src[v] : zero;
            if (MODE == 2) {
                uint4 *dlo = reinterpret_cast<uint4 *>(lo_plane + (size_t)i * d_pad);
                for (int64_t v = lane; v < nvec; v += 32) dlo[v] = zero;
            }
        }
        __syncwarp();  // orders the fill before the scattered entry stores; queue visible
        if (!kept) continue;
        kept_count += 1;
        if (!__all_sync(kFull, ordered)) {
            // columns not strictly increasing: look for a repeated column
            // among the queued entries (pairwise; such cells are rare)
            bool dup = false;
            if (!ovf) {
                for (int a = lane; a < nq; a += 32)
                    for (int b = 0; b < a; ++b) dup = dup || q_code[a] == q_code[b];
            }
            if (lane == 0) atomicOr(status, ovf ? 4 : 0);
            if (__any_sync(kFull, dup) && lane == 0) atomicOr(status, 2);
        }
        double scale = 1.0;
        if (norm) {
            double total;
            if (__all_sync(kFull, ok)) {
                total = warp_sum(tsum);
            } else {
                OrderedSum ts;
                for_entries_by<4, false>(c, lo, hi, lookup,
                                         [&](int32_t m, float x) { ts.add(m >= 0 ? (double)x : 0.0); });
                total = ts.acc;
            }
            scale = total > 0.0 ? c.target_sum / total : 1.0;
        }
        E *row_lo = lo_plane + (size_t)i * d_pad;
        auto put = [&](int32_t sub, float x) {
            const double s = scale_value(t, sub, transform_value(c, scale, x));
            if (MODE == 0) {
                row[sub] = s;
            } else {
                const double z = shift ? __dadd_rn(s, __ldg(shift + sub)) : s;
                if (MODE == 1) {
                    row[sub] = (E)__double2float_rn(z);
                } else {
                    __nv_bfloat16 h, l;
                    split_bf16(z, h, l);
                    row[sub] = h;
                    row_lo[sub] = l;
                }
                atomicAdd(s_col + sub, s);
            }
        };
        if (!ovf) {
            for (int e = lane; e < nq; e += 32) put((int32_t)q_code[e], q_x[e]);
        } else {
            for_entries_by<8, true>(c, lo, hi, lookup, [&](int32_t m, float x) {
                if (m >= 0 && m < dd) put(m, x);
            });
        }
        __syncwarp();  // queue reuse
    }
    if (lane == 0 && kept_count) atomicAdd(reinterpret_cast<unsigned long long *>(n_kept), (unsigned long long)kept_count);
    if (priv) {
        __syncthreads();
        for (int64_t j = threadIdx.x; j < d; j += blockDim.x)
            if (s_col[j] != 0.0) atomicAdd(colsum + j, s_col[j]);
    }
}

template <int MODE, bool SMAP>
static int launch_densify_k(const DevChunk &c, const int32_t *code, const DevScale &t, const double *shift,
                            const GramWork &w, int64_t m_pad, size_t smem, cudaStream_t st) {
    CREST_TRY(ensure_smem_attr((const void *)k_densify<MODE, SMAP>, smem));
    int64_t blocks = ceil_div(m_pad, kDensifyWarps);
    const int64_t cap = (int64_t)device_sms();
    if (blocks > cap) blocks = cap;
    k_densify<MODE, SMAP><<<(unsigned)blocks, kDensifyWarps * 32, smem, st>>>(c, code, t, shift, w.d, w.d_pad, m_pad,
                                                                               w.tile, w.colsum_chunk, w.n_kept,
                                                                               w.counter, w.status);
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

template <int MODE>
static int launch_densify_t(const DevChunk &c, const int32_t *code, const DevScale &t, const double *shift,
                            const GramWork &w, int64_t m_pad, cudaStream_t st) {
    const size_t fixed16 = densify_smem_fixed<MODE, true>(w.d, w.d_pad);
    if (codes_in_smem(c.n_gene_map, w.d, fixed16))
        return launch_densify_k<MODE, true>(c, code, t, shift, w, m_pad,
                                            fixed16 + 2 * (size_t)round_up(c.n_gene_map, 8), st);
    const size_t fixed = densify_smem_fixed<MODE, false>(w.d, w.d_pad);
    CREST_REQUIRE(fixed <= (size_t)kMaxSmem, CREST_EINVAL, "d=%lld too large for the densify shared buffers",
                  (long long)w.d);
    return launch_densify_k<MODE, false>(c, code, t, shift, w, m_pad, fixed, st);
}

int launch_densify(const DevChunk &c, const int32_t *code, const DevScale &t, const GramWork &w,
                   cudaStream_t st) {
    CREST_REQUIRE(c.n_spans <= w.m_cap, CREST_EINVAL, "tile holds %lld cells, chunk has %lld",
                  (long long)w.m_cap, (long long)c.n_spans);
    const int64_t m_pad = round_up(c.n_spans > 0 ? c.n_spans : 1, 64);
    CREST_CUDA_TRY(cudaMemsetAsync(w.n_kept, 0, 2 * sizeof(int64_t), st));  // kept count + work counter
    CREST_CUDA_TRY(cudaMemsetAsync(w.colsum_chunk, 0, sizeof(double) * (size_t)(w.d > 0 ? w.d : 1), st));
    const double *shift = nullptr;
    if (w.precision != CREST_GRAM_FP64 && t.scale) {
        CREST_TRY(launch_tile_shift(w, t, st));
        shift = w.shift;
    }
    prof::Scope ps("densify", st);
    if (w.precision == CREST_GRAM_FP64) return launch_densify_t<0>(c, code, t, nullptr, w, m_pad, st);
    if (w.precision == CREST_GRAM_FP32) return launch_densify_t<1>(c, code, t, shift, w, m_pad, st);
    return launch_densify_t<2>(c, code, t, shift, w, m_pad, st);
}

// ------------------------------------------------------------ FP64 SYRK
// Upper-triangular TILE x TILE block tiles; each thread owns P x Q outputs and
// accumulates G[a][b] + T[0][a]T[0][b] + T[1][a]T[1][b] + ... in cell order
// with separately rounded products, exactly like src/kernels.rs:303-305, so
// the cells cannot be split and a tile is one CTA's.  Both panels go through
// a cp.async ring of 16 cells a stage.
//
// Bound by the FP64 pipe (64 products or sums a cycle and SM: 8192 cells x
// 1000 genes 0.55 ms for the busiest SM's 64 x 64 tile) and by the latency of
// the few warps that a triangle of tiles leaves: 696 us now, 932 with the
// panels loaded between two barriers, 720 with four cells unrolled.  Tiles of
// 32 x 32 with 2 x 4 outputs a thread make four times the CTAs and twice the
// warps: while an SM gets at most three of them they end before one 64 x 64
// tile does (8192 cells, 300 / 700 / 850 genes: 345 / 446 / 596 us against
// 690; 1000 genes: 773 against 696).
__device__ __forceinline__ void tri_decode(int64_t t, int64_t nb, int &bi, int &bj) {
    // t enumerates (bi <= bj) row-major: row bi has nb - bi tiles
    int r = 0;
    int64_t rem = t;
    while (rem >= nb - r) {
        rem -= nb - r;
        ++r;
    }
    bi = r;
    bj = r + (int)rem;
}

constexpr int kSyrkF64Stages = 4, kSyrkF64Cells = 16;

template <int TILE, int P, int Q>
__global__ void __launch_bounds__(TILE / P * (TILE / Q)) k_syrk_f64(const double *__restrict__ T, int64_t d,
                                                                    int64_t d_pad, int64_t m_pad, int64_t nb,
                                                                    double *__restrict__ G) {
    constexpr int TX = TILE / Q, TY = TILE / P, NT = TX * TY;
    constexpr int kPanelF64 = kSyrkF64Cells * TILE;
    extern __shared__ __align__(16) double f64_ring[];  // [stage][A, B][cell][TILE genes]
    int bi, bj;
    tri_decode(blockIdx.x, nb, bi, bj);
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int64_t a0 = (int64_t)bi * TILE, b0 = (int64_t)bj * TILE;
    double acc[P][Q];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int64_t a = a0 + ty + TY * p, b = b0 + tx + TX * q;
            acc[p][q] = (a < d && b < d && a <= b) ? G[a * d + b] : 0.0;
        }
    // 16 bytes a copy, two genes of a cell; a pass of the block covers ROWS cells of one panel
    constexpr int ROWS = NT / (TILE / 2), PASSES = kSyrkF64Cells / ROWS;
    static_assert(ROWS * PASSES == kSyrkF64Cells, "passes must divide the cells of a step");
    const int kk0 = threadIdx.x / (TILE / 2), g = threadIdx.x % (TILE / 2) * 2;
    const double *src_a = T + kk0 * d_pad + a0 + g, *src_b = src_a + (b0 - a0);
    const unsigned ring = (unsigned)__cvta_generic_to_shared(f64_ring + kk0 * TILE + g);
    auto load = [&](int stage) {  // the next step's panels
#pragma unroll
        for (int r = 0; r < PASSES; ++r) {
            const unsigned to = ring + (unsigned)((stage * 2 * kPanelF64 + r * ROWS * TILE) * sizeof(double));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(to), "l"(src_a + r * ROWS * d_pad) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(to + kPanelF64 * (unsigned)sizeof(double)),
                         "l"(src_b + r * ROWS * d_pad)
                         : "memory");
        }
        src_a += kSyrkF64Cells * d_pad;
        src_b += kSyrkF64Cells * d_pad;
    };
    const int steps = (int)(m_pad / kSyrkF64Cells);  // m_pad is a multiple of 64
#pragma unroll
    for (int t = 0; t < kSyrkF64Stages - 1; ++t) {
        if (t < steps) load(t);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int t = 0; t < steps; ++t) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kSyrkF64Stages - 2) : "memory");
        __syncthreads();
        if (t + kSyrkF64Stages - 1 < steps) load((t + kSyrkF64Stages - 1) % kSyrkF64Stages);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const double *As = f64_ring + (t % kSyrkF64Stages) * (2 * kPanelF64) + ty;
        const double *Bs = As - ty + kPanelF64 + tx;
#pragma unroll 8
        for (int kk = 0; kk < kSyrkF64Cells; ++kk) {
            double av[P], bv[Q];
#pragma unroll
            for (int p = 0; p < P; ++p) av[p] = As[kk * TILE + TY * p];
#pragma unroll
            for (int q = 0; q < Q; ++q) bv[q] = Bs[kk * TILE + TX * q];
#pragma unroll
            for (int p = 0; p < P; ++p)
#pragma unroll
                for (int q = 0; q < Q; ++q) acc[p][q] = __dadd_rn(acc[p][q], __dmul_rn(av[p], bv[q]));
        }
    }
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int64_t a = a0 + ty + TY * p, b = b0 + tx + TX * q;
            if (a < d && b < d && a <= b) G[a * d + b] = acc[p][q];
        }
}

template <int TILE, int P, int Q>
static int launch_syrk_f64(const GramWork &w, int64_t m_pad, double *gram, cudaStream_t st) {
    constexpr size_t smem = sizeof(double) * kSyrkF64Stages * 2 * kSyrkF64Cells * TILE;
    const int64_t nb = ceil_div(w.d, TILE);
    CREST_TRY(ensure_smem_attr((const void *)k_syrk_f64<TILE, P, Q>, smem));
    prof::Scope ps("syrk_fp64", st);
    k_syrk_f64<TILE, P, Q><<<(unsigned)(nb * (nb + 1) / 2), TILE / P * (TILE / Q), smem, st>>>(
        (const double *)w.tile, w.d, w.d_pad, m_pad, nb, gram);
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

// colsum[j] += T[0][j] + T[1][j] + ... in cell order (FP64 form).
__global__ void k_colsum_f64(const double *__restrict__ T, int64_t d, int64_t d_pad, int64_t m,
                             double *__restrict__ colsum) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= d) return;
    double acc = colsum[j];
    for (int64_t i = 0; i < m; ++i) acc = __dadd_rn(acc, T[i * d_pad + j]);
    colsum[j] = acc;
}

// ------------------------------------------------------------ FP32 SYRK
// 128x128 upper-triangular block tiles, 256 threads, 8x8 register tile per
// thread, K in steps of 16 cells through a three-stage cp.async ring.  The
// FP32 register accumulators are folded into FP64 register sums every
// kFoldSteps K steps, so an FP32 rounding chain only ever spans
// kFoldSteps*16 cells: the error of a chain grows with its length times the
// partial's magnitude, and at 1M cells 256-cell chains left the top-50
// subspace 0.03 degree from the FP64 Gram's; 32-cell chains keep it an order
// of magnitude closer.
//
// The work is (tiles) x (groups of 32 cells), dealt evenly to one CTA per SM
// in runs over that order: a CTA's run covers the end of one tile, whole
// tiles, and the start of another.  A whole tile goes straight into G with
// the shift correction; a part of one leaves its FP64 sums in the CTA's
// workspace (two parts at most), and k_syrk_f32_parts adds a tile's parts in
// order with the correction, so results do not depend on scheduling.  Bound
// by the FP32 pipe (packed FFMA2, each half rounded as a plain fused
// multiply-add; 70 TFLOP/s, 62 % busy) and the conversions of the folds: 30,000 cells x
// 1,501 genes 4.2 ms with a CTA per tile (78 of 148 SMs), 1.7 ms now.
constexpr int kBM = 128, kBK = 16, kFoldSteps = 2, kSyrkStages = 3;
constexpr int kPanel = kBK * kBM;  // floats of one panel
constexpr size_t kSyrkF32Smem = sizeof(float) * kSyrkStages * 2 * kPanel;
constexpr int kGroupCells = kBK * kFoldSteps;

typedef unsigned long long u64;
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 twice(float v) {
    u64 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}

// One CTA's run of the work, in groups of cells.
__host__ __device__ inline int64_t syrk_run_start(int64_t cta, int64_t units, int64_t ctas) { return cta * units / ctas; }
// The CTA whose run holds a unit.
__host__ __device__ inline int64_t syrk_owner(int64_t unit, int64_t units, int64_t ctas) {
    return ((unit + 1) * ctas - 1) / units;
}

// CTAs of a launch.  Even runs leave parts of tiles to be written, read and
// added in a second launch, the more the more tiles there are: with one CTA per
// SM about as long as kPartsGroups x tiles / SMs groups take.  A CTA per tile is
// taken where it is longer than even runs by no more than that (no tile is then
// in parts, nor when whole tiles come out even).  Even runs against a CTA per
// tile: 2,000 genes (136 tiles), 64 / 384 / 1,024 / 2,048 cells 34 / 73 / 130 /
// 227 us against 23 / 56 / 123 / 229; 1,501 (78), 64 / 192 / 256 / 512 cells 34 /
// 39 / 42 / 56 against 23 / 36 / 43 / 70; 1,000 (36), 64 / 128 cells 20 / 22
// against 22 / 29.
constexpr int64_t kPartsGroups = 6;
inline int64_t syrk_ctas(int64_t tiles, int64_t groups, int64_t sms) {
    if (tiles <= sms && groups * (sms - tiles) <= kPartsGroups * tiles) return tiles;
    return std::min(sms, tiles * groups);
}

// Row / column of this thread's output (p, q) in a tile.
__device__ __forceinline__ int syrk_row(int tid, int p) { return (p < 4 ? 0 : 60) + (tid >> 4) * 4 + p; }
__device__ __forceinline__ int syrk_col(int tid, int q) { return (q < 4 ? 0 : 60) + (tid & 15) * 4 + q; }

// The column side of the shift correction, and one row of outputs into G with
// it: the loads of a row go out together (one after another, each behind the
// store of the element before, the 64 outputs of a thread took 5 to 12 us more).
struct SyrkCols {
    double shift[8], colsum[8];
};
__device__ __forceinline__ void syrk_cols(SyrkCols &c, int64_t b0, int tid, int64_t d, const double *shift,
                                          const double *colsum_c) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int64_t b = b0 + syrk_col(tid, q);
        c.shift[q] = shift && b < d ? __ldg(shift + b) : 0.0;
        c.colsum[q] = shift && b < d ? __ldg(colsum_c + b) : 0.0;
    }
}
__device__ __forceinline__ void syrk_add_row(const double (&v)[8], const SyrkCols &c, int64_t a, int64_t b0, int tid,
                                             int64_t d, const double *shift, const double *colsum_c, double nk,
                                             double *G) {
    if (a >= d) return;
    const double ba = shift ? __ldg(shift + a) : 0.0, ca = shift ? __ldg(colsum_c + a) : 0.0;
    double g[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int64_t b = b0 + syrk_col(tid, q);
        g[q] = b < d && b >= a ? G[a * d + b] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int64_t b = b0 + syrk_col(tid, q);
        const double x = shift ? v[q] - ba * c.colsum[q] - ca * c.shift[q] - nk * ba * c.shift[q] : v[q];
        if (b < d && b >= a) G[a * d + b] = g[q] + x;
    }
}

__global__ void __launch_bounds__(256, 1) k_syrk_f32(const float *__restrict__ T, int64_t d, int64_t d_pad,
                                                     int64_t m_pad, int64_t nb, int64_t tiles,
                                                     const double *__restrict__ shift,
                                                     const double *__restrict__ colsum_c,
                                                     const int64_t *__restrict__ n_kept, double *__restrict__ G,
                                                     double *__restrict__ parts) {
    extern __shared__ __align__(16) float syrk_sm[];  // [stage][A, B][cell][gene]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int64_t groups = m_pad / kGroupCells, units = tiles * groups;
    const int64_t u0 = syrk_run_start(blockIdx.x, units, gridDim.x), u1 = syrk_run_start(blockIdx.x + 1, units, gridDim.x);
    // loader: a panel is 16 cells x 128 genes, two 16-byte pieces per thread and panel
    const int lk = tid >> 5, lg = (tid & 31) * 4;
    for (int64_t u = u0; u < u1;) {
        const int64_t t = u / groups, g0 = u - t * groups, g1 = min(groups, g0 + (u1 - u));
        int bi, bj;
        tri_decode(t, nb, bi, bj);
        const float *Ta = T + (int64_t)bi * kBM + lg, *Tb = T + (int64_t)bj * kBM + lg;
        const int64_t k_begin = g0 * kGroupCells;
        const int steps = (int)(g1 - g0) * kFoldSteps;
        auto load = [&](int s) {
            float *a = syrk_sm + (s % kSyrkStages) * 2 * kPanel, *b = a + kPanel;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int kk = lk + 8 * r;
                const int64_t row = (k_begin + (int64_t)s * kBK + kk) * d_pad;
                const unsigned sa = (unsigned)__cvta_generic_to_shared(a + kk * kBM + lg);
                const unsigned sb = (unsigned)__cvta_generic_to_shared(b + kk * kBM + lg);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(Ta + row) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sb), "l"(Tb + row) : "memory");
            }
        };
        u64 acc[8][4];
        double acc64[8][8];
#pragma unroll
        for (int p = 0; p < 8; ++p)
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                acc[p][q >> 1] = 0ull;
                acc64[p][q] = 0.0;
            }
        __syncthreads();  // the ring's last readers of the part before
#pragma unroll
        for (int s = 0; s < kSyrkStages - 1; ++s) {
            if (s < steps) load(s);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        for (int s = 0; s < steps; ++s) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(kSyrkStages - 2) : "memory");
            __syncthreads();
            if (s + kSyrkStages - 1 < steps) load(s + kSyrkStages - 1);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            const float *a = syrk_sm + (s % kSyrkStages) * 2 * kPanel, *b = a + kPanel;
#pragma unroll
            for (int kk = 0; kk < kBK; ++kk) {
                const float4 a_lo = *reinterpret_cast<const float4 *>(a + kk * kBM + ty * 4);
                const float4 a_hi = *reinterpret_cast<const float4 *>(a + kk * kBM + 64 + ty * 4);
                const ulonglong2 b_lo = *reinterpret_cast<const ulonglong2 *>(b + kk * kBM + tx * 4);
                const ulonglong2 b_hi = *reinterpret_cast<const ulonglong2 *>(b + kk * kBM + 64 + tx * 4);
                const float av[8] = {a_lo.x, a_lo.y, a_lo.z, a_lo.w, a_hi.x, a_hi.y, a_hi.z, a_hi.w};
                const u64 bv[4] = {b_lo.x, b_lo.y, b_hi.x, b_hi.y};
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    const u64 a2 = twice(av[p]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) acc[p][q] = fma2(a2, bv[q], acc[p][q]);
                }
            }
            if ((s + 1) % kFoldSteps == 0) {
#pragma unroll
                for (int p = 0; p < 8; ++p)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        acc64[p][2 * q] += (double)__uint_as_float((unsigned)acc[p][q]);
                        acc64[p][2 * q + 1] += (double)__uint_as_float((unsigned)(acc[p][q] >> 32));
                        acc[p][q] = 0ull;
                    }
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        if (g1 - g0 == groups) {
            const double nk = (double)*n_kept;
            SyrkCols cols;
            syrk_cols(cols, (int64_t)bj * kBM, tid, d, shift, colsum_c);
#pragma unroll
            for (int p = 0; p < 8; ++p)
                syrk_add_row(acc64[p], cols, (int64_t)bi * kBM + syrk_row(tid, p), (int64_t)bj * kBM, tid, d, shift,
                             colsum_c, nk, G);
        } else {  // part 0 of the CTA when its run begins here, else part 1
            double *o = parts + (2 * (int64_t)blockIdx.x + (u == u0 ? 0 : 1)) * kBM * kBM + tid;
#pragma unroll
            for (int p = 0; p < 8; ++p)
#pragma unroll
                for (int q = 0; q < 8; ++q) o[(p * 8 + q) * 256] = acc64[p][q];
        }
        u += g1 - g0;
    }
}

// Tiles in parts: blockIdx.x = tile, blockIdx.y = row p of the threads' outputs.
__global__ void __launch_bounds__(256) k_syrk_f32_parts(int64_t d, int64_t m_pad, int64_t nb, int64_t tiles,
                                                        int64_t ctas, const double *__restrict__ shift,
                                                        const double *__restrict__ colsum_c,
                                                        const int64_t *__restrict__ n_kept, double *__restrict__ G,
                                                        const double *__restrict__ parts) {
    const int64_t groups = m_pad / kGroupCells, units = tiles * groups, t = blockIdx.x;
    const int64_t c0 = syrk_owner(t * groups, units, ctas), c1 = syrk_owner((t + 1) * groups - 1, units, ctas);
    if (c0 == c1) return;  // in one run: whole
    int bi, bj;
    tri_decode(t, nb, bi, bj);
    const int tid = threadIdx.x, p = blockIdx.y;
    const double nk = (double)*n_kept;
    double v[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int64_t c = c0; c <= c1; ++c) {
        const int part = syrk_run_start(c, units, ctas) / groups == t ? 0 : 1;  // the first of its run, or a later one
        const double *o = parts + (2 * c + part) * kBM * kBM + p * 8 * 256 + tid;
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] += o[q * 256];
    }
    SyrkCols cols;
    syrk_cols(cols, (int64_t)bj * kBM, tid, d, shift, colsum_c);
    syrk_add_row(v, cols, (int64_t)bi * kBM + syrk_row(tid, p), (int64_t)bj * kBM, tid, d, shift, colsum_c, nk, G);
}

size_t syrk_f32_parts_bytes() { return sizeof(double) * 2 * (size_t)device_sms() * kBM * kBM; }

__global__ void k_add_colsum(const double *__restrict__ src, int64_t d, double *__restrict__ dst) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < d) dst[j] += src[j];
}

int launch_syrk_fold(const GramWork &w, int64_t m, const DevScale &t, double *gram, double *colsum,
                     cudaStream_t st, bool add_colsum) {
    if (w.d == 0) return CREST_OK;
    const int64_t m_pad = round_up(m > 0 ? m : 1, 64);
    if (w.precision == CREST_GRAM_FP64) {
        const int64_t nb = ceil_div(w.d, 32);
        if (nb * (nb + 1) / 2 <= 3 * (int64_t)device_sms()) {  // up to 928 genes
            CREST_TRY((launch_syrk_f64<32, 2, 4>(w, m_pad, gram, st)));
        } else {
            CREST_TRY((launch_syrk_f64<64, 4, 4>(w, m_pad, gram, st)));
        }
        k_colsum_f64<<<(unsigned)ceil_div(w.d, 128), 128, 0, st>>>((const double *)w.tile, w.d, w.d_pad, m, colsum);
        CREST_CUDA_TRY(cudaGetLastError());
        return CREST_OK;
    }
    const double *shift = t.scale ? w.shift : nullptr;  // the tile's exact zero-entry value
    if (w.precision == CREST_GRAM_FP32) {
        const int64_t nb = w.d_pad / kBM;
        const int64_t tiles = nb * (nb + 1) / 2;
        prof::Scope ps("syrk_fp32", st);
        CREST_TRY(ensure_smem_attr((const void *)k_syrk_f32, (size_t)kSyrkF32Smem));
        const int64_t ctas = syrk_ctas(tiles, m_pad / kGroupCells, device_sms());
        k_syrk_f32<<<(unsigned)ctas, 256, kSyrkF32Smem, st>>>((const float *)w.tile, w.d, w.d_pad, m_pad, nb, tiles, shift,
                                                             w.colsum_chunk, w.n_kept, gram, w.part64);
        CREST_CUDA_TRY(cudaGetLastError());
        if (tiles % ctas) {
            k_syrk_f32_parts<<<dim3((unsigned)tiles, 8), 256, 0, st>>>(w.d, m_pad, nb, tiles, ctas, shift, w.colsum_chunk,
                                                                      w.n_kept, gram, w.part64);
            CREST_CUDA_TRY(cudaGetLastError());
        }
    } else {
        CREST_TRY(syrk_bf16x3_fold(w, m_pad, t, gram, st));
    }
    if (add_colsum) {
        k_add_colsum<<<(unsigned)ceil_div(w.d, 256), 256, 0, st>>>(w.colsum_chunk, w.d, colsum);
        CREST_CUDA_TRY(cudaGetLastError());
    }
    return CREST_OK;
}

}  // namespace crest
