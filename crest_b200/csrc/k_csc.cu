// Gene-major (CSC) copy of a device-resident CSR matrix and the per-gene
// statistics read from it (src/kernels.rs:144-160 gene_stats).
//
// Per-gene sums over cells are a scatter in the CSR layout: every stored
// entry adds four f64 values at its gene, and without a native f64 atomic in
// shared memory that scatter ran at 0.07 of HBM bandwidth.  In the CSC copy
// each gene's entries are contiguous, so the sums become segmented reductions
// with no atomics per entry: a warp reduces a segment of one gene's column
// (cell ids and raw values, coalesced) and adds its five partial sums to the
// gene's outputs once.
//
// What an entry adds depends only on its cell and its count, and most counts
// are small: the transformed value and its expm1 are tabulated per cell for
// the counts 1 .. T before the pass, and an entry gathers its pair (one
// 32-byte sector from L2, the bound of the pass) instead of evaluating log1p
// and a double-precision expm1.  Other values take the evaluation.
//
// The copy is built once per matrix (it holds raw counts; maps and transforms
// are applied when it is read): a per-gene count (shared-memory histograms of
// blocks of cells), a host prefix sum, then a scatter in which each block of
// cells reserves one run per gene with a global atomic and places its entries
// with shared-memory atomics.  Entry order within a column follows that
// reservation order, so per-gene sums are added in no fixed order (as with
// atomics); they agree with the reference's to rounding.  Entries whose gene
// id is past the matrix's gene count are left out (every gene map drops them).
#include <vector>

#include "host.cuh"
#include "prof.cuh"
#include "rowwarp.cuh"

namespace crest {

// The transformed value of a count in a cell and its expm1; ev = -2 (below
// any expm1) marks a dropped cell.
struct __align__(16) CellValue {
    double ev;
    float v;
    float pad;
};

constexpr int kCscThreads = 1024;
constexpr int kCscBlockCells = 128;
constexpr int64_t kSegEntries = 2048;  // of a segment: 64 per lane of its warp
constexpr int kTabCounts = 8;          // counts tabulated per cell, at most
constexpr size_t kTabBytes = 32u << 20;
// Counts 1 .. T of n_cells cells: as many as keep the table a quarter of L2, or
// none when those are fewer than four (above 524,288 cells): a warp then meets
// an untabulated count in nearly every step and evaluates anyway.  Table against
// none: 250,000 cells (8 counts, 100 M entries) 385 us / 869, 500,000 (4, 50 M)
// 354 / 455, 700,000 (2, 70 M) 654 / 618, 1 M (2, 100 M) 902 / 852, 2 M (1, 200 M)
// 1752 / 1662, 8 M (1, 96 M) 1240 / 891.
constexpr int kTabLeast = 4;
inline int tab_counts(int64_t n_cells) {
    const int64_t fit = (int64_t)(kTabBytes / sizeof(CellValue)) / std::max<int64_t>(n_cells, 1);
    return fit < kTabLeast ? 0 : (int)std::min<int64_t>(kTabCounts, fit);
}

// cells [c0, c1) of a block, one warp per cell: f(gene, value, cell)
template <class F>
__device__ __forceinline__ void block_entries(const int64_t *__restrict__ indptr, const uint32_t *__restrict__ genes,
                                              const float *__restrict__ values, int64_t c0, int64_t c1, F &&f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int64_t cell = c0 + warp; cell < c1; cell += nw) {
        const int64_t lo = indptr[cell], hi = indptr[cell + 1];
        for (int64_t e = lo + lane; e < hi; e += 32) f(__ldg(genes + e), values ? __ldg(values + e) : 0.0f, cell);
    }
}

// count[g] += entries of gene g (blocks of 8 x kCscBlockCells cells)
__global__ void __launch_bounds__(kCscThreads, 1) k_col_count(const int64_t *__restrict__ indptr,
                                                              const uint32_t *__restrict__ genes, int64_t n_cells,
                                                              int64_t n_genes, unsigned long long *__restrict__ count) {
    extern __shared__ uint32_t hist[];
    const int64_t span = (int64_t)kCscBlockCells * 8;
    for (int64_t b0 = (int64_t)blockIdx.x * span; b0 < n_cells; b0 += (int64_t)gridDim.x * span) {
        const int64_t b1 = b0 + span < n_cells ? b0 + span : n_cells;
        for (int64_t g = threadIdx.x; g < n_genes; g += blockDim.x) hist[g] = 0u;
        __syncthreads();
        block_entries(indptr, genes, nullptr, b0, b1, [&](uint32_t g, float, int64_t) {
            if ((int64_t)g < n_genes) atomicAdd(hist + g, 1u);
        });
        __syncthreads();
        for (int64_t g = threadIdx.x; g < n_genes; g += blockDim.x)
            if (hist[g]) atomicAdd(count + g, (unsigned long long)hist[g]);
        __syncthreads();
    }
}

// cursor[g]: entries of gene g placed so far, relative to col_ptr[g].
__global__ void __launch_bounds__(kCscThreads, 1)
    k_col_scatter(const int64_t *__restrict__ indptr, const uint32_t *__restrict__ genes,
                  const float *__restrict__ values, int64_t n_cells, int64_t n_genes,
                  const int64_t *__restrict__ col_ptr, uint32_t *__restrict__ cursor, uint32_t *__restrict__ col_cell,
                  float *__restrict__ col_val) {
    extern __shared__ uint32_t slot[];  // per gene: entries of the block, then the next free offset of its run
    for (int64_t b0 = (int64_t)blockIdx.x * kCscBlockCells; b0 < n_cells; b0 += (int64_t)gridDim.x * kCscBlockCells) {
        const int64_t b1 = b0 + kCscBlockCells < n_cells ? b0 + kCscBlockCells : n_cells;
        for (int64_t g = threadIdx.x; g < n_genes; g += blockDim.x) slot[g] = 0u;
        __syncthreads();
        block_entries(indptr, genes, nullptr, b0, b1, [&](uint32_t g, float, int64_t) {
            if ((int64_t)g < n_genes) atomicAdd(slot + g, 1u);
        });
        __syncthreads();
        for (int64_t g = threadIdx.x; g < n_genes; g += blockDim.x) {  // one run per gene present
            const uint32_t k = slot[g];
            if (k) slot[g] = atomicAdd(cursor + g, k);
        }
        __syncthreads();
        block_entries(indptr, genes, values, b0, b1, [&](uint32_t g, float x, int64_t cell) {
            if ((int64_t)g >= n_genes) return;
            const int64_t pos = __ldg(col_ptr + g) + atomicAdd(slot + g, 1u);
            col_cell[pos] = (uint32_t)cell;
            col_val[pos] = x;
        });
        __syncthreads();
    }
}

// Per store cell: target / total of its kept genes (1 without
// normalisation, or when the total is 0), or -1 for a dropped cell; and the
// table of its small counts, tab[x - 1][cell] (one count after another, since
// a gene's entries mostly share theirs and often come from nearby cells).
__global__ void k_cell_table(DevChunk c, int64_t n_cells, const double *__restrict__ total, int counts,
                             double *__restrict__ cs, CellValue *__restrict__ tab) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_cells) return;
    double scale = -1.0;
    if (i < c.n_cell_map && c.cell_map[i] >= 0) {
        scale = 1.0;
        if (c.target_sum > 0.0) {
            const double t = total[i];
            scale = t > 0.0 ? c.target_sum / t : 1.0;
        }
    }
    cs[i] = scale;
    for (int x = 1; x <= counts; ++x) {
        CellValue e;
        e.v = scale < 0.0 ? 0.0f : transform_value(c, scale, (float)x);
        e.ev = scale < 0.0 ? -2.0 : expm1((double)e.v);
        e.pad = 0.0f;
        tab[(int64_t)(x - 1) * n_cells + i] = e;
    }
}

// Five sums of one segment of a gene's column per warp: out[m * 5 + s] +=
// (x, x^2, expm1 x, expm1(x)^2, 1) over the segment's entries of kept
// cells, x the transformed value.  A lane has kStatsUnroll entries' gathers and the
// next entries in flight; blocks are of two warps, so that a long segment
// holds up one other.  100,000 cells, 213M entries: 2.97 ms when every entry
// was evaluated (7.5 instructions an entry, latency between them) in CTA-wide
// segments, 0.72 ms from the table (12 TB/s of sectors and columns from L2
// and HBM; 0.80 with the entries loaded only when needed and blocks of eight
// warps).
constexpr int kStatsUnroll = 4, kStatsThreads = 64;

__global__ void __launch_bounds__(kStatsThreads) k_gene_stats_csc(DevChunk c, const int64_t *__restrict__ seg_lo,
                                                                  const int32_t *__restrict__ seg_gene, int64_t n_segs,
                                                                  const int64_t *__restrict__ col_ptr,
                                                                  const uint32_t *__restrict__ col_cell,
                                                                  const float *__restrict__ col_val, int64_t n_cells,
                                                                  const double *__restrict__ cell_scale, int counts,
                                                                  const CellValue *__restrict__ tab,
                                                                  double *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const float top = (float)counts;
    for (int64_t s = warp; s < n_segs; s += n_warps) {
        const int32_t g = seg_gene[s];
        const int32_t m = g < c.n_gene_map ? __ldg(c.gene_map + g) : -1;
        if (m < 0) continue;  // uniform over the warp
        const int64_t e0 = seg_lo[s], end = col_ptr[g + 1];
        const int n = (int)(end - e0 < kSegEntries ? end - e0 : kSegEntries);
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        int kept = 0;
        uint32_t ncell[kStatsUnroll];
        float nx[kStatsUnroll];
        auto fetch = [&](int b) {
#pragma unroll
            for (int u = 0; u < kStatsUnroll; ++u) {
                const bool in = b + 32 * u < n;
                ncell[u] = in ? __ldcs(col_cell + e0 + b + 32 * u) : 0u;
                nx[u] = in ? __ldcs(col_val + e0 + b + 32 * u) : 1.0f;
            }
        };
        fetch(lane);
        for (int b = lane; b < n; b += 32 * kStatsUnroll) {
            uint32_t cell[kStatsUnroll];
            float x[kStatsUnroll];
            double2 e[kStatsUnroll];
            bool use[kStatsUnroll], slow[kStatsUnroll];
#pragma unroll
            for (int u = 0; u < kStatsUnroll; ++u) {
                use[u] = b + 32 * u < n;
                cell[u] = ncell[u];
                x[u] = nx[u];
            }
            fetch(b + 32 * kStatsUnroll);
#pragma unroll
            for (int u = 0; u < kStatsUnroll; ++u) {
                // x in 1 .. counts: adding 2^23 leaves the integer in the low mantissa bits
                const float t = x[u] + 8388608.0f;
                const int k = (int)(__float_as_uint(t) & 0xffu);
                slow[u] = !(x[u] >= 1.0f && x[u] <= top && t - 8388608.0f == x[u]);
                e[u] = make_double2(0.0, 0.0);
                if (!slow[u])
                    e[u] = __ldg(reinterpret_cast<const double2 *>(tab + (int64_t)(k - 1) * n_cells + cell[u]));
            }
#pragma unroll
            for (int u = 0; u < kStatsUnroll; ++u) {
                double ev = e[u].x;
                float vf = __int_as_float(__double2loint(e[u].y));
                if (slow[u]) {
                    const double scale = __ldg(cell_scale + cell[u]);
                    vf = transform_value(c, scale, x[u]);
                    ev = expm1((double)vf);
                    use[u] = use[u] && !(scale < 0.0);  // a cell whose factor is NaN is a kept one
                } else {
                    use[u] = use[u] && ev != -2.0;
                }
                if (use[u]) {
                    const double v = (double)vf;
                    a0 += v;
                    a1 += __dmul_rn(v, v);
                    a2 += ev;
                    a3 += __dmul_rn(ev, ev);
                    ++kept;
                }
            }
        }
        a0 = warp_sum(a0);
        a1 = warp_sum(a1);
        a2 = warp_sum(a2);
        a3 = warp_sum(a3);
        kept = __reduce_add_sync(kFull, kept);
        if (lane < 5) {
            const double t = lane == 0 ? a0 : lane == 1 ? a1 : lane == 2 ? a2 : lane == 3 ? a3 : (double)kept;
            if (t != 0.0) atomicAdd(out + (size_t)m * 5 + lane, t);
        }
    }
}

int build_csc(const int64_t *indptr, const uint32_t *genes, const float *values, int64_t n_cells, int64_t n_genes,
              int64_t nnz, CscMatrix &out, cudaStream_t st) {
    CREST_REQUIRE(4 * (size_t)n_genes <= (size_t)kMaxSmem, CREST_EINVAL, "too many genes for the CSC build");
    CREST_TRY(out.col_ptr.ensure(8 * (size_t)(n_genes + 1)));
    CREST_TRY(out.col_cell.ensure(4 * (size_t)std::max<int64_t>(nnz, 1)));
    CREST_TRY(out.col_val.ensure(4 * (size_t)std::max<int64_t>(nnz, 1)));
    DevBuf cursor;  // per-gene counts (u64), then per-gene placement cursors (u32)
    CREST_TRY(cursor.ensure(8 * (size_t)std::max<int64_t>(n_genes, 1)));
    CREST_CUDA_TRY(cudaMemsetAsync(cursor.ptr, 0, 8 * (size_t)n_genes, st));
    const size_t smem = 4 * (size_t)n_genes;
    CREST_TRY(ensure_smem_attr((const void *)k_col_count, smem));
    CREST_TRY(ensure_smem_attr((const void *)k_col_scatter, smem));
    const int grid = device_sms();
    {
        prof::Scope ps("csc_build", st);
        k_col_count<<<grid, kCscThreads, smem, st>>>(indptr, genes, n_cells, n_genes,
                                                      cursor.as<unsigned long long>());
        CREST_CUDA_TRY(cudaGetLastError());
    }
    std::vector<unsigned long long> cnt(n_genes);
    CREST_CUDA_TRY(cudaMemcpyAsync(cnt.data(), cursor.ptr, 8 * (size_t)n_genes, cudaMemcpyDeviceToHost, st));
    CREST_CUDA_TRY(cudaStreamSynchronize(st));
    std::vector<int64_t> ptr(n_genes + 1, 0);
    for (int64_t g = 0; g < n_genes; ++g) {
        CREST_REQUIRE(cnt[g] < (1ull << 32), CREST_EINVAL, "gene %lld has 2^32 or more entries", (long long)g);
        ptr[g + 1] = ptr[g] + (int64_t)cnt[g];
    }
    std::vector<int64_t> seg_lo;
    std::vector<int32_t> seg_gene;
    for (int64_t g = 0; g < n_genes; ++g)
        for (int64_t e = ptr[g]; e < ptr[g + 1]; e += kSegEntries) {
            seg_lo.push_back(e);
            seg_gene.push_back((int32_t)g);
        }
    out.n_segs = (int64_t)seg_lo.size();
    CREST_TRY(upload(out.col_ptr, ptr.data(), n_genes + 1, st));
    CREST_TRY(upload(out.seg_lo, seg_lo.data(), out.n_segs, st));
    CREST_TRY(upload(out.seg_gene, seg_gene.data(), out.n_segs, st));
    CREST_CUDA_TRY(cudaMemsetAsync(cursor.ptr, 0, 4 * (size_t)n_genes, st));
    {
        prof::Scope ps("csc_build", st);
        k_col_scatter<<<grid, kCscThreads, smem, st>>>(indptr, genes, values, n_cells, n_genes,
                                                        out.col_ptr.as<int64_t>(), cursor.as<uint32_t>(),
                                                        out.col_cell.as<uint32_t>(), out.col_val.as<float>());
        CREST_CUDA_TRY(cudaGetLastError());
    }
    CREST_CUDA_TRY(cudaStreamSynchronize(st));
    cursor.release();
    out.n_genes = n_genes;
    return CREST_OK;
}

int launch_gene_stats_csc(const DevChunk &c, CscMatrix &m, const double *total, double *out, cudaStream_t st) {
    if (m.n_segs == 0) return CREST_OK;
    const int64_t n = std::max<int64_t>(c.n_spans, 1);
    const int counts = tab_counts(n);
    CREST_TRY(m.cell_scale.ensure(8 * (size_t)n));
    CREST_TRY(m.cell_table.ensure(sizeof(CellValue) * (size_t)n * counts));
    prof::Scope ps("gene_stats_csc", st);
    if (c.n_spans)
        k_cell_table<<<(unsigned)ceil_div(c.n_spans, 256), 256, 0, st>>>(
            c, c.n_spans, total, counts, m.cell_scale.as<double>(), m.cell_table.as<CellValue>());
    const int64_t blocks = std::min<int64_t>(ceil_div(m.n_segs, kStatsThreads / 32), (int64_t)device_sms() * 128);
    k_gene_stats_csc<<<(unsigned)blocks, kStatsThreads, 0, st>>>(
        c, m.seg_lo.as<int64_t>(), m.seg_gene.as<int32_t>(), m.n_segs, m.col_ptr.as<int64_t>(),
        m.col_cell.as<uint32_t>(), m.col_val.as<float>(), c.n_spans, m.cell_scale.as<double>(), counts,
        m.cell_table.as<CellValue>(), out);
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

}  // namespace crest
