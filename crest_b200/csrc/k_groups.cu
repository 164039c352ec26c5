// Per (group, gene) sums of the transformed matrix: the streaming pass behind
// differential expression (rank_genes_groups t-test) and pseudobulk totals
// (src/kernels.rs:388-442 group_gene_sums; src/py.rs:311-357).
//
// For every stored entry of a kept cell whose row has a group
// (group_of_row[row] != 0xffffffff) and whose gene is kept:
//   x = the lazily transformed value (normalize_total / log1p, f32),
//   x = min(x, clip[group][gene]) when a clip table is given (seurat_v3),
//   sum[group][gene] += x, sumsq += x * x, nnz += 1        (f64)
// One warp per cell: the cell's normalisation factor from a first read of the
// row (as every pass here; nothing is kept from one call for the next), then
// the entries.  The transformed value of a count depends on the cell only, so
// lane l evaluates that of l + 1 once per cell and an entry takes it from there
// by a shuffle; other values are evaluated.  Per entry, two f64 atomics and one
// integer atomic go to global memory: the (n_groups x n_vars) outputs stay in
// L2, and these three updates of three arrays bound the pass, not the
// evaluation they replace (50,000 cells, 70M entries, every cell in a group:
// 1.22 ms, as with every entry evaluated and three f64 atomics; with a
// twentieth of the cells in a group 125 us against 168).  The reference sums
// each (group, gene) in entry order; here the order of the atomics is not fixed,
// so results agree to rounding.
//
// The counts are 32-bit integers, which halves that part of the read-back, in
// outputs of kNarrowCounts (65,536 group and gene pairs) and more.  Smaller outputs have
// few lines for all the entries to meet on, and counts side by side in half as
// many make it worse, so there they are as wide as the sums (doubles): 2 x 2,000
// pairs, 30M entries 1208 us against 1587, 20 x 500, 2M 76 / 92, 40 x 500 33 / 39,
// 2 x 5,000, 5M 132 / 140, 2 x 33,538, 70M 1446 / 1471 (2 x 20,000, 57M 1130 /
// 1109); 20 x 20,000 1087 / 1068, 40 x 33,538 1376 / 1342.
#include "kernels.cuh"
#include "prof.cuh"
#include "rowwarp.cuh"

namespace crest {

template <class N>
__global__ void __launch_bounds__(256) k_group_gene_sums(DevChunk c, const uint32_t *__restrict__ group_of_row,
                                                         int64_t n_vars, const double *__restrict__ clip,
                                                         double *__restrict__ sum, double *__restrict__ sumsq,
                                                         N *__restrict__ nnz) {
    const int lane = lane_id();
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = warp; i < c.n_spans; i += n_warps) {
        int64_t lo, hi;
        const int64_t row = span_row(c, i, lo, hi);
        if (row < 0) continue;
        const uint32_t grp = __ldg(group_of_row + row);
        if (grp == 0xffffffffu) continue;
        const double scale = cell_scale(c, lo, hi);
        const float own = transform_value(c, scale, (float)(lane + 1));
        const int64_t base = (int64_t)grp * n_vars;
        for_entries<8>(c, lo, hi, [&](int32_t m, float xf) {
            const bool small = xf >= 1.0f && xf <= 32.0f && xf == rintf(xf);
            float v = __shfl_sync(kFull, own, small ? (int)xf - 1 : 0);
            if (m < 0) return;
            if (!small) v = transform_value(c, scale, xf);
            const int64_t at = base + m;
            double x = (double)v;
            if (clip) x = fmin(x, __ldg(clip + at));
            atomicAdd(sum + at, x);
            if (sumsq) atomicAdd(sumsq + at, __dmul_rn(x, x));
            if (nnz) atomicAdd(nnz + at, (N)1);
        });
    }
}

int launch_group_gene_sums(const DevChunk &c, const uint32_t *group_of_row, int64_t n_vars, const double *clip,
                           double *sum, double *sumsq, void *nnz, bool narrow, cudaStream_t st) {
    if (c.n_spans == 0) return CREST_OK;
    prof::Scope ps("group_gene_sums_csr", st);
    int64_t blocks = ceil_div(c.n_spans, 8);
    const int64_t cap = (int64_t)device_sms() * 16;
    if (blocks > cap) blocks = cap;
    const unsigned grid = (unsigned)std::max<int64_t>(blocks, 1);
    if (narrow)
        k_group_gene_sums<<<grid, 256, 0, st>>>(c, group_of_row, n_vars, clip, sum, sumsq, static_cast<uint32_t *>(nnz));
    else
        k_group_gene_sums<<<grid, 256, 0, st>>>(c, group_of_row, n_vars, clip, sum, sumsq, static_cast<double *>(nnz));
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

}  // namespace crest
