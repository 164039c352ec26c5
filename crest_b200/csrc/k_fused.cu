// K7: the differentiable normalise -> log1p -> scale -> project map and its
// backward, for training-style use of the PCA projection (no counterpart in
// the reference; the forward arithmetic is the reference's transform).
//
// Input: a CSR matrix over d genes (HVG columns already selected) with
// per-cell size factors sf, loadings W (d x k, row-major), fixed per-gene
// mean / std of the scale step and its clip value.  Per stored entry e of
// cell c and gene g (the size factor divides, y = x / sf):
//
//   y = x / sf_c                      (f32, correctly rounded)
//   l = log1pf(y)                     (f32, glibc's algorithm)
//   z = (l - mean_g) / std_g          (f64)
//   s = clip(z) - clip(-mean_g / std_g)
//   score[c, :] = sum_e s_e W[g_e, :] (f64 accumulation, stored as f32)
//
// Backward, given G = dL/dscore (n x k):
//   dL/ds_e  = G[c, :] . W[g_e, :]
//   dL/dz_e  = dL/ds_e  when -max <= z <= max (or no clipping), else 0
//   dL/dy_e  = dL/dz_e / (std_g (1 + y))
//   dL/dx_e  = dL/dy_e / sf_c
//   dL/dsf_c = - sum_e dL/dy_e y_e / sf_c
//   dL/dW[g, :] = sum over entries of gene g of s_e G[c_e, :]
// log1p and the scaled values are recomputed in the backward pass.  The W
// gradient is formed gene by gene: a per-gene histogram of the entries and
// its scan give every gene a segment, the entry pass writes (s_e, c_e) of
// each entry into its gene's segment (counting sort; the order inside a
// segment is not fixed), and a warp per chunk of a segment sums s_e G[c_e, :]
// in f64.
#include "host.cuh"
#include "prof.cuh"
#include "rowwarp.cuh"

namespace crest {
namespace {

struct FusedArgs {
    const int64_t *indptr;
    const int32_t *indices;
    const float *values;
    int64_t n, d;
    const float *sf;
    const float *W;
    int k;
    const double *mean, *std;
    double max_value;
    int *bad;  // set when a gene id is outside [0, d)
};

// (s, pass, y) of one entry; pass is the clip derivative (1 inside the band).
__device__ __forceinline__ double fused_value(const FusedArgs &a, int32_t g, float x, float sfc, float &y,
                                              double &pass) {
    y = __fdiv_rn(x, sfc);
    const float l = crest_log1pf(y);
    const double mu = __ldg(a.mean + g), sd = __ldg(a.std + g);
    const double z = __ddiv_rn(__dsub_rn((double)l, mu), sd);
    const double mv = a.max_value;
    pass = (mv > 0.0 && (z < -mv || z > mv)) ? 0.0 : 1.0;
    return __dsub_rn(clip_mv(z, mv), clip_mv(__ddiv_rn(-mu, sd), mv));
}

// Rows of W and G are read from copies padded with zeros to 4 LPR floats
// (LPR = 8, 16 or 32 lanes, k <= 32, 64 or 128): LPR lanes take a row as one
// 16-byte load each, so a row is whole 128-byte lines and a warp works on
// 32 / LPR entries at a time, four columns per lane.  The copy has a row 0
// even when there are no rows (d = 0): slots without an entry, and entries
// whose gene id is outside [0, d), load that row and drop what they load.
// The launch also clears the call's flag (`clear`, when it has no other fill):
// a fill of its own costs a small call 2 us.
__global__ void k_pad_rows(const float *__restrict__ in, int64_t rows, int64_t rows_out, int k, int kp,
                           float *__restrict__ out, int *clear) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0 && clear) *clear = 0;
    if (i >= rows_out * kp) return;
    const int64_t r = i / kp;
    const int j = (int)(i - r * kp);
    out[i] = r < rows && j < k ? in[r * k + j] : 0.0f;
}

// One entry of the W gradient: s_e and its cell.
struct __align__(16) EntryCell {
    double s;
    int32_t cell;
    int32_t pad;
};

// One entry as a warp hands it round through shared memory: its factor and
// its row.
struct __align__(16) EntryRow {
    double s;
    int64_t row;
};

constexpr int kFly = 8;  // rows in flight per lane: loaded before their products are added

// acc += the sum over `cnt` entries of ent[] of s * row of `base`, each group
// of LPR lanes taking every (32 / LPR)-th entry.
template <int LPR>
__device__ __forceinline__ void add_rows(const EntryRow *ent, int cnt, const float4 *__restrict__ base, int lane,
                                         double (&acc)[4]) {
    constexpr int SUBS = 32 / LPR;
    const int sub = lane / LPR;
    const float4 *col = base + lane % LPR;
    for (int u = 0; u < cnt; u += kFly * SUBS) {
        float4 w[kFly];
        if (u + kFly * SUBS <= cnt) {
#pragma unroll
            for (int t = 0; t < kFly; ++t) w[t] = __ldg(col + ent[u + t * SUBS + sub].row * LPR);
#pragma unroll
            for (int t = 0; t < kFly; ++t) {
                const double s = ent[u + t * SUBS + sub].s;
                acc[0] = fma(s, (double)w[t].x, acc[0]);
                acc[1] = fma(s, (double)w[t].y, acc[1]);
                acc[2] = fma(s, (double)w[t].z, acc[2]);
                acc[3] = fma(s, (double)w[t].w, acc[3]);
            }
        } else {  // the last entries, guarded
#pragma unroll
            for (int t = 0; t < kFly; ++t)
                if (u + t * SUBS + sub < cnt) w[t] = __ldg(col + ent[u + t * SUBS + sub].row * LPR);
#pragma unroll
            for (int t = 0; t < kFly; ++t) {
                if (u + t * SUBS + sub >= cnt) continue;
                const double s = ent[u + t * SUBS + sub].s;
                acc[0] = fma(s, (double)w[t].x, acc[0]);
                acc[1] = fma(s, (double)w[t].y, acc[1]);
                acc[2] = fma(s, (double)w[t].z, acc[2]);
                acc[3] = fma(s, (double)w[t].w, acc[3]);
            }
        }
    }
}
// The groups' sums together, in every lane.
template <int LPR>
__device__ __forceinline__ void add_groups(double (&acc)[4]) {
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] += __shfl_xor_sync(kFull, acc[q], o);
}

// Cells are spread one to a warp, or one to a block of kCellWarps warps that
// take its 32-entry segments in turn: a warp needs about 5 us per segment, a
// chain of loads and divisions, so with few cells the segments of a cell are
// the parallelism (512 cells x 175 entries: forward 38 -> 10 us, entry pass of
// the backward 44 -> 14 us).
constexpr int kCellWarps = 8;

template <int LPR, int WPC>
struct CellLoop {
    int64_t first, step;  // cells
    int seg;              // this warp's first segment of a cell, and then every WPC-th
    __device__ __forceinline__ CellLoop()
        : first(WPC == 1 ? ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5 : blockIdx.x),
          step(WPC == 1 ? ((int64_t)gridDim.x * blockDim.x) >> 5 : gridDim.x),
          seg(WPC == 1 ? 0 : threadIdx.x >> 5) {}
};

// Each 32-entry segment is transformed lane-parallel and handed round through
// shared memory; each group of lanes folds its entries into its scores, the
// groups' (and warps') sums are added at the end.  Bound by the row loads (two
// lines per entry at k = 50) and the conversions of W to double: 50,000 cells
// x 186 entries, k = 50: 411 us with a row as two loads by the whole warp and
// (gene, value) broadcast by shuffles, 295 us this way (at 64 registers; with
// 96 the lower occupancy costs 80 us).
template <int LPR, int WPC>
__global__ void __launch_bounds__(256, 4) k_fused_fwd(FusedArgs a, const float4 *__restrict__ Wp,
                                                      float *__restrict__ scores) {
    __shared__ EntryRow ent[8][32];
    __shared__ double part[WPC == 1 ? 1 : 8][4 * LPR];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const CellLoop<LPR, WPC> cells;
    for (int64_t c = cells.first; c < a.n; c += cells.step) {
        const int64_t lo = a.indptr[c] + 32 * cells.seg, hi = a.indptr[c + 1];
        const float sfc = a.sf[c];
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        int32_t gn = 0;  // the next segment's entry is fetched while this one is folded
        float xn = 0.0f;
        if (lo + lane < hi) {
            gn = __ldg(a.indices + lo + lane);
            xn = __ldg(a.values + lo + lane);
        }
        for (int64_t s0 = lo; s0 < hi; s0 += 32 * WPC) {
            const int64_t e = s0 + lane;
            const int32_t g = gn;
            const float x = xn;
            if (e + 32 * WPC < hi) {
                gn = __ldg(a.indices + e + 32 * WPC);
                xn = __ldg(a.values + e + 32 * WPC);
            }
            EntryRow ec{0.0, 0};
            if (e < hi) {
                if (g >= 0 && g < a.d) {
                    float y;
                    double pass;
                    ec.s = fused_value(a, g, x, sfc, y, pass);
                    ec.row = g;
                } else {  // out-of-range gene id: reported, contributes nothing
                    *a.bad = 1;
                }
            }
            __syncwarp();
            ent[wid][lane] = ec;
            __syncwarp();
            add_rows<LPR>(ent[wid], hi - s0 < 32 ? (int)(hi - s0) : 32, Wp, lane, acc);
        }
        add_groups<LPR>(acc);
        if (WPC == 1) {
            if (lane < LPR)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (4 * lane + q < a.k) scores[c * a.k + 4 * lane + q] = __double2float_rn(acc[q]);
        } else {
            if (lane < LPR)
#pragma unroll
                for (int q = 0; q < 4; ++q) part[WPC == 1 ? 0 : wid][4 * lane + q] = acc[q];
            __syncthreads();
            for (int j = threadIdx.x; j < a.k; j += blockDim.x) {
                double v = 0.0;
#pragma unroll
                for (int w = 0; w < WPC; ++w) v += part[w][j];
                scores[c * a.k + j] = __double2float_rn(v);
            }
            __syncthreads();
        }
    }
}

// Per-gene entry counts: block-private counters in shared memory when d
// fits (kHistSmem genes), else global atomics; ids outside [0, d) are left
// out (the entry pass reports them).
constexpr int kHistSmem = 12288;

__global__ void __launch_bounds__(256) k_gene_hist(const int32_t *__restrict__ indices, int64_t nnz, int64_t d,
                                                   int32_t *__restrict__ count) {
    __shared__ int32_t s_cnt[kHistSmem];
    const bool priv = d <= kHistSmem;
    if (priv)
        for (int64_t g = threadIdx.x; g < d; g += blockDim.x) s_cnt[g] = 0;
    __syncthreads();
    const int64_t per = ceil_div(nnz, (int64_t)gridDim.x);
    const int64_t e0 = per * blockIdx.x, e1 = e0 + per < nnz ? e0 + per : nnz;
    for (int64_t e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
        const int32_t g = __ldg(indices + e);
        if (g < 0 || g >= d) continue;
        if (priv)
            atomicAdd(s_cnt + g, 1);
        else
            atomicAdd(count + g, 1);
    }
    __syncthreads();
    if (priv)
        for (int64_t g = threadIdx.x; g < d; g += blockDim.x)
            if (s_cnt[g]) atomicAdd(count + g, s_cnt[g]);
}

// The W gradient takes a gene's entries in chunks, a warp each: 256, or fewer
// (a multiple of 32) when that leaves the chip's warps without one.
inline int entry_chunk(int64_t nnz) {
    int64_t c = 256;
    while (c > 32 && nnz < c * 64 * device_sms()) c /= 2;
    return (int)c;
}

// Exclusive scans of the per-gene counts and of their chunks (one block):
// offsets[0..d] and chunks[0..d].
__global__ void __launch_bounds__(1024) k_scan_counts(const int32_t *count, int64_t d, int chunk, int64_t *offsets,
                                                      int32_t *chunks) {
    __shared__ int64_t part[32];
    __shared__ int32_t cpart[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t per = (d + 1023) / 1024, b0 = tid * per, b1 = b0 + per < d ? b0 + per : d;
    int64_t s = 0;
    int32_t cs = 0;
    for (int64_t i = b0; i < b1; ++i) {
        s += count[i];
        cs += (count[i] + chunk - 1) / chunk;
    }
    int64_t inc = s;
    int32_t cinc = cs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t t = __shfl_up_sync(kFull, inc, o);
        const int32_t ct = __shfl_up_sync(kFull, cinc, o);
        if (lane >= o) {
            inc += t;
            cinc += ct;
        }
    }
    if (lane == 31) {
        part[wid] = inc;
        cpart[wid] = cinc;
    }
    __syncthreads();
    int64_t run = inc - s;
    int32_t crun = cinc - cs;
    for (int w = 0; w < wid; ++w) {
        run += part[w];
        crun += cpart[w];
    }
    for (int64_t i = b0; i < b1; ++i) {
        offsets[i] = run;
        chunks[i] = crun;
        run += count[i];
        crun += (count[i] + chunk - 1) / chunk;
    }
    if (tid == 1023) {  // the last thread's running sums are the totals, whatever its share was
        offsets[d] = run;
        chunks[d] = crun;
    }
}

// Sums over groups of LPR lanes of 8 values per lane: lane l of a group ends
// with the sum of value l / (LPR / 8).
template <int LPR>
__device__ __forceinline__ double group_sums8(double (&p)[8], int lane) {
#pragma unroll
    for (int h = 4; h; h >>= 1) {
        const int o = LPR / 8 * h;
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double mine = up ? p[i + h] : p[i], other = up ? p[i] : p[i + h];
            p[i] = mine + __shfl_xor_sync(kFull, other, o);
        }
    }
    double v = p[0];
#pragma unroll
    for (int o = LPR / 16; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// Entry pass of the backward: dL/dx and dL/dsf, and (s_e, c) of every entry
// into its gene's segment.  The transform and the gradients of
// 32 entries are lane-parallel; their dot products with the cell's row of G
// (four columns per lane, as double) take the W rows like the forward pass
// and are summed over a group's lanes eight steps at a time.  Bound by
// instruction issue: 50,000 cells x 186 entries, k = 50: 489 us with a lane
// reading its entry's whole W row 16 bytes at a time (32 lines per load),
// 413 us this way.
template <int LPR, int WPC>
__global__ void __launch_bounds__(256, 4) k_fused_bwd_entries(FusedArgs a, const float4 *__restrict__ Wp,
                                                           const float4 *__restrict__ Gp, float *__restrict__ grad_x,
                                                           float *__restrict__ grad_sf,
                                                           const int64_t *__restrict__ offsets,
                                                           int32_t *__restrict__ fill, EntryCell *__restrict__ by_gene) {
    constexpr int SUBS = 32 / LPR, kStep = 8 * SUBS;
    __shared__ int32_t row_of[8][32];
    __shared__ double dsf_part[8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, sub = lane / LPR;
    const CellLoop<LPR, WPC> cells;
    const float4 *col = Wp + lane % LPR;
    // where the sum of this lane's entry (step lane / SUBS of group lane % SUBS) is found
    const int src = lane % SUBS * LPR + lane / SUBS % 8 * (LPR / 8);
    for (int64_t c = cells.first; c < a.n; c += cells.step) {
        const float4 g4 = __ldg(Gp + c * LPR + lane % LPR);
        const double gr[4] = {(double)g4.x, (double)g4.y, (double)g4.z, (double)g4.w};
        const int64_t lo = a.indptr[c] + 32 * cells.seg, hi = a.indptr[c + 1];
        const float sfc = a.sf[c];
        double dsf = 0.0;
        int32_t gn = 0;
        float xn = 0.0f;
        if (lo + lane < hi) {
            gn = __ldg(a.indices + lo + lane);
            xn = __ldg(a.values + lo + lane);
        }
        for (int64_t s0 = lo; s0 < hi; s0 += 32 * WPC) {
            const int64_t e = s0 + lane;
            const int cnt = hi - s0 < 32 ? (int)(hi - s0) : 32;
            const int32_t g = gn;
            const float x = xn;
            if (e + 32 * WPC < hi) {
                gn = __ldg(a.indices + e + 32 * WPC);
                xn = __ldg(a.values + e + 32 * WPC);
            }
            const bool ok = e < hi && g >= 0 && g < a.d;
            __syncwarp();
            row_of[wid][lane] = ok ? g : 0;  // row 0 where there is no entry: its sum is not used
            __syncwarp();
            double gs = 0.0;
            for (int f = 0; f < cnt; f += kStep) {
                float4 w[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) w[t] = __ldg(col + (int64_t)row_of[wid][f + t * SUBS + sub] * LPR);
                double p[8];
#pragma unroll
                for (int t = 0; t < 8; ++t)
                    p[t] = fma(gr[3], (double)w[t].w,
                               fma(gr[2], (double)w[t].z, fma(gr[1], (double)w[t].y, gr[0] * (double)w[t].x)));
                const double sum = __shfl_sync(kFull, group_sums8<LPR>(p, lane), src);
                if (lane / kStep == f / kStep) gs = sum;
            }
            if (e >= hi) continue;
            if (!ok) {  // out-of-range gene id: reported, no gradient
                *a.bad = 1;
                grad_x[e] = 0.0f;
                continue;
            }
            float y;
            double pass;
            EntryCell ec;
            ec.s = fused_value(a, g, x, sfc, y, pass);
            const double dy = gs * pass / (__ldg(a.std + g) * (1.0 + (double)y));
            grad_x[e] = (float)(dy / (double)sfc);
            dsf -= dy * (double)y / (double)sfc;
            ec.cell = (int32_t)c;
            ec.pad = 0;
            by_gene[offsets[g] + atomicAdd(fill + g, 1)] = ec;
        }
        dsf = warp_sum(dsf);
        if (WPC == 1) {
            if (lane == 0) grad_sf[c] = (float)dsf;
        } else {
            if (lane == 0) dsf_part[wid] = dsf;
            __syncthreads();
            if (threadIdx.x == 0) {
                double v = 0.0;
#pragma unroll
                for (int w = 0; w < WPC; ++w) v += dsf_part[w];
                grad_sf[c] = (float)v;
            }
            __syncthreads();
        }
    }
}

// dL/dW[g, :] = sum over gene g's segment of s_e G[c_e, :], a warp per chunk
// of the entries of one gene, so that genes of any length spread over the
// chip; a chunk's partial row is added to the gene's double row with one
// atomic per column.  The gathers of G rows from L2 bound it.  9.3M entries,
// k = 50: 1040 us with a block per gene, 200 us this way.
template <int LPR>
__global__ void __launch_bounds__(256, 4) k_fused_bwd_w(int64_t d, int k, int chunk, const int64_t *__restrict__ offsets,
                                                     const int32_t *__restrict__ chunks,
                                                     const EntryCell *__restrict__ by_gene,
                                                     const float4 *__restrict__ Gp, double *__restrict__ sum_W) {
    __shared__ EntryRow ent[8][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int32_t total = chunks[d];
    for (int64_t ch = warp; ch < total; ch += n_warps) {
        int64_t g0 = 0, g1 = d;  // the gene whose chunks include ch: chunks[g] <= ch < chunks[g + 1]
        while (g1 - g0 > 1) {
            const int64_t mid = (g0 + g1) >> 1;
            if (__ldg(chunks + mid) <= ch)
                g0 = mid;
            else
                g1 = mid;
        }
        const int64_t t0 = offsets[g0] + (ch - __ldg(chunks + g0)) * chunk;
        const int64_t t1 = t0 + chunk < offsets[g0 + 1] ? t0 + chunk : offsets[g0 + 1];
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        EntryCell next{0.0, 0, 0};
        if (t0 + lane < t1) next = by_gene[t0 + lane];
        for (int64_t b = t0; b < t1; b += 32) {
            __syncwarp();
            ent[wid][lane] = EntryRow{next.s, next.cell};
            if (b + 32 + lane < t1) next = by_gene[b + 32 + lane];
            __syncwarp();
            add_rows<LPR>(ent[wid], t1 - b < 32 ? (int)(t1 - b) : 32, Gp, lane, acc);
        }
        add_groups<LPR>(acc);
        if (lane < LPR)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (4 * lane + q < k) atomicAdd(sum_W + g0 * k + 4 * lane + q, acc[q]);
    }
}

__global__ void k_to_float(const double *__restrict__ in, int64_t n, float *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)in[i];
}

// A block per cell while all cells' blocks are resident at once (four a SM):
// then it costs nothing even where a cell has one segment.  Beyond, it pays
// where cells have several segments, which the backward knows (nnz): up to 64
// cells an SM when they average 128 entries or more.  Warp against block per
// cell, backward up to the W gradient: k = 50, 900 cells x 190 entries 52 against
// 38 us, 4,736 x 190 153 / 114, 9,600 x 190 242 / 196, 9,600 x 128 174 / 151,
// 20,000 x 128 302 / 280 but 229 / 259 at k = 100; 1,200 x 60 36 / 36, 2,400 x 60
// 42 / 44, 2,400 x 20 31 / 43.  Forward: 592 x 190 28 / 15, 1,200 x 190 28 / 21,
// 4,736 x 190 44 / 49, 600 x 20 17 / 20, 1,200 x 20 18 / 22: less to win and no
// count of the entries at hand, so it keeps the first line.
bool cell_per_block(int64_t n) { return n <= (int64_t)device_sms() * 4; }
bool cell_per_block(int64_t n, int64_t nnz) {
    return cell_per_block(n) || (n <= (int64_t)device_sms() * 64 && nnz >= 128 * n);
}

int grid_warps(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 8), device_sms() * 16)); }

struct FusedWork {
    DevBuf by_gene, offsets, chunks, wpad, gpad;
    DevBuf zeroed;  // cleared by one fill at the start of a call
    DevBuf bad;
    HostBuf host;   // pinned, for the few bytes a call reads back
};

// fn<LPR> for rows padded to kp columns, fn<LPR, WPC> with a cell per warp or per block
#define CREST_FUSED_LAUNCH(fn, kp, grid, st, ...)                           \
    do {                                                                    \
        if ((kp) == 32) fn<8><<<(grid), 256, 0, (st)>>>(__VA_ARGS__);       \
        else if ((kp) == 64) fn<16><<<(grid), 256, 0, (st)>>>(__VA_ARGS__); \
        else fn<32><<<(grid), 256, 0, (st)>>>(__VA_ARGS__);                 \
    } while (0)
#define CREST_FUSED_CELLS_W(fn, kp, wpc, grid, st, ...)                          \
    do {                                                                         \
        if ((kp) == 32) fn<8, wpc><<<(grid), 256, 0, (st)>>>(__VA_ARGS__);       \
        else if ((kp) == 64) fn<16, wpc><<<(grid), 256, 0, (st)>>>(__VA_ARGS__); \
        else fn<32, wpc><<<(grid), 256, 0, (st)>>>(__VA_ARGS__);                 \
    } while (0)
#define CREST_FUSED_CELLS(fn, kp, n, by_block, st, ...)                                           \
    do {                                                                                          \
        if (by_block) CREST_FUSED_CELLS_W(fn, kp, kCellWarps, (unsigned)(n), st, __VA_ARGS__); \
        else CREST_FUSED_CELLS_W(fn, kp, 1, grid_warps(n), st, __VA_ARGS__);                      \
    } while (0)

int padded_columns(int64_t k) { return k <= 32 ? 32 : k <= 64 ? 64 : 128; }

int pad_rows(const float *in, int64_t rows, int64_t k, int kp, DevBuf &buf, cudaStream_t st, int *clear = nullptr) {
    const int64_t rows_out = std::max<int64_t>(rows, 1);
    CREST_TRY(buf.ensure(sizeof(float) * (size_t)(rows_out * kp)));
    k_pad_rows<<<(unsigned)ceil_div(rows_out * kp, 256), 256, 0, st>>>(in, rows, rows_out, (int)k, kp, buf.as<float>(),
                                                                          clear);
    CREST_CUDA_TRY(cudaGetLastError());
    return CREST_OK;
}

FusedWork &fused_work(int dev) {
    static thread_local FusedWork ws[64];
    return ws[dev];
}

int bad_ids(FusedWork &w, const int *flag, cudaStream_t st) {
    CREST_TRY(w.host.ensure(sizeof(int)));
    int &h = *w.host.as<int>();
    CREST_CUDA_TRY(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    CREST_CUDA_TRY(cudaStreamSynchronize(st));
    CREST_REQUIRE(h == 0, CREST_EINVAL, "fused map: indices must be gene ids in [0, d)");
    return CREST_OK;
}

int current_device(int *dev) {
    CREST_CUDA_TRY(cudaGetDevice(dev));
    CREST_REQUIRE(*dev >= 0 && *dev < 64, CREST_ERUNTIME, "device index %d out of range", *dev);
    return CREST_OK;
}

int check_fused(const FusedArgs &a) {
    CREST_REQUIRE(a.n >= 0 && a.d >= 0 && a.k >= 1 && a.k <= 128, CREST_EINVAL,
                  "fused map: need n, d >= 0 and 1 <= k <= 128 (k=%d)", a.k);
    CREST_REQUIRE(a.indptr && a.sf && a.W && a.mean && a.std, CREST_EINVAL, "fused map: NULL argument");
    return CREST_OK;
}

}  // namespace
}  // namespace crest

using namespace crest;

extern "C" int crest_fused_forward(const int64_t *indptr, const int32_t *indices, const float *values, int64_t n,
                                   int64_t d, const float *size_factors, const float *W, int64_t k,
                                   const double *mean, const double *std, double max_value, float *scores) {
    FusedArgs a{indptr, indices, values, n, d, size_factors, W, (int)k, mean, std, max_value, nullptr};
    CREST_TRY(check_fused(a));
    CREST_REQUIRE(scores, CREST_EINVAL, "fused map: NULL scores");
    CREST_TRY(require_device());
    if (n == 0) return CREST_OK;
    int dev = 0;
    CREST_TRY(current_device(&dev));
    FusedWork &w = fused_work(dev);
    cudaStream_t st = cudaStreamPerThread;
    CREST_TRY(w.bad.ensure(sizeof(int)));
    a.bad = w.bad.as<int>();
    {
        prof::Scope ps("fused_fwd", st);
        const int kp = padded_columns(k);
        CREST_TRY(pad_rows(W, d, k, kp, w.wpad, st, a.bad));
        CREST_FUSED_CELLS(k_fused_fwd, kp, n, cell_per_block(n), st, a, w.wpad.as<float4>(), scores);
    }
    CREST_CUDA_TRY(cudaGetLastError());
    return bad_ids(w, a.bad, st);
}

extern "C" int crest_fused_backward(const int64_t *indptr, const int32_t *indices, const float *values, int64_t n,
                                    int64_t d, const float *size_factors, const float *W, int64_t k,
                                    const double *mean, const double *std, double max_value,
                                    const float *grad_scores, float *grad_values, float *grad_sf, float *grad_W) {
    FusedArgs a{indptr, indices, values, n, d, size_factors, W, (int)k, mean, std, max_value, nullptr};
    CREST_TRY(check_fused(a));
    CREST_REQUIRE(grad_scores && grad_values && grad_sf && grad_W, CREST_EINVAL, "fused map: NULL gradient");
    CREST_TRY(require_device());
    int dev = 0;
    CREST_TRY(current_device(&dev));
    FusedWork &w = fused_work(dev);
    cudaStream_t st = cudaStreamPerThread;
    int64_t nnz = 0, p0 = 0;
    if (n > 0) {
        CREST_TRY(w.host.ensure(2 * sizeof(int64_t)));
        int64_t *ends = w.host.as<int64_t>();
        CREST_CUDA_TRY(cudaMemcpyAsync(ends, indptr, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        CREST_CUDA_TRY(cudaMemcpyAsync(ends + 1, indptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        CREST_CUDA_TRY(cudaStreamSynchronize(st));
        p0 = ends[0];
        nnz = ends[1];
    }
    CREST_REQUIRE(p0 == 0 && nnz >= 0 && nnz < ((int64_t)1 << 31), CREST_EINVAL,
                  "fused map: indptr must start at 0 and hold < 2^31 entries");
    // [sums of dW (f64, d x k)] [entries per gene] [entries placed per gene] [bad flag]
    const size_t at_count = sizeof(double) * (size_t)(d * k), at_fill = at_count + sizeof(int32_t) * (size_t)d,
                 at_bad = at_fill + sizeof(int32_t) * (size_t)d, zeroed = at_bad + sizeof(int);
    CREST_TRY(w.zeroed.ensure(zeroed));
    CREST_TRY(w.by_gene.ensure(sizeof(EntryCell) * (size_t)std::max<int64_t>(nnz, 1)));
    CREST_TRY(w.offsets.ensure(sizeof(int64_t) * (size_t)(d + 1)));
    CREST_TRY(w.chunks.ensure(sizeof(int32_t) * (size_t)(d + 1)));
    CREST_CUDA_TRY(cudaMemsetAsync(w.zeroed.ptr, 0, zeroed, st));
    unsigned char *z = w.zeroed.as<unsigned char>();
    double *sum_W = reinterpret_cast<double *>(z);
    int32_t *count = reinterpret_cast<int32_t *>(z + at_count), *fill = reinterpret_cast<int32_t *>(z + at_fill);
    a.bad = reinterpret_cast<int *>(z + at_bad);
    int64_t *offsets = w.offsets.as<int64_t>();
    int32_t *chunks = w.chunks.as<int32_t>();
    EntryCell *by_gene = w.by_gene.as<EntryCell>();
    const int kp = padded_columns(k), chunk = entry_chunk(nnz);
    {
        prof::Scope ps("fused_bwd", st);
        if (d > 0) {
            if (nnz)
                k_gene_hist<<<(unsigned)std::min<int64_t>(ceil_div(nnz, 1024), device_sms() * 4), 256, 0, st>>>(
                    indices, nnz, d, count);
            k_scan_counts<<<1, 1024, 0, st>>>(count, d, chunk, offsets, chunks);
        }
        CREST_TRY(pad_rows(W, d, k, kp, w.wpad, st));
        CREST_TRY(pad_rows(grad_scores, n, k, kp, w.gpad, st));
        if (n > 0)
            CREST_FUSED_CELLS(k_fused_bwd_entries, kp, n, cell_per_block(n, nnz), st, a, w.wpad.as<float4>(),
                              w.gpad.as<float4>(), grad_values, grad_sf, offsets, fill, by_gene);
        CREST_CUDA_TRY(cudaGetLastError());
    }
    if (d > 0) {
        prof::Scope ps("fused_bwd_w", st);
        const int64_t most = nnz / chunk + std::min(d, nnz);  // chunks, at most
        const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(ceil_div(most, 8), (int64_t)device_sms() * 16));
        CREST_FUSED_LAUNCH(k_fused_bwd_w, kp, (unsigned)blocks, st, d, (int)k, chunk, offsets, chunks, by_gene,
                           w.gpad.as<float4>(), sum_W);
        k_to_float<<<(unsigned)ceil_div(d * k, 256), 256, 0, st>>>(sum_W, d * k, grad_W);
        CREST_CUDA_TRY(cudaGetLastError());
    }
    return bad_ids(w, a.bad, st);
}
