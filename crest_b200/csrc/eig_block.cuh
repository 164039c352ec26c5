// Kernels of the block eigensolver (k_eig.cu) on its narrow blocks, p <= 64
// columns: the coefficients of one Cholesky-QR pass, the Rayleigh-Ritz
// rotations, and their application to the long block rows.
#pragma once

#include <stdint.h>

namespace crest {
namespace {

constexpr int kBlk = 64;        // widest block these kernels take
constexpr int kBlkMax = 112;    // widest block of the solver
constexpr int kRrThreads = 16 * 32 + 32;  // of k_rr: the blocks' warps and one for the rotations
constexpr int kRotRows = 16;    // rows of V and W per block of k_apply_rot
constexpr int kRotChunk = 32;   // rounds of rotations staged at a time

// What the host reads back after one Rayleigh-Ritz step, in one copy.
struct EigOut {
    double theta[kBlkMax], res[kBlkMax];
    int fail;     // bit 0: a Cholesky factor failed; bit 1: one more pass is needed
    int rounds;   // rotation rounds of the last step
    int ticket;   // blocks of k_apply_rot that have finished
};

// Whether value u of index j stands before value v of index i in descending
// order, the lower index first among equals and NaN last: a total order, so
// ranks by it are a permutation whatever the values are (by u > v alone every
// NaN takes rank 0 and other places of the permutation stay unwritten).
__device__ __forceinline__ bool stands_before(double u, int j, double v, int i) {
    if (isnan(u) || isnan(v)) return !isnan(u) || (isnan(v) && j < i);
    return u > v || (u == v && j < i);
}

// One Cholesky-QR pass on the active columns Ya = V[:, j0 ..) of a block
// whose first j0 columns are orthonormal: from S = V^T Ya (p x q, ld p; its
// first j0 rows T = Vl^T Ya, the rest the Gram matrix of Ya) the coefficients
// Rc (p x q) with V Rc = (Ya - Vl T) R^-1, so a pass costs one product for S
// and one for V Rc whatever j0 is.
//
// B = Ya^T Ya - T^T T is the Gram matrix with the locked directions taken
// out.  It is equilibrated, B' = D B D with D = diag(B)^-1/2 (column scaling
// leaves the span unchanged and removes the norm disparity a Chebyshev
// filter creates), shifted by shift_coef * q >= shift_coef * ||B'||_2, and
// eliminated: B' = U^T P U with unit U and pivots P; R^-1 = D U^-1 P^-1/2.
// The matrices stay in registers: thread (ty, tx) of 16 x 16 holds rows
// ty + 16 a and columns tx + 16 b of B' and of the inverse under
// construction.  Step k needs only column k of one and row k of the other,
// published in a double-buffered shared line, so a step is one barrier, 13
// shared loads, one reciprocal and at most 32 independent updates; the
// kernel is bound by that chain of q steps (one CTA).  (A form with both
// matrices in shared memory, each update waiting for the previous one's
// store, took 75 us per call at q = 64, this one 25 us with its launch.)
//
// out->fail bit 0 (and Rc = the identity, Ya left as it is) when a column is
// zero or a pivot is not positive; bit 1 when this was an unshifted pass and
// a pivot below 1/4, or a column that lay almost wholly in the locked span,
// shows that the columns were not yet nearly orthonormal: the passes so far
// then do not guarantee orthonormal columns to working precision.
__global__ void __launch_bounds__(256) k_ortho_coef(const double *__restrict__ S, int p, int j0, double shift_coef,
                                                    double *__restrict__ Rc, EigOut *out) {
    __shared__ double col[2][kBlk], row[2][kBlk];
    __shared__ double dsc[kBlk], piv_[kBlk];
    __shared__ double T[kBlk * kBlk / 4];   // j0 x q, j0 + q = p <= 64
    __shared__ double Ri[kBlk][kBlk + 1];   // R^-1
    __shared__ int bad, again;
    const int q = p - j0, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    if (tid == 0) bad = again = 0;
    for (int e = tid; e < j0 * q; e += 256) T[e] = S[e % j0 + (int64_t)(e / j0) * p];
    __syncthreads();
    double A[4][4], R[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int i = ty + 16 * a, j = tx + 16 * b;
            double v = i == j ? 1.0 : 0.0;  // rows and columns past q: the identity
            if (i < q && j < q) {
                v = S[j0 + i + (int64_t)j * p];
                const double full = v;
                for (int t = 0; t < j0; ++t) v = fma(-T[t + i * j0], T[t + j * j0], v);
                if (i == j && v < 1e-6 * full) again = 1;
            }
            if (i == j) {
                if (!(v > 0.0)) bad = 1;
                dsc[i] = v > 0.0 ? 1.0 / sqrt(v) : 1.0;
            }
            A[a][b] = v;
            R[a][b] = i == j ? 1.0 : 0.0;
        }
    __syncthreads();
    const double shift = shift_coef * (double)q;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int i = ty + 16 * a, j = tx + 16 * b;
            A[a][b] = i == j ? 1.0 + shift : A[a][b] * dsc[i] * dsc[j];
        }
#pragma unroll
    for (int kb = 0; kb < 4; ++kb) {
        if (16 * kb >= q) break;
        for (int kt = 0; kt < 16; ++kt) {
            const int k = 16 * kb + kt, buf = k & 1;
            if (k >= q) break;
            if (tx == kt)
#pragma unroll
                for (int a = kb; a < 4; ++a) col[buf][ty + 16 * a] = A[a][kb];
            if (ty == kt)
#pragma unroll
                for (int b = 0; b <= kb; ++b) row[buf][tx + 16 * b] = R[kb][b];
            __syncthreads();  // the other buffer is free: its readers passed this barrier after their reads
            const double akk = col[buf][k], piv = akk > 0.0 ? akk : 1.0, rp = 1.0 / piv;
            double cj[4], rj[4], mi[4];
#pragma unroll
            for (int b = kb; b < 4; ++b) cj[b] = col[buf][tx + 16 * b];
#pragma unroll
            for (int b = 0; b <= kb; ++b) rj[b] = row[buf][tx + 16 * b];
#pragma unroll
            for (int a = kb; a < 4; ++a) mi[a] = ty + 16 * a > k ? col[buf][ty + 16 * a] * rp : 0.0;
#pragma unroll
            for (int a = kb; a < 4; ++a) {
#pragma unroll
                for (int b = kb; b < 4; ++b) A[a][b] = fma(-mi[a], cj[b], A[a][b]);
#pragma unroll
                for (int b = 0; b <= kb; ++b) R[a][b] = fma(-mi[a], rj[b], R[a][b]);
            }
            if (tid == 0) {
                if (!(akk > 0.0)) bad = 1;
                if (shift_coef == 0.0 && akk < 0.25) again = 1;
                piv_[k] = piv;
            }
        }
    }
    __syncthreads();
    if (tid < q) piv_[tid] = 1.0 / sqrt(piv_[tid]);
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int c = ty + 16 * a, r = tx + 16 * b;
            if (c >= q || r >= q) continue;
            const double v = bad ? (r == c ? 1.0 : 0.0) : (r <= c ? dsc[r] * R[a][b] * piv_[c] : 0.0);
            Ri[r][c] = v;
            Rc[j0 + r + (int64_t)c * p] = v;
        }
    __syncthreads();
    for (int e = tid; e < j0 * q; e += 256) {
        const int t = e % j0, c = e / j0;
        double v = 0.0;
        if (!bad)
            for (int r = 0; r <= c; ++r) v = fma(-T[t + r * j0], Ri[r][c], v);
        Rc[t + (int64_t)c * p] = v;
    }
    if (tid == 0 && (bad | again)) atomicOr(&out->fail, (bad ? 1 : 0) | (again ? 2 : 0));
}

// ---------------------------------------------------- Rayleigh-Ritz rotations
// Cyclic Jacobi on the symmetric q x q matrix (H + H^T) / 2, padded to an
// even n with a decoupled zero index.  Round-robin ordering: n/2 disjoint
// pairs per round, n - 1 rounds per sweep; in round r pair i couples the
// index in its slot a with the one in its slot b.  Between rounds the
// indices move: a 0 stays, a 1 -> b 0, a i -> a i-1, b i -> b i+1,
// b last -> a last, so after a sweep every index is where it began (a i = i,
// b i = n-1-i).  The matrix is kept by slot position: thread (w, l) owns the
// 2 x 2 block coupling pair l with pair l + w + 1 (mod n/2), reads it from
// fixed, conflict-free addresses, rotates it from both sides and stores its
// elements at the fixed addresses of their next positions in a second
// buffer.  Only one of each pair of symmetric blocks exists.  A rotation is
// skipped when |A_pq| <= n u sqrt(|A_pp A_qq|) (or below 1e-18 ||A||_F):
// below that level it only moves rounding noise around; the solver stops
// after a sweep without rotations, or after max_sweeps.
//
// The eigenvectors are not formed: every round's (c, s) go to `rot`
// (x_a' = c x_a - s x_b, x_b' = s x_a + c x_b), and k_apply_rot applies them
// to the rows of the block.  vals: the diagonal in descending order; perm[i]
// = the place of index i in that order.
//
// One CTA.  A round is the chain of the last warp, which forms the rotations:
// in round r it also computes the one element of the block that couples each
// pair's next indices, so the angles of round r + 1 (two reciprocal square
// roots) are formed while the other warps rotate their blocks, and a round
// takes one barrier.  Its loads are issued before theirs (barrier 1): behind
// the 16 warps' loads they wait 130 ns.  Two sweeps of q = 64 take 67 us;
// angles and blocks in turns between two barriers took 80, and the matrix by
// index with both triangles and the eigenvectors in shared memory 157 (1024
// shared-memory wavefronts a round, here 440).
__device__ __forceinline__ int rr_next(int pos, int half) {  // pos = 2 pair + slot
    const int i = pos >> 1;
    if (pos & 1) return i == half - 1 ? 2 * i : pos + 2;
    return i == 0 ? 0 : i == 1 ? 1 : pos - 2;
}

// Address of the element coupling two positions of different pairs, or of
// the two slots of one pair (area behind the blocks).
constexpr int kRrBlocks = 4 * 16 * 32;
__device__ __forceinline__ int rr_addr(int P, int Q, int half) {
    int i = P >> 1, j = Q >> 1, si = P & 1, sj = Q & 1;
    if (i == j) return kRrBlocks + i;
    int dlt = j - i;
    if (dlt < 0) dlt += half;
    if (2 * dlt > half || (2 * dlt == half && i > j)) {
        const int t = i;
        i = j;
        j = t;
        const int u = si;
        si = sj;
        sj = u;
        dlt = half - dlt;
    }
    return ((si * 2 + sj) * 16 + dlt - 1) * 32 + i;
}

__global__ void __launch_bounds__(kRrThreads) k_rr(const double *__restrict__ H, int q, int ldh, int max_sweeps,
                                                   double2 *__restrict__ rot, double *__restrict__ vals,
                                                   int *__restrict__ perm, EigOut *out) {
    __shared__ double E[2][kRrBlocks + 32];
    __shared__ double D[kBlk];  // diagonal by position, at the end
    __shared__ double2 cs[2][32];
    __shared__ double red[kRrThreads / 32];
    __shared__ int rotated[2];
    const int tid = threadIdx.x, l = tid & 31, w = tid >> 5;
    const int n = q + (q & 1), half = n / 2;
    const bool angles = w == kRrThreads / 32 - 1;  // the warp that forms the rotations
    auto at = [&](int pos) { return pos & 1 ? n - 1 - (pos >> 1) : pos >> 1; };  // index at a position before round 0
    auto val = [&](int r, int c) {
        return r < q && c < q ? 0.5 * (H[r + (int64_t)c * ldh] + H[c + (int64_t)r * ldh]) : 0.0;
    };
    const int dlt = w + 1, lj = l + dlt >= half ? l + dlt - half : l + dlt;
    const bool own = !angles && l < half && 2 * dlt <= half && (2 * dlt < half || l < half - dlt);
    const bool pair = angles && l < half;
    int src = 0, dst[4] = {0, 0, 0, 0};
    double ss = 0.0;
    if (own) {
        src = w * 32 + l;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int P = 2 * l + (e >> 1), Q = 2 * lj + (e & 1);
            const double v = val(at(P), at(Q));
            E[0][src + e * 512] = v;
            ss += 2.0 * v * v;
            dst[e] = rr_addr(rr_next(P, half), rr_next(Q, half), half);
        }
    }
    // of the pair l: its diagonal (app, aqq), its coupling, where the zeroed
    // coupling moves, and the element that couples its next indices (those at
    // positions X and Y): the four elements of that block by address
    double app = 0.0, aqq = 0.0, apq = 0.0;
    int dzero = 0, X = 0, Y = 0, from[4] = {0, 0, 0, 0};
    if (pair) {
        const int P = 2 * l;
        app = val(at(P), at(P));
        aqq = val(at(P + 1), at(P + 1));
        apq = val(at(P), at(P + 1));
        ss += app * app + aqq * aqq + 2.0 * apq * apq;
        dzero = rr_addr(rr_next(P, half), rr_next(P + 1, half), half);
        X = l == 0 ? 0 : l == half - 1 ? P + 1 : P + 2;
        Y = l == 0 ? (half > 1 ? 2 : 1) : P - 1;
#pragma unroll
        for (int e = 0; e < 4; ++e) from[e] = rr_addr((X & ~1) + (e >> 1), (Y & ~1) + (e & 1), half);
    }
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (l == 0) red[w] = ss;
    __syncthreads();
    double floor_abs = 0.0;
    if (angles) {
        double t = 0.0;
        for (int i = 0; i < kRrThreads / 32; ++i) t += red[i];
        floor_abs = 1e-18 * sqrt(t);
    }
    const double eps = (double)n * 0x1.0p-52, eps2 = eps * eps;
    double c = 1.0, s = 0.0, t = 0.0;
    bool any = false;  // a rotation in the sweep of the round formed last
    auto rotation = [&](int round) {
        c = 1.0;
        s = t = 0.0;
        if (pair && fabs(apq) > floor_abs && apq * apq > eps2 * fabs(app * aqq)) {
            // cos 2x = |dd| / h, sin 2x = +-two / h: c = sqrt((1 + cos 2x) / 2),
            // s = sin 2x / (2 c), t = s / c, as two reciprocal square roots
            const double dd = aqq - app, two = 2.0 * apq, rh = rsqrt(fma(dd, dd, two * two));
            const double c2 = fma(0.5 * fabs(dd), rh, 0.5), rc = rsqrt(c2);
            c = c2 * rc;
            s = (dd >= 0.0 ? apq : -apq) * rh * rc;
            t = s * rc;
            any = true;
        }
        if (pair) {
            cs[round & 1][l] = make_double2(c, s);
            rot[(int64_t)round * 32 + l] = make_double2(c, s);
        }
    };
    if (angles) rotation(0);
    const int total = max_sweeps * (n - 1);
    int rounds = 0, left = n - 1, cur = 0;  // rounds left in the sweep
    for (int sweep = 0;;) {
        __syncthreads();  // the matrix before this round and its rotations are complete
        if (angles) {
            // its loads go first: it is the longer chain, and behind the other
            // warps' loads they would wait for all of those
            const double2 x = cs[cur][X >> 1], y = cs[cur][Y >> 1];
            const double *e = E[cur];
            const double m00 = e[from[0]], m01 = e[from[1]], m10 = e[from[2]], m11 = e[from[3]];
            asm volatile("bar.arrive 1, %0;" ::"n"(kRrThreads) : "memory");
            // the pair itself: its coupling becomes zero and moves on with its
            // indices, like its diagonal
            const double g = t != 0.0 ? t * apq : 0.0, a = app - g, b = aqq + g;
            if (pair) E[cur ^ 1][dzero] = t != 0.0 ? 0.0 : apq;
            const double ad = __shfl_down_sync(0xffffffffu, a, 1), bu = __shfl_up_sync(0xffffffffu, b, 1);
            app = l == 0 ? a : l == half - 1 ? b : ad;
            aqq = l == 0 ? ad : bu;
            if (left == 1) {
                const bool sweep_any = __any_sync(0xffffffffu, any);
                if (l == 0) rotated[sweep & 1] = sweep_any;
                any = false;
            }
            const double x0 = X & 1 ? x.y : x.x, x1 = X & 1 ? x.x : -x.y;
            const double y0 = Y & 1 ? y.y : y.x, y1 = Y & 1 ? y.x : -y.y;
            apq = (x0 * m00 + x1 * m10) * y0 + (x0 * m01 + x1 * m11) * y1;
            if (rounds + 1 < total) rotation(rounds + 1);
        } else {
            asm volatile("bar.sync 1, %0;" ::"n"(kRrThreads) : "memory");
            if (own) {
                const double2 ri = cs[cur][l], rj = cs[cur][lj];
                const double *e = E[cur] + src;
                const double m00 = e[0], m01 = e[512], m10 = e[1024], m11 = e[1536];
                const double r00 = ri.x * m00 - ri.y * m10, r01 = ri.x * m01 - ri.y * m11;
                const double r10 = ri.y * m00 + ri.x * m10, r11 = ri.y * m01 + ri.x * m11;
                double *o = E[cur ^ 1];
                o[dst[0]] = rj.x * r00 - rj.y * r01;
                o[dst[1]] = rj.y * r00 + rj.x * r01;
                o[dst[2]] = rj.x * r10 - rj.y * r11;
                o[dst[3]] = rj.y * r10 + rj.x * r11;
            }
        }
        cur ^= 1;
        ++rounds;
        if (--left) continue;
        __syncthreads();
        if (!rotated[sweep & 1] || ++sweep == max_sweeps) break;
        left = n - 1;
    }
    if (pair) {
        D[2 * l] = app;
        D[2 * l + 1] = aqq;
    }
    __syncthreads();
    if (tid < n) {  // index tid sits at its first position again
        const int pos = tid < half ? 2 * tid : 2 * (n - 1 - tid) + 1;
        const double v = D[pos];
        int rank = 0;
        for (int P = 0; P < n; ++P) {
            const int i = at(P);
            if (i < q && stands_before(D[P], i, v, tid)) ++rank;
        }
        if (tid < q) {
            perm[tid] = rank;
            vals[rank] = v;
        }
    }
    if (tid == 0) {
        out->rounds = rounds;
        out->ticket = 0;
    }
}

// Applies the rounds logged by k_rr to the active columns of V and W = C V
// (d x q at ld; columns in index order), puts the columns in Ritz order into
// Vo and Wo, and leaves ||W_j - theta_j V_j|| in res.  A block takes kRotRows
// rows of both; in a warp, lane i holds the pair in slots a i, b i of four
// row vectors in registers, and the move between rounds is two shuffles per
// vector.  This replaces the accumulation of the rotations into a matrix and
// two products with it.  The per-block sums of squares are added in block
// order by the last block to finish.
__global__ void __launch_bounds__(256) k_apply_rot(const double *__restrict__ V, const double *__restrict__ W,
                                                   double *__restrict__ Vo, double *__restrict__ Wo, int64_t ld, int q,
                                                   const double2 *__restrict__ rot, const double *__restrict__ theta,
                                                   const int *__restrict__ perm, double *__restrict__ part,
                                                   double *__restrict__ res, EigOut *out) {
    __shared__ double tile[2][kBlk][kRotRows + 1];
    __shared__ double2 cs[kRotChunk][32];
    __shared__ double red[4][kBlk];
    __shared__ bool last;
    const int tid = threadIdx.x, l = tid & 31, w = tid >> 5;
    const int n = q + (q & 1), half = n / 2;
    const int64_t row0 = (int64_t)blockIdx.x * kRotRows;  // ld is a multiple of kRotRows
    for (int e = tid; e < kRotRows * q; e += 256) {
        const int r = e % kRotRows, c = e / kRotRows;
        tile[0][c][r] = V[row0 + r + c * ld];
        tile[1][c][r] = W[row0 + r + c * ld];
    }
    const int rounds = out->rounds;
    __syncthreads();
    double xa[4], xb[4];
    const int ib = n - 1 - l;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const int r = 2 * w + (v & 1);
        xa[v] = l < half ? tile[v >> 1][l][r] : 0.0;
        xb[v] = l < half && ib < q ? tile[v >> 1][ib][r] : 0.0;
    }
    for (int r0 = 0; r0 < rounds; r0 += kRotChunk) {
        const int nr = min(kRotChunk, rounds - r0);
        __syncthreads();
        for (int e = tid; e < nr * 32; e += 256) cs[e >> 5][e & 31] = rot[(int64_t)r0 * 32 + e];
        __syncthreads();
#pragma unroll 2
        for (int r = 0; r < nr; ++r) {
            const double2 g = cs[r][l];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const double a = g.x * xa[v] - g.y * xb[v], b = g.y * xa[v] + g.x * xb[v];
                const double ad = __shfl_down_sync(0xffffffffu, a, 1), bu = __shfl_up_sync(0xffffffffu, b, 1);
                xa[v] = l == 0 ? a : l == half - 1 ? b : ad;
                xb[v] = l == 0 ? ad : bu;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const int r = 2 * w + (v & 1);
        if (l < half) tile[v >> 1][perm[l]][r] = xa[v];
        if (l < half && ib < q) tile[v >> 1][perm[ib]][r] = xb[v];
    }
    __syncthreads();
    for (int e = tid; e < kRotRows * q; e += 256) {
        const int r = e % kRotRows, c = e / kRotRows;
        Vo[row0 + r + c * ld] = tile[0][c][r];
        Wo[row0 + r + c * ld] = tile[1][c][r];
    }
    const int c = tid & 63, h = tid >> 6;
    double s = 0.0;
    if (c < q) {
        const double th = theta[c];
#pragma unroll
        for (int r = 0; r < kRotRows / 4; ++r) {
            const double e = tile[1][c][h * (kRotRows / 4) + r] - th * tile[0][c][h * (kRotRows / 4) + r];
            s += e * e;
        }
    }
    red[h][c] = s;
    __syncthreads();
    if (tid < kBlk) {
        part[(int64_t)blockIdx.x * kBlk + tid] = red[0][tid] + red[1][tid] + red[2][tid] + red[3][tid];
        __threadfence();
    }
    __syncthreads();
    if (tid == 0) last = atomicAdd(&out->ticket, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // block order within each of four interleaved groups, then the groups
    double t = 0.0;
    for (unsigned b = h; b < gridDim.x; b += 4) t += __ldcg(part + (int64_t)b * kBlk + c);
    red[h][c] = t;
    __syncthreads();
    if (tid < q) res[tid] = sqrt(red[0][tid] + red[1][tid] + red[2][tid] + red[3][tid]);
}

// X = alpha W + beta V over n elements (the first step of the filter recurrence).
__global__ void k_axpby(const double *__restrict__ W, const double *__restrict__ V, double alpha, double beta, int64_t n,
                        double *__restrict__ X) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) X[i] = alpha * W[i] + beta * V[i];
}

}  // namespace
}  // namespace crest
