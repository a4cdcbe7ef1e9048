// Persistent cooperative Cholesky factorisation, and the inverse of the factor alongside.
//
// One cooperative launch covers the whole factorisation: for every 64-column panel, block 0
// factors the diagonal block (and inverts it), all blocks solve the panel rows, then update the
// trailing lower triangle tile by tile on the DMMA path. Block 0's chain (its first rows of the
// panel, the next diagonal block) sets the time; the blocks signal one another through counters
// and wait only for what they read. A failed pivot (non-positive or NaN, the dpotrf test used by
// the reference's positive-definiteness checks, linalg/hdsdp_linsolver.c:521-553) is stored
// in *info and published with the diagonal block's signal, at which every block leaves. The status
// and sum log L_ii go to the host from the same launch.
//
// Measured (factor only / with K = L^-1, ms, copy and status included): order 64 0.038 / 0.048
// -> 0.017 / 0.021, 200 0.111 / 0.123 -> 0.049 / 0.061, 500 0.205 / 0.222 -> 0.105 / 0.115,
// 1000 0.394 / 0.408 -> 0.209 / 0.226, 2000 0.782 / 0.957 -> 0.529 / 0.754 (before: shuffled
// 16-column sweeps, two grid barriers a panel, five launches a factorisation).
//
// K = L^-1, where it is wanted, is formed by block rows one panel behind: K_i = Dinv_i X_i, then
// X_below -= L_below,i K_i.
#include "la.h"
#include <cooperative_groups.h>
#include <mutex>
#include <algorithm>
#include <vector>
#include <utility>

namespace cg = cooperative_groups;

namespace hb {

#ifdef HB_CHOL_STAMPS
// Diagnostic build only (never defined in the library build): per-phase %globaltimer
// stamps of the cooperative factorisation, written by thread 0 of a block.
__device__ unsigned long long *g_chol_stamps = nullptr;
void chol_set_stamps(unsigned long long *p) { cudaMemcpyToSymbol(g_chol_stamps, &p, sizeof(p)); }
#define CHOL_STAMP(slot)                                                  \
    do {                                                                  \
        if (threadIdx.x == 0 && g_chol_stamps && (slot) < 8192) {         \
            unsigned long long t_;                                        \
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));        \
            g_chol_stamps[(slot)] = t_;                                   \
        }                                                                 \
    } while (0)
#else
#define CHOL_STAMP(slot) \
    do {                 \
    } while (0)
#endif

namespace {
constexpr int NB = 64;

constexpr int TP = 68;                         // tile pitch (conflict-free DMMA fragment reads)
constexpr int SM_DOUBLES = 4 * 64 * TP;        // four 64 x 68 tiles
constexpr int COOP_THREADS = 256;

__device__ __forceinline__ void cpa8(double *sdst, const double *gsrc, bool pred) {
    const unsigned saddr = (unsigned) __cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(gsrc), "r"(pred ? 8 : 0));
}
__device__ __forceinline__ void cpa_wait_all() {
    asm volatile("cp.async.commit_group;\n" ::);
    asm volatile("cp.async.wait_group 0;\n" ::);
}

// 16-byte copy of which the first `bytes` (0, 8 or 16) come from global memory and the
// rest is zero filled; both addresses 16-byte aligned.
__device__ __forceinline__ void cpa16(double *sdst, const double *gsrc, int bytes) {
    const unsigned saddr = (unsigned) __cvta_generic_to_shared(sdst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(saddr), "l"(gsrc), "r"(bytes));
}

// Stage columns 0..ncols-1 of the R-row tile G (column-major, pitch ldg) into S (pitch PS):
// entries with row < nr and column < nc are copied, the rest of those columns is zero. Two rows
// move per copy when G and ldg keep every pair 16-byte aligned. With `lower` the entries above
// the diagonal (zeros in global memory) are not fetched. The caller waits with cpa_wait_all().
template <int R = 64, int PS = TP>
__device__ __forceinline__ void stage_tile(double *S, const double *G, long ldg, int nr, int nc, int ncols,
                                           bool lower = false) {
    if (((((size_t) G) & 15) == 0) && ((ldg & 1) == 0)) {
#pragma unroll 4
        for (int idx = threadIdx.x; idx < (R / 2) * ncols; idx += blockDim.x) {
            const int r = (idx % (R / 2)) * 2, c = idx / (R / 2);
            const int cnt = (c < nc && !(lower && r + 1 < c)) ? min(2, max(0, nr - r)) : 0;
            cpa16(&S[r + c * PS], cnt ? G + (size_t) r + (size_t) c * ldg : G, 8 * cnt);
        }
    } else {
        for (int idx = threadIdx.x; idx < R * ncols; idx += blockDim.x) {
            const int r = idx % R, c = idx / R;
            const bool ok = r < nr && c < nc;
            cpa8(&S[r + c * PS], ok ? G + (size_t) r + (size_t) c * ldg : G, ok);
        }
    }
}

__device__ __forceinline__ void dmma_c(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}


// ---------------------------------------------------------------------------------
// Diagonal-block factorisation: eight 8-column sweeps over the 64 x 64 block T stacked on the
// identity. The same elimination that turns T into L turns the identity below it into
// E = L^-T, so the inverse costs no pass of its own.
//
// What bounds it is the chain of 64 pivots, each a reciprocal square root (50 cycles), a
// product and a fused multiply-add (8.5 each). So warp 0 does nothing but the 8 x 8 pivot
// blocks, every lane factoring the block for itself in registers, without shuffles or shared
// memory between the pivots. Warps 1-7 keep one 8-row block each in DMMA accumulators for the
// whole factorisation (warp j the block row T_j until sweep j - 1, then E_(j-1), which comes to
// life with that sweep) and bring it up to date while warp 0 is in the next sweep. A block with
// its update by the previous panel takes 7.3 us (13,000 cycles, of which 740 a
// sweep are warp 0's arithmetic); 16.3 us with 16-column sweeps by shuffles and a separate
// inverse.
// ---------------------------------------------------------------------------------

// c += -(A B^T) over 64 columns for operand fragments na = -A and the 8-row block B in shared
// memory (pitch TP), two chains of products
__device__ __forceinline__ void mma8_64(double (&c)[2], const double (&na)[16], const double *B) {
    const int at = ((threadIdx.x & 31) >> 2) + (threadIdx.x & 3) * TP;
    double b[16], d[2] = {};
#pragma unroll
    for (int k = 0; k < 16; ++k) b[k] = B[at + 4 * k * TP];
#pragma unroll
    for (int k = 0; k < 16; k += 2) {
        dmma_c(c[0], c[1], na[k], b[k]);
        dmma_c(d[0], d[1], na[k + 1], b[k + 1]);
    }
    c[0] += d[0];
    c[1] += d[1];
}

// 1 / sqrt(p) for positive normal p: the hardware's approximation (rsqrt.approx, about 20 bits)
// and one step of Householder's third-order iteration y (1 + e/2 + 3 e^2 / 8), e = 1 - p y^2.
// Straight-line code, so that the other work of a column is scheduled under it. The roundings of
// p y and of the last step leave at most 1.5 2^-53 of relative error, the iteration itself a few
// hundredths of that.
__device__ __forceinline__ double rsqrt_normal(double p) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(p));
    const double e = fma(-(p * y), y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// The lower part of the 8 x 8 block d (pitch TP, 16-byte aligned) in every lane's registers.
__device__ __forceinline__ void load8(const double *d, double (&a)[8][8]) {
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int r = c & ~1; r < 8; r += 2) {
            const double2 v = *reinterpret_cast<const double2 *>(d + r + c * TP);
            a[r][c] = v.x;
            a[r + 1][c] = v.y;
        }
}

// One sweep by one warp over the 8 x 8 pivot block a: every lane factors it for itself and
// carries its row x along, x <- x L^-T. Two columns at a time: with the 2 x 2 pivot p11, p21,
// p22 and its determinant, 1/L_22 = sqrt(p11) / sqrt(det), so both reciprocal square roots run
// at once (46 cycles of latency a column instead of 66). False when a pivot is not a positive number whose
// products with its neighbour stay in the normal range (sweep8_any then takes the block).
__device__ __forceinline__ bool sweep8(double (&a)[8][8], double (&x)[8]) {
    bool fine = true;
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
        const double p11 = a[c][c], p21 = a[c + 1][c], p22 = a[c + 1][c + 1];
        const double det = fma(p11, p22, -(p21 * p21));
        // high words: p11 and p22 between 2^-500 and 2^500, det at least 2^-1020
        fine = fine && (unsigned) __double2hiint(p11) - 0x20b00000u < 0x3e800000u &&
               (unsigned) __double2hiint(p22) - 0x20b00000u < 0x3e800000u &&
               (unsigned) __double2hiint(det) - 0x00300000u < 0x7fb00000u;
        const double r1 = rsqrt_normal(p11), rd = rsqrt_normal(det);
        const double l21 = p21 * r1, r2 = rd * (p11 * r1);
        x[c] *= r1;
        x[c + 1] = (x[c + 1] - x[c] * l21) * r2;
#pragma unroll
        for (int r = c + 2; r < 8; ++r) {
            a[r][c] *= r1;
            a[r][c + 1] = (a[r][c + 1] - a[r][c] * l21) * r2;
        }
#pragma unroll
        for (int q = c + 2; q < 8; ++q) {
#pragma unroll
            for (int r = q; r < 8; ++r) a[r][q] = a[r][q] - a[r][c] * a[q][c] - a[r][c + 1] * a[q][c + 1];
            x[q] = x[q] - x[c] * a[q][c] - x[c + 1] * a[q][c + 1];
        }
    }
    return fine;
}

// The lane's row at the start of a sweep: lanes 8-15 carry the pivot block's rows (and end with
// L_ss), lanes 0-7 the identity's (E_ss = L_ss^-T); the upper half warp repeats them.
__device__ __forceinline__ void load_row8(const double *d, double (&x)[8]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const double t = d[(lane & 7) + c * TP];
        x[c] = (lane & 8) ? t : ((lane & 7) == c ? 1.0 : 0.0);
    }
}

// The sweep over the pivot block d for any pivots, a column at a time with rsqrt(), the lane's
// row to out (pitch po); returns the first column whose pivot is not positive, or 8.
__device__ __noinline__ int sweep8_any(const double *d, double *out, int po) {
    double a[8][8], x[8];
    load_row8(d, x);
    load8(d, a);
    int bad = 8;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const double p = a[c][c];
        if (!(p > 0.0) && bad == 8) bad = c;
        const double rs = rsqrt(p);
        x[c] *= rs;
#pragma unroll
        for (int r = c + 1; r < 8; ++r) a[r][c] *= rs;
#pragma unroll
        for (int q = c + 1; q < 8; ++q) {
#pragma unroll
            for (int r = q; r < 8; ++r) a[r][q] -= a[r][c] * a[q][c];
            x[q] -= x[c] * a[q][c];
        }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) out[c * po] = x[c];
    return bad;
}

// Shared-memory regions of the factorisation kernel (64 x TP doubles each): tile
// products use regions 0 and 1; the diagonal-block factorisation keeps its block in
// region 3, the previous panel's rows in region 2 and its exchange buffers in region 1.
constexpr int R_X = 1, R_P = 2, R_T = 3;
// (addressed through the array itself, not a pointer argument, so that every access is known to
// be to shared memory)
extern __shared__ double dyn_smem[];
__device__ __forceinline__ double *region(int r) { return dyn_smem + r * 64 * TP; }

// Factor the nb x nb diagonal block at (j0, j0) and write its inverse to Dinv (lower part; the
// rest of Dinv is zero from the allocation on). With `staged` the block and the previous
// panel's 64 rows P are in regions 3 and 2 (copies possibly still in flight) and the block is
// first updated, A_jj -= P P^T. Executed by one block of 256 threads. Returns false, to every
// thread alike, on a failed pivot (then *info is set, ahead of whatever the block releases next)
// or when mid() gave up. The strictly upper part of the diagonal block in L holds zeros
// (copy_lower_k and every later write keep it so), which lets whole column segments be staged.
//
// Sweep s turns column block s. Warp 0 factors the pivot block and publishes E_ss = L_ss^-T
// (barrier 1). Every row block multiplies its tile of column s by E_ss; those of T are published
// as operands (barrier 2, without warp 0), and each row block is updated with them. The owner
// of row s + 1 updates the next pivot block before all else and hands it to warp 0 (barrier 3).
//
// mid() is called by one thread of warp 2 near the end, where that warp has time to spare; false
// means that it gave up (and has set *info).
template <class Mid>
__device__ __forceinline__ bool potf2_dev(double *L, long ld, int j0, int nb, double *Dinv, long ldd, int *info,
                                          bool staged, Mid mid) {
    double *T = region(R_T), *P = region(R_P);
    // E_ss and L_ss of alternate sweeps (8 columns, pitch PU), the published tiles of column s
    // (pitch PB). An 8 x 8 tile held as accumulators serves as a DMMA operand as it is: register h
    // of a lane is column 2 (lane % 4) + h, so product h takes those columns of both operands. The
    // pitches keep the reads of the other operand free of bank conflicts in that order.
    constexpr int PU = 72, PB = 66;
    double *U = region(R_X), *Ls = U + 16 * PU, *B = U + 32 * PU;
    __shared__ int fail, lost;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *Ljj = L + (size_t) j0 + (size_t) j0 * ld;
    double *Dj = Dinv + j0;
    const bool vec = ((((size_t) Dj) & 15) == 0) && ((ldd & 1) == 0);   // two rows of Dinv a store
    if (!staged) stage_tile(T, Ljj, ld, nb, nb, 64, true);
    cpa_wait_all();
    if (tid == 0) fail = lost = 0;
    for (int r = nb + tid; r < 64; r += blockDim.x) T[r + r * TP] = 1.0;  // pad with the identity
    __syncthreads();
    const int sb = 4096 + (j0 / 64) * 32;
    (void) sb;
    CHOL_STAMP(sb);
    const int nq = (nb + 7) / 8;               // column blocks (the padding beyond them is the identity)
    const int fr = lane >> 2, fc = lane & 3;   // row, and column or column pair, of a fragment's entry
    double na[16];                             // -P_j as operand fragments
    if (staged && warp < nq)
#pragma unroll
        for (int k = 0; k < 16; ++k) na[k] = -P[8 * warp + fr + (4 * k + fc) * TP];
    if (warp == 0) {
        if (staged) {
            double *c = T + fr + 2 * fc * TP, acc[2] = {c[0], c[TP]};
            mma8_64(acc, na, P);
            c[0] = acc[0];
            c[TP] = acc[1];
            __syncwarp();
        }
        for (int s = 0; s < nq; ++s) {
            const int o = 8 * s;
            const double *d = T + o + o * TP;
            if (s > 0) asm volatile("bar.sync 3, 64;" ::: "memory");
            double a[8][8], x[8];
            load_row8(d, x);
            load8(d, a);
            double *out = ((lane & 8) ? Ls : U) + (s & 1) * 8 * PU + (lane & 7);
            const bool fine = sweep8(a, x);
#pragma unroll
            for (int c = 0; c < 8; ++c) out[c * PU] = x[c];
            int bad = 8;
            if (!fine) bad = sweep8_any(d, out, PU);
            if (bad < 8) fail = o + bad + 1;
            asm volatile("bar.arrive 1, 256;" ::: "memory");
            CHOL_STAMP(sb + 1 + s);
            if (bad < 8) break;
        }
    } else {
        const int j = warp;
        const bool live = j < nq;
        // acc[r]: the row block's tile of column block s + r (a row of T has j - s + 1 of them)
        double acc[8][2];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double *c = T + 8 * j + fr + (8 * q + 2 * fc) * TP;
            acc[q][0] = c[0];
            acc[q][1] = c[TP];
        }
        if (staged && live) {
            mma8_64(acc[0], na, P);
            mma8_64(acc[1], na, P + 8);
        }
        for (int s = 0; s < nq; ++s) {
            const double *Us = U + (s & 1) * 8 * PU;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const double2 u = *reinterpret_cast<const double2 *>(Us + 2 * fc + fr * PU);
            // warp 0 may be a sweep further on by now and have failed there: that one's verdict is
            // for the next sweep, which all of these warps reach together
            const int failed = *(volatile int *) &fail;
            const bool low = j > s;
            // the tile of column s times E_ss
            double c[2] = {}, f[2] = {};
            dmma_c(c[0], c[1], acc[0][0], u.x);
            dmma_c(f[0], f[1], acc[0][1], u.y);
            c[0] += f[0];
            c[1] += f[1];
            if (failed && failed <= 8 * (s + 1)) break;
            if (live && (low || j - 1 < s)) {
                if (low) {
                    if (j == s + 1) {
                        double *t = T + 8 * j + fr + (8 * j + 2 * fc) * TP;
                        dmma_c(acc[1][0], acc[1][1], -c[0], c[0]);
                        dmma_c(acc[1][0], acc[1][1], -c[1], c[1]);
                        t[0] = acc[1][0];
                        t[TP] = acc[1][1];
                        asm volatile("bar.arrive 3, 64;" ::: "memory");
                    }
                    double *b = B + 8 * j + fr + 2 * fc * PB;
                    b[0] = c[0];
                    b[PB] = c[1];
                    if (8 * j + fr < nb) {
                        double *g = Ljj + (size_t) (8 * j + fr) + (size_t) (8 * s + 2 * fc) * ld;
                        g[0] = c[0];
                        g[ld] = c[1];
                    }
                } else {
                    const int r = 8 * s + 2 * fc;
                    double *g = Dj + (size_t) r + (size_t) (8 * (j - 1) + fr) * ldd;
                    if (r + 1 < nb && vec) {
                        *reinterpret_cast<double2 *>(g) = make_double2(c[0], c[1]);
                    } else {
                        if (r < nb) g[0] = c[0];
                        if (r + 1 < nb) g[1] = c[1];
                    }
                }
            }
            asm volatile("bar.sync 2, 224;" ::: "memory");
            if (j == 2 && s == max(0, nq - 2)) {
                if (lane == 0 && !mid()) lost = 1;
                __syncwarp();   // the products below are the whole warp's
            }
            if (live) {
                if (j == s + 1) {
                    // from here on row block s of E: E_ss, and -E_ss T(q, s)^T to its right
#pragma unroll
                    for (int r = 1; r < 8; ++r) acc[r][0] = acc[r][1] = 0.0;
                    c[0] = Us[fr + 2 * fc * PU];
                    c[1] = Us[fr + (2 * fc + 1) * PU];
                }
                // every operand first (those past the last column block are read, not used)
                const int last = (j > s + 1) ? j - s : nq - 1 - s;
                const double *b = B + 8 * s + fr + 2 * fc * PB;
                double bv[8][2];
#pragma unroll
                for (int r = 1; r < 8; ++r) {
                    bv[r][0] = b[8 * r];
                    bv[r][1] = b[8 * r + PB];
                }
                c[0] = -c[0];
                c[1] = -c[1];
#pragma unroll
                for (int r = 1; r < 8; ++r)
                    if (r <= last) dmma_c(acc[r][0], acc[r][1], c[0], bv[r][0]);
#pragma unroll
                for (int r = 1; r < 8; ++r)
                    if (r <= last) dmma_c(acc[r][0], acc[r][1], c[1], bv[r][1]);
                if (staged && j > s + 1) mma8_64(acc[2], na, P + 8 * (s + 2));
#pragma unroll
                for (int r = 0; r < 7; ++r) {
                    acc[r][0] = acc[r + 1][0];
                    acc[r][1] = acc[r + 1][1];
                }
            }
            if (j == 1) {
                // the pivot block of L and of Dinv
                const double *l = Ls + (s & 1) * 8 * PU;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = lane & 7, c = (lane >> 3) + 4 * h, gr = 8 * s + r, gc = 8 * s + c;
                    if (gr < nb && r >= c) Ljj[(size_t) gr + (size_t) gc * ld] = l[r + c * PU];
                    if (gr < nb && r >= c) Dj[(size_t) gr + (size_t) gc * ldd] = Us[c + r * PU];
                }
            }
        }
    }
    __syncthreads();
    CHOL_STAMP(sb + 11);
    const int failed = fail, gaveUp = lost;
    if (!failed && !gaveUp) return true;
    if (tid == 0 && !gaveUp) *info = j0 + failed;
    __syncthreads();
    return false;
}

// Tile product on the DMMA path over K = nb <= 64:
//   mode 0:  C -= A * op(B)      mode 1:  C = A * op(B)      mode 2:  C = -A * op(B)
// A(r, k) = A[r + k*lda]; op(B)(k, c) = bt ? B[c + k*ldb] : B[k + c*ldb].
// C is the 64 x 64 tile at C (pitch ldc) clipped to mr x nc; with diag set only
// row >= col entries are written.
struct TileJob {
    double *C;
    long ldc;
    int mr, nc;
    const double *A;
    long lda;
    int ar;
    const double *B;
    long ldb;
    int bt, bc, nb;
    bool diag;
    int mode;
};

// An MR x NC tile (32 or 64 each) of a job by the block's 8 warps, 16 columns and MR NC / 128
// rows a warp, in 8 x 8 DMMA tiles. Operands sit in shared memory as A (row r, column k at
// r + k (MR + 4)) and B, by rows of op(B)^T (c + k (NC + 4)) or, untransposed, by columns of
// op(B) (k + c TP): pitches that are 4 modulo 16 keep the fragment reads of either free of bank
// conflicts. Every entry is the same chain of products over k = 0, 4, 8, ... whatever the tile,
// so the result does not depend on the tile size.
template <int MR, int NC>
struct Tile {
    static constexpr int WN = NC / 16, WM = 8 / WN, RW = MR / WM, TI = RW / 8, PA = MR + 4, PB = NC + 4;
    static constexpr int A_DOUBLES = 64 * PA;
    // Warps w and w + 4 share an SM sub-partition: of a 64 x 64 tile they take opposite rows and
    // columns (0 and 3, 1 and 2 of the column parts), so that a triangular operand leaves every
    // sub-partition the same work.
    static __device__ __forceinline__ int row0() {
        const int w = threadIdx.x >> 5;
        return (WN == 4 ? ((w & 1) ^ (w >> 2)) : (w & 3)) * RW;
    }
    static __device__ __forceinline__ int col0() {
        const int w = threadIdx.x >> 5;
        return (WN == 4 ? ((w < 4) ? (w >> 1) : 3 - ((w - 4) >> 1)) : (w >> 2)) * 16;
    }
    // issue the copies of the operands (zero padded); tri 1: op(B)^T is lower triangular, tri 2: A is
    static __device__ __forceinline__ void stage(const TileJob &J, double *As, double *Bs, int tri = 0) {
        const int kp = (J.nb + 3) & ~3;
        stage_tile<MR, PA>(As, J.A, J.lda, J.ar, J.nb, kp, tri == 2);
        if (J.bt) stage_tile<NC, PB>(Bs, J.B, J.ldb, J.bc, J.nb, kp, tri == 1);
        else stage_tile<64, TP>(Bs, J.B, J.ldb, J.nb, J.bc, NC);
    }
    // this thread's C entries of a mode-0 job (zero otherwise), in fragment order
    static __device__ __forceinline__ void load_c(const TileJob &J, double (&cv)[TI][2][2]) {
        const int lane = threadIdx.x & 31, wm = row0(), wn = col0();
#pragma unroll
        for (int i = 0; i < TI; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = wm + i * 8 + (lane >> 2), c = wn + j * 8 + (lane & 3) * 2 + e;
                    cv[i][j][e] = (J.mode == 0 && r < J.mr && c < J.nc && !(J.diag && r < c))
                                      ? J.C[(size_t) r + (size_t) c * J.ldc]
                                      : 0.0;
                }
    }
    // acc = A op(B) over k < kp, the zero part of a triangular operand skipped
    template <bool BT>
    static __device__ __forceinline__ void mma(const double *As, const double *Bs, int kp, double (&acc)[TI][2][2],
                                               int tri) {
        const int lane = threadIdx.x & 31, wm = row0(), wn = col0();
#pragma unroll
        for (int i = 0; i < TI; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
        if (tri == 1) kp = min(kp, wn + 16);
        if (tri == 2) kp = min(kp, wm + RW);
#pragma unroll 4
        for (int k = 0; k < kp; k += 4) {
            const int kk = k + (lane & 3);
            double a[TI], b[2];
#pragma unroll
            for (int i = 0; i < TI; ++i) a[i] = As[(wm + i * 8 + (lane >> 2)) + kk * PA];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int c = wn + j * 8 + (lane >> 2);
                b[j] = BT ? Bs[c + kk * PB] : Bs[kk + c * TP];
            }
#pragma unroll
            for (int i = 0; i < TI; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) dmma_c(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
    }
    // write the result; with Ct also transposed to Ct (pitch ldct), with Csm also into shared
    // memory (pitch TP, zeros outside the written entries)
    static __device__ __forceinline__ void store(const TileJob &J, const double (&cv)[TI][2][2],
                                                 const double (&acc)[TI][2][2], double *Ct, long ldct, double *Csm) {
        const int lane = threadIdx.x & 31, wm = row0(), wn = col0();
#pragma unroll
        for (int i = 0; i < TI; ++i) {
            const int r = wm + i * 8 + (lane >> 2);
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = wn + j * 8 + (lane & 3) * 2 + e;
                    const bool valid = r < J.mr && c < J.nc && !(J.diag && r < c);
                    const double val =
                        (J.mode == 0) ? cv[i][j][e] - acc[i][j][e] : (J.mode == 2) ? -acc[i][j][e] : acc[i][j][e];
                    if (valid) {
                        J.C[(size_t) r + (size_t) c * J.ldc] = val;
                        if (Ct) Ct[(size_t) c + (size_t) r * ldct] = val;
                    }
                    if (Csm) Csm[r + c * TP] = valid ? val : 0.0;
                }
        }
    }
    // One tile product. Operands are staged first, so C may alias A or B (in-place solves).
    // issued() is called when their copies are on the way.
    template <class Issued>
    static __device__ __forceinline__ void run(const TileJob &J, int tri, double *Ct, long ldct, double *Csm,
                                               Issued issued) {
        double *As = dyn_smem, *Bs = dyn_smem + A_DOUBLES;
        stage(J, As, Bs, tri);
        issued();
        double cv[TI][2][2];
        load_c(J, cv);  // while the operand copies are in flight
        cpa_wait_all();
        __syncthreads();
        double acc[TI][2][2];
        if (J.bt) mma<true>(As, Bs, (J.nb + 3) & ~3, acc, tri);
        else mma<false>(As, Bs, (J.nb + 3) & ~3, acc, tri);
        store(J, cv, acc, Ct, ldct, Csm);
        __syncthreads();
    }
    static __device__ __forceinline__ void run(const TileJob &J, int tri = 0, double *Ct = nullptr, long ldct = 0) {
        run(J, tri, Ct, ldct, nullptr, []() {});
    }
};
using Tile64 = Tile<64, 64>;

// A job's part of MR x NC at row r0 and column c0 of its tile; false when nothing of it is left.
__device__ __forceinline__ bool sub_job(TileJob &J, int MR, int NC, int r0, int c0) {
    if (J.diag && r0 + MR <= c0) return false;   // above the diagonal
    J.mr = min(MR, J.mr - r0);
    J.nc = min(NC, J.nc - c0);
    if (J.mr <= 0 || J.nc <= 0) return false;
    J.ar = J.mr;
    J.bc = J.nc;
    J.C += (size_t) r0 + (size_t) c0 * J.ldc;
    J.A += r0;
    J.B += J.bt ? (size_t) c0 : (size_t) c0 * J.ldb;
    J.diag = J.diag && r0 < c0 + NC;
    return true;
}

// Mode-0 jobs t0, t0 + step, ... (< t1) of one block, double buffered: the operands
// of the next job are copied into the other pair of regions (0/1 and 2/3) and its C
// entries loaded into registers while the current job's products run. The jobs'
// C tiles must be disjoint from each other and from every operand.
template <typename JobOf>
__device__ void tile_stream(JobOf job_of, long t0, long t1, long step) {
    if (t0 >= t1) return;
    TileJob cur, nxt;
    job_of(t0, cur);
    int b = 0;
    Tile64::stage(cur, region(2 * b), region(2 * b + 1));
    asm volatile("cp.async.commit_group;\n" ::);
    double cv[4][2][2], cvn[4][2][2];
    Tile64::load_c(cur, cv);
    for (long t = t0;; t += step) {
        const bool more = t + step < t1;
        if (more) {
            job_of(t + step, nxt);
            Tile64::stage(nxt, region(2 * (b ^ 1)), region(2 * (b ^ 1) + 1));
            asm volatile("cp.async.commit_group;\n" ::);
            Tile64::load_c(nxt, cvn);
            asm volatile("cp.async.wait_group 1;\n" ::);
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::);
        }
        __syncthreads();
        double acc[4][2][2];
        if (cur.bt) Tile64::mma<true>(region(2 * b), region(2 * b + 1), (cur.nb + 3) & ~3, acc, 0);
        else Tile64::mma<false>(region(2 * b), region(2 * b + 1), (cur.nb + 3) & ~3, acc, 0);
        Tile64::store(cur, cv, acc, nullptr, 0, nullptr);
        __syncthreads();  // the buffer just read may be refilled
        if (!more) break;
        cur = nxt;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                cv[i][j][0] = cvn[i][j][0];
                cv[i][j][1] = cvn[i][j][1];
            }
        b ^= 1;
    }
}

__device__ __forceinline__ void tri_index(long t, int &ti, int &tj) {
    ti = (int) ((sqrtf(8.0f * (float) t + 1.0f) - 1.0f) * 0.5f);   // settled by the loops below
    while ((long) ti * (ti + 1) / 2 > t) --ti;
    while ((long) (ti + 1) * (ti + 2) / 2 <= t) ++ti;
    tj = (int) (t - (long) ti * (ti + 1) / 2);
}

// Right-looking blocked Cholesky with one-panel look-ahead: while the other blocks solve panel
// j and update the trailing matrix with it, block 0 solves the panel's first chunk, updates the
// diagonal block j + 1 with it and factors it.
//
// With K set, the inverse factor K = L^-1 (and KT = K^T) is formed alongside, right
// looking by 64-row blocks, on the blocks that would otherwise wait for block 0:
// before panel j, the rows below block j-1 of K receive
// X(r, c) -= L(r, j-1) K(j-1, c) (the first update of a tile assigns -L K); while the
// trailing matrix is updated, block row j is finalised as K(j, c) = Dinv_j X(j, c) and
// K(j, j) = Dinv_j. The strictly upper blocks of K and the strictly lower blocks of KT
// are never written (they must hold zeros).
//
// A phase whose tiles would leave half the blocks idle takes them in quarters (32 x 32) or
// halves: a 64 x 64 tile takes a block about 5 us (2.1 us of DMMA, 128 KB through the SM's L2
// port), a quarter 2 us, so the line lies where the quarters need a second round.
__device__ __forceinline__ TileJob k_update_job(const double *L, long ld, double *K, int n, int r, int c, int k) {
    const int mr = min(64, n - 64 * r);
    return TileJob{K + (size_t) 64 * r + (size_t) 64 * c * ld, ld, mr, 64, L + (size_t) 64 * r + (size_t) 64 * k * ld,
                   ld, mr, K + (size_t) 64 * k + (size_t) 64 * c * ld, ld, 0, 64, 64, false, (k == c) ? 2 : 0};
}

// part h of `parts` (1, or 2: column halves) of block (bj, c) of K's final form
__device__ __forceinline__ void k_final_tile(const double *Dinv, long ldd, double *K, double *KT, long ld, int n,
                                             int bj, int c, int h, int parts) {
    const int mr = min(64, n - 64 * bj), c0 = 32 * h;
    if (c < bj) {
        double *X = K + (size_t) 64 * bj + (size_t) 64 * c * ld;
        TileJob J{X, ld, mr, 64, Dinv + (size_t) 64 * bj, ldd, mr, X, ld, 0, 64, mr, false, 1};
        double *Ct = KT + (size_t) (64 * c + c0) + (size_t) 64 * bj * ld;
        if (parts == 1) Tile64::run(J, 2, Ct, ld);
        else if (sub_job(J, 64, 32, 0, c0)) Tile<64, 32>::run(J, 2, Ct, ld);
    } else {
        for (int idx = threadIdx.x; idx < 64 * 64 / parts; idx += blockDim.x) {
            const int r = idx & 63, cc = c0 + (idx >> 6);
            if (r < mr && cc < mr) {
                const double v = Dinv[(size_t) (64 * bj + r) + (size_t) cc * ldd];
                K[(size_t) (64 * bj + r) + (size_t) (64 * bj + cc) * ld] = v;
                KT[(size_t) (64 * bj + cc) + (size_t) (64 * bj + r) * ld] = v;
            }
        }
        __syncthreads();
    }
}

// The factorisation on a grid of ngrid blocks, this one being block bid, with the signals of
// `sync` between them. The cooperative kernel runs it on its grid (ONE false, at least two
// blocks: block 0 does the diagonal blocks and the rows that feed them and nothing else, the
// others the rest); a batched launch runs it with one block per matrix (ONE, bid 0, ngrid 1).
// Every tile is computed by the same operations whatever the grid, so the result does not
// depend on it.
//
// Block 0 is the chain that sets the time, so it waits for the others only where it must: it
// needs the last panel's updates (which are done long before it has finished the diagonal block
// it is in), and the others need its diagonal blocks and its rows of the panel.
//
// Whether to go on is decided once per block and never from *info, which others may be writing:
// block 0 by what potf2_dev returns to all of its threads, the others by what their waits return.
// After a failure in diagonal block q every other block still takes part in panel q and leaves at
// its wait for diagonal block q, whenever it gets there, so no arrival that others count on is lost.
template <bool ONE, class Sync>
__device__ __forceinline__ void potrf_body(double *L, long ld, int n, double *Dinv, long ldd, int *info, double *K,
                                           double *KT, int bid, int ngrid, Sync &sync) {
    const int nblk = (n + 63) / 64;
    const int nworker = ONE ? 1 : ngrid - 1, wid = ONE ? 0 : bid - 1;
    for (int jn = 0; jn < n; jn += NB) {
        // the next diagonal block starts at jn, the panel being finished at j0 = jn - 64
        const bool first = jn == 0;
        const int bj = jn / NB - 1;
        // K's rows r >= bj are updated by block row bj - 1 before the diagonal block bj is waited
        // for: they need only the other blocks' last updates
        const long nx = (K && bj >= 1) ? (long) (nblk - bj) * bj : 0;
        if ((ONE || bid > 0) && nx > 0) {
            auto kjob = [&](long u) { return k_update_job(L, ld, K, n, bj + (int) (u / bj), (int) (u % bj), bj - 1); };
            if (!sync.update_wait_all(bj)) return;
            if (2 * nx <= nworker) {
                // half the blocks would stay idle: quarter tiles
                for (long t = wid; t < 4 * nx; t += nworker) {
                    TileJob J = kjob(t >> 2);
                    if (sub_job(J, 32, 32, 32 * (int) (t & 1), 32 * (int) ((t >> 1) & 1))) Tile<32, 32>::run(J);
                }
            } else {
                tile_stream([&](long u, TileJob &J) { J = kjob(u); }, wid, nx, nworker);
            }
        }
        if (!first && bid > 0 && !sync.diag_wait(jn / NB)) return;
        const int j0 = jn - NB, rows = n - jn, nchunk = (rows + 63) / 64, nbn = min(NB, rows);
        double *P = L + (size_t) jn + (size_t) j0 * ld, *A22 = L + (size_t) jn + (size_t) jn * ld;
        const int pb = bj * 16 + (bid == 1 ? 8 : 0);
        (void) pb;
        auto chunk = [&](int ch) {
            const int mr = min(64, rows - ch * 64);
            return TileJob{P + ch * 64, ld, mr, NB, P + ch * 64, ld, mr, Dinv + j0, ldd, 1, NB, NB, false, 1};
        };
        if (!first && bid <= 1) CHOL_STAMP(pb + 0);
        if (ONE || bid == 0) {
            if (!first) {
                // the next diagonal block (its updates by earlier panels are complete) and chunk 0
                // of the panel, the rows that update it
                stage_tile(region(R_T), A22, ld, nbn, nbn, 64, true);
                Tile64::run(chunk(0), 1, nullptr, 0, region(R_P), [&]() { sync.diag_release(jn / NB); });
                if (bid <= 1) CHOL_STAMP(pb + 1);
                if (!ONE) sync.panel_arrive();
                if (bid <= 1) CHOL_STAMP(pb + 2);
            }
            const bool good = potf2_dev(L, ld, jn, nbn, Dinv, ldd, info, !first, [&]() {
                // the panel's updates by the other blocks, before the next panel
                return first || sync.update_wait(jn / NB);
            });
            if (!first && bid <= 1) CHOL_STAMP(pb + 4);
            if (!good) {
                sync.diag_failed(jn / NB);
                return;
            }
        }
        if (!first && (ONE || bid > 0)) {
            // the rest of the panel, by half chunks where the blocks outnumber them
            const int c1 = nchunk - 1;
            if (2 * c1 <= nworker) {
                for (int t = wid; t < 2 * c1; t += nworker) {
                    TileJob J = chunk(1 + (t >> 1));
                    const int r0 = 32 * (t & 1);
                    J.mr = J.ar = min(32, J.mr - r0);
                    J.C += r0;
                    J.A += r0;
                    if (J.mr > 0) Tile<32, 64>::run(J, 1);
                }
            } else {
                for (int t = wid; t < c1; t += nworker) Tile64::run(chunk(1 + t), 1);
            }
            if (bid == 1) CHOL_STAMP(pb + 1);
            if (!ONE) sync.panel_arrive();
            if (!sync.panel_wait(jn / NB)) return;
            if (bid == 1) CHOL_STAMP(pb + 2);
            // the trailing matrix (tile 0 is the next diagonal block) and K's block row bj
            const long ntile = (long) nchunk * (nchunk + 1) / 2, nk = K ? bj + 1 : 0;
            auto trailing = [&](long t, TileJob &J) {
                int ti, tj;
                tri_index(t, ti, tj);
                const int mr = min(64, rows - ti * 64), nc = min(64, rows - tj * 64);
                J = TileJob{A22 + (size_t) ti * 64 + (size_t) tj * 64 * ld, ld, mr, nc, P + ti * 64, ld, mr,
                            P + tj * 64, ld, 1, nc, NB, ti == tj, 0};
            };
            if (2 * (ntile - 1 + nk) <= nworker) {
                const long nt4 = 4 * (ntile - 1);
                for (long t = wid; t < nt4 + 2 * nk; t += nworker) {
                    if (t < nt4) {
                        TileJob J;
                        trailing(1 + (t >> 2), J);
                        if (sub_job(J, 32, 32, 32 * (int) (t & 1), 32 * (int) ((t >> 1) & 1))) Tile<32, 32>::run(J);
                    } else {
                        k_final_tile(Dinv, ldd, K, KT, ld, n, bj, (int) ((t - nt4) >> 1), (int) ((t - nt4) & 1), 2);
                    }
                }
            } else {
                tile_stream(trailing, 1 + wid, ntile, nworker);
                for (long t = 1 + wid; t < ntile + nk; t += nworker)
                    if (t >= ntile) k_final_tile(Dinv, ldd, K, KT, ld, n, bj, (int) (t - ntile), 0, 1);
            }
            if (bid == 1) CHOL_STAMP(pb + 3);
            sync.update_arrive();
        }
        if (!first && bid <= 1) CHOL_STAMP(pb + 5);
    }
    if (bid == 0) sync.diag_release(nblk);
    else if (!sync.diag_wait(nblk)) return;
    if (!K) return;
    // the last block row of K: its update by block row nblk - 2, then its final form
    const int bj = nblk - 1;
    if (2 * bj <= ngrid) {
        for (int t = bid; t < 4 * bj; t += ngrid) {
            TileJob J = k_update_job(L, ld, K, n, bj, t >> 2, bj - 1);
            if (sub_job(J, 32, 32, 32 * (t & 1), 32 * ((t >> 1) & 1))) Tile<32, 32>::run(J);
        }
        if (bj >= 1 && !sync.all()) return;
        for (int t = bid; t < 2 * (bj + 1); t += ngrid) k_final_tile(Dinv, ldd, K, KT, ld, n, bj, t >> 1, t & 1, 2);
        return;
    }
    for (int c = bid; c < bj; c += ngrid) Tile64::run(k_update_job(L, ld, K, n, bj, c, bj - 1));
    if (bj >= 1 && !sync.all()) return;
    for (int c = bid; c <= bj; c += ngrid) k_final_tile(Dinv, ldd, K, KT, ld, n, bj, c, 0, 1);
}

// The signals between the blocks of a cooperative launch: words in global memory that start at zero
// and only grow. One thread of a block signals and polls for all of it: thread kThread (of warp 3,
// which has time to spare in the diagonal blocks), or in block 0's update_wait() the thread that
// calls it. Waits are bounded and return the same to every thread of the block: false when the wait
// gave up, which sets *info to -1, or, for a diagonal block, when it failed.
struct GridSync {
    unsigned *c;    // 0: all(), 1: panel, 2: updates, 3: diagonal blocks done (and kFailed)
    int *info;
    unsigned nall = 0;
    static constexpr int kThread = 96;
    static constexpr unsigned kFailed = 1u << 31;   // the last one counted by word 3 has failed
    __device__ __forceinline__ void add(int k) {
        __syncthreads();
        if (threadIdx.x == kThread) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c + k) : "memory");
        }
    }
    // one thread: the word once it has reached the target (but for kFailed); false on giving up
    __device__ __forceinline__ bool poll(int k, unsigned target, unsigned &v) {
        for (long it = 0; it < (1L << 22); ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c + k) : "memory");
            if ((v & ~kFailed) >= target) return true;
        }
        *(volatile int *) info = -1;
        return false;
    }
    __device__ __forceinline__ bool wait(int k, unsigned target) {
        unsigned v;
        return !__syncthreads_or(threadIdx.x == kThread && !poll(k, target, v));
    }
    // every block has finished its part of panel p (block 0 its chunk 0)
    __device__ __forceinline__ void panel_arrive() { add(1); }
    __device__ __forceinline__ bool panel_wait(int p) { return wait(1, (unsigned) p * gridDim.x); }
    // the blocks beside block 0 have finished their updates by panel p (awaited by one thread of block 0)
    __device__ __forceinline__ void update_arrive() { add(2); }
    __device__ __forceinline__ bool update_wait(int p) {
        unsigned v;
        return poll(2, (unsigned) p * (gridDim.x - 1), v);
    }
    __device__ __forceinline__ bool update_wait_all(int p) { return wait(2, (unsigned) p * (gridDim.x - 1)); }
    // block 0 has finished d diagonal blocks (and seen the updates before the last of them)
    __device__ __forceinline__ void diag_release(unsigned d) {   // after a block barrier
        if (threadIdx.x == kThread) {
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(c + 3), "r"(d) : "memory");
        }
    }
    // diagonal block q has failed, those before it are done
    __device__ __forceinline__ void diag_failed(int q) { diag_release((unsigned) (q + 1) | kFailed); }
    // d diagonal blocks done; false when the d-th of them failed
    __device__ __forceinline__ bool diag_wait(int d) {
        unsigned v;
        return !__syncthreads_or(threadIdx.x == kThread &&
                                 (!poll(3, (unsigned) d, v) || v == ((unsigned) d | kFailed)));
    }
    __device__ __forceinline__ bool all() {
        add(0);
        return wait(0, ++nall * gridDim.x);
    }
};

// the same for a grid of one block
struct BlockSync {
    __device__ __forceinline__ void panel_arrive() {}
    __device__ __forceinline__ bool panel_wait(int) {
        __syncthreads();
        return true;
    }
    __device__ __forceinline__ void update_arrive() { __syncthreads(); }
    __device__ __forceinline__ bool update_wait(int) { return true; }
    __device__ __forceinline__ bool update_wait_all(int) { return true; }
    __device__ __forceinline__ void diag_release(unsigned) {}
    __device__ __forceinline__ void diag_failed(int) {}
    __device__ __forceinline__ bool diag_wait(int) { return true; }
    __device__ __forceinline__ bool all() {
        __syncthreads();
        return true;
    }
};

// sum_i log L_ii summed as the log-diagonal kernel sums it with its 1024 threads (terms v,
// v + 1024, ... per thread, a shuffle tree per warp, then one over the 32 warp sums), by
// COOP_THREADS threads each standing in for four: the same additions in the same order. The
// sum is thread 0's.
__device__ double logdiag_1024(int n, const double *L, long ld) {
    __shared__ double red[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    constexpr int kV = 1024 / COOP_THREADS;
#pragma unroll
    for (int q = 0; q < kV; ++q) {
        double x = 0.0;
        for (int v = t + COOP_THREADS * q; v < n; v += 1024) x += log(__ldcg(L + (size_t) v + (size_t) v * ld));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[w + (COOP_THREADS / 32) * q] = x;
    }
    __syncthreads();
    double x = 0.0;
    if (w == 0) {
        x = red[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    }
    __syncthreads();
    return x;
}

// The factor's status at the end of its kernel, by one block: the word *info and, with
// `logdet`, sum log L_ii in the double after it, both also straight into the host's pinned
// mirror when there is one.
__device__ void write_status(int n, const double *L, long ld, int *info, double *hinfo, int logdet) {
    double sum = 0.0;
    if (logdet) sum = logdiag_1024(n, L, ld);
    if (threadIdx.x != 0) return;
    const int v = *(volatile int *) info;
    if (logdet) reinterpret_cast<double *>(info)[1] = sum;
    if (hinfo) {
        reinterpret_cast<volatile int *>(hinfo)[0] = v;
        if (logdet) hinfo[1] = sum;
    }
}

__global__ void __launch_bounds__(COOP_THREADS, 1)
    potrf_coop_kernel(double *L, long ld, int n, double *Dinv, long ldd, int *info, double *K, double *KT,
                      double *hinfo, int logdet) {
    GridSync sync{reinterpret_cast<unsigned *>(info) + kInfoCounters, info};
    potrf_body<false>(L, ld, n, Dinv, ldd, info, K, KT, (int) blockIdx.x, (int) gridDim.x, sync);
    // block 0 has the last word on *info: the others' waits end before its own work does, and blocks
    // still on their way out after a failed pivot leave it alone
    if (blockIdx.x == 0 && (logdet || hinfo)) write_status(n, L, ld, info, hinfo, logdet);
}

// Several factorisations in one launch, one CTA each: the copy of the lower triangle, the
// factorisation of the cooperative kernel on a grid of one block (with K = L^-1 and K^T for
// a fused factor), and sum log L_ii next to the info word as the log-diagonal kernel forms
// it; the results are those of the cooperative kernel on any grid.
struct SmallFactorJob {
    const double *S;
    double *L, *Dinv, *K, *KT;
    long lds, ld;
    int *info;
    double *hinfo;   // device address of the factor's pinned status words (written directly)
    int n, logdet;
};
constexpr int kSmallBatch = 36;
struct SmallFactorBatch {
    SmallFactorJob job[kSmallBatch];
};

__device__ void small_factor_job(const SmallFactorJob &J) {
    const int n = J.n;
    for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
        const int r = idx % n, c = idx / n;
        J.L[(size_t) r + (size_t) c * J.ld] = (r >= c) ? J.S[(size_t) r + (size_t) c * J.lds] : 0.0;
    }
    if (threadIdx.x == 0) *J.info = 0;
    __threadfence_block();
    __syncthreads();
    BlockSync sync;
    potrf_body<true>(J.L, J.ld, n, J.Dinv, J.ld, J.info, J.K, J.KT, 0, 1, sync);
    __threadfence_block();
    __syncthreads();
    write_status(n, J.L, J.ld, J.info, J.hinfo, J.logdet);
}

__global__ void __launch_bounds__(COOP_THREADS, 1) potrf_small_batch_kernel(const SmallFactorBatch B) {
    small_factor_job(B.job[blockIdx.x]);
}

// the same, the jobs in global memory (more than fit the parameters)
__global__ void __launch_bounds__(COOP_THREADS, 1) potrf_batch_array_kernel(const SmallFactorJob *__restrict__ jobs) {
    const SmallFactorJob J = jobs[blockIdx.x];
    small_factor_job(J);
}

// Blocked substitution for L L^T x = b, one cooperative launch. The 64-row blocks of
// the vector are dealt to the CTAs (block k to CTA k mod grid); a CTA keeps, in shared
// memory, the accumulated products of its unfinished blocks with the solved ones.
// Forward sweep: the owner of block j forms t_j = Dinv_j (b_j - acc_j) and publishes it
// with flag_f[j] = epoch; every CTA then adds L_kj t_j to its unfinished blocks. The
// chain from block to block is kept short: each CTA prefetches into shared memory the
// tile L_{k,k-1} and Dinv_k of its next block k while it works on older ones, and when
// t_{k-1} appears it finishes and publishes block k before any other update. The other
// updates of a step are one pass over all of the CTA's unfinished blocks (many loads in
// flight). After a grid barrier the backward sweep does the same from the last block up
// with L^T and Dinv^T. Every wait on a flag is bounded; on giving up the CTA raises
// g_tri_err and the others skip their work (every CTA still reaches the grid barrier).
__device__ int g_tri_err = 0;
constexpr long TRI_WAIT_LIMIT = 1L << 22;

__device__ __forceinline__ bool tri_wait(const unsigned *flag, unsigned epoch) {
    for (long it = 0; it < TRI_WAIT_LIMIT; ++it) {
        if ((int) (*(volatile const unsigned *) flag - epoch) >= 0) return true;
        if ((it & 1023) == 1023 && *(volatile int *) &g_tri_err) return false;
    }
    atomicExch(&g_tri_err, 1);
    return false;
}

__global__ void __launch_bounds__(COOP_THREADS, 1)
    tri_solve_coop_kernel(const double *__restrict__ L, long ld, int n, const double *__restrict__ Dinv, long ldd,
                          const double *b, double *t, double *x, unsigned *flag_f, unsigned *flag_b,
                          unsigned epoch) {
    cg::grid_group grid = cg::this_grid();
    double *sm = dyn_smem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = gridDim.x, me = blockIdx.x;
    const int nblk = (n + 63) / 64;
    const int nown = (me < nblk) ? (nblk - 1 - me) / G + 1 : 0;
    double *Lt = sm;                       // 64 x TP: the tile that feeds the next block
    double *Dt = sm + 64 * TP;             // 64 x TP: that block's Dinv
    double *acc = sm + 2 * 64 * TP;        // nown x 64
    double *xs = acc + (size_t) nown * 64; // the solved block being applied
    double *xn = xs + 64;                  // the block this CTA just published
    double *red = xn + 64;                 // 4 x 64 partial sums
    __shared__ int abort_;
    if (tid == 0) abort_ = 0;
    auto kof = [&](int c) { return me + c * G; };
    auto nbof = [&](int j) { return min(64, n - 64 * j); };
    auto fetch = [&](const double *v, int j, const unsigned *flag) {
        if (tid == 0 && !tri_wait(flag + j, epoch)) abort_ = 1;
        __threadfence();
        __syncthreads();
        if (tid < 64) xs[tid] = (!abort_ && tid < nbof(j)) ? __ldcg(v + 64 * j + tid) : 0.0;
        __syncthreads();
    };
    auto take_next = [&]() {
        if (tid < 64) xs[tid] = xn[tid];
        __syncthreads();
    };
    // v = rhs_k - acc_c; out_k = Dt v (transpose: Dt^T v) into xn and out, then publish
    auto finish = [&](int c, const double *rhs, double *out, bool transpose, unsigned *flag) {
        const int k = kof(c), nb = nbof(k);
        double *a = acc + (size_t) c * 64;
        if (tid < 64) red[tid] = (tid < nb) ? rhs[64 * k + tid] - a[tid] : 0.0;
        __syncthreads();
        for (int o = warp; o < 64; o += 8) {
            double sum = 0.0;
            for (int q = lane; q < 64; q += 32) sum += (transpose ? Dt[q + o * TP] : Dt[o + q * TP]) * red[q];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            if (lane == 0) xn[o] = (o < nb) ? sum : 0.0;
        }
        __syncthreads();
        if (tid < nb) out[64 * k + tid] = xn[tid];
        __threadfence();
        __syncthreads();
        if (tid == 0) atomicExch(flag + k, epoch);
    };
    auto wait_tiles = [&]() {
        asm volatile("cp.async.wait_all;\n" ::);
        __syncthreads();
    };

    // ---- forward sweep: t = L^-1 b
    for (int i = tid; i < nown * 64; i += blockDim.x) acc[i] = 0.0;
    __syncthreads();
    if (nown > 0 && !*(volatile int *) &g_tri_err) {
        // next block k: L_{k,k-1} (rows of k, columns of k-1) and Dinv_k
        auto prefetch_f = [&](int k) {
            if (k > 0) stage_tile(Lt, L + (size_t) (64 * k) + (size_t) (64 * (k - 1)) * ld, ld, nbof(k), 64, 64);
            stage_tile(Dt, Dinv + (size_t) (64 * k), ldd, nbof(k), nbof(k), 64);
            asm volatile("cp.async.commit_group;\n" ::);
        };
        int c = 0;
        bool have = false;
        prefetch_f(kof(0));
        if (me == 0) {
            wait_tiles();
            finish(0, b, t, false, flag_f);
            have = true;
            c = 1;
            if (c < nown) prefetch_f(kof(c));
        }
        const int last = kof(nown - 1);
        for (int j = 0; j < last && !abort_; ++j) {
            if (have) {
                take_next();
                have = false;
            } else {
                fetch(t, j, flag_f);
                if (abort_) break;
            }
            if (c < nown && kof(c) == j + 1) {
                // the next block: acc += L_{j+1,j} t_j from the prefetched tile, then finish it
                wait_tiles();
                {
                    const int r = tid & 63, q = tid >> 6;
                    double sum = 0.0;
#pragma unroll
                    for (int cc = 16 * q; cc < 16 * q + 16; ++cc) sum += Lt[r + cc * TP] * xs[cc];
                    red[q * 64 + r] = sum;
                }
                __syncthreads();
                if (tid < 64) acc[(size_t) c * 64 + tid] += red[tid] + red[64 + tid] + red[128 + tid] + red[192 + tid];
                __syncthreads();
                finish(c, b, t, false, flag_f);
                have = true;
                ++c;
                if (c < nown) prefetch_f(kof(c));
            }
            // every other unfinished block (all beyond block j + 1): acc_k += L_kj t_j
            for (int item = tid; item < (nown - c) * 64; item += blockDim.x) {
                const int cc = c + (item >> 6), r = item & 63, k = kof(cc);
                if (r >= nbof(k)) continue;
                const double *row = L + (size_t) (64 * k + r) + (size_t) (64 * j) * ld;
                double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll 4
                for (int q = 0; q < 64; q += 4) {
                    s0 += row[(size_t) q * ld] * xs[q];
                    s1 += row[(size_t) (q + 1) * ld] * xs[q + 1];
                    s2 += row[(size_t) (q + 2) * ld] * xs[q + 2];
                    s3 += row[(size_t) (q + 3) * ld] * xs[q + 3];
                }
                acc[(size_t) cc * 64 + r] += (s0 + s1) + (s2 + s3);
            }
            __syncthreads();
        }
    }
    asm volatile("cp.async.wait_all;\n" ::);
    grid.sync();
    // ---- backward sweep: x = L^-T t
    for (int i = tid; i < nown * 64; i += blockDim.x) acc[i] = 0.0;
    __syncthreads();
    if (nown > 0 && !*(volatile int *) &g_tri_err) {
        // next block k (downwards): L_{k+1,k} (rows of k+1, columns of k) and Dinv_k
        auto prefetch_b = [&](int k) {
            if (k < nblk - 1) stage_tile(Lt, L + (size_t) (64 * (k + 1)) + (size_t) (64 * k) * ld, ld, nbof(k + 1), 64, 64);
            stage_tile(Dt, Dinv + (size_t) (64 * k), ldd, nbof(k), nbof(k), 64);
            asm volatile("cp.async.commit_group;\n" ::);
        };
        int c = nown - 1;
        bool have = false;
        prefetch_b(kof(c));
        if (kof(c) == nblk - 1) {
            wait_tiles();
            finish(c, t, x, true, flag_b);
            have = true;
            --c;
            if (c >= 0) prefetch_b(kof(c));
        }
        for (int j = nblk - 1; j > me && !abort_; --j) {
            if (have) {
                take_next();
                have = false;
            } else {
                fetch(x, j, flag_b);
                if (abort_) break;
            }
            if (c >= 0 && kof(c) == j - 1) {
                // the next block: acc += L_{j,j-1}^T x_j from the prefetched tile, then finish it
                wait_tiles();
                for (int o = warp; o < 64; o += 8) {
                    double sum = 0.0;
                    for (int q = lane; q < 64; q += 32) sum += Lt[q + o * TP] * xs[q];
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
                    if (lane == 0) acc[(size_t) c * 64 + o] += sum;
                }
                __syncthreads();
                finish(c, t, x, true, flag_b);
                have = true;
                --c;
                if (c >= 0) prefetch_b(kof(c));
            }
            // every other unfinished block (all below block j - 1): acc_k += L_jk^T x_j,
            // a warp per output column, four columns at a time
            const int nbj = nbof(j);
            for (int item = warp * 4; item < (c + 1) * 64; item += 32) {
                double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int cc = (item + u) >> 6, o = (item + u) & 63, k = kof(cc);
                    const double *col = L + (size_t) (64 * j) + (size_t) (64 * k + o) * ld;
                    for (int q = lane; q < nbj; q += 32) s4[u] += col[q] * xs[q];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) s4[u] += __shfl_xor_sync(0xffffffffu, s4[u], off);
                }
                if (lane == 0) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc[(size_t) ((item + u) >> 6) * 64 + ((item + u) & 63)] += s4[u];
                }
            }
            __syncthreads();
        }
    }
    asm volatile("cp.async.wait_all;\n" ::);
}

// L = the lower triangle of S; with info, the status words and the counters after them cleared
__global__ void copy_lower_k(int n, const double *S, long lds, double *L, long ldl, int *info) {
    if (info && blockIdx.x == 0 && threadIdx.x < kInfoBytes / 4) info[threadIdx.x] = 0;
    const int r = (blockIdx.x % ((n + 255) / 256)) * 256 + threadIdx.x;
    if (r >= n) return;
    const int step = gridDim.x / ((n + 255) / 256);
#pragma unroll 4
    for (int c = blockIdx.x / ((n + 255) / 256); c < n; c += step)
        L[(size_t) r + (size_t) c * ldl] = (r >= c) ? S[(size_t) r + (size_t) c * lds] : 0.0;
}

int sm_count() { return device_sm_count(); }

// resident CTAs of the cooperative factorisation, per device
int coop_grid() {
    static std::atomic<int> cached[kMaxDevices];
    const int dev = current_device();
    int v = cached[dev].load(std::memory_order_acquire);
    if (v) return v;
    static std::atomic<unsigned long long> init;
    once_per_device(init, [&] {
        const int smem = SM_DOUBLES * (int) sizeof(double);
        HB_CUDA(cudaFuncSetAttribute(potrf_coop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        int per = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, potrf_coop_kernel, COOP_THREADS, smem);
        cached[dev].store(std::max(1, device_sm_count() * std::max(per, 1)), std::memory_order_release);
    });
    return cached[dev].load(std::memory_order_acquire);
}

}  // namespace

// blocks of copy_lower_k: a whole number of row ranges of 256, about four columns a thread
static int copy_lower_grid(int n) {
    const int rb = (n + 255) / 256;
    return rb * std::max(1, std::min((n + 3) / 4, 148 * 16 / rb));
}

// `status`: the kernel also writes the status and sum log L_ii (d_info, and the pinned mirror
// where it is mapped; *mirrored tells the caller that no copy is needed)
bool coop_factorize_enqueue(cudaStream_t s, DenseFactor &F, const double *S, long ldS, bool status, bool *mirrored) {
    const int n = F.n;
    copy_lower_k<<<hb::counted(copy_lower_grid(n)), 256, 0, s>>>(n, S, ldS, F.L, F.ld, F.d_info);
    double *hinfo = nullptr;
    if (status && cudaHostGetDevicePointer((void **) &hinfo, F.h_info, 0) != cudaSuccess) {
        cudaGetLastError();
        hinfo = nullptr;
    }
    if (mirrored) *mirrored = hinfo != nullptr;
    int logdet = (status && F.stat_logdet) ? 1 : 0;
    const void *fn = (const void *) potrf_coop_kernel;
    const long t0 = (long) ((n - 1) / 64 + 1);
    // with the fused inverse, the update of K's rows needs up to t0^2 / 4 tiles per phase
    // at most one block per SM, so that the block factoring the diagonal never shares an SM
    // (four quarter tiles a tile where the blocks outnumber the tiles)
    const long want = 1 + 4 * (F.fuse_k ? t0 * (t0 + 1) / 2 + t0 * t0 / 4 : t0 * (t0 + 1) / 2);
    const int grid = (int) std::max(2L, std::min<long>(std::min(coop_grid(), sm_count()), want));
    double *Lp = F.L;
    long ld = F.ld;
    int nn = n;
    double *Dp = F.Dinv;
    long ldd = F.ld;
    int *ip = F.d_info;
    double *Kp = F.fuse_k ? F.K : nullptr;
    double *KTp = F.fuse_k ? F.KT : nullptr;
    void *args[] = {&Lp, &ld, &nn, &Dp, &ldd, &ip, &Kp, &KTp, &hinfo, &logdet};
    const bool timed = kstat_on(F.kfamily);
    if (timed) kstat_begin(F.kfamily, s, (double) n * n * n / 3.0);
    cudaError_t e = cudaLaunchCooperativeKernel(fn, hb::counted(grid), COOP_THREADS, args, SM_DOUBLES * sizeof(double), s);
    if (timed) kstat_end(s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

// ---- recursive blocked form (orders above kRecLeafMaxN, with K = L^-1) ----------------
//   L11 L11^T = A11 (recursively; a block of at most kRecLeafMaxN rows on the cooperative
//   kernel, which also forms its K and K^T), L21 = A21 K11^T, A22 -= L21 L21^T,
//   L22 L22^T = A22 (recursively), K21 = -K22 (L21 K11), KT12 = K21^T.
// The split falls on a 64-row boundary, so every diagonal block's 64 x 64 inverses land in
// Dinv where the one-launch factorisation puts them. Each diagonal block reports its status
// in a word of its own; the first failure (with its global pivot index) becomes the
// factor's status.
namespace {
constexpr int kRecMaxLeaves = 128;   // status words of kInfoBytes each
struct RecLeaves {
    int off[kRecMaxLeaves];
    int count;
};

__global__ void rec_info_kernel(const RecLeaves R, const int *leaf_info, int *info) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int v = 0;
    for (int q = 0; q < R.count && v == 0; ++q)
        if (const int w = leaf_info[kInfoBytes / 4 * q]) v = w < 0 ? -1 : w + R.off[q];
    *info = v;
}

// B (cols x rows) = A^T for A rows x cols
__global__ void transpose_rect_kernel(int rows, int cols, const double *A, long lda, double *B, long ldb) {
    __shared__ double tile[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = bx + threadIdx.x, c = by + j;
        if (r < rows && c < cols) tile[j][threadIdx.x] = A[(size_t) r + (size_t) c * lda];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = by + threadIdx.x, c = bx + j;   // B(r, c) = A(c, r)
        if (r < cols && c < rows) B[(size_t) r + (size_t) c * ldb] = tile[threadIdx.x][j];
    }
}

int rec_split(int n) { return ((n / 2) / 64) * 64; }

// the diagonal block [off, off + n) of F on the cooperative kernel, its K and K^T into Kp / KTp
// (leading dimension F.ld)
bool rec_leaf(cudaStream_t s, DenseFactor &F, int off, int n, double *Kp, double *KTp, RecLeaves &R) {
    if (R.count >= kRecMaxLeaves) return false;
    DenseFactor V;   // a view of the diagonal block in F's buffers (never released)
    V.n = n;
    V.ld = F.ld;
    V.L = F.L + off + (size_t) off * F.ld;
    V.Dinv = F.Dinv + off;
    V.K = Kp;
    V.KT = KTp;
    V.d_info = F.d_rec_info + kInfoBytes / 4 * R.count;
    V.fuse_k = true;
    V.kfamily = F.kfamily;
    R.off[R.count++] = off;
    return coop_factorize_enqueue(s, V, V.L, F.ld, false, nullptr);
}

bool rec_factor(cudaStream_t s, DenseFactor &F, int off, int n, RecLeaves &R) {
    const long ld = F.ld;
    if (n <= kRecLeafMaxN)
        return rec_leaf(s, F, off, n, F.K + off + (size_t) off * ld, F.KT + off + (size_t) off * ld, R);
    const int n1 = rec_split(n), n2 = n - n1;
    if (!rec_factor(s, F, off, n1, R)) return false;
    double *L21 = F.L + (off + n1) + (size_t) off * ld;
    double *A22 = F.L + (off + n1) + (size_t) (off + n1) * ld;
    const double *K11 = F.K + off + (size_t) off * ld, *KT11 = F.KT + off + (size_t) off * ld;
    const double *K22 = F.K + (off + n1) + (size_t) (off + n1) * ld;
    double *K21 = F.K + (off + n1) + (size_t) off * ld, *KT12 = F.KT + off + (size_t) (off + n1) * ld;
    double *W = F.d_rec_w;   // n2 x n1, leading dimension ld
    gemm(s, n2, n1, n1, 1.0, L21, ld, 0, KT11, ld, 0, 0.0, W, ld, GEMM_B_UPPER);      // A21 K11^T
    copy_matrix(s, n2, n1, W, ld, L21, ld);
    gemm(s, n2, n2, n1, -1.0, L21, ld, 0, L21, ld, 1, 1.0, A22, ld, GEMM_C_LOWER);    // A22 -= L21 L21^T
    if (!rec_factor(s, F, off + n1, n2, R)) return false;
    gemm(s, n2, n1, n1, 1.0, L21, ld, 0, K11, ld, 0, 0.0, W, ld, GEMM_B_LOWER);       // L21 K11
    gemm(s, n2, n1, n2, -1.0, K22, ld, 0, W, ld, 0, 0.0, K21, ld, GEMM_A_LOWER);      // -K22 (L21 K11)
    dim3 grid((n2 + 31) / 32, (n1 + 31) / 32), block(32, 8);
    transpose_rect_kernel<<<hb::counted(grid), block, 0, s>>>(n2, n1, K21, ld, KT12, ld);
    return cudaGetLastError() == cudaSuccess;
}

// X (rows x nL, leading dimension ldx) <- X L^-T for the diagonal block L of F at [Loff, Loff +
// nL), split as the factorisation split it: a leaf is one GEMM with that block's K^T (kept in
// the strip), otherwise Xa <- Xa La^-T, Xc -= Xa Lb^T, Xc <- Xc Lc^-T
bool rec_trsm(cudaStream_t s, DenseFactor &F, double *X, long ldx, int rows, int Loff, int nL) {
    const long ld = F.ld;
    if (nL <= kRecLeafMaxN) {
        gemm(s, rows, nL, nL, 1.0, X, ldx, 0, F.d_rec_kts + Loff, ld, 0, 0.0, F.d_rec_w, ld, GEMM_B_UPPER);
        copy_matrix(s, rows, nL, F.d_rec_w, ld, X, ldx);
        return true;
    }
    const int n1 = rec_split(nL), nc = nL - n1;
    if (!rec_trsm(s, F, X, ldx, rows, Loff, n1)) return false;
    gemm(s, rows, nc, n1, -1.0, X, ldx, 0, F.L + (Loff + n1) + (size_t) Loff * ld, ld, 1, 1.0, X + (size_t) n1 * ldx,
         ldx, 0);
    return rec_trsm(s, F, X + (size_t) n1 * ldx, ldx, rows, Loff + n1, nc);
}

// the recursive form without K: the diagonal blocks' K (and K^T) go to the strips
bool rec_factor_nok(cudaStream_t s, DenseFactor &F, int off, int n, RecLeaves &R) {
    const long ld = F.ld;
    if (n <= kRecLeafMaxN) return rec_leaf(s, F, off, n, F.d_rec_ks + off, F.d_rec_kts + off, R);
    const int n1 = rec_split(n), n2 = n - n1;
    if (!rec_factor_nok(s, F, off, n1, R)) return false;
    double *L21 = F.L + (off + n1) + (size_t) off * ld;
    double *A22 = F.L + (off + n1) + (size_t) (off + n1) * ld;
    if (!rec_trsm(s, F, L21, ld, n2, off, n1)) return false;                            // A21 L11^-T
    gemm(s, n2, n2, n1, -1.0, L21, ld, 0, L21, ld, 1, 1.0, A22, ld, GEMM_C_LOWER);    // A22 -= L21 L21^T
    return rec_factor_nok(s, F, off + n1, n2, R);
}
}  // namespace

bool rec_factorize_enqueue(cudaStream_t s, DenseFactor &F, const double *S, long ldS) {
    const int n = F.n;
    if (!F.d_rec_info && hb::cmalloc(&F.d_rec_info, kInfoBytes * kRecMaxLeaves) != cudaSuccess) {
        F.d_rec_info = nullptr;
        return false;
    }
    if (!F.d_rec_w && hb::cmalloc(&F.d_rec_w, sizeof(double) * F.ld * ((n + 1) / 2)) != cudaSuccess) {
        F.d_rec_w = nullptr;
        return false;
    }
    HB_CUDA(cudaMemsetAsync(F.d_rec_info, 0, kInfoBytes * kRecMaxLeaves, s));
    copy_lower_k<<<hb::counted(copy_lower_grid(n)), 256, 0, s>>>(n, S, ldS, F.L, F.ld, nullptr);
    RecLeaves R;
    R.count = 0;
    const bool ok = rec_factor(s, F, 0, n, R);
    rec_info_kernel<<<hb::counted(1), 32, 0, s>>>(R, F.d_rec_info, F.d_info);
    if (!ok) device_error_flag() = 1;
    return ok && cudaGetLastError() == cudaSuccess;
}

bool rec_factorize_nok_enqueue(cudaStream_t s, DenseFactor &F, const double *S, long ldS) {
    const int n = F.n;
    const size_t strip = (size_t) F.ld * kRecLeafMaxN;
    if (!F.d_rec_info && hb::cmalloc(&F.d_rec_info, kInfoBytes * kRecMaxLeaves) != cudaSuccess) {
        F.d_rec_info = nullptr;
        return false;
    }
    if (!F.d_rec_w && hb::cmalloc(&F.d_rec_w, sizeof(double) * strip) != cudaSuccess) {
        F.d_rec_w = nullptr;
        return false;
    }
    if (!F.d_rec_ks) {
        // zero outside the blocks' triangles, which the cooperative kernel never writes
        if (hb::cmalloc(&F.d_rec_ks, sizeof(double) * strip) != cudaSuccess ||
            hb::cmalloc(&F.d_rec_kts, sizeof(double) * strip) != cudaSuccess) {
            if (F.d_rec_ks) hb::cache_free(F.d_rec_ks);
            F.d_rec_ks = F.d_rec_kts = nullptr;
            return false;
        }
        HB_CUDA(cudaMemsetAsync(F.d_rec_ks, 0, sizeof(double) * strip, s));
        HB_CUDA(cudaMemsetAsync(F.d_rec_kts, 0, sizeof(double) * strip, s));
    }
    HB_CUDA(cudaMemsetAsync(F.d_rec_info, 0, kInfoBytes * kRecMaxLeaves, s));
    copy_lower_k<<<hb::counted(copy_lower_grid(n)), 256, 0, s>>>(n, S, ldS, F.L, F.ld, nullptr);
    RecLeaves R;
    R.count = 0;
    const bool ok = rec_factor_nok(s, F, 0, n, R);
    rec_info_kernel<<<hb::counted(1), 32, 0, s>>>(R, F.d_rec_info, F.d_info);
    if (!ok) device_error_flag() = 1;
    return ok && cudaGetLastError() == cudaSuccess;
}

// The factorisations of F[0..count) (each n <= kSmallFactorMaxN) of S[i] (ldS[i]) in launches of up to
// kSmallBatch CTAs, the status words written into each factor's pinned host mirror by the
// kernel; returns false (nothing enqueued) if a mirror has no device address, or false
// after a failed launch.
bool small_factor_batch_enqueue(cudaStream_t s, DenseFactor *const *F, const double *const *S, const long *ldS,
                                int count) {
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        HB_CUDA(cudaFuncSetAttribute((const void *) potrf_small_batch_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, SM_DOUBLES * (int) sizeof(double)));
        HB_CUDA(cudaFuncSetAttribute((const void *) potrf_batch_array_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, SM_DOUBLES * (int) sizeof(double)));
    });
    std::vector<SmallFactorJob> jobs(count);
    for (int q = 0; q < count; ++q) {
        DenseFactor &G = *F[q];
        double *hd = nullptr;
        if (cudaHostGetDevicePointer((void **) &hd, G.h_info, 0) != cudaSuccess || !hd) {
            cudaGetLastError();
            return false;
        }
        jobs[q] = SmallFactorJob{S[q], G.L, G.Dinv, G.fuse_k ? G.K : nullptr, G.fuse_k ? G.KT : nullptr, ldS[q], G.ld,
                                 G.d_info, hd, G.n, G.stat_logdet ? 1 : 0};
    }
    if (count <= kSmallBatch) {
        SmallFactorBatch B;
        for (int q = 0; q < count; ++q) B.job[q] = jobs[q];
        potrf_small_batch_kernel<<<hb::counted(count), COOP_THREADS, SM_DOUBLES * sizeof(double), s>>>(B);
        return cudaGetLastError() == cudaSuccess;
    }
    // more jobs than fit the parameters: one launch over a device copy of them, in a buffer kept
    // per host thread and device (every caller waits for the launch before its thread enqueues
    // another batch, so the buffer is free again by then)
    struct JobBuf {
        SmallFactorJob *p = nullptr;
        size_t cap = 0;
    };
    thread_local JobBuf buf[kMaxDevices];
    JobBuf &b = buf[current_device()];
    if (b.cap < (size_t) count) {
        if (b.p) hb::cache_free(b.p);
        b.cap = (size_t) count;
        if (hb::cmalloc(&b.p, sizeof(SmallFactorJob) * b.cap) != cudaSuccess) {
            b.p = nullptr;
            b.cap = 0;
            return false;
        }
    }
    HB_CUDA(cudaMemcpyAsync(b.p, jobs.data(), sizeof(SmallFactorJob) * count, cudaMemcpyHostToDevice, s));
    potrf_batch_array_kernel<<<hb::counted(count), COOP_THREADS, SM_DOUBLES * sizeof(double), s>>>(b.p);
    return cudaGetLastError() == cudaSuccess;
}

namespace {
// y -= A x (rows x cols, column-major): 32 rows a block, its warps taking the columns in turn
constexpr int kGemvThreads = 1024;
__global__ void __launch_bounds__(kGemvThreads)
    gemv_sub_kernel(int rows, int cols, const double *__restrict__ A, long lda, const double *__restrict__ x, double *y) {
    __shared__ double part[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = blockIdx.x * 32 + lane;
    double p[4] = {};
    if (r < rows) {
        const double *a = A + r;
        int c = w;
        for (; c + 96 < cols; c += 128) {
#pragma unroll
            for (int q = 0; q < 4; ++q) p[q] += __ldg(a + (size_t) (c + 32 * q) * lda) * __ldg(x + c + 32 * q);
        }
        for (int q = 0; c < cols; c += 32, ++q) p[q] += __ldg(a + (size_t) c * lda) * __ldg(x + c);
    }
    part[w][lane] = (p[0] + p[1]) + (p[2] + p[3]);
    __syncthreads();
    // warp w sums row w of the block
    double v = part[lane][w];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int row = blockIdx.x * 32 + w;
    if (lane == 0 && row < rows) y[row] -= v;
}

// the diagonal blocks of the recursive factorisation, in order
void rec_leaves(int off, int n, std::vector<std::pair<int, int>> &out) {
    if (n <= kRecLeafMaxN) {
        out.push_back({off, n});
        return;
    }
    const int n1 = rec_split(n);
    rec_leaves(off, n1, out);
    rec_leaves(off + n1, n - n1, out);
}

// Substitution by the diagonal blocks of the recursive factorisation, with their inverses from
// the strips: a block is a product with K and one with the rows (columns) of L below it. The two
// passes over L bound it (order 8000: 80 us of DRAM time); 64-row blocks in one cooperative
// launch are a chain of 2 n / 64 waits (order 4485 / 6000 / 8000: 684 / 972 / 1300 us, now 130 / 160 /
// 314).
bool rec_solve(cudaStream_t s, DenseFactor &F, const double *b, double *x) {
    const int n = F.n;
    const long ld = F.ld;
    std::vector<std::pair<int, int>> leaf;
    rec_leaves(0, n, leaf);
    double *t = F.d_tmp;
    HB_CUDA(cudaMemcpyAsync(t, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    for (auto [o, m] : leaf) {   // x <- L^-1 b, t the right-hand side left
        coldot(s, m, m, F.d_rec_kts + o, ld, t + o, x + o, 1.0, 0.0, 2);
        const int rows = n - o - m;
        if (rows > 0)
            gemv_sub_kernel<<<hb::counted((rows + 31) / 32), kGemvThreads, 0, s>>>(
                rows, m, F.L + (o + m) + (size_t) o * ld, ld, x + o, t + o + m);
    }
    for (size_t q = leaf.size(); q-- > 0;) {   // t <- L^-T x
        const auto [o, m] = leaf[q];
        const int rows = n - o - m;
        if (rows > 0) coldot(s, rows, m, F.L + (o + m) + (size_t) o * ld, ld, t + o + m, x + o, -1.0, 1.0, 0);
        coldot(s, m, m, F.d_rec_ks + o, ld, x + o, t + o, 1.0, 0.0, 1);
    }
    HB_CUDA(cudaMemcpyAsync(x, t, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    return cudaGetLastError() == cudaSuccess;
}
}  // namespace

bool chol_solve(cudaStream_t s, DenseFactor &F, const double *b, double *x) {
    const int n = F.n;
    if (n <= 0) return true;
    if (F.rec_strips) {
        if (!F.d_tmp) HB_CUDA(hb::cmalloc(&F.d_tmp, sizeof(double) * n));
        return F.d_tmp && rec_solve(s, F, b, x);
    }
    const int nblk = (n + 63) / 64;
    if (!F.d_flags) {
        HB_CUDA(hb::cmalloc(&F.d_flags, sizeof(unsigned) * 2 * nblk));
        HB_CUDA(cudaMemsetAsync(F.d_flags, 0, sizeof(unsigned) * 2 * nblk, s));
        F.epoch = 0;
    }
    if (!F.d_tmp) HB_CUDA(hb::cmalloc(&F.d_tmp, sizeof(double) * n));
    if (!F.d_flags || !F.d_tmp) return false;
    F.epoch += 1;
    const void *fn = (const void *) tri_solve_coop_kernel;
    const int G = std::min(nblk, sm_count());
    const int nown = (nblk + G - 1) / G;
    const int smem = (2 * 64 * TP + nown * 64 + 2 * 64 + 4 * 64) * (int) sizeof(double);
    {
        // the largest dynamic shared memory requested so far, per device
        static std::mutex mu;
        static int smem_set[kMaxDevices] = {0};
        std::lock_guard<std::mutex> g(mu);
        int &cur = smem_set[current_device()];
        if (smem > cur) {
            if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
                return false;
            cur = smem;
        }
    }
    const double *Lp = F.L;
    long ld = F.ld;
    int nn = n;
    const double *Dp = F.Dinv;
    long ldd = F.ld;
    const double *bp = b;
    double *tp = F.d_tmp, *xp = x;
    unsigned *ff = F.d_flags, *fb = F.d_flags + nblk;
    unsigned ep = F.epoch;
    void *args[] = {&Lp, &ld, &nn, &Dp, &ldd, &bp, &tp, &xp, &ff, &fb, &ep};
    cudaError_t e = cudaLaunchCooperativeKernel(fn, hb::counted(G), COOP_THREADS, args, smem, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

int chol_solve_error() {
    int h = 0;
    cudaMemcpyFromSymbol(&h, g_tri_err, sizeof(int));
    if (h) {
        const int z = 0;
        cudaMemcpyToSymbol(g_tri_err, &z, sizeof(int));
    }
    return h;
}

}  // namespace hb
