// Banded direct solve of the FP64 system matrices (the 2.5-D path).
//
// The reference factors every wavenumber's matrix with CHOLMOD and solves
// each current source with the factor (core/src/bert/dcfemmodelling.cpp:
// 2199-2210, core/src/cholmodWrapper.cpp:309-420).  The 2-D meshes of the
// 2.5-D path have a small bandwidth in their own node order (the para
// meshes: 17-28; otherwise reverse Cuthill-McKee is used when it is
// smaller), so the exact Cholesky factor L of A (L L^T = A, no pivoting, A
// SPD) fits a band of b+1 diagonals and costs n b^2 / 2 multiply-adds:
//
// Blocks of B = max(b, 8) consecutive rows in band order make the matrix block
// tridiagonal (N = ceil(n / B) dense blocks).  A serial band Cholesky has n
// dependent columns and one substitution chain per right-hand side; block
// cyclic reduction has log2(N) levels whose blocks are independent:
//   level s (stride): every odd multiple i of s is eliminated between its
//   neighbours l = i - s and r = i + s,
//     V_l = D_i^-1 A(i,l),  V_r = D_i^-1 A(i,r),
//     D_l -= A(l,i) V_l,  D_r -= A(r,i) V_r,  A(l,r) = -A(l,i) V_r,
//     f_l -= V_l^T f_i,  f_r -= V_r^T f_i,
//   then from the last level back x_i = D_i^-1 f_i - V_l x_l - V_r x_r.
// Every D_i is a Schur complement of an SPD matrix (a symmetric permutation of
// the Cholesky elimination), so its inverse by Gauss-Jordan needs no pivoting.
//
// Bound: the FP64 pipe (GB300: 1.2 TFLOP/s).  Per right-hand side the products
// cost 10 n B flops against the 4 n b of the serial substitutions, and the
// factor 11 n B^2 against n b^2, but every SM works on them.  Factor and solve,
// serial -> reduction: 16 electrodes (n 684, 14 wavenumbers) 3.54 -> 0.26 ms; 41
// electrodes (n 3618, b 19, 17 wavenumbers, 697 right-hand sides) 26.2 -> 1.15
// ms; 72 electrodes on a fine mesh (n 25992, b 25, 1296 right-hand sides) 229.6
// -> 11.7 ms, its widest level (k_cr_back, 2.2 ms) with the FP64 pipe 97 % active.
// The last levels hold few blocks; there the columns are split finer and the
// inverse's chain of B dependent steps (25-38 us per level) is what remains.
//
// Error against a refined extended-precision solution, potentials of 16- and
// 41-electrode lines on 30 grounds (log-normal sigma 1 to 4, bodies of 1e3 and 1e5
// times either way): 0.58 times the serial band's on average (geometric mean of the
// largest errors), 0.07 to 2.9 times on single grounds.
//
// Blocks wider than kCrMax rows (their inverse and one operand would not fit
// shared memory), and a response repeated after running out of memory (the 4 n B
// values per wavenumber), take the serial band Cholesky: B[j (b+1) + d] = L(j+d, j), one
// block per wavenumber factoring column by column, one thread per
// right-hand side in the substitutions.
//
// Rows are visited in the chosen order through a permutation, so the
// right-hand-side and solution blocks stay in the mesh's node order.  A pivot
// that is not positive stops the solve with an error (A must be SPD).
#include <algorithm>
#include <cmath>
#include <queue>

#include "ertgb_internal.cuh"

namespace ertgb {

namespace {

constexpr int kBandThreads = 256;

__global__ void __launch_bounds__(kBandThreads) k_band_fill(int64_t n, int b, int nK, int64_t nnz,
                                                             const int32_t *__restrict__ rowptr,
                                                             const int32_t *__restrict__ colidx,
                                                             const int32_t *__restrict__ pos,
                                                             const double *__restrict__ S, double *__restrict__ B) {
    const int64_t total = n * nK;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = t / n, i = t - k * n;
        const int64_t pi = pos[i];
        double *Bk = B + k * n * (b + 1);
        for (int32_t s = rowptr[i]; s < rowptr[i + 1]; s++) {
            const int64_t pj = pos[colidx[s]];
            if (pj <= pi) Bk[pj * (b + 1) + (pi - pj)] = S[k * nnz + s];
        }
    }
}

// one block per wavenumber: the band Cholesky factor in place
__global__ void __launch_bounds__(kBandThreads) k_band_factor(int64_t n, int b, double *__restrict__ B,
                                                               int32_t *__restrict__ bad) {
    __shared__ double col[kMaxBand + 1];
    double *A = B + (int64_t)blockIdx.x * n * (b + 1);
    const int tid = threadIdx.x;
    for (int64_t j = 0; j < n; j++) {
        const int m = (int)(n - 1 - j < (int64_t)b ? n - 1 - j : (int64_t)b);
        double *Aj = A + j * (b + 1);
        if (tid == 0) {
            double d = Aj[0];
            if (!(d > 0.0) || !isfinite(d)) {
                atomicAdd(bad, 1);
                d = 1.0;
            }
            col[0] = sqrt(d);
            Aj[0] = col[0];
        }
        __syncthreads();
        const double ljj = col[0];
        for (int i = 1 + tid; i <= m; i += kBandThreads) {
            const double v = Aj[i] / ljj;
            Aj[i] = v;
            col[i] = v;
        }
        __syncthreads();
        // a_{j+i, j+l} -= L_i L_l for 1 <= l <= i <= m (every pair a distinct entry)
        for (int l = 1; l <= m; l++) {
            const double cl = col[l];
            double *Al = A + (j + l) * (b + 1) - l;
            for (int i = l + tid; i <= m; i += kBandThreads) Al[i] -= col[i] * cl;
        }
        __syncthreads();
    }
}

// ------------------------------------------------ block cyclic reduction
constexpr int kCrMax = kDenseMax;  // widest block: D and one operand in shared memory (2 x 100 KB)
constexpr int kCrThreads = 256;
constexpr int kCrChunk = 32;     // inner-dimension chunk of the right-hand-side products
constexpr int kCrOut = 16;       // outputs per thread of the right-hand-side products, at most

// Matrix blocks of every wavenumber: D (diagonal, later its inverse), C
// (coupling of a block to the next active one), V_l and V_r, each N x B x B
// row-major.
struct CrMat {
    double *D, *C, *VL, *VR;
    int N, B;
    __device__ double *d(int k, int i) const { return D + ((int64_t)k * N + i) * B * B; }
    __device__ double *c(int k, int i) const { return C + ((int64_t)k * N + i) * B * B; }
    __device__ double *vl(int k, int i) const { return VL + ((int64_t)k * N + i) * B * B; }
    __device__ double *vr(int k, int i) const { return VR + ((int64_t)k * N + i) * B * B; }
};

__global__ void __launch_bounds__(kBandThreads) k_cr_fill(int64_t n, int nK, int64_t nnz,
                                                           const int32_t *__restrict__ rowptr,
                                                           const int32_t *__restrict__ colidx,
                                                           const int32_t *__restrict__ pos,
                                                           const double *__restrict__ S, CrMat m) {
    const int64_t rows = (int64_t)m.N * m.B, total = rows * nK;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t / rows);
        const int64_t i = t - k * rows;
        if (i >= n) {  // rows past the matrix: identity
            const int bi = (int)(i / m.B), r = (int)(i - (int64_t)bi * m.B);
            m.d(k, bi)[r * m.B + r] = 1.0;
            continue;
        }
        const int pi = pos[i], bi = pi / m.B, r = pi - bi * m.B;
        for (int32_t s = rowptr[i]; s < rowptr[i + 1]; s++) {
            const int pj = pos[colidx[s]], bj = pj / m.B, c = pj - bj * m.B;
            if (bj == bi) m.d(k, bi)[r * m.B + c] = S[(int64_t)k * nnz + s];
            else if (bj == bi + 1) m.c(k, bi)[r * m.B + c] = S[(int64_t)k * nnz + s];
        }
    }
}

// Elimination of block i = s + 2 s blockIdx.x: its inverse by Gauss-Jordan in
// shared memory, then V_l and V_r.  A thread owns one column of the inverse and
// every G-th row, so a step costs it one product and its rows' multiply-adds;
// the pivot's reciprocal is taken once, by the thread that updated the pivot,
// before the barrier that ends a step.  s = 0: the last block, inverse only.
__global__ void __launch_bounds__(kCrThreads) k_cr_eliminate(CrMat m, int s, int32_t *__restrict__ bad) {
    extern __shared__ double cr_smem[];
    const int B = m.B, k = blockIdx.y, tid = threadIdx.x;
    const int i = s ? s + 2 * s * (int)blockIdx.x : 0;
    double *A = cr_smem, *X = A + B * B, *prow = X + B * (B + 1), *pcol = prow + 2 * B, *rd = pcol + 2 * B;
    double *Di = m.d(k, i);
    for (int q = tid; q < B * B; q += kCrThreads) A[q] = Di[q];
    __syncthreads();
    const int G = kCrThreads / B, g = tid / B, j = tid - g * B;  // B <= kCrThreads: G >= 1
    auto reciprocal = [&](double d) {
        if (!(d > 0.0) || !isfinite(d)) {
            atomicAdd(bad, 1);
            d = 1.0;
        }
        return 1.0 / d;
    };
    if (tid < B) {
        prow[tid] = A[tid];
        pcol[tid] = A[tid * B];
        if (tid == 0) rd[0] = reciprocal(A[0]);
    }
    __syncthreads();
    for (int p = 0; p < B; p++) {
        const double *pr = prow + (p & 1) * B, *pc = pcol + (p & 1) * B;
        double *nr = prow + ((p + 1) & 1) * B, *nc = pcol + ((p + 1) & 1) * B;
        const double d = rd[p & 1];
        if (g < G) {
            const double f = pr[j] * d;  // the scaled pivot row at this thread's column
            for (int r = g; r < B; r += G) {
                double v;
                if (r == p) v = j == p ? d : f;
                else if (j == p) v = -pc[r] * d;
                else v = fma(-pc[r], f, A[r * B + j]);
                A[r * B + j] = v;
                if (r == p + 1) {
                    nr[j] = v;
                    if (j == p + 1) rd[(p + 1) & 1] = reciprocal(v);
                }
                if (j == p + 1) nc[r] = v;
            }
        }
        __syncthreads();
    }
    for (int q = tid; q < B * B; q += kCrThreads) Di[q] = A[q];
    if (!s) return;
    // V_l = D^-1 A(i,l) = D^-1 C[l]^T, V_r = D^-1 C[i]
    const double *Cl = m.c(k, i - s), *Ci = m.c(k, i);
    const int LD = B + 1;
    for (int q = tid; q < B * B; q += kCrThreads) {
        const int r = q / B;
        X[(q - r * B) * LD + r] = Cl[q];
    }
    __syncthreads();
    double *VL = m.vl(k, i), *VR = m.vr(k, i);
    const bool right = i + s < m.N;
    for (int pass = 0; pass < 2; pass++) {
        double *V = pass ? VR : VL;
        for (int q = tid; q < B * B; q += kCrThreads) {
            const int r = q / B, c = q - r * B;
            const double *a = A + r * B, *x = X + c;
            double s0 = 0.0, s1 = 0.0;
            int e = 0;
            for (; e + 1 < B; e += 2) {
                s0 = fma(a[e], x[e * LD], s0);
                s1 = fma(a[e + 1], x[(e + 1) * LD], s1);
            }
            if (e < B) s0 = fma(a[e], x[e * LD], s0);
            V[q] = s0 + s1;
        }
        if (pass || !right) break;
        __syncthreads();
        for (int q = tid; q < B * B; q += kCrThreads) {
            const int r = q / B;
            X[r * LD + (q - r * B)] = Ci[q];
        }
        __syncthreads();
    }
}

// Tile of right-hand sides: columns [c0, c0 + nc) of wavenumber k.
struct CrRhs {
    const int32_t *perm;
    double *x;
    int64_t n, Rpad;
    int nE, ntile;  // tiles per wavenumber
};

// acc += M F for one block product: M is B x B with element (row, q) at
// M[q * B + row] (trans) or M[row * B + q]; F the nc columns of block fb.
// Outputs o of a thread: (row, column) = divmod(tid + o kCrThreads, nc).
template <int NO, bool TRANS>
__device__ __forceinline__ void cr_product(const CrMat &m, const CrRhs &R, const double *__restrict__ M, int k, int fb,
                                           int c0, int nc, double sign, double *Ms, double *Fs, const int (&ro)[NO],
                                           const int (&co)[NO], double (&acc)[NO]) {
    const int B = m.B, tid = threadIdx.x;
    for (int q0 = 0; q0 < B; q0 += kCrChunk) {
        const int qn = min(kCrChunk, B - q0);
        __syncthreads();  // the previous chunk is consumed
        for (int t = tid; t < qn * B; t += kCrThreads) {
            if (TRANS) {
                Ms[t] = sign * M[q0 * B + t];
            } else {
                const int r = t / qn, q = t - r * qn;
                Ms[q * B + r] = sign * M[r * B + q0 + q];
            }
        }
        for (int t = tid; t < qn * nc; t += kCrThreads) {
            const int q = t / nc, c = t - q * nc;
            const int64_t row = (int64_t)fb * B + q0 + q;
            Fs[t] = row < R.n ? R.x[(int64_t)R.perm[row] * R.Rpad + (int64_t)k * R.nE + c0 + c] : 0.0;
        }
        __syncthreads();
        for (int q = 0; q < qn; q++) {
#pragma unroll
            for (int o = 0; o < NO; o++)
                if (tid + o * kCrThreads < B * nc) acc[o] = fma(Ms[q * B + ro[o]], Fs[q * nc + co[o]], acc[o]);
        }
    }
}

// Update of the kept block j = 2 s e by its eliminated neighbours: the matrix
// part (blocks [0, n_kept)) and the right-hand-side part (the others, one tile
// of columns each) of one level share a launch: neither reads what the other
// writes.
template <int NO>
__global__ void __launch_bounds__(kCrThreads) k_cr_update(CrMat m, int s, int n_kept, CrRhs R) {
    extern __shared__ double cr_smem[];
    const int B = m.B, k = blockIdx.y, tid = threadIdx.x;
    if ((int)blockIdx.x < n_kept) {
        const int j = 2 * s * (int)blockIdx.x, i1 = j - s, i2 = j + s;
        double *A = cr_smem, *X = A + B * B;
        double *Dj = m.d(k, j), *Cj = m.c(k, j);
        const int half = B * (B + 1) / 2;
        // D_j -= P^T-or-P times V, symmetric: the lower triangle, mirrored
        auto rank_update = [&](bool trans) {
            for (int q = tid; q < half; q += kCrThreads) {
                int r = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
                while ((r + 1) * (r + 2) / 2 <= q) r++;
                while (r * (r + 1) / 2 > q) r--;
                const int c = q - r * (r + 1) / 2;
                const double *a = trans ? A + r : A + r * B;
                const int st = trans ? B : 1;
                double s0 = 0.0, s1 = 0.0;
                int e = 0;
                for (; e + 1 < B; e += 2) {
                    s0 = fma(a[e * st], X[e * B + c], s0);
                    s1 = fma(a[(e + 1) * st], X[(e + 1) * B + c], s1);
                }
                if (e < B) s0 = fma(a[e * st], X[e * B + c], s0);
                const double v = Dj[r * B + c] - (s0 + s1);
                Dj[r * B + c] = v;
                Dj[c * B + r] = v;
            }
        };
        if (i2 < m.N) {
            const double *VL = m.vl(k, i2), *VR = m.vr(k, i2);
            for (int q = tid; q < B * B; q += kCrThreads) {
                A[q] = Cj[q];
                X[q] = VL[q];
            }
            __syncthreads();
            rank_update(false);
            if (i2 + s < m.N) {
                __syncthreads();
                for (int q = tid; q < B * B; q += kCrThreads) X[q] = VR[q];
                __syncthreads();
                for (int q = tid; q < B * B; q += kCrThreads) {
                    const int r = q / B, c = q - r * B;
                    double s0 = 0.0, s1 = 0.0;
                    int e = 0;
                    for (; e + 1 < B; e += 2) {
                        s0 = fma(A[r * B + e], X[e * B + c], s0);
                        s1 = fma(A[r * B + e + 1], X[(e + 1) * B + c], s1);
                    }
                    if (e < B) s0 = fma(A[r * B + e], X[e * B + c], s0);
                    Cj[q] = -(s0 + s1);
                }
            }
        }
        if (i1 >= 0) {
            const double *C1 = m.c(k, i1), *VR = m.vr(k, i1);
            __syncthreads();
            for (int q = tid; q < B * B; q += kCrThreads) {
                A[q] = C1[q];
                X[q] = VR[q];
            }
            __syncthreads();
            rank_update(true);
        }
        return;
    }
    // f_j -= V_r(i1)^T f_i1 + V_l(i2)^T f_i2
    const int t = (int)blockIdx.x - n_kept, j = 2 * s * (t / R.ntile), i1 = j - s, i2 = j + s, tile = t % R.ntile;
    const int c0 = (int)((int64_t)R.nE * tile / R.ntile), nc = (int)((int64_t)R.nE * (tile + 1) / R.ntile) - c0;
    double *Ms = cr_smem, *Fs = Ms + kCrChunk * B;
    int ro[NO], co[NO];
    double acc[NO];
#pragma unroll
    for (int o = 0; o < NO; o++) {
        const int q = tid + o * kCrThreads;
        ro[o] = q / nc;
        co[o] = q - ro[o] * nc;
        acc[o] = 0.0;
    }
    if (i1 >= 0) cr_product<NO, true>(m, R, m.vr(k, i1), k, i1, c0, nc, -1.0, Ms, Fs, ro, co, acc);
    if (i2 < m.N) cr_product<NO, true>(m, R, m.vl(k, i2), k, i2, c0, nc, -1.0, Ms, Fs, ro, co, acc);
#pragma unroll
    for (int o = 0; o < NO; o++) {
        const int64_t row = (int64_t)j * B + ro[o];
        if (tid + o * kCrThreads < B * nc && row < R.n)
            R.x[(int64_t)R.perm[row] * R.Rpad + (int64_t)k * R.nE + c0 + co[o]] += acc[o];
    }
}

// x_i = D_i^-1 f_i - V_l x_l - V_r x_r of the blocks eliminated at stride s
// (s = 0: the last block, no neighbours); one tile of columns per block
template <int NO>
__global__ void __launch_bounds__(kCrThreads) k_cr_back(CrMat m, int s, CrRhs R) {
    extern __shared__ double cr_smem[];
    const int B = m.B, k = blockIdx.y, tid = threadIdx.x, tile = (int)blockIdx.x % R.ntile;
    const int i = s ? s + 2 * s * ((int)blockIdx.x / R.ntile) : 0;
    const int c0 = (int)((int64_t)R.nE * tile / R.ntile), nc = (int)((int64_t)R.nE * (tile + 1) / R.ntile) - c0;
    double *Ms = cr_smem, *Fs = Ms + kCrChunk * B;
    int ro[NO], co[NO];
    double acc[NO];
#pragma unroll
    for (int o = 0; o < NO; o++) {
        const int q = tid + o * kCrThreads;
        ro[o] = q / nc;
        co[o] = q - ro[o] * nc;
        acc[o] = 0.0;
    }
    cr_product<NO, false>(m, R, m.d(k, i), k, i, c0, nc, 1.0, Ms, Fs, ro, co, acc);
    if (s) {
        cr_product<NO, false>(m, R, m.vl(k, i), k, i - s, c0, nc, -1.0, Ms, Fs, ro, co, acc);
        if (i + s < m.N) cr_product<NO, false>(m, R, m.vr(k, i), k, i + s, c0, nc, -1.0, Ms, Fs, ro, co, acc);
    }
#pragma unroll
    for (int o = 0; o < NO; o++) {
        const int64_t row = (int64_t)i * B + ro[o];
        if (tid + o * kCrThreads < B * nc && row < R.n)
            R.x[(int64_t)R.perm[row] * R.Rpad + (int64_t)k * R.nE + c0 + co[o]] = acc[o];
    }
}

// Column tiles of a level with nblk independent blocks per wavenumber: at most
// kCrOut outputs per thread and 48 columns, narrower (8 at least) while the
// launch has fewer than two blocks per SM.
int cr_tiles(int B, int nE, int64_t blocks, int nsm) {
    int nc = std::min(48, kCrOut * kCrThreads / B);
    int nt = (nE + nc - 1) / nc;
    while (blocks * nt < 2 * nsm && nE / (2 * nt) >= 8) nt *= 2;
    return nt;
}

template <template <int> class F, typename... A> void by_outputs(int B, int nc, A &&...args) {
    const int no = (B * nc + kCrThreads - 1) / kCrThreads;
    if (no <= 2) F<2>::go(args...);
    else if (no <= 4) F<4>::go(args...);
    else if (no <= 8) F<8>::go(args...);
    else F<kCrOut>::go(args...);
}

// the inverse, one operand, two pivot rows and columns, two reciprocals
size_t eliminate_smem(int B) {
    return sizeof(double) * ((size_t)B * B + (size_t)B * (B + 1) + 4 * B + 2);
}

// The limit is per function, not per launch, and a batch solves its problems on
// several host threads: always the same value, the widest block's need.
template <class K> void allow_smem(K kern) {
    ERTGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)eliminate_smem(kCrMax)));
}

template <int NO> struct CrUpdateL {
    static void go(dim3 g, size_t smem, cudaStream_t st, const CrMat &m, int s, int n_kept, const CrRhs &R) {
        allow_smem(k_cr_update<NO>);
        k_cr_update<NO><<<g, kCrThreads, smem, st>>>(m, s, n_kept, R);
    }
};
template <int NO> struct CrBackL {
    static void go(dim3 g, size_t smem, cudaStream_t st, const CrMat &m, int s, const CrRhs &R) {
        allow_smem(k_cr_back<NO>);
        k_cr_back<NO><<<g, kCrThreads, smem, st>>>(m, s, R);
    }
};

// Factor and solve; x holds the right-hand sides and receives the solution.
// Returns the kernels launched.
int cr_solve(Context &c, CrMat m, const int32_t *perm, double *x, int32_t *bad, cudaStream_t st) {
    const int B = m.B, N = m.N, nK = c.nK;
    int nsm = 0, launches = 0;
    ERTGB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    const size_t elim = eliminate_smem(B);
    allow_smem(k_cr_eliminate);
    auto rhs_smem = [&](int nc) { return sizeof(double) * (size_t)kCrChunk * (B + nc); };
    std::vector<int> strides;
    for (int s = 1; s < N; s *= 2) strides.push_back(s);
    CrRhs R{perm, x, c.mesh.n, c.Rpad, c.nE, 1};
    for (int s : strides) {
        const int n_elim = (N - 1 - s) / (2 * s) + 1, n_kept = (N - 1) / (2 * s) + 1;
        k_cr_eliminate<<<dim3((unsigned)n_elim, (unsigned)nK), kCrThreads, elim, st>>>(m, s, bad);
        R.ntile = cr_tiles(B, c.nE, (int64_t)n_kept * nK, nsm);
        const int nc = (c.nE + R.ntile - 1) / R.ntile;
        const size_t smem = std::max(sizeof(double) * 2 * (size_t)B * B, rhs_smem(nc));
        by_outputs<CrUpdateL>(B, nc, dim3((unsigned)(n_kept * (1 + R.ntile)), (unsigned)nK), smem, st, m, s, n_kept, R);
        launches += 2;
    }
    k_cr_eliminate<<<dim3(1, (unsigned)nK), kCrThreads, elim, st>>>(m, 0, bad);
    auto back = [&](int s) {  // s = 0: the last block
        const int nblk = s ? (N - 1 - s) / (2 * s) + 1 : 1;
        R.ntile = cr_tiles(B, c.nE, (int64_t)nblk * nK, nsm);
        const int nc = (c.nE + R.ntile - 1) / R.ntile;
        by_outputs<CrBackL>(B, nc, dim3((unsigned)(nblk * R.ntile), (unsigned)nK), rhs_smem(nc), st, m, s, R);
    };
    back(0);
    for (size_t l = strides.size(); l-- > 0;) back(strides[l]);
    ERTGB_CUDA(cudaGetLastError());
    return launches + 2 + (int)strides.size();
}

// one block per wavenumber, one thread per right-hand side of it: forward
// and backward substitution in place on x (node-major n x Rpad), rows
// visited in band order through perm
__global__ void __launch_bounds__(kBandThreads) k_band_solve(int64_t n, int b, int nE, int64_t Rpad,
                                                              const double *__restrict__ B,
                                                              const int32_t *__restrict__ perm,
                                                              double *__restrict__ x) {
    const int k = blockIdx.x;
    const double *L = B + (int64_t)k * n * (b + 1);
    for (int e = threadIdx.x; e < nE; e += blockDim.x) {
        double *xc = x + (int64_t)k * nE + e;
        for (int64_t j = 0; j < n; j++) {
            const double *Lj = L + j * (b + 1);
            const int m = (int)(n - 1 - j < (int64_t)b ? n - 1 - j : (int64_t)b);
            const double y = xc[(int64_t)perm[j] * Rpad] / Lj[0];
            xc[(int64_t)perm[j] * Rpad] = y;
            for (int i = 1; i <= m; i++) xc[(int64_t)perm[j + i] * Rpad] -= Lj[i] * y;
        }
        for (int64_t j = n - 1; j >= 0; j--) {
            const double *Lj = L + j * (b + 1);
            const int m = (int)(n - 1 - j < (int64_t)b ? n - 1 - j : (int64_t)b);
            double s = xc[(int64_t)perm[j] * Rpad];
            for (int i = 1; i <= m; i++) s -= Lj[i] * xc[(int64_t)perm[j + i] * Rpad];
            xc[(int64_t)perm[j] * Rpad] = s / Lj[0];
        }
    }
}

// bandwidth of the pattern under the order pos (old index -> new)
int bandwidth(int64_t n, const std::vector<int32_t> &rp, const std::vector<int32_t> &ci,
              const std::vector<int32_t> &pos) {
    int64_t bw = 0;
    for (int64_t i = 0; i < n; i++)
        for (int32_t q = rp[i]; q < rp[i + 1]; q++) bw = std::max<int64_t>(bw, std::abs((int64_t)pos[i] - pos[ci[q]]));
    return (int)std::min<int64_t>(bw, INT32_MAX);
}

// reverse Cuthill-McKee: breadth-first from a low-degree node of each
// component, neighbours by increasing degree, the order reversed
std::vector<int32_t> rcm_order(int64_t n, const std::vector<int32_t> &rp, const std::vector<int32_t> &ci) {
    std::vector<int32_t> order;
    order.reserve((size_t)n);
    std::vector<char> seen((size_t)n, 0);
    auto deg = [&](int64_t i) { return rp[i + 1] - rp[i]; };
    std::vector<int32_t> byDeg((size_t)n);
    for (int64_t i = 0; i < n; i++) byDeg[(size_t)i] = (int32_t)i;
    std::stable_sort(byDeg.begin(), byDeg.end(), [&](int32_t a, int32_t c) { return deg(a) < deg(c); });
    std::vector<int32_t> nb;
    for (int32_t start : byDeg) {
        if (seen[start]) continue;
        std::queue<int32_t> q;
        q.push(start);
        seen[start] = 1;
        while (!q.empty()) {
            const int32_t v = q.front();
            q.pop();
            order.push_back(v);
            nb.clear();
            for (int32_t p = rp[v]; p < rp[v + 1]; p++)
                if (!seen[ci[p]]) {
                    seen[ci[p]] = 1;
                    nb.push_back(ci[p]);
                }
            std::stable_sort(nb.begin(), nb.end(), [&](int32_t a, int32_t c) { return deg(a) < deg(c); });
            for (int32_t w : nb) q.push(w);
        }
    }
    std::reverse(order.begin(), order.end());
    return order;
}

void band_plan(Context &c) {
    MeshData &m = c.mesh;
    BandPlan &P = m.band;
    if (P.built) return;
    P.built = true;
    const int64_t n = m.n;
    std::vector<int32_t> ident((size_t)n);
    for (int64_t i = 0; i < n; i++) ident[(size_t)i] = (int32_t)i;
    const int b0 = bandwidth(n, m.rowptr, m.colidx, ident);
    std::vector<int32_t> perm = ident;
    int b = b0;
    if (b0 > 16) {
        std::vector<int32_t> rcm = rcm_order(n, m.rowptr, m.colidx), pos((size_t)n);
        for (int64_t i = 0; i < n; i++) pos[(size_t)rcm[(size_t)i]] = (int32_t)i;
        const int b1 = bandwidth(n, m.rowptr, m.colidx, pos);
        if (b1 < b0) {
            perm = rcm;
            b = b1;
        }
    }
    P.b = b;
    P.ok = b <= kMaxBand;
    if (!P.ok) return;
    P.perm = perm;
    P.pos.assign((size_t)n, 0);
    for (int64_t i = 0; i < n; i++) P.pos[(size_t)perm[(size_t)i]] = (int32_t)i;
    P.d_perm.upload(P.perm, c.stream);
    P.d_pos.upload(P.pos, c.stream);
}

}  // namespace

void dense_inverse(double *A, int n, int32_t *bad, cudaStream_t s) {
    const CrMat M{A, nullptr, nullptr, nullptr, 1, n};
    allow_smem(k_cr_eliminate);
    k_cr_eliminate<<<1, kCrThreads, eliminate_smem(n), s>>>(M, 0, bad);
    ERTGB_CUDA(cudaGetLastError());
}

int band_solve(Context &c, cudaStream_t s) {
    MeshData &m = c.mesh;
    band_plan(c);
    const BandPlan &P = m.band;
    if (!P.ok)
        throw Error(ERTGB_BAD_INPUT, "the banded direct solve needs a matrix bandwidth of at most " +
                                         std::to_string(kMaxBand) + " (this matrix: " + std::to_string(P.b) +
                                         "); use an iterative preconditioner");
    const int64_t n = m.n, b = P.b;
    DBuf<int32_t> &bad = c.d_ic_bad;
    bad.alloc(1);
    bad.zero(s);
    // the solution overwrites a copy of the right-hand sides (d_r keeps them)
    c.d_x.alloc((size_t)n * c.Rpad);
    ERTGB_CUDA(cudaMemcpyAsync(c.d_x.p, c.d_r.p, sizeof(double) * n * c.Rpad, cudaMemcpyDeviceToDevice, s));
    const int B = (int)std::max<int64_t>(b, 8), N = (int)ceil_div(n, B);
    const size_t blk = (size_t)c.nK * N * B * B;
    const bool reduction = B <= kCrMax && !c.lean;
    if (reduction) {
        c.d_band.alloc(4 * blk);
        const CrMat M{c.d_band.p, c.d_band.p + blk, c.d_band.p + 2 * blk, c.d_band.p + 3 * blk, N, B};
        ERTGB_CUDA(cudaMemsetAsync(M.D, 0, sizeof(double) * 2 * blk, s));
        k_cr_fill<<<(unsigned)std::min<int64_t>(ceil_div((int64_t)N * B * c.nK, kBandThreads), 4096), kBandThreads, 0,
                    s>>>(n, c.nK, m.nnz, m.d_rowptr.p, m.d_colidx.p, P.d_pos.p, c.d_S.p, M);
        c.stats.launches_response += 1 + cr_solve(c, M, P.d_perm.p, c.d_x.p, bad.p, s);
    } else {
        const size_t per = (size_t)n * (size_t)(b + 1);
        c.d_band.alloc(per * c.nK);
        ERTGB_CUDA(cudaMemsetAsync(c.d_band.p, 0, sizeof(double) * per * c.nK, s));
        k_band_fill<<<(unsigned)std::min<int64_t>(ceil_div(n * c.nK, kBandThreads), 4096), kBandThreads, 0, s>>>(
            n, (int)b, c.nK, m.nnz, m.d_rowptr.p, m.d_colidx.p, P.d_pos.p, c.d_S.p, c.d_band.p);
        k_band_factor<<<c.nK, kBandThreads, 0, s>>>(n, (int)b, c.d_band.p, bad.p);
        k_band_solve<<<c.nK, std::min(kBandThreads, ((c.nE + 31) / 32) * 32), 0, s>>>(n, (int)b, c.nE, c.Rpad,
                                                                                      c.d_band.p, P.d_perm.p, c.d_x.p);
        c.stats.launches_response += 3;
    }
    ERTGB_CUDA(cudaGetLastError());
    int32_t h = 0;
    ERTGB_CUDA(cudaMemcpyAsync(&h, bad.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    ERTGB_CUDA(cudaStreamSynchronize(s));
    c.stats.iterations = 0;
    c.stats.max_rel_residual = 0.0;
    c.stats.n_rhs = (int32_t)c.R;
    if (h) throw Error(ERTGB_NOT_CONVERGED, "banded Cholesky: " + std::to_string(h) + " pivots not positive");
    return ERTGB_OK;
}

}  // namespace ertgb
