// Multilevel preconditioner of the mixed-precision PCG on 3-D meshes.
//
// A single-level factor (Jacobi, FSAI, the network's) leaves the smooth error
// of a 3-D potential problem to the CG recurrence: its iterations grow with
// the mesh (FSAI 448 at 23k nodes, 1088 at 145k).  Coarse levels (coarsen.cpp)
// take that error out; one symmetric V(1,1) cycle per iteration keeps the
// count at 20-40 on log-normal ground of sigma 1, whatever the mesh.  P knows the
// geometry only, so rough ground takes more (23k nodes, Jacobi / FSAI: 84 / 42 at
// sigma 2, 126 / 60 at 3, 270 / 96 at 4; single level 1024 / 384, 2560 / 384 and
// 4960 / 512).  Fine-level smoother: the chosen factor, w G^T G, or Jacobi;
// Jacobi on the coarse levels; the dense inverse (FP64, at most 64 rows)
// at the bottom.
//
// Jacobi levels.  With D = diag(dw), dw_i = 1.5 / sum_j |a_ij| (the spectrum
// of D A lies in [0, 1.5]) and the right-hand side b, the two sweeps need one
// product with A between them:
//     r = b - (A D) b            residual after the first sweep
//     e = coarse(P^T r)
//     z = D (b + r) + (P - D A P) e
// because D b + P e + D (b - A (D b + P e)) = D (b + r) + (P - D A P) e.
// A P is there from the Galerkin product, holds about 10 entries per row
// against A's 14 and gathers rows of the four times smaller coarse block.
// Factor level: with t = G b and x = w G^T t,
//     r = b - A x,  e = coarse(P^T r),  r -= (A P) e,  t += G r,
//     z = w G^T t + P e   ( = x + P e + w G^T G r )
// so neither sweep reads the iterate it corrects.
//
// Bound: the gathers of dense-block rows through L1 / L2, as the operator
// itself (k_spmm32_q); the small levels are latency and launches.  Solve, single
// level -> this: 23k nodes, 96 sources (FSAI) 23.9 -> 5.6 ms; 88k nodes, 96
// sources (FSAI) 160.5 -> 18.2; 145k nodes, 256 sources (learned) 748 -> 77;
// 38k nodes, 35 sources (Jacobi) 48.9 -> 6.9.
//
// Precision: matrices, Galerkin products and the coarsest inverse in FP64.  The
// mixed solver's cycle holds their FP32 copies and FP32 vectors, as its factors
// were applied before (its FP64 true residual decides convergence); the FP64
// solver's cycle is FP64 throughout (Jacobi levels; 23k nodes, 96 sources: 671
// iterations -> 39, 78.5 -> 20.8 ms).
#include <algorithm>
#include <cmath>

#include "ertgb_internal.cuh"

namespace ertgb {

namespace {

constexpr int64_t kMlMinRows = 1024;  // smallest matrix with coarse levels (ml_setup)
constexpr int kMlMaxLevels = 16;
constexpr int64_t kMlCoarsest = 64;   // largest bottom level (its inverse is one block of that many dependent steps)
constexpr double kOmega = 1.5;        // damping against a spectrum bound of 1
constexpr int kPower = 8;             // power iterations for the factor's damping
constexpr float kPowerSafety = 1.1f;  // the Rayleigh quotient is a lower bound
constexpr int kT = 256, kGroups = kT / 8;
constexpr int64_t kFill = 304;        // blocks that fill the chip: two on each of its 152 SMs

// position of column c in the ascending row [q0, q1)
__device__ __forceinline__ int32_t find_col(const int32_t *__restrict__ ci, int32_t q0, int32_t q1, int32_t c) {
    while (q0 + 1 < q1) {
        const int32_t h = (q0 + q1) >> 1;
        if (ci[h] <= c) q0 = h;
        else q1 = h;
    }
    return q0;
}

// Row i of A P and what follows from it, one warp per row: lanes own entries
// (i, J) of A P's pattern and scan the row's products a_ij P_jJ, which the warp
// reads once (no search, no conflicting sums; one thread per row with a search
// per product took 276 us a level on a 23k-node mesh).  Also
//   dw_i = kOmega / sum_j |a_ij|  (a row without a positive diagonal or with a
//     value that is not finite counts as bad),
//   Q = P - diag(dw) A P  (Jacobi level) or Q = -A P (factor level).
template <typename T>
__global__ void k_ml_rows(int64_t n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                          const double *__restrict__ val, const int32_t *__restrict__ prp,
                          const int32_t *__restrict__ pci, const float *__restrict__ pv,
                          const int32_t *__restrict__ arp, const int32_t *__restrict__ aci, int jacobi,
                          double *__restrict__ ap, T *__restrict__ dw, T *__restrict__ Q,
                          int32_t *__restrict__ bad) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const int32_t s0 = rp[i], s1 = rp[i + 1];
        double sum = 0.0;
        int diag = 0;
        for (int32_t s = s0 + lane; s < s1; s += 32) {
            const double a = val[s];
            sum += fabs(a);
            diag |= ci[s] == i && a > 0.0;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        diag = __any_sync(0xffffffffu, diag);
        const T d = (T)(kOmega / sum);
        if (lane == 0) {
            if (!diag || !isfinite(sum)) atomicAdd(bad, 1);
            dw[i] = d;
        }
        const int32_t a0 = arp[i], a1 = arp[i + 1], p0 = prp[i], p1 = prp[i + 1];
        for (int32_t q = a0 + lane; q < a1; q += 32) {
            const int32_t J = aci[q];
            double acc = 0.0;
            for (int32_t s = s0; s < s1; s++) {
                const double a = val[s];
                const int32_t j = ci[s];
                for (int32_t p = prp[j]; p < prp[j + 1]; p++)
                    if (pci[p] == J) acc = fma(a, (double)pv[p], acc);
            }
            ap[q] = acc;
            if (jacobi) {
                double e = 0.0;
                for (int32_t p = p0; p < p1; p++)
                    if (pci[p] == J) e = (double)pv[p];
                Q[q] = (T)(e - (double)d * acc);
            } else {
                Q[q] = (T)-acc;
            }
        }
    }
}

// AS = A diag(dw)
template <typename T>
__global__ void k_ml_scale(int64_t nnz, const int32_t *__restrict__ ci, const double *__restrict__ val,
                           const T *__restrict__ dw, T *__restrict__ AS) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nnz; t += (int64_t)gridDim.x * blockDim.x)
        AS[t] = (T)(val[t] * (double)dw[ci[t]]);
}

// P^T (A P), one warp per coarse row: the fine rows in order, lanes over the
// distinct columns of a row of A P
__global__ void k_ml_galerkin(int64_t nc, const int32_t *__restrict__ trp, const int32_t *__restrict__ tci,
                              const float *__restrict__ tv, const int32_t *__restrict__ arp,
                              const int32_t *__restrict__ aci, const double *__restrict__ ap,
                              const int32_t *__restrict__ crp, const int32_t *__restrict__ cci, double *cv) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t I = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; I < nc; I += warps) {
        const int32_t c0 = crp[I], c1 = crp[I + 1];
        for (int32_t q = c0 + lane; q < c1; q += 32) cv[q] = 0.0;
        __syncwarp();
        for (int32_t t = trp[I]; t < trp[I + 1]; t++) {
            const int32_t i = tci[t];
            const double w = (double)tv[t];
            for (int32_t p = arp[i] + lane; p < arp[i + 1]; p += 32) {
                const int32_t q = find_col(cci, c0, c1, aci[p]);
                cv[q] = fma(w, ap[p], cv[q]);
            }
            __syncwarp();
        }
    }
}

__global__ void k_ml_densify(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                             const double *__restrict__ val, double *__restrict__ A) {
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        for (int j = threadIdx.x; j < n; j += blockDim.x) A[(int64_t)i * n + j] = 0.0;
        __syncthreads();
        for (int32_t s = rp[i] + threadIdx.x; s < rp[i + 1]; s += blockDim.x) A[(int64_t)i * n + ci[s]] = val[s];
        __syncthreads();
    }
}

template <typename T> __global__ void k_ml_symmetric(int n, const double *__restrict__ A, T *__restrict__ B) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < (int64_t)n * n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / n, j = t - i * n;
        B[t] = (T)(0.5 * (A[t] + A[j * n + i]));
    }
}

// Sparse product over dense-block rows, the operator's layout (k_spmm32_q):
// 8-lane groups, CH float4 per lane; a group takes a row alone (SPLIT = 1), or a
// warp's four groups share one row's entries (SPLIT = 4, CH = 1): the short
// levels have few rows of up to a hundred entries and are bound by that chain.
// The row-local rest of the cycle's step is the epilogue:
enum Ep {
    EP_PLAIN,  // y = B x
    EP_RESID,  // y = b - B x
    EP_POST,   // y = dw (b + r) + B x
    EP_SCALE,  // y = w B x
    EP_ACC,    // y += B x
    EP_FINAL,  // y = w B x + P e
};
// four adjacent columns
template <typename T> struct Four;
template <> struct Four<float> { using V = float4; };
struct alignas(32) Double4 { double x, y, z, w; };
template <> struct Four<double> { using V = Double4; };
__device__ __forceinline__ float4 load4(const float4 *p) { return __ldg(p); }
__device__ __forceinline__ Double4 load4(const Double4 *p) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p)), b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    return {a.x, a.y, b.x, b.y};
}

// Operands of one product; unused ones stay null.
template <typename T> struct Args {
    const T *b = nullptr, *r = nullptr, *dw = nullptr, *w = nullptr;
    const int32_t *prp = nullptr, *pci = nullptr;  // EP_FINAL: P by rows and the coarse block it multiplies
    const T *pv = nullptr, *e = nullptr;
    double *part = nullptr;                        // DOT: column partials of b . y
    int NB = 0;                                    // their block rows
};

template <typename T, typename V> __device__ __forceinline__ void axpy4(V &y, T v, const V &x) {
    y.x = fma(v, x.x, y.x);
    y.y = fma(v, x.y, y.y);
    y.z = fma(v, x.z, y.z);
    y.w = fma(v, x.w, y.w);
}

template <typename T, int CH, int SPLIT, int EP, bool DOT>
__global__ void __launch_bounds__(kT, 2)
    k_ml_spmm(int64_t n, int64_t Rpad, int tile_rows, const int32_t *__restrict__ rowptr,
              const int32_t *__restrict__ colidx, const T *__restrict__ vals, const T *__restrict__ x,
              T *__restrict__ y, Args<T> A) {
    using V = typename Four<T>::V;
    static_assert(SPLIT == 1 || (CH == 1 && !DOT), "split rows: one chunk, no partials");
    constexpr int ROWS = kGroups / SPLIT;  // rows of a block at a time
    __shared__ T red[DOT ? kGroups : 1][DOT ? 32 * CH + 1 : 1];
    const int l8 = threadIdx.x & 7, g = threadIdx.x >> 3, sub = SPLIT == 1 ? 0 : g % SPLIT;
    const int64_t t0 = (int64_t)blockIdx.y * 32 * CH + l8 * 4;
    const T ws = (EP == EP_SCALE || EP == EP_FINAL) ? *A.w : (T)0;
    V dot[CH];
#pragma unroll
    for (int j = 0; j < CH; j++) dot[j] = V{0, 0, 0, 0};
    const int64_t ntile = (n + tile_rows - 1) / tile_rows;
    for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x)
        for (int64_t row = tile * tile_rows + g / SPLIT, end = min(n, (tile + 1) * tile_rows); row < end; row += ROWS) {
            V acc[CH];
#pragma unroll
            for (int j = 0; j < CH; j++) acc[j] = V{0, 0, 0, 0};
            const int32_t s1 = rowptr[row + 1];
#pragma unroll(CH == 1 ? 8 : 4)
            for (int32_t s = rowptr[row] + sub; s < s1; s += SPLIT) {
                const int64_t col = colidx[s];
                const T v = vals[s];
                const V *xc = reinterpret_cast<const V *>(x + col * Rpad + t0);
#pragma unroll
                for (int j = 0; j < CH; j++) axpy4(acc[j], v, load4(xc + 8 * j));
            }
            if (SPLIT == 4) {
#pragma unroll
                for (int o = 8; o < 32; o *= 2) {  // the warp's groups hold parts of one row
                    acc[0].x += __shfl_xor_sync(0xffffffffu, acc[0].x, o);
                    acc[0].y += __shfl_xor_sync(0xffffffffu, acc[0].y, o);
                    acc[0].z += __shfl_xor_sync(0xffffffffu, acc[0].z, o);
                    acc[0].w += __shfl_xor_sync(0xffffffffu, acc[0].w, o);
                }
                if (sub) continue;
            }
            const int64_t o = row * Rpad + t0;
            V *yr = reinterpret_cast<V *>(y + o);
            if (EP == EP_SCALE || EP == EP_FINAL) {
#pragma unroll
                for (int j = 0; j < CH; j++) acc[j] = V{ws * acc[j].x, ws * acc[j].y, ws * acc[j].z, ws * acc[j].w};
            }
            if (EP == EP_FINAL) {
                for (int32_t p = A.prp[row], p1 = A.prp[row + 1]; p < p1; p++) {
                    const T v = A.pv[p];
                    const V *ec = reinterpret_cast<const V *>(A.e + (int64_t)A.pci[p] * Rpad + t0);
#pragma unroll
                    for (int j = 0; j < CH; j++) axpy4(acc[j], v, load4(ec + 8 * j));
                }
            }
            // every operand of the row is loaded before the first store
            constexpr bool B = EP == EP_RESID || EP == EP_POST || DOT;
            V bv[B ? CH : 1], rv[EP == EP_POST || EP == EP_ACC ? CH : 1];
#pragma unroll
            for (int j = 0; j < CH; j++) {
                if (B) bv[j] = load4(reinterpret_cast<const V *>(A.b + o) + 8 * j);
                if (EP == EP_POST) rv[j] = load4(reinterpret_cast<const V *>(A.r + o) + 8 * j);
                if (EP == EP_ACC) rv[j] = yr[8 * j];
            }
            const T dwi = EP == EP_POST ? A.dw[row] : (T)0;
#pragma unroll
            for (int j = 0; j < CH; j++) {
                V v = acc[j];
                if (EP == EP_RESID) v = V{bv[j].x - v.x, bv[j].y - v.y, bv[j].z - v.z, bv[j].w - v.w};
                if (EP == EP_POST)
                    v = V{fma(dwi, bv[j].x + rv[j].x, v.x), fma(dwi, bv[j].y + rv[j].y, v.y),
                          fma(dwi, bv[j].z + rv[j].z, v.z), fma(dwi, bv[j].w + rv[j].w, v.w)};
                if (EP == EP_ACC) v = V{rv[j].x + v.x, rv[j].y + v.y, rv[j].z + v.z, rv[j].w + v.w};
                yr[8 * j] = v;
                if (DOT) {
                    dot[j].x = fma(bv[j].x, v.x, dot[j].x);
                    dot[j].y = fma(bv[j].y, v.y, dot[j].y);
                    dot[j].z = fma(bv[j].z, v.z, dot[j].z);
                    dot[j].w = fma(bv[j].w, v.w, dot[j].w);
                }
            }
        }
    if (!DOT) return;
#pragma unroll
    for (int j = 0; j < CH; j++) {
        const int c = 32 * j + l8 * 4;
        red[g][c] = dot[j].x;
        red[g][c + 1] = dot[j].y;
        red[g][c + 2] = dot[j].z;
        red[g][c + 3] = dot[j].w;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < 32 * CH; c += kT) {
        double sum = 0.0;
#pragma unroll
        for (int gg = 0; gg < kGroups; gg++) sum += (double)red[gg][c];
        A.part[(int64_t)blockIdx.x * Rpad + (int64_t)blockIdx.y * 32 * CH + c] = sum;
    }
}

// coarsest level: e = A^-1 b, one block per 8 rows and 32 columns with b's
// columns in shared memory (16 KB at most)
template <typename T>
__global__ void __launch_bounds__(256) k_ml_dense(int n, int64_t Rpad, const T *__restrict__ inv,
                                                  const T *__restrict__ b, T *__restrict__ e) {
    __shared__ T bs[kMlCoarsest * 32];
    const int64_t c0 = (int64_t)blockIdx.y * 32;
    for (int t = threadIdx.x; t < n * 32; t += 256) bs[t] = b[(int64_t)(t >> 5) * Rpad + c0 + (t & 31)];
    __syncthreads();
    const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= n) return;
    T s0 = 0, s1 = 0;
    int q = 0;
    for (; q + 1 < n; q += 2) {
        s0 = fma(inv[row * n + q], bs[q * 32 + lane], s0);
        s1 = fma(inv[row * n + q + 1], bs[(q + 1) * 32 + lane], s1);
    }
    if (q < n) s0 = fma(inv[row * n + q], bs[q * 32 + lane], s0);
    e[(int64_t)row * Rpad + c0 + lane] = s0 + s1;
}

// power iteration: 32 start columns of fixed pseudo-random values
__global__ void k_ml_start(int64_t total, float *__restrict__ x) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        uint32_t h = (uint32_t)t * 2654435761u;
        h ^= h >> 15;
        h *= 2246822519u;
        h ^= h >> 13;
        x[t] = (float)(int32_t)h * (1.f / 2147483648.f);
    }
}

// w = kOmega / (safety * max over the columns of (t . y) / (x . t)), t = A x,
// y = G^T G t: the Rayleigh quotients of G^T G A in A's inner product
__global__ void k_ml_damping(int NB, const double *__restrict__ part_xt, const double *__restrict__ part_ty,
                             float *__restrict__ w, int32_t *__restrict__ bad) {
    double a = 0.0, b = 0.0;
    for (int i = 0; i < NB; i++) {
        a += part_xt[i * 32 + threadIdx.x];
        b += part_ty[i * 32 + threadIdx.x];
    }
    float l = a > 0.0 ? (float)(b / a) : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l = fmaxf(l, __shfl_xor_sync(0xffffffffu, l, o));
    if (threadIdx.x == 0) {
        if (!(l > 0.f) || !isfinite(l)) {
            atomicAdd(bad, 1);
            l = 1.f;
        }
        *w = (float)kOmega / (kPowerSafety * l);
    }
}

// T in a parameter that the others' types decide
template <typename T> struct SameT { using type = T; };
template <typename T> using Same = typename SameT<T>::type;

// Rows per tile and columns per block: 128 rows and the widest column chunk
// while that fills the SMs twice; shorter levels 32 rows (one per group) and 32
// columns, and the shortest one row per warp.
template <int EP, bool DOT, typename T>
void spmm(cudaStream_t s, int64_t n, int64_t Rpad, const int32_t *rp, const int32_t *ci, const T *v,
          const Same<T> *x, T *y, const Args<Same<T>> &a) {
    const int64_t chunks = Rpad / 32;
    int ch = chunks % 4 == 0 ? 4 : chunks % 3 == 0 ? 3 : chunks % 2 == 0 ? 2 : 1;
    if (sizeof(T) == 8) ch = chunks % 2 == 0 ? 2 : 1;  // registers; the FP64 pipe is the bound
    int tile = 128;
    bool split = false;
    if (ceil_div(n, tile) * (chunks / ch) < kFill) {
        tile = 32;
        if (!DOT && ceil_div(n, tile) * (chunks / ch) < kFill) {
            ch = 1;
            if (ceil_div(n, tile) * chunks < kFill) {
                tile = 8;
                split = true;
            }
        }
    }
    const int64_t gx = DOT ? a.NB : std::min<int64_t>(ceil_div(n, tile), 4096);
    const dim3 g((unsigned)gx, (unsigned)(chunks / ch));
    if (split) {
        if constexpr (!DOT) k_ml_spmm<T, 1, 4, EP, false><<<g, kT, 0, s>>>(n, Rpad, tile, rp, ci, v, x, y, a);
        return;
    }
    if constexpr (sizeof(T) == 4) {
        if (ch == 4) {
            k_ml_spmm<T, 4, 1, EP, DOT><<<g, kT, 0, s>>>(n, Rpad, tile, rp, ci, v, x, y, a);
            return;
        }
        if (ch == 3) {
            k_ml_spmm<T, 3, 1, EP, DOT><<<g, kT, 0, s>>>(n, Rpad, tile, rp, ci, v, x, y, a);
            return;
        }
    }
    switch (ch) {
        case 2: k_ml_spmm<T, 2, 1, EP, DOT><<<g, kT, 0, s>>>(n, Rpad, tile, rp, ci, v, x, y, a); break;
        default: k_ml_spmm<T, 1, 1, EP, DOT><<<g, kT, 0, s>>>(n, Rpad, tile, rp, ci, v, x, y, a); break;
    }
}

// Host hierarchy of the context's mesh onto the device (once per mesh and set
// of fixed rows)
void build(Context &c, cudaStream_t s) {
    MeshData &m = c.mesh;
    Multilevel &M = m.ml;
    std::vector<uint8_t> fixed;
    if (c.have_fixed) {
        fixed.assign((size_t)m.n, 0);
        for (int32_t v : m.dir_nodes) fixed[v] = 1;
        for (int32_t v : c.calib) fixed[v] = 1;
    }
    if (M.tried && M.fixed == fixed) return;
    M.tried = false;  // a failed allocation leaves it so: the next solve builds again
    M.ok = false;
    M.levels.clear();
    // the unit-resistivity matrix
    std::vector<double> unit((size_t)m.nnz);
    DBuf<double> tmp;
    const double *src = c.d_S1.p;
    if (c.d_S1.n != (size_t)m.nnz) {  // total potential: not kept
        tmp.alloc((size_t)m.nnz);
        assemble_all(c, nullptr, tmp.p, s);
        src = tmp.p;
    }
    ERTGB_CUDA(cudaMemcpyAsync(unit.data(), src, sizeof(double) * unit.size(), cudaMemcpyDeviceToHost, s));
    ERTGB_CUDA(cudaStreamSynchronize(s));
    std::vector<HostLevel> H;
    if (!build_levels(m.rowptr, m.colidx, unit, kMlCoarsest, kMlMaxLevels, H)) {
        M.tried = true;
        M.fixed = fixed;
        return;
    }
    for (size_t k = 0; k < H.size(); k++) {
        auto l = std::make_unique<MlLevel>();
        const HostLevel &h = H[k];
        l->n = h.n;
        l->nc = h.nc;
        l->nnz = (int64_t)h.ci.size();
        l->nnzP = (int64_t)h.P_ci.size();
        l->nnzAP = (int64_t)h.AP_ci.size();
        if (k) {
            l->rp.upload(h.rp, s);
            l->ci.upload(h.ci, s);
            l->val.alloc((size_t)l->nnz);
        }
        if (k + 1 < H.size()) {
            l->P_rp.upload(h.P_rp, s);
            l->P_ci.upload(h.P_ci, s);
            l->P_v.upload(h.P_v, s);
            l->PT_rp.upload(h.PT_rp, s);
            l->PT_ci.upload(h.PT_ci, s);
            l->PT_v.upload(h.PT_v, s);
            l->PT64.upload(std::vector<double>(h.PT_v.begin(), h.PT_v.end()), s);
            ERTGB_CUDA(cudaStreamSynchronize(s));  // the copy's source ends here
            l->AP_rp.upload(h.AP_rp, s);
            l->AP_ci.upload(h.AP_ci, s);
            l->AP.alloc((size_t)l->nnzAP);
        }
        M.levels.push_back(std::move(l));
    }
    const int64_t last = M.levels.back()->n;
    M.inv64.alloc((size_t)(last * last));
    M.bad.alloc(1);
    M.w.alloc(1);
    ERTGB_CUDA(cudaStreamSynchronize(s));  // host lists are freed on return
    M.ok = M.tried = true;
    M.fixed = fixed;
}

inline unsigned grid_rows(int64_t n, int per = kT) { return (unsigned)std::min<int64_t>(ceil_div(n, per), 1 << 16); }

}  // namespace

// largest eigenvalue of G^T G A from kPower power iterations on 32 columns
static int factor_damping(Context &c, cudaStream_t s) {
    MeshData &m = c.mesh;
    Multilevel &M = m.ml;
    const int NB = 152;
    M.px.alloc((size_t)m.n * 32);
    M.pt.alloc((size_t)m.n * 32);
    M.pg.alloc((size_t)m.n * 32);
    M.ppart.alloc((size_t)2 * NB * 32);
    k_ml_start<<<grid_rows(m.n * 32), kT, 0, s>>>(m.n * 32, M.px.p);
    for (int i = 0; i < kPower; i++) {
        const bool end = i + 1 == kPower;
        Args<float> a;
        a.NB = NB;
        a.b = M.px.p;
        a.part = M.ppart.p;
        if (end) spmm<EP_PLAIN, true>(s, m.n, 32, m.d_rowptr.p, m.d_colidx.p, c.d_S32.p, M.px.p, M.pt.p, a);
        else spmm<EP_PLAIN, false>(s, m.n, 32, m.d_rowptr.p, m.d_colidx.p, c.d_S32.p, M.px.p, M.pt.p, a);
        spmm<EP_PLAIN, false>(s, m.n, 32, m.d_Lrowptr.p, m.d_Lcolidx.p, c.d_G32.p, M.pt.p, M.pg.p, a);
        a.b = M.pt.p;
        a.part = M.ppart.p + NB * 32;
        if (end) spmm<EP_PLAIN, true>(s, m.n, 32, m.d_Urowptr.p, m.d_Ucolidx.p, c.d_GT32.p, M.pg.p, M.px.p, a);
        else spmm<EP_PLAIN, false>(s, m.n, 32, m.d_Urowptr.p, m.d_Ucolidx.p, c.d_GT32.p, M.pg.p, M.px.p, a);
    }
    k_ml_damping<<<1, 32, 0, s>>>(NB, M.ppart.p, M.ppart.p + NB * 32, M.w.p, M.bad.p);
    return 3 * kPower + 2;
}

template <typename T> static bool setup(Context &c, const double *fine, bool factor, int64_t Rpad, cudaStream_t s) {
    MeshData &m = c.mesh;
    build(c, s);
    Multilevel &M = m.ml;
    if (!M.ok) return false;
    const size_t L = M.levels.size();
    M.factor = factor;
    M.bad.zero(s);
    int launches = 0;
    for (size_t k = 0; k + 1 < L; k++) {
        MlLevel &l = *M.levels[k];
        MlLevel &d = *M.levels[k + 1];
        MlValues<T> &v = l.values<T>();
        const int32_t *rp = k ? l.rp.p : m.d_rowptr.p, *ci = k ? l.ci.p : m.d_colidx.p;
        const double *val = k ? l.val.p : fine;
        const bool jac = k || !factor;
        if (jac) v.AS.alloc((size_t)l.nnz);
        v.Q.alloc((size_t)l.nnzAP);
        v.dw.alloc((size_t)l.n);
        k_ml_rows<T><<<grid_rows(32 * l.n), kT, 0, s>>>(l.n, rp, ci, val, l.P_rp.p, l.P_ci.p, l.P_v.p, l.AP_rp.p, l.AP_ci.p,
                                                     jac ? 1 : 0, l.AP.p, v.dw.p, v.Q.p, M.bad.p);
        if (jac) k_ml_scale<T><<<grid_rows(l.nnz), kT, 0, s>>>(l.nnz, ci, val, v.dw.p, v.AS.p);
        k_ml_galerkin<<<grid_rows(32 * l.nc), kT, 0, s>>>(l.nc, l.PT_rp.p, l.PT_ci.p, l.PT_v.p, l.AP_rp.p, l.AP_ci.p,
                                                          l.AP.p, d.rp.p, d.ci.p, d.val.p);
        launches += 3;
        if (k) {
            v.b.alloc((size_t)l.n * Rpad);
            v.r.alloc((size_t)l.n * Rpad);
            v.e.alloc((size_t)l.n * Rpad);
        }
    }
    MlLevel &z = *M.levels.back();
    MlValues<T> &zv = z.values<T>();
    zv.b.alloc((size_t)z.n * Rpad);
    zv.e.alloc((size_t)z.n * Rpad);
    zv.AS.alloc((size_t)(z.n * z.n));  // the inverse
    k_ml_densify<<<(unsigned)z.n, 128, 0, s>>>((int)z.n, z.rp.p, z.ci.p, z.val.p, M.inv64.p);
    dense_inverse(M.inv64.p, (int)z.n, M.bad.p, s);
    k_ml_symmetric<T><<<grid_rows(z.n * z.n), kT, 0, s>>>((int)z.n, M.inv64.p, zv.AS.p);
    launches += 3;
    if constexpr (sizeof(T) == 4) {
        if (factor) launches += factor_damping(c, s);
    }
    ERTGB_CUDA(cudaGetLastError());
    int32_t bad = 0;
    ERTGB_CUDA(cudaMemcpyAsync(&bad, M.bad.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    ERTGB_CUDA(cudaStreamSynchronize(s));
    c.stats.launches_response += launches;
    return bad == 0;
}

// 3-D (one wavenumber k = 0): the 2.5-D path has its direct solve.  One response
// without -> with coarse levels: 1350 nodes, 12 electrodes 5.2 -> 2.3 ms
// (Jacobi), 4.0 -> 2.2 (FSAI); 4224 nodes, 48 electrodes 11.9 -> 3.2, 11.6 ->
// 3.5; nothing smaller than kMlMinRows was measured.  CEM and bypass matrices
// keep the single level.
template <typename T>
static bool guarded_setup(Context &c, const double *val, bool factor, int64_t cols, cudaStream_t s) {
    const MeshData &m = c.mesh;
    if (c.lean || !c.coarse_levels || m.dim != 3 || c.nK != 1 || c.k[0] != 0.0 || m.n < kMlMinRows) return false;
    if (!m.ext_rows.empty() || m.n_ext > 0) return false;
    return setup<T>(c, val, factor, cols, s);
}

bool ml_setup(Context &c, const double *val, bool factor, int64_t cols, cudaStream_t s) {
    return guarded_setup<float>(c, val, factor, cols, s);
}

bool ml_setup64(Context &c, const double *val, int64_t cols, cudaStream_t s) {
    return guarded_setup<double>(c, val, false, cols, s);
}

template <typename T>
static void cycle(Context &c, const MlBlock<T> &v, int NB, double *pz, cudaStream_t s) {
    MeshData &m = c.mesh;
    Multilevel &M = m.ml;
    const int64_t n = m.n, R = v.cols;
    const size_t L = M.levels.size();
    MlLevel &f = *M.levels[0];
    MlValues<T> &fv = f.values<T>();
    const T *b = v.b;
    T *z = v.z, *r = v.r;
    Args<T> a;
    a.b = b;
    bool factor = false;
    if constexpr (sizeof(T) == 4) {
        factor = M.factor;
        if (factor) {
            a.w = M.w.p;
            spmm<EP_PLAIN, false>(s, n, R, m.d_Lrowptr.p, m.d_Lcolidx.p, c.d_G32.p, b, v.t, a);
            spmm<EP_SCALE, false>(s, n, R, m.d_Urowptr.p, m.d_Ucolidx.p, c.d_GT32.p, v.t, z, a);
            spmm<EP_RESID, false>(s, n, R, m.d_rowptr.p, m.d_colidx.p, c.d_S32.p, z, r, a);
        }
    }
    if (!factor) spmm<EP_RESID, false>(s, n, R, m.d_rowptr.p, m.d_colidx.p, fv.AS.p, b, r, a);
    auto restrict_to = [&](MlLevel &l, const T *from, T *to) {
        if constexpr (sizeof(T) == 4) spmm<EP_PLAIN, false>(s, l.nc, R, l.PT_rp.p, l.PT_ci.p, l.PT_v.p, from, to, Args<T>{});
        else spmm<EP_PLAIN, false>(s, l.nc, R, l.PT_rp.p, l.PT_ci.p, l.PT64.p, from, to, Args<T>{});
    };
    restrict_to(f, r, M.levels[1]->values<T>().b.p);
    for (size_t k = 1; k + 1 < L; k++) {
        MlLevel &l = *M.levels[k];
        MlValues<T> &lv = l.values<T>();
        Args<T> q;
        q.b = lv.b.p;
        spmm<EP_RESID, false>(s, l.n, R, l.rp.p, l.ci.p, lv.AS.p, lv.b.p, lv.r.p, q);
        restrict_to(l, lv.r.p, M.levels[k + 1]->values<T>().b.p);
    }
    MlLevel &d = *M.levels[L - 1];
    MlValues<T> &dv = d.values<T>();
    k_ml_dense<T><<<dim3((unsigned)ceil_div(d.n, 8), (unsigned)(R / 32)), 256, 0, s>>>((int)d.n, R, dv.AS.p, dv.b.p,
                                                                                       dv.e.p);
    for (size_t k = L - 2; k >= 1; k--) {
        MlLevel &l = *M.levels[k];
        MlValues<T> &lv = l.values<T>();
        Args<T> q;
        q.b = lv.b.p;
        q.r = lv.r.p;
        q.dw = lv.dw.p;
        spmm<EP_POST, false>(s, l.n, R, l.AP_rp.p, l.AP_ci.p, lv.Q.p, M.levels[k + 1]->values<T>().e.p,
                             lv.e.p, q);
    }
    const T *e = M.levels[1]->values<T>().e.p;
    a.part = pz;
    a.NB = NB;
    if constexpr (sizeof(T) == 4) {
        if (factor) {
            spmm<EP_ACC, false>(s, n, R, f.AP_rp.p, f.AP_ci.p, fv.Q.p, e, r, Args<T>{});
            spmm<EP_ACC, false>(s, n, R, m.d_Lrowptr.p, m.d_Lcolidx.p, c.d_G32.p, r, v.t, Args<T>{});
            a.prp = f.P_rp.p;
            a.pci = f.P_ci.p;
            a.pv = f.P_v.p;
            a.e = e;
            spmm<EP_FINAL, true>(s, n, R, m.d_Urowptr.p, m.d_Ucolidx.p, c.d_GT32.p, v.t, z, a);
        }
    }
    if (!factor) {
        a.r = r;
        a.dw = fv.dw.p;
        if (pz) spmm<EP_POST, true>(s, n, R, f.AP_rp.p, f.AP_ci.p, fv.Q.p, e, z, a);
        else spmm<EP_POST, false>(s, n, R, f.AP_rp.p, f.AP_ci.p, fv.Q.p, e, z, a);
    }
    ERTGB_CUDA(cudaGetLastError());
}

void ml_cycle(Context &c, const MlBlock<float> &v, int NB, double *pz, cudaStream_t s) { cycle(c, v, NB, pz, s); }

void ml_cycle64(Context &c, const MlBlock<double> &v, int NB, double *pz, cudaStream_t s) { cycle(c, v, NB, pz, s); }

int ml_launches(const Context &c) {
    const Multilevel &M = c.mesh.ml;
    return (M.factor ? 7 : 3) + 3 * ((int)M.levels.size() - 2) + 1;
}

}  // namespace ertgb
