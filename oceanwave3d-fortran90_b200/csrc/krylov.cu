// GMRES building blocks on the device (FP64 in both precision forms).
//
// The reference drives SPARSKIT2's gmres through reverse communication
// (src/wrappers/iterative_solution.f90:50-134); here the Arnoldi process,
// the Givens rotations and the least-squares update stay on the device, for
// right (flexible) and left preconditioning alike: each Arnoldi step is one
// reduction pass and one update pass of delayed classical Gram-Schmidt
// (DCGS2, below), whose last block forms the Hessenberg column, the Givens
// rotation, the residual estimate and the stopping test.
// Reductions are deterministic: every block writes a partial sum, the last
// block to finish (atomic ticket) adds the partials in block order.
// Basis vectors are stored unnormalised with a scale factor s_i = 1/|V_i|,
// which saves the normalisation pass.
#include "ow3d_internal.h"
#include <algorithm>
#include <cmath>

namespace ow3d {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxDots = kMaxKrylov + 1;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums over the warp of M values per lane (M a power of two <= 32): lane l gets
// the sum of value l / (32 / M), in each of the 32 / M lanes that share it. A
// step folds the lanes' values in half, so M values cost M - 1 + log2(32 / M)
// shuffles instead of 5 M.
template <int M>
__device__ __forceinline__ double warp_sums(double* v) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int n = M; n > 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const double send = up ? v[i] : v[i + n / 2], keep = up ? v[i + n / 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    double s = v[0];
#pragma unroll
    for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Block-reduce `nv` values per thread into partial[v*nblocks + blockIdx.x].
__device__ void block_store_partials(const double* acc, int nv, double* partial, int nblocks) {
    __shared__ double red[kThreads / 32][kMaxDots + 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int v = 0; v < nv; ++v) {
        double s = warp_sum(acc[v]);
        if (lane == 0) red[wid][v] = s;
    }
    __syncthreads();
    for (int v = threadIdx.x; v < nv; v += blockDim.x) {
        double s = 0;
        for (int w = 0; w < (int)(blockDim.x / 32); ++w) s += red[w][v];
        partial[(int64_t)v * nblocks + blockIdx.x] = s;
    }
}

// The last block to finish sums the partials: warp w reduces vectors
// v = w, w + nwarps, ...; lane l adds blocks l, l+32, ... in order and the
// warp tree combines the lanes (a fixed order: deterministic results).
// Returns true in that block. G vectors a warp at a time, U L2 loads of each in
// flight per lane: <1, 20> takes the one sum of a pass over the grid's at most
// 592 blocks in one round.
template <int G, int U>
__device__ bool last_block_reduce(double* partial, int nv, int nblocks, unsigned int* counter, double* out) {
    __shared__ bool amlast;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int t = atomicAdd(counter, 1u);
        amlast = (t == gridDim.x * gridDim.y - 1);
    }
    __syncthreads();
    if (!amlast) return false;
    __threadfence();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int v0 = wid; v0 < nv; v0 += G * nw) {
        double s[G];
#pragma unroll
        for (int g = 0; g < G; ++g) s[g] = 0.0;
        for (int b = lane; b < nblocks; b += U * 32) {
            double q[G][U];
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int v = v0 + g * nw, bb = b + 32 * u;
                    q[g][u] = v < nv && bb < nblocks ? __ldcg(partial + (int64_t)v * nblocks + bb) : 0.0;
                }
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int u = 0; u < U; ++u) s[g] += q[g][u];
        }
#pragma unroll
        for (int g = 0; g < G; ++g) s[g] = warp_sum(s[g]);
        if (lane == 0)
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (v0 + g * nw < nv) out[v0 + g * nw] = s[g];
    }
    __syncthreads();
    if (threadIdx.x == 0) *counter = 0u;
    return true;
}

// Initial residual norm: beta = |v|, tolerance rtol*beta + atol.
// hnext (nonzero only inside a captured step graph): the condition of the
// graph node that runs the next Arnoldi step, set to "not done".
__global__ void __launch_bounds__(kThreads) k_norm_init(const double* __restrict__ v, int64_t n, double* partial,
                                                        unsigned int* counter, int nblocks, KrylovState* ks,
                                                        double rtol, double atol, cudaGraphConditionalHandle hnext) {
    pdl_entry();
    double acc[1] = {0.0};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += stride) acc[0] += v[t] * v[t];
    block_store_partials(acc, 1, partial, nblocks);
    __shared__ double res[1];
    if (last_block_reduce<1, 20>(partial, 1, nblocks, counter, res)) {
        if (threadIdx.x == 0) {
            const double beta = sqrt(res[0]);
            ks->beta = beta;
            ks->iters += 1;   // the residual's matvec (iterative_solution.f90:58-60 counts it)
            if (ks->iters == 1) ks->tol = rtol * beta + atol;   // fixed at the first residual
            ks->resid = beta;
            for (int i = 0; i < kMaxKrylov + 2; ++i) ks->g[i] = 0.0;
            ks->g[0] = beta;
            ks->scale[0] = beta > 0 ? 1.0 / beta : 0.0;
            ks->k = 0;
            ks->reorth = 0;
            if (beta <= ks->tol) { ks->done = 1; ks->converged = 1; }
            if (hnext) cudaGraphSetConditional(hnext, ks->done ? 0u : 1u);
        }
    }
}

// Upper-triangular solve R y = g for the current k: the block brings R and g to
// shared memory, one thread runs the rows' chain of multiply-adds there. (The
// same chain on R in memory, load after load: 18-32 us at 16-22 columns; the
// columns subtracted by a warp's lanes would be shorter still, but in another
// order of sums, which a preconditioner in FP32 magnifies.)
// With in_basis set (left preconditioning), the coefficients of the vectors
// the Arnoldi steps multiplied are taken to the final basis, y <- T y, so
// that the update is x += sum_i y_i v_i.
__global__ void __launch_bounds__(kThreads) k_backsolve(KrylovState* ks, int in_basis) {
    pdl_entry();
    __shared__ double R[kMaxKrylov + 1][kMaxKrylov + 1], y[kMaxKrylov + 1];   // R[row][column]
    __shared__ int kk;
    const int k0 = ks->k, tid = threadIdx.x;
    for (int t = tid; t < k0 * k0; t += blockDim.x) {
        const int c = t / k0, r = t - c * k0;
        if (r <= c) R[r][c] = ks->R[c][r];
        if (c == 0) y[r] = ks->g[r];
    }
    __syncthreads();
    if (tid == 0) {
        int k = k0;
        while (k > 0 && R[k - 1][k - 1] == 0.0) --k;
        for (int i = k - 1; i >= 0; --i) {
            double t = y[i];
#pragma unroll 4
            for (int j = i + 1; j < k; ++j) t -= R[i][j] * y[j];
            y[i] = t / R[i][i];
        }
        kk = k;
    }
    __syncthreads();
    const int k = kk;
    for (int i = tid; i <= kMaxKrylov; i += blockDim.x) {
        double c = i < k ? y[i] : 0.0;
        if (in_basis && i < k) {
            c = 0.0;
            for (int j = i; j < k; ++j) c += ks->T[j][i] * y[j];
        }
        ks->y[i] = c;
    }
    __syncthreads();
    if (tid == 0) ks->k = k;
}

// x += sum_i y_i * (use_scale ? scale_i : 1) * Z_i
template <typename TZ>
__global__ void __launch_bounds__(kThreads) k_solution_update(double* __restrict__ x, const TZ* __restrict__ Z,
                                                              int64_t ldz, int64_t n,
                                                              const KrylovState* ks, int use_scale) {
    pdl_entry();
    __shared__ double coef[kMaxDots];
    const int k = ks->k;
    for (int v = threadIdx.x; v < k; v += blockDim.x) coef[v] = ks->y[v] * (use_scale ? ks->scale[v] : 1.0);
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += stride) {
        double a = x[t];
        int v = 0;
        for (; v + 8 <= k; v += 8) {   // eight vectors' loads in flight
            TZ z[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) z[u] = __ldcs(Z + (int64_t)(v + u) * ldz + t);
#pragma unroll
            for (int u = 0; u < 8; ++u) a += coef[v + u] * (double)z[u];
        }
        for (; v < k; ++v) a += coef[v] * (double)__ldcs(Z + (int64_t)v * ldz + t);
        x[t] = a;
    }
}

__global__ void k_krylov_reset(KrylovState* ks) {
    pdl_entry();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    ks->k = 0; ks->done = 0; ks->converged = 0; ks->iters = 0; ks->reorth = 0; ks->status = 0;
    ks->tol = 0; ks->resid = 0; ks->beta = 0;
}

// ---------------------------------------------------------------- DCGS2
// Arnoldi orthogonalisation by delayed classical Gram-Schmidt with
// reorthogonalisation (Swirydowicz, Langou, Ananthan, Yang, Thomas, "Low
// synchronization Gram-Schmidt and generalized minimal residual algorithms",
// NLAA 2021): the second Gram-Schmidt pass of V_j rides on step j's single
// reduction, so each Arnoldi step reads the basis twice (reduce, update)
// instead of four times. V_0..V_{j-1} are final, V_j has had one pass.

// The scalar work of a step runs in the warp that ends a kernel's last block,
// with its columns in shared memory: lane l takes entries l and l + 32, and
// only the sums and the chain of rotations are serial, on shared memory
// instead of a chain of loads from the state in memory.
// The order of every FP64 sum here and in the reductions below is part of the
// method's results in the mixed precision form: a change of rounding in the
// last place of a coefficient reaches the FP32 preconditioner's input and
// comes out at 1e-9 to 5e-9 of a small sloping flume's surface.
struct ColScratch {
    double h[kMaxKrylov + 2], cs[kMaxKrylov + 1], sn[kMaxKrylov + 1], sig[kMaxKrylov + 1], hq[kMaxKrylov + 1];
};

// One warp: rotate the unrotated column col of H (w.h[0..col+1]) with
// rotations 0..col-1 into R, form rotation col, rotate g from its value
// before rotation col (g0); w.cs, w.sn hold rotations 0..col-1 and get
// rotation col. Returns |g[col+1]|.
__device__ double dcgs_rotate(KrylovState* ks, ColScratch& w, int col, double g0) {
    const int lane = threadIdx.x & 31;
    double a = w.h[0];
    double al = 0.0, gc = 0.0;
    if (lane == 0) {
        for (int i = 0; i < col; ++i) {
            const double n = w.h[i + 1];
            w.h[i] = w.cs[i] * a + w.sn[i] * n;
            a = w.cs[i] * n - w.sn[i] * a;
        }
        const double yv = w.h[col + 1];
        const double r = sqrt(a * a + yv * yv);
        double c = 1.0, sg = 0.0, d = a;
        if (r != 0.0) { c = a / r; sg = yv / r; d = r; }
        w.h[col] = d;
        w.h[col + 1] = r != 0.0 ? 0.0 : yv;
        w.cs[col] = c; w.sn[col] = sg;
        ks->cs[col] = c; ks->sn[col] = sg;
        al = -sg * g0;
        gc = c * g0;
        ks->g[col] = gc;
        ks->g[col + 1] = al;
    }
    __syncwarp();
    for (int r = lane; r <= col + 1; r += 32) ks->R[col][r] = w.h[r];
    __syncwarp();
    return fabs(__shfl_sync(0xffffffffu, al, 0));
}

// One warp, after step j's reduction: res[2i] = <V_i, V_j>, res[2i+1] = <V_i, W>, i <= j.
// The vector step j multiplied, scale_j V_j with V_j after one pass and
// scale_j its provisional scale, is scale_j (nu q_j + sum sigma_i q_i) in
// the final basis: column j of T (used by left preconditioning, whose
// solution is a combination of those vectors).
__device__ void dcgs_column(KrylovState* ks, ColScratch& w, int j, const double* res) {
    const int lane = threadIdx.x & 31;
    double sig[2] = {0.0, 0.0}, sc[2] = {0.0, 0.0}, hq[2] = {0.0, 0.0};
    double g0 = 0.0, scj = ks->scale[j], ss = 0.0, corr = 0.0;
    if (j >= 1) g0 = ks->gsave[j - 1];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int i = lane + 32 * q;
        if (i < j) {
            sc[q] = ks->scale[i];
            const double h = ks->H[j - 1][i];
            if (i < j - 1) { w.cs[i] = ks->cs[i]; w.sn[i] = ks->sn[i]; }
            sig[q] = __dmul_rn(sc[q], res[2 * i]);
            hq[q] = __dmul_rn(sc[q], res[2 * i + 1]);
            w.sig[i] = sig[q];
            w.hq[i] = hq[q];
            ks->T[j][i] = scj * sig[q];
            // complete column j-1: W_{j-1} = sum (h + sigma) q_i + nu q_j
            ks->H[j - 1][i] = w.h[i] = __dadd_rn(h, sig[q]);
        }
    }
    __syncwarp();
#pragma unroll 4
    for (int i = 0; i < j; ++i) {
        const double si = w.sig[i];
        ss = __fma_rn(si, si, ss);
        corr = __fma_rn(si, w.hq[i], corr);
    }
    if (j >= 1) {
        const double nu = sqrt(fmax(res[2 * j] - ss, 0.0));
        if (lane == 0) {
            ks->T[j][j] = scj * nu;
            ks->H[j - 1][j] = nu;
            w.h[j] = nu;
        }
        scj = nu > 0 ? 1.0 / nu : 0.0;
        __syncwarp();
        const double resid = dcgs_rotate(ks, w, j - 1, g0);
        if (lane == 0) { ks->scale[j] = scj; ks->resid = resid; }
    } else if (lane == 0) {
        ks->T[0][0] = 1.0;   // scale_0 V_0 is final: v_0
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int i = lane + 32 * q;
        if (i < j) {
            ks->H[j][i] = hq[q];
            ks->coefB[i] = hq[q] * sc[q];
            ks->coefA[i] = sig[q] * sc[q];
        }
    }
    if (lane == 0) {
        const double hj = (j >= 1 ? res[2 * j + 1] - corr : res[2 * j + 1]) * scj;
        ks->H[j][j] = hj;
        ks->coefB[j] = hj * scj;
    }
}

// Reduction: res[2v] = <V_v, V_j>, res[2v+1] = <V_v, W> for v <= j. The
// vectors are cut into chunks of kDotE * blockDim.x element pairs; a block takes
// chunks in turn, keeps its thread's kDotE pairs of V_j and W in registers, and
// streams the V_v of the chunk, kDotG vectors' loads in flight together. The
// warp sums of kDotG vectors' 2 kDotG values fold into each other (warp_sums:
// 9 shuffles for four vectors instead of 40), and a warp adds them to its own
// shared-memory slots; the block's slots become partial[u * gridDim.x + b];
// the last block reduces the partials in a fixed order and runs dcgs_column.
// Long vectors take one block per chunk, which reads every vector from memory
// once per step. Short ones, whose few chunks leave most SMs idle and whose
// time is the latency of the groups one after another, split the groups over
// gridDim.y blocks, which read V_j and W again (from L2); the sums are the same.
constexpr int kDotE = 4;
constexpr int kDotG = 4;

__global__ void __launch_bounds__(kThreads, 2) k_dcgs_reduce(const double* __restrict__ V, int64_t ldv, int j,
                                                          const double* __restrict__ W, int64_t n, double* partial,
                                                          unsigned int* counter, KrylovState* ks) {
    constexpr int E = kDotE, G = kDotG;
    pdl_entry();
    if (ks->done) return;
    __shared__ double acc[2 * kMaxDots + 2 * G][kThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nv = 2 * (j + 1);
    for (int u = threadIdx.x; u < (nv + 2 * G) * nw; u += blockDim.x) acc[u / nw][u % nw] = 0.0;
    __syncthreads();
    const int64_t n2 = (n + 1) / 2;
    const int64_t chunk = (int64_t)E * blockDim.x;
    const int64_t nchunks = (n2 + chunk - 1) / chunk;
    const double2* q2 = reinterpret_cast<const double2*>(V + (int64_t)j * ldv);
    const double2* w2 = reinterpret_cast<const double2*>(W);
    constexpr int L = 32 / (2 * G);   // lanes that share a sum
    for (int64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        const int64_t t0 = ch * chunk + threadIdx.x;
        double2 q[E], w[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int64_t t = t0 + (int64_t)e * blockDim.x;
            if (t < n2) { q[e] = q2[t]; w[e] = w2[t]; }
            else { q[e] = make_double2(0.0, 0.0); w[e] = make_double2(0.0, 0.0); }
        }
        // the older basis vectors are read once per pass, so they are streamed
        // (evict-first) rather than let them push the multigrid levels and
        // their coefficient tables out of L2 before the next V-cycle
        for (int v0 = blockIdx.y * G; v0 <= j; v0 += gridDim.y * G) {
            double2 x[G][E];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int v = v0 + g;
                const double2* a2 = reinterpret_cast<const double2*>(V + (int64_t)min(v, j) * ldv);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int64_t t = t0 + (int64_t)e * blockDim.x;
                    x[g][e] = (v < j && t < n2) ? __ldcs(a2 + t) : make_double2(0.0, 0.0);
                }
            }
            double s[2 * G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                double sa = 0, sb = 0;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const double2 xe = (v0 + g == j) ? q[e] : x[g][e];
                    sa += xe.x * q[e].x + xe.y * q[e].y;
                    sb += xe.x * w[e].x + xe.y * w[e].y;
                }
                s[2 * g] = sa;
                s[2 * g + 1] = sb;
            }
            const double r = warp_sums<2 * G>(s);
            // the lanes' sums of vectors past j are zero and land past nv
            if (lane % L == 0) acc[2 * v0 + lane / L][wid] += r;
        }
    }
    __syncthreads();
    for (int u = threadIdx.x; u < nv; u += blockDim.x) {
        if ((u / (2 * G)) % gridDim.y != blockIdx.y) continue;
        double t = 0;
        for (int w = 0; w < nw; ++w) t += acc[u][w];
        partial[(int64_t)u * gridDim.x + blockIdx.x] = t;
    }
    __shared__ double res[2 * kMaxDots];
    if (!last_block_reduce<3, 4>(partial, nv, gridDim.x, counter, res)) return;
    __shared__ ColScratch scratch;
    if (wid == 0) dcgs_column(ks, scratch, j, res);
}

// Update: V_j <- V_j - sum_{i<j} coefA_i V_i,  W <- W - sum_{i<j} coefB_i V_i - coefB_j V_j(new),
// |W|^2; the last block completes column j's provisional norm, its rotation,
// the residual estimate and the stopping test.
__global__ void __launch_bounds__(kThreads) k_dcgs_update(double* __restrict__ V, int64_t ldv, int j,
                                                          double* __restrict__ W, int64_t n, double* partial,
                                                          unsigned int* counter, int nblocks, KrylovState* ks,
                                                          int maxmv, int m, cudaGraphConditionalHandle hnext) {
    pdl_entry();
    if (ks->done) return;
    __shared__ double cA[kMaxDots], cB[kMaxDots + 1];
    for (int v = threadIdx.x; v <= j; v += blockDim.x) { cB[v] = ks->coefB[v]; if (v < j) cA[v] = ks->coefA[v]; }
    __syncthreads();
    const double cBj = cB[j];
    double acc[1] = {0.0};
    const int64_t n2 = (n + 1) / 2;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    double2* vj2 = reinterpret_cast<double2*>(V + (int64_t)j * ldv);
    double2* w2 = reinterpret_cast<double2*>(W);
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n2; t += stride) {
        // v_j is next read as an older vector of the following reduction
        // (streamed), so it is written back evict-first too
        double2 q = __ldcs(vj2 + t), a = w2[t];
        for (int v0 = 0; v0 < j; v0 += 8) {
            double2 vv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (v0 + u < j) vv[u] = __ldcs(reinterpret_cast<const double2*>(V + (int64_t)(v0 + u) * ldv) + t);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (v0 + u < j) {
                    q.x -= cA[v0 + u] * vv[u].x; q.y -= cA[v0 + u] * vv[u].y;
                    a.x -= cB[v0 + u] * vv[u].x; a.y -= cB[v0 + u] * vv[u].y;
                }
        }
        a.x -= cBj * q.x; a.y -= cBj * q.y;
        if (j > 0) __stcs(vj2 + t, q);
        w2[t] = a;
        acc[0] += a.x * a.x + a.y * a.y;
    }
    block_store_partials(acc, 1, partial, nblocks);
    __shared__ double res[1];
    if (!last_block_reduce<1, 20>(partial, 1, nblocks, counter, res)) return;
    __shared__ ColScratch w;
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    for (int i = lane; i <= j; i += 32) {
        w.h[i] = ks->H[j][i];
        if (i < j) { w.cs[i] = ks->cs[i]; w.sn[i] = ks->sn[i]; }
    }
    const double g0 = ks->g[j], tol = ks->tol, nrm = sqrt(res[0]);
    const int iters = ks->iters + 1;
    if (lane == 0) {
        w.h[j + 1] = nrm;
        ks->H[j][j + 1] = nrm;
        ks->scale[j + 1] = nrm > 0 ? 1.0 / nrm : 0.0;
        ks->gsave[j] = g0;
    }
    __syncwarp();
    const double resid = dcgs_rotate(ks, w, j, g0);
    if (lane == 0) {
        const bool conv = resid <= tol;
        const int done = conv || j + 1 >= m || iters >= maxmv || nrm == 0.0;
        ks->resid = resid;
        ks->k = j + 1;
        ks->iters = iters;
        if (conv) ks->converged = 1;
        if (done) ks->done = 1;
        if (hnext) cudaGraphSetConditional(hnext, done ? 0u : 1u);
    }
}

__global__ void k_solve_log(const KrylovState* ks, SolveLog* out) {
    pdl_entry();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    out->iters = ks->iters;
    out->converged = ks->converged;
    out->resid = ks->resid;
    out->beta = ks->beta;
    out->tol = ks->tol;
}

}  // namespace

void launch_dcgs_reduce(const double* V, int64_t ldv, int j, const double* W, int64_t n, const DotScratch& sc,
                        KrylovState* ks, cudaStream_t st) {
    // one block per chunk up to the scratch's blocks; 2(j+1) partial rows
    const int64_t chunk = (int64_t)kDotE * kThreads, chunks = ((n + 1) / 2 + chunk - 1) / chunk;
    int64_t nb = std::min<int64_t>(chunks, sc.nblocks);
    nb = std::min<int64_t>(nb, ((int64_t)(kMaxKrylov + 2) * sc.nblocks) / (2 * (j + 1)));   // scratch rows
    if (nb < 1) nb = 1;
    // groups side by side while all blocks fit on the chip at once, two per SM
    const int64_t ny = std::max<int64_t>(1, std::min<int64_t>((j + kDotG) / kDotG, 2 * 148 / nb));
    launch_k(k_dcgs_reduce, dim3((unsigned)nb, (unsigned)ny), dim3(kThreads), 0, st, V, ldv, j, W, n, sc.partial,
             sc.counter, ks);
}

// Blocks of a pass over n2 items with one partial sum per block.
static int pass_blocks(int64_t n2, const DotScratch& sc) {
    return (int)std::max<int64_t>(1, std::min<int64_t>(sc.nblocks, (n2 + kThreads - 1) / kThreads));
}

void launch_dcgs_update(double* V, int64_t ldv, int j, double* W, int64_t n, const DotScratch& sc, KrylovState* ks,
                        int maxmv, int m, cudaStream_t st, cudaGraphConditionalHandle hnext) {
    const int nb = pass_blocks((n + 1) / 2, sc);
    launch_k(k_dcgs_update, dim3(nb), dim3(kThreads), 0, st, V, ldv, j, W, n, sc.partial, sc.counter, nb, ks, maxmv, m, hnext);
}
void launch_solve_log(const KrylovState* ks, SolveLog* out, cudaStream_t st) {
    launch_k(k_solve_log, dim3(1), dim3(32), 0, st, ks, out);
}

void launch_norm_init(const double* v, int64_t n, const DotScratch& sc, KrylovState* ks, double rtol, double atol,
                      cudaStream_t st, cudaGraphConditionalHandle hnext) {
    const int nb = pass_blocks(n, sc);
    launch_k(k_norm_init, dim3(nb), dim3(kThreads), 0, st, v, n, sc.partial, sc.counter, nb, ks, rtol, atol, hnext);
}

void launch_backsolve(KrylovState* ks, cudaStream_t st, int in_basis) {
    launch_k(k_backsolve, dim3(1), dim3(kThreads), 0, st, ks, in_basis);
}

template <typename TZ>
void launch_solution_update(double* x, const TZ* Z, int64_t ldz, int64_t n, const KrylovState* ks, int use_scale,
                            cudaStream_t st) {
    int nb = (int)((n + kThreads - 1) / kThreads);
    if (nb > 148 * 8) nb = 148 * 8;
    if (nb < 1) nb = 1;
    launch_k(k_solution_update<TZ>, dim3(nb), dim3(kThreads), 0, st, x, Z, ldz, n, ks, use_scale);
}
template void launch_solution_update<double>(double*, const double*, int64_t, int64_t, const KrylovState*, int,
                                             cudaStream_t);
template void launch_solution_update<float>(double*, const float*, int64_t, int64_t, const KrylovState*, int,
                                            cudaStream_t);

void launch_krylov_reset(KrylovState* ks, cudaStream_t st) { launch_k(k_krylov_reset, dim3(1), dim3(32), 0, st, ks); }

// Restart after a full subspace: keep the matvec count and the tolerance.
__global__ void k_krylov_restart(KrylovState* ks) {
    pdl_entry();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    ks->k = 0; ks->done = 0; ks->converged = 0; ks->reorth = 0;
}
void launch_krylov_restart(KrylovState* ks, cudaStream_t st) { launch_k(k_krylov_restart, dim3(1), dim3(32), 0, st, ks); }

}  // namespace ow3d
