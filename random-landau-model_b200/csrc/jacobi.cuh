// Batched two-sided cyclic Jacobi eigensolver for small complex Hermitian matrices, double
// precision, one CTA per matrix with the matrix and its rotations resident in shared memory.
//
// It is the small-order alternative to the Householder path of heev.cu (reduction,
// tridiagonal solve, back-transformation), both replacing the reference's per-matrix
// LAPACKE_zheevd (diag_wrappers/mkl_diag.cpp:2-9).  Same contract: the upper triangle of each
// column-major matrix is read, eigenvalues ascend, eigenvector k overwrites column k.
//
// Algorithm (cyclic Jacobi with the round-robin "tournament" ordering, so that the n/2 rotations
// of one round touch disjoint index pairs and run in parallel):
//   for each sweep, until the off-diagonal mass is below 1e-32 of the total mass:
//     for each of the m-1 rounds (m = n rounded up to even; index n is a bye for odd n):
//       1. thread k computes the rotation of pair k from A_pp, A_qq and b = A_pq: with
//          h = A_qq - A_pp and u = 2 sgn(h) / (|h| + sqrt(h^2 + 4 |b|^2)) the tangent is
//          t = u |b|, c = 1/sqrt(1 + t^2), J = [[c, c u b], [-c u conj(b), c]] on (p, q);
//          then J^H A J has (p, q) entry 0 and diagonal A_pp - u |b|^2, A_qq + u |b|^2;
//       2. A <- J^H A J by 2 x 2 blocks: a thread takes the block of two pairs, applies both
//          rotations and writes it back (only the upper triangle is kept: an entry that lies
//          below the diagonal is read and written as its conjugate); V <- V J, a thread per
//          (row, pair).
// Two __syncthreads per round; there are no other waits.  The blocks of a round are disjoint,
// so no two threads touch the same element.  The round is a chain of latencies (the three
// dependent square roots and divisions of the rotation, the shared-memory round trips), so it
// is kept short: with separate column and row phases over A and a rotation through |b|, tau
// and t the order-16 kernel took 202 us on 81 matrices and 1,143 us on 8,450; now 133 and 875.
// On many matrices the bound is the shared-memory pipe (by count of the accesses about 200
// wavefronts of the 265 cycles a round takes per matrix and SM, a third of them V's).
//
// Shared memory: A with an odd leading dimension (the row phase's stride-ld accesses of 16
// bytes then hit distinct banks), V with leading dimension n, the round's rotations, the
// block reduction partials.  16 (n (n|1) + n^2) bytes: 33 KB at n = 32, 131 KB at n = 64,
// 206 KB at n = 80, the largest order served (JAC_MAX_N).
#pragma once
#include "common.cuh"

#include <algorithm>

namespace rlmb {

static constexpr int JAC_MAX_N = 80;
static constexpr int JAC_MAX_SWEEPS = 30;

struct JacRot {
    double c;           // cosine
    cplx se;            // s e
    int p, q;           // p < q; q = n: the bye of an odd order
    int on;             // 0: no rotation this round (bye, or A_pq already zero)
};

// Warps per matrix: enough that the matrices resident per SM (as many as fit in its 228 KB of
// shared memory, or the batch's share of them) bring about 20 warps, and no more than give
// every thread a task; from order ~60 on a matrix alone fills the SM's shared memory and its
// own 8 warps must hide the latency.
__host__ __device__ inline size_t jacobi_smem(int n);
inline int jacobi_threads(int n, int nb) {
    const int np = (n + (n & 1)) / 2;
    int per_sm = (int)((size_t)233472 / (jacobi_smem(n) + 1024));
    per_sm = std::min(std::min(std::max(per_sm, 1), 32), (nb + 147) / 148);
    const int tasks = np * (np - 1) / 2 + n * np;
    int w = std::min((20 + per_sm - 1) / per_sm, 8);
    w = std::max(std::min(w, tasks / 32), 1);
    return 32 * std::max(w, (std::max(np, n) + 31) / 32);   // step 1 needs a thread per pair
}
__host__ __device__ inline int jacobi_ld(int n) { return n | 1; }
__host__ __device__ inline size_t jacobi_smem(int n) {
    const int m = n + (n & 1);
    return (size_t)sizeof(cplx) * ((size_t)n * jacobi_ld(n) + (size_t)n * n) + sizeof(JacRot) * (size_t)(m / 2) +
           sizeof(double) * (2 * 32 + 2 * (size_t)n) + sizeof(int) * (size_t)n;
}

// Pair k of round rd of the tournament of m players, p < q.
__device__ __forceinline__ void jac_pair(int k, int rd, int m, int& p, int& q) {
    int a = m - 1, b = rd;
    if (k > 0) {
        a = rd + k;
        if (a >= m - 1) a -= m - 1;
        b = rd - k;
        if (b < 0) b += m - 1;
    }
    p = a < b ? a : b;
    q = a < b ? b : a;
}

// (x_p, x_q) <- (c x_p - conj(se) x_q, se x_p + c x_q): columns p, q of A J or V J
__device__ __forceinline__ void jac_rot_cols(cplx& xp, cplx& xq, double c, cplx se) {
    const cplx p0 = xp, q0 = xq;
    xp = cscale(p0, c);
    xq = cscale(q0, c);
    cfmac(xp, se, mk(-q0.x, -q0.y));
    cfma(xq, se, p0);
}
// (y_p, y_q) <- (c y_p - se y_q, conj(se) y_p + c y_q): rows p, q of J^H A
__device__ __forceinline__ void jac_rot_rows(cplx& yp, cplx& yq, double c, cplx se) {
    const cplx p0 = yp, q0 = yq;
    yp = cscale(p0, c);
    yq = cscale(q0, c);
    cfma(yp, se, mk(-q0.x, -q0.y));
    cfmac(yq, se, p0);
}

// One CTA of jacobi_threads(n) threads per matrix; dynamic shared memory jacobi_smem(n).
__global__ void __launch_bounds__(256) k_jacobi(cplx* __restrict__ Ag, double* __restrict__ W, int* __restrict__ info,
                                                int n) {
    extern __shared__ __align__(16) unsigned char jac_smem[];
    const int ld = jacobi_ld(n);
    const int m = n + (n & 1);
    const int np = m / 2;
    cplx* A = reinterpret_cast<cplx*>(jac_smem);
    cplx* V = A + (size_t)n * ld;
    JacRot* rot = reinterpret_cast<JacRot*>(V + (size_t)n * n);
    double* red = reinterpret_cast<double*>(rot + np);   // [2][32] warp partials
    double* lam = red + 64;                              // eigenvalues
    int* rank = reinterpret_cast<int*>(lam + 2 * n);
    const int tid = threadIdx.x;
    const int nt = blockDim.x;
    const int G = nt / n;              // (threads of a whole column: loads, stores, masses)
    const int r = tid % n, g = tid / n;
    const bool act = g < G;
    const int nblk = np * (np - 1) / 2, nv = n * np;
    const size_t mat = blockIdx.x;
    cplx* Am = Ag + mat * (size_t)n * n;

    // load: the upper triangle of column c is rows 0..c (the lower one is not kept)
    for (int c = g; act && c < n; c += G) {
        if (r <= c) {
            cplx v = Am[(size_t)c * n + r];
            if (c == r) v.y = 0.0;
            A[(size_t)c * ld + r] = v;
        }
        V[(size_t)c * n + r] = mk(c == r ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();

    int converged = 0;
    for (int sweep = 0; sweep <= JAC_MAX_SWEEPS; ++sweep) {
        // off-diagonal and diagonal mass
        double off = 0.0, dia = 0.0;
        for (int c = g; act && c < n; c += G) {
            const double a2 = r <= c ? cabs2(A[(size_t)c * ld + r]) : 0.0;
            if (c == r) dia += a2;
            else off += 2.0 * a2;
        }
        off = warp_sum(off);
        dia = warp_sum(dia);
        if ((tid & 31) == 0) {
            red[tid >> 5] = off;
            red[32 + (tid >> 5)] = dia;
        }
        __syncthreads();
        off = 0.0;
        dia = 0.0;
        for (int w = 0; w < nt / 32; ++w) {
            off += red[w];
            dia += red[32 + w];
        }
        __syncthreads();   // red is rewritten by the next sweep's check
        if (off <= 1e-32 * (off + dia)) {
            converged = 1;
            break;
        }
        if (sweep == JAC_MAX_SWEEPS) break;
        for (int rd = 0; rd < m - 1; ++rd) {
            // 1. rotations of the round, thread k for pair k
            if (tid < np) {
                int p, q;
                jac_pair(tid, rd, m, p, q);
                JacRot R;
                R.p = p;
                R.q = q;
                R.on = 0;
                R.c = 1.0;
                R.se = mk(0.0, 0.0);
                if (q < n) {
                    const cplx b = A[(size_t)q * ld + p];
                    const double b2 = cabs2(b);
                    if (b2 > 0.0) {
                        const double a = A[(size_t)p * ld + p].x, d = A[(size_t)q * ld + q].x;
                        const double h = d - a;
                        const double u = copysign(2.0, h) / (fabs(h) + sqrt(fma(4.0, b2, h * h)));
                        const double c = rsqrt(fma(u * b2, u, 1.0));
                        R.on = 1;
                        R.c = c;
                        R.se = cscale(b, u * c);
                        A[(size_t)p * ld + p] = mk(a - u * b2, 0.0);
                        A[(size_t)q * ld + q] = mk(d + u * b2, 0.0);
                        A[(size_t)q * ld + p] = mk(0.0, 0.0);
                    }
                }
                rot[tid] = R;
            }
            __syncthreads();
            // 2. the blocks of two pairs (k, l), k < l, then V
            for (int t = tid; t < nblk + nv; t += nt) {
                if (t < nblk) {
                    int l = (int)((1.0f + sqrtf(8.0f * t + 1.0f)) * 0.5f);
                    if (l * (l - 1) / 2 > t) --l;
                    else if (l * (l + 1) / 2 <= t) ++l;
                    const JacRot K = rot[t - l * (l - 1) / 2], L = rot[l];
                    if (!K.on && !L.on) continue;
                    const int kq = K.q, lq = L.q;
                    const bool ok = kq < n, ol = lq < n;   // (an odd order's bye has no second index)
                    const int kr = ok ? kq : K.p, lr = ol ? lq : L.p;
                    const bool f0 = K.p > L.p, f1 = kr > L.p, f2 = K.p > lr, f3 = kr > lr;   // kept as the conjugate
                    cplx* a0 = A + (f0 ? K.p * ld + L.p : L.p * ld + K.p);
                    cplx* a1 = A + (f1 ? kr * ld + L.p : L.p * ld + kr);
                    cplx* a2 = A + (f2 ? K.p * ld + lr : lr * ld + K.p);
                    cplx* a3 = A + (f3 ? kr * ld + lr : lr * ld + kr);
                    cplx pp = *a0, qp = *a1, pq = *a2, qq = *a3;
                    if (f0) pp.y = -pp.y;
                    if (f1) qp.y = -qp.y;
                    if (f2) pq.y = -pq.y;
                    if (f3) qq.y = -qq.y;
                    if (L.on) {
                        jac_rot_cols(pp, pq, L.c, L.se);
                        jac_rot_cols(qp, qq, L.c, L.se);
                    }
                    if (K.on) {
                        jac_rot_rows(pp, qp, K.c, K.se);
                        jac_rot_rows(pq, qq, K.c, K.se);
                    }
                    if (f0) pp.y = -pp.y;
                    if (f1) qp.y = -qp.y;
                    if (f2) pq.y = -pq.y;
                    if (f3) qq.y = -qq.y;
                    *a0 = pp;
                    if (ok) *a1 = qp;
                    if (ol) *a2 = pq;
                    if (ok && ol) *a3 = qq;
                } else {
                    const int k = (t - nblk) / n, row = (t - nblk) - k * n;
                    const JacRot R0 = rot[k];
                    if (!R0.on) continue;
                    cplx* vp = V + (size_t)R0.p * n + row;
                    cplx* vq = V + (size_t)R0.q * n + row;
                    cplx xp = *vp, xq = *vq;
                    jac_rot_cols(xp, xq, R0.c, R0.se);
                    *vp = xp;
                    *vq = xq;
                }
            }
            __syncthreads();
        }
    }

    // ascending order: the rank of eigenvalue t among all (ties by index)
    if (tid < n) lam[tid] = A[(size_t)tid * ld + tid].x;
    __syncthreads();
    if (tid < n) {
        const double l = lam[tid];
        int rk = 0;
        for (int j = 0; j < n; ++j) {
            const double lj = lam[j];
            rk += (lj < l || (lj == l && j < tid)) ? 1 : 0;
        }
        rank[tid] = rk;
        W[mat * n + rk] = l;
    }
    __syncthreads();
    for (int c = g; act && c < n; c += G) Am[(size_t)rank[c] * n + r] = V[(size_t)c * n + r];
    if (tid == 0 && info) info[mat] = converged ? 0 : 1;
}

}  // namespace rlmb
