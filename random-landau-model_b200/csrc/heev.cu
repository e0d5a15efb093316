// Batched complex Hermitian eigensolver (sm_100a), double precision or mixed precision.
//
// Replaces the reference's dense solver calls: mkl_heevd (diag_wrappers/mkl_diag.cpp:2-9,
// LAPACKE_zheevd col-major 'U'), cusolver_diag_hamil (diag_wrappers/cusolver_diag.cu:3-22)
// and magma_diag_hamil (diag_wrappers/magma_diag.cu:2-49).  The LAPACK arithmetic those
// calls reach is restated from its published algorithms:
//
//   reduction      A = Q T Q^H (zhetrd, uplo='U').  From order 256: panels of 16 columns
//                  (32 from order 1024 in double precision; k_hetrd_panel_c, zlatrd restated)
//                  whose rank-32 (rank-64) updates run as batched GEMMs over all SMs
//                  (launch_zgemm); the last leading
//                  block (order <= 64, or all of a smaller matrix) by the unblocked,
//                  look-ahead k_hetrd (zhetd2), its triangle resident in shared memory.
//   tridiagonal    below order 600 k_tridiag: eigenvalues by Sturm counts (dstebz restated,
//                  seeded from a shared grid, Newton-accelerated); eigenvectors by twisted
//                  factorisation, or for clusters inverse iteration / twisted solves with
//                  modified Gram-Schmidt (dstein restated).  From order 600 divide and
//                  conquer (tridiag_dc.cuh: secular equations, Gu-Eisenstat vectors, DMMA
//                  merges).  Either one may be pinned or autotuned per order.
//   back-transform X = Q Z (zunmtr): with X resident on the SM in blocks of 16 reflectors
//                  (k_larft, then k_ormtr_mma in double precision up to order 408, k_ormtr in
//                  single precision below 256), else T factors from batched Gram GEMMs and
//                  three GEMM launches per block of 64 reflectors.
//   mixed mode     the reduction and back-transformation in single precision, then double
//                  refinement of every eigenpair (k_ref_*, Ogita-Aishima restated, with
//                  cluster Rayleigh-Ritz).
//   small orders   up to order 20 (12 in the mesh solves, autotuned up to 80) the whole eigensolve
//                  is batched two-sided Jacobi instead (jacobi.cuh).
//
// Waits are __syncthreads inside one CTA and the hardware barriers of a cluster
// (k_hetrd_panel_c, k_dc_merge), except the panel queue's per-column counts (k_hetrd_panel_q), whose spins
// are bounded in time and abort the chunk when they run out.
#include "common.cuh"
#include "jacobi.cuh"
#include "tridiag_dc.cuh"
#include "small_eig.cuh"
#include "zgemm.cuh"
#include "zgemm_tc.cuh"
#include "zgemm_tma.cuh"

#include <cfloat>
#include <map>
#include <vector>
#include <cmath>

namespace rlmb {


// --------------------------------------------------------------- block reductions
template <int NT, class R>
__device__ __forceinline__ R block_sum(R v, R* red) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    R s = 0;
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) s += red[i];
    return s;
}
template <int NT, class C, class R>
__device__ __forceinline__ C block_sum_c(C v, R* red) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) {
        red[2 * w] = v.x;
        red[2 * w + 1] = v.y;
    }
    __syncthreads();
    C s = cz<C>();
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) {
        s.x += red[2 * i];
        s.y += red[2 * i + 1];
    }
    return s;
}

template <class C>
__device__ __forceinline__ void smem_atomic_add(C* p, C v) {
    atomicAdd(&p->x, v.x);
    atomicAdd(&p->y, v.y);
}

// ------------------------------------------------------------------ k_hetrd
// Storage of the active leading block: global column-major (ld = n) while it is large,
// packed upper triangle in shared memory (column c at c(c+1)/2) once it fits.
template <class C>
struct GlobalStore {
    C* a;
    int n;
    __device__ __forceinline__ C* at(int r, int c) const { return a + (size_t)c * n + r; }
};
template <class C>
struct SharedStore {
    C* s;
    __device__ __forceinline__ C* at(int r, int c) const { return s + (c * (c + 1) / 2 + r); }
};

// One 16 x 16 tile (rows from r0, columns from c0) of the upper triangle of the leading m x m
// block: applies the rank-2 update A -= v w^H + w v^H of the previous reflector (UPD) and forms
// the tile's part of A' vn.  Lane (lr = lane % 8, lc = lane / 8) holds rows lr + 8 i (i < 2) and
// columns lc + 4 j (j < 4), so that the cross-lane sums are over 4 lanes per row and 8 per
// column.  rowsum: on lanes with bit 3 clear, row r0 + lr + 8 (lane / 16); colsum: on even
// lanes, column c0 + lc + 4 (lr / 2).  The vectors are readable up to the next multiple of 16.
template <bool INSIDE, bool UPD, class C, class R, class S>
__device__ __forceinline__ void hetrd_tile(const S& st, int m, int r0, int c0, const C* __restrict__ v,
                                           const C* __restrict__ w, const C* __restrict__ vn, C& rowsum, C& colsum,
                                           R& quad) {
    const int lane = threadIdx.x & 31, lr = lane & 7, lc = lane >> 3;
    C vr[2], wr[2], vnr[2], rs[2], es[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = r0 + lr + 8 * i;
        if (UPD) {
            vr[i] = v[r];
            wr[i] = w[r];
        }
        vnr[i] = vn[r];
        rs[i] = cz<C>();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = c0 + lc + 4 * j;
        C x[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = r0 + lr + 8 * i;
            x[i] = INSIDE || (c < m && r <= c) ? *st.at(r, c) : cz<C>();
        }
        const C vnc = vn[c];
        es[j] = cz<C>();
        C vc, wc;
        if (UPD) {
            vc = cconj(v[c]);
            wc = cconj(w[c]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = r0 + lr + 8 * i;
            const bool in = INSIDE || (c < m && r <= c);
            if (UPD) {
                C u = cmul(vr[i], wc);   // (summed apart: onto x, every term would round at x's size)
                cfma(u, wr[i], vc);
                x[i] = csub(x[i], u);
                if (!INSIDE && r == c) x[i].y = 0;
                if (in) *st.at(r, c) = x[i];
                else x[i] = cz<C>();
            }
            if (!INSIDE && r == c) {   // the diagonal: real, counted once
                const C d = cscale(vnc, x[i].x);
                rs[i] = cadd(rs[i], d);
                quad -= vnr[i].x * d.x + vnr[i].y * d.y;
                x[i] = cz<C>();
            }
            cfma(rs[i], x[i], vnc);
            cfmac(es[j], x[i], vnr[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) quad += 2 * (vnr[i].x * rs[i].x + vnr[i].y * rs[i].y);
    const bool b4 = (lane & 16) != 0;
    rowsum = cadd(b4 ? rs[1] : rs[0], shfl_xor(b4 ? rs[0] : rs[1], 16));
    rowsum = cadd(rowsum, shfl_xor(rowsum, 8));
    const bool b2 = (lane & 4) != 0, b1 = (lane & 2) != 0;
    C y[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) y[j] = cadd(b2 ? es[j + 2] : es[j], shfl_xor(b2 ? es[j] : es[j + 2], 4));
    colsum = cadd(b1 ? y[1] : y[0], shfl_xor(b1 ? y[0] : y[1], 2));
    colsum = cadd(colsum, shfl_xor(colsum, 1));
}

// The pass over all tiles of the leading m x m block, dealt to the CTA's warps.  PARTS: tile
// t's sums go to its own slots part[32 t ..] (16 rows, then 16 columns; hetrd_sum adds them up),
// else into pn by shared-memory atomics.  Returns this lane's share of vn^H A' vn.
template <int NT, bool PARTS, bool UPD, class C, class R, class S>
__device__ __forceinline__ R hetrd_pass(S st, int m, const C* __restrict__ v, const C* __restrict__ w,
                                        const C* __restrict__ vn, C* pn) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane & 7, lc = lane >> 3;
    const int nb = (m + 15) / 16, nt = nb * (nb + 1) / 2;
    R quad = 0;
    for (int t = warp; t < nt; t += NT / 32) {
        // t-th tile (row block rb <= column block cb), column blocks in turn
        int cb = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
        if ((cb + 1) * (cb + 2) / 2 <= t) ++cb;
        else if (cb * (cb + 1) / 2 > t) --cb;
        const int rb = t - cb * (cb + 1) / 2, r0 = 16 * rb, c0 = 16 * cb;
        C rowsum, colsum;
        if (rb < cb && c0 + 16 <= m) hetrd_tile<true, UPD, C, R>(st, m, r0, c0, v, w, vn, rowsum, colsum, quad);
        else hetrd_tile<false, UPD, C, R>(st, m, r0, c0, v, w, vn, rowsum, colsum, quad);
        if (PARTS) {
            if (!(lane & 8)) pn[32 * t + lr + 8 * (lane >> 4)] = rowsum;
            if (!(lane & 1)) pn[32 * t + 16 + lc + 4 * (lr >> 1)] = colsum;
        } else {
            const int r = r0 + lr + 8 * (lane >> 4), c = c0 + lc + 4 * (lr >> 1);
            if (!(lane & 8) && r < m) smem_atomic_add(&pn[r], rowsum);
            if (!(lane & 1) && c < m) smem_atomic_add(&pn[c], colsum);
        }
    }
    return quad;
}
// (A' vn)[r] of the leading m x m block from the tiles' parts.
template <class C>
__device__ __forceinline__ C hetrd_sum(const C* __restrict__ part, int m, int r) {
    const int nb = (m + 15) / 16, b = r >> 4;
    const C* q = part + 16 * b * (b + 1) + (r & 15);   // tile (0, b)
    C s = q[16];
    for (int rb = 0; rb < b; ++rb) {                   // column sums of tiles (0, b) .. (b, b)
        q += 32;
        s = cadd(s, q[16]);
    }
    for (int cb = b; cb < nb; ++cb) {                  // row sums of tiles (b, b) .. (b, nb - 1)
        s = cadd(s, *q);
        q += 32 * (cb + 1);
    }
    return s;
}

// Householder reflector of zlarfg for (alpha, x) with ||x||^2 = xnorm2: returns beta, tau
// and the scale applied to x.  Called by whole warps with the same arguments in every lane.
template <class C, class R>
__device__ __forceinline__ void reflector(const C alpha, R xnorm2, R& beta, C& tau, C& scal) {
    if (xnorm2 == 0 && alpha.y == 0) {
        beta = alpha.x;
        tau = cz<C>();
        scal = cm<C>(1, 0);
        return;
    }
    const R nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2);
    beta = alpha.x >= 0 ? -nrm : nrm;
    // tau = ((beta - alpha.x) / beta, -alpha.y / beta), scal = conj(den) / |den|^2: every warp computes
    // the reflector, its lanes one of the four quotients each, so that a warp issues one division
    // (quotients, not products with an inverse: that of a denormal |den|^2 overflows)
    const C den = cm<C>(alpha.x - beta, alpha.y);
    const int k = threadIdx.x & 3;
    const R num = k == 0 ? beta - alpha.x : k == 1 ? -alpha.y : k == 2 ? den.x : -den.y;
    const R quo = num / (k < 2 ? beta : cabs2(den));
    tau.x = __shfl_sync(0xffffffffu, quo, 0);
    tau.y = __shfl_sync(0xffffffffu, quo, 1);
    scal.x = __shfl_sync(0xffffffffu, quo, 2);
    scal.y = __shfl_sync(0xffffffffu, quo, 3);
}

// Unblocked reduction A = Q T Q^H (zhetd2, uplo='U') with look-ahead: step i's rank-2
// update and step i-1's matrix-vector product share one pass over the leading block.
// a: n*n col-major (upper triangle), real type R (double, or float in the mixed mode); the
// leading m x m block is reduced (m < n after the blocked panels of k_hetrd_panel_c, which
// own E and TAU from index m - 1 on).
// On exit column c (c >= 1) rows 0..c-2 hold the reflector of step c-1 (its entry c-1 is
// 1 and not stored), D/E the tridiagonal (double) and TAU the reflector scalars.  The
// leading block moves into shared memory once its packed upper triangle fits in
// `tri_cap` elements.
// Three barriers per column: w of the last reflector, the next column brought up to date and
// its norm; the new reflector; the pass.  x^H v in w = x - tau/2 (x^H v) v is tau v^H A v, which
// the pass sums on the way.  Small blocks (PARTS, m <= HT_PARTS_MAX) keep the pass's sums per
// tile, so that it needs neither atomics nor a cleared accumulator.
// Bound: instruction issue (several CTAs per SM hide the chains of the reflector).  With one
// row and 16 columns per lane, shared double atomics and eight barriers per column 4,624 matrices
// of order 64 took 4.03 ms, 2,304 of order 32 0.69 ms and 128 of order 129 0.93 ms; now 1.85,
// 0.17 and 0.46.
static constexpr int HT_PARTS_MAX = 144;
// vectors are read up to the next multiple of 16, times zero; with sums by atomics, where shared memory
// sets the largest order, that may be the next array
__host__ __device__ constexpr int hetrd_pad(int m) { return m <= HT_PARTS_MAX ? (m + 15) / 16 * 16 : m; }
__host__ __device__ constexpr int hetrd_pn(int m) {   // elements of pn
    return m <= HT_PARTS_MAX ? 16 * (hetrd_pad(m) / 16) * (hetrd_pad(m) / 16 + 1) : hetrd_pad(m);
}
template <int NT, class R, bool PARTS>
__global__ void __launch_bounds__(NT, NT >= 512 ? 1 : 512 / NT)
k_hetrd(typename Cx<R>::T* __restrict__ A, double* __restrict__ D, double* __restrict__ E,
        typename Cx<R>::T* __restrict__ TAU, int n, int m, int tri_cap) {
    typedef typename Cx<R>::T C;
    constexpr int NW = NT / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int mp = hetrd_pad(m);
    C* v = reinterpret_cast<C*>(smem_raw);   // [mp] reflector of step i
    C* vn = v + mp;                           // [mp] the next one / column buffer
    C* w = vn + mp;                           // [mp] w of step i
    C* pn = w + mp;                           // [hetrd_pn(m)] A' v
    C* alpha = pn + hetrd_pn(m);              // [1] (PARTS; else the entry of pn after the column's)
    R* normp = reinterpret_cast<R*>(alpha + (PARTS ? 1 : 0));   // [NW] parts of the column's norm
    R* quadp = normp + NW;                    // [NW] parts of v^H A' v
    C* tri = reinterpret_cast<C*>(smem_raw) + 3 * mp + hetrd_pn(m) + (PARTS ? 1 : 0) + 2 * NW * sizeof(R) / sizeof(C);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t mat = blockIdx.x;
    GlobalStore<C> gs{A + mat * (size_t)n * n, n};
    SharedStore<C> ss{tri};
    double* dd = D + mat * n;
    double* ee = E + mat * n;
    C* tt = TAU + mat * n;
    for (int r = tid; r < 3 * mp + hetrd_pn(m); r += NT) v[r] = cz<C>();
    if (lane == 0) quadp[warp] = 0;
    if (tid == 0 && m == n) {
        ee[n - 1] = 0.0;
        tt[n - 1] = cz<C>();
    }
    __syncthreads();
    bool resident = false;
    C tau = cz<C>();
    bool act = false;
    // column i: rows 0..i of the leading block; step i's reflector (v) came from column i + 1
    for (int i = m - 1; i >= 0; --i) {
        if (!resident && (i + 1) * (i + 2) / 2 <= tri_cap) {
            // move the leading (i+1)x(i+1) upper triangle into shared memory
            for (int c = warp; c <= i; c += NW)
                for (int r = lane; r <= c; r += 32) *ss.at(r, c) = *gs.at(r, c);
            resident = true;
            __syncthreads();
        }
        // (1) w of step i, and column i brought up to date with it
        if (!PARTS) alpha = pn + min(i + 1, m - 1);
        R q2 = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) q2 += quadp[k];
        const R al = (R)-0.5 * cabs2(tau) * q2;   // x^H v = conj(tau) v^H A v, al = -tau/2 x^H v
        C wi = cmul(tau, PARTS ? hetrd_sum(pn, i + 1, i) : pn[i]);
        wi.x += al;                               // (v[i] = 1)
        if (!act) wi = cz<C>();
        R part = 0;
        for (int r = tid; r <= i; r += NT) {
            C wr = cz<C>(), x = resident ? *ss.at(r, i) : *gs.at(r, i);
            if (act) {
                const C vr = v[r];
                wr = cmul(tau, PARTS ? hetrd_sum(pn, i + 1, r) : pn[r]);
                wr.x += al * vr.x;
                wr.y += al * vr.y;
                C u = cmul(vr, cconj(wi));
                x = csub(x, cadd(u, wr));
            }
            w[r] = wr;
            vn[r] = x;
            if (r < i - 1) part += cabs2(x);
            if (r == i - 1) *alpha = x;
            if (r == i) dd[i] = x.x;
        }
        if (i == 0) break;
        part = warp_sum(part);
        if (lane == 0) normp[warp] = part;
        __syncthreads();
        // (2) reflector of step i-1: alpha = A'[i-1][i], x = A'[0..i-2][i]
        R xn2 = 0, beta;
#pragma unroll
        for (int k = 0; k < NW; ++k) xn2 += normp[k];
        C scal;
        const bool upd = act;
        reflector(*alpha, xn2, beta, tau, scal);
        act = !(tau.x == 0 && tau.y == 0);
        for (int r = tid; r < i; r += NT) {
            if (!PARTS) pn[r] = cz<C>();
            if (r == i - 1) {
                vn[r] = cm<C>(1, 0);
                *gs.at(r, i) = cm<C>(beta, 0);
            } else {
                const C x = act ? cmul(scal, vn[r]) : vn[r];
                vn[r] = x;
                *gs.at(r, i) = x;   // reflector storage stays in global memory
            }
        }
        if (tid == 0) {
            ee[i - 1] = beta;
            tt[i - 1] = tau;
        }
        __syncthreads();
        // (3) update [0..i-1]^2 with (v, w), accumulate pn = A' vn
        R quad;
        if (upd)
            quad = resident ? hetrd_pass<NT, PARTS, true, C, R>(ss, i, v, w, vn, pn)
                            : hetrd_pass<NT, PARTS, true, C, R>(gs, i, v, w, vn, pn);
        else
            quad = resident ? hetrd_pass<NT, PARTS, false, C, R>(ss, i, v, w, vn, pn)
                            : hetrd_pass<NT, PARTS, false, C, R>(gs, i, v, w, vn, pn);
        quad = warp_sum(quad);
        if (lane == 0) quadp[warp] = quad;
        __syncthreads();
        C* t = v;
        v = vn;
        vn = t;
    }
}

// ------------------------------------------------------------ k_tridiag
// Eigen-decomposition of the real symmetric tridiagonal (d, e), scaled by a power of two to unit
// norm.  A CTA of T threads takes up to T eigenvalues of one matrix at a time (T: the order
// rounded up to a warp, at most TRI_THREADS); eigenvalues in k_tridiag<1, T>, eigenvectors in
// k_tridiag<2, T>, stored row-major in Z (Z[j*n + k] = component j of eigenvector k) so that the
// recurrences of the threads touch consecutive addresses.  Per-thread scratch columns live in
// the interleaved workspace LU (5 * n * tri_columns(n) doubles per matrix, same layout).
// Bound: instruction issue in phase 1 (the counts), the latency of the scratch columns in phase
// 2.  With 256 threads whatever the order, range and sign tests on the FP64 pipe in every step
// and vectors walked from thread-dependent indices (uncoalesced) the phases took 9.7 and 12.4 ms
// on 4,224 matrices of order 256, 0.74 and 0.70 on 4,624 of order 64, 1.16 and 0.54 on 18 of
// order 300; now 5.7 and 5.4, 0.42 and 0.22, 0.34 and 0.18.
static constexpr int TRI_THREADS = 256;
static constexpr int INV_MAXITS = 5;
// scratch columns per matrix: one per eigenvector up to order 384 (a chunk of few matrices then
// spreads a matrix over two CTAs), else one per thread of one CTA
__host__ __device__ constexpr int tri_columns(int n) { return n <= 384 ? (n + 31) / 32 * 32 : TRI_THREADS; }

// Sturm count by the leading principal minors of T - x I,
//   p_j = (d_j - x) p_{j-1} - e_{j-1}^2 p_{j-2},   p_{-1} = 1:
// the number of sign changes along p_{-1}, p_0, ..., p_{n-1} is the number of eigenvalues below
// x (Sturm).  A minor below 2^-100 of its predecessor is replaced by -2^-100 of that, a change of T by
// less than 2^-99 |T| that keeps the recurrence from dying out where couplings or d_j - x vanish
// (a replacement of fixed size would be a large change of T after smaller minors).  The pair
// (p_j, p_{j-1}) is kept in range by exact powers of two, every fourth step: |T| is about 1, so
// four steps grow it by less than 2^12, and p_j, above 2^-500 where the pair is in range, shrinks by
// 2^400 at most.  Signs, sizes and exponents are looked at as integers, which leaves the FP64 pipe
// the recurrences.  The derivatives p_j' ride along for the Newton step ratio = p_{n-1}/p_{n-1}'.
static constexpr int STURM_BIG = (1023 + 400) << 20, STURM_SMALL = (1023 - 400) << 20, STURM_TINY = 100 << 20;
__device__ __forceinline__ double sturm_nonzero(double pn, double p) {
    const int hp = __double2hiint(p);
    return (__double2hiint(pn) & 0x7fffffff) < (hp & 0x7fffffff) - STURM_TINY
               ? __hiloint2double((hp ^ 0x80000000) - STURM_TINY, __double2loint(p)) : pn;
}
__device__ __forceinline__ int sturm_change(double a, double b) {
    return (int)((unsigned)(__double2hiint(a) ^ __double2hiint(b)) >> 31);
}
// 2^-k for the larger of the two, if that is out of range (else 1)
__device__ __forceinline__ bool sturm_range(double p, double pm, double& sc) {
    const int m = max(__double2hiint(p) & 0x7fffffff, __double2hiint(pm) & 0x7fffffff);
    if (m <= STURM_BIG && m >= STURM_SMALL) return false;
    sc = __hiloint2double((1023 - min((m >> 20) - 1023, 1000)) << 20, 0);
    return true;
}
__device__ __forceinline__ int sturm_poly(const double* __restrict__ d, const double* __restrict__ e2, int n,
                                          double x, double& ratio) {
    double pm = 1.0, p = sturm_nonzero(d[0] - x, 1.0);   // p_{j-1}, p_j
    double dpm = 0.0, dp = -1.0;                          // their derivatives in x
    int cnt = sturm_change(p, 1.0);
    auto step = [&](int j) {
        const double a = d[j] - x, ee = e2[j - 1];
        const double pn = sturm_nonzero(fma(a, p, -ee * pm), p);
        const double dpn = fma(a, dp, -fma(ee, dpm, p));
        cnt += sturm_change(pn, p);
        pm = p;
        dpm = dp;
        p = pn;
        dp = dpn;
    };
    int j = 1;
    for (; j + 4 <= n; j += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) step(j + u);
        double sc;
        if (sturm_range(p, pm, sc)) {
            p *= sc;
            pm *= sc;
            dp *= sc;
            dpm *= sc;
        }
    }
    for (; j < n; ++j) step(j);
    ratio = p / dp;
    return cnt;
}
// The counts at two shifts, the two recurrences interleaved (no derivatives).
__device__ __forceinline__ void sturm_count2(const double* __restrict__ d, const double* __restrict__ e2, int n,
                                             double xa, double xb, int& ca, int& cb) {
    double pma = 1.0, pa = sturm_nonzero(d[0] - xa, 1.0), pmb = 1.0, pb = sturm_nonzero(d[0] - xb, 1.0);
    int na = sturm_change(pa, 1.0), nb = sturm_change(pb, 1.0);
    auto step = [&](int j) {
        const double ee = e2[j - 1], dj = d[j];
        const double qa = sturm_nonzero(fma(dj - xa, pa, -ee * pma), pa);
        const double qb = sturm_nonzero(fma(dj - xb, pb, -ee * pmb), pb);
        na += sturm_change(qa, pa);
        nb += sturm_change(qb, pb);
        pma = pa;
        pa = qa;
        pmb = pb;
        pb = qb;
    };
    int j = 1;
    for (; j + 4 <= n; j += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) step(j + u);
        double sc;
        if (sturm_range(pa, pma, sc)) {
            pa *= sc;
            pma *= sc;
        }
        if (sturm_range(pb, pmb, sc)) {
            pb *= sc;
            pmb *= sc;
        }
    }
    for (; j < n; ++j) step(j);
    ca = na;
    cb = nb;
}

// deterministic start vector entries in (-1, 1)
__device__ __forceinline__ double start_entry(int k, int j) {
    uint32_t h = (uint32_t)k * 0x9E3779B1u ^ ((uint32_t)j * 0x85EBCA77u + 0x165667B1u);
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    h *= 0x297A2D39u;
    h ^= h >> 15;
    return ((double)h + 0.5) * (2.0 / 4294967296.0) - 1.0;
}

// Eigenvector of an isolated eigenvalue x of (d, e) by the twisted factorisation of
// T - x I (Parlett & Dhillon): forward pivots D+ (the Sturm recurrence) and backward
// pivots D-, twist index r minimising |gamma_r| = |D+_r + D-_r - (d_r - x)|, then
// z_r = 1, z_j = L_j z_{j+1} (j < r), z_j = M_j z_{j-1} (j > r) with the multipliers
// L_j = -e_j / D+_j and M_j = -e_{j-1} / D-_j.
// The multipliers, not the pivots, go to the thread's scratch columns lp and lm (stride `ls`), so
// that only the factorisation divides.  Every loop runs over the same j in all threads -- the
// parts of z beside the twist start at thread-dependent indices, but are walked from the ends
// with the value held at 1 until the twist is reached -- so that a warp's accesses stay
// coalesced, and loads are issued eight steps ahead of their use.
static constexpr int TW_AHEAD = 8;
__device__ void twisted_vector(const double* __restrict__ d, const double* __restrict__ e, int n, double x,
                               double pivmin, double* __restrict__ z, int k, double* __restrict__ lp,
                               double* __restrict__ lm, int ls) {
    if (n == 1) {
        z[k] = 1.0;
        return;
    }
    auto pivot = [&](double q) { return fabs(q) <= pivmin ? -pivmin : q; };
    // D+ (forward, stationary) and D- (backward, progressive) are independent division
    // chains: one loop advances both, step t forward to t + 1 and backward to n - 2 - t
    double qf = pivot(d[0] - x), qb = pivot(d[n - 1] - x);
    auto advance = [&](int t) {
        const int jb = n - 1 - t;
        const double l = -e[t] / qf, m = -e[jb - 1] / qb;
        lp[(size_t)t * ls] = l;
        lm[(size_t)jb * ls] = m;
        qf = pivot(fma(e[t], l, d[t + 1] - x));
        qb = pivot(fma(e[jb - 1], m, d[jb - 1] - x));
    };
    int r = 0;
    double gbest = DBL_MAX;
    auto twist = [&](int j, double gam) {
        gam = fabs(gam);
        if (gam < gbest) {
            gbest = gam;
            r = j;
        }
    };
    // until the chains have met: after step t0 - 1, D+ is at t0 and D- at n - 1 - t0
    const int t0 = n / 2;
    for (int t = 0; t < t0; ++t) advance(t);
    if (n & 1) twist(t0, qf + qb - (d[t0] - x));
    else {   // D+ is at n/2, D- at n/2 - 1: their other halves are the last multipliers
        twist(t0, t0 + 1 < n ? fma(e[t0], lm[(size_t)(t0 + 1) * ls], qf) : qf);
        twist(t0 - 1, t0 >= 2 ? fma(e[t0 - 2], lp[(size_t)(t0 - 2) * ls], qb) : qb);
    }
    // beyond: gamma_j = D+_j + e_j M_{j+1} and D-_j + e_{j-1} L_{j-1}, from multipliers stored
    // by the other chain
    for (int t = t0; t < n - 1; t += TW_AHEAD) {
        double am[TW_AHEAD], ap[TW_AHEAD];
#pragma unroll
        for (int u = 0; u < TW_AHEAD; ++u) {
            const int jf = t + u + 1, jb = n - 2 - t - u;   // D+_jf, D-_jb after step t + u
            am[u] = jf + 1 < n ? lm[(size_t)(jf + 1) * ls] : 0.0;
            ap[u] = jb >= 1 ? lp[(size_t)(jb - 1) * ls] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < TW_AHEAD; ++u) {
            if (t + u >= n - 1) break;
            advance(t + u);
            const int jf = t + u + 1, jb = n - 2 - t - u;
            twist(jf, jf + 1 < n ? fma(e[jf], am[u], qf) : qf);
            twist(jb, jb >= 1 ? fma(e[jb - 1], ap[u], qb) : qb);
        }
    }
    // z from the twist outwards; WRITE: times scale, to memory
    double nrm2 = 1.0, big = 1.0, rn = 1.0;
    auto walk = [&](auto write) {
        double zz = rn;
        for (int j0 = n - 2; j0 >= 0; j0 -= TW_AHEAD) {   // j = r - 1 .. 0
            double l[TW_AHEAD];
#pragma unroll
            for (int u = 0; u < TW_AHEAD; ++u) l[u] = j0 - u >= 0 ? lp[(size_t)(j0 - u) * ls] : 0.0;
#pragma unroll
            for (int u = 0; u < TW_AHEAD; ++u) {
                const int j = j0 - u;
                if (j >= 0 && j < r) {
                    zz *= l[u];
                    if constexpr (decltype(write)::value) {
                        z[(size_t)j * n + k] = zz;
                    } else {
                        nrm2 = fma(zz, zz, nrm2);
                        if (fabs(zz) > fabs(big)) big = zz;
                    }
                }
            }
        }
        if constexpr (decltype(write)::value) z[(size_t)r * n + k] = rn;
        zz = rn;
        for (int j0 = 1; j0 < n; j0 += TW_AHEAD) {   // j = r + 1 .. n - 1
            double l[TW_AHEAD];
#pragma unroll
            for (int u = 0; u < TW_AHEAD; ++u) l[u] = j0 + u < n ? lm[(size_t)(j0 + u) * ls] : 0.0;
#pragma unroll
            for (int u = 0; u < TW_AHEAD; ++u) {
                const int j = j0 + u;
                if (j < n && j > r) {
                    zz *= l[u];
                    if constexpr (decltype(write)::value) {
                        z[(size_t)j * n + k] = zz;
                    } else {
                        nrm2 = fma(zz, zz, nrm2);
                        if (fabs(zz) > fabs(big)) big = zz;
                    }
                }
            }
        }
    };
    walk(std::false_type{});
    rn = 1.0 / sqrt(nrm2);
    if (big < 0.0) rn = -rn;
    walk(std::true_type{});
}

// PHASE 1 (k_stebz): eigenvalues into W.  PHASE 2 (k_stein): eigenvectors from W.
// Grid (matrices, CTAs per matrix); CTA y of Y takes the eigenvalues y, y + Y, ...
template <int PHASE, int T>
__global__ void __launch_bounds__(T, 512 / T)
k_tridiag(const double* __restrict__ D, const double* __restrict__ E, double* __restrict__ W,
          double* __restrict__ Z, double* __restrict__ LU, int* __restrict__ info, int n) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* d = reinterpret_cast<double*>(smem_raw);   // [n]
    double* e = d + n;                                  // [n]
    double* e2 = e + n;                                 // [n]
    double* lam = e2 + n;                               // [n]
    int* leader = reinterpret_cast<int*>(lam + n);      // [n] first index of k's cluster
    __shared__ double s_gx[T + 1];                      // (first the warps' parts of the norms, then grid points)
    __shared__ int s_fail;
    static_assert(4 * (T / 32) <= T + 1, "s_gx holds the norms' parts");
    double (*s_red)[T / 32] = reinterpret_cast<double (*)[T / 32]>(s_gx);
    const int tid = threadIdx.x;
    const size_t mat = blockIdx.x;
    const int sub = blockIdx.y, subs = gridDim.y;
    const size_t nn = (size_t)n * n;
    double* z = Z + mat * nn;
    // per-thread scratch columns (stride ls): U diag / super1 / super2, multipliers and swap
    // flags of the LU of T - x I; the twisted solve uses the first two for its multipliers
    const int ls = tri_columns(n);
    const size_t lus = (size_t)n * ls;
    double* la = LU + mat * 5 * lus + sub * ((n + subs - 1) / subs) + tid;
    double* lb = la + lus;
    double* lc2 = lb + lus;
    double* lm = lc2 + lus;
    double* lp = lm + lus;

    // Gershgorin interval, one-norm (of the rows), largest |e|
    double gl = DBL_MAX, gu = -DBL_MAX, onenrm = 0.0, emax = 0.0;
    for (int j = tid; j < n; j += T) {
        const double dj = D[mat * n + j];
        const double ej = j < n - 1 ? E[mat * n + j] : 0.0;
        const double ep = j > 0 ? E[mat * n + j - 1] : 0.0;
        d[j] = dj;
        e[j] = ej;
        const double off = fabs(ep) + fabs(ej);
        gl = fmin(gl, dj - off);
        gu = fmax(gu, dj + off);
        onenrm = fmax(onenrm, fabs(dj) + off);
        emax = fmax(emax, fabs(ej));
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
        gl = fmin(gl, __shfl_xor_sync(0xffffffffu, gl, m));
        gu = fmax(gu, __shfl_xor_sync(0xffffffffu, gu, m));
        onenrm = fmax(onenrm, __shfl_xor_sync(0xffffffffu, onenrm, m));
        emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, m));
    }
    if ((tid & 31) == 0) {
        s_red[0][tid >> 5] = gl;
        s_red[1][tid >> 5] = gu;
        s_red[2][tid >> 5] = onenrm;
        s_red[3][tid >> 5] = emax;
    }
    if (tid == 0) s_fail = 0;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < T / 32; ++w) {
        gl = fmin(gl, s_red[0][w]);
        gu = fmax(gu, s_red[1][w]);
        onenrm = fmax(onenrm, s_red[2][w]);
        emax = fmax(emax, s_red[3][w]);
    }
    if (!(onenrm > 1e3 * DBL_MIN)) {
        // T = 0 to underflow: eigenvalues are the diagonal (sorted), eigenvectors unit vectors
        if (PHASE == 2 || sub > 0) return;
        if (tid == 0) {
            for (int k = 0; k < n; ++k) leader[k] = k;
            for (int k = 1; k < n; ++k)
                for (int q = k; q > 0 && d[leader[q]] < d[leader[q - 1]]; --q) {
                    const int tmp = leader[q];
                    leader[q] = leader[q - 1];
                    leader[q - 1] = tmp;
                }
        }
        __syncthreads();
        for (int k = tid; k < n; k += T) {
            W[mat * n + k] = d[leader[k]];
            for (int j = 0; j < n; ++j) z[(size_t)j * n + k] = j == leader[k] ? 1.0 : 0.0;
        }
        if (tid == 0 && info) info[mat] = 0;
        return;
    }
    // scale T to a one-norm in [1, 2) (exactly; the eigenvalues are scaled back)
    const int ex = min(max(ilogb(onenrm), -1000), 1000);
    const double scale = ldexp(1.0, -ex), unscale = ldexp(1.0, ex);
    gl *= scale;
    gu *= scale;
    onenrm *= scale;
    emax *= scale;
    for (int j = tid; j < n; j += T) {   // (this thread's own entries)
        d[j] *= scale;
        e[j] *= scale;
        e2[j] = e[j] * e[j];
    }
    const double pivmin = DBL_MIN * fmax(1.0, emax * emax);
    {
        const double tnorm = fmax(fabs(gl), fabs(gu));
        gl -= 2.1 * tnorm * DBL_EPSILON * n + 4.2 * pivmin;
        gu += 2.1 * tnorm * DBL_EPSILON * n + 4.2 * pivmin;
    }
    __syncthreads();
    // ---- eigenvalue k: bisection on Sturm counts (dstebz bracketing, restated), accelerated
    //      by safeguarded Newton steps on det(T - x I), taken from the current point or from
    //      either end of the bracket, with the step scaled by the number m of eigenvalues in
    //      the bracket (exact for an m-fold root)
    if (PHASE == 1) {
    const double atol = 2.0 * DBL_EPSILON * onenrm;
    // one collective pass first: Sturm counts at the T+1 equally spaced points of
    // the Gershgorin interval (count 0 at its left end, n at its right end), so that every
    // eigenvalue starts from the grid cell holding it instead of the whole interval
    __shared__ int s_gc[T + 1];
    {
        const int t = tid;
        s_gx[t] = t == 0 ? gl : gl + (gu - gl) * ((double)t / T);
        if (t == 0) {
            s_gc[0] = 0;
            s_gx[T] = gu;
            s_gc[T] = n;
        } else {
            double rr;
            s_gc[t] = sturm_poly(d, e2, n, s_gx[t], rr);
        }
    }
    __syncthreads();
    for (int k = tid * subs + sub; k < n; k += T * subs) {
        int cell = 0;   // largest grid point with count <= k
        for (int step = T / 2; step >= 1; step >>= 1)
            if (cell + step < T && s_gc[cell + step] <= k) cell += step;
        double lo = s_gx[cell], hi = s_gx[cell + 1];
        int clo = s_gc[cell], chi = s_gc[cell + 1];
        // Newton steps p/p' recorded at the bracket ends (valid flags), bracket widths of the
        // last two steps (bisection is forced when the bracket did not halve over two steps)
        double rlo = 0.0, rhi = 0.0;
        bool vlo = false, vhi = false;
        double w1 = hi - lo, w2 = hi - lo;
        double x = 0.5 * (lo + hi);
        double res = x;
        for (int it = 0; it < 200; ++it) {
            double ratio;
            const int c = sturm_poly(d, e2, n, x, ratio);
            const bool rok = isfinite(ratio);
            if (c > k) { hi = x; chi = c; rhi = ratio; vhi = rok; } else { lo = x; clo = c; rlo = ratio; vlo = rok; }
            const double tol = fmax(atol, 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)));
            if (hi - lo <= tol) { res = 0.5 * (lo + hi); break; }
            double xn = 0.5 * (lo + hi);
            // Newton candidates x - m p/p' from x and from the two bracket ends, m = eigenvalues
            // in the bracket (the modified step converges on an m-fold cluster); the smallest
            // step first: a step within tol is verified by paired counts, else the first
            // candidate inside the bracket is taken
            const double m = (double)(chi - clo);
            double cs[3], cn[3];
            int nc = 0;
            if (rok) { cs[nc] = fabs(m * ratio); cn[nc++] = x - m * ratio; }
            if (vlo && x != lo) { cs[nc] = fabs(m * rlo); cn[nc++] = lo - m * rlo; }
            if (vhi && x != hi) { cs[nc] = fabs(m * rhi); cn[nc++] = hi - m * rhi; }
            for (int i = 1; i < nc; ++i)
                for (int j = i; j > 0 && cs[j] < cs[j - 1]; --j) {
                    const double ts = cs[j], tn = cn[j];
                    cs[j] = cs[j - 1]; cn[j] = cn[j - 1];
                    cs[j - 1] = ts; cn[j - 1] = tn;
                }
            bool accepted = false;
            for (int ci = 0; ci < nc; ++ci) {
                const double nt = cn[ci];
                if (cs[ci] <= tol) {
                    // converged step: accept only if Sturm counts bracket index k at nt +- 2 tol
                    const double a0 = fmax(lo, nt - 2.0 * tol), b0 = fmin(hi, nt + 2.0 * tol);
                    int ca, cb;
                    sturm_count2(d, e2, n, a0, b0, ca, cb);
                    if (ca <= k && cb > k) { res = fmin(fmax(nt, lo), hi); accepted = true; break; }
                    if (ca > k) { hi = a0; chi = ca; vhi = false; } else { lo = b0; clo = cb; vlo = false; }
                    xn = 0.5 * (lo + hi);
                    break;
                }
                if (nt > lo && nt < hi) { xn = nt; break; }
            }
            if (accepted) break;
            if (hi - lo > 0.5 * w2) xn = 0.5 * (lo + hi);
            w2 = w1;
            w1 = hi - lo;
            if (xn <= lo || xn >= hi) { res = 0.5 * (lo + hi); break; }
            x = xn;
            res = x;
        }
        W[mat * n + k] = res * unscale;
    }
    if (tid == 0 && sub == 0 && info) info[mat] = 0;
    return;
    }
    for (int k = tid; k < n; k += T) lam[k] = W[mat * n + k] * scale;
    __syncthreads();
    // ---- clusters (relative gap 1e-4 of the norm) and eigenvalue output
    const double ortol = 1e-4 * onenrm;
    for (int k = tid; k < n; k += T) {
        int lead = k;
        while (lead > 0 && lam[lead] - lam[lead - 1] <= ortol) --lead;
        leader[k] = lead;
    }
    __syncthreads();
    // ---- eigenvectors: isolated eigenvalues by one twisted solve; clusters (handled by the
    //      leader's thread) by twisted solves + modified Gram-Schmidt when their members are
    //      still separated, else by inverse iteration with modified Gram-Schmidt
    const double eps = DBL_EPSILON;
    const double dtpcrt = sqrt(0.1 / n);
    for (int k0 = tid * subs + sub; k0 < n; k0 += T * subs) {
        if (leader[k0] != k0) continue;
        int k1 = k0;
        while (k1 + 1 < n && leader[k1 + 1] == k0) ++k1;
        if (k1 == k0) {
            twisted_vector(d, e, n, lam[k0], pivmin, z, k0, la, lb, ls);
            continue;
        }
        // a cluster whose members are still 1e-9 * ||T|| apart: each twisted vector is
        // accurate to ~eps ||T|| / gap, so a twisted solve per member followed by modified
        // Gram-Schmidt inside the cluster replaces the iterations
        double mingap = DBL_MAX;
        for (int k = k0 + 1; k <= k1; ++k) mingap = fmin(mingap, lam[k] - lam[k - 1]);
        if (mingap > 1e-9 * onenrm) {
            for (int k = k0; k <= k1; ++k) {
                twisted_vector(d, e, n, lam[k], pivmin, z, k, la, lb, ls);
                for (int q = k0; q < k; ++q) {
                    double dot = 0.0;
                    for (int j = 0; j < n; ++j) dot += z[(size_t)j * n + q] * z[(size_t)j * n + k];
                    for (int j = 0; j < n; ++j) z[(size_t)j * n + k] -= dot * z[(size_t)j * n + q];
                }
                double x2s = 0.0, big = 0.0;
                for (int j = 0; j < n; ++j) {
                    const double t = z[(size_t)j * n + k];
                    x2s += t * t;
                    if (fabs(t) > fabs(big)) big = t;
                }
                double rn = 1.0 / sqrt(fmax(x2s, DBL_MIN));
                if (big < 0.0) rn = -rn;
                for (int j = 0; j < n; ++j) z[(size_t)j * n + k] *= rn;
            }
            continue;
        }
        double xjm = lam[k0];
        for (int k = k0; k <= k1; ++k) {
            double x = lam[k];
            if (k > k0) {
                const double pertol = 10.0 * fabs(x) * eps + 10.0 * eps * onenrm * 1e-3;
                if (x - xjm < pertol) x = xjm + pertol;
            }
            xjm = x;
            // LU with partial pivoting of T - x I (dlagtf).  The active row carries
            // (u0, u1) = its entries in columns j, j+1; the row pivoted into position j is
            // stored as U diag / super1 / super2 (la, lb, lc2), the multiplier in lm and
            // the swap flag in lp, all at [j * ls] of this thread's columns.
            double u0 = d[0] - x, u1 = n > 1 ? e[0] : 0.0;
            for (int j = 0; j < n - 1; ++j) {
                const double cj = e[j];
                const double anext = d[j + 1] - x;
                const double bnext = j + 1 < n - 1 ? e[j + 1] : 0.0;
                const size_t o = (size_t)j * ls;
                if (fabs(u0) >= fabs(cj)) {
                    const double mult = u0 != 0.0 ? cj / u0 : 0.0;
                    la[o] = u0;
                    lb[o] = u1;
                    lc2[o] = 0.0;
                    lm[o] = mult;
                    lp[o] = 0.0;
                    u0 = anext - mult * u1;
                    u1 = bnext;
                } else {
                    const double mult = u0 / cj;
                    la[o] = cj;
                    lb[o] = anext;
                    lc2[o] = bnext;
                    lm[o] = mult;
                    lp[o] = 1.0;
                    u0 = u1 - mult * anext;
                    u1 = -mult * bnext;
                }
            }
            la[(size_t)(n - 1) * ls] = u0;
            lb[(size_t)(n - 1) * ls] = 0.0;
            lc2[(size_t)(n - 1) * ls] = 0.0;
            // tiny pivots are perturbed to +-tolp in the solves (dlagts job = -1)
            double umax = 0.0;
            for (int j = 0; j < n; ++j) umax = fmax(umax, fabs(la[(size_t)j * ls]));
            const double tolp = fmax(eps * fmax(umax, onenrm), DBL_MIN);
            for (int j = 0; j < n; ++j) z[(size_t)j * n + k] = start_entry(k, j);
            int nrmchk = 0;
            bool conv = false;
            for (int its = 0; its < INV_MAXITS; ++its) {
                // scale the right-hand side to ||b||_1 = n * onenrm * max(eps, |u_nn|)
                double b1 = 0.0;
                for (int j = 0; j < n; ++j) b1 += fabs(z[(size_t)j * n + k]);
                const double unn = fabs(la[(size_t)(n - 1) * ls]);
                const double sc = n * onenrm * fmax(eps, unn) / fmax(b1, DBL_MIN);
                // forward: y = L^{-1} P b  (the active right-hand side value is carried)
                double rc = z[k] * sc;
                for (int j = 0; j < n - 1; ++j) {
                    const size_t o = (size_t)j * n + k;
                    const size_t ol = (size_t)j * ls;
                    const double bnext = z[(size_t)(j + 1) * n + k] * sc;
                    const double mult = lm[ol];
                    if (lp[ol] != 0.0) {
                        z[o] = bnext;
                        rc = rc - mult * bnext;
                    } else {
                        z[o] = rc;
                        rc = bnext - mult * rc;
                    }
                }
                z[(size_t)(n - 1) * n + k] = rc;
                // backward: U x = y
                double x1 = 0.0, x2 = 0.0;   // x_{j+1}, x_{j+2}
                double xmax = 0.0;
                for (int j = n - 1; j >= 0; --j) {
                    const size_t o = (size_t)j * n + k;
                    const size_t ol = (size_t)j * ls;
                    double u = la[ol];
                    if (fabs(u) < tolp) u = u >= 0.0 ? tolp : -tolp;
                    const double xj = (z[o] - lb[ol] * x1 - lc2[ol] * x2) / u;
                    z[o] = xj;
                    x2 = x1;
                    x1 = xj;
                }
                // modified Gram-Schmidt against the earlier members of the cluster, twice: what is left of an
                // iterate that is all but one of them is the first pass's rounding
                for (int pass = 0; pass < 2; ++pass)
                    for (int q = k0; q < k; ++q) {
                        double dot = 0.0;
                        for (int j = 0; j < n; ++j) dot += z[(size_t)j * n + q] * z[(size_t)j * n + k];
                        for (int j = 0; j < n; ++j) z[(size_t)j * n + k] -= dot * z[(size_t)j * n + q];
                    }
                for (int j = 0; j < n; ++j) xmax = fmax(xmax, fabs(z[(size_t)j * n + k]));
                if (xmax < dtpcrt) continue;   // not yet amplified enough
                if (++nrmchk < 3) continue;    // two extra iterations after acceptance
                conv = true;
                break;
            }
            // normalise, largest component positive (dstein)
            double x2s = 0.0, big = 0.0;
            for (int j = 0; j < n; ++j) {
                const double t = z[(size_t)j * n + k];
                x2s += t * t;
                if (fabs(t) > fabs(big)) big = t;
            }
            double rn = 1.0 / sqrt(fmax(x2s, DBL_MIN));
            if (big < 0.0) rn = -rn;
            for (int j = 0; j < n; ++j) z[(size_t)j * n + k] *= rn;
            if (!conv) atomicAdd(&s_fail, 1);
        }
    }
    __syncthreads();
    if (tid == 0 && info && s_fail) atomicAdd(&info[mat], s_fail);   // (cleared by phase 1)
}

// --------------------------------------------------------------- back-transformation
// X = Q Z with Q = H_{n-2} ... H_0 (H_i = I - tau_i v_i v_i^H, v_i on rows 0..i, v_i[i] = 1,
// v_i[0..i-1] stored in A[0..i-1][i+1]).  Reflectors are grouped in blocks of ORM_NB
// consecutive indices i0..i1; a block's product P = H_{i1} ... H_{i0} = I - V T V^H
// (compact WY form, T lower triangular, built by k_larft) is applied as
//   X <- X - V (T (V^H X)),
// blocks in increasing order (LAPACK zlarft / zlarfb, restated).
static constexpr int ORM_NB = 16;     // reflectors per block
static constexpr int ORM_RPT = 16;    // rows of the Z chunk held per thread
static constexpr int ORM_VS = ORM_NB + 1;   // padded shared-memory row stride of a V block

template <class C>
__device__ __forceinline__ C refl_entry(const C* __restrict__ a, int n, int i, int r) {
    // component r of reflector i (zero for i > n-2 padding)
    if (i > n - 2 || r > i) return cz<C>();
    if (r == i) return cm<C>(1, 0);
    return a[(size_t)(i + 1) * n + r];
}

// its address, or null with the implicit value in imm
template <class C>
__device__ __forceinline__ const C* refl_addr(const C* __restrict__ a, int n, int i, int r, cplx& imm) {
    if (i <= n - 2 && r < i) return a + (size_t)(i + 1) * n + r;
    imm.x = i <= n - 2 && r == i ? 1.0 : 0.0;
    return nullptr;
}

// T factor of one block of one matrix, grid (blocks, matrices):
//   T[k][k] = tau_k,  T[k][q] = -tau_k sum_{l=q}^{k-1} (v_k^H v_l) T[l][q]   (q < k)
template <class R>
__global__ void __launch_bounds__(128)
k_larft(const typename Cx<R>::T* __restrict__ A, const typename Cx<R>::T* __restrict__ TAU,
        typename Cx<R>::T* __restrict__ Tw, int n) {
    typedef typename Cx<R>::T C;
    __shared__ C G[ORM_NB][ORM_NB];
    __shared__ C T[ORM_NB][ORM_NB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t mat = blockIdx.y;
    const C* a = A + mat * (size_t)n * n;
    const C* tau = TAU + mat * n;
    const int i0 = blockIdx.x * ORM_NB;
    // G[k][l] = v_k^H v_l for l < k: rows 0..i0+l overlap; a warp takes k = warp, warp + 4, ...
    // with the entries of v_k in registers' reach for all l
    for (int k = warp; k < ORM_NB; k += 4) {
        const int ik = i0 + k;
        if (ik > n - 2) break;
        for (int l0 = 0; l0 < k; l0 += 4) {
            C s[4] = {cz<C>(), cz<C>(), cz<C>(), cz<C>()};
            const int top = i0 + min(l0 + 3, k - 1);
            for (int r = lane; r <= top; r += 32) {
                const C vk = refl_entry(a, n, ik, r);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (l0 + u < k) cfmac(s[u], vk, refl_entry(a, n, i0 + l0 + u, r));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const C t = warp_sum(s[u]);
                if (lane == 0 && l0 + u < k) G[k][l0 + u] = t;
            }
        }
    }
    __syncthreads();
    if (warp == 0) {
        for (int k = 0; k < ORM_NB; ++k) {
            const int ik = i0 + k;
            const C tk = ik <= n - 2 ? tau[ik] : cz<C>();
            if (lane < ORM_NB) {
                C val = cz<C>();
                if (lane == k) {
                    val = tk;
                } else if (lane < k && ik <= n - 2) {
                    C s = cz<C>();
                    for (int l = lane; l < k; ++l) cfma(s, G[k][l], T[l][lane]);
                    val = cscale(cmul(tk, s), (R)-1);
                }
                T[k][lane] = val;
            }
            __syncwarp();
        }
    }
    __syncthreads();
    C* out = Tw + (mat * gridDim.x + blockIdx.x) * ORM_NB * ORM_NB;
    for (int i = threadIdx.x; i < ORM_NB * ORM_NB; i += 128) out[i] = T[i / ORM_NB][i % ORM_NB];
}

// The same in double precision on the FP64 tensor path, one warp per block and LM_WARPS blocks per
// CTA: G = V^H V as the three 8 x 8 tiles on and below the diagonal (both fragments of a product
// are the same entries, 4 rows x 8 reflectors of V straight from memory), then lane q forms
// column q of T in registers.  grid (ceil(blocks / LM_WARPS), matrices).
// Bound: the latency of V's loads.  As dot products with a warp sum each it took 0.43 ms for
// 4,624 matrices of order 64 and 0.11 ms for 2,304 of order 32; now 0.10 and 0.03.
static constexpr int LM_WARPS = 4;
__global__ void __launch_bounds__(32 * LM_WARPS)
k_larft_mma(const cplx* __restrict__ A, const cplx* __restrict__ TAU, cplx* __restrict__ Tw, int n, int nblk) {
    __shared__ cplx Gs[LM_WARPS][ORM_NB][ORM_NB + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int j = blockIdx.x * LM_WARPS + warp;
    if (j >= nblk) return;
    const size_t mat = blockIdx.y;
    const cplx* a = A + mat * (size_t)n * n;
    const int i0 = j * ORM_NB, rows = min(i0 + ORM_NB, n - 1);
    const int ia = i0 + g, ib = i0 + 8 + g;   // this lane's reflectors
    double r0[2] = {0, 0}, m0[2] = {0, 0}, r1[2] = {0, 0}, m1[2] = {0, 0}, r2[2] = {0, 0}, m2[2] = {0, 0};
    auto product = [&](double (&re)[2], double (&im)[2], cplx x, cplx y) {   // conj(x) y
        dmma884(re, x.x, y.x);
        dmma884(im, x.x, y.y);
        dmma884(re, x.y, y.y);
        dmma884(im, -x.y, y.x);
    };
#pragma unroll 4
    for (int k = 0; k < rows; k += 4) {
        const cplx x = refl_entry(a, n, ia, k + q), y = refl_entry(a, n, ib, k + q);
        product(r0, m0, x, x);
        product(r1, m1, y, x);
        product(r2, m2, y, y);
    }
    cplx (&G)[ORM_NB][ORM_NB + 1] = Gs[warp];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        G[g][2 * q + e] = mk(r0[e], m0[e]);
        G[8 + g][2 * q + e] = mk(r1[e], m1[e]);
        G[8 + g][8 + 2 * q + e] = mk(r2[e], m2[e]);
    }
    __syncwarp();
    // T[k][c] = -tau_k sum_{l < k} G[k][l] T[l][c], T[c][c] = tau_c, zero above the diagonal
    const int c = lane & 15;
    cplx t[ORM_NB];
    const cplx tl = i0 + c <= n - 2 ? TAU[mat * n + i0 + c] : mk(0, 0);
    cplx* out = Tw + (mat * nblk + j) * ORM_NB * ORM_NB;
#pragma unroll
    for (int k = 0; k < ORM_NB; ++k) {
        const cplx tk = mk(__shfl_sync(0xffffffffu, tl.x, k), __shfl_sync(0xffffffffu, tl.y, k));
        cplx s0 = mk(0, 0), s1 = mk(0, 0);
#pragma unroll
        for (int l = 0; l < k; ++l) cfma(l & 1 ? s1 : s0, G[k][l], t[l]);
        const cplx s = cadd(s0, s1);
        t[k] = k == c ? tk : k < c ? mk(0, 0) : cscale(cmul(tk, s), -1.0);
        if (lane < ORM_NB) out[k * ORM_NB + c] = t[k];
    }
}

// asynchronous global -> shared copy of one complex element (16 or 8 bytes)
__device__ __forceinline__ void cp_async_elem(double2* smem_dst, const double2* gmem_src) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_elem(float2* smem_dst, const float2* gmem_src) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Stage block j of V (rows 0..i1, layout [r][k]) and its T factor into shared memory:
// stored reflector entries by cp.async, the implicit 1 and the zeros below by plain stores.
template <class C>
__device__ __forceinline__ void stage_block(const C* __restrict__ a, const C* __restrict__ tsrc,
                                            C* vsb, C* tsb, int n, int j) {
    const int t = threadIdx.x;
    const int i0 = j * ORM_NB;
    const int i1 = min(i0 + ORM_NB - 1, n - 2);
    for (int idx = t; idx < (i1 + 1) * ORM_NB; idx += blockDim.x) {
        const int r = idx / ORM_NB, k = idx % ORM_NB;
        const int i = i0 + k;
        C* dst = &vsb[r * ORM_VS + k];
        if (i <= n - 2 && r < i) cp_async_elem(dst, &a[(size_t)(i + 1) * n + r]);
        else *dst = (i <= n - 2 && r == i) ? cm<C>(1, 0) : cz<C>();
    }
    if (t < ORM_NB * ORM_NB) cp_async_elem(&tsb[t], &tsrc[t]);
    cp_async_commit();
}

// Apply all blocks to a chunk of CH columns of Z (row-major Z[r*n + col], real) and write
// the chunk of X (column-major, column = eigenvector).  NT threads; thread t owns column
// t % CH and the rows g + RG*q (g = t / CH, RG = NT/CH, q < RPT) in registers.  With dbuf
// the next block's V and T are copied asynchronously while the current block is applied.
template <int CH, int NT, int RPT, class R, int MINB = 1>
__global__ void __launch_bounds__(NT, MINB)
k_ormtr(const typename Cx<R>::T* __restrict__ A, const typename Cx<R>::T* __restrict__ Tw,
        const double* __restrict__ Z, typename Cx<R>::T* __restrict__ X, int n, int dbuf) {
    typedef typename Cx<R>::T C;
    constexpr int RG = NT / CH, NW = NT / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* vsbuf[2];
    vsbuf[0] = reinterpret_cast<C*>(smem_raw);                    // [n][ORM_VS]
    vsbuf[1] = dbuf ? vsbuf[0] + (size_t)n * ORM_VS : vsbuf[0];
    C* tsbuf[2];
    tsbuf[0] = vsbuf[0] + (size_t)(dbuf ? 2 : 1) * n * ORM_VS;       // [ORM_NB][ORM_NB]
    tsbuf[1] = dbuf ? tsbuf[0] + ORM_NB * ORM_NB : tsbuf[0];
    C* wsum = tsbuf[0] + (size_t)(dbuf ? 2 : 1) * ORM_NB * ORM_NB;   // [NW][ORM_NB][CH]
    C* w2 = wsum + NW * ORM_NB * CH;                               // [ORM_NB][CH]
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int c = t % CH, g = t / CH;
    const size_t mat = blockIdx.y;
    const int col = blockIdx.x * CH + c;
    const C* a = A + mat * (size_t)n * n;
    const double* z = Z + mat * (size_t)n * n;
    const int nblk = (n - 1 + ORM_NB - 1) / ORM_NB;
    const C* tw = Tw + mat * (size_t)nblk * ORM_NB * ORM_NB;
    C x[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
        const int r = g + RG * q;
        x[q] = (r < n && col < n) ? cm<C>(z[(size_t)r * n + col], 0) : cz<C>();
    }
    if (dbuf && nblk > 0) stage_block(a, tw, vsbuf[0], tsbuf[0], n, 0);
    for (int j = 0; j < nblk; ++j) {
        const int i0 = j * ORM_NB;
        const int i1 = min(i0 + ORM_NB - 1, n - 2);
        if (dbuf) {
            if (j + 1 < nblk) {
                stage_block(a, tw + (size_t)(j + 1) * ORM_NB * ORM_NB, vsbuf[(j + 1) & 1],
                            tsbuf[(j + 1) & 1], n, j + 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
        } else {
            stage_block(a, tw + (size_t)j * ORM_NB * ORM_NB, vsbuf[0], tsbuf[0], n, j);
            cp_async_wait<0>();
        }
        __syncthreads();
        const C* vs = vsbuf[j & 1];
        const C* ts = tsbuf[j & 1];
        // partial W = V^H X over this thread's rows
        C wp[ORM_NB];
#pragma unroll
        for (int k = 0; k < ORM_NB; ++k) wp[k] = cz<C>();
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
            const int r = g + RG * q;
            if (r <= i1) {
                const C* vr = vs + r * ORM_VS;
#pragma unroll
                for (int k = 0; k < ORM_NB; ++k) cfmac(wp[k], vr[k], x[q]);
            }
        }
        // reduce over the row groups: inside the warp, then across the NW warps
#pragma unroll
        for (int s2 = CH; s2 < 32; s2 <<= 1)
#pragma unroll
            for (int k = 0; k < ORM_NB; ++k) wp[k] = cadd(wp[k], shfl_xor(wp[k], s2));
        if (lane < CH)
#pragma unroll
            for (int k = 0; k < ORM_NB; ++k) wsum[(warp * ORM_NB + k) * CH + lane] = wp[k];
        __syncthreads();
        C wk = cz<C>();
        if (t < ORM_NB * CH) {
            for (int w8 = 0; w8 < NW; ++w8) wk = cadd(wk, wsum[w8 * ORM_NB * CH + t]);
            wsum[t] = wk;   // W[k][c] at t = k*CH + c (slot of warp 0, already read)
        }
        __syncthreads();
        if (t < ORM_NB * CH) {
            const int k = t / CH, cc = t % CH;
            C s = cz<C>();
            for (int q2 = 0; q2 <= k; ++q2) cfma(s, ts[k * ORM_NB + q2], wsum[q2 * CH + cc]);
            w2[t] = s;
        }
        __syncthreads();
        // X -= V W2 on rows <= i1
        C wc[ORM_NB];
#pragma unroll
        for (int k = 0; k < ORM_NB; ++k) wc[k] = w2[k * CH + c];
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
            const int r = g + RG * q;
            if (r <= i1) {
                const C* vr = vs + r * ORM_VS;
                C s = cz<C>();
#pragma unroll
                for (int k = 0; k < ORM_NB; ++k) cfma(s, vr[k], wc[k]);
                x[q] = csub(x[q], s);
            }
        }
        __syncthreads();
    }
    // write the chunk column-major through shared memory (coalesced along rows)
    C* xs = vsbuf[0];   // [CH][n]
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
        const int r = g + RG * q;
        if (r < n) xs[(size_t)c * n + r] = x[q];
    }
    __syncthreads();
    C* xo = X + mat * (size_t)n * n;
    const int col0 = blockIdx.x * CH;
    for (int idx = t; idx < CH * n; idx += NT) {
        const int cc = idx / n, r = idx % n;
        if (col0 + cc < n) xo[(size_t)(col0 + cc) * n + r] = xs[idx];
    }
}

// The same in double precision on the FP64 tensor path (DMMA, m8n8k4): one CTA keeps CW columns
// of X in shared memory (X[r][c], rows padded to 8) for the whole transformation, so that X
// crosses device memory once whatever the number of blocks.  Per block of 16 reflectors, staged
// as V[r][k]:
//   W = V^H X     2 x CW/8 tiles of 8 x 8, WH warps per tile (each an equal share of the rows,
//                 the shares added by the next product's loads)
//   W <- T W      one tile per warp
//   X -= V W      a warp takes 8-row tiles, W's fragments in registers
// Column c of row r of X and V sits at c ^ om_swz(r), so that the 8 lanes of a 16-byte phase hit
// distinct banks in every fragment: 2 columns x 4 rows (W's operands), 4 even columns x 2 rows
// (X in the accumulator's layout), 4 columns x 2 rows (V in the last product).
// 256 threads where two CTAs or more fit an SM, 512 where X and V leave room for one.
// Bound: the DMMA pipe (8 n^3 flops) and, between the products, barriers and V's staging.
// (order 256: the pipe is 57 % busy).  k_ormtr took 2.76 ms for 4,624 matrices of order 64 and
// 0.34 ms for 2,304 of order 32; this kernel 0.66 and 0.07.  Against the GEMM form (X read twice
// and written once per 64 reflectors), T factors included: order 256, 1,408 matrices 14.5 ->
// 11.0 ms, order 380, 296 matrices 8.6 -> 7.3 ms.
static constexpr int OM_TS = ORM_NB + 2;   // row stride of T
__device__ __forceinline__ int om_swz(int r) { return (r & 1) * 5 + (r & 2); }   // 0, 5, 2, 7 by r mod 4
template <int CW, int NT>
struct OrmtrMma {
    static constexpr int CT = CW / 8, WH = NT / 64 / CT, WS = CW + 2;
    static __host__ __device__ constexpr size_t smem(int n) {
        return sizeof(cplx) * ((size_t)((n + 7) / 8 * 8) * (CW + ORM_NB) + WH * ORM_NB * WS + ORM_NB * OM_TS);
    }
};
template <int CW, int NT>
__global__ void __launch_bounds__(NT, 512 / NT)
k_ormtr_mma(const cplx* __restrict__ A, const cplx* __restrict__ Tw, const double* __restrict__ Z,
            cplx* __restrict__ X, int n) {
    constexpr int CT = OrmtrMma<CW, NT>::CT, WH = OrmtrMma<CW, NT>::WH, WS = OrmtrMma<CW, NT>::WS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int np = (n + 7) / 8 * 8;
    cplx* xs = reinterpret_cast<cplx*>(smem_raw);   // [np][CW]
    cplx* vs = xs + (size_t)np * CW;                // [np][16]
    cplx* ws = vs + (size_t)np * ORM_NB;            // [WH][16][WS]
    cplx* ts = ws + WH * ORM_NB * WS;               // [16][OM_TS]
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, g = lane >> 2, q = lane & 3;
    const int sq = om_swz(q), sg = om_swz(g);       // swizzles of rows 4 k + q and 8 k + g
    const size_t mat = blockIdx.y;
    const int col0 = blockIdx.x * CW;
    const cplx* a = A + mat * (size_t)n * n;
    const double* z = Z + mat * (size_t)n * n;
    const int nblk = (n - 1 + ORM_NB - 1) / ORM_NB;
    const cplx* tw = Tw + mat * (size_t)nblk * ORM_NB * ORM_NB;
    for (int i = t; i < np * CW; i += NT) {
        const int r = i / CW, c = i % CW;
        xs[r * CW + (c ^ om_swz(r))] = mk(r < n && col0 + c < n ? z[(size_t)r * n + col0 + c] : 0.0, 0.0);
    }
    const int m = warp & 1, nt = (warp >> 1) % CT, part = warp / (2 * CT);   // the warp's tile of W, its share
    for (int j = 0; j < nblk; ++j) {
        const int i0 = j * ORM_NB, i1 = min(i0 + ORM_NB - 1, n - 2);
        const int rows = (i1 + 1 + 7) / 8 * 8;
        // stage V (rows 0 .. rows-1, the implicit ones and the zeros included) and T
        for (int k = warp; k < ORM_NB; k += NT / 32) {
            const int ir = i0 + k;
            const cplx* src = a + (size_t)(ir + 1) * n;
            for (int r = lane; r < rows; r += 32) {
                cplx* dst = &vs[r * ORM_NB + (k ^ om_swz(r))];
                if (ir <= n - 2 && r < ir) cp_async_elem(dst, src + r);
                else *dst = mk(ir <= n - 2 && r == ir ? 1.0 : 0.0, 0.0);
            }
        }
        if (t < ORM_NB * ORM_NB)
            cp_async_elem(&ts[(t / ORM_NB) * OM_TS + t % ORM_NB], &tw[(size_t)j * ORM_NB * ORM_NB + t]);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        {   // W tile (m, nt) = V^H X over this warp's rows
            double ra[2] = {0, 0}, rb[2] = {0, 0}, ia[2] = {0, 0}, ib[2] = {0, 0};
            const cplx* vp = vs + q * ORM_NB + ((8 * m + g) ^ sq);
            const cplx* xp = xs + q * CW + ((8 * nt + g) ^ sq);
#pragma unroll 4
            for (int k = 4 * part; k < rows; k += 4 * WH) {
                const cplx v = vp[k * ORM_NB], x = xp[k * CW];
                dmma884(ra, v.x, x.x);
                dmma884(rb, v.y, x.y);
                dmma884(ia, v.x, x.y);
                dmma884(ib, -v.y, x.x);
            }
            cplx* wp = ws + (part * ORM_NB + 8 * m + g) * WS + 8 * nt + 2 * q;
            wp[0] = mk(ra[0] + rb[0], ia[0] + ib[0]);
            wp[1] = mk(ra[1] + rb[1], ia[1] + ib[1]);
        }
        __syncthreads();
        cplx w2[2];
        if (part == 0) {   // T W tile (m, nt): T is lower triangular, so the upper tile row needs half of it
            double cr[2] = {0, 0}, ci[2] = {0, 0};
#pragma unroll
            for (int k = 0; k < ORM_NB; k += 4) {
                if (k >= 8 * (m + 1)) break;
                const cplx v = ts[(8 * m + g) * OM_TS + k + q];
                cplx x = ws[(k + q) * WS + 8 * nt + g];
#pragma unroll
                for (int h = 1; h < WH; ++h) x = cadd(x, ws[(h * ORM_NB + k + q) * WS + 8 * nt + g]);
                dmma884(cr, v.x, x.x);
                dmma884(cr, -v.y, x.y);
                dmma884(ci, v.x, x.y);
                dmma884(ci, v.y, x.x);
            }
            w2[0] = mk(cr[0], ci[0]);
            w2[1] = mk(cr[1], ci[1]);
        }
        __syncthreads();
        if (part == 0) {
            cplx* wp = ws + (8 * m + g) * WS + 8 * nt + 2 * q;
            wp[0] = w2[0];
            wp[1] = w2[1];
        }
        __syncthreads();
        {   // X -= V W
            cplx b[4][CT];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int c = 0; c < CT; ++c) b[k][c] = ws[(4 * k + q) * WS + 8 * c + g];
            for (int r0 = 8 * warp; r0 < rows; r0 += NT / 4) {
                cplx v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = vs[(r0 + g) * ORM_NB + ((4 * k + q) ^ sg)];
#pragma unroll
                for (int c = 0; c < CT; ++c) {
                    cplx* xp = xs + (r0 + g) * CW;
                    const int k0 = (8 * c + 2 * q) ^ sg, k1 = k0 ^ 1;
                    const cplx x0 = xp[k0], x1 = xp[k1];
                    // (summed apart: accumulated onto X, every DMMA would round at X's size)
                    double cr[2] = {0, 0}, ci[2] = {0, 0};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        dmma884(cr, v[k].x, b[k][c].x);
                        dmma884(ci, v[k].x, b[k][c].y);
                        dmma884(cr, -v[k].y, b[k][c].y);
                        dmma884(ci, v[k].y, b[k][c].x);
                    }
                    xp[k0] = mk(x0.x - cr[0], x0.y - ci[0]);
                    xp[k1] = mk(x1.x - cr[1], x1.y - ci[1]);
                }
            }
        }
        __syncthreads();
    }
    if (nblk == 0) __syncthreads();
    cplx* xo = X + mat * (size_t)n * n;
    for (int c = warp; c < CW; c += NT / 32)
        for (int r = lane; r < n && col0 + c < n; r += 32) xo[(size_t)(col0 + c) * n + r] = xs[r * CW + (c ^ om_swz(r))];
}

// ------------------------------------------------ back-transformation for large orders
// For orders whose 16-reflector blocks do not fit the register/shared-memory scheme of
// k_ormtr, X = Q Z is applied with blocks of BT_NB = 64 reflectors (or 128, a tuning choice)
// as tiled complex GEMMs per block (LAPACK zlarfb restated): W' = T (V^H X), then
// X -= V W'.  X lives in global memory (column-major, column = eigenvector) and is read twice
// and written once per block.
static constexpr int BT_NB = 64;
static constexpr int BT_GEMM_MIN = 256;   // mixed mode: order from which the GEMM back-transformation runs
static constexpr int BT_MMA_MAX = 408;    // double precision: order up to which k_ormtr_mma runs (the largest that fits)
// Blocks of 128 reflectors (T from two 64-reflector halves, k_larft128) halve the passes
// over X, but at order 3000 they were no faster in double precision and 10 % slower in single
// precision (the block GEMMs are bound by the tensor pipes, not by X's traffic): they are a
// tuning choice (HeevTune::bt_nb, rlmb_set_heev_config), not the built-in one.
static constexpr int BT128_MIN = 1 << 30;

// T factor of block j (reflectors 64j .. 64j+63) of one matrix from its Gram matrix
// G = V_j^H V_j (column-major 64 x 64, computed by a batched GEMM into the same slot of Tw):
//   T[k][k] = tau_k,  T[k][q] = -tau_k sum_{l=q}^{k-1} G[k][l] T[l][q]   (q < k),
// written back row-major (T[k][q] at k*64 + q); grid (blocks, matrices), 128 threads.
// The recurrence reads G only above its diagonal (S[l][k], l < k, with S[l][k] = G[k][l])
// and T only on and below it, so T overwrites the lower half of the one shared table S as
// it is formed.  Two threads share row q of T (even and odd l), halving the dependent chain.
template <class R>
__global__ void __launch_bounds__(2 * BT_NB)
k_larft64(const typename Cx<R>::T* __restrict__ TAU, typename Cx<R>::T* __restrict__ Tw, int n) {
    typedef typename Cx<R>::T C;
    typedef C Row[BT_NB + 1];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Row* S = reinterpret_cast<Row*>(smem_raw);   // S[l][k] = G[k][l] (l < k); T[k][q] at S[k][q] (q <= k)
    const int j = blockIdx.x, q = threadIdx.x >> 1, h = threadIdx.x & 1;
    const size_t mat = blockIdx.y;
    const C* tau = TAU + mat * n;
    const int nblk = (n - 1 + BT_NB - 1) / BT_NB;
    const int i0 = j * BT_NB;
    C* blk = Tw + (mat * nblk + j) * BT_NB * BT_NB;
    for (int idx = threadIdx.x; idx < BT_NB * BT_NB; idx += 2 * BT_NB) S[idx / BT_NB][idx % BT_NB] = blk[idx];
    __syncthreads();
    for (int k = 0; k < BT_NB; ++k) {
        const int ik = i0 + k;
        const C tk = ik <= n - 2 ? tau[ik] : cz<C>();
        C sum = cz<C>();
        if (q < k)
            for (int l = q + h; l < k; l += 2) cfma(sum, S[l][k], S[l][q]);
        sum = cadd(sum, shfl_xor(sum, 1));
        if (h == 0 && q <= k) S[k][q] = q == k ? tk : cscale(cmul(tk, sum), (R)-1);
        __syncthreads();
    }
    for (int idx = threadIdx.x; idx < BT_NB * BT_NB; idx += 2 * BT_NB) {
        const int k = idx / BT_NB, c = idx % BT_NB;
        blk[idx] = c <= k ? S[k][c] : cz<C>();
    }
}

// T factor of a block of 128 reflectors (128j .. 128j+127) from its 128 x 128 Gram matrix
// G = V^H V (column-major, in the block's slot of Tw), written back row-major:
//   T = [[T1, 0], [T21, T2]],   T21 = -T2 (G21 T1),   G21 = V2^H V1,
// where T1 and T2 are the T factors of the two halves (the k_larft64 recurrence, run on both
// at once by the two halves of the CTA) -- the same matrix the zlarft recurrence gives for
// all 128 reflectors.  Grid (blocks, matrices), 256 threads; shared memory: S1, S2 (the
// halves' recurrence tables as in k_larft64) and Y (G21, then G21 T1).
template <class R>
__global__ void __launch_bounds__(256)
k_larft128(const typename Cx<R>::T* __restrict__ TAU, typename Cx<R>::T* __restrict__ Tw, int n) {
    typedef typename Cx<R>::T C;
    constexpr int H = 64, B = 128;
    typedef C Row[H + 1];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Row* S1 = reinterpret_cast<Row*>(smem_raw);
    Row* S2 = S1 + H;
    Row* Y = S2 + H;
    const int j = blockIdx.x, tid = threadIdx.x;
    const size_t mat = blockIdx.y;
    const C* tau = TAU + mat * n;
    const int nblk = (n - 1 + B - 1) / B;
    const int i0 = j * B;
    C* blk = Tw + (mat * nblk + j) * B * B;
    // S1[l][k] = G(k, l), S2[l][k] = G(64 + k, 64 + l), Y[k][l] = G21(k, l) = G(64 + k, l)
    for (int idx = tid; idx < H * H; idx += 256) {
        const int a = idx / H, b = idx % H;
        S1[a][b] = blk[(size_t)a * B + b];
        S2[a][b] = blk[(size_t)(H + a) * B + H + b];
        Y[b][a] = blk[(size_t)a * B + H + b];
    }
    __syncthreads();
    {
        const int half = tid >> 7, q = (tid & 127) >> 1, h = tid & 1;
        Row* S = half ? S2 : S1;
        const int ib = i0 + H * half;
        for (int k = 0; k < H; ++k) {
            const int ik = ib + k;
            const C tk = ik <= n - 2 ? tau[ik] : cz<C>();
            C sum = cz<C>();
            if (q < k)
                for (int l = q + h; l < k; l += 2) cfma(sum, S[l][k], S[l][q]);
            sum = cadd(sum, shfl_xor(sum, 1));
            if (h == 0 && q <= k) S[k][q] = q == k ? tk : cscale(cmul(tk, sum), (R)-1);
            __syncthreads();
        }
    }
    // thread: row k of the 64 x 64 products, columns q = c4 + 4 i
    const int k = tid >> 2, c4 = tid & 3;
    C acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = cz<C>();
    // Y <- G21 T1: (G21 T1)[k][q] = sum_{l >= q} G21[k][l] T1[l][q], T1[l][q] = S1[l][q]
    for (int l = 0; l < H; ++l) {
        const C g = Y[k][l];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int q = c4 + 4 * i;
            if (l >= q) cfma(acc[i], g, S1[l][q]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) Y[k][c4 + 4 * i] = acc[i];
    __syncthreads();
    // T21 = -T2 Y: T21[k][q] = -sum_{l <= k} T2[k][l] Y[l][q], T2[k][l] = S2[k][l]
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = cz<C>();
    for (int l = 0; l <= k; ++l) {
        const C t2 = S2[k][l];
#pragma unroll
        for (int i = 0; i < 16; ++i) cfma(acc[i], t2, Y[l][c4 + 4 * i]);
    }
    // row-major T: rows 0..63 [T1 0], rows 64..127 [T21 T2]
    for (int idx = tid; idx < H * H; idx += 256) {
        const int a = idx / H, b = idx % H;
        blk[(size_t)a * B + b] = b <= a ? S1[a][b] : cz<C>();
        blk[(size_t)a * B + H + b] = cz<C>();
        blk[(size_t)(H + a) * B + H + b] = b <= a ? S2[a][b] : cz<C>();
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) blk[(size_t)(H + k) * B + c4 + 4 * i] = cscale(acc[i], (R)-1);
}

// Z (row-major real) -> X (column-major complex), grid-stride over all batch entries.
template <class C>
__global__ void k_z_to_x(const double* __restrict__ Z, C* __restrict__ X, int n, size_t total) {
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const size_t nn = (size_t)n * n;
        const size_t mat = idx / nn, rem = idx % nn;
        const int c = (int)(rem / n), r = (int)(rem % n);
        X[idx] = cm<C>(Z[mat * nn + (size_t)r * n + c], 0);
    }
}

// ------------------------------------------------------------------ GEMM operands
// Element accessors for the GEMM engines of launch_zgemm (A: elem(mat, r, k), B: elem(mat, k, c)).

// A(r, k) = P(r, k) of a column-major P (entry at p[k*ld + r]): r contiguous.
template <class C, class PT>
struct OpColA {
    static constexpr bool RFAST = true;
    const PT* p;
    int ld;
    size_t stride;
    __device__ __forceinline__ C elem(size_t mat, int r, int k) const {
        return from_c64<C>(to_c64(p[mat * stride + (size_t)k * ld + r]));
    }
    static constexpr bool CONJ = false;
    __device__ __forceinline__ const PT* addr(size_t mat, int r, int k, cplx&) const {
        return p + mat * stride + (size_t)k * ld + r;
    }
};

// A(r, k) = P(k, r), conjugated if CONJ, of a column-major P (entry (k, r) at p[r*ld + k]):
// the (conjugate) transpose, k contiguous.
template <class C, class PT, bool CJ>
struct OpRowA {
    static constexpr bool RFAST = false;
    static constexpr bool CONJ = CJ;
    const PT* p;
    int ld;
    size_t stride;
    __device__ __forceinline__ C elem(size_t mat, int r, int k) const {
        C v = from_c64<C>(to_c64(p[mat * stride + (size_t)r * ld + k]));
        if (CONJ) v.y = -v.y;
        return v;
    }
    __device__ __forceinline__ const PT* addr(size_t mat, int r, int k, cplx&) const {
        return p + mat * stride + (size_t)r * ld + k;
    }
};

// B(k, c) = P(k, c) of a column-major P (entry at p[c*ld + k]): k contiguous.
template <class C, class PT>
struct OpColB {
    static constexpr bool KFAST = true;
    const PT* p;
    int ld;
    size_t stride;
    __device__ __forceinline__ C elem(size_t mat, int k, int c) const {
        return from_c64<C>(to_c64(p[mat * stride + (size_t)c * ld + k]));
    }
    static constexpr bool CONJ = false;
    __device__ __forceinline__ const PT* addr(size_t mat, int k, int c, cplx&) const {
        return p + mat * stride + (size_t)c * ld + k;
    }
};

// Reflectors i0 + q of a reduced matrix as columns of V (V(r, q) = v_{i0+q}[r], with the
// implicit 1 and the zeros): OpRefl gives A = V (r contiguous), OpReflH A = V^H.
template <class C>
struct OpRefl {
    static constexpr bool RFAST = true;
    const C* a;
    int n, i0;
    __device__ __forceinline__ C elem(size_t mat, int r, int q) const {
        return refl_entry(a + mat * (size_t)n * n, n, i0 + q, r);
    }
    static constexpr bool CONJ = false;
    __device__ __forceinline__ const C* addr(size_t mat, int r, int q, cplx& imm) const {
        return refl_addr(a + mat * (size_t)n * n, n, i0 + q, r, imm);
    }
};
template <class C>
struct OpReflH {
    static constexpr bool RFAST = false;
    const C* a;
    int n, i0;
    __device__ __forceinline__ C elem(size_t mat, int q, int r) const {
        C v = refl_entry(a + mat * (size_t)n * n, n, i0 + q, r);
        v.y = -v.y;
        return v;
    }
    static constexpr bool CONJ = true;
    __device__ __forceinline__ const C* addr(size_t mat, int q, int r, cplx& imm) const {
        return refl_addr(a + mat * (size_t)n * n, n, i0 + q, r, imm);
    }
};

// Gram matrices of all blocks of bs reflectors in one batched GEMM: batch index z = mat * nblk
// + j; A(q, r) = conj(v_{bs j+q}[r]), B(r, l) = v_{bs j+l}[r].
template <class C>
struct OpBlkReflH {
    static constexpr bool RFAST = false;
    const C* a;
    int n, nblk, bs;
    __device__ __forceinline__ C elem(size_t z, int q, int r) const {
        C v = refl_entry(a + (z / nblk) * (size_t)n * n, n, (int)(z % nblk) * bs + q, r);
        v.y = -v.y;
        return v;
    }
    static constexpr bool CONJ = true;
    __device__ __forceinline__ const C* addr(size_t z, int q, int r, cplx& imm) const {
        return refl_addr(a + (z / nblk) * (size_t)n * n, n, (int)(z % nblk) * bs + q, r, imm);
    }
};
template <class C>
struct OpBlkRefl {
    static constexpr bool KFAST = true;
    const C* a;
    int n, nblk, bs;
    __device__ __forceinline__ C elem(size_t z, int r, int l) const {
        return refl_entry(a + (z / nblk) * (size_t)n * n, n, (int)(z % nblk) * bs + l, r);
    }
    static constexpr bool CONJ = false;
    __device__ __forceinline__ const C* addr(size_t z, int r, int l, cplx& imm) const {
        return refl_addr(a + (z / nblk) * (size_t)n * n, n, (int)(z % nblk) * bs + l, r, imm);
    }
};

// Complete a Hermitian matrix stored in the upper triangle (column-major, 'U') in place:
// lower triangle = conjugate of the upper, imaginary part of the diagonal zeroed.  Tiles of
// 32 x 32 through shared memory, both sides coalesced; grid (n/32, n/32, matrices), only
// tiles on or below the diagonal work.  Reads (strict upper) and writes (strict lower and
// diagonal) never overlap.
__global__ void k_herm_fill(cplx* __restrict__ A, int n) {
    __shared__ cplx tile[32][33];
    const int cb = blockIdx.x, rb = blockIdx.y;   // output tile: rows rb, columns cb
    if (rb < cb) return;
    cplx* a = A + (size_t)blockIdx.z * n * n;
    const int tx = threadIdx.x, ty = threadIdx.y;   // 32 x 8
    // input: upper entries (c, r) at a[r*n + c] for r in block rb, c in block cb
    for (int j = ty; j < 32; j += 8) {
        const int r = rb * 32 + j, c = cb * 32 + tx;
        if (r < n && c < n && c < r) tile[j][tx] = a[(size_t)r * n + c];
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8) {
        const int c = cb * 32 + j, r = rb * 32 + tx;
        if (r < n && c < n) {
            if (r > c) a[(size_t)c * n + r] = cconj(tile[tx][j]);
            else if (r == c) a[(size_t)c * n + r].y = 0.0;
        }
    }
}

// Epilogues
template <class C>
struct EpStore {   // P(r, c) = acc, column-major P with leading dimension ld
    C* p;
    int ld;
    size_t stride;
    __device__ __forceinline__ bool skip(int, int, int) const { return false; }
    __device__ __forceinline__ void store(size_t mat, int r, int c, C acc) const {
        p[mat * stride + (size_t)c * ld + r] = acc;
    }
};
template <class C>
struct EpSub {     // X(r, c) -= acc
    C* x;
    int n;
    __device__ __forceinline__ bool skip(int, int, int) const { return false; }
    __device__ __forceinline__ void store(size_t mat, int r, int c, C acc) const {
        C* q = x + mat * (size_t)n * n + (size_t)c * n + r;
        *q = csub(*q, acc);
    }
    // the GEMM engines prefetch X(r, c) (the DMMA engine into shared memory, the tcgen05
    // engine into registers) and pass it back as `old`
    __device__ __forceinline__ const C* pre_src(size_t mat, int r, int c) const {
        return x + mat * (size_t)n * n + (size_t)c * n + r;
    }
    __device__ __forceinline__ void store_pre(size_t mat, int r, int c, C acc, C old) const {
        x[mat * (size_t)n * n + (size_t)c * n + r] = csub(old, acc);
    }
};

// ------------------------------------------------------------- blocked k_hetrd (large n)
// For large orders the reduction runs in panels of pw (16 or 32) columns (LAPACK zlatrd + zher2k,
// uplo='U', restated): k_hetrd_panel_c reduces columns m-1 .. m-pw of the leading m x m
// block one CTA per matrix, keeping each column's reflector v and its w = tau A' v - ...
// in the panel buffers V, W instead of updating the leading block: column c is first
// brought up to date with the panel's earlier pairs, its matrix-vector product reads the
// leading c x c block as stored (read only) and is corrected by the same pairs.  The
// rank-2*pw update A -= V W^H + W V^H of the remaining leading block then runs as a GEMM
// over all SMs (launch_zgemm, EpHer2k), and the last block (order <= HT_TAIL) is reduced by
// k_hetrd.  D, E, TAU and the reflector storage are those of the unblocked reduction.
// Panel width: in double precision 32 columns from order HP_W_WIDE_MIN (at n = 3000 the
// rank-64 updates save 17 % of the update time, the panels cost the same), 16 below (measured
// faster than 8, 12, 24 and 32 at orders 256-1000).  Single precision keeps 16: with 32 the
// panel folds up to 31 pairs into each column in FP32, and two refinement steps then left an
// orthogonality defect of 2.6e-10 at n = 1600 (1e-12 with 16), for a 3 % saving.  Shared
// memory and the pair storage are laid out for the plan's width; HP_W_MAX bounds it.
static constexpr int HP_W_MAX = 32;
static constexpr int HP_W_WIDE_MIN = 1024;
static constexpr int HT_TAIL = 64;   // order below which the unblocked kernel finishes
static constexpr int HT_BLOCKED_MIN = 256;   // orders from which the blocked reduction runs
// Orders from which divide and conquer is the built-in tridiagonal solver.  Bisection is the faster
// one up to order ~2000 (order 640, 289 matrices 5.5 ms against 16.2; order 1200, 148 matrices 14.4
// against 37.4; order 2000, 25 matrices 25 against 33), but leaves its vectors orthogonal to 1e-13
// .. 7e-13 at orders 640 to 2000 where divide and conquer's are to 4e-15 .. 8e-15; callers who
// want the speed pin it (rlmb_set_tridiag_solver).
static constexpr int DC_DEFAULT_MIN = 600;
// Orders up to which k_jacobi is the built-in solver: of the batched eigensolver (part of its
// documented behaviour, and of the phases its callers' vectors come with), and of the mesh solves,
// whose results are gauge invariant and which take the faster one (8,192 matrices: order 10
// 0.29 ms against the Householder path's 0.40, order 12 0.40 against 0.45, order 13 0.54 against
// 0.48, order 16, 8,450 matrices, 0.85 against 0.55; 81 matrices of order 12 0.105 against 0.087).
// Up to JAC_DEFAULT_MAX the mixed mode's mesh solves take the double-precision path too: it is the
// more accurate and the faster one (calls of 81 and 8,450 matrices: order 20, double precision,
// 0.17 and 1.06 ms; order 21, mixed, 0.38 and 6.5, double precision 0.18 and 1.11).
static constexpr int JAC_DEFAULT_MAX = 20;
static constexpr int JAC_MESH_MAX = 12;
static constexpr int QUEUE_NT_DEFAULT = 512;   // panel queue CTAs: 512 threads, one per SM
static constexpr int TUNE_MIN_N = 16;         // orders the autotuner tunes: TUNE_MIN_N .. TUNE_MAX_N
static constexpr int TUNE_MAX_N = 1024;

// p += A v for the Hermitian leading m x m block stored in the upper triangle of a
// (column-major, leading dimension ld; read only), v and p in shared memory.  Work is dealt
// to warps as strips of HV_W columns (dealt back and forth for balance); a lane holds one
// row of a 32-row block of the strip:
// its row contributions go to p[r] (shared atomics, once per block), its column
// contributions conj(A[r][c]) v[r] stay in registers for the whole strip and are reduced
// across the warp once at the end.  Interior blocks (entirely above the diagonal and inside
// the matrix) run without predicates.
// Strip width: 8 columns in double precision, 16 in single precision, so that a lane has the
// same bytes of loads in flight (128) in both modes: the product streams the leading block
// from memory and is bound by the loads each SM keeps in flight, not by its arithmetic.
template <class C>
__host__ __device__ constexpr int hv_width() { return sizeof(C) == 8 ? 16 : 8; }
template <int NT, class C>
__device__ __forceinline__ void hemv_upper(const C* __restrict__ a, int ld, int m, const C* __restrict__ v,
                                           C* p) {
    constexpr int HV_W = hv_width<C>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = NT / 32;
    const int nstrips = (m + HV_W - 1) / HV_W;
    // strip s holds s*HV_W/32 + 1 row blocks: deal them back and forth (warp w takes strips
    // w, 2NW-1-w, 2NW+w, ...) so that every warp gets a similar amount of work
    for (int base = 0; base < nstrips; base += NW) {
        const int s = ((base / NW) & 1) ? base + NW - 1 - warp : base + warp;
        if (s >= nstrips) continue;
        const int c0 = s * HV_W;
        C vc[HV_W], e[HV_W];
#pragma unroll
        for (int j = 0; j < HV_W; ++j) {
            vc[j] = c0 + j < m ? v[c0 + j] : cz<C>();
            e[j] = cz<C>();
        }
        const C* colp = a + (size_t)c0 * ld;
        const int rend = min(c0 + HV_W, m);   // rows that meet the strip on or above the diagonal
        const bool full = c0 + HV_W <= m;
#pragma unroll 1
        for (int r0 = 0; r0 < rend; r0 += 32) {
            const int r = r0 + lane;
            const bool interior = full && r0 + 32 <= c0;
            C x[HV_W];
            if (interior) {
#pragma unroll
                for (int j = 0; j < HV_W; ++j) x[j] = colp[(size_t)j * ld + r];
            } else {
#pragma unroll
                for (int j = 0; j < HV_W; ++j) {
                    const int cc = c0 + j;
                    x[j] = (cc < m && r <= cc) ? colp[(size_t)j * ld + r] : cz<C>();
                }
            }
            const C vr = r < m ? v[r] : cz<C>();
            C rowacc = cz<C>();
#pragma unroll
            for (int j = 0; j < HV_W; ++j) {
                if (interior || r < c0 + j) {
                    cfma(rowacc, x[j], vc[j]);
                    cfmac(e[j], x[j], vr);
                } else if (r == c0 + j) {
                    rowacc = cadd(rowacc, cscale(vc[j], x[j].x));
                }
            }
            if (r < rend) smem_atomic_add(&p[r], rowacc);
        }
        // column sums: lane l ends with the sum over the warp of e[l & (HV_W - 1)]
#pragma unroll
        for (int mask = 16; mask >= HV_W; mask >>= 1)
#pragma unroll
            for (int j = 0; j < HV_W; ++j) e[j] = cadd(e[j], shfl_xor(e[j], mask));
#pragma unroll
        for (int sh = HV_W / 2; sh >= 1; sh >>= 1) {
            const bool up = (lane & sh) != 0;
#pragma unroll
            for (int j = 0; j < sh; ++j) {
                const C send = up ? e[j] : e[j + sh];
                const C keep = up ? e[j + sh] : e[j];
                e[j] = cadd(keep, shfl_xor(send, sh));
            }
        }
        if (lane < HV_W && c0 + lane < m) smem_atomic_add(&p[c0 + lane], e[0]);
    }
}

// Loads of the panel pairs V, W: around L1 (ld.global.cg), other CTAs wrote them during the same
// launch.
template <class C>
__device__ __forceinline__ C pv_ld(const C* p) {
    return __ldcg(p);
}

// Column j of the panel (column c = m - 1 - j of the leading m x m block) of matrix mat, by
// the NT threads of one CTA; vn, pn, coef, red: the CTA's shared work arrays.
template <int NT, class R>
__device__ __forceinline__ void panel_column(typename Cx<R>::T* __restrict__ A, double* __restrict__ D,
                                             double* __restrict__ E, typename Cx<R>::T* __restrict__ TAU,
                                             typename Cx<R>::T* __restrict__ PV, typename Cx<R>::T* __restrict__ PW,
                                             int n, int m, size_t mat, int j, int pw, typename Cx<R>::T* vn,
                                             typename Cx<R>::T* pn, typename Cx<R>::T* coef, R* red) {
    typedef typename Cx<R>::T C;
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    GlobalStore<C> gs{A + mat * (size_t)n * n, n};
    double* dd = D + mat * n;
    double* ee = E + mat * n;
    C* tt = TAU + mat * n;
    C* V = PV + mat * (size_t)pw * n;   // pair q at V + q*n, W + q*n
    C* W = PW + mat * (size_t)pw * n;
    if (m == n && j == 0 && tid == 0) {
        ee[n - 1] = 0.0;
        tt[n - 1] = cz<C>();
    }
    const int c = m - 1 - j;
    // (1) column c brought up to date with the panel's pairs q < j
    R part = 0;
    for (int r = tid; r <= c; r += NT) {
        C x = *gs.at(r, c);
        for (int q = 0; q < j; ++q) {
            const C* vq = V + (size_t)q * n;
            const C* wq = W + (size_t)q * n;
            C u = cmul(pv_ld(vq + r), cconj(pv_ld(wq + c)));
            cfma(u, pv_ld(wq + r), cconj(pv_ld(vq + c)));
            x = csub(x, u);
        }
        if (r == c) x.y = 0;
        vn[r] = x;
        if (r < c - 1) part += cabs2(x);
        if (r < c) pn[r] = cz<C>();
    }
    const R xn2 = block_sum<NT>(part, red);
    // (2) reflector of step c-1: alpha = A'[c-1][c], x = A'[0..c-2][c]
    R beta;
    C tau, scal;
    reflector(vn[c - 1], xn2, beta, tau, scal);
    const bool act = !(tau.x == 0 && tau.y == 0);
    __syncthreads();
    if (tid == 0) dd[c] = vn[c].x;
    for (int r = tid; r < c - 1; r += NT) {
        const C x = act ? cmul(scal, vn[r]) : vn[r];
        vn[r] = x;
        *gs.at(r, c) = x;
    }
    if (tid == 0) {
        vn[c - 1] = cm<C>(1, 0);
        *gs.at(c - 1, c) = cm<C>(beta, 0);
        ee[c - 1] = beta;
        tt[c - 1] = tau;
    }
    __syncthreads();
    // (3) pn = A v over the stored leading c x c block (read only)
    if (act) hemv_upper<NT>(gs.a, n, c, vn, pn);
    // (4) w_q^H v (even slots) and v_q^H v (odd slots) for q < j
    for (int t2 = warp; t2 < 2 * j; t2 += NW) {
        const int q = t2 >> 1;
        const C* y = (t2 & 1) ? V + (size_t)q * n : W + (size_t)q * n;
        C sd = cz<C>();
        for (int r = lane; r < c; r += 32) cfmac(sd, pv_ld(y + r), vn[r]);
        sd = warp_sum(sd);
        if (lane == 0) coef[t2] = sd;
    }
    __syncthreads();
    // (5) x = tau (pn - sum_q V_q (w_q^H v) + W_q (v_q^H v)); w = x - tau/2 (x^H v) v
    C dpart = cz<C>();
    for (int r = tid; r < c; r += NT) {
        C x = pn[r];
        for (int q = 0; q < j; ++q) {
            C u = cmul(pv_ld(V + (size_t)q * n + r), coef[2 * q]);
            cfma(u, pv_ld(W + (size_t)q * n + r), coef[2 * q + 1]);
            x = csub(x, u);
        }
        x = cmul(tau, x);
        pn[r] = x;
        cfmac(dpart, x, vn[r]);
    }
    const C xv = block_sum_c<NT>(dpart, red);
    const C al = cscale(cmul(tau, xv), (R)-0.5);
    C* vj = V + (size_t)j * n;
    C* wj = W + (size_t)j * n;
    for (int r = tid; r < c; r += NT) {
        vj[r] = vn[r];
        wj[r] = act ? cadd(pn[r], cmul(al, vn[r])) : cz<C>();
    }
    __syncthreads();
}

// Shared work arrays of the panel kernels: vn [m] (column / reflector), pn [m] (A' v
// accumulator), coef [2*HP_W_MAX] (w_q^H v, v_q^H v), red [2*warps].
template <int NT, class R>
__host__ __device__ constexpr size_t panel_smem(int m) {
    return (2 * (size_t)m + 2 * HP_W_MAX) * sizeof(typename Cx<R>::T) + 2 * (NT / 32) * sizeof(R);
}

// The panel for chunks of more matrices than SMs (see panel_waves_full; and for vectors too long for
// k_hetrd_panel_c's rings, see tridiagonalise): one resident CTA of NT
// threads per SM (grid <= SMs) takes units (matrix, column) from a queue, unit u = claim - base = matrix
// u % nb, column u / nb, so that every SM keeps NT threads of loads in flight whatever the
// number of matrices (one CTA per matrix would leave SMs with a single CTA when the chunk has
// between one and two matrices per SM).  Column j of a matrix needs column j - 1 (its panel
// pair): q[2 + mat] counts the columns of each matrix completed in the chunk; a unit waits
// for done = col0 + j, a wait bounded by TC_WAIT_NS that sets the abort flag q[1] (and counts
// in g_tc_fault) when it runs out.  The claims of a launch end with one failed claim per CTA,
// so launch k's units start at base = k * (nb * pw + grid).  Units are claimed in order and
// wait only on earlier claims, which CTAs already running hold: no wait depends on a CTA
// that has not started.
template <int NT, class R>
__global__ void __launch_bounds__(NT, NT >= 512 ? 1 : 2)
k_hetrd_panel_q(typename Cx<R>::T* __restrict__ A, double* __restrict__ D, double* __restrict__ E,
                typename Cx<R>::T* __restrict__ TAU, typename Cx<R>::T* __restrict__ PV,
                typename Cx<R>::T* __restrict__ PW, int n, int m, int pw, int nb, int* q, long long base, int col0,
                int* __restrict__ info) {
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* vn = reinterpret_cast<C*>(smem_raw);
    C* pn = vn + m;
    C* coef = pn + m;
    R* red = reinterpret_cast<R*>(coef + 2 * HP_W_MAX);
    __shared__ long long s_unit;
    __shared__ int s_go;
    const int tid = threadIdx.x;
    const long long units = (long long)nb * pw;
    for (;;) {
        if (tid == 0) {
            long long u = (long long)atomicAdd(reinterpret_cast<unsigned long long*>(q + 4), 1ull) - base;
            if (*(volatile int*)(q + 1)) u = units;   // aborted: stop claiming work
            s_unit = u;
            s_go = 1;
            if (u < units && u >= nb) {   // column j > 0: wait for column j - 1 of the matrix
                const int mat = (int)(u % nb), j = (int)(u / nb);
                const int* dp = q + 8 + mat;
                int v;
                asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(dp) : "memory");
                if (v < col0 + j) {
                    const unsigned long long t0 = tc_ns();
                    for (;;) {
                        __nanosleep(64);
                        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(dp) : "memory");
                        if (v >= col0 + j) break;
                        if (*(volatile int*)(q + 1) || tc_ns() - t0 > TC_WAIT_NS) {
                            if (atomicExch(q + 1, 1) == 0) atomicAdd(&g_tc_fault, 1);
                            if (info) info[mat] = -1;
                            s_go = 0;
                            break;
                        }
                    }
                }
            }
        }
        __syncthreads();
        const long long u = s_unit;
        const int go = s_go;
        __syncthreads();
        if (u >= units || !go) break;
        __threadfence();
        const int mat = (int)(u % nb), j = (int)(u / nb);
        panel_column<NT, R>(A, D, E, TAU, PV, PW, n, m, mat, j, pw, vn, pn, coef, red);
        // every thread's writes of the column, then the release of the column count
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            const int v = col0 + j + 1;
            int* dp = q + 8 + mat;
            asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(dp), "r"(v) : "memory");
        }
    }
}

// ---- the panel by a cluster of CTAs per matrix
// barrier of the cluster (or of the CTA, P = 1): orders global and (distributed) shared memory
__device__ __forceinline__ void panel_sync(int P) {
    if (P == 1) {
        __syncthreads();
    } else {
        cluster_arrive();
        cluster_wait();
    }
}
// the address of this CTA's shared variable p in CTA `rank` of the cluster
template <class T>
__device__ __forceinline__ T* panel_peer(T* p, int rank, int P) {
    if (P == 1) return p;
    T* q;
    asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(rank));
    return q;
}

// p += A v for the Hermitian leading m x m block stored in the upper triangle of a
// (column-major, leading dimension ld; read only), dealt over the GW = P * warps warps of a
// cluster (this warp: gw), each CTA summing into its own p (shared).  A unit is a segment of
// seg 32-row blocks of a strip of HU_W columns: segment g meets the strips from 32 g seg / HU_W
// on, and the units are counted off segment by segment, so that every warp gets the same
// number within one.  A block is taken in four quarters of 4 columns, lane (lr = lane % 8,
// lc = lane / 8) holding rows lr + 8 i (i < 4) and column lc of each: the cross-lane sums are
// then over 4 lanes per row (three exchanges and one shared add per 512 entries) and over 8
// lanes per column, once per unit.  The entries come through shared memory by cp.async, every
// lane copying what it will read itself (no synchronisation): four quarters per warp, one
// being multiplied while the next three are on their way, whatever the unit they belong to.
static constexpr int HU_W = 16;
static constexpr int HU_RING = 4 * 32 * 4;   // entries of a warp's ring: quarters x lanes x columns
template <class C>
struct HemvPos {
    int u, g, c0, r0, r1;   // unit counted from segment g on, its strip, block and last row
    bool ok, inside;        // a block; wholly above the diagonal and in the matrix
    const C* src;           // this lane's first entry of the block
    // the first unit at or after u counted from segment g on
    __device__ __forceinline__ void unit(const C* a, int ld, int m, int seg) {
        const int lane = threadIdx.x & 31, nstrips = (m + HU_W - 1) / HU_W;
        for (;; ++g) {
            const int s0 = g * seg * (32 / HU_W), cnt = nstrips - s0;
            if (cnt <= 0) {
                ok = false;
                return;
            }
            if (u < cnt) {
                c0 = (s0 + u) * HU_W;
                r0 = g * seg * 32;
                r1 = min(min(c0 + HU_W, m), (g + 1) * seg * 32);   // rows on or above the diagonal
                ok = true;
                inside = c0 + HU_W <= m && r0 + 32 <= c0;
                src = a + (size_t)(c0 + (lane >> 3)) * ld + r0 + (lane & 7);
                return;
            }
            u -= cnt;
        }
    }
};
template <int I>
__device__ __forceinline__ void hemv_copy(unsigned dst, const cplx* src) {
    asm volatile("cp.async.cg.shared.global [%0+%2], [%1+%3], 16;\n" ::"r"(dst), "l"(src), "n"(I * 32 * 16), "n"(I * 8 * 16) : "memory");
}
template <int I>
__device__ __forceinline__ void hemv_copy(unsigned dst, const cplxf* src) {
    asm volatile("cp.async.ca.shared.global [%0+%2], [%1+%3], 8;\n" ::"r"(dst), "l"(src), "n"(I * 32 * 8), "n"(I * 8 * 8) : "memory");
}
// Quarter q of block t (src: its entries of this lane) into the lane's ring slots at dst.
template <class C>
__device__ __forceinline__ void hemv_fetch(const C* __restrict__ a, int m, const HemvPos<C>& t, int q, const C* src,
                                           unsigned dst) {
    if (t.inside) {
        hemv_copy<0>(dst, src);
        hemv_copy<1>(dst, src);
        hemv_copy<2>(dst, src);
        hemv_copy<3>(dst, src);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int r = t.r0 + (lane & 7), c = t.c0 + 4 * q + (lane >> 3);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int n = c < m && r + 8 * i <= c ? (int)sizeof(C) : 0;   // outside: zeros
        const C* s = n ? src + 8 * i : a;
        if constexpr (sizeof(C) == 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + i * 32 * 16), "l"(s), "r"(n) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst + i * 32 * 8), "l"(s), "r"(n) : "memory");
    }
}
// The first block's four quarters on their way (one group each).
template <class C>
__device__ __forceinline__ HemvPos<C> hemv_begin(const C* __restrict__ a, int ld, int m, int gw, int seg, C* ring) {
    HemvPos<C> t{};
    t.u = gw;
    t.unit(a, ld, m, seg);
    const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + (threadIdx.x & 31));
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (t.ok) hemv_fetch(a, m, t, q, t.src + (size_t)(4 * q) * ld, dst + q * 128 * (int)sizeof(C));
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    return t;
}
// The product from position t (hemv_begin) on; returns this lane's share of v^H A v.  v and p
// are readable up to 32 entries beyond m (entries of A there are 0).
template <class C, class R>
__device__ __forceinline__ R hemv_units(const C* __restrict__ a, int ld, int m, const C* __restrict__ v, C* p,
                                        HemvPos<C> t, int GW, int seg, C* ring) {
    const int lane = threadIdx.x & 31, lr = lane & 7, lc = lane >> 3;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + lane);
    const size_t qstep = (size_t)4 * ld;
    R quad = 0;
    C es[4], vc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) es[j] = vc[j] = cz<C>();
    bool first = true;   // block of its unit
#pragma unroll 1
    while (t.ok) {
        if (first) {
            const C* vp = v + t.c0 + lc;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                vc[j] = vp[4 * j];
                es[j] = cz<C>();
            }
        }
        HemvPos<C> nx = t;
        nx.r0 += 32;
        nx.src += 32;
        const bool last = nx.r0 >= t.r1;
        if (last) {
            nx.u += GW;
            nx.unit(a, ld, m, seg);
        } else {
            nx.inside = t.inside && nx.r0 + 32 <= t.c0;
        }
        C rs[4], vr[4];
        const C* vp = v + t.r0 + lr;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            rs[i] = cz<C>();
            vr[i] = vp[8 * i];
        }
        const C* src = nx.src;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            asm volatile("cp.async.wait_group 3;\n" ::: "memory");
            C x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = ring[q * 128 + i * 32 + lane];
            if (!t.inside) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (t.r0 + lr + 8 * i == t.c0 + lc + 4 * q) {   // the diagonal: real, counted once
                        const C d = cscale(vc[q], x[i].x);
                        rs[i] = cadd(rs[i], d);
                        quad -= vr[i].x * d.x + vr[i].y * d.y;
                        x[i] = cz<C>();
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                cfma(rs[i], x[i], vc[q]);
                cfmac(es[q], x[i], vr[i]);
            }
            if (nx.ok) hemv_fetch(a, m, nx, q, src, dst + q * 128 * (int)sizeof(C));
            src += qstep;
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) quad += 2 * (vr[i].x * rs[i].x + vr[i].y * rs[i].y);
        {   // row sums over the four lanes of a row: lane ends with row r0 + lane
            const bool u1 = (lane & 16) != 0, u0 = (lane & 8) != 0;
            C y[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const C send = u1 ? rs[i] : rs[i + 2], keep = u1 ? rs[i + 2] : rs[i];
                y[i] = cadd(keep, shfl_xor(send, 16));
            }
            const C send = u0 ? y[0] : y[1], keep = u0 ? y[1] : y[0];
            const C s = cadd(keep, shfl_xor(send, 8));
            if (t.inside || t.r0 + lane < min(t.c0 + HU_W, m)) smem_atomic_add(&p[t.r0 + lane], s);
        }
        if (last) {   // column sums over the eight lanes of a column: lane ends with column lc + 4 (lr / 2)
            const bool u2 = (lane & 4) != 0, u1 = (lane & 2) != 0;
            C y[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const C send = u2 ? es[j] : es[j + 2], keep = u2 ? es[j + 2] : es[j];
                y[j] = cadd(keep, shfl_xor(send, 4));
            }
            const C send = u1 ? y[0] : y[1], keep = u1 ? y[1] : y[0];
            C e = cadd(keep, shfl_xor(send, 2));
            e = cadd(e, shfl_xor(e, 1));
            const int c = t.c0 + lc + 4 * (lr >> 1);
            if ((lr & 1) == 0 && c < m) smem_atomic_add(&p[c], e);
        }
        first = last;
        t = nx;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    return quad;
}

static constexpr int PC_MAX = 16;   // CTAs per cluster
template <int NT, class R>
__host__ __device__ constexpr size_t panel_c_smem(int m, int P) {
    typedef typename Cx<R>::T C;
    return (2 * (size_t)(m + 32) + (NT / 32) * HU_RING + (size_t)P * 2 * HP_W_MAX + 4 * HP_W_MAX + 4) * sizeof(C) +
           2 * (size_t)P * (NT / 32) * sizeof(R);
}

// The panel of one matrix by a cluster of P CTAs (blockIdx.x = matrix * P + rank): the leading
// block's product is dealt over all the cluster's warps, the rows of the column vectors over
// its CTAs in blocks of 8 (a warp takes 8 rows, its four 8-lane groups every fourth pair).  Per
// column two cluster barriers:
//   rows   w of the previous column, and with it the next column brought up to date, in one
//          pass over the panel pairs; every CTA receives the column and its norm's parts
//   -- barrier --   reflector (each CTA redundantly), A v and the pairs' products with v
//   -- barrier --   sums of the CTAs' parts over distributed shared memory
// x^H v for w = x - tau/2 (x^H v) v comes from v^H A v and the pairs' products, so that it
// needs no barrier of its own.
// Bound: the stream of the leading block (25 matrices of order 2500, clusters of 5: 198 to 204 ms
// for 1.04 TB, 5.2 TB/s), with the instructions of the product close behind (two thirds of the time
// remained with the loads taken out).  One CTA per matrix, 25 SMs at work, took 923 ms, and 957 at
// order 3000 in single precision, now 208.
// ONE: one CTA per matrix, no cluster.
template <int NT, class R, bool ONE>
__global__ void __launch_bounds__(NT, NT > 256 ? 1 : 512 / NT)
k_hetrd_panel_c(typename Cx<R>::T* __restrict__ A, double* __restrict__ D, double* __restrict__ E,
                typename Cx<R>::T* __restrict__ TAU, typename Cx<R>::T* __restrict__ PV,
                typename Cx<R>::T* __restrict__ PW, int n, int m, int pw, int Pr) {
    typedef typename Cx<R>::T C;
    constexpr int NW = NT / 32;
    const int P = ONE ? 1 : Pr;
    if (!ONE) cluster_arrive();   // (the wait stands before the first access to a peer's shared memory)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* ring = reinterpret_cast<C*>(smem_raw) + (threadIdx.x >> 5) * HU_RING;   // this warp's staging
    C* v = reinterpret_cast<C*>(smem_raw) + NW * HU_RING;   // [m] column / reflector
    C* pn = v + m + 32;                           // [m] this CTA's part of A v
    C* coefp = pn + m + 32;                            // [P][2 * HP_W_MAX] the CTAs' parts of w_q^H v, v_q^H v
    C* coef = coefp + (size_t)P * 2 * HP_W_MAX;   // [2 * HP_W_MAX] their sums
    C* rowc = coef + 2 * HP_W_MAX;                // [2 * HP_W_MAX] V_q, W_q at the next column's index
    C* scal_s = rowc + 2 * HP_W_MAX;              // [0..1] alpha by parity, [2] al, [3] w at the next column's index
    R* quadp = reinterpret_cast<R*>(scal_s + 4);  // [P * NW] parts of v^H A v
    R* normp = quadp + (size_t)P * NW;            // [P * NW] parts of the column's norm
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t mat = blockIdx.x / P;
    const int rank = ONE ? 0 : (int)(blockIdx.x % P);
    C* a = A + mat * (size_t)n * n;
    double* dd = D + mat * n;
    double* ee = E + mat * n;
    C* tt = TAU + mat * n;
    C* V = PV + mat * (size_t)pw * n;
    C* W = PW + mat * (size_t)pw * n;
    const int rl = lane & 7, ql = lane >> 3;   // row of the block of 8, pair group
    if (m == n && rank == 0 && tid == 0) {
        ee[n - 1] = 0.0;
        tt[n - 1] = cz<C>();
    }
    C tau = cz<C>();
    bool act = false;
    HemvPos<C> pos{};
    int seg = 1;
    for (int r = m + tid; r < m + 32; r += NT) v[r] = cz<C>();   // (read, times zero, by the product's last blocks)
    if (!ONE) cluster_wait();   // every CTA of the cluster has started: step -1 writes to its peers
    for (int j = -1; j < pw; ++j) {
        const int c = m - 1 - j;   // column of step j; the pass below finishes step j and starts step j + 1
        if (j >= 0) {
            panel_sync(P);
            // reflector of step c-1 from the column's norm and alpha = column[c-1]
            R xn2 = 0;
            for (int i = lane; i < P * NW; i += 32) xn2 += normp[i];
            xn2 = warp_sum(xn2);
            R beta;
            C scal;
            reflector(scal_s[j & 1], xn2, beta, tau, scal);
            act = !(tau.x == 0 && tau.y == 0);
            // (each CTA the whole vector; to memory its own rows)
            for (int r = tid; r < c; r += NT) {
                const C x = r == c - 1 ? cm<C>(1, 0) : act ? cmul(scal, v[r]) : v[r];
                v[r] = x;
                pn[r] = cz<C>();
                if (ONE) {
                    a[(size_t)c * n + r] = r == c - 1 ? cm<C>(beta, 0) : x;
                    V[(size_t)j * n + r] = x;
                }
            }
            if (rank == 0 && tid == 0) {
                ee[c - 1] = beta;
                tt[c - 1] = tau;
            }
            // the pairs at row c - 1, for the next column
            C vq = cz<C>(), wq = cz<C>();
            if (warp == 0 && lane < j) {
                vq = __ldcg(V + (size_t)lane * n + c - 1);
                wq = __ldcg(W + (size_t)lane * n + c - 1);
            }
            __syncthreads();
            if (!ONE)
                for (int r = ((tid >> 3) * P + rank) * 8 + (tid & 7); r < c; r += NT * P) {
                    const C x = v[r];
                    a[(size_t)c * n + r] = r == c - 1 ? cm<C>(beta, 0) : x;
                    V[(size_t)j * n + r] = x;
                }
            R quad = 0;
            if (act) quad = hemv_units<C, R>(a, n, c, v, pn, pos, P * NW, seg, ring);
            else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            quad = warp_sum(quad);
            if (lane < P) panel_peer(quadp, lane, P)[rank * NW + warp] = quad;
            // this CTA's rows of w_q^H v (even slots) and v_q^H v (odd slots), two pairs per warp at
            // a time: their four sums cross the warp together, each ending in eight lanes
            for (int q0 = 2 * warp; q0 < j; q0 += 2 * NW) {
                const C *w0 = W + (size_t)q0 * n, *v0 = V + (size_t)q0 * n;
                const size_t step = q0 + 1 < j ? n : 0;   // (a last pair alone is summed twice)
                C sd[4] = {cz<C>(), cz<C>(), cz<C>(), cz<C>()};
#pragma unroll 2
                for (int r = ((lane >> 3) * P + rank) * 8 + (lane & 7); r < c; r += 32 * P) {
                    const C vr = v[r];
                    cfmac(sd[0], w0[r], vr);
                    cfmac(sd[1], v0[r], vr);
                    cfmac(sd[2], w0[step + r], vr);
                    cfmac(sd[3], v0[step + r], vr);
                }
                const bool u1 = (lane & 16) != 0, u0 = (lane & 8) != 0;
                C y[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) y[i] = cadd(u1 ? sd[i + 2] : sd[i], shfl_xor(u1 ? sd[i] : sd[i + 2], 16));
                C s = cadd(u0 ? y[1] : y[0], shfl_xor(u0 ? y[0] : y[1], 8));
                s = cadd(s, shfl_xor(s, 4));
                s = cadd(s, shfl_xor(s, 2));
                s = cadd(s, shfl_xor(s, 1));
                const int t2 = 2 * q0 + (lane >> 3);   // (an absent second pair's slots are not read)
                for (int k = lane & 7; k < P; k += 8) panel_peer(coefp, k, P)[rank * 2 * HP_W_MAX + t2] = s;
            }
            panel_sync(P);
            if (warp == 0) {
                C ca = cz<C>(), cb = cz<C>(), y = cz<C>();
                R q2 = 0;
                for (int i = lane; i < P * NW; i += 32) q2 += quadp[i];
                if (lane < j) {
                    for (int k = 0; k < P; ++k) {
                        ca = cadd(ca, coefp[k * 2 * HP_W_MAX + 2 * lane]);
                        cb = cadd(cb, coefp[k * 2 * HP_W_MAX + 2 * lane + 1]);
                    }
                    coef[2 * lane] = ca;
                    coef[2 * lane + 1] = cb;
                    rowc[2 * lane] = vq;
                    rowc[2 * lane + 1] = wq;
                    q2 -= 2 * (ca.x * cb.x + ca.y * cb.y);
                    cfma(y, vq, ca);
                    cfma(y, wq, cb);
                    y = cscale(y, (R)-1);
                }
                if (lane < P) y = cadd(y, panel_peer(pn, lane, P)[c - 1]);
                y = warp_sum(y);
                q2 = warp_sum(q2);
                if (lane == 0) {
                    // x = tau y, x^H v = conj(tau) (v^H y), al = -tau/2 x^H v = -|tau|^2/2 v^H y
                    const R al = (R)-0.5 * cabs2(tau) * q2;
                    C w = cmul(tau, y);
                    w.x += al;   // v[c-1] = 1
                    scal_s[2] = cm<C>(al, 0);
                    scal_s[3] = act ? w : cz<C>();
                }
            }
            __syncthreads();
        }
        // the next product's first entries on their way (the leading block does not change)
        const bool next = j + 1 < pw;
        if (next) {
            const int mc = c - 1, ns = (mc + HU_W - 1) / HU_W;
            const int blocks = ns * (ns + 2) / 4;   // 32-row blocks over all strips
            seg = min(max(blocks / (4 * P * NW), 1), 32);
            pos = hemv_begin(a, n, mc, warp * P + rank, seg, ring);
        }
        // rows: w_j, and the next column (index c - 1) brought up to date with the pairs 0 .. j
        const int cn = c - 1;
        const R al = j >= 0 ? scal_s[2].x : (R)0;
        const C wcn = j >= 0 ? scal_s[3] : cz<C>();
        R part = 0;
        const int top = j >= 0 ? cn : m - 1;   // (step -1: the first column as stored)
        const int col = j >= 0 ? cn : m - 1;
        for (int b = warp * P + rank; b * 8 <= top; b += NW * P) {
            const int r = b * 8 + rl;
            const bool in = r <= top;
            C x = cz<C>(), y = cz<C>(), s2 = cz<C>();
            if (in) {
                if (next && ql == 0) x = a[(size_t)col * n + r];
                if (j >= 0) {
                    for (int k = ql; k < P; k += 4) y = cadd(y, panel_peer(pn, k, P)[r]);
                    C s1 = cz<C>();
                    const C *vq = V + (size_t)ql * n + r, *wq = W + (size_t)ql * n + r;
                    const size_t step = (size_t)4 * n;
#pragma unroll 2
                    for (int q = ql; q < j; q += 4, vq += step, wq += step) {
                        const C vr = *vq, wr = *wq;
                        cfma(s1, vr, coef[2 * q]);
                        cfma(s1, wr, coef[2 * q + 1]);
                        cfma(s2, vr, cconj(rowc[2 * q + 1]));
                        cfma(s2, wr, cconj(rowc[2 * q]));
                    }
                    y = csub(y, s1);
                }
            }
            if (j >= 0) {
                x = csub(x, s2);
                y = cadd(y, shfl_xor(y, 8));
                y = cadd(y, shfl_xor(y, 16));
                x = cadd(x, shfl_xor(x, 8));
                x = cadd(x, shfl_xor(x, 16));
                if (in) {
                    const C vr = V[(size_t)j * n + r];
                    C w = cmul(tau, y);
                    w.x += al * vr.x;
                    w.y += al * vr.y;
                    if (!act) w = cz<C>();
                    if (ql == 0) W[(size_t)j * n + r] = w;
                    C u = cmul(vr, cconj(wcn));
                    u = cadd(u, w);   // conj(v[cn]) = 1
                    x = csub(x, u);
                }
            } else {
                x = cm<C>(__shfl_sync(0xffffffffu, x.x, rl), __shfl_sync(0xffffffffu, x.y, rl));
            }
            if (next && in) {
                if (r == col) x.y = 0;
                for (int k = ql; k < P; k += 4) {
                    panel_peer(v, k, P)[r] = x;
                    if (r == col - 1) panel_peer(scal_s, k, P)[(j + 1) & 1] = x;
                }
                if (ql == 0) {
                    if (r == col) dd[col] = x.x;
                    if (r < col - 1) part += cabs2(x);
                }
            }
        }
        if (next) {
            part = warp_sum(part);
            if (lane < P) panel_peer(normp, lane, P)[rank * NW + warp] = part;
        }
    }
    panel_sync(P);   // no CTA leaves while a peer may still read its shared memory
}

template <int NT, class R>
static cudaLaunchConfig_t panel_c_config(cudaLaunchAttribute* at, cudaStream_t st, int m, int nb, int P) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nb * P);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = panel_c_smem<NT, R>(m, P);
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = P;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}
template <int NT, class R>
static cudaError_t panel_c_attrs(int m, int P) {
    auto kern = k_hetrd_panel_c<NT, R, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)panel_c_smem<NT, R>(m, P));
    if (e == cudaSuccess && P > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}
template <int NT, class R>
static cudaError_t launch_panel_c(cudaStream_t st, typename Cx<R>::T* A, double* D, double* E, typename Cx<R>::T* TAU,
                                  typename Cx<R>::T* PV, typename Cx<R>::T* PW, int n, int m, int pw, int nb, int P) {
    const cudaError_t e = panel_c_attrs<NT, R>(m, P);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = panel_c_config<NT, R>(at, st, m, nb, P);
    return cudaLaunchKernelEx(&cfg, k_hetrd_panel_c<NT, R, false>, A, D, E, TAU, PV, PW, n, m, pw, P);
}

// Shape of the cluster panel for a chunk of nb matrices, P = 0 where one CTA per matrix (or the
// panel queue) is the better one.  The clusters of one launch should all run at once: of the
// shapes whose nb clusters fit the device together the one with the most threads per matrix is
// taken (measured best at orders 300 to 1000 with 1 to 81 matrices, wider CTAs winning ties),
// if that is at least 1.5 (below order 512: 2) times the 512 threads of one CTA per matrix:
// panels of order 300, double precision, 18 matrices 3.46 -> 2.63 ms, 36 3.47 -> 2.86, but 81
// 3.49 -> 3.71; of order 512 10.9 -> 5.9, 11.3 -> 6.9, 13.1 -> 10.9; of order 2500, 25 matrices,
// 923 -> 198.
struct PanelShape {
    int nt, P;
};
template <int NT, class R>
static void panel_shape_try(int m, int nb, PanelShape* best) {
    for (int P = PC_MAX; P >= 2; --P) {
        if (NT * P <= best->nt * best->P) return;
        if (panel_c_smem<NT, R>(m, P) > 227 * 1024) continue;
        int active = 0;
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = panel_c_config<NT, R>(at, 0, m, nb, P);
        if (panel_c_attrs<NT, R>(m, P) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, k_hetrd_panel_c<NT, R, false>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (active >= nb) *best = PanelShape{NT, P};
    }
}
template <class R>
static PanelShape panel_shape(int m, int nb) {
    PanelShape s{0, 0};
    if (nb > 148) return s;
    panel_shape_try<512, R>(m, nb, &s);
    panel_shape_try<384, R>(m, nb, &s);
    panel_shape_try<256, R>(m, nb, &s);
    if (s.nt * s.P < (m >= 512 ? 768 : 1024)) s.P = 0;
    return s;
}

// One CTA per matrix (k_hetrd_panel_c without a cluster): 512 threads, or 256 or 128 with two
// or four CTAs per SM, which between them keep the SM busier through each other's chains of
// small steps.  A wave of 148 k matrices takes about 1, 1.8 and 3.4 units of time for k = 1, 2
// and 4 (orders 256 to 640), the last one of several counts in part, but a second wave of one
// CTA per SM nearly whole: 149 matrices of order 400 take 21.1 ms with 512 threads and 18.2 with 256
// (the eigensolve), 200 23.3 and 20.6.  Panels in double
// precision, against a kernel with one row and 8 columns per lane and seven barriers per column:
// order 256, 592 matrices 9.64 -> 8.00 ms (128 threads), order 512, 592 matrices 51.3 -> 45.2
// (128), 296 matrices 25.8 -> 23.8 (256), order 1000, 100 matrices 78.4 -> 63.6 (512); in
// single precision order 256 7.59 -> 5.15, order 512 37.8 -> 28.9.
// Returns the threads (64 serve the orders whose vectors leave a ring for no more warps), 0 if
// none fits.  pinned: 512 or 256, or the next smaller that fits; 0: the rule.
template <class R>
static int panel_threads(int m, int nb, int pinned) {
    const size_t smem[4] = {panel_c_smem<512, R>(m, 1), panel_c_smem<256, R>(m, 1), panel_c_smem<128, R>(m, 1),
                            panel_c_smem<64, R>(m, 1)};
    const double unit[3] = {1.0, 1.8, 3.4};
    int best = 0;
    double best_cost = 0.0;
    for (int i = 0; i < 3; ++i) {
        const int nt = 512 >> i, per_sm = (int)std::min<size_t>((size_t)1 << i, (size_t)(228 * 1024) / (smem[i] + 1024));
        if (per_sm < 1 || smem[i] > 227 * 1024 || (pinned && nt > pinned)) continue;
        if (pinned) return nt;
        const double waves = (double)nb / (148.0 * per_sm);
        const double cost = (per_sm == 1 << i ? unit[i] : unit[i] / (1 << i) * per_sm * 1.3) *
                            (waves <= 1.0 ? 1.0 : std::max(waves + 0.35, 1.0 + 0.85 / per_sm));
        if (best == 0 || cost < best_cost) {
            best = nt;
            best_cost = cost;
        }
    }
    return best ? best : smem[3] <= 227 * 1024 ? 64 : 0;
}
// One CTA per matrix rather than the panel queue for more matrices than SMs: where two 256-thread
// CTAs fit an SM (order 1200 at most, above which the queue is even) and their waves of 296 are
// at least 80 % full, a single wave 60 %: eigensolves of 149 matrices of order 520 take 36.6 ms by
// the queue and 38.4 by 256 threads, 160 38.8 and 39.5, 180 43.0 and 41.8; of order 1100 273 and
// 290, 292 and 303, 325.5 and 324.5.  Panels of order 600, 592 matrices 101.6 -> 73.5 ms; of order
// 1000, 296 matrices 180.2 -> 144.8; but order 800, 300 matrices 102.5 -> 113.7.
template <class R>
static bool panel_waves_full(int m, int nb) {
    const int waves = (nb + 295) / 296;
    return m <= 1200 && panel_c_smem<256, R>(m, 1) <= 113 * 1024 && nb >= (waves == 1 ? 0.6 : 0.8) * 296 * waves;
}
template <int NT, class R>
static cudaError_t launch_panel_one(cudaStream_t st, typename Cx<R>::T* A, double* D, double* E, typename Cx<R>::T* TAU,
                                    typename Cx<R>::T* PV, typename Cx<R>::T* PW, int n, int m, int pw, int nb) {
    auto kern = k_hetrd_panel_c<NT, R, true>;
    const size_t smem = panel_c_smem<NT, R>(m, 1);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<nb, NT, smem, st>>>(A, D, E, TAU, PV, PW, n, m, pw, 1);
    return cudaGetLastError();
}

// [V | W] (r, k) and [W | V]^H (k, c) of a panel: the operands of A -= V W^H + W V^H.
template <class C, int w>
struct OpPanelA {
    static constexpr bool RFAST = true;
    const C* pv;
    const C* pw;
    int n;
    __device__ __forceinline__ C elem(size_t mat, int r, int k) const {
        const size_t o = mat * (size_t)w * n;
        return k < w ? pv[o + (size_t)k * n + r] : pw[o + (size_t)(k - w) * n + r];
    }
    static constexpr bool CONJ = false;
    __device__ __forceinline__ const C* addr(size_t mat, int r, int k, cplx&) const {
        return (k < w ? pv + (size_t)k * n : pw + (size_t)(k - w) * n) + mat * (size_t)w * n + r;
    }
};
template <class C, int w>
struct OpPanelB {
    static constexpr bool KFAST = false;
    const C* pv;
    const C* pw;
    int n;
    __device__ __forceinline__ C elem(size_t mat, int k, int c) const {
        const size_t o = mat * (size_t)w * n;
        return cconj(k < w ? pw[o + (size_t)k * n + c] : pv[o + (size_t)(k - w) * n + c]);
    }
    static constexpr bool CONJ = true;
    __device__ __forceinline__ const C* addr(size_t mat, int k, int c, cplx&) const {
        return (k < w ? pw + (size_t)k * n : pv + (size_t)(k - w) * n) + mat * (size_t)w * n + c;
    }
};
// A(r, c) -= acc on and above the diagonal (real diagonal); tiles below it are skipped.
template <class C>
struct EpHer2k {
    C* a;
    int n;
    __device__ __forceinline__ bool skip(int r0, int c0, int) const { return r0 > c0 + ZG_BN - 1; }
    __device__ __forceinline__ bool skip_tile(int r0, int c0, int, int cols) const { return r0 > c0 + cols - 1; }
    __device__ __forceinline__ void store(size_t mat, int r, int c, C acc) const {
        if (r > c) return;
        C* q = a + mat * (size_t)n * n + (size_t)c * n + r;
        C x = csub(*q, acc);
        if (r == c) x.y = 0;
        *q = x;
    }
    // the GEMM engines prefetch A(r, c) (on and above the diagonal) when the tile starts
    __device__ __forceinline__ const C* pre_src(size_t mat, int r, int c) const {
        return r > c ? nullptr : a + mat * (size_t)n * n + (size_t)c * n + r;
    }
    __device__ __forceinline__ void store_pre(size_t mat, int r, int c, C acc, C old) const {
        C x = csub(old, acc);
        if (r == c) x.y = 0;
        a[mat * (size_t)n * n + (size_t)c * n + r] = x;
    }
};

// The GEMMs of the reduction and back-transformation in the working precision C: double on
// the FP64 tensor path (DMMA engine, BM-row tiles), single precision (the mixed mode) on the
// tcgen05 tensor cores with split TF32 operands.
template <class C, int BM, class LA, class LB, class EP>
static cudaError_t launch_work_gemm(cudaStream_t st, const LA& la, const LB& lb, const EP& ep, int M, int N, int K,
                                    int nb) {
    if constexpr (std::is_same<C, cplxf>::value) return launch_zgemm_tc<C>(st, la, lb, ep, M, N, K, nb);
    else return launch_zgemm<C, BM>(st, la, lb, ep, M, N, K, nb);
}

// ------------------------------------------------- mixed mode: FP64 refinement kernels
// The mixed mode reduces and back-transforms in single precision (k_hetrd<.., float>,
// k_larft / k_ormtr or the blocked path on float), solves the tridiagonal in double
// (k_tridiag), then refines the eigenpairs (X, lambda) of H in double, in the manner of
// Ogita & Aishima (2018, "Iterative refinement for symmetric eigenvalue decomposition"),
// one or two steps:
//   R = H X - X diag(lambda)                            k_ref_resid     (double)
//   E = X^H R,  F_ij = E_ij / (lambda_j - lambda_i)     k_ref_coupling  (double, i != j)
//   F_jj = (1 - x_j^H x_j) / 2,
//   lambda_j += Re(x_j^H r_j) / x_j^H x_j               k_ref_diag      (double)
//   X <- X + X F                                        k_ref_update    (single product,
//                                                                        double sum)
// X F is a first-order correction of the size of the current error, so a single-precision
// product carries it; R, E and the diagonal need double.  Each step roughly squares the
// relative error of the vectors.
// Two neighbouring eigenpairs whose gap is within 8 x their residual norms ||r_j|| are not
// separated by the current vectors (first-order theory needs |x_i^H r_j| << gap), and for
// gaps below 2^-14 of the spectral radius the first-order correction cannot restore
// orthogonality to double precision (its error is ~ u ||H|| / gap; LAPACK's inverse
// iteration likewise re-orthogonalises eigenvalues closer than 1e-3 ||T||, dstein): chains
// of such gaps form clusters (k_ref_clusters).  Inside a cluster of at most RF_KMAX members the vectors are re-resolved
// by a Rayleigh-Ritz step on the cluster's subspace in double (k_ref_cluster_solve: S =
// X_C^H H X_C = E_CC + G_CC Lambda, G_CC = X_C^H X_C, S y = mu G y; k_ref_cluster_apply:
// X_C <- X_C Y, lambda_C <- mu).  Larger clusters, and any other pair whose gap is within
// 8 |E_ij|, are orthogonalised only, F_ij = -(x_i^H x_j)/2, and keep Rayleigh quotients.
static constexpr int RF_KMAX = 16;             // largest cluster resolved by Rayleigh-Ritz
static constexpr double RF_RES = 8.0;          // gap / residual ratio below which pairs cluster
static constexpr double RF_CLUSTER = 0x1p-14;  // relative gap below which pairs cluster

// R = H X - X diag(lambda): epilogue of the GEMM H X (H completed by k_herm_fill).
template <class XT>
struct EpResid {
    const XT* x;
    const double* w;
    cplx* res;
    int n;
    __device__ __forceinline__ bool skip(int, int, int) const { return false; }
    __device__ __forceinline__ void store(size_t mat, int r, int c, cplx acc) const {
        const size_t o = mat * (size_t)n * n + (size_t)c * n + r;
        const cplx xr = to_c64(x[o]);
        const double lam = w[mat * n + c];
        res[o] = mk(acc.x - lam * xr.x, acc.y - lam * xr.y);
    }
};

// R = H X - X diag(lambda) for a cyclic band matrix H of half-bandwidth o (H(r, k) = 0 unless
// the cyclic distance of r and k is at most o -- the rlm Hamiltonian's structure,
// rlm/hamiltonian_rlm_cpu.cpp:26-38), in double, with 32 + 2o <= n.  An output tile of 32 rows
// x 64 columns needs only the 32 + 2o rows k = r0 - o .. r0 + 31 + o (cyclic) of X: the tile's
// band rows of H, zero-padded to a dense 32 x (32 + 2o) block, times those rows of X, in
// chunks of 16.  Row r of H is read as the conjugate of column r (contiguous in k) of the
// Hermitian matrix stored in full.  Thread (tr, tc) computes rows 2 tr, 2 tr + 1 and columns
// tc + 16 j (j < 4) of the tile: 8 complex multiply-adds per 6 shared-memory loads.
template <class XT>
__global__ void __launch_bounds__(256)
k_ref_resid_band(const cplx* __restrict__ A, const XT* __restrict__ X, const double* __restrict__ W,
                 cplx* __restrict__ Res, int n, int o) {
    __shared__ cplx hs[16][32 + 1];   // hs[kk][rl] = H(r0 + rl, k(kk))
    __shared__ cplx xs[16][64 + 1];   // xs[kk][cl] = X(k(kk), c0 + cl)
    const int t = threadIdx.x, tr = t >> 4, tc = t & 15;
    const size_t mat = blockIdx.z;
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 64;
    const size_t nn = (size_t)n * n;
    const cplx* Am = A + mat * nn;
    const XT* Xm = X + mat * nn;
    const int span = 32 + 2 * o;   // k(kk) = (r0 - o + kk) mod n, kk < span
    cplx acc[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = mk(0, 0);
    for (int k0 = 0; k0 < span; k0 += 16) {
        {   // H band: (kk, rl) = (t % 16, t / 16 + 16 h)
            const int kk = t & 15;
            const int kg = k0 + kk;
            int k = r0 - o + kg;
            k = k < 0 ? k + n : (k >= n ? k - n : k);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int rl = (t >> 4) + 16 * h, r = r0 + rl;
                const int dist = kg - rl;   // k - r + o
                cplx v = mk(0, 0);
                if (kg < span && r < n && dist >= 0 && dist <= 2 * o) v = cconj(Am[(size_t)r * n + k]);
                hs[kk][rl] = v;
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int cl = (t >> 4) + 16 * h, c = c0 + cl;
                xs[kk][cl] = (kg < span && c < n) ? to_c64(Xm[(size_t)c * n + k]) : mk(0, 0);
            }
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            const cplx h0 = hs[kk][2 * tr], h1 = hs[kk][2 * tr + 1];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const cplx x = xs[kk][tc + 16 * j];
                cfma(acc[0][j], h0, x);
                cfma(acc[1][j], h1, x);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = c0 + tc + 16 * j;
        if (c >= n) continue;
        const double lam = W[mat * n + c];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = r0 + 2 * tr + i;
            if (r >= n) continue;
            const size_t off = mat * nn + (size_t)c * n + r;
            const cplx xr = to_c64(X[off]);
            Res[off] = mk(acc[i][j].x - lam * xr.x, acc[i][j].y - lam * xr.y);
        }
    }
}

// The same band product on the FP64 tensor path: operands of the DMMA engine (64-row output
// tiles) for R = H X - X diag(lambda) with a cyclic band H of half-width o, 64 + 2o <= n.  The
// tile of rows r0 = 64 blockIdx.x .. r0 + 63 needs only the columns k(kk) = (r0 - o + kk) mod n,
// kk < 64 + 2o, of H, which becomes the inner dimension:
//   A(r, kk) = H(r, k(kk)) where 0 <= kk - (r - r0) <= 2o, else 0 (read as the conjugate of
//              column r of the stored Hermitian H, contiguous in kk);
//   B(kk, c) = X(k(kk), c).
// 64 + 2o inner terms per output against 2o + 1 nonzero ones (1.29x at o = 110), on a pipe
// ~4x faster than the FP64 FMA of k_ref_resid_band.
static constexpr int RB_BM = 64;
struct OpBandA {
    static constexpr bool RFAST = false;
    const cplx* p;
    int n, o;
    __device__ __forceinline__ cplx elem(size_t mat, int r, int kk) const {
        const int r0 = r - r % RB_BM;
        const int dist = kk - (r - r0);
        if (dist < 0 || dist > 2 * o) return mk(0.0, 0.0);
        int k = r0 - o + kk;
        k = k < 0 ? k + n : (k >= n ? k - n : k);
        return cconj(p[mat * (size_t)n * n + (size_t)r * n + k]);
    }
    static constexpr bool CONJ = true;
    __device__ __forceinline__ const cplx* addr(size_t mat, int r, int kk, cplx&) const {
        const int r0 = r - r % RB_BM, dist = kk - (r - r0);
        if (dist < 0 || dist > 2 * o) return nullptr;   // (0)
        int k = r0 - o + kk;
        k = k < 0 ? k + n : (k >= n ? k - n : k);
        return p + mat * (size_t)n * n + (size_t)r * n + k;
    }
};
template <class XT>
struct OpBandB {
    static constexpr bool KFAST = true;
    const XT* p;
    int n, o;
    __device__ __forceinline__ cplx elem(size_t mat, int kk, int c) const {
        int k = (int)blockIdx.x * RB_BM - o + kk;   // the tile's r0 (the engine's row tile is RB_BM)
        k = k < 0 ? k + n : (k >= n ? k - n : k);
        return to_c64(p[mat * (size_t)n * n + (size_t)c * n + k]);
    }
    static constexpr bool CONJ = false;
    __device__ __forceinline__ const XT* addr(size_t mat, int kk, int c, cplx&) const {
        int k = (int)blockIdx.x * RB_BM - o + kk;
        k = k < 0 ? k + n : (k >= n ? k - n : k);
        return p + mat * (size_t)n * n + (size_t)c * n + k;
    }
};

// R = H X - X diag(W): cyclic band H on DMMA where the band fits a 64-row tile's span, else the
// FP64-FMA band kernel; dense H as a full DMMA GEMM.
template <class XT>
static cudaError_t launch_resid(cudaStream_t st, const cplx* A, const XT* X, const double* W, cplx* Res, int n,
                                int band, int nb) {
    const size_t nn = (size_t)n * n;
    if (band >= 0 && RB_BM + 2 * band <= n)
        return launch_zgemm<cplx, RB_BM>(st, OpBandA{A, n, band}, OpBandB<XT>{X, n, band},
                                         EpResid<XT>{X, W, Res, n}, n, n, RB_BM + 2 * band, nb);
    if (band >= 0) {
        k_ref_resid_band<XT><<<dim3((n + 31) / 32, (n + 63) / 64, nb), 256, 0, st>>>(A, X, W, Res, n, band);
        return cudaGetLastError();
    }
    return launch_zgemm<cplx, 64>(st, OpColA<cplx, cplx>{A, n, nn}, OpColB<cplx, XT>{X, n, nn},
                                  EpResid<XT>{X, W, Res, n}, n, n, n, nb);
}

// Per eigenvector j (one warp each), in double: G_jj = x_j^H x_j, q_j = Re(x_j^H r_j) and
// ||r_j||, stored as ST[3 (mat n + j) + {0, 1, 2}].
template <class XT>
__global__ void k_ref_colstats(const XT* __restrict__ X, const cplx* __restrict__ Res, double* __restrict__ ST,
                               int n, int nmat) {
    const int lane = threadIdx.x & 31;
    const size_t gw = (size_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (gw >= (size_t)nmat * n) return;
    const size_t mat = gw / n;
    const int j = (int)(gw % n);
    const XT* x = X + mat * (size_t)n * n + (size_t)j * n;
    const cplx* r = Res + mat * (size_t)n * n + (size_t)j * n;
    double g = 0.0, q = 0.0, rr = 0.0;
    for (int k = lane; k < n; k += 32) {
        const cplx xv = to_c64(x[k]), rv = r[k];
        g += xv.x * xv.x + xv.y * xv.y;
        q += xv.x * rv.x + xv.y * rv.y;
        rr += rv.x * rv.x + rv.y * rv.y;
    }
    g = warp_sum(g);
    q = warp_sum(q);
    rr = warp_sum(rr);
    if (lane == 0) {
        ST[3 * gw] = g;
        ST[3 * gw + 1] = q;
        ST[3 * gw + 2] = sqrt(rr);
    }
}

// Clusters of the ascending eigenvalues of each matrix (one thread per matrix): chains of
// consecutive pairs with gap <= RF_RES * max(||r||/||x||) or <= RF_CLUSTER * spectral radius.
// cl[j] = (first index, size).
__global__ void k_ref_clusters(const double* __restrict__ W, const double* __restrict__ ST, int2* __restrict__ cl,
                               int n, int nmat) {
    const int mat = blockIdx.x * blockDim.x + threadIdx.x;
    if (mat >= nmat) return;
    const double* w = W + (size_t)mat * n;
    const double* st = ST + (size_t)mat * n * 3;
    int2* c = cl + (size_t)mat * n;
    const double tie = RF_CLUSTER * fmax(fabs(w[0]), fabs(w[n - 1]));
    int a = 0;
    double rho_prev = st[2] / sqrt(fmax(st[0], DBL_MIN));
    for (int j = 1; j <= n; ++j) {
        bool split = true;
        double rho = 0.0;
        if (j < n) {
            rho = st[3 * j + 2] / sqrt(fmax(st[3 * j], DBL_MIN));
            const double gap = w[j] - w[j - 1];
            split = gap > tie && gap > RF_RES * fmax(rho, rho_prev);
        }
        if (split) {
            for (int m = a; m < j; ++m) c[m] = make_int2(a, j - a);
            a = j;
        }
        rho_prev = rho;
    }
}

// double overlap of two columns (single or double storage)
template <class XT>
__device__ __forceinline__ cplx col_dot(const XT* __restrict__ xi, const XT* __restrict__ xj, int n) {
    cplx g = mk(0, 0);
    for (int k = 0; k < n; ++k) cfmac(g, to_c64(xi[k]), to_c64(xj[k]));
    return g;
}

// F_ij = (X^H R)_ij / (lambda_j - lambda_i) for i != j; zero on the diagonal (set by
// k_ref_diag) and inside Rayleigh-Ritz clusters; -(x_i^H x_j)/2 inside larger clusters and
// for pairs too close for a first-order correction.  Epilogue of the GEMM X^H R taken in
// double: F + F^H must cancel the orthogonality defect (E_ij - conj(E_ji) = (lambda_i -
// lambda_j) x_i^H x_j).
template <class XT>
struct EpCoupling {
    const XT* x;
    const double* w;
    const int2* cl;
    cplxf* f;
    int n;
    __device__ __forceinline__ bool skip(int, int, int) const { return false; }
    __device__ __forceinline__ void store(size_t mat, int i, int j, cplx acc) const {
        cplxf val = make_float2(0.f, 0.f);
        if (i != j) {
            const double* wm = w + mat * n;
            const int2* cm_ = cl + mat * n;
            const double gap = wm[j] - wm[i];
            const int2 cj = cm_[j];
            const bool same = cm_[i].x == cj.x;
            if (same && cj.y <= RF_KMAX) {
                val = make_float2(0.f, 0.f);   // resolved by k_ref_cluster_solve
            } else if (!same && fabs(gap) > 8.0 * sqrt(cabs2(acc))) {
                const double ig = 1.0 / gap;
                val = make_float2((float)(acc.x * ig), (float)(acc.y * ig));
            } else {
                const XT* xm = x + mat * (size_t)n * n;
                const cplx g = col_dot(xm + (size_t)i * n, xm + (size_t)j * n, n);
                val = make_float2((float)(-0.5 * g.x), (float)(-0.5 * g.y));
            }
        }
        f[mat * (size_t)n * n + (size_t)j * n + i] = val;
    }
};

// Rayleigh-Ritz on each cluster of 2..RF_KMAX members (one warp per cluster, found at its
// first index): G = X_C^H X_C and E = X_C^H R_C by warp sums in double, S = E + G Lambda
// (Hermitian part), then in one lane G = L L^H, C = L^-1 S L^-H, Jacobi C = V diag(mu) V^H,
// Y = L^-H V (ascending mu).  Y[j][p] (column j's coefficients) and mu[j] go to YB / MU.
// Lane 0's part of k_ref_cluster_solve for the cluster of k members starting at eigenpair a
// of matrix mat: G (Gram) and S (Rayleigh) of the cluster in, Y and mu out.
__device__ __noinline__ void cluster_rr_serial(cplx* G, cplx* S, cplx* T, int k, size_t mat, int a, int n,
                                               const double* __restrict__ w, cplx* __restrict__ YB,
                                               double* __restrict__ MU) {
    // Hermitian parts
    for (int p = 0; p < k; ++p)
        for (int q = p; q < k; ++q) {
            const cplx gs = cscale(cadd(G[p + q * k], cconj(G[q + p * k])), 0.5);
            const cplx ss = cscale(cadd(S[p + q * k], cconj(S[q + p * k])), 0.5);
            G[p + q * k] = gs;
            G[q + p * k] = cconj(gs);
            S[p + q * k] = ss;
            S[q + p * k] = cconj(ss);
        }
    // Cholesky G = L L^H (L lower, stored in G's lower triangle and diagonal)
    for (int j = 0; j < k; ++j) {
        double d = G[j + j * k].x;
        for (int m = 0; m < j; ++m) d -= cabs2(G[j + m * k]);
        if (!(d > 0.0)) {   // not positive definite: leave the cluster as it is
            for (int q = 0; q < k; ++q) {
                cplx* yo = YB + (mat * n + a + q) * RF_KMAX;
                for (int p = 0; p < k; ++p) yo[p] = mk(p == q ? 1.0 : 0.0, 0.0);
                MU[mat * n + a + q] = w[a + q];
            }
            return;
        }
        const double ljj = sqrt(d);
        G[j + j * k] = mk(ljj, 0.0);
        for (int i = j + 1; i < k; ++i) {
            cplx s = G[i + j * k];
            for (int m = 0; m < j; ++m) s = csub(s, cmul(G[i + m * k], cconj(G[j + m * k])));
            G[i + j * k] = cscale(s, 1.0 / ljj);
        }
    }
    // T = L^-1 S (columns), then C = L^-1 T^H  (= L^-1 S L^-H, Hermitian)
    for (int q = 0; q < k; ++q)
        for (int i = 0; i < k; ++i) {
            cplx s = S[i + q * k];
            for (int m = 0; m < i; ++m) s = csub(s, cmul(G[i + m * k], T[m + q * k]));
            T[i + q * k] = cscale(s, 1.0 / G[i + i * k].x);
        }
    for (int q = 0; q < k; ++q)
        for (int i = 0; i < k; ++i) {
            cplx s = cconj(T[q + i * k]);
            for (int m = 0; m < i; ++m) s = csub(s, cmul(G[i + m * k], S[m + q * k]));
            S[i + q * k] = cscale(s, 1.0 / G[i + i * k].x);   // S now holds C
        }
    for (int p = 0; p < k; ++p)
        for (int q = p + 1; q < k; ++q) {
            const cplx h = cscale(cadd(S[p + q * k], cconj(S[q + p * k])), 0.5);
            S[p + q * k] = h;
            S[q + p * k] = cconj(h);
        }
    for (int p = 0; p < k; ++p) S[p + p * k].y = 0.0;
    for (int i = 0; i < k * k; ++i) T[i] = mk(i % (k + 1) == 0 ? 1.0 : 0.0, 0.0);
    herm_jacobi(S, T, k);   // T <- V
    // ascending order
    int order[RF_KMAX];
    for (int i = 0; i < k; ++i) order[i] = i;
    for (int i = 1; i < k; ++i)
        for (int j = i; j > 0 && S[order[j] * (k + 1)].x < S[order[j - 1] * (k + 1)].x; --j) {
            const int tmp = order[j];
            order[j] = order[j - 1];
            order[j - 1] = tmp;
        }
    // Y = L^-H V by back substitution, column by column
    for (int q = 0; q < k; ++q) {
        const int col = order[q];
        cplx y[RF_KMAX];
        for (int i = k - 1; i >= 0; --i) {
            cplx s = T[i + col * k];
            for (int m = i + 1; m < k; ++m) s = csub(s, cmul(cconj(G[m + i * k]), y[m]));
            y[i] = cscale(s, 1.0 / G[i + i * k].x);
        }
        cplx* yo = YB + (mat * n + a + q) * RF_KMAX;
        for (int p = 0; p < k; ++p) yo[p] = y[p];
        MU[mat * n + a + q] = S[col * (k + 1)].x;
    }
}

template <class XT>
__global__ void k_ref_cluster_solve(const XT* __restrict__ X, const cplx* __restrict__ Res,
                                    const double* __restrict__ W, const int2* __restrict__ CL,
                                    cplx* __restrict__ YB, double* __restrict__ MU, int n, int nmat) {
    const int lane = threadIdx.x & 31;
    // G, S and T of this warp's cluster in shared memory (column-major [p + q*k]); only lane 0
    // writes and reads them
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx* G = reinterpret_cast<cplx*>(smem_raw) + (size_t)(threadIdx.x / 32) * 3 * RF_KMAX * RF_KMAX;
    cplx* S = G + RF_KMAX * RF_KMAX;
    cplx* T = S + RF_KMAX * RF_KMAX;
    // grid-stride over the eigenpairs: most are not cluster leaders and are skipped at once
    const size_t nwarps = (size_t)gridDim.x * (blockDim.x / 32);
    for (size_t gw = (size_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; gw < (size_t)nmat * n;
         gw += nwarps) {
        const size_t mat = gw / n;
        const int a = (int)(gw % n);
        const int2 c = CL[mat * n + a];
        const int k = c.y;
        if (c.x != a || k < 2 || k > RF_KMAX) continue;
        const XT* x = X + mat * (size_t)n * n;
        const cplx* res = Res + mat * (size_t)n * n;
        const double* w = W + mat * n;
        for (int p = 0; p < k; ++p)
            for (int q = 0; q < k; ++q) {
                const XT* xp = x + (size_t)(a + p) * n;
                const XT* xq = x + (size_t)(a + q) * n;
                const cplx* rq = res + (size_t)(a + q) * n;
                cplx g = mk(0, 0), e = mk(0, 0);
                for (int r = lane; r < n; r += 32) {
                    const cplx xpr = to_c64(xp[r]);
                    cfmac(g, xpr, to_c64(xq[r]));
                    cfmac(e, xpr, rq[r]);
                }
                g = warp_sum(g);
                e = warp_sum(e);
                if (lane == 0) {
                    G[p + q * k] = g;
                    S[p + q * k] = mk(e.x + w[a + q] * g.x, e.y + w[a + q] * g.y);
                }
            }
        if (lane == 0) cluster_rr_serial(G, S, T, k, mat, a, n, w, YB, MU);
        __syncwarp();
    }
}

// Per eigenvector j (one thread each): lambda_j += q_j / G_jj (Rayleigh quotient) and
// F_jj = (1 - G_jj) / 2 from k_ref_colstats -- except for members of Rayleigh-Ritz clusters
// (F_jj = 0, lambda from k_ref_cluster_apply).
__global__ void k_ref_diag(const double* __restrict__ ST, const int2* __restrict__ CL, double* __restrict__ W,
                           cplxf* __restrict__ F, int n, int nmat) {
    const size_t gj = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gj >= (size_t)nmat * n) return;
    const size_t mat = gj / n;
    const int j = (int)(gj % n);
    const int2 c = CL[gj];
    cplxf* fjj = F + mat * (size_t)n * n + (size_t)j * n + j;
    if (c.y >= 2 && c.y <= RF_KMAX) {
        *fjj = make_float2(0.f, 0.f);
        return;
    }
    const double g = ST[3 * gj], q = ST[3 * gj + 1];
    W[gj] += q / g;
    *fjj = make_float2((float)(0.5 * (1.0 - g)), 0.f);
}

// X_out = X + X F: epilogue of the single-precision GEMM X F, sum in double, into a
// buffer other than X.
template <class XT>
struct EpUpdate {
    const XT* x;
    cplx* out;
    int n;
    __device__ __forceinline__ bool skip(int, int, int) const { return false; }
    __device__ __forceinline__ void store(size_t mat, int r, int c, cplxf acc) const {
        const size_t o = mat * (size_t)n * n + (size_t)c * n + r;
        const cplx xr = to_c64(x[o]);
        out[o] = mk(xr.x + (double)acc.x, xr.y + (double)acc.y);
    }
};

// X_C <- X_C Y and lambda_C <- mu for every Rayleigh-Ritz cluster (one warp per cluster,
// rows dealt to lanes; every row is read before it is written, so in place).
__global__ void k_ref_cluster_apply(cplx* __restrict__ X, const int2* __restrict__ CL, const cplx* __restrict__ YB,
                                    const double* __restrict__ MU, double* __restrict__ W, int n, int nmat) {
    const int lane = threadIdx.x & 31;
    const size_t gw = (size_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (gw >= (size_t)nmat * n) return;
    const size_t mat = gw / n;
    const int a = (int)(gw % n);
    const int2 c = CL[gw];
    const int k = c.y;
    if (c.x != a || k < 2 || k > RF_KMAX) return;
    cplx y[RF_KMAX * RF_KMAX];   // y[p + q*k]
    for (int q = 0; q < k; ++q)
        for (int p = 0; p < k; ++p) y[p + q * k] = YB[(mat * n + a + q) * RF_KMAX + p];
    cplx* x = X + mat * (size_t)n * n + (size_t)a * n;
    for (int r = lane; r < n; r += 32) {
        cplx old[RF_KMAX];
        for (int p = 0; p < k; ++p) old[p] = x[(size_t)p * n + r];
        for (int q = 0; q < k; ++q) {
            cplx s = mk(0, 0);
            for (int p = 0; p < k; ++p) cfma(s, old[p], y[p + q * k]);
            x[(size_t)q * n + r] = s;
        }
    }
    if (lane < k) W[mat * n + a + lane] = MU[mat * n + a + lane];
}

// double -> single copy of the matrices (the single-precision reduction works on the copy;
// the double input stays for the residual)
__global__ void k_to_single(const cplx* __restrict__ A, cplxf* __restrict__ B, size_t total) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
        B[i] = from_c64<cplxf>(A[i]);
}

// Launch shape of k_hetrd: NT threads, as much of the leading triangle resident as fits (all
// of it up to order ~155 in double precision).  Threads: the tiles of a pass are few (3 at order
// 32, 10 at 64) and every warp repeats the column's scalar steps, so one warp up to order 40, 64
// threads up to 48, 128 up to 100 with several CTAs per SM, 256 where one fits or the matrices
// are fewer than the SMs; 512 where the sums go through atomics.  2,304 matrices of order 32 took
// 0.26 ms with 64 threads and 0.17 with 32; 128 of order 129 0.46 with 512 and 0.44 with 256;
// order 64 is even between 64 and 128.
struct HetrdCfg {
    int nt;
    int tri_cap;
    size_t smem;
};
template <class R>
static HetrdCfg hetrd_config(int m, int nb) {
    const size_t ce = 2 * sizeof(R);   // complex element
    const int nt = m > HT_PARTS_MAX ? 512 : nb <= 148 || m > 100 ? 256 : m <= 40 ? 32 : m <= 48 ? 64 : 128;
    const size_t vec = (3 * (size_t)hetrd_pad(m) + hetrd_pn(m) + (m > HT_PARTS_MAX ? 0 : 2)) * ce + 2 * (nt / 32) * sizeof(R);
    const size_t budget = 220 * 1024;
    size_t cap = budget > vec ? (budget - vec) / ce : 0;
    cap = std::min(cap, (size_t)m * (m + 1) / 2);
    return {nt, (int)cap, vec + cap * ce};
}
template <int NT, class R, bool PARTS>
static cudaError_t launch_hetrd_t(const HetrdCfg& c, cudaStream_t st, int nb, typename Cx<R>::T* A, double* D,
                                  double* E, typename Cx<R>::T* TAU, int n, int m) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_hetrd<NT, R, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.smem);
    if (e != cudaSuccess) return e;
    k_hetrd<NT, R, PARTS><<<nb, NT, c.smem, st>>>(A, D, E, TAU, n, m, c.tri_cap);
    return cudaGetLastError();
}
template <class R>
static cudaError_t launch_hetrd(cudaStream_t st, int nb, typename Cx<R>::T* A, double* D, double* E,
                                typename Cx<R>::T* TAU, int n, int m) {
    const HetrdCfg c = hetrd_config<R>(m, nb);
    if (c.smem > 227 * 1024) return cudaErrorInvalidValue;
    if (m > HT_PARTS_MAX) return launch_hetrd_t<512, R, false>(c, st, nb, A, D, E, TAU, n, m);
    const auto launch = c.nt == 32 ? launch_hetrd_t<32, R, true> : c.nt == 64 ? launch_hetrd_t<64, R, true>
                      : c.nt == 128 ? launch_hetrd_t<128, R, true> : launch_hetrd_t<256, R, true>;
    return launch(c, st, nb, A, D, E, TAU, n, m);
}

// Launch choices of one eigensolve configuration that the autotuner may set (0 / -1: the
// built-in choice for the order).
struct HeevTune {
    int blocked = -1;    // 1: blocked reduction (16-column panels + GEMM updates), 0: unblocked only
    int gemm_bt = -1;    // 1: GEMM back-transformation, 0: register-resident k_ormtr (where it fits)
    int panel_nt = 0;    // threads per panel CTA, 256 or 512
    int xtile = 0;       // row tile of the double-precision X -= V W' update, 64 or 128
    int bt_nb = 0;       // reflectors per block of the GEMM back-transformation, 64 or 128
    int jacobi = -1;     // 1: batched Jacobi (k_jacobi, orders <= JAC_MAX_N), 0: the Householder path
    int queue_nt = 0;    // panel queue CTAs: 512 threads (one per SM) or 256 (two per SM); 0: built-in
    int panel_w = 0;     // panel width, 16 or 32; 0: built-in (32 from order HP_W_WIDE_MIN in FP64)
    int dc = -1;         // tridiagonal stage: 1 divide and conquer (orders <= DC_MAX_N), 0 bisection +
                         // inverse iteration (k_tridiag)
};

// Shape of one eigensolve chunk: kernel configurations and the scratch layout per matrix
// (byte offsets, each region a multiple of 256 bytes so that every region of a chunk
// starts aligned whatever the chunk size).
struct HeevPlan {
    int n;
    bool jacobi;         // k_jacobi in double precision (either mode); nothing below applies
    size_t smem_jac;
    bool dc;             // divide-and-conquer tridiagonal stage (tridiag_dc.cuh) instead of k_tridiag
    size_t off_q2, off_u, off_rot, off_sc;   // its second Q, U, rotations and scale
    bool mixed;          // single-precision reduction + double refinement
    int refine_steps;    // mixed mode: 1 or 2
    bool rq;             // mixed mode, one step: then the eigenvalues as Rayleigh quotients (H kept until then)
    int band;            // >= 0: every matrix is a cyclic band of this half-bandwidth (rlm), else -1
    size_t smem_tri;
    bool small_bt;       // k_ormtr (register-resident Z chunk) or the blocked GEMM path
    int ch, dbuf, orm_nt;
    size_t smem_orm;
    int nblk16, bt_nb, nblkbt;   // k_ormtr blocks; GEMM back-transformation block size and count
    int npanels, m_tail;  // blocked reduction: panels of pw columns, then k_hetrd on m_tail
    int pw;               // panel width, 16 or 32
    int panel_nt, xtile;  // tuned launch choices (0: built-in)
    int queue_nt;         // threads of the panel queue's CTAs (512: one per SM, 256: two per SM)
    bool queue_pinned;    // set by the caller: the queue wherever it applies
    // per: bytes per matrix of the chunk's regions (offsets off_*, times the chunk size);
    // per2: bytes per matrix of the mixed mode's refinement regions (Res, X1), which the
    // refinement uses for one sub-chunk of matrices at a time
    size_t per2, off2_x1;
    size_t off_d, off_e, off_tau, off_a, off_z, off_lu, off_x, off_t, off_w, off_res, off_x1, off_cl,
        off_y, off_mu, off_st, off_pv, off_q, per;
};

static HeevPlan heev_plan(int n, bool mixed, int refine_steps = 2, int band = -1, HeevTune tune = HeevTune{}) {
    HeevPlan p{};
    p.panel_nt = tune.panel_nt;
    p.xtile = tune.xtile;
    p.queue_nt = tune.queue_nt ? tune.queue_nt : QUEUE_NT_DEFAULT;
    p.queue_pinned = tune.queue_nt != 0;
    p.n = n;
    p.mixed = mixed;
    p.band = band >= 0 && 32 + 2 * band <= n ? band : -1;   // the band residual needs 32 + 2o <= n
    // refine_steps 3 (heev_steps): one step, then the Rayleigh-quotient eigenvalue pass
    p.rq = mixed && refine_steps == 3;
    p.refine_steps = mixed ? (refine_steps == 3 ? 1 : refine_steps) : 0;
    p.jacobi = n <= JAC_MAX_N && (tune.jacobi < 0 ? n <= JAC_DEFAULT_MAX : tune.jacobi > 0);
    if (p.jacobi) {   // no scratch: the matrix and its rotations live in shared memory
        p.smem_jac = jacobi_smem(n);
        p.per = 256;
        return p;
    }
    const size_t ce = mixed ? sizeof(cplxf) : sizeof(cplx);   // working complex element
    p.pw = tune.panel_w ? tune.panel_w : n >= HP_W_WIDE_MIN && !mixed ? 32 : 16;
    const bool blocked = tune.blocked < 0 ? n >= HT_BLOCKED_MIN : (tune.blocked > 0 && n > HT_TAIL + p.pw);
    p.npanels = blocked ? (n - HT_TAIL + p.pw - 1) / p.pw : 0;
    p.m_tail = n - p.npanels * p.pw;
    p.smem_tri = 4 * (size_t)n * sizeof(double) + n * sizeof(int);
    p.nblk16 = (n - 1 + ORM_NB - 1) / ORM_NB;
    p.bt_nb = tune.bt_nb ? tune.bt_nb : n >= BT128_MIN ? 2 * BT_NB : BT_NB;
    p.nblkbt = (n - 1 + p.bt_nb - 1) / p.bt_nb;
    bool fits;
    if (mixed) {   // k_ormtr<float>
        int ch = 16;
        while (ch > 1 && (n + 256 / ch - 1) / (256 / ch) > ORM_RPT) ch >>= 1;
        p.ch = ch;
        const int onw = 8;   // warps of k_ormtr (256 threads; 512 threads of 8 rows, or 8 columns
                             // of 8 rows at two CTAs per SM, measured slower)
        size_t smem = ((size_t)2 * n * ORM_VS + 2 * ORM_NB * ORM_NB + onw * ORM_NB * ch + ORM_NB * ch) * ce;
        p.dbuf = smem <= 220 * 1024 ? 1 : 0;
        if (!p.dbuf)
            smem = ((size_t)std::max(n * ORM_VS, n * ch) + ORM_NB * ORM_NB + onw * ORM_NB * ch + ORM_NB * ch) * ce;
        p.smem_orm = smem;
        fits = (n + 256 / ch - 1) / (256 / ch) <= ORM_RPT && smem <= 220 * 1024;
    } else {       // k_ormtr_mma: 32 columns per CTA, 16 where X and V leave no room for more
        p.ch = OrmtrMma<32, 512>::smem(n) <= 227 * 1024 ? 32 : 16;
        p.orm_nt = p.ch == 32 && OrmtrMma<32, 256>::smem(n) <= 113 * 1024 ? 256 : 512;
        p.smem_orm = p.ch == 16 ? OrmtrMma<16, 512>::smem(n)
                   : p.orm_nt == 256 ? OrmtrMma<32, 256>::smem(n) : OrmtrMma<32, 512>::smem(n);
        fits = p.smem_orm <= 227 * 1024;
    }
    // X resident on the SM where it fits: below order 256 in the mixed mode, up to BT_MMA_MAX in
    // double precision (it beats the GEMM path there), the GEMM path otherwise
    p.small_bt = fits && (tune.gemm_bt < 0 ? (mixed ? n < BT_GEMM_MIN : n <= BT_MMA_MAX) : tune.gemm_bt == 0);
    const size_t nn = (size_t)n * n;
    auto r256 = [](size_t v) { return (v + 255) / 256 * 256; };
    size_t off = 0;
    p.off_d = off; off += r256(n * sizeof(double));
    p.off_e = off; off += r256(n * sizeof(double));
    p.off_tau = off; off += r256(n * ce);
    p.off_a = off; off += mixed ? r256(nn * ce) : 0;        // single-precision copy of H, then F
    p.dc = n <= DC_MAX_N && (tune.dc < 0 ? n >= DC_DEFAULT_MIN : tune.dc > 0);
    p.off_z = off; off += r256(nn * sizeof(double));
    p.off_lu = off; off += p.dc ? 0 : r256(5 * (size_t)n * tri_columns(n) * sizeof(double));
    p.off_q2 = off; off += p.dc ? r256(nn * sizeof(double)) : 0;
    p.off_u = off; off += p.dc ? r256(nn * sizeof(double)) : 0;
    p.off_rot = off; off += p.dc ? r256((size_t)n * sizeof(DcRot)) : 0;
    p.off_sc = off; off += p.dc ? 256 : 0;
    p.off_x = off; off += r256(nn * ce);
    p.off_t = off; off += r256((p.small_bt ? (size_t)p.nblk16 * ORM_NB * ORM_NB : (size_t)p.nblkbt * p.bt_nb * p.bt_nb) * ce);
    p.off_w = off; off += p.small_bt ? 0 : r256(2 * (size_t)p.bt_nb * n * ce);   // G and W' of a block
    p.off_res = 0;   // (the refinement regions: per2 below)
    p.off_x1 = 0;
    p.off_cl = off; off += mixed ? r256(n * sizeof(int2)) : 0;
    p.off_y = off; off += mixed ? r256((size_t)n * RF_KMAX * sizeof(cplx)) : 0;
    p.off_mu = off; off += mixed ? r256(n * sizeof(double)) : 0;
    p.off_st = off; off += mixed ? r256(3 * (size_t)n * sizeof(double)) : 0;
    p.off_pv = off; off += p.npanels > 0 ? r256(2 * (size_t)p.pw * n * ce) : 0;   // panel V, W
    p.off_q = off; off += p.npanels > 0 ? r256(16) : 0;   // panel queue: claims, abort flag, column counts
    p.per = off;
    p.per2 = mixed ? r256(nn * sizeof(cplx)) : 0;                              // residual R
    p.off2_x1 = p.per2;
    p.per2 += p.refine_steps >= 2 || p.rq ? r256(nn * sizeof(cplx)) : 0;         // step-1 vectors
    return p;
}

// The allocation-free path's configuration: the built-in one with the bisection tridiagonal
// solver, whose scratch sets its order limit.
static HeevPlan noalloc_plan(int n) {
    HeevTune t;
    t.dc = 0;
    return heev_plan(n, false, 2, -1, t);
}

// Bytes of scratch one matrix of order n needs in heev_chunk_on_scratch (double precision).
size_t heev_scratch_bytes_per_matrix(int n) { return noalloc_plan(n).per; }

// Largest chunk of matrices one heev_chunk call may take: the grid y / z extent (65535) of
// the per-matrix launches, and of the (matrix, block) batches of the GEMM back-transformation.
size_t heev_max_chunk(int n) {
    const HeevPlan p = noalloc_plan(n);
    size_t c = 65535;
    if (!p.small_bt) c = std::min<size_t>(c, 65535 / std::max(p.nblkbt, 1));
    return c;
}

#define RLMB_CHUNK_LAUNCHED()                                     \
    do {                                                          \
        if (ctx) {                                                \
            prof_end(ctx);                                        \
            ctx->launches++;                                      \
        } else {                                                  \
            ++*launches;                                          \
        }                                                         \
        if (cudaGetLastError() != cudaSuccess) return RLMB_ERR_CUDA; \
    } while (0)
#define RLMB_CHUNK_PROF(name) \
    do {                      \
        if (ctx) prof_begin(ctx, name); \
    } while (0)

// Householder tridiagonalisation in the working precision R: blocked panels (k_hetrd_panel_c +
// rank-2*pw GEMM update) down to order m_tail, then k_hetrd on the leading block.  PV holds
// the panel pairs of the chunk (V of every matrix, then W of every matrix).
template <class R>
static int tridiagonalise(rlmb_context* ctx, cudaStream_t st, const HeevPlan& p, int nb, typename Cx<R>::T* A,
                          double* D, double* E, typename Cx<R>::T* TAU, typename Cx<R>::T* PV, int* Q, int* info,
                          long long* launches) {
    typedef typename Cx<R>::T C;
    const int n = p.n;
    int m = n;
    if (p.npanels > 0) {
        const int pw = p.pw;
        C* PWb = PV + (size_t)nb * pw * n;
        int dev = 0, sms = 148;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return RLMB_ERR_CUDA;
        // above order 512, chunks of more matrices than SMs: one 512-thread CTA per SM taking
        // (matrix, column) units from a queue (k_hetrd_panel_q), built in where one CTA per matrix
        // would leave its last wave mostly empty (panel_waves_full)
        const int qnt = p.queue_nt == 256 ? 256 : 512;
        const int qper = qnt == 256 ? 2 : 1;   // resident queue CTAs per SM
        const bool queue = p.panel_nt == 0 && n > 512 && nb > sms && (p.queue_pinned || !panel_waves_full<R>(n, nb)) &&
                           (qnt == 512 ? panel_smem<512, R>(n) <= 227 * 1024 : panel_smem<256, R>(n) <= 113 * 1024);
        // chunks of few matrices: a cluster of CTAs per matrix; otherwise one CTA per matrix,
        // with the pinned number of threads if there is one
        PanelShape shape{};
        if (p.panel_nt == 0 && !queue) shape = panel_shape<R>(n, nb);
        // Where neither runs and the vectors leave the rings of k_hetrd_panel_c no room for 512 threads
        // (double precision: above order 3000; no cluster fits above 5080), the queue's kernel, whose
        // loads need no rings, takes the panels until the leading block has shrunk enough.  With the 256 to
        // 64 threads that fit, eigensolves of 100 matrices of order 4000 took 7.4 s, now 6.4, one of order
        // 5600 12.7 s, now 3.5, and one of 6300 20.1, now 9.8.
        auto too_long = [](int order) { return panel_c_smem<512, R>(order, 1) > 227 * 1024; };
        const bool long_queue = p.panel_nt == 0 && n > 512 && !queue && shape.P == 0 && too_long(n) && qnt == 512 &&
                                panel_smem<512, R>(n) <= 227 * 1024;
        if (queue || long_queue) {
            const void* qk = qnt == 256 ? (const void*)k_hetrd_panel_q<256, R> : (const void*)k_hetrd_panel_q<512, R>;
            const size_t smem = qnt == 256 ? panel_smem<256, R>(n) : panel_smem<512, R>(n);
            if (cudaFuncSetAttribute(qk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
                return RLMB_ERR_CUDA;
        }
        const int grid = std::min(nb, qper * sms);
        // the queue's counters, and its abort flag, which k_panel_abort_info reads in every case
        if (cudaMemsetAsync(Q, 0, (8 + (size_t)nb) * sizeof(int), st) != cudaSuccess) return RLMB_ERR_CUDA;
        for (int k = 0; k < p.npanels; ++k) {
            RLMB_CHUNK_PROF("k_hetrd_panel");
            const bool by_queue = queue || (long_queue && too_long(m));
            if (k > 0 && (shape.P > 0 ? shape.nt < 512 : long_queue && by_queue)) {   // (the vectors have shrunk)
                const PanelShape wider = panel_shape<R>(m, nb);
                if (wider.P > 0) shape = wider;
            }
            if (shape.P > 0) {
                const auto launch = shape.nt == 512 ? launch_panel_c<512, R>
                                  : shape.nt == 384 ? launch_panel_c<384, R> : launch_panel_c<256, R>;
                if (launch(st, A, D, E, TAU, PV, PWb, n, m, pw, nb, shape.P) != cudaSuccess) return RLMB_ERR_CUDA;
            } else if (by_queue && qnt == 256) {
                k_hetrd_panel_q<256, R><<<grid, 256, panel_smem<256, R>(n), st>>>(
                    A, D, E, TAU, PV, PWb, n, m, pw, nb, Q, (long long)k * ((long long)nb * pw + grid), k * pw, info);
            } else if (by_queue) {
                k_hetrd_panel_q<512, R><<<grid, 512, panel_smem<512, R>(n), st>>>(
                    A, D, E, TAU, PV, PWb, n, m, pw, nb, Q, (long long)k * ((long long)nb * pw + grid), k * pw, info);
            } else {
                const int nt = panel_threads<R>(m, nb, p.panel_nt);
                const auto launch = nt == 512 ? launch_panel_one<512, R> : nt == 256 ? launch_panel_one<256, R>
                                  : nt == 128 ? launch_panel_one<128, R> : launch_panel_one<64, R>;
                if (nt == 0 || launch(st, A, D, E, TAU, PV, PWb, n, m, pw, nb) != cudaSuccess) return RLMB_ERR_CUDA;
            }
            RLMB_CHUNK_LAUNCHED();
            m -= pw;
            RLMB_CHUNK_PROF("k_hetrd_her2k");
            // (the width a compile-time constant of the operands: their loads are the tile's work)
            const cudaError_t eu =
                pw == 32 ? launch_work_gemm<C, 64>(st, OpPanelA<C, 32>{PV, PWb, n}, OpPanelB<C, 32>{PV, PWb, n},
                                                   EpHer2k<C>{A, n}, m, m, 64, nb)
                         : launch_work_gemm<C, 64>(st, OpPanelA<C, 16>{PV, PWb, n}, OpPanelB<C, 16>{PV, PWb, n},
                                                   EpHer2k<C>{A, n}, m, m, 32, nb);
            if (eu != cudaSuccess)
                return RLMB_ERR_CUDA;
            RLMB_CHUNK_LAUNCHED();
        }
    }
    RLMB_CHUNK_PROF("k_hetrd");
    if (launch_hetrd<R>(st, nb, A, D, E, TAU, n, m) != cudaSuccess) return RLMB_ERR_CUDA;
    RLMB_CHUNK_LAUNCHED();
    return RLMB_OK;
}

// After the tridiagonal solve (which writes every matrix's info): a panel queue that ran out
// of its bounded wait marks every matrix of the chunk as failed.
__global__ void k_panel_abort_info(const int* __restrict__ Q, int* __restrict__ info, int nb) {
    if (!*(volatile const int*)(Q + 1)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x) info[i] = -1;
}

// Back-transformation X = Q Z in the working precision R (X column-major, column =
// eigenvector): k_larft + k_ormtr, or the blocked GEMM path (Gram GEMM + k_larft64, then
// three GEMMs per block of 64 reflectors).
template <class R>
static int back_transform(rlmb_context* ctx, cudaStream_t st, const HeevPlan& p, int nb,
                          const typename Cx<R>::T* Aw, const typename Cx<R>::T* TAUw, const double* Zw,
                          typename Cx<R>::T* Xw, typename Cx<R>::T* Tw, typename Cx<R>::T* Wp,
                          long long* launches) {
    typedef typename Cx<R>::T C;
    const int n = p.n;
    const size_t nn = (size_t)n * n;
    if (p.small_bt) {
        if (n > 1) {
            RLMB_CHUNK_PROF("k_larft");
            if constexpr (std::is_same<R, double>::value)
                k_larft_mma<<<dim3((p.nblk16 + LM_WARPS - 1) / LM_WARPS, nb), 32 * LM_WARPS, 0, st>>>(Aw, TAUw, Tw, n,
                                                                                                     p.nblk16);
            else k_larft<R><<<dim3(p.nblk16, nb), 128, 0, st>>>(Aw, TAUw, Tw, n);
            RLMB_CHUNK_LAUNCHED();
        }
        const dim3 grid((n + p.ch - 1) / p.ch, nb);
        RLMB_CHUNK_PROF("k_ormtr");
        if constexpr (std::is_same<R, double>::value) {
            auto ormtr = p.ch == 16 ? k_ormtr_mma<16, 512> : p.orm_nt == 256 ? k_ormtr_mma<32, 256> : k_ormtr_mma<32, 512>;
            if (cudaFuncSetAttribute(ormtr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem_orm) != cudaSuccess)
                return RLMB_ERR_CUDA;
            ormtr<<<grid, p.orm_nt, p.smem_orm, st>>>(Aw, Tw, Zw, Xw, n);
        } else {
            auto ormtr = p.ch == 16 ? k_ormtr<16, 256, ORM_RPT, R> : p.ch == 8 ? k_ormtr<8, 256, ORM_RPT, R>
                       : p.ch == 4 ? k_ormtr<4, 256, ORM_RPT, R> : p.ch == 2 ? k_ormtr<2, 256, ORM_RPT, R>
                       : k_ormtr<1, 256, ORM_RPT, R>;
            if (cudaFuncSetAttribute(ormtr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem_orm) != cudaSuccess)
                return RLMB_ERR_CUDA;
            ormtr<<<grid, 256, p.smem_orm, st>>>(Aw, Tw, Zw, Xw, n, p.dbuf);
        }
        RLMB_CHUNK_LAUNCHED();
        return RLMB_OK;
    }
    const int bs = p.bt_nb, nblk = p.nblkbt;
    RLMB_CHUNK_PROF("k_larft");
    if (launch_work_gemm<C, 64>(st, OpBlkReflH<C>{Aw, n, nblk, bs}, OpBlkRefl<C>{Aw, n, nblk, bs},
                            EpStore<C>{Tw, bs, (size_t)bs * bs}, bs, bs, n, nb * nblk) != cudaSuccess)
        return RLMB_ERR_CUDA;
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_larft");
    if (bs == BT_NB) {
        const size_t smem_t = BT_NB * (BT_NB + 1) * sizeof(C);
        if (cudaFuncSetAttribute(k_larft64<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_t) != cudaSuccess)
            return RLMB_ERR_CUDA;
        k_larft64<R><<<dim3(nblk, nb), 2 * BT_NB, smem_t, st>>>(TAUw, Tw, n);
    } else {
        const size_t smem_t = 3 * BT_NB * (BT_NB + 1) * sizeof(C);
        if (cudaFuncSetAttribute(k_larft128<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_t) != cudaSuccess)
            return RLMB_ERR_CUDA;
        k_larft128<R><<<dim3(nblk, nb), 256, smem_t, st>>>(TAUw, Tw, n);
    }
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ormtr");
    k_z_to_x<C><<<2048, 256, 0, st>>>(Zw, Xw, n, (size_t)nb * nn);
    RLMB_CHUNK_LAUNCHED();
    // per block j of bs reflectors (zlarfb): G = V^H X, W' = T G, X -= V W'; G and W' are
    // [n][bs] per matrix (column c of G at c*bs)
    C* G = Wp;
    C* W2 = Wp + (size_t)nb * bs * n;
    const size_t gs = (size_t)bs * n;
    for (int j = 0; j < nblk; ++j) {
        const int i0 = j * bs;
        const int rows = std::min(i0 + bs - 1, n - 2) + 1;   // rows 0..i1 carry the block
        RLMB_CHUNK_PROF("k_ormtr");
        if (launch_work_gemm<C, 64>(st, OpReflH<C>{Aw, n, i0}, OpColB<C, C>{Xw, n, nn}, EpStore<C>{G, bs, gs},
                                bs, n, rows, nb) != cudaSuccess)
            return RLMB_ERR_CUDA;
        RLMB_CHUNK_LAUNCHED();
        RLMB_CHUNK_PROF("k_ormtr");
        if (launch_work_gemm<C, 64>(st, OpRowA<C, C, false>{Tw + (size_t)j * bs * bs, bs, (size_t)nblk * bs * bs},
                                OpColB<C, C>{G, bs, gs}, EpStore<C>{W2, bs, gs}, bs, n, bs, nb) != cudaSuccess)
            return RLMB_ERR_CUDA;
        RLMB_CHUNK_LAUNCHED();
        RLMB_CHUNK_PROF("k_ormtr");
        // X -= V W': 64-row tiles (two CTAs per SM) on the DMMA engine unless tuned to 128
        // (the tcgen05 engine of the single-precision mode has its own tile)
        const cudaError_t ex =
            p.xtile == 128 ? launch_work_gemm<C, 128>(st, OpRefl<C>{Aw, n, i0}, OpColB<C, C>{W2, bs, gs},
                                                      EpSub<C>{Xw, n}, rows, n, bs, nb)
                           : launch_work_gemm<C, 64>(st, OpRefl<C>{Aw, n, i0}, OpColB<C, C>{W2, bs, gs},
                                                     EpSub<C>{Xw, n}, rows, n, bs, nb);
        if (ex != cudaSuccess) return RLMB_ERR_CUDA;
        RLMB_CHUNK_LAUNCHED();
    }
    return RLMB_OK;
}

// cuTensorMapEncodeTiled, looked up once from the driver through the runtime.
TmaEncodeFn tma_encode_fn() {
    static TmaEncodeFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<TmaEncodeFn>(p);
        else
            cudaGetLastError();
    }
    return fn;
}

// Planes of the TMA-fed GEMMs of one refinement chunk: up to 4 GB, at least one matrix.
static int refine_planes(rlmb_context* ctx, int n, int nb) {
    const size_t per = tma_plane_bytes(n, n, n);
    const size_t want = std::max(per, std::min((size_t)nb * per, (size_t)4 << 30));
    return ensure_tma_planes(ctx, want);
}

// One refinement step from the vectors X (single or double) to Out (double, not X).
template <class XT>
static int refine_step(rlmb_context* ctx, cudaStream_t st, int n, int band, int nb, const cplx* A, const XT* X,
                       double* W, cplx* Res, cplxf* F, int2* CL, cplx* YB, double* MU, double* ST,
                       cplx* Out, long long* launches) {
    const size_t nn = (size_t)n * n;
    const unsigned gw = (unsigned)(((size_t)nb * n + 7) / 8);   // one warp per column
    RLMB_CHUNK_PROF("k_ref_resid");
    if (launch_resid<XT>(st, A, X, W, Res, n, band, nb) != cudaSuccess) return RLMB_ERR_CUDA;
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_colstats");
    k_ref_colstats<XT><<<gw, 256, 0, st>>>(X, Res, ST, n, nb);
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_clusters");
    k_ref_clusters<<<(nb + 127) / 128, 128, 0, st>>>(W, ST, CL, n, nb);
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_coupling");
    // E = X^H R on the TMA-fed engine with double-precision accumulation: its error, relative
    // to |X| |R|, is the orthogonality defect the step leaves (F + F^H cancels x_i^H x_j only
    // as well as E is known)
    if (!ctx) return RLMB_ERR_ARG;
    if (int rc = refine_planes(ctx, n, nb)) return rc;
    if (launch_zgemm_tma<cplx>(st, OpRowA<cplx, XT, true>{X, n, nn}, OpColB<cplx, cplx>{Res, n, nn},
                               EpCoupling<XT>{X, W, CL, F, n}, n, n, n, nb, ctx->tws, ctx->tws_bytes) != cudaSuccess)
        return RLMB_ERR_CUDA;
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_cluster");
    {
        const size_t smem_cs = 8 * 3 * RF_KMAX * RF_KMAX * sizeof(cplx);   // 8 warps x (G, S, T)
        if (cudaFuncSetAttribute(k_ref_cluster_solve<XT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_cs) !=
            cudaSuccess)
            return RLMB_ERR_CUDA;
        // a bounded grid (8 warps per CTA, two CTAs per SM by shared memory) strides over gw warps
        const unsigned grid = (unsigned)std::min<size_t>(gw, 4 * 2 * 148);
        k_ref_cluster_solve<XT><<<grid, 256, smem_cs, st>>>(X, Res, W, CL, YB, MU, n, nb);
    }
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_diag");
    k_ref_diag<<<(unsigned)(((size_t)nb * n + 255) / 256), 256, 0, st>>>(ST, CL, W, F, n, nb);
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_update");
    // X F is a correction of the size of the current error: FP32 sums over K (one drain per
    // tile) carry it to well below the step's target
    if (launch_zgemm_tma<cplxf>(st, OpColA<cplx, XT>{X, n, nn}, OpColB<cplxf, cplxf>{F, n, nn},
                                EpUpdate<XT>{X, Out, n}, n, n, n, nb, ctx->tws, ctx->tws_bytes, false) != cudaSuccess)
        return RLMB_ERR_CUDA;
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_cluster");
    k_ref_cluster_apply<<<gw, 256, 0, st>>>(Out, CL, YB, MU, W, n, nb);
    RLMB_CHUNK_LAUNCHED();
    return RLMB_OK;
}

// w_j <- w_j + Re(x_j^H r_j) / x_j^H x_j for every column: the Rayleigh quotient of x_j, r = H x - x w.
__global__ void k_ref_rq(const double* __restrict__ ST, double* __restrict__ W, size_t total) {
    const size_t gj = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gj < total) W[gj] += ST[3 * gj + 1] / ST[3 * gj];
}

// The eigenvalue pass after one refinement step: residual of the refined double-precision
// vectors X against H (banded for the rlm meshes), column statistics, Rayleigh quotients.
static int rayleigh_pass(cudaStream_t st, int n, int band, int nb, const cplx* A, const cplx* X, double* W,
                         cplx* Res, double* ST, rlmb_context* ctx, long long* launches) {
    const unsigned gw = (unsigned)(((size_t)nb * n + 7) / 8);
    RLMB_CHUNK_PROF("k_ref_resid");
    if (launch_resid<cplx>(st, A, X, W, Res, n, band, nb) != cudaSuccess) return RLMB_ERR_CUDA;
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_colstats");
    k_ref_colstats<cplx><<<gw, 256, 0, st>>>(X, Res, ST, n, nb);
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_ref_diag");
    k_ref_rq<<<(unsigned)(((size_t)nb * n + 255) / 256), 256, 0, st>>>(ST, W, (size_t)nb * n);
    RLMB_CHUNK_LAUNCHED();
    return RLMB_OK;
}

template <int T>
static cudaError_t launch_tridiag(int phase, cudaStream_t st, const HeevPlan& p, int nb, const double* D, const double* E,
                                  double* W, double* Z, double* LU, int* info) {
    auto kern = phase == 1 ? k_tridiag<1, T> : k_tridiag<2, T>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem_tri);
    if (e != cudaSuccess) return e;
    const int subs = nb <= 148 && p.n > T && (phase == 1 || tri_columns(p.n) >= p.n) ? (p.n + T - 1) / T : 1;
    kern<<<dim3(nb, subs), T, p.smem_tri, st>>>(D, E, W, Z, LU, info, p.n);
    return cudaGetLastError();
}

static cudaLaunchConfig_t dc_merge_config(cudaLaunchAttribute* at, cudaStream_t st, int nb, int Y, size_t smem) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nb * Y);
    cfg.blockDim = dim3(DC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = Y;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}
// CTAs per matrix of k_dc_merge (its shared-memory attribute set): the most, up to 8, with which
// every cluster of the chunk runs at once.
static int dc_cluster(int nb, int n, size_t smem) {
    for (int Y = 8; Y > 1; --Y) {
        if (nb * Y > 148) continue;
        int active = 0;
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = dc_merge_config(at, 0, nb, Y, smem);
        if (cudaOccupancyMaxActiveClusters(&active, k_dc_merge, &cfg) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (active >= nb) return Y;
    }
    return 1;
}
static cudaError_t launch_dc_merge(cudaStream_t st, int nb, int Y, const double* E, const double* SC, double* W,
                                   const double* Qo, double* Qn, double* U, DcRot* ROT, int* info, int n, int S) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = dc_merge_config(at, st, nb, Y, dc_smem(S, n));
    return cudaLaunchKernelEx(&cfg, k_dc_merge, E, SC, W, Qo, Qn, U, ROT, info, n, S, Y);
}

// Eigenvalues W and eigenvectors Z (row-major) of the chunk's tridiagonals (D, E): bisection +
// inverse iteration (k_tridiag), or divide and conquer level by level (k_dc_*), ending in Zw.
static int tridiag_solve(rlmb_context* ctx, cudaStream_t st, const HeevPlan& p, int nb, unsigned char* base,
                         const double* Dw, const double* Ew, double* W, double* Zw, double* LUw, int* info,
                         long long* launches) {
    const int n = p.n;
    const size_t B = (size_t)nb;
    if (!p.dc) {
        // threads: the order rounded up to a power-of-two number of warps; above 256 chunks of few
        // matrices take two CTAs per matrix where the scratch has a column per eigenvector
        const auto go = n <= 32 ? launch_tridiag<32> : n <= 64 ? launch_tridiag<64> : n <= 128 ? launch_tridiag<128>
                                                                                            : launch_tridiag<TRI_THREADS>;
        RLMB_CHUNK_PROF("k_stebz");
        if (go(1, st, p, nb, Dw, Ew, W, Zw, LUw, info) != cudaSuccess) return RLMB_ERR_CUDA;
        RLMB_CHUNK_LAUNCHED();
        RLMB_CHUNK_PROF("k_stein");
        if (go(2, st, p, nb, Dw, Ew, W, Zw, LUw, info) != cudaSuccess) return RLMB_ERR_CUDA;
        RLMB_CHUNK_LAUNCHED();
        return RLMB_OK;
    }
    double* Q2 = reinterpret_cast<double*>(base + p.off_q2 * B);
    double* Uw = reinterpret_cast<double*>(base + p.off_u * B);
    DcRot* Rw = reinterpret_cast<DcRot*>(base + p.off_rot * B);
    double* SCw = reinterpret_cast<double*>(base + p.off_sc * B);
    const int levels = dc_levels(n);
    // ping-pong so that the last level writes Zw
    double* qa = levels % 2 ? Q2 : Zw;
    double* qb = levels % 2 ? Zw : Q2;
    size_t smem_max = 0;   // (not monotone in S: small levels run 16 groups per CTA)
    for (int S = 2; S / 2 < n; S *= 2) smem_max = std::max(smem_max, dc_smem(S, n));
    if (smem_max > 227 * 1024) return RLMB_ERR_ARG;
    if (cudaFuncSetAttribute(k_dc_merge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max) != cudaSuccess ||
        cudaFuncSetAttribute(k_dc_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DgTiles)) !=
            cudaSuccess)
        return RLMB_ERR_CUDA;
    const int Y = dc_cluster(nb, n, smem_max);
    RLMB_CHUNK_PROF("k_dc_merge");
    k_dc_init<<<nb, 256, 0, st>>>(Dw, Ew, W, qa, SCw, info, n);
    RLMB_CHUNK_LAUNCHED();
    for (int S = 2; S / 2 < n; S *= 2) {
        RLMB_CHUNK_PROF("k_dc_merge");
        if (launch_dc_merge(st, nb, Y, Ew, SCw, W, qa, qb, Uw, Rw, info, n, S) != cudaSuccess) return RLMB_ERR_CUDA;
        RLMB_CHUNK_LAUNCHED();
        if (S > DC_SMALL) {
            const int nsub = (n + S - 1) / S;
            const int mh = std::min(S / 2, n);
            const dim3 grid((mh + DG_BM - 1) / DG_BM, (std::min(S, n) + DG_BN - 1) / DG_BN, nb * nsub * 2);
            if (grid.z > 65535) return RLMB_ERR_ARG;
            RLMB_CHUNK_PROF("k_dc_gemm");
            k_dc_gemm<<<grid, 256, sizeof(DgTiles), st>>>(qa, Uw, qb, n, S, nsub);
            RLMB_CHUNK_LAUNCHED();
        }
        std::swap(qa, qb);
    }
    RLMB_CHUNK_PROF("k_dc_merge");
    k_dc_finish<<<std::min<size_t>(2048, (B * n + 255) / 256), 256, 0, st>>>(W, SCw, n, B * n);
    RLMB_CHUNK_LAUNCHED();
    return RLMB_OK;
}

// The kernel sequence of one eigensolve chunk of nb matrices of order n on scratch laid out
// per matrix as heev_plan describes (nb * plan.per bytes, no allocation).  Every scratch
// region is written by a kernel before any kernel reads it.  ctx (optional) receives the
// launch count and profile; otherwise *launches is advanced.
static int heev_chunk(rlmb_context* ctx, cudaStream_t st, const HeevPlan& p, cplx* A, double* W, int* info,
                      int nb, void* scratch, int nb2, long long* launches) {
    const int n = p.n;
    unsigned char* base = static_cast<unsigned char*>(scratch);
    const size_t B = (size_t)nb;
    double* Dw = reinterpret_cast<double*>(base + p.off_d * B);
    double* Ew = reinterpret_cast<double*>(base + p.off_e * B);
    double* Zw = reinterpret_cast<double*>(base + p.off_z * B);
    double* LUw = reinterpret_cast<double*>(base + p.off_lu * B);
    int* Qw = reinterpret_cast<int*>(base + p.off_q * B);
    const size_t nn = (size_t)n * n;
    if (p.jacobi) {
        if (p.smem_jac > 227 * 1024) return RLMB_ERR_ARG;
        if (cudaFuncSetAttribute(k_jacobi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem_jac) != cudaSuccess)
            return RLMB_ERR_CUDA;
        RLMB_CHUNK_PROF("k_jacobi");
        k_jacobi<<<nb, jacobi_threads(n, nb), p.smem_jac, st>>>(A, W, info, n);
        RLMB_CHUNK_LAUNCHED();
        return RLMB_OK;
    }
    if ((p.mixed ? hetrd_config<float>(p.m_tail, nb) : hetrd_config<double>(p.m_tail, nb)).smem > 227 * 1024 ||
        p.smem_tri > 227 * 1024)
        return RLMB_ERR_ARG;
    // (the last orders before that do not fit beside k_tridiag's own arrays: refused before any work)
    if (!p.dc && n > 6000 &&
        (cudaFuncSetAttribute(k_tridiag<1, TRI_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem_tri) != cudaSuccess ||
         cudaFuncSetAttribute(k_tridiag<2, TRI_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem_tri) != cudaSuccess)) {
        cudaGetLastError();
        return RLMB_ERR_CUDA;
    }
    if (!p.mixed) {
        cplx* TAUw = reinterpret_cast<cplx*>(base + p.off_tau * B);
        cplx* Xw = reinterpret_cast<cplx*>(base + p.off_x * B);
        cplx* Tw = reinterpret_cast<cplx*>(base + p.off_t * B);
        cplx* Wp = reinterpret_cast<cplx*>(base + p.off_w * B);
        if (int rc = tridiagonalise<double>(ctx, st, p, nb, A, Dw, Ew, TAUw,
                                            reinterpret_cast<cplx*>(base + p.off_pv * B), Qw, info, launches))
            return rc;
        if (int rc = tridiag_solve(ctx, st, p, nb, base, Dw, Ew, W, Zw, LUw, info, launches)) return rc;
        if (info && p.npanels > 0) {
            RLMB_CHUNK_PROF("k_stein");
            k_panel_abort_info<<<(nb + 255) / 256, 256, 0, st>>>(Qw, info, nb);
            RLMB_CHUNK_LAUNCHED();
        }
        if (int rc = back_transform<double>(ctx, st, p, nb, A, TAUw, Zw, Xw, Tw, Wp, launches)) return rc;
        if (cudaMemcpyAsync(A, Xw, B * nn * sizeof(cplx), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return RLMB_ERR_CUDA;
        return RLMB_OK;
    }
    cplxf* TAUw = reinterpret_cast<cplxf*>(base + p.off_tau * B);
    cplxf* As = reinterpret_cast<cplxf*>(base + p.off_a * B);
    cplxf* Xw = reinterpret_cast<cplxf*>(base + p.off_x * B);
    cplxf* Tw = reinterpret_cast<cplxf*>(base + p.off_t * B);
    cplxf* Wp = reinterpret_cast<cplxf*>(base + p.off_w * B);
    // refinement regions for nb2 matrices at a time, after the chunk's regions
    unsigned char* base2 = base + p.per * B;
    cplx* Res = reinterpret_cast<cplx*>(base2);
    cplx* X1 = reinterpret_cast<cplx*>(base2 + p.off2_x1 * (size_t)nb2);
    int2* CL = reinterpret_cast<int2*>(base + p.off_cl * B);
    cplx* YB = reinterpret_cast<cplx*>(base + p.off_y * B);
    double* MU = reinterpret_cast<double*>(base + p.off_mu * B);
    double* ST = reinterpret_cast<double*>(base + p.off_st * B);
    RLMB_CHUNK_PROF("k_herm_fill");
    k_herm_fill<<<dim3((n + 31) / 32, (n + 31) / 32, nb), dim3(32, 8), 0, st>>>(A, n);
    RLMB_CHUNK_LAUNCHED();
    RLMB_CHUNK_PROF("k_to_single");
    k_to_single<<<2048, 256, 0, st>>>(A, As, B * nn);
    RLMB_CHUNK_LAUNCHED();
    if (int rc = tridiagonalise<float>(ctx, st, p, nb, As, Dw, Ew, TAUw,
                                       reinterpret_cast<cplxf*>(base + p.off_pv * B), Qw, info, launches))
        return rc;
    if (int rc = tridiag_solve(ctx, st, p, nb, base, Dw, Ew, W, Zw, LUw, info, launches)) return rc;
    if (info && p.npanels > 0) {
        RLMB_CHUNK_PROF("k_stein");
        k_panel_abort_info<<<(nb + 255) / 256, 256, 0, st>>>(Qw, info, nb);
        RLMB_CHUNK_LAUNCHED();
    }
    if (int rc = back_transform<float>(ctx, st, p, nb, As, TAUw, Zw, Xw, Tw, Wp, launches)) return rc;
    // refinement, nb2 matrices at a time: the single-precision copy of H is free now and
    // holds F.  Step 1 starts from the single-precision vectors, step 2 from step 1's double
    // vectors (X1); the last step writes the caller's buffer (every step's residual reads H
    // first).
    if (nb2 < 1) return RLMB_ERR_ARG;
    for (int m0 = 0; m0 < nb; m0 += nb2) {
        const int ns = std::min(nb2, nb - m0);
        const size_t o = (size_t)m0 * nn, on = (size_t)m0 * n;
        cplx* Am = A + o;
        double* Wm = W + on;
        cplxf* Fm = As + o;
        int2* CLm = CL + on;
        cplx* YBm = YB + (size_t)m0 * n * RF_KMAX;
        double* MUm = MU + on;
        double* STm = ST + 3 * on;
        if (int rc = refine_step<cplxf>(ctx, st, n, p.band, ns, Am, Xw + o, Wm, Res, Fm, CLm, YBm, MUm, STm,
                                        p.refine_steps >= 2 || p.rq ? X1 : Am, launches))
            return rc;
        if (p.rq) {   // eigenvalues as Rayleigh quotients of the step-1 vectors, then the vectors out
            if (int rc = rayleigh_pass(st, n, p.band, ns, Am, X1, Wm, Res, STm, ctx, launches)) return rc;
            if (cudaMemcpyAsync(Am, X1, (size_t)ns * nn * sizeof(cplx), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
                return RLMB_ERR_CUDA;
        }
        if (p.refine_steps >= 2)
            if (int rc = refine_step<cplx>(ctx, st, n, p.band, ns, Am, X1, Wm, Res, Fm, CLm, YBm, MUm, STm, Am,
                                           launches))
                return rc;
    }
    return RLMB_OK;
}
#undef RLMB_CHUNK_LAUNCHED
#undef RLMB_CHUNK_PROF

int heev_chunk_on_scratch(cudaStream_t st, cplx* A, double* W, int* info, int n, int nb, void* scratch,
                          long long* launches) {
    return heev_chunk(nullptr, st, noalloc_plan(n), A, W, info, nb, scratch, 0, launches);
}

}  // namespace rlmb

using namespace rlmb;

// ----------------------------------------------------------------------- autotuner
// Per context, per (order, precision): the launch choices of HeevTune picked by timing every
// feasible candidate -- unblocked or blocked reduction (from order 128), panels by the built-in
// rules or of 512 threads, SM-resident or GEMM back-transformation, 64- or 128-reflector blocks and 64- or
// 128-row X-update tiles (double precision) of the latter, either tridiagonal solver (bisection +
// inverse iteration, or divide and conquer), and up to order JAC_MAX_N the batched Jacobi solver -- on copies of up to 2 x SMs of the call's own matrices (at most 2 GB of them),
// each candidate run twice and timed the second time with CUDA events.  Orders
// TUNE_MIN_N .. TUNE_MAX_N are tuned; others keep the built-in choices.
struct TuneEntry {
    HeevTune t;
    double ms_per_matrix;
};
typedef std::map<std::pair<int, int>, TuneEntry> TuneCache;
static TuneCache& tune_cache(rlmb_context* ctx) {
    if (!ctx->tune) ctx->tune = new TuneCache();
    return *static_cast<TuneCache*>(ctx->tune);
}
void rlmb::tune_free(rlmb_context* ctx) {
    delete static_cast<TuneCache*>(ctx->tune);
    ctx->tune = nullptr;
}

static std::vector<HeevTune> tune_candidates(int n, bool mixed) {
    std::vector<HeevTune> out;
    if (n <= JAC_MAX_N) {
        HeevTune t;
        t.jacobi = 1;
        out.push_back(t);
    }
    for (int blocked = 0; blocked <= 1; ++blocked) {
        if (blocked && n < 128) continue;
        for (int gemm = 0; gemm <= 1; ++gemm)
            for (int nt : {0, 512}) {   // panels by the rules, or 512 threads per matrix
                if (!blocked && nt != 512) continue;   // no panels: one entry
                for (int xt : {64, 128})
                    for (int bs : {64, 128}) {
                        if ((!gemm || mixed) && xt == 128) continue;
                        if (!gemm && bs == 128) continue;
                        HeevTune t;
                        t.jacobi = 0;
                        t.blocked = blocked;
                        t.gemm_bt = gemm;
                        t.panel_nt = blocked ? nt : 0;
                        t.xtile = gemm && !mixed ? xt : 0;
                        t.bt_nb = gemm ? bs : 0;
                        const HeevPlan p = heev_plan(n, mixed, 2, -1, t);
                        if (!gemm && !p.small_bt) continue;   // register back-transformation does not fit
                        for (int dc = 0; dc <= (n <= DC_MAX_N ? 1 : 0); ++dc) {   // tridiagonal solver
                            t.dc = dc;
                            out.push_back(t);
                        }
                    }
            }
    }
    return out;
}

static int autotune(rlmb_context* ctx, int n, bool mixed, int refine_steps, int band, const cplx* A, int batch,
                    HeevTune* best) {
    int dev = 0, sms = 148;
    RLMB_CUDA_TRY(cudaGetDevice(&dev));
    RLMB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const size_t nn = (size_t)n * n;
    const size_t cap = std::min<size_t>((size_t)2 * sms, ((size_t)2 << 30) / (nn * sizeof(cplx)));
    const int tb = (int)std::max<size_t>(1, std::min<size_t>((size_t)batch, cap));
    const std::vector<HeevTune> cands = tune_candidates(n, mixed);
    size_t per = 0;
    for (const HeevTune& t : cands) {
        const HeevPlan pl = heev_plan(n, mixed, refine_steps, band, t);
        per = std::max(per, pl.per + pl.per2);
    }
    void* buf = nullptr;
    const size_t work = (size_t)tb * (2 * nn * sizeof(cplx) + n * sizeof(double) + sizeof(int)) + 1024;
    if (cudaMalloc(&buf, work) != cudaSuccess) {
        cudaGetLastError();
        return RLMB_ERR_ALLOC;
    }
    if (int rc = ensure_workspace(ctx, (size_t)tb * per)) {
        cudaFree(buf);
        return rc;
    }
    cplx* src = static_cast<cplx*>(buf);
    cplx* wk = src + (size_t)tb * nn;
    double* w = reinterpret_cast<double*>(wk + (size_t)tb * nn);
    int* info = reinterpret_cast<int*>(w + (size_t)tb * n);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    int rc = RLMB_OK;
    if (cudaMemcpyAsync(src, A, (size_t)tb * nn * sizeof(cplx), cudaMemcpyDeviceToDevice, ctx->stream) != cudaSuccess ||
        cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)
        rc = RLMB_ERR_CUDA;
    double best_ms = 1e300;
    long long unused = 0;
    void* prof = ctx->prof;
    ctx->prof = nullptr;   // tuning launches stay out of the caller's profile
    for (size_t c = 0; c < cands.size() && rc == RLMB_OK; ++c) {
        const HeevPlan p = heev_plan(n, mixed, refine_steps, band, cands[c]);
        float ms = 0.f;
        for (int rep = 0; rep < 2 && rc == RLMB_OK; ++rep) {
            if (cudaMemcpyAsync(wk, src, (size_t)tb * nn * sizeof(cplx), cudaMemcpyDeviceToDevice, ctx->stream) !=
                    cudaSuccess ||
                cudaEventRecord(e0, ctx->stream) != cudaSuccess) {
                rc = RLMB_ERR_CUDA;
                break;
            }
            rc = heev_chunk(ctx, ctx->stream, p, wk, w, info, tb, ctx->ws, tb, &unused);
            if (rc == RLMB_OK && (cudaEventRecord(e1, ctx->stream) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
                                  cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess))
                rc = RLMB_ERR_CUDA;
        }
        if (rc == RLMB_OK && ms / tb < best_ms) {
            best_ms = ms / tb;
            *best = cands[c];
        }
    }
    ctx->prof = prof;
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaStreamSynchronize(ctx->stream);
    cudaFree(buf);
    if (rc == RLMB_OK) tune_cache(ctx)[{n, mixed ? 1 : 0}] = TuneEntry{*best, best_ms};
    return rc;
}

// Refinement steps handed to heev_plan: 1 or 2, or 3 for one step followed by the eigenvalue pass.
static int heev_steps(const rlmb_context* ctx) { return ctx->refine_steps == 1 && ctx->rq_pass ? 3 : ctx->refine_steps; }

bool rlmb::heev_mesh_differs(rlmb_context* ctx, int n) {
    const TuneCache& tc = tune_cache(ctx);
    const auto it = tc.find({n, ctx->precision == RLMB_PRECISION_MIXED ? 1 : 0});
    return n > JAC_MESH_MAX && n <= JAC_DEFAULT_MAX && (it == tc.end() || it->second.t.jacobi < 0);
}

// The batched eigensolve of rlmb_heevd_batched with a structure hint: band >= 0 declares every
// matrix a cyclic band of that half-bandwidth (the rlm Hamiltonian), which the mixed mode's
// refinement uses for its residual; band < 0 is a dense matrix.
int rlmb::heevd_batched_band(rlmb_context* ctx, double* d_a, double* d_w, int n, int batch, int* d_info, int band,
                             bool mesh) {
    if (!ctx || !d_a || !d_w || n <= 0 || batch < 0) return RLMB_ERR_ARG;
    if (batch == 0) return RLMB_OK;
    RLMB_CUDA_TRY(cudaSetDevice(ctx->device));
    bool mixed = ctx->precision == RLMB_PRECISION_MIXED;
    HeevTune tune;
    {
        TuneCache& tc = tune_cache(ctx);
        auto it = tc.find({n, mixed ? 1 : 0});
        if (it != tc.end()) {
            tune = it->second.t;
        } else if (ctx->autotune && !ctx->frozen && n >= TUNE_MIN_N && n <= TUNE_MAX_N) {
            if (int rc = autotune(ctx, n, mixed, heev_steps(ctx), band, reinterpret_cast<const cplx*>(d_a), batch, &tune))
                return rc;
        }
    }
    // a mesh solve takes the faster solver (its results do not see the vectors' phases) where the
    // batched eigensolver runs Jacobi, and like Jacobi in double precision in either mode
    if (mesh && tune.jacobi < 0 && n <= JAC_DEFAULT_MAX) {
        tune.jacobi = n <= JAC_MESH_MAX;
        mixed = false;
    }
    const HeevPlan plan = heev_plan(n, mixed, heev_steps(ctx), band, tune);
    const size_t per = plan.per;
    // workspace: 8 GB, or for large orders enough for two resident matrices per SM (one
    // CTA each in k_tridiag); where the workspace has to grow for that, capped at 60 % of the
    // free memory
    const size_t per2 = plan.per2;
    size_t budget = std::max<size_t>(std::max<size_t>((size_t)8 << 30, 2 * 148 * (per + per2)), per + per2);
    if (ctx->frozen) budget = std::max<size_t>(per + per2, ctx->ws_bytes);   // capture: the workspace as sized before
    size_t nb2 = 0, chunk = 0;
    auto cut = [&]() {
        // the refinement regions take up to an eighth of the budget (its GEMMs fill the GPU from a
        // few matrices on); the chunk -- all of whose matrices the one-CTA-per-matrix reduction and
        // tridiagonal kernels run at once -- takes the rest
        nb2 = per2 ? std::max<size_t>(1, std::min<size_t>((size_t)batch, budget / 8 / per2)) : 0;
        chunk = std::max<size_t>(1, std::min<size_t>((budget - nb2 * per2) / per, (size_t)batch));
        chunk = std::min<size_t>(chunk, 65535);   // grid y / z extent of the per-matrix launches
        if (!plan.small_bt) chunk = std::min<size_t>(chunk, 65535 / std::max(plan.nblkbt, 1));   // (matrix, block) batches
        if (plan.dc) chunk = std::min<size_t>(chunk, dc_max_chunk(n));   // (matrix, subproblem, half) GEMM batches
        // equal chunks: a short last chunk would leave most SMs idle in the one-CTA-per-matrix kernels
        const size_t nchunks = (batch + chunk - 1) / chunk;
        chunk = (batch + nchunks - 1) / nchunks;
        if (per2) {   // equal refinement sub-chunks too
            nb2 = std::min(nb2, chunk);
            const size_t nsub = (chunk + nb2 - 1) / nb2;
            nb2 = (chunk + nsub - 1) / nsub;
        }
    };
    cut();
    if (!ctx->frozen && chunk * per + nb2 * per2 > ctx->ws_bytes) {
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
            cudaGetLastError();
            free_b = (size_t)8 << 30;
        }
        budget = std::max<size_t>(std::min<size_t>(budget, free_b / 10 * 6 + ctx->ws_bytes), per + per2);
        cut();
    }
    if (int rc = ensure_workspace(ctx, chunk * per + nb2 * per2)) return rc;
    const size_t nn = (size_t)n * n;
    long long unused = 0;
    for (size_t b0 = 0; b0 < (size_t)batch; b0 += chunk) {
        const int nb = (int)std::min(chunk, (size_t)batch - b0);
        if (int rc = heev_chunk(ctx, ctx->stream, plan, reinterpret_cast<cplx*>(d_a) + b0 * nn, d_w + b0 * n,
                                d_info ? d_info + b0 : nullptr, nb, ctx->ws, (int)nb2, &unused))
            return rc;
    }
    return RLMB_OK;
}

extern "C" int rlmb_heevd_batched(rlmb_context* ctx, double* d_a, double* d_w, int n, int batch, int* d_info) {
    return rlmb::heevd_batched_band(ctx, d_a, d_w, n, batch, d_info, -1, false);
}

extern "C" int rlmb_set_autotune(rlmb_context* ctx, int on) {
    if (!ctx) return RLMB_ERR_ARG;
    ctx->autotune = on ? 1 : 0;
    return RLMB_OK;
}

extern "C" int rlmb_heev_config(rlmb_context* ctx, int n, int precision, int* blocked, int* gemm_bt,
                                int* panel_threads, int* x_tile, int* bt_block, double* ms_per_matrix) {
    if (!ctx || n <= 0 || (precision != RLMB_PRECISION_FP64 && precision != RLMB_PRECISION_MIXED)) return RLMB_ERR_ARG;
    auto& tc = tune_cache(ctx);
    auto it = tc.find({n, precision});
    HeevTune t;
    double ms = 0.0;
    if (it != tc.end()) {
        t = it->second.t;
        ms = it->second.ms_per_matrix;
    }
    const HeevPlan p = heev_plan(n, precision == RLMB_PRECISION_MIXED, 2, -1, t);
    if (blocked) *blocked = p.npanels > 0;
    if (gemm_bt) *gemm_bt = !p.small_bt;
    if (panel_threads) *panel_threads = p.panel_nt;
    if (x_tile) *x_tile = p.xtile == 128 ? 128 : 64;
    if (bt_block) *bt_block = p.bt_nb;
    if (ms_per_matrix) *ms_per_matrix = ms;
    return it != tc.end() ? 1 : 0;
}

extern "C" int rlmb_set_heev_config(rlmb_context* ctx, int n, int precision, int blocked, int gemm_bt,
                                    int panel_threads, int x_tile, int bt_block) {
    if (!ctx || n <= 0 || (precision != RLMB_PRECISION_FP64 && precision != RLMB_PRECISION_MIXED) || blocked < -1 ||
        blocked > 1 || gemm_bt < -1 || gemm_bt > 1 || (panel_threads != 0 && panel_threads != 256 && panel_threads != 512) ||
        (x_tile != 0 && x_tile != 64 && x_tile != 128) || (bt_block != 0 && bt_block != 64 && bt_block != 128))
        return RLMB_ERR_ARG;
    auto& tc = tune_cache(ctx);
    auto it = tc.find({n, precision});
    HeevTune t;
    if (it != tc.end()) {   // the solver and panel-queue choices are set separately
        t.jacobi = it->second.t.jacobi;
        t.dc = it->second.t.dc;
        t.queue_nt = it->second.t.queue_nt;
        t.panel_w = it->second.t.panel_w;
    }
    t.blocked = blocked;
    t.gemm_bt = gemm_bt;
    t.panel_nt = panel_threads;
    t.xtile = x_tile;
    t.bt_nb = bt_block;
    tc[{n, precision}] = TuneEntry{t, 0.0};
    return RLMB_OK;
}

extern "C" int rlmb_set_heev_solver(rlmb_context* ctx, int n, int precision, int solver) {
    if (!ctx || n <= 0 || (precision != RLMB_PRECISION_FP64 && precision != RLMB_PRECISION_MIXED) ||
        (solver != RLMB_SOLVER_AUTO && solver != RLMB_SOLVER_HOUSEHOLDER && solver != RLMB_SOLVER_JACOBI) ||
        (solver == RLMB_SOLVER_JACOBI && n > JAC_MAX_N))
        return RLMB_ERR_ARG;
    auto& tc = tune_cache(ctx);
    auto it = tc.find({n, precision});
    TuneEntry e{HeevTune{}, 0.0};
    if (it != tc.end()) e = it->second;
    e.t.jacobi = solver == RLMB_SOLVER_AUTO ? -1 : solver == RLMB_SOLVER_JACOBI ? 1 : 0;
    tc[{n, precision}] = e;
    return RLMB_OK;
}

extern "C" int rlmb_set_panel_queue(rlmb_context* ctx, int n, int precision, int threads) {
    if (!ctx || n <= 0 || (precision != RLMB_PRECISION_FP64 && precision != RLMB_PRECISION_MIXED) ||
        (threads != 0 && threads != 256 && threads != 512))
        return RLMB_ERR_ARG;
    auto& tc = tune_cache(ctx);
    auto it = tc.find({n, precision});
    TuneEntry e{HeevTune{}, 0.0};
    if (it != tc.end()) e = it->second;
    e.t.queue_nt = threads;
    tc[{n, precision}] = e;
    return RLMB_OK;
}

extern "C" int rlmb_set_panel_width(rlmb_context* ctx, int n, int precision, int width) {
    if (!ctx || n <= 0 || (precision != RLMB_PRECISION_FP64 && precision != RLMB_PRECISION_MIXED) ||
        (width != 0 && width != 16 && width != 32))
        return RLMB_ERR_ARG;
    auto& tc = tune_cache(ctx);
    auto it = tc.find({n, precision});
    TuneEntry e{HeevTune{}, 0.0};
    if (it != tc.end()) e = it->second;
    e.t.panel_w = width;
    tc[{n, precision}] = e;
    return RLMB_OK;
}

extern "C" int rlmb_set_tridiag_solver(rlmb_context* ctx, int n, int precision, int solver) {
    if (!ctx || n <= 0 || (precision != RLMB_PRECISION_FP64 && precision != RLMB_PRECISION_MIXED) ||
        (solver != RLMB_TRIDIAG_AUTO && solver != RLMB_TRIDIAG_BISECTION && solver != RLMB_TRIDIAG_DC) ||
        (solver == RLMB_TRIDIAG_DC && n > DC_MAX_N))
        return RLMB_ERR_ARG;
    auto& tc = tune_cache(ctx);
    auto it = tc.find({n, precision});
    TuneEntry e{HeevTune{}, 0.0};
    if (it != tc.end()) e = it->second;
    e.t.dc = solver == RLMB_TRIDIAG_AUTO ? -1 : solver == RLMB_TRIDIAG_DC ? 1 : 0;
    tc[{n, precision}] = e;
    return RLMB_OK;
}

extern "C" int rlmb_tridiag_solver(rlmb_context* ctx, int n, int precision, int* solver) {
    if (!ctx || n <= 0 || !solver || (precision != RLMB_PRECISION_FP64 && precision != RLMB_PRECISION_MIXED))
        return RLMB_ERR_ARG;
    auto& tc = tune_cache(ctx);
    auto it = tc.find({n, precision});
    const HeevTune t = it != tc.end() ? it->second.t : HeevTune{};
    *solver = heev_plan(n, precision == RLMB_PRECISION_MIXED, 2, -1, t).dc ? RLMB_TRIDIAG_DC : RLMB_TRIDIAG_BISECTION;
    return RLMB_OK;
}

extern "C" int rlmb_heev_solver(rlmb_context* ctx, int n, int precision, int* solver) {
    if (!ctx || n <= 0 || !solver || (precision != RLMB_PRECISION_FP64 && precision != RLMB_PRECISION_MIXED))
        return RLMB_ERR_ARG;
    auto& tc = tune_cache(ctx);
    auto it = tc.find({n, precision});
    const HeevTune t = it != tc.end() ? it->second.t : HeevTune{};
    *solver = heev_plan(n, precision == RLMB_PRECISION_MIXED, 2, -1, t).jacobi ? RLMB_SOLVER_JACOBI
                                                                              : RLMB_SOLVER_HOUSEHOLDER;
    return RLMB_OK;
}

// Batched complex GEMM C = A B (column-major complex128, A m x k, B k x n, C m x n, matrices
// packed back to back) on either engine: the FP64 tensor path (DMMA) or the tcgen05 TF32
// tensor cores with split operands (FP32-class accuracy).
extern "C" int rlmb_zgemm_batched(rlmb_context* ctx, const double* d_a, const double* d_b, double* d_c, int m,
                                  int n, int k, int batch, int engine) {
    if (!ctx || (k > 0 && (!d_a || !d_b)) || !d_c || m <= 0 || n <= 0 || k < 0 || batch < 0 ||
        (engine != RLMB_GEMM_FP64 && engine != RLMB_GEMM_TF32X3 && engine != RLMB_GEMM_TF32X3_F64ACC))
        return RLMB_ERR_ARG;
    if (batch == 0) return RLMB_OK;
    if (batch > 65535) return RLMB_ERR_ARG;
    RLMB_CUDA_TRY(cudaSetDevice(ctx->device));
    const cplx* A = reinterpret_cast<const cplx*>(d_a);
    const cplx* B = reinterpret_cast<const cplx*>(d_b);
    cplx* Cm = reinterpret_cast<cplx*>(d_c);
    const OpColA<cplx, cplx> la{A, m, (size_t)m * k};
    const OpColB<cplx, cplx> lb{B, k, (size_t)k * n};
    const EpStore<cplx> ep{Cm, m, (size_t)m * n};
    if (engine == RLMB_GEMM_TF32X3_F64ACC && k > 0) {
        const size_t per = tma_plane_bytes(m, n, k);
        if (int rc = ensure_tma_planes(ctx, std::max(per, std::min((size_t)batch * per, (size_t)4 << 30)))) return rc;
    }
    prof_begin(ctx, engine == RLMB_GEMM_FP64 ? "k_zgemm_dmma" : engine == RLMB_GEMM_TF32X3 ? "k_zgemm_tc" : "k_zgemm_tma");
    const cudaError_t e =
        engine == RLMB_GEMM_FP64     ? launch_zgemm<cplx, 64>(ctx->stream, la, lb, ep, m, n, k, batch)
        : engine == RLMB_GEMM_TF32X3 ? launch_zgemm_tc<cplx>(ctx->stream, la, lb, ep, m, n, k, batch)
                                     : launch_zgemm_tma<cplx>(ctx->stream, la, lb, ep, m, n, k, batch, ctx->tws, ctx->tws_bytes);
    prof_end(ctx);
    ctx->launches++;
    return e == cudaSuccess ? RLMB_OK : RLMB_ERR_CUDA;
}

// Number of tcgen05 GEMM tiles whose bounded mbarrier waits ran out since the library was
// loaded on the current device (synchronises the device).
extern "C" int rlmb_tc_fault_count(rlmb_context* ctx, int* count) {
    if (!ctx || !count) return RLMB_ERR_ARG;
    RLMB_CUDA_TRY(cudaSetDevice(ctx->device));
    RLMB_CUDA_TRY(cudaDeviceSynchronize());
    RLMB_CUDA_TRY(cudaMemcpyFromSymbol(count, g_tc_fault, sizeof(int)));
    return RLMB_OK;
}
