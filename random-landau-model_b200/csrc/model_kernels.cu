// Assembly and Chern-step kernels of the rlm and hlm twist-mesh pipelines (sm_100a, FP64).
#include "model_kernels.cuh"
#include "small_eig.cuh"
#include "zgemm.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>

namespace rlmb {

// ======================================================================= rlm
// V_mn (rlm/matrix_coefficients.cpp:27-44): the phase of impurity i factorises,
// e^{-i 2pi((m-o)x + (n-o)y)} = e^{-i 2pi (m-o) x} e^{-i 2pi (n-o) y}, so V is a
// (dim x N_imp) by (N_imp x dim) complex product.  One CTA computes a 32x32 tile of
// (m, n) over one chunk of impurities; partial tiles are summed in a fixed order by
// k_vmn_reduce (deterministic).
static constexpr int VMN_T = 32;       // output tile edge
static constexpr int VMN_KC = 32;      // impurities staged per step
static constexpr int VMN_KSPLIT = 2048;  // impurities per CTA at most
// Impurities per CTA: 2048 where the tiles of one sample fill the GPU with that, down to 64 where
// they are few (a CTA's time is its chain of staged steps: n_phi = 129, 2 samples, 4 tiles each,
// 200 us with 2048, 17 us now; n_phi = 16, one tile, 29 us, now 11).  It depends on the
// sample's sizes alone, so that a sample's sums are the same in any batch.
static int vmn_chunk(int nimp, int dim) {
    const int nt = (dim + VMN_T - 1) / VMN_T, want = (148 + nt * nt - 1) / (nt * nt);
    const int chunk = ((nimp + want - 1) / want + VMN_KC - 1) / VMN_KC * VMN_KC;
    return std::min(std::max(chunk, 64), VMN_KSPLIT);
}

__global__ void __launch_bounds__(256)
k_vmn_partial(const double* __restrict__ X, const double* __restrict__ Y,
              const double* __restrict__ S, int nimp, int dim, int off_head, int nsplit, int chunk,
              cplx* __restrict__ partial) {
    __shared__ cplx ex[VMN_T][VMN_KC + 1];   // s_i e^{-i 2pi (m-o) x_i}
    __shared__ cplx ey[VMN_T][VMN_KC + 1];   // e^{-i 2pi (n-o) y_i}
    const int tid = threadIdx.x;
    const int m0 = blockIdx.x * VMN_T, n0 = blockIdx.y * VMN_T;
    const int sample = blockIdx.z / nsplit, split = blockIdx.z % nsplit;
    const double* x = X + (size_t)sample * nimp;
    const double* y = Y + (size_t)sample * nimp;
    const double* s = S + (size_t)sample * nimp;
    const int i_begin = split * chunk, i_end = min(nimp, i_begin + chunk);
    // thread owns outputs (m0 + tm + 8*u, n0 + tn) for u = 0..3
    const int tn = tid & 31, tm = tid >> 5;
    cplx acc[4] = {mk(0, 0), mk(0, 0), mk(0, 0), mk(0, 0)};
    for (int ib = i_begin; ib < i_end; ib += VMN_KC) {
        __syncthreads();
        for (int idx = tid; idx < VMN_T * VMN_KC; idx += 256) {
            const int r = idx / VMN_KC, k = idx % VMN_KC;
            const int i = ib + k;
            cplx vx = mk(0, 0), vy = mk(0, 0);
            if (i < i_end) {
                double sn, cs;
                sincospi(2.0 * (double)(m0 + r - off_head) * x[i], &sn, &cs);
                vx = mk(cs * s[i], -sn * s[i]);
                sincospi(2.0 * (double)(n0 + r - off_head) * y[i], &sn, &cs);
                vy = mk(cs, -sn);
            }
            ex[r][k] = vx;
            ey[r][k] = vy;
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < VMN_KC; ++k) {
            const cplx b = ey[tn][k];
#pragma unroll
            for (int u = 0; u < 4; ++u) cfma(acc[u], ex[tm + 8 * u][k], b);
        }
    }
    for (int u = 0; u < 4; ++u) {
        const int m = m0 + tm + 8 * u, n = n0 + tn;
        if (m < dim && n < dim)
            partial[(((size_t)sample * nsplit + split) * dim + m) * dim + n] = acc[u];
    }
}

__global__ void k_vmn_reduce(const cplx* __restrict__ partial, const cplx* __restrict__ coeff_mn,
                             int dim, int nsplit, int nsamples, cplx* __restrict__ vmn) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t per = (size_t)dim * dim;
    if (idx >= per * nsamples) return;
    const size_t sample = idx / per, mn = idx % per;
    cplx sum = mk(0, 0);
    for (int k = 0; k < nsplit; ++k) sum = cadd(sum, partial[(sample * nsplit + k) * per + mn]);
    vmn[idx] = cmul(sum, coeff_mn[mn]);
}

// Samples whose partial sums are held at once: 256 MB of them (a sample of few tiles has up to 37
// splits), within the grid's z extent, at least one.
static int vmn_group(int nsplit, int nsamples, int dim) {
    const size_t sample = (size_t)nsplit * dim * dim * sizeof(cplx);
    const size_t most = std::min<size_t>(((size_t)256 << 20) / sample, 65535 / nsplit);
    return (int)std::max<size_t>(1, std::min<size_t>(most, nsamples));
}
int launch_rlm_potential(rlmb_context* ctx, const double* x, const double* y, const double* s,
                         int nimp, int nsamples, const cplx* coeff_mn, int dim, int off_head,
                         cplx* partial_ws, cplx* vmn) {
    const int chunk = vmn_chunk(nimp, dim), nsplit = (nimp + chunk - 1) / chunk;
    const int nt = (dim + VMN_T - 1) / VMN_T;
    const int per = vmn_group(nsplit, nsamples, dim);
    for (int s0 = 0; s0 < nsamples; s0 += per) {
        const int ns = std::min(per, nsamples - s0);
        const size_t o = (size_t)s0 * nimp, dd = (size_t)dim * dim;
        prof_begin(ctx, "k_vmn_partial");
        k_vmn_partial<<<dim3(nt, nt, ns * nsplit), 256, 0, ctx->stream>>>(x + o, y + o, s + o, nimp, dim, off_head, nsplit,
                                                                         chunk, partial_ws);
        RLMB_LAUNCHED(ctx);
        prof_begin(ctx, "k_vmn_reduce");
        k_vmn_reduce<<<(unsigned)((dd * ns + 255) / 256), 256, 0, ctx->stream>>>(partial_ws, coeff_mn, dim, nsplit, ns,
                                                                                vmn + s0 * dd);
        RLMB_LAUNCHED(ctx);
    }
    return RLMB_OK;
}
size_t rlm_potential_ws_elems(int nimp, int nsamples, int dim) {
    const int chunk = vmn_chunk(nimp, dim), nsplit = (nimp + chunk - 1) / chunk;
    return (size_t)vmn_group(nsplit, nsamples, dim) * nsplit * dim * dim;
}

// H(theta_1, theta_2) (rlm/hamiltonian_rlm_cpu.cpp:14-48).  For k >= j:
//   F[j][k] = sum_m conj(c_t2[m]) c_jm[j][m] * sum_{n in {o+k-j, o+k-j-N}} V[m][n] c_t1[n]
// stored row-major as the reference does: buf[j*N+k] = F[j][k] (k > j), conj(F[j][j]) on
// the diagonal, buf[k*N+j] = conj(F[j][k]); zero outside the cyclic band.
//
// The sum over m does not see theta_1: with
//   S_t2[j][n] = sum_m conj(c_t2[m]) c_jm[j][m] V[m][n]
// every entry is F[j][k] = sum_{n} S_t2[j][n] c_t1[n] (one or two terms).  S is one complex
// N x dim by dim x dim product per theta_2 (the FP64 tensor-path GEMM engine), shared by all
// theta_1, and the fill is bound by writing H.  Evaluating the m sum per entry and k-point
// took 8.9 ms at n_phi = 512, g = 16, 2 samples (2.4 GB of H); this form takes 0.50 ms (4.8 TB/s of H).
struct ThetaList {   // theta_2 indices of one group, ascending
    static constexpr int MAX = 64;
    int n;
    int t2[MAX];
};

// A(j, m) = conj(c_t2[m]) c_jm[j][m], batch z = sample * list.n + slot
struct OpThetaA {
    static constexpr bool RFAST = false;
    const cplx* cmt;
    const cplx* cjm;
    int dim;
    ThetaList list;
    __device__ __forceinline__ cplx elem(size_t z, int j, int m) const {
        const int t2 = list.t2[z % list.n];
        return cmulc(cmt[(size_t)t2 * dim + m], cjm[(size_t)j * dim + m]);
    }
};
// B(m, n) = V[m][n] of the batch's sample
struct OpVmnB {
    static constexpr bool KFAST = false;
    const cplx* vmn;
    int dim, per;
    __device__ __forceinline__ cplx elem(size_t z, int m, int n) const {
        return vmn[((size_t)(z / per) * dim + m) * dim + n];
    }
};
// S[z][j][n], n contiguous
struct EpRowMajor {
    cplx* s;
    int rows, cols;
    __device__ __forceinline__ bool skip(int, int, int) const { return false; }
    __device__ __forceinline__ void store(size_t z, int j, int n, cplx acc) const {
        s[(z * rows + j) * cols + n] = acc;
    }
};

// One warp per row j of a k-point's buffer, lanes along k.  kp0: first k-point of the launch;
// a k-point whose theta_2 is not in the list belongs to another launch.
__global__ void __launch_bounds__(256)
k_rlm_assemble(const cplx* __restrict__ S, const cplx* __restrict__ cmt, const int* __restrict__ t1s,
               const int* __restrict__ t2s, const __grid_constant__ ThetaList list, int n_phi, int dim, int o,
               int kpts_per_sample, int n_theta, int kp0, cplx* __restrict__ H) {
    const int kp = kp0 + blockIdx.y;
    // (without lists: the whole mesh, theta_2 fastest)
    const int mesh = t2s ? 0 : kp % kpts_per_sample, t1 = t2s ? t1s[kp] : mesh / n_theta, t2 = t2s ? t2s[kp] : mesh % n_theta;
    int lo = 0, hi = list.n - 1;   // the slot of t2
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (list.t2[mid] < t2) lo = mid + 1;
        else hi = mid;
    }
    if (list.t2[lo] != t2) return;
    const int j = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (j >= n_phi) return;
    const int sample = blockIdx.y / kpts_per_sample;
    const cplx* s = S + ((size_t)sample * list.n + lo) * n_phi * dim;
    const cplx* c1 = cmt + (size_t)t1 * dim;
    cplx* h = H + ((size_t)kp * n_phi + j) * n_phi;
    for (int k = threadIdx.x & 31; k < n_phi; k += 32) {
        const int row = min(j, k), delta = max(j, k) - row;
        const cplx* sr = s + (size_t)row * dim;
        cplx f = mk(0, 0);
        if (delta <= o) cfma(f, sr[o + delta], c1[o + delta]);
        if (n_phi - delta <= o) cfma(f, sr[o + delta - n_phi], c1[o + delta - n_phi]);
        h[k] = k > j ? f : cconj(f);
    }
}

// theta_2 slabs of S held at once: at most 64 per sample and 256 MB in all, at least one.
static size_t rlm_slab_cap(int n_phi, int dim) {
    const size_t slab = (size_t)n_phi * dim * sizeof(cplx);
    return std::max<size_t>(1, ((size_t)256 << 20) / slab);
}
size_t rlm_assemble_ws_elems(int n_phi, int dim, int nsamples, int n_t2) {
    const size_t want = (size_t)nsamples * std::min(n_t2, (int)ThetaList::MAX);
    return std::min(want, rlm_slab_cap(n_phi, dim)) * n_phi * dim;
}

// k-points kp = 0 .. count-1 (kpts_per_sample consecutive ones per sample, angles d_t1 / d_t2, or
// without these the n_t2 x n_t2 mesh of every sample);
// uniq_t2: the n_t2 distinct theta_2 indices among them, ascending (host); ws:
// rlm_assemble_ws_elems(n_phi, dim, samples, n_t2) elements.
int launch_rlm_assemble(rlmb_context* ctx, const cplx* vmn, const cplx* cmt, const cplx* cjm,
                        const int* d_t1, const int* d_t2, int count, int kpts_per_sample,
                        int n_phi, int dim, int o, const int* uniq_t2, int n_t2, cplx* ws, cplx* H) {
    const int nsamples = (count + kpts_per_sample - 1) / kpts_per_sample;
    const size_t cap = rlm_slab_cap(n_phi, dim);
    const int group = (int)std::min<size_t>(std::min(n_t2, (int)ThetaList::MAX), cap);
    // samples per launch: their slabs within the cap, both grids within 65535 in y / z
    const int per = (int)std::max<size_t>(1, std::min<size_t>({(size_t)nsamples, cap / group, (size_t)65535 / group,
                                                               (size_t)65535 / kpts_per_sample}));
    for (int s0 = 0; s0 < nsamples; s0 += per) {
        const int ns = std::min(per, nsamples - s0);
        const int kp0 = s0 * kpts_per_sample, kps = std::min(ns * kpts_per_sample, count - kp0);
        for (int u = 0; u < n_t2; u += group) {
            ThetaList list;
            list.n = std::min(group, n_t2 - u);
            for (int i = 0; i < ThetaList::MAX; ++i) list.t2[i] = i < list.n ? uniq_t2[u + i] : 0;
            prof_begin(ctx, "k_rlm_assemble");
            RLMB_CUDA_TRY((launch_zgemm<cplx, 64>(ctx->stream, OpThetaA{cmt, cjm, dim, list},
                                                  OpVmnB{vmn + (size_t)s0 * dim * dim, dim, list.n},
                                                  EpRowMajor{ws, n_phi, dim}, n_phi, dim, dim, ns * list.n)));
            RLMB_LAUNCHED(ctx);
            for (int q = 0; q < kps; q += 65535) {
                prof_begin(ctx, "k_rlm_assemble");
                k_rlm_assemble<<<dim3((n_phi + 7) / 8, std::min(65535, kps - q)), 256, 0, ctx->stream>>>(
                    ws, cmt, d_t1, d_t2, list, n_phi, dim, o, kpts_per_sample, n_t2, kp0 + q, H);
                RLMB_LAUNCHED(ctx);
            }
        }
    }
    return RLMB_OK;
}

// rlm links: U1(t1,t2) = <u_n(t1,t2)|u_n(t1+1,t2)>, U2(t1,t2) = <u_n(t1,t2)|u_n(t1,t2+1)>
// on the full (g+1)^2 mesh of one sample, eigenvector n of k-point t at X[(t*N + n)*N].
// blockIdx.x = k-point * chunks + chunk of 8 states (a batch may hold more than 65,535 k-points).
__global__ void __launch_bounds__(256)
k_rlm_links(const cplx* __restrict__ X, int n_phi, int g, int chunks, cplx* __restrict__ U1, cplx* __restrict__ U2) {
    const int kpt = blockIdx.x / chunks;        // sample * (g+1)^2 + t1*(g+1) + t2
    const int per = (g + 1) * (g + 1);
    const int sample = kpt / per, t = kpt % per, t1 = t / (g + 1), t2 = t % (g + 1);
    const int lane = threadIdx.x & 31;
    const int state = blockIdx.x % chunks * 8 + (threadIdx.x >> 5);
    if (state >= n_phi) return;
    const size_t nn = (size_t)n_phi * n_phi;
    const cplx* a = X + (size_t)kpt * nn + (size_t)state * n_phi;
    const cplx* b1 = t1 < g ? a + (size_t)(g + 1) * nn : nullptr;
    const cplx* b2 = t2 < g ? a + nn : nullptr;
    cplx s1 = mk(0, 0), s2 = mk(0, 0);
    for (int r = lane; r < n_phi; r += 32) {
        const cplx av = a[r];
        if (b1) cfmac(s1, av, b1[r]);
        if (b2) cfmac(s2, av, b2[r]);
    }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (lane == 0) {
        const size_t o = ((size_t)sample * per + t) * n_phi + state;
        U1[o] = b1 ? s1 : mk(1.0, 0.0);
        U2[o] = b2 ? s2 : mk(1.0, 0.0);
    }
}

int launch_rlm_links(rlmb_context* ctx, const cplx* X, int n_phi, int g, int nsamples, cplx* U1, cplx* U2) {
    const int chunks = (n_phi + 7) / 8;
    prof_begin(ctx, "k_rlm_links");
    k_rlm_links<<<(unsigned)chunks * nsamples * (g + 1) * (g + 1), 256, 0, ctx->stream>>>(X, n_phi, g, chunks, U1, U2);
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// Plaquette phases and sample accumulation (rlm/main_rlm_cpu.cpp:155-158,187-190,230-239;
// hlm/main_hlm_cpu.cpp:111-115,143-147,184-187; diag_wrappers/chern.cpp:47-72).
// Mesh arrays are [sample][t1 (g+1)][t2 (n2)][N]; for hlm n2 = g and slot g of a line is
// the periodic copy of slot 0.  Plaquette (line L = 1..g, m = 0..g-1):
//   prod = U1(L-1,m) * U2(L,m) * conj(U1(L-1,m+1)) * conj(U2(L-1,m))
// contributes -arg(prod)/2pi (rlm, then + 1/N) or +arg(prod)/2pi (hlm).
//
// One thread per (state, plaquette slot): TX states (neighbouring, so that the mesh arrays are
// read in whole sectors) times TY slots per CTA, slot y taking plaquettes y, y + TY, ...; the
// slots' sums are added by shuffles and through shared memory in a fixed order.  The work is
// one atan2 per plaquette and state, so what matters is that a small number of states on a
// fine mesh still fills the GPU's warps: with one thread per state the rlm n_phi = 16, g = 64,
// 2-sample mesh took 2,960 us (32 threads walking 4,096 plaquettes each), with this split 33 us.
template <int TX, int TY>
__global__ void __launch_bounds__(TX * TY)
k_plaquettes(const cplx* __restrict__ U1, const cplx* __restrict__ U2, const double* __restrict__ W, int n_phi,
             int g, int hlm, double* __restrict__ energies, double* __restrict__ chern) {
    constexpr int NW = TX * TY / 32;
    __shared__ double red[2][NW][TX];
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sample = blockIdx.y, n = blockIdx.x * TX + tx;
    const int n2 = hlm ? g : g + 1;
    const size_t base = (size_t)sample * (g + 1) * n2;
    auto at = [&](int t1, int t2) -> size_t {
        if (hlm && t2 == g) t2 = 0;
        return (base + (size_t)t1 * n2 + t2) * n_phi + n;
    };
    double c = 0.0, e = 0.0;
    if (n < n_phi) {
        for (int p = ty; p < g * g; p += TY) {
            const int L = p / g + 1, m = p % g;
            cplx prod = U1[at(L - 1, m)];
            prod = cmul(prod, U2[at(L, m)]);
            prod = cmul(prod, cconj(U1[at(L - 1, m + 1)]));
            prod = cmul(prod, cconj(U2[at(L - 1, m)]));
            const double phase = atan2(prod.y, prod.x) / (M_PI * 2.0);
            c += hlm ? phase : -phase;
        }
        for (int p = ty; p < (g + 1) * n2; p += TY) {
            const int t1 = p / n2, t2 = p % n2;
            const double w = W[at(t1, t2)];
            e += hlm && t2 == 0 ? 2.0 * w : w;   // (hlm: slot g repeats slot 0)
        }
    }
#pragma unroll
    for (int m = TX; m < 32; m <<= 1) {
        c += __shfl_xor_sync(0xffffffffu, c, m);
        e += __shfl_xor_sync(0xffffffffu, e, m);
    }
    if (lane < TX) {
        red[0][warp][lane] = c;
        red[1][warp][lane] = e;
    }
    __syncthreads();
    if (threadIdx.x < TX && n < n_phi) {
        c = 0.0;
        e = 0.0;
        for (int i = 0; i < NW; ++i) {
            c += red[0][i][tx];
            e += red[1][i][tx];
        }
        const size_t idx = (size_t)sample * n_phi + n;
        energies[idx] = e / ((double)(g + 1) * (g + 1));
        chern[idx] = hlm ? c : c + 1.0 / n_phi;
    }
}

// Slots per state: about the mesh's plaquettes, at most 256 (g = 64: 16 plaquettes per
// thread); coarse meshes take 16 slots and 16 states per CTA, whose rows are whole 256-byte
// lines.
int launch_plaquettes(rlmb_context* ctx, const cplx* U1, const cplx* U2, const double* W, int n_phi,
                      int g, int nsamples, int hlm, double* energies, double* chern) {
    const size_t mesh = (size_t)(g + 1) * (hlm ? g : g + 1) * n_phi;
    prof_begin(ctx, "k_plaquettes");
    for (int s0 = 0; s0 < nsamples; s0 += 65535) {   // grid y extent
        const int ns = std::min(nsamples - s0, 65535);
        const cplx *u1 = U1 + s0 * mesh, *u2 = U2 + s0 * mesh;
        const double* w = W + s0 * mesh;
        double *oe = energies + (size_t)s0 * n_phi, *oc = chern + (size_t)s0 * n_phi;
        if (g <= 4)
            k_plaquettes<16, 16><<<dim3((n_phi + 15) / 16, ns), 256, 0, ctx->stream>>>(u1, u2, w, n_phi, g, hlm, oe, oc);
        else if (g <= 32)
            k_plaquettes<4, 64><<<dim3((n_phi + 3) / 4, ns), 256, 0, ctx->stream>>>(u1, u2, w, n_phi, g, hlm, oe, oc);
        else
            k_plaquettes<4, 256><<<dim3((n_phi + 3) / 4, ns), 1024, 0, ctx->stream>>>(u1, u2, w, n_phi, g, hlm, oe, oc);
    }
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// Reference-layout FHS for one line pair (diag_wrappers/chern.cpp:3-75): prev/cur hold
// (g+1) k-points of N states of length dim_vec; out[m + n*g] = -arg(prod)/2pi.
__global__ void __launch_bounds__(256)
k_fhs_line(const cplx* __restrict__ prev, const cplx* __restrict__ cur, int n_phi, int dim_vec,
           int g, double* __restrict__ out) {
    const int m = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int n = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (n >= n_phi) return;
    const size_t kstride = (size_t)n_phi * dim_vec;
    const cplx* pm = prev + (size_t)m * kstride + (size_t)n * dim_vec;
    const cplx* pm1 = pm + kstride;
    const cplx* cm = cur + (size_t)m * kstride + (size_t)n * dim_vec;
    const cplx* cm1 = cm + kstride;
    cplx l0 = mk(0, 0), l1 = mk(0, 0), l2 = mk(0, 0), l3 = mk(0, 0);
    for (int r = lane; r < dim_vec; r += 32) {
        const cplx a = pm[r], b = cm[r], c = cm1[r], d = pm1[r];
        cfmac(l0, a, b);   // <prev,m | cur,m>
        cfmac(l1, b, c);   // <cur,m | cur,m+1>
        cfmac(l2, c, d);   // <cur,m+1 | prev,m+1>
        cfmac(l3, d, a);   // <prev,m+1 | prev,m>
    }
    l0 = warp_sum(l0);
    l1 = warp_sum(l1);
    l2 = warp_sum(l2);
    l3 = warp_sum(l3);
    if (lane == 0) {
        cplx prod = mk(1.0, 0.0);
        prod = cmul(prod, l0);
        prod = cmul(prod, l1);
        prod = cmul(prod, l2);
        prod = cmul(prod, l3);
        out[m + (size_t)n * g] = -atan2(prod.y, prod.x) / (M_PI * 2.0);
    }
}

int launch_fhs_line(rlmb_context* ctx, const cplx* prev, const cplx* cur, int n_phi, int dim_vec,
                    int g, double* out) {
    dim3 grid((n_phi + 7) / 8, g);
    prof_begin(ctx, "k_fhs_line");
    k_fhs_line<<<grid, 256, 0, ctx->stream>>>(prev, cur, n_phi, dim_vec, g, out);
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// ======================================================================= hlm
// Clean Bloch vectors (hlm/hamiltonian_hlm_cpu.cpp:18-51).  For each k-point t of the
// mesh (t1 in [0,g], t2 in [0,g)) and Bloch index c = kx*ly + ky: the Q x Q Harper matrix
// exactly as the reference writes its column-major array (:25-32), diagonalised by
// cyclic complex Jacobi rotations, band `band` of the ascending spectrum, scaled by
// 1/sqrt(N |h|^2) -- the norm of the full plane-wave column (:43-51).
__global__ void k_hlm_bloch(int lx, int ly, int Q, int band, int g, int t1_0, int t1_1, int t2_0,
                            int t2_1, cplx* __restrict__ hb) {
    const int Lxp = lx / Q, N = Lxp * ly;
    const int n2 = t2_1 - t2_0;
    const long total = (long)(t1_1 - t1_0) * n2 * N;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int c = (int)(idx % N);
    const int t = (int)(idx / N);
    const int t1 = t1_0 + t / n2, t2 = t2_0 + t % n2;
    const int kx = c / ly, ky = c % ly;
    const double inv_g = 1.0 / g, pi2 = 2.0 * M_PI;
    const double kxs = kx + t1 * inv_g, kys = ky + t2 * inv_g;
    cplx a[RLMB_MAX_Q * RLMB_MAX_Q];   // column-major [r + c*Q]
    cplx v[RLMB_MAX_Q * RLMB_MAX_Q];
    for (int i = 0; i < Q * Q; ++i) a[i] = mk(0, 0);
    const double inv_Q = 1.0 / Q;
    for (int p = 0; p < Q; ++p) {
        a[p * Q + p] = mk(-2.0 * cos(kys * (pi2 / ly) + pi2 * p * inv_Q), 0.0);
        if (p + 1 < Q) a[p * Q + p + 1] = a[(p + 1) * Q + p] = mk(-1.0, 0.0);
    }
    const double ph = kxs * Q * (pi2 / lx);
    a[Q * (Q - 1)] = mk(-cos(ph), -sin(ph));
    a[Q - 1] = cconj(a[Q * (Q - 1)]);
    // heevd reads the upper triangle (col-major): A[r][c] = a[r + c*Q], r <= c
    for (int cc = 0; cc < Q; ++cc)
        for (int r = 0; r < Q; ++r) {
            if (r < cc) a[cc + r * Q] = cconj(a[r + cc * Q]);
            else if (r == cc) a[r + cc * Q].y = 0.0;
        }
    for (int i = 0; i < Q * Q; ++i) v[i] = mk(i % (Q + 1) == 0 ? 1.0 : 0.0, 0.0);
    herm_jacobi(a, v, Q);
    // eigenvector of the band-th smallest eigenvalue
    int order[RLMB_MAX_Q];
    for (int i = 0; i < Q; ++i) order[i] = i;
    for (int i = 1; i < Q; ++i)
        for (int j = i; j > 0 && a[order[j] * (Q + 1)].x < a[order[j - 1] * (Q + 1)].x; --j) {
            const int tmp = order[j];
            order[j] = order[j - 1];
            order[j - 1] = tmp;
        }
    const int col = order[band];
    double h2 = 0.0;
    for (int q = 0; q < Q; ++q) h2 += cabs2(v[q + col * Q]);
    const double sc = 1.0 / sqrt((double)N * h2);
    cplx* out = hb + ((size_t)t * N + c) * Q;
    for (int q = 0; q < Q; ++q) out[q] = cscale(v[q + col * Q], sc);
}

int launch_hlm_bloch(rlmb_context* ctx, int lx, int ly, int Q, int band, int g, int t1_0, int t1_1,
                     int t2_0, int t2_1, cplx* hb) {
    const int N = lx * ly / Q;
    const long total = (long)(t1_1 - t1_0) * (t2_1 - t2_0) * N;
    prof_begin(ctx, "k_hlm_bloch");
    k_hlm_bloch<<<(unsigned)((total + 127) / 128), 128, 0, ctx->stream>>>(lx, ly, Q, band, g, t1_0,
                                                                         t1_1, t2_0, t2_1, hb);
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// Full basis column W(r, c) = e^{-i phi_c(r)} hhat_c[q(r)] (hlm/hamiltonian_hlm_cpu.cpp:37-42)
__global__ void k_hlm_basis_expand(const cplx* __restrict__ hb, int lx, int ly, int Q, int g, int t1,
                                   int t2, cplx* __restrict__ W) {
    const int Lxp = lx / Q, N = Lxp * ly, ns = lx * ly;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)N * ns) return;
    const int c = (int)(idx / ns), r = (int)(idx % ns);
    const int kx = c / ly, ky = c % ly;
    const int j = r / lx, xm = r % lx, q = xm % Q, m = xm - q;
    const double inv_g = 1.0 / g, pi2 = 2.0 * M_PI;
    const double kxs = kx + t1 * inv_g, kys = ky + t2 * inv_g;
    const double phase = kxs * (pi2 / lx) * m + kys * (pi2 / ly) * j;
    double sn, cs;
    sincos(phase, &sn, &cs);
    W[idx] = cmul(mk(cs, -sn), hb[(size_t)c * Q + q]);
}

int launch_hlm_basis_expand(rlmb_context* ctx, const cplx* hb, int lx, int ly, int Q, int g, int t1,
                            int t2, cplx* W) {
    const long total = (long)(lx * ly / Q) * lx * ly;
    prof_begin(ctx, "k_hlm_basis_expand");
    k_hlm_basis_expand<<<(unsigned)((total + 255) / 256), 256, 0, ctx->stream>>>(hb, lx, ly, Q, g, t1, t2, W);
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// Sublattice Fourier transform of the on-site potential (blockIdx.x = sample * chunks + chunk of 128
// entries):
//   Vt[q][dx][dy] = sum_{m'<Lx', j<ly} V[j*lx + Q m' + q] e^{+i 2pi (dx m'/Lx' + dy j/ly)}
// so that W^H diag(V) W [a][b] = sum_q conj(hhat_a[q]) hhat_b[q] Vt[q][kxa-kxb][kya-kyb]:
// the twist phases of the two columns cancel in the difference.
__global__ void k_hlm_vtilde(const double* __restrict__ pot, int lx, int ly, int Q, int chunks, cplx* __restrict__ vt) {
    const int Lxp = lx / Q, N = Lxp * ly, ns = lx * ly;
    const int sample = blockIdx.x / chunks;
    const int idx = blockIdx.x % chunks * blockDim.x + threadIdx.x;
    if (idx >= ns) return;
    const int q = idx / N, rest = idx % N, dx = rest / ly, dy = rest % ly;
    const double* V = pot + (size_t)sample * ns;
    cplx acc = mk(0, 0);
    for (int mp = 0; mp < Lxp; ++mp) {
        const int fx = (dx * mp) % Lxp;
        for (int j = 0; j < ly; ++j) {
            const int fy = (dy * j) % ly;
            // exact fraction fx/Lxp + fy/ly, taken through sincospi
            const double f = 2.0 * ((double)fx / Lxp + (double)fy / ly);
            double sn, cs;
            sincospi(f, &sn, &cs);
            const double val = V[j * lx + Q * mp + q];
            acc.x = fma(val, cs, acc.x);
            acc.y = fma(val, sn, acc.y);
        }
    }
    vt[(size_t)sample * ns + idx] = acc;
}

int launch_hlm_vtilde(rlmb_context* ctx, const double* pot, int lx, int ly, int Q, int nsamples, cplx* vt) {
    const int chunks = (lx * ly + 127) / 128;
    prof_begin(ctx, "k_hlm_vtilde");
    k_hlm_vtilde<<<(unsigned)chunks * nsamples, 128, 0, ctx->stream>>>(pot, lx, ly, Q, chunks, vt);
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// Projected H of k-point (sample, t) into column-major buf[b*N + a] = H[a][b].
// blockIdx.x = (sample * kpts + k) * slices + slice, kpts = number of mesh k-points given in tlist.
// Thread = row a (its Bloch indices and hhat_a held in registers); the CTA's slice of the
// columns b is walked in order, so consecutive threads store consecutive entries of a
// column (coalesced) and every per-b quantity is a warp-uniform shared-memory broadcast.
// The sublattice offsets (kxa - kxb) mod Lx', (kya - kyb) mod ly advance by wrap-around
// subtraction instead of integer division.  QT: the flux denominator Q as a compile-time
// constant (hhat_a in registers), or 0 for the generic form (hhat_a re-read from shared
// memory).
template <int QT>
__global__ void __launch_bounds__(256)
k_hlm_project(const cplx* __restrict__ hb, const cplx* __restrict__ vt, const int* __restrict__ tlist,
              int g, int lx, int ly, int Qr, int kpts, int slices, cplx* __restrict__ H) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Q = QT > 0 ? QT : Qr;
    const int Lxp = lx / Q, N = Lxp * ly, ns = lx * ly;
    cplx* sh = reinterpret_cast<cplx*>(smem_raw);   // [N*Q] hhat of this k-point
    cplx* sv = sh + (size_t)N * Q;                   // [ns]  Vt of this sample
    const int job = blockIdx.x / slices, slice = blockIdx.x % slices;
    const int sample = job / kpts, k = job % kpts;
    const int t = tlist ? tlist[k] : k / g * (g + 1) + k % g;   // (without a list: the mesh, theta_2 < g)
    for (int i = threadIdx.x; i < N * Q; i += blockDim.x) sh[i] = hb[(size_t)t * N * Q + i];
    for (int i = threadIdx.x; i < ns; i += blockDim.x) sv[i] = vt[(size_t)sample * ns + i];
    __syncthreads();
    cplx* h = H + (size_t)job * N * N;
    // columns of this CTA: [b0, b1)
    const int per = (N + slices - 1) / slices;
    const int b0 = slice * per, b1 = min(N, b0 + per);
    if (b0 >= b1) return;
    for (int a = threadIdx.x; a < N; a += blockDim.x) {
        const int kxa = a / ly, kya = a % ly;
        constexpr int QR = QT > 0 ? QT : 1;
        cplx ha[QR];
#pragma unroll
        for (int q = 0; q < QR; ++q) ha[q] = cconj(sh[a * Q + q]);
        const int kxb = b0 / ly, kyb0 = b0 % ly;
        int kyb = kyb0;
        int dx = kxa - kxb;
        if (dx < 0) dx += Lxp;
        int dy = kya - kyb;
        if (dy < 0) dy += ly;
        for (int b = b0; b < b1; ++b) {
            cplx acc = mk(0, 0);
            const cplx* hbq = sh + b * Q;
            if constexpr (QT > 0) {
#pragma unroll
                for (int q = 0; q < QT; ++q) cfma(acc, cmul(ha[q], hbq[q]), sv[(q * Lxp + dx) * ly + dy]);
            } else {
                for (int q = 0; q < Q; ++q)
                    cfma(acc, cmul(cconj(sh[a * Q + q]), hbq[q]), sv[(q * Lxp + dx) * ly + dy]);
            }
            h[(size_t)b * N + a] = acc;
            // next column: kyb + 1 (wrapping into kxb + 1)
            if (++kyb == ly) {
                kyb = 0;
                dy = kya;
                if (--dx < 0) dx += Lxp;
            } else if (--dy < 0) {
                dy += ly;
            }
        }
    }
}

int launch_hlm_project(rlmb_context* ctx, const cplx* hb, const cplx* vt, const int* d_tlist, int g, int lx,
                       int ly, int Q, int kpts, int nsamples, cplx* H) {
    const int N = lx * ly / Q;
    const size_t smem = ((size_t)N * Q + (size_t)lx * ly) * sizeof(cplx);
    if (smem > 200 * 1024) return RLMB_ERR_ARG;
    auto kern = Q == 1 ? k_hlm_project<1> : Q == 2 ? k_hlm_project<2> : Q == 3 ? k_hlm_project<3>
              : Q == 4 ? k_hlm_project<4> : k_hlm_project<0>;
    RLMB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int slices = std::max(1, std::min(N / 32, 16));   // column slices of >= 32 columns per k-point
    prof_begin(ctx, "k_hlm_project");
    kern<<<(unsigned)slices * kpts * nsamples, 256, smem, ctx->stream>>>(hb, vt, d_tlist, g, lx, ly, Q, kpts, slices, H);
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// hlm link overlaps from the eigenvectors U of the projected problems, without forming
// the n_sites-long states W U (hlm/hamiltonian_hlm_cpu.cpp:180):
//   <psi_n(a)|psi_n(b)> = U_n(a)^H S U_n(b),  S = W(a)^H W(b).
// S is block diagonal: theta_2 links (same t1) couple equal kx only,
//   S[(kx,ky),(kx,ky')] = Lx' D_ly(ky - ky' + (t2 - t2')/g) <hhat|hhat'>,
// theta_1 links (same t2) couple equal ky only,
//   S[(kx,ky),(kx',ky)] = ly D_Lx'(kx - kx' + (t1 - t1')/g) <hhat|hhat'>,
// with D_L(s) = sum_{j<L} e^{i 2pi s j / L}.  The theta_2 = g neighbour is the periodic
// copy of theta_2 = 0 (hlm/main_hlm_cpu.cpp:149-150).
// blockIdx.x = state chunk, blockIdx.y = sample*kpts + t (t = t1*g + t2), blockIdx.z = dir.
static constexpr int LINK_STATES = 16;

__global__ void __launch_bounds__(256)
k_hlm_links_generic(const cplx* __restrict__ hb, const cplx* __restrict__ X, int lx, int ly, int Q, int g,
            cplx* __restrict__ U1, cplx* __restrict__ U2) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Lxp = lx / Q, N = Lxp * ly;
    const int dir = blockIdx.y;                       // 0: theta_1 link, 1: theta_2 link
    const int kpts = (g + 1) * g;
    const int job = blockIdx.x, sample = job / kpts, t = job % kpts;
    const int t1 = t / g, t2 = t % g;
    if (dir == 0 && t1 == g) return;                  // no theta_1 neighbour of the last line
    const int L = dir == 0 ? Lxp : ly;                // block size
    const int tb1 = dir == 0 ? t1 + 1 : t1;
    const int tb2 = dir == 0 ? t2 : (t2 + 1 == g ? 0 : t2 + 1);
    const int tb = tb1 * g + tb2;
    // theta offset (t - t') / g entering D: theta_1 link: -1/g; theta_2 link: (t2 - t2')/g
    const double shift = dir == 0 ? -1.0 / g : (double)(t2 - tb2) / g;
    cplx* S = reinterpret_cast<cplx*>(smem_raw);      // [N][L]: S[a][l], b = partner l of a
    cplx* ub = S + (size_t)N * L;                     // [LINK_STATES][N]
    __shared__ cplx Dtab[64];
    __shared__ cplx red[8][LINK_STATES];
    for (int dlt = threadIdx.x; dlt < L; dlt += blockDim.x) {
        // D_L(dlt + shift), dlt = (index difference) mod L
        cplx acc = mk(0, 0);
        for (int j = 0; j < L; ++j) {
            double sn, cs;
            sincospi(2.0 * (dlt + shift) * j / L, &sn, &cs);
            acc = cadd(acc, mk(cs, sn));
        }
        Dtab[dlt] = acc;
    }
    __syncthreads();
    // Bloch tables cover the (g+1) x (g+1) mesh: index t1*(g+1) + t2
    const cplx* ha = hb + ((size_t)t1 * (g + 1) + t2) * N * Q;
    const cplx* hbb = hb + ((size_t)tb1 * (g + 1) + tb2) * N * Q;
    const double pref = dir == 0 ? (double)ly : (double)Lxp;
    for (int idx = threadIdx.x; idx < N * L; idx += blockDim.x) {
        const int a = idx / L, l = idx % L;
        const int kxa = a / ly, kya = a % ly;
        int b, dlt;
        if (dir == 0) { b = l * ly + kya; dlt = (kxa - l + Lxp) % Lxp; }
        else { b = kxa * ly + l; dlt = (kya - l + ly) % ly; }
        cplx ov = mk(0, 0);
        for (int q = 0; q < Q; ++q) cfmac(ov, ha[(size_t)a * Q + q], hbb[(size_t)b * Q + q]);
        S[idx] = cscale(cmul(Dtab[dlt], ov), pref);
    }
    const size_t nn = (size_t)N * N;
    const cplx* Xa = X + ((size_t)sample * kpts + t) * nn;
    const cplx* Xb = X + ((size_t)sample * kpts + tb) * nn;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int s0 = 0; s0 < N; s0 += LINK_STATES) {
        const int ns = min(LINK_STATES, N - s0);
        __syncthreads();
        for (int i = threadIdx.x; i < LINK_STATES * N; i += blockDim.x) {
            const int s = i / N, bidx = i % N;
            ub[i] = s < ns ? Xb[(size_t)(s0 + s) * N + bidx] : mk(0, 0);
        }
        __syncthreads();
        cplx part[LINK_STATES];
#pragma unroll
        for (int s = 0; s < LINK_STATES; ++s) part[s] = mk(0, 0);
        for (int a = threadIdx.x; a < N; a += blockDim.x) {
            const int kxa = a / ly, kya = a % ly;
            const cplx* Sa = S + (size_t)a * L;
#pragma unroll
            for (int s = 0; s < LINK_STATES; ++s) {
                if (s < ns) {
                    cplx y = mk(0, 0);
                    for (int l = 0; l < L; ++l) {
                        const int b = dir == 0 ? l * ly + kya : kxa * ly + l;
                        cfma(y, Sa[l], ub[s * N + b]);
                    }
                    cfmac(part[s], Xa[(size_t)(s0 + s) * N + a], y);
                }
            }
        }
#pragma unroll
        for (int s = 0; s < LINK_STATES; ++s) {
            const cplx v = warp_sum(part[s]);
            if (lane == 0) red[w][s] = v;
        }
        __syncthreads();
        if (threadIdx.x < ns) {
            cplx tot = mk(0, 0);
            for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot = cadd(tot, red[i][threadIdx.x]);
            const size_t o = ((size_t)sample * kpts + t) * N + s0 + threadIdx.x;
            if (dir == 0) U1[o] = tot; else U2[o] = tot;
        }
    }
}

int launch_hlm_links_generic(rlmb_context* ctx, const cplx* hb, const cplx* X, int lx, int ly, int Q, int g,
                     int nsamples, cplx* U1, cplx* U2) {
    const int N = lx * ly / Q;
    const int Lmax = std::max(lx / Q, ly);
    if (Lmax > 64) return RLMB_ERR_ARG;
    const size_t smem = ((size_t)N * Lmax + (size_t)LINK_STATES * N) * sizeof(cplx);
    if (smem > 200 * 1024) return RLMB_ERR_ARG;
    RLMB_CUDA_TRY(cudaFuncSetAttribute(k_hlm_links_generic, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid(nsamples * (g + 1) * g, 2);
    prof_begin(ctx, "k_hlm_links_generic");
    k_hlm_links_generic<<<grid, 256, smem, ctx->stream>>>(hb, X, lx, ly, Q, g, U1, U2);
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// One CTA per (sample, k-point t): both links of t.  S blocks of the two directions are
// built once in shared memory; thread = state n, which loads one Bloch block of U'(n) into
// registers and reuses it for the block's L rows (S entries are warp-uniform broadcasts).
static constexpr int LINK_MAXL = 32;

template <int L>
__device__ __forceinline__ cplx link_dir(const cplx* __restrict__ S, const cplx* __restrict__ ua,
                                         const cplx* __restrict__ ub, int nblk, int ly, int dir) {
    // blocks: dir 1 (theta_2) -> block kx, rows a = kx*ly + i, partners kx*ly + l;
    //         dir 0 (theta_1) -> block ky, rows a = i*ly + ky, partners l*ly + ky.
    cplx acc = mk(0, 0);
    for (int beta = 0; beta < nblk; ++beta) {
        cplx u[L];
#pragma unroll
        for (int l = 0; l < L; ++l) u[l] = ub[dir ? beta * ly + l : l * ly + beta];
#pragma unroll 2
        for (int i = 0; i < L; ++i) {
            const int a = dir ? beta * ly + i : i * ly + beta;
            const cplx* Sa = S + (size_t)a * L;
            cplx y = mk(0, 0);
#pragma unroll
            for (int l = 0; l < L; ++l) cfma(y, Sa[l], u[l]);
            cfmac(acc, ua[a], y);
        }
    }
    return acc;
}

__device__ void build_link_S(cplx* S, cplx* Dtab, const cplx* __restrict__ ha, const cplx* __restrict__ hbb,
                             int N, int L, int ly, int Lxp, int Q, int dir, double shift, bool transposed = false) {
    for (int dlt = threadIdx.x; dlt < L; dlt += blockDim.x) {
        // D_L(dlt + shift) = sum_j e^{i 2pi (dlt + shift) j / L}, dlt = index difference mod L
        cplx acc = mk(0, 0);
        for (int j = 0; j < L; ++j) {
            double sn, cs;
            sincospi(2.0 * (dlt + shift) * j / L, &sn, &cs);
            acc = cadd(acc, mk(cs, sn));
        }
        Dtab[dlt] = acc;
    }
    __syncthreads();
    const double pref = dir == 0 ? (double)ly : (double)Lxp;
    for (int idx = threadIdx.x; idx < N * L; idx += blockDim.x) {
        const int a = idx / L, l = idx % L;
        const int kxa = a / ly, kya = a % ly;
        int b, dlt;
        if (dir == 0) { b = l * ly + kya; dlt = (kxa - l + Lxp) % Lxp; }
        else { b = kxa * ly + l; dlt = (kya - l + ly) % ly; }
        cplx ov = mk(0, 0);
        for (int q = 0; q < Q; ++q) cfmac(ov, ha[(size_t)a * Q + q], hbb[(size_t)b * Q + q]);
        S[transposed ? (size_t)l * N + a : (size_t)idx] = cscale(cmul(Dtab[dlt], ov), pref);
    }
}

template <int L1, int L2>
__global__ void __launch_bounds__(256)
k_hlm_links(const cplx* __restrict__ hb, const cplx* __restrict__ X, int lx, int ly, int Q, int g,
            cplx* __restrict__ U1, cplx* __restrict__ U2) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Lxp = lx / Q, N = Lxp * ly;
    const int kpts = (g + 1) * g;
    const int job = blockIdx.x, sample = job / kpts, t = job % kpts;
    const int t1 = t / g, t2 = t % g;
    cplx* S1 = reinterpret_cast<cplx*>(smem_raw);      // theta_1 link: [N][Lxp]
    cplx* S2 = S1 + (size_t)N * L1;                      // theta_2 link: [N][ly]
    __shared__ cplx Dtab[LINK_MAXL];
    const bool has1 = t1 < g;
    const int t2n = t2 + 1 == g ? 0 : t2 + 1;            // theta_2 = g is the copy of theta_2 = 0
    const cplx* ha = hb + ((size_t)t1 * (g + 1) + t2) * N * Q;
    if (has1) {
        build_link_S(S1, Dtab, ha, hb + ((size_t)(t1 + 1) * (g + 1) + t2) * N * Q, N, L1, ly, Lxp, Q, 0,
                     -1.0 / g);
        __syncthreads();
    }
    build_link_S(S2, Dtab, ha, hb + ((size_t)t1 * (g + 1) + t2n) * N * Q, N, L2, ly, Lxp, Q, 1,
                 (double)(t2 - t2n) / g);
    __syncthreads();
    const size_t nn = (size_t)N * N;
    const cplx* Xa = X + ((size_t)sample * kpts + t) * nn;
    const cplx* Xb1 = X + ((size_t)sample * kpts + (t1 + 1) * g + t2) * nn;
    const cplx* Xb2 = X + ((size_t)sample * kpts + t1 * g + t2n) * nn;
    for (int n = threadIdx.x; n < N; n += blockDim.x) {
        const cplx* ua = Xa + (size_t)n * N;
        const size_t o = ((size_t)sample * kpts + t) * N + n;
        if (has1) U1[o] = link_dir<L1>(S1, ua, Xb1 + (size_t)n * N, ly, ly, 0);
        U2[o] = link_dir<L2>(S2, ua, Xb2 + (size_t)n * N, Lxp, ly, 1);
    }
}

// The same links with one warp per state n: the warp stages rows n of the two neighbours'
// eigenvector matrices in shared memory, its lanes walk the Bloch index a of row n of its own
// matrix (coalesced 16-byte loads of all three rows), and the S blocks are stored transposed
// (S[l][a]) so that consecutive lanes read consecutive words.  Per-lane partial overlaps are
// reduced across the warp.
template <int L1, int L2>
__global__ void __launch_bounds__(256)
k_hlm_links_w(const cplx* __restrict__ hb, const cplx* __restrict__ X, int lx, int ly, int Q, int g,
              cplx* __restrict__ U1, cplx* __restrict__ U2) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Lxp = lx / Q, N = Lxp * ly;
    const int kpts = (g + 1) * g;
    const int job = blockIdx.x, sample = job / kpts, t = job % kpts;
    const int t1 = t / g, t2 = t % g;
    cplx* T1 = reinterpret_cast<cplx*>(smem_raw);      // theta_1 link, transposed: T1[l][a]
    cplx* T2 = T1 + (size_t)N * L1;                      // theta_2 link, T2[l][a]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    cplx* r1 = T2 + (size_t)N * L2 + (size_t)w * 2 * N;   // this warp's two staged rows
    cplx* r2 = r1 + N;
    __shared__ cplx Dtab[LINK_MAXL];
    const bool has1 = t1 < g;
    const int t2n = t2 + 1 == g ? 0 : t2 + 1;            // theta_2 = g is the copy of theta_2 = 0
    const cplx* ha = hb + ((size_t)t1 * (g + 1) + t2) * N * Q;
    if (has1) {
        build_link_S(T1, Dtab, ha, hb + ((size_t)(t1 + 1) * (g + 1) + t2) * N * Q, N, L1, ly, Lxp, Q, 0,
                     -1.0 / g, true);
        __syncthreads();
    }
    build_link_S(T2, Dtab, ha, hb + ((size_t)t1 * (g + 1) + t2n) * N * Q, N, L2, ly, Lxp, Q, 1,
                 (double)(t2 - t2n) / g, true);
    __syncthreads();
    const size_t nn = (size_t)N * N;
    const cplx* Xa = X + ((size_t)sample * kpts + t) * nn;
    const cplx* Xb1 = X + ((size_t)sample * kpts + (t1 + 1) * g + t2) * nn;
    const cplx* Xb2 = X + ((size_t)sample * kpts + t1 * g + t2n) * nn;
    for (int n = w; n < N; n += blockDim.x >> 5) {
        for (int b = lane; b < N; b += 32) {
            if (has1) r1[b] = Xb1[(size_t)n * N + b];
            r2[b] = Xb2[(size_t)n * N + b];
        }
        __syncwarp();
        cplx acc1 = mk(0, 0), acc2 = mk(0, 0);
        for (int a = lane; a < N; a += 32) {
            const int kxa = a / ly, kya = a % ly;
            const cplx ua = Xa[(size_t)n * N + a];
            if (has1) {   // theta_1 link: partners b = l * ly + kya
                cplx y = mk(0, 0);
#pragma unroll
                for (int l = 0; l < L1; ++l) cfma(y, T1[(size_t)l * N + a], r1[l * ly + kya]);
                cfmac(acc1, ua, y);
            }
            cplx y = mk(0, 0);   // theta_2 link: partners b = kxa * ly + l
#pragma unroll
            for (int l = 0; l < L2; ++l) cfma(y, T2[(size_t)l * N + a], r2[kxa * ly + l]);
            cfmac(acc2, ua, y);
        }
        acc1 = warp_sum(acc1);
        acc2 = warp_sum(acc2);
        if (lane == 0) {
            const size_t o = ((size_t)sample * kpts + t) * N + n;
            if (has1) U1[o] = acc1;
            U2[o] = acc2;
        }
        __syncwarp();   // the staged rows are rewritten for the next state
    }
}

// The same links on the FP64 tensor path (DMMA), block sizes 8 and 16: per direction every Bloch
// block of L partners is a product Y[n][i] = sum_l U'_n[l] S[i][l], K = L, of the states with the
// block's S, followed by the products with conj(U_n[i]).  One CTA of 16 warps per k-point; a warp
// owns every sixteenth block and keeps its S fragments in registers for all states, which pass
// through shared memory eight at a time (U and U', cp.async, the next eight on their way), in
// the order that makes a block's entries contiguous.  Rows are padded by 4 entries so that the
// two rows of a fragment's 8-lane phase hit distinct banks.
// Bound: reading the eigenvectors (three rows of the mesh per k-point and direction) and the
// barriers between groups of states.  k_hlm_links_w, bound by its shared-memory operands (two per
// multiply-add), took 10.6 ms for the 4,224 k-points of the 48 x 16 lattice; this one 5.6.
static constexpr int LM_T = 512, LM_NS = 8;
template <int L1, int L2>
constexpr size_t links_mma_smem() {
    return sizeof(cplx) * ((size_t)L1 * L2 * (L1 > L2 ? L1 : L2) + 2 * 2 * LM_NS * (L1 * L2 + 4) + 16 * LM_NS);
}
template <int L, int NBLK>
__device__ __forceinline__ void links_mma_dir(const cplx* __restrict__ S, cplx* __restrict__ stage, cplx* __restrict__ red,
                                              const cplx* __restrict__ Xa, const cplx* __restrict__ Xb, int ly, int dir,
                                              cplx* __restrict__ U) {
    constexpr int N = L * NBLK, XS = N + 4, NB = (NBLK + 15) / 16;   // blocks per warp
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    // S fragments: (l = 4 k + q, i = 8 it + g) of this warp's blocks
    cplx b[NB][L / 8][L / 4];
#pragma unroll
    for (int u = 0; u < NB; ++u) {
        const int beta = warp + 16 * u;
#pragma unroll
        for (int it = 0; it < L / 8; ++it) {
            const int i = 8 * it + g, a = dir ? beta * ly + i : i * ly + beta;
#pragma unroll
            for (int k = 0; k < L / 4; ++k) b[u][it][k] = beta < NBLK ? S[a * L + 4 * k + q] : mk(0, 0);
        }
    }
    auto fetch = [&](int n0, int buf) {   // states n0 .. n0 + 7 of U and U'
        cplx* d = stage + buf * 2 * LM_NS * XS;
        for (int i = tid; i < LM_NS * N; i += LM_T) {
            const int s = i / N, a = i % N;
            const int at = s * XS + (dir ? a : (a % ly) * L + a / ly);
            if (n0 + s < N) {
                const unsigned da = (unsigned)__cvta_generic_to_shared(d + at);
                const unsigned db = (unsigned)__cvta_generic_to_shared(d + LM_NS * XS + at);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(da), "l"(Xa + (size_t)(n0 + s) * N + a) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(db), "l"(Xb + (size_t)(n0 + s) * N + a) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    fetch(0, 0);
    for (int n0 = 0, buf = 0; n0 < N; n0 += LM_NS, buf ^= 1) {
        if (n0 + LM_NS < N) fetch(n0 + LM_NS, buf ^ 1);
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        const cplx* xa = stage + buf * 2 * LM_NS * XS + g * XS;
        const cplx* xb = xa + LM_NS * XS;
        cplx acc = mk(0, 0);
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int beta = warp + 16 * u;
            if (beta >= NBLK) break;
            double cr[L / 8][2], ci[L / 8][2];
#pragma unroll
            for (int it = 0; it < L / 8; ++it) cr[it][0] = cr[it][1] = ci[it][0] = ci[it][1] = 0.0;
#pragma unroll
            for (int k = 0; k < L / 4; ++k) {
                const cplx x = xb[beta * L + 4 * k + q];
#pragma unroll
                for (int it = 0; it < L / 8; ++it) {
                    dmma884(cr[it], x.x, b[u][it][k].x);
                    dmma884(ci[it], x.x, b[u][it][k].y);
                    dmma884(cr[it], -x.y, b[u][it][k].y);
                    dmma884(ci[it], x.y, b[u][it][k].x);
                }
            }
#pragma unroll
            for (int it = 0; it < L / 8; ++it)
#pragma unroll
                for (int e = 0; e < 2; ++e) cfmac(acc, xa[beta * L + 8 * it + 2 * q + e], mk(cr[it][e], ci[it][e]));
        }
        acc = cadd(acc, shfl_xor(acc, 1));
        acc = cadd(acc, shfl_xor(acc, 2));
        if (q == 0) red[warp * LM_NS + g] = acc;
        __syncthreads();
        if (tid < LM_NS && n0 + tid < N) {
            cplx s = mk(0, 0);
#pragma unroll
            for (int w = 0; w < 16; ++w) s = cadd(s, red[w * LM_NS + tid]);
            U[n0 + tid] = s;
        }
        // (red is written again after the next group's first barrier, the buffers after this one)
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
}
template <int L1, int L2>
__global__ void __launch_bounds__(LM_T)
k_hlm_links_mma(const cplx* __restrict__ hb, const cplx* __restrict__ X, int lx, int ly, int Q, int g,
                cplx* __restrict__ U1, cplx* __restrict__ U2) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int N = L1 * L2;
    const int kpts = (g + 1) * g;
    const int job = blockIdx.x, sample = job / kpts, t = job % kpts;
    const int t1 = t / g, t2 = t % g;
    cplx* S = reinterpret_cast<cplx*>(smem_raw);   // [N][L]
    cplx* stage = S + N * (L1 > L2 ? L1 : L2);      // [2][U, U'][8][N + 4]
    cplx* red = stage + 2 * 2 * LM_NS * (N + 4);    // [16][8]
    __shared__ cplx Dtab[LINK_MAXL];
    const int t2n = t2 + 1 == g ? 0 : t2 + 1;       // theta_2 = g is the copy of theta_2 = 0
    const cplx* ha = hb + ((size_t)t1 * (g + 1) + t2) * N * Q;
    const size_t nn = (size_t)N * N;
    const cplx* Xa = X + ((size_t)sample * kpts + t) * nn;
    const size_t o = ((size_t)sample * kpts + t) * N;
    if (t1 < g) {
        build_link_S(S, Dtab, ha, hb + ((size_t)(t1 + 1) * (g + 1) + t2) * N * Q, N, L1, ly, L1, Q, 0, -1.0 / g);
        __syncthreads();
        links_mma_dir<L1, L2>(S, stage, red, Xa, X + ((size_t)sample * kpts + (t1 + 1) * g + t2) * nn, ly, 0, U1 + o);
    }
    build_link_S(S, Dtab, ha, hb + ((size_t)t1 * (g + 1) + t2n) * N * Q, N, L2, ly, L1, Q, 1, (double)(t2 - t2n) / g);
    __syncthreads();
    links_mma_dir<L2, L1>(S, stage, red, Xa, X + ((size_t)sample * kpts + t1 * g + t2n) * nn, ly, 1, U2 + o);
}

template <int L1, int L2>
static int launch_links_thread(rlmb_context* ctx, const cplx* hb, const cplx* X, int lx, int ly, int Q, int g,
                               int nsamples, cplx* U1, cplx* U2) {
    const int N = lx * ly / Q;
    const size_t smem = (size_t)N * (L1 + L2) * sizeof(cplx);
    if (smem > 220 * 1024) return RLMB_ERR_ARG;
    RLMB_CUDA_TRY(cudaFuncSetAttribute(k_hlm_links<L1, L2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
    prof_begin(ctx, "k_hlm_links");
    k_hlm_links<L1, L2><<<nsamples * (g + 1) * g, 256, smem, ctx->stream>>>(hb, X, lx, ly, Q, g, U1, U2);
    RLMB_LAUNCHED(ctx);
    return RLMB_OK;
}

// Blocks of 8 and 16 are whole DMMA tiles; else warp-per-state links where their shared memory fits
// (the transposed S blocks and two staged rows per warp), else the thread-per-state kernel.
template <int L1, int L2>
static int launch_links_t(rlmb_context* ctx, const cplx* hb, const cplx* X, int lx, int ly, int Q, int g,
                          int nsamples, cplx* U1, cplx* U2) {
    if constexpr ((L1 == 8 || L1 == 16) && (L2 == 8 || L2 == 16)) {
        const size_t smem = links_mma_smem<L1, L2>();
        RLMB_CUDA_TRY(cudaFuncSetAttribute(k_hlm_links_mma<L1, L2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        prof_begin(ctx, "k_hlm_links");
        k_hlm_links_mma<L1, L2><<<nsamples * (g + 1) * g, LM_T, smem, ctx->stream>>>(hb, X, lx, ly, Q, g, U1, U2);
        RLMB_LAUNCHED(ctx);
        return RLMB_OK;
    } else {
        const int N = lx * ly / Q;
        const size_t smem_w = ((size_t)N * (L1 + L2) + (size_t)8 * 2 * N) * sizeof(cplx);
        if (smem_w > 220 * 1024) return launch_links_thread<L1, L2>(ctx, hb, X, lx, ly, Q, g, nsamples, U1, U2);
        RLMB_CUDA_TRY(cudaFuncSetAttribute(k_hlm_links_w<L1, L2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem_w));
        prof_begin(ctx, "k_hlm_links");
        k_hlm_links_w<L1, L2><<<nsamples * (g + 1) * g, 256, smem_w, ctx->stream>>>(hb, X, lx, ly, Q, g, U1, U2);
        RLMB_LAUNCHED(ctx);
        return RLMB_OK;
    }
}

int launch_hlm_links(rlmb_context* ctx, const cplx* hb, const cplx* X, int lx, int ly, int Q, int g,
                     int nsamples, cplx* U1, cplx* U2) {
    const int Lxp = lx / Q;
    // block sizes are compile-time so the U' block lives in registers; others are unsupported
#define RLMB_LINKS_CASE(A, B) \
    if (Lxp == A && ly == B) return launch_links_t<A, B>(ctx, hb, X, lx, ly, Q, g, nsamples, U1, U2);
    RLMB_LINKS_CASE(1, 1) RLMB_LINKS_CASE(1, 2) RLMB_LINKS_CASE(1, 3) RLMB_LINKS_CASE(1, 4)
    RLMB_LINKS_CASE(2, 2) RLMB_LINKS_CASE(2, 3) RLMB_LINKS_CASE(2, 4) RLMB_LINKS_CASE(2, 6)
    RLMB_LINKS_CASE(2, 8) RLMB_LINKS_CASE(3, 3) RLMB_LINKS_CASE(3, 6) RLMB_LINKS_CASE(4, 4)
    RLMB_LINKS_CASE(4, 8) RLMB_LINKS_CASE(8, 8) RLMB_LINKS_CASE(8, 16) RLMB_LINKS_CASE(16, 16)
    RLMB_LINKS_CASE(16, 8) RLMB_LINKS_CASE(4, 2) RLMB_LINKS_CASE(3, 2) RLMB_LINKS_CASE(6, 6)
    RLMB_LINKS_CASE(8, 4) RLMB_LINKS_CASE(12, 12) RLMB_LINKS_CASE(16, 32) RLMB_LINKS_CASE(32, 32)
    RLMB_LINKS_CASE(32, 16)
#undef RLMB_LINKS_CASE
    return launch_hlm_links_generic(ctx, hb, X, lx, ly, Q, g, nsamples, U1, U2);
}

}  // namespace rlmb
