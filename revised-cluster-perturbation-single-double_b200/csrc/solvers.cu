// Device-resident Davidson (src/lib_cc/mod_davidson.f90:40-728) and DIIS
// (src/libsrint/dosodiis2_d.f:1-119, dodiis.f, minv.f): one cluster of CTAs
// owns the whole subspace logic, so an iteration costs one step launch + the
// batched sigma contraction + one Ritz-matrix update.
#include "solvers.cuh"

#include <algorithm>
#include <atomic>

#include <cooperative_groups.h>

namespace cpsd {

namespace {
namespace cg = cooperative_groups;

constexpr int DT = 512;  // threads of a solver CTA

// The CTAs that own one subspace: a thread-block cluster (one CTA for short
// vectors), CTA r holding elements [lo, hi) of every vector.  Sums over whole
// vectors are formed per CTA and exchanged through distributed shared memory:
// every CTA then adds the partial sums in rank order, so all of them see the
// same bits and follow the same control flow without a broadcast.
struct Team {
    int size, rank, lo, hi;
    int flip = 0;
    __device__ Team(int n) {  // the cluster's own split of n elements
        const cg::cluster_group c = cg::this_cluster();
        size = (int)c.num_blocks();
        rank = (int)c.block_rank();
        const int chunk = ((n + size - 1) / size + 31) & ~31;
        lo = min(n, rank * chunk);
        hi = min(n, lo + chunk);
    }
    __device__ void sync() const {
        if (size > 1) cg::this_cluster().sync();
        else __syncthreads();
    }
    // the buffer of the next exchange (of two: a CTA that fills it has passed
    // the exchange after its last use, so nobody reads it any more)
    __device__ double *next(double *buf, int stride) {
        flip ^= 1;
        return buf + flip * stride;
    }
    // sum (or maximum) over the CTAs of entry e of an exchange buffer, to be
    // called after sync()
    __device__ double sum(const double *part, int e) const {
        if (size == 1) return part[e];
        double t = 0.0;
        for (int r = 0; r < size; r++) t += cg::this_cluster().map_shared_rank(const_cast<double *>(part), r)[e];
        return t;
    }
    __device__ double amax(const double *part, int e) const {
        if (size == 1) return part[e];
        double t = -1.0;
        for (int r = 0; r < size; r++)
            t = fmax(t, cg::this_cluster().map_shared_rank(const_cast<double *>(part), r)[e]);
        return t;
    }
    // no CTA leaves while another may still read its shared memory
    __device__ void leave() const {
        if (size > 1) cg::this_cluster().sync();
    }
};

// CTAs of a team: `per` elements each, up to `most` CTAs (16, of one GPC: above
// the portable 8)
int team_size(i64 n, i64 per, int most) {
    int c = 1;
    while (2 * c <= most && (i64)c * per < n) c *= 2;
    return c;
}

cudaLaunchConfig_t team_config(int teams, int size, size_t smem, cudaLaunchAttribute *at) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(teams * size));
    cfg.blockDim = dim3(DT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream();
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)size;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}
template <class... P, class... A>
int launch_team(void (*kern)(P...), int teams, int size, size_t smem, const char *what, A... args) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = team_config(teams, size, smem, at);
    return cuda_check(cudaLaunchKernelEx(&cfg, kern, P(args)...), what);
}
// Largest cluster of `kern` with up to smem bytes a CTA that the current device
// runs: 16 on a whole B200, fewer where part of the SMs is set aside.  Asked
// once per kernel and device, with the kernel's attributes set.
constexpr int TEAM_MAXDEV = 64;
template <class... P>
int team_most(void (*kern)(P...), size_t smem, std::atomic<int> (&cache)[TEAM_MAXDEV], int *most) {
    int dev = 0;
    CPSD_TRY(cuda_check(cudaGetDevice(&dev), "cudaGetDevice"));
    *most = dev < TEAM_MAXDEV ? cache[dev].load(std::memory_order_acquire) : 0;
    if (!*most) {
        if (smem)
            CPSD_TRY(cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                                "solver smem attr"));
        CPSD_TRY(cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1),
                            "solver cluster attr"));
        int size = 16;
        for (; size > 1; size /= 2) {
            cudaLaunchAttribute at[1];
            const cudaLaunchConfig_t cfg = team_config(1, size, smem, at);
            int active = 0;
            if (cudaOccupancyMaxActiveClusters(&active, kern, &cfg) == cudaSuccess && active > 0) break;
            cudaGetLastError();  // a size that the device refuses
        }
        *most = size;
        if (dev < TEAM_MAXDEV) cache[dev].store(size, std::memory_order_release);
    }
    *most = std::min(*most, ctx().team_cap);
    return CPSD_OK;
}

// value of the first element of largest magnitude (BLAS idamax semantics)
__device__ double block_amax(const double *x, int n, double *sh, int *shi) {
    double best = -1.0;
    int bi = 0x7fffffff;
    for (int k = threadIdx.x; k < n; k += DT) {
        double a = fabs(x[k]);
        if (a > best) {
            best = a;
            bi = k;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        double ob = __shfl_down_sync(0xffffffffu, best, o);
        int oi = __shfl_down_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) {
            best = ob;
            bi = oi;
        }
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) {
        sh[w] = best;
        shi[w] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = -1.0;
        int ii = 0x7fffffff;
        for (int i = 0; i < DT / 32; i++)
            if (sh[i] > b || (sh[i] == b && shi[i] < ii)) {
                b = sh[i];
                ii = shi[i];
            }
        shi[DT / 32] = ii;
    }
    __syncthreads();
    int idx = shi[DT / 32];
    __syncthreads();
    return (idx < n) ? x[idx] : 0.0;
}

// dot product of two length-n vectors by one warp (result in every lane)
__device__ double warp_dot(const double *x, const double *y, int n) {
    const int lane = threadIdx.x & 31;
    double a = 0.0;
#pragma unroll 4
    for (int k = lane; k < n; k += 32) a = fma(x[k], y[k], a);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

constexpr int GL = DAV_MAXD + 1;

// Index that round robin pairing r (0 <= r < m - 1) of m = 2, 4, .. indices has
// at place i: places 2k and 2k + 1 are a pair, {m - 1, r} for k = 0 and {r - k,
// r + k} modulo m - 1 for the others
__device__ __forceinline__ int jacobi_at(int i, int m, int r) {
    const int k = i >> 1;
    if (i & 1) return r + k < m - 1 ? r + k : r + k - (m - 1);
    return k == 0 ? m - 1 : r - k >= 0 ? r - k : r - k + m - 1;
}

// The symmetric n x n matrix a(i, j) into S (ld GL) in the places of the first
// pairing of m = n rounded up to even, zero where an index is n: the padding of
// an odd n, which sits at place 0 throughout
template <class F>
__device__ void jacobi_place(double *S, int n, F a) {
    const int m = (n + 1) & ~1;
    for (int e = threadIdx.x; e < DAV_MAXD * DAV_MAXD; e += DT) {
        const int p = e / DAV_MAXD, q = e % DAV_MAXD;
        const int i = p < m ? jacobi_at(p, m, 0) : n, j = q < m ? jacobi_at(q, m, 0) : n;
        S[p * GL + q] = i < n && j < n ? a(i, j) : 0.0;
    }
    __syncthreads();
}

// Cyclic Jacobi by the whole block on the symmetric n x n matrix that
// jacobi_place put into S: w receives the eigenvalues; the eigenvector of w[k]
// is column place[k] of the returned matrix (ld GL), which is V or V2.  S, S2,
// V and V2 are of the same size.  The order of the rotations is part of the
// result, as it decides the sign of every eigenvector.  Classic threshold
// (Golub & Van Loan, Alg. 8.5.3): an element with a_pq^2 <= 1e-34 |a_pp a_qq|
// is negligible and set to zero.  The
// n(n-1)/2 rotations of a sweep run as n-1 rounds of n/2 disjoint rotations
// (round-robin pairing, n padded to even), each round one parallel update of
// S and V.  The iteration ends at the first round whose matrix has no
// element above the threshold: later rounds would change nothing.  The
// rotation of a pair is the smaller root t of t^2 + 2 tau t - 1 = 0, tau =
// d / b, d = a_qq - a_pp, b = 2 a_pq, by its half angle:
//   h = 1 / sqrt(d^2 + b^2),  u = (1 + |d| h) / 2,  r = 1 / sqrt(u),
//   c = u r,  s = sgn(d b) |b| h r / 2,
// two reciprocal roots after one another and no division, and one correction
// of c^2 + s^2 to 1; a pair whose d^2 + b^2 leaves the normal range is scaled
// first.
//
// Latency bounds it: about 80 rounds at n = 20, each a chain of the rotation
// parameters, a barrier, one 2 x 2 update and a barrier.  So pair k always
// sits in rows and columns 2k and 2k + 1 and the update writes to the places
// of the next round's pairing, in the other of two buffers: every address of
// a thread is the same in all rounds.  (Indexing the pairs anew took 1250
// cycles a round; roots, divisions and the index arithmetic 2000.)
__device__ double *block_jacobi(double *S, double *V, double *S2, double *V2, int n, double *w, int *place) {
    __shared__ double cs[DAV_MAXD / 2], sn[DAV_MAXD / 2], tn[DAV_MAXD / 2];
    __shared__ int rotate;  // last round that saw an element above the threshold
    const int tid = threadIdx.x;
    const int m = (n + 1) & ~1, half = m / 2;
    for (int e = tid; e < DAV_MAXD * DAV_MAXD; e += DT) {
        const int i = e / DAV_MAXD, j = e % DAV_MAXD;
        V[i * GL + j] = (j < m && i == jacobi_at(j, m, 0)) ? 1.0 : 0.0;
        V2[i * GL + j] = 0.0;
    }
    if (tid == 0) rotate = 0;
    // round robin: the players of a circle move one place on, the one at
    // place 0 stays; place 2k faces 2k + 1
    auto next = [&](int i) {
        if (i == 0 || m == 2) return i;
        if (i == m - 2) return m - 1;           // end of the upper row turns back
        if ((i & 1) == 0) return i + 2;         // upper row moves out
        return i == 1 ? 2 : i - 2;              // lower row moves in
    };
    // this thread's elements i < j of the threshold test (warps 1..: at most
    // two of the 496), numbered along the rows
    int to[2] = {-1, -1}, tp[2] = {0, 0}, tq[2] = {0, 0};
    if (tid >= 32)
#pragma unroll
        for (int w = 0; w < 2; w++) {
            int e = tid - 32 + w * (DT - 32);
            if (e < m * (m - 1) / 2) {
                int i = 0;
                while (e >= m - 1 - i) e -= m - 1 - i++;
                const int j = i + 1 + e;
                to[w] = i * GL + j;
                tp[w] = i * (GL + 1);
                tq[w] = j * (GL + 1);
            }
        }
    // its 2 x 2 block (pair k rows, pair l columns) of S (first half of the
    // threads), or its two (row, pair) items of V (second half)
    const bool on_s = tid < DT / 2;
    const int e0 = on_s ? tid : tid - DT / 2;
    const int k0 = e0 / half, l0 = e0 - k0 * half;
    const int e1 = e0 + DT / 2, k1 = e1 / half, l1 = e1 - k1 * half;
    const bool live0 = on_s ? k0 < half : k0 < m, live1 = !on_s && k1 < m;
    const int cp = next(2 * l0), cq = next(2 * l0 + 1);
    int r0, r1, w00, w01, w10, w11;
    if (on_s) {
        r0 = 2 * k0 * GL + 2 * l0;
        r1 = r0 + GL;
        w00 = next(2 * k0) * GL + cp;
        w01 = next(2 * k0) * GL + cq;
        w10 = next(2 * k0 + 1) * GL + cp;
        w11 = next(2 * k0 + 1) * GL + cq;
    } else {
        r0 = k0 * GL + 2 * l0;
        r1 = k1 * GL + 2 * l1;
        w00 = k0 * GL + cp;
        w01 = k0 * GL + cq;
        w10 = k1 * GL + next(2 * l1);
        w11 = k1 * GL + next(2 * l1 + 1);
    }
    const bool dia = on_s && k0 == l0;
    double *A = S, *B = S2, *E = V, *F = V2;
    int r = 0;  // pairing of the round
    // indices of this thread's rotation (threads below half)
    int pa = jacobi_at(2 * tid, m, 0), pb = tid;
    __syncthreads();
    for (int round = 1; round <= 50 * (m - 1); round++) {
        // does any element of the matrix still call for a rotation?
        // (asked by warps 1.., beside warp 0's rotation parameters)
        bool above = false;
#pragma unroll
        for (int w = 0; w < 2; w++)
            if (to[w] >= 0) {
                const double x = A[to[w]];
                above |= !(x * x <= 1.0e-34 * fabs(A[tp[w]] * A[tq[w]]) || x == 0.0);
            }
        if (above) rotate = round;
        const double *src = on_s ? A : E;
        double b00 = 0.0, b01 = 0.0, b10 = 0.0, b11 = 0.0;
        if (live0) {
            b00 = src[r0];
            b01 = src[r0 + 1];
        }
        if (on_s ? live0 : live1) {
            b10 = src[r1];
            b11 = src[r1 + 1];
        }
        if (tid < half) {
            const int o = 2 * tid * (GL + 1);
            const double app = A[o], aqq = A[o + GL + 1], apq = A[o + 1];
            double d = aqq - app, b = 2.0 * apq, h2 = fma(d, d, b * b);
            const bool keep = apq * apq <= 1.0e-34 * fabs(app * aqq) || apq == 0.0;
            if (!keep && !(h2 > 1.0e-290 && h2 < 1.0e290)) {
                const double f = 1.0 / fmax(fabs(d), fabs(b));
                d *= f;
                b *= f;
                h2 = fma(d, d, b * b);
            }
            const double h = rsqrt(h2), u = fma(0.5 * fabs(d), h, 0.5), ru = rsqrt(u);
            double c = u * ru, s = 0.5 * fabs(b) * h * ru;
            // c and s hold the rounding of h apart from one another: scaled to
            // c^2 + s^2 = 1 (the defect itself, not 1 less half of it, which
            // would round one way only)
            const double z = fma(-s, s, fma(-c, c, 1.0));
            c = fma(0.5 * c, z, c);
            s = fma(0.5 * s, z, s);
            // equal diagonal elements: t = 1 from the lower to the higher index
            if (d == 0.0 ? pa > pb : (d > 0.0) != (b > 0.0)) s = -s;
            cs[tid] = keep ? 1.0 : c;
            sn[tid] = keep ? 0.0 : s;
            tn[tid] = keep ? 0.0 : s * ru;  // s / c
        }
        __syncthreads();
        if (rotate != round) break;
        // S <- J^T S J on the 2x2 blocks, V <- V J
        const double cl = cs[l0 < half ? l0 : 0], sl = sn[l0 < half ? l0 : 0];
        if (on_s) {
            if (live0) {
                const double ck = cs[k0], sk = sn[k0];
                const double t00 = cl * b00 - sl * b01, t01 = sl * b00 + cl * b01;
                const double t10 = cl * b10 - sl * b11, t11 = sl * b10 + cl * b11;
                const double tk = tn[k0];
                // a pair's own block: a_pp - t a_pq, a_qq + t a_pq, so that c^2
                // + s^2 being 1 to rounding only does not add up in the
                // eigenvalues, and an annihilated (or negligible) element
                B[w00] = dia ? fma(-tk, b01, b00) : ck * t00 - sk * t10;
                B[w01] = dia ? 0.0 : ck * t01 - sk * t11;
                B[w10] = dia ? 0.0 : sk * t00 + ck * t10;
                B[w11] = dia ? fma(tk, b01, b11) : sk * t01 + ck * t11;
            }
        } else {
            if (live0) {
                F[w00] = cl * b00 - sl * b01;
                F[w01] = sl * b00 + cl * b01;
            }
            if (live1) {
                const double c = cs[l1], s = sn[l1];
                F[w10] = c * b10 - s * b11;
                F[w11] = s * b10 + c * b11;
            }
        }
        double *x = A;
        A = B;
        B = x;
        x = E;
        E = F;
        F = x;
        r = r + 1 < m - 1 ? r + 1 : 0;
        pa = tid == 0 ? pa : pa + 1 < m - 1 ? pa + 1 : 0;
        pb = pb + 1 < m - 1 ? pb + 1 : 0;
        __syncthreads();
    }
    if (tid < m) {
        const int k = jacobi_at(tid, m, r);
        if (k < n) {
            w[k] = A[tid * (GL + 1)];
            place[k] = tid;
        }
    }
    __syncthreads();
    return E;
}

// ------------------------------------------------ general real eigenproblem
// Eigenvalues and right eigenvectors of a general real n x n matrix (n <= 32)
// by one warp, in the form LAPACK's dgeev('N', 'V') returns them to the
// reference's Davidson (src/lib_cc/mod_davidson.f90:185-186): wr / wi the
// eigenvalues, a complex pair at (k, k + 1) with wi[k] > 0 first; column k
// of V the eigenvector of a real eigenvalue, columns k and k + 1 the real and
// imaginary parts of the eigenvector of wr[k] + i wi[k]; every eigenvector
// of unit 2-norm with its largest component real.  Method (Golub & Van Loan,
// Matrix Computations, 4th ed., sections 7.4-7.5 and 7.6.4):
//   1. Householder reduction to upper Hessenberg form, H = Z^T A Z;
//   2. Francis double-shift QR sweeps on the active window [l, hi] to real
//      Schur form T, Z accumulated; a subdiagonal element at most eps times
//      its two diagonal neighbours deflates; sweeps 10 and 20 of a window
//      use the ad-hoc exceptional shift of the LAPACK/EISPACK QR codes;
//      a 2 x 2 block with real eigenvalues is rotated to triangular form;
//   3. eigenvectors of T by back substitution (lane e solves for eigenvalue
//      e, complex arithmetic for a pair), then V = Z X and normalisation.
// Lane i owns row i or column i of every update; every lane walks the same
// control flow (deflation tests, shifts and reflectors are computed from
// shared values by all lanes alike).  H, Z and X are row-major with leading
// dimension GL (odd, so that a lane per row hits distinct banks); H is
// destroyed, Z and X are scratch, V (leading dimension GL, may alias Z)
// receives the vectors.  Returns the number of QR sweeps, or -1 when a
// window did not converge within 30 max(10, n) sweeps.

__device__ __forceinline__ double warp_allsum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_allmax(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

struct cplx {
    double re, im;
};
__device__ __forceinline__ cplx cmul(cplx a, cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ cplx csub(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }
// a / b by Smith's scaling (R. L. Smith, CACM 5 (1962) 435); |b| >= tiny
__device__ cplx cdiv(cplx a, cplx b, double tiny) {
    if (fabs(b.re) + fabs(b.im) < tiny) b = {tiny, 0.0};
    if (fabs(b.re) >= fabs(b.im)) {
        const double r = b.im / b.re, d = b.re + b.im * r;
        return {(a.re + a.im * r) / d, (a.im - a.re * r) / d};
    }
    const double r = b.re / b.im, d = b.im + b.re * r;
    return {(a.re * r + a.im) / d, (a.im * r - a.re) / d};
}

// x of the 2 x 2 system [[t00 - lam, t01], [t10, t11 - lam]] x = -rhs
// (Cramer's rule with the determinant kept away from zero)
__device__ void solve2(double t00, double t01, double t10, double t11, cplx lam, cplx r0, cplx r1, double tiny,
                       cplx *x0, cplx *x1) {
    const cplx a = {t00 - lam.re, -lam.im}, d = {t11 - lam.re, -lam.im};
    const cplx det = csub(cmul(a, d), {t01 * t10, 0.0});
    const cplx b0 = {-r0.re, -r0.im}, b1 = {-r1.re, -r1.im};
    *x0 = cdiv(csub(cmul(b0, d), {t01 * b1.re, t01 * b1.im}), det, tiny);
    *x1 = cdiv(csub(cmul(a, b1), {t10 * b0.re, t10 * b0.im}), det, tiny);
}

__device__ int warp_geev(double *H, double *Z, double *X, double *V, double *wr, double *wi, int n) {
    const int lane = threadIdx.x & 31;
    const double eps = 2.220446049250313e-16;
    for (int i = 0; i < n; i++)
        if (lane < n) Z[i * GL + lane] = (i == lane) ? 1.0 : 0.0;
    __syncwarp();
    // ---- 1. Hessenberg form: reflector k zeroes column k below row k + 1
    for (int k = 0; k + 2 < n; k++) {
        const double xi = (lane > k && lane < n) ? H[lane * GL + k] : 0.0;
        const double tail2 = warp_allsum(lane > k + 1 ? xi * xi : 0.0);
        if (tail2 == 0.0) continue;  // column already reduced (same on every lane)
        const double x0 = H[(k + 1) * GL + k];
        const double alpha = -copysign(sqrt(tail2 + x0 * x0), x0);
        const double beta = 1.0 / (alpha * (alpha - x0));  // 2 / v^T v
        if (lane < n) X[lane] = (lane == k + 1) ? x0 - alpha : (lane > k + 1 ? xi : 0.0);
        __syncwarp();
        if (lane >= k && lane < n) {  // H <- P H, lane = column
            double s = 0.0;
            for (int i = k + 1; i < n; i++) s += X[i] * H[i * GL + lane];
            s *= beta;
            for (int i = k + 1; i < n; i++) H[i * GL + lane] -= s * X[i];
            if (lane == k) {
                H[(k + 1) * GL + k] = alpha;
                for (int i = k + 2; i < n; i++) H[i * GL + k] = 0.0;
            }
        }
        __syncwarp();
        if (lane < n) {  // H <- H P and Z <- Z P, lane = row
            double s = 0.0, t = 0.0;
            for (int j = k + 1; j < n; j++) {
                s += H[lane * GL + j] * X[j];
                t += Z[lane * GL + j] * X[j];
            }
            s *= beta;
            t *= beta;
            for (int j = k + 1; j < n; j++) {
                H[lane * GL + j] -= s * X[j];
                Z[lane * GL + j] -= t * X[j];
            }
        }
        __syncwarp();
    }
    // 1-norm of H: the scale of the deflation test when both diagonal
    // neighbours vanish
    double cn = 0.0;
    if (lane < n)
        for (int i = 0; i < n; i++) cn += fabs(H[i * GL + lane]);
    const double anorm = warp_allmax(cn);
    const double tiny = fmax(eps * anorm, 1.0e-300);
    // ---- 2. real Schur form
    const int maxits = 30 * max(10, n);
    int hi = n - 1, its = 0, sweeps = 0;
    while (hi >= 0) {
        int l = hi;
        for (; l > 0; l--) {
            double s = fabs(H[(l - 1) * GL + l - 1]) + fabs(H[l * GL + l]);
            if (s == 0.0) s = anorm;
            if (fabs(H[l * GL + l - 1]) <= eps * s) break;
        }
        __syncwarp();
        if (l > 0 && lane == 0) H[l * GL + l - 1] = 0.0;
        __syncwarp();
        if (l == hi) {  // 1 x 1 block
            if (lane == 0) {
                wr[hi] = H[hi * GL + hi];
                wi[hi] = 0.0;
            }
            hi--;
            its = 0;
            continue;
        }
        if (l == hi - 1) {  // 2 x 2 block
            const int m = hi - 1;
            const double a = H[m * GL + m], b = H[m * GL + hi], c = H[hi * GL + m], d = H[hi * GL + hi];
            const double p = 0.5 * (a - d), disc = p * p + b * c;
            if (disc >= 0.0) {
                // real pair: rotate by G = [cs -sn; sn cs] whose first column
                // is the eigenvector (z, c) of lam1 = d + z
                const double z = p + copysign(sqrt(disc), p);
                const double lam1 = d + z, lam2 = (z != 0.0) ? d - (b * c) / z : lam1;
                const double r = hypot(z, c), cs = z / r, sn = c / r;
                if (lane >= m && lane < n) {
                    const double hm = H[m * GL + lane], hh = H[hi * GL + lane];
                    H[m * GL + lane] = cs * hm + sn * hh;
                    H[hi * GL + lane] = -sn * hm + cs * hh;
                }
                __syncwarp();
                if (lane < n) {
                    if (lane <= hi) {
                        const double hm = H[lane * GL + m], hh = H[lane * GL + hi];
                        H[lane * GL + m] = cs * hm + sn * hh;
                        H[lane * GL + hi] = -sn * hm + cs * hh;
                    }
                    const double zm = Z[lane * GL + m], zh = Z[lane * GL + hi];
                    Z[lane * GL + m] = cs * zm + sn * zh;
                    Z[lane * GL + hi] = -sn * zm + cs * zh;
                }
                __syncwarp();
                if (lane == 0) {
                    H[hi * GL + m] = 0.0;
                    H[m * GL + m] = lam1;
                    H[hi * GL + hi] = lam2;
                    wr[m] = lam1;
                    wr[hi] = lam2;
                    wi[m] = wi[hi] = 0.0;
                }
            } else if (lane == 0) {  // complex pair: the block stays
                wr[m] = wr[hi] = 0.5 * (a + d);
                wi[m] = sqrt(-disc);
                wi[hi] = -wi[m];
            }
            __syncwarp();
            hi -= 2;
            its = 0;
            continue;
        }
        if (its >= maxits) return -1;
        its++;
        sweeps++;
        double h11, h12, h21, h22;  // the shifts are the eigenvalues of [h11 h12; h21 h22]
        if (its == 10 || its == 20) {
            const double s = (its == 10) ? fabs(H[(l + 1) * GL + l]) + fabs(H[(l + 2) * GL + l + 1])
                                         : fabs(H[hi * GL + hi - 1]) + fabs(H[(hi - 1) * GL + hi - 2]);
            h11 = 0.75 * s + ((its == 10) ? H[l * GL + l] : H[hi * GL + hi]);
            h12 = -0.4375 * s;
            h21 = s;
            h22 = h11;
        } else {
            h11 = H[(hi - 1) * GL + hi - 1];
            h12 = H[(hi - 1) * GL + hi];
            h21 = H[hi * GL + hi - 1];
            h22 = H[hi * GL + hi];
        }
        const double tr = h11 + h22, det = h11 * h22 - h12 * h21;
        // first column of (H - s1)(H - s2) in the window
        const double hll = H[l * GL + l], h1l = H[(l + 1) * GL + l];
        double x = hll * hll + H[l * GL + l + 1] * h1l - tr * hll + det;
        double y = h1l * (hll + H[(l + 1) * GL + l + 1] - tr);
        double z = h1l * H[(l + 2) * GL + l + 1];
        for (int k = l; k <= hi - 1; k++) {
            const bool three = k < hi - 1;  // reflector length 3, else 2
            if (!three) z = 0.0;
            const double t2 = y * y + z * z;
            if (t2 != 0.0) {
                const double alpha = -copysign(sqrt(x * x + t2), x);
                const double beta = 1.0 / (alpha * (alpha - x));
                const double v0 = x - alpha, v1 = y, v2 = z;
                const int q = max(l, k - 1);
                if (lane >= q && lane < n) {  // rows k.. of columns q..n-1
                    double a0 = H[k * GL + lane], a1 = H[(k + 1) * GL + lane];
                    double a2 = three ? H[(k + 2) * GL + lane] : 0.0;
                    const double s = beta * (v0 * a0 + v1 * a1 + v2 * a2);
                    a0 -= s * v0;
                    a1 -= s * v1;
                    a2 -= s * v2;
                    if (lane == k - 1) {  // the bulge column: exactly (alpha, 0, 0)
                        a0 = alpha;
                        a1 = a2 = 0.0;
                    }
                    H[k * GL + lane] = a0;
                    H[(k + 1) * GL + lane] = a1;
                    if (three) H[(k + 2) * GL + lane] = a2;
                }
                __syncwarp();
                if (lane < n) {  // columns k.. of rows 0..min(k+3, hi); Z all rows
                    if (lane <= min(k + 3, hi)) {
                        const double a0 = H[lane * GL + k], a1 = H[lane * GL + k + 1];
                        const double a2 = three ? H[lane * GL + k + 2] : 0.0;
                        const double s = beta * (a0 * v0 + a1 * v1 + a2 * v2);
                        H[lane * GL + k] = a0 - s * v0;
                        H[lane * GL + k + 1] = a1 - s * v1;
                        if (three) H[lane * GL + k + 2] = a2 - s * v2;
                    }
                    const double c0 = Z[lane * GL + k], c1 = Z[lane * GL + k + 1];
                    const double c2 = three ? Z[lane * GL + k + 2] : 0.0;
                    const double s = beta * (c0 * v0 + c1 * v1 + c2 * v2);
                    Z[lane * GL + k] = c0 - s * v0;
                    Z[lane * GL + k + 1] = c1 - s * v1;
                    if (three) Z[lane * GL + k + 2] = c2 - s * v2;
                }
                __syncwarp();
            }
            if (three) {
                x = H[(k + 1) * GL + k];
                y = H[(k + 2) * GL + k];
                z = (k < hi - 2) ? H[(k + 3) * GL + k] : 0.0;
            }
        }
    }
    __syncwarp();
    // ---- 3. eigenvectors of T (lane e: eigenvalue e; a pair by its first lane)
    if (lane < n && wi[lane] >= 0.0) {
        const int e = lane;
        const cplx lam = {wr[e], wi[e]};
        const bool pair = wi[e] > 0.0;
        const int top = pair ? e + 1 : e;  // last nonzero row of x
        for (int i = top + 1; i < n; i++) {
            X[i * GL + e] = 0.0;
            if (pair) X[i * GL + e + 1] = 0.0;
        }
        // x[i] kept as (X[i][e], X[i][e+1]) for a pair, X[i][e] otherwise
        if (pair) {
            // eigenvector of the block [a b; c d] for lam: (lam - d, c) or
            // (b, lam - a), whichever is longer
            const double a = H[e * GL + e], b = H[e * GL + e + 1], c = H[(e + 1) * GL + e], d = H[(e + 1) * GL + e + 1];
            const cplx u0 = {lam.re - d, lam.im}, w1 = {lam.re - a, lam.im};
            const double nu = u0.re * u0.re + u0.im * u0.im + c * c, nw = b * b + w1.re * w1.re + w1.im * w1.im;
            const cplx x0 = (nu >= nw) ? u0 : cplx{b, 0.0}, x1 = (nu >= nw) ? cplx{c, 0.0} : w1;
            X[e * GL + e] = x0.re;
            X[e * GL + e + 1] = x0.im;
            X[(e + 1) * GL + e] = x1.re;
            X[(e + 1) * GL + e + 1] = x1.im;
        } else {
            X[e * GL + e] = 1.0;
        }
        auto xval = [&](int j) -> cplx {
            return pair ? cplx{X[j * GL + e], X[j * GL + e + 1]} : cplx{X[j * GL + e], 0.0};
        };
        auto rowsum = [&](int i, int j0) -> cplx {  // sum_{j >= j0} T[i][j] x[j]
            cplx r = {0.0, 0.0};
            for (int j = j0; j <= top; j++) {
                const cplx xj = xval(j);
                r.re += H[i * GL + j] * xj.re;
                r.im += H[i * GL + j] * xj.im;
            }
            return r;
        };
        for (int i = e - 1; i >= 0;) {
            if (i > 0 && H[i * GL + i - 1] != 0.0) {  // rows i-1, i: a 2 x 2 block
                const cplx r0 = rowsum(i - 1, i + 1), r1 = rowsum(i, i + 1);
                cplx x0, x1;
                solve2(H[(i - 1) * GL + i - 1], H[(i - 1) * GL + i], H[i * GL + i - 1], H[i * GL + i], lam, r0, r1,
                       tiny, &x0, &x1);
                X[(i - 1) * GL + e] = x0.re;
                X[i * GL + e] = x1.re;
                if (pair) {
                    X[(i - 1) * GL + e + 1] = x0.im;
                    X[i * GL + e + 1] = x1.im;
                }
                i -= 2;
            } else {
                const cplx r = rowsum(i, i + 1);
                const cplx xi = cdiv({-r.re, -r.im}, {H[i * GL + i] - lam.re, -lam.im}, tiny);
                X[i * GL + e] = xi.re;
                if (pair) X[i * GL + e + 1] = xi.im;
                i -= 1;
            }
        }
    }
    __syncwarp();
    // V = Z X into H (T is no longer read); lane e: column e
    if (lane < n) {
        const int top = (wi[lane] > 0.0) ? lane + 1 : lane;
        for (int i = 0; i < n; i++) {
            double s = 0.0;
            for (int j = 0; j <= top; j++) s += Z[i * GL + j] * X[j * GL + lane];
            H[i * GL + lane] = s;
        }
    }
    __syncwarp();
    // unit 2-norm, largest component real (a pair: by its first lane)
    if (lane < n && wi[lane] >= 0.0) {
        const int e = lane;
        if (wi[e] == 0.0) {
            double s = 0.0;
            for (int i = 0; i < n; i++) s += H[i * GL + e] * H[i * GL + e];
            const double f = 1.0 / sqrt(s);
            for (int i = 0; i < n; i++) H[i * GL + e] *= f;
        } else {
            double s = 0.0, best = -1.0;
            int kb = 0;
            for (int i = 0; i < n; i++) {
                const double m2 = H[i * GL + e] * H[i * GL + e] + H[i * GL + e + 1] * H[i * GL + e + 1];
                s += m2;
                if (m2 > best) {
                    best = m2;
                    kb = i;
                }
            }
            // multiply by conj(v_kb) / (|v_kb| |v|)
            const double mk = sqrt(best), f = 1.0 / (sqrt(s) * mk);
            const double cr = H[kb * GL + e] * f, ci = H[kb * GL + e + 1] * f;
            for (int i = 0; i < n; i++) {
                const double re = H[i * GL + e], im = H[i * GL + e + 1];
                H[i * GL + e] = re * cr + im * ci;
                H[i * GL + e + 1] = im * cr - re * ci;
            }
            H[kb * GL + e + 1] = 0.0;
        }
    }
    __syncwarp();
    // each column to unit norm where it is off by more than 1e-10, as the
    // reference does with the real and imaginary parts it keeps
    // (mod_davidson.f90:211-217)
    if (lane < n) {
        double s = 0.0;
        for (int i = 0; i < n; i++) s += H[i * GL + lane] * H[i * GL + lane];
        const double t = sqrt(s), f = (fabs(t - 1.0) > 1.0e-10) ? 1.0 / t : 1.0;
        for (int i = 0; i < DAV_MAXD; i++) V[i * GL + lane] = (i < n) ? H[i * GL + lane] * f : 0.0;
    } else {
        for (int i = 0; i < DAV_MAXD; i++) V[i * GL + lane] = 0.0;
    }
    __syncwarp();
    return sweeps;
}

// Schmidt_2D (mod_davidson.f90:642-680) on the dim columns (length len <= 32)
// of v (leading dimension GL), in place by the whole block: modified
// Gram-Schmidt, each column projected on the earlier ones in the reference's
// order; a warp per later column takes out column j as soon as it is final
__device__ void block_schmidt_2d(double *v, int len, int dim) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int j = 0; j < dim; j++) {
        if (j > 0) {
            if (w == 0) {
                const double x = lane < len ? v[j * GL + lane] : 0.0;
                const double nrm = sqrt(warp_allsum(x * x));
                if (lane < len) v[j * GL + lane] = x * (1.0 / nrm);
            }
            __syncthreads();
        }
        const double y = lane < len ? v[j * GL + lane] : 0.0;
        for (int i = j + 1 + w; i < dim; i += DT / 32) {
            const double x = lane < len ? v[i * GL + lane] : 0.0;
            const double ov = warp_allsum(x * y);
            if (lane < len) v[i * GL + lane] = x + -ov * y;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(DT) k_dav_init(DavState *st, DavBuffers b) {
    DavState &s = *st;
    const int n = s.dimA, D = s.D, nr = s.nroot;
    for (int e = threadIdx.x >> 5; e < nr * nr; e += DT / 32) {
        const int i = e / nr, j = e % nr;
        double v = warp_dot(b.fileEV + (size_t)j * (n + 1) + 1, b.AB[0] + (size_t)i * n, n);
        if ((threadIdx.x & 31) == 0) s.Abar[j + i * D] = v;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < nr; i++) s.eigenVal[i] = b.fileEV[(size_t)i * (n + 1)];
        s.iterations = 1;
        s.dimIter = nr;
        s.dimFree = D - nr;
        s.dim_exceed = 0;
        s.cur = 0;
        s.done = 0;
        s.converged = 0;
        s.pending = 0;
    }
}

// Shared memory of a Davidson step.  S, X and V hold the Ritz problem, then S
// the collapse coefficients; ex is the double-buffered exchange of a step's
// partial sums (overlaps with the basis and Gram matrix of the new vectors,
// or the collapsed Ritz matrix), tot their sums over the CTAs.
constexpr int DAV_EX = 2 * DAV_MAXD * DAV_MAXD;
constexpr int DOT_RT = 4;  // row tiles of eight vectors per pass of the products
struct DavShared {
    double S[DAV_MAXD * GL], V[DAV_MAXD * GL], X[DAV_MAXD * GL];
    double ex[2][DAV_EX], tot[DAV_EX];
    double red[DT / 32][DOT_RT * 64];  // one pass's products of each warp
    double L[DAV_MAXD * GL];           // Cholesky factor of the new vectors
    double2 cf[DAV_MAXD][4];           // coefficients of eight outputs
    double vR[DAV_MAXD], vI[DAV_MAXD], ev[DAV_MAXD], rnorm[DAV_MAXD];
    int lw[DAV_MAXD], act[DAV_MAXD], cvd[DAV_MAXD];
    int place[DAV_MAXD];  // column of an eigenvector
    int general, eig_fail, warn, nnew;
};

// The basis, its sigma vectors and the work vectors of a step live in shared
// memory when this many doubles hold a CTA's part of them (n up to 4096
// with 16 CTAs, a basis of 20 and 5 roots): copied there while the Ritz
// problem is solved, they cost one latency instead of one for each of the
// step's eight passes.
constexpr int DAV_LOCAL = 13312;
// elements a CTA, up to 16 CTAs: n = 858, 5 roots, 94 us a step at 112, 100 at
// 224, 111 at 448 (150 on one CTA); n = 174, 3 roots, 44 us at 112, 42.5 at 224
constexpr int DAV_PER = 192;
// leading dimension of vectors in shared memory: 4 mod 16, so that 8 vectors
// by 4 elements fall on different banks
__host__ __device__ constexpr int dav_ld(int nc) { return (nc + 11) / 16 * 16 + 4; }

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// coefficients c(i, r0 + q), q < 8, of nb vectors into cf (zero past nr)
template <class F>
__device__ void put_coefs(double2 (*cf)[4], int nb, int r0, int nr, F coef) {
    __syncthreads();
    for (int e = threadIdx.x; e < nb * 8; e += DT) {
        const int i = e >> 3, q = e & 7;
        reinterpret_cast<double *>(cf[i])[q] = r0 + q < nr ? coef(i, r0 + q) : 0.0;
    }
    __syncthreads();
}

// out(r, k, sum_i c(i, r) x_i[k], sum_i c(i, r) y_i[k]) for r < nr and the nc
// elements k of this CTA, 8 outputs a pass so that every x_i, y_i is loaded
// once for them (sums in basis order); the coefficients are read as pairs, a
// broadcast of four loads a basis vector
template <class F, class G>
__device__ void combine(double2 (*cf)[4], int nc, int nb, int nr, const double *x, const double *y, i64 ld, F coef,
                        G out) {
    for (int r0 = 0; r0 < nr; r0 += 8) {
        put_coefs(cf, nb, r0, nr, coef);
        for (int k = threadIdx.x; k < nc; k += DT) {
            double a[8], c[8];
#pragma unroll
            for (int q = 0; q < 8; q++) a[q] = c[q] = 0.0;
#pragma unroll 4
            for (int i = 0; i < nb; i++) {
                const double u = x[i * ld + k], v = y[i * ld + k];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const double2 f = cf[i][q];
                    a[2 * q] += f.x * u;
                    a[2 * q + 1] += f.y * u;
                    c[2 * q] += f.x * v;
                    c[2 * q + 1] += f.y * v;
                }
            }
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (r0 + q < nr) out(r0 + q, k, a[q], c[q]);
        }
    }
}

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// part[i * nw + q] = x_i . w_act[q] over this CTA's elements for i < nx and,
// with gram, part[(nx + p) * nw + q] = w_act[p] . w_act[q].  FP64 tensor
// instructions: a warp takes every 16th group of 8 elements, tiles of 8
// vectors by 8; so each vector is read once for eight products.  Ends with a
// block barrier.
__device__ void team_dots(DavShared &sm, int nc, const double *x, i64 ldx, int nx, const double *w, i64 ldw,
                          const int *act, int nw, bool gram, double *part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int rows = nx + (gram ? nw : 0);
    for (int q0 = 0; q0 < nw; q0 += 8) {
        const double *wp = q0 + g < nw ? w + act[q0 + g] * ldw : nullptr;
        for (int i0 = 0; i0 < rows; i0 += 8 * DOT_RT) {
            const double *xp[DOT_RT];
            double acc[DOT_RT][2];
#pragma unroll
            for (int r = 0; r < DOT_RT; r++) {
                const int i = i0 + 8 * r + g;
                xp[r] = i < nx ? x + i * ldx : i < rows ? w + act[i - nx] * ldw : nullptr;
                acc[r][0] = acc[r][1] = 0.0;
            }
            const int nt = min(DOT_RT, (rows - i0 + 7) / 8);
#pragma unroll 2
            for (int k = 8 * warp; k < nc; k += 8 * (DT / 32)) {
                const int ka = k + c, kb = ka + 4;
                const double ba = wp && ka < nc ? wp[ka] : 0.0, bb = wp && kb < nc ? wp[kb] : 0.0;
                double aa[DOT_RT], ab[DOT_RT];
#pragma unroll
                for (int r = 0; r < DOT_RT; r++) {
                    aa[r] = xp[r] && ka < nc ? xp[r][ka] : 0.0;
                    ab[r] = xp[r] && kb < nc ? xp[r][kb] : 0.0;
                }
#pragma unroll
                for (int r = 0; r < DOT_RT; r++)
                    if (r < nt) {
                        dmma884(acc[r], aa[r], ba);
                        dmma884(acc[r], ab[r], bb);
                    }
            }
#pragma unroll
            for (int r = 0; r < DOT_RT; r++)
                if (r < nt)
                    *reinterpret_cast<double2 *>(&sm.red[warp][r * 64 + g * 8 + 2 * c]) = make_double2(acc[r][0], acc[r][1]);
            __syncthreads();
            if ((int)threadIdx.x < nt * 64) {
                const int i = i0 + (int)threadIdx.x / 8, q = q0 + ((int)threadIdx.x & 7);
                if (i < rows && q < nw) {
                    double v = 0.0;
#pragma unroll
                    for (int u = 0; u < DT / 32; u++) v += sm.red[u][threadIdx.x];
                    part[i * nw + q] = v;
                }
            }
            __syncthreads();
        }
    }
}

// One Davidson step by the CTAs of a cluster.  Latency bounds it for SF-CIS
// (n of a few hundred), bandwidth for (R1, R2) vectors, which 16 SMs stream.
// The CTAs meet four times a step: Ritz norms and residuals together, then
// three times for the new vectors.
__global__ void __launch_bounds__(DT) k_dav_step(DavState *st, DavBuffers b, int local) {
    extern __shared__ double dav_smem[];
    DavShared &sm = *reinterpret_cast<DavShared *>(dav_smem);
    double *const S = sm.S, *const X = sm.X, *const vR = sm.vR, *const vI = sm.vI;
    double *V = sm.V;  // eigenvector k in column place[k]; in sm.tot until the new vectors' sums go there
    int *const lw = sm.lw, *const place = sm.place;
    DavState &s = *st;
    const int tid = threadIdx.x;
    const int D = s.D, n = s.dimA, nroot = s.nroot;
    if (s.done) return;
    Team t(n);
    const int lo = t.lo, nc = t.hi - t.lo;
    // the sigma vectors staged by the step before belong to the subspace now
    const int iterations = s.iterations + s.pending;
    int dimIter = s.dimIter + (s.pending ? s.nNew : 0), cur = s.cur, dimFree = s.dimFree;
    const int dim_exceed = s.dim_exceed, ndimIter = s.ndimIter, ndimFree = s.ndimFree;
    const bool over = iterations > s.maxcyc;
    // this CTA's part of the vectors: x_i[k] at x[i ld + k]
    const i64 ld = local ? dav_ld(nc) : n;
    double *const room = dav_smem + (sizeof(DavShared) + 15) / 16 * 2;
    double *Bl = local ? room : b.B[cur] + lo, *ABl = local ? room + D * ld : b.AB[cur] + lo;
    double *const W0 = local ? room + 2 * D * ld : b.w0 + lo, *const W1 = local ? W0 + nroot * ld : b.w1 + lo;
    const double dk0 = tid < nc ? b.diag[lo + tid] : 0.0;  // the first element's diagonal
    if (local && !over)
        for (int e = tid; e < dimIter * nc; e += DT) {
            const int i = e / nc, k = e - i * nc;
            cp_async8(Bl + i * ld + k, b.B[cur] + (size_t)i * n + lo + k);
            cp_async8(ABl + i * ld + k, b.AB[cur] + (size_t)i * n + lo + k);
        }
    int &general = sm.general, &eig_fail = sm.eig_fail, &warn = sm.warn;
    // ---- step 3: eigenpairs of Abar, dgeev in the reference
    // (mod_davidson.f90:185-219).  Abar = B^T A B is symmetric when A is
    // (spin-flip CIS with real integrals); when it is symmetric to 1e-12 of
    // its largest element, the parallel Jacobi on 0.5 (Abar + Abar^T) gives
    // dgeev's eigenpairs (to rounding) fastest; otherwise one warp solves
    // the general problem (warp_geev: real parts of the eigenvalues, real
    // and imaginary parts of complex eigenvectors as dgeev returns them,
    // complex values counted as the reference's imaginary-eigenvalue
    // warning).  Every CTA solves it for itself.
    if (tid == 0) eig_fail = warn = 0;
    if (!over) {
        if (tid < 32) {
            double am = 0.0, ad = 0.0;
            if (tid < dimIter)
                for (int i = 0; i < dimIter; i++) {
                    const double aij = s.Abar[i + tid * D], aji = s.Abar[tid + i * D];
                    am = fmax(am, fabs(aij));
                    ad = fmax(ad, fabs(aij - aji));
                }
            am = warp_allmax(am);
            ad = warp_allmax(ad);
            if (tid == 0) general = ad > 1.0e-12 * am;
        }
        __syncthreads();
        if (!general) {
            jacobi_place(S, dimIter, [&](int i, int j) { return 0.5 * (s.Abar[i + j * D] + s.Abar[j + i * D]); });
            V = block_jacobi(S, V, X, sm.tot, dimIter, vR, place);
        } else {
            for (int e = tid; e < dimIter * dimIter; e += DT) {
                const int i = e / dimIter, j = e % dimIter;
                S[i * GL + j] = s.Abar[i + j * D];
            }
            __syncthreads();
            if (tid < 32) {
                place[tid] = tid;
                const int sw = warp_geev(S, V, X, V, vR, vI, dimIter);
                if (tid == 0) {
                    eig_fail = sw < 0;
                    warn = 0;
                    for (int i = 0; i < dimIter; i++)
                        if (fabs(vI[i]) > 1.0e-10) warn++;
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    t.sync();  // every CTA has read the state
    if (over || eig_fail) {  // cycle limit, or the QR iteration did not converge: stop the solver
        if (t.rank == 0 && tid == 0) {
            s.iterations = iterations;
            s.dimIter = dimIter;
            s.pending = 0;
            if (eig_fail) {
                s.eig_fail = 1;
                s.nonsym_steps++;
                s.warn_imag += warn;
            }
            s.done = 1;
            if (b.mailbox) b.mailbox[0] = 0;
        }
        return;
    }
    // eigenvalues, their order and the chosen roots (vecR(i, k) = V[i][place[k]])
    // sort (mod_davidson.f90:620-640): position = number of smaller values;
    // equal values keep the order that the reference's exchanges leave
    if (tid < 32) {
        int rank = 0;
        bool tie = false;
        if (tid < dimIter) {
            const double x = vR[tid];
            for (int j = 0; j < dimIter; j++) {
                rank += vR[j] < x;
                tie |= j != tid && !(vR[j] < x) && !(x < vR[j]);
            }
        }
        tie = __any_sync(0xffffffffu, tie);
        if (tid < dimIter) lw[tie ? tid : rank] = tid + 1;
        __syncwarp();
        if (tie && tid == 0)
            for (int i = 0; i < dimIter - 1; i++)
                for (int j = i + 1; j < dimIter; j++)
                    if (vR[lw[j] - 1] < vR[lw[i] - 1]) {
                        int t = lw[j];
                        lw[j] = lw[i];
                        lw[i] = t;
                    }
        __syncwarp();
        // root tracking by largest component (mod_davidson.f90:227-251),
        // searched over the positions not yet given to a root: the
        // reference also searches the assigned ones and, when one of them
        // wins, gives one eigenvector to two roots, whose collapse then
        // orthonormalises a repeated vector (division by zero); wherever the
        // reference assigns distinct vectors the choice is the same.  Lane j
        // holds position j; the first position of the largest component wins
        if (!s.lowest)
            for (int iroot = 0; iroot < nroot; iroot++) {
                const int mine = tid < dimIter ? lw[tid] : 0;
                double best = tid >= iroot && tid < dimIter ? fabs(V[iroot * GL + place[mine - 1]]) : 0.0;
                int at = best > 0.0 ? tid : iroot;
                if (!(best > 0.0)) best = 0.0;
                for (int o = 16; o > 0; o >>= 1) {
                    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oa = __shfl_xor_sync(0xffffffffu, at, o);
                    if (ob > best || (ob == best && oa < at)) {
                        best = ob;
                        at = oa;
                    }
                }
                const int idx = __shfl_sync(0xffffffffu, mine, at);
                const int left = __shfl_up_sync(0xffffffffu, mine, 1);
                if (tid > iroot && tid <= at) lw[tid] = left;
                if (tid == iroot) lw[tid] = idx;
                __syncwarp();
            }
    }
    __syncthreads();
    if (tid < nroot) sm.ev[tid] = vR[lw[tid] - 1];
    __syncthreads();
    // ---- collapse when the subspace was full (mod_davidson.f90:266-325)
    if (dim_exceed) {
        const int nd = ndimIter;
        for (int e = tid; e < nd * dimIter; e += DT) {
            const int k = e % dimIter, i = e / dimIter;
            S[i * GL + k] = V[k * GL + place[lw[i] - 1]];
        }
        if (tid < nd) sm.act[tid] = tid;
        __syncthreads();
        block_schmidt_2d(S, dimIter, nd);
        cur = 1 - cur;
        double *const gB = b.B[cur] + lo, *const gAB = b.AB[cur] + lo;
        // in shared memory an element's new values replace the old ones once
        // all of them are formed
        if (local && nd > 8) {
            for (int r0 = 0; r0 < nd; r0 += 8) {
                combine(sm.cf, nc, dimIter, min(8, nd - r0), ABl, Bl, ld,
                        [&](int i, int r) { return S[(r0 + r) * GL + i]; },
                        [&](int r, int k, double x, double y) {
                            gAB[(size_t)(r0 + r) * n + k] = x;
                            gB[(size_t)(r0 + r) * n + k] = y;
                        });
            }
            __syncthreads();
            for (int e = tid; e < nd * nc; e += DT) {
                const int i = e / nc, k = e - i * nc;
                ABl[i * ld + k] = gAB[(size_t)i * n + k];
                Bl[i * ld + k] = gB[(size_t)i * n + k];
            }
        } else {
            combine(sm.cf, nc, dimIter, nd, ABl, Bl, ld, [&](int i, int r) { return S[r * GL + i]; },
                    [&](int r, int k, double x, double y) {
                        gAB[(size_t)r * n + k] = x;
                        gB[(size_t)r * n + k] = y;
                        if (local) {
                            ABl[r * ld + k] = x;
                            Bl[r * ld + k] = y;
                        }
                    });
            if (!local) {
                ABl = gAB;
                Bl = gB;
            }
        }
        __syncthreads();
        dimFree = ndimFree;
        dimIter = nd;
        double *part = t.next(sm.ex[0], DAV_EX);
        team_dots(sm, nc, ABl, ld, nd, Bl, ld, sm.act, nd, false, part);
        t.sync();
        if (t.rank == 0)
            for (int e = tid; e < nd * nd; e += DT) s.Abar[e % nd + (e / nd) * D] = t.sum(part, e);
    }
    // ---- steps 4-6.  The Ritz vector, residual, convergence test and
    // preconditioned vector of a root depend only on the subspace before this
    // step (the new vectors go to positions >= dimIter), so they are formed
    // for all roots at once in per-root slices of w0 / w1.  The norm t of a
    // Ritz vector q and the largest element of A q - w q are found in one
    // pass: where t is off 1 by more than 1e-10, both are divided by it.
    if (dim_exceed) {
        for (int ir = 0; ir < nroot; ir++)
            for (int k = tid; k < nc; k += DT) {
                W0[ir * ld + k] = ABl[ir * ld + k];
                W1[ir * ld + k] = Bl[ir * ld + k];
            }
    } else {
        combine(sm.cf, nc, dimIter, nroot, ABl, Bl, ld, [&](int i, int r) { return V[i * GL + place[lw[r] - 1]]; },
                [&](int r, int k, double x, double y) {
                    W0[r * ld + k] = x;
                    W1[r * ld + k] = y;
                });
    }
    {
        const int w = tid >> 5;
        double *const rq = sm.red[0], *const rb = rq + DT;  // [root][warp]
        for (int r0 = 0; r0 < nroot; r0 += 4) {  // a thread's own elements: no barrier needed
            double q2[4], big[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int ir = min(r0 + u, nroot - 1);
                const double ev = sm.ev[ir];
                q2[u] = 0.0;
                big[u] = -1.0;
                for (int k = tid; k < nc; k += DT) {
                    const double q = W1[ir * ld + k], a = fabs(W0[ir * ld + k] - ev * q);
                    q2[u] = fma(q, q, q2[u]);
                    if (a > big[u]) big[u] = a;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                q2[u] = warp_allsum(q2[u]);
                big[u] = warp_allmax(big[u]);
            }
            if ((tid & 31) == 0)
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (r0 + u < nroot) {
                        rq[(r0 + u) * (DT / 32) + w] = q2[u];
                        rb[(r0 + u) * (DT / 32) + w] = big[u];
                    }
        }
        __syncthreads();
        double *part = t.next(sm.ex[0], DAV_EX);
        if (tid < nroot) {
            double q2 = 0.0, big = -1.0;
            for (int i = 0; i < DT / 32; i++) {
                q2 += rq[tid * (DT / 32) + i];
                big = fmax(big, rb[tid * (DT / 32) + i]);
            }
            part[tid] = q2;
            part[DAV_MAXD + tid] = big;
        }
        t.sync();
        if (tid < nroot) {
            const double nrm = sqrt(t.sum(part, tid)), big = t.amax(part, DAV_MAXD + tid);
            const double f = fabs(nrm - 1.0) > 1.0e-10 ? 1.0 / nrm : 1.0;
            sm.rnorm[tid] = f;
            sm.cvd[tid] = (big >= 0.0 ? big * f : 0.0) < s.maxError ? 1 : 0;
        }
        __syncthreads();
    }
    int nconv = 0, na = 0;  // na: roots that get a new vector
    for (int ir = 0; ir < nroot; ir++) nconv += sm.cvd[ir];
    if (dimFree > 0)
        for (int ir = 0; ir < nroot; ir++) {
            if (sm.cvd[ir]) continue;
            if (tid == 0) sm.act[na] = ir;
            na++;
        }
    for (int k = tid; k < nc; k += DT) {
        const double dk = k == tid ? dk0 : b.diag[lo + k];
#pragma unroll 4
        for (int ir = 0; ir < nroot; ir++) {
            const double f = sm.rnorm[ir], ev = sm.ev[ir];
            const double q = W1[ir * ld + k] * f, r = W0[ir * ld + k] * f - ev * q;
            b.fileEV[(size_t)ir * (n + 1) + 1 + lo + k] = q;
            double d = ev - dk;
            if (fabs(d) < 1.0e-4) d = (d < 0.0) ? -1.0e-4 : 1.0e-4;
            if (!sm.cvd[ir]) W1[ir * ld + k] = r / d;
        }
    }
    __syncthreads();
    // SchmidtS (mod_davidson.f90:682-727) of all new vectors together: twice
    // projected on the basis (overlaps of a pass computed at once, as
    // classical Gram-Schmidt applied twice), then made orthonormal among
    // themselves in root order by the Cholesky factor of their Gram matrix,
    // a vector that keeps less than 1e-6 of its length being dropped; one
    // more pass of both takes out what the divisions by those lengths
    // amplified.  Same vectors as the reference's one-by-one projections, to
    // rounding, with three exchanges instead of five for every root.
    int nNew = 0;
    for (int pass = 0; pass < 3 && na > 0; pass++) {
        // pass 0: overlaps and lengths; 1, 2: overlaps and Gram matrix
        double *part = t.next(sm.ex[0], DAV_EX);
        team_dots(sm, nc, Bl, ld, dimIter, W1, ld, sm.act, na, true, part);
        t.sync();
        const int no = dimIter * na;
        for (int e = tid; e < no + na * na; e += DT) sm.tot[e] = t.sum(part, e);
        __syncthreads();
        if (pass > 0) {  // Gram matrix less the projections
            for (int e = tid; e < na * na; e += DT) {
                const int q = e / na, p = e - q * na;
                double g = sm.tot[no + e];
#pragma unroll 4
                for (int i = 0; i < dimIter; i++) g -= sm.tot[i * na + q] * sm.tot[i * na + p];
                sm.L[q * GL + p] = g;
            }
            __syncthreads();
        }
        if (tid < 32) {
            double *const L = sm.L;  // L(q, p) at [q * GL + p]
            if (pass == 0) {
                // reciprocal lengths only: the vectors are scaled to unit length
                for (int e = tid; e < na * na; e += 32) L[(e / na) * GL + e % na] = 0.0;
                __syncwarp();
                if (tid < na) L[tid * GL + tid] = 1.0 / sqrt(sm.tot[no + tid * na + tid]);
                if (tid == 0) sm.nnew = na;
            } else {
                // Cholesky factor column by column (lane = row); the
                // reciprocal diagonal is kept, zero for a dropped vector
                int kept = 0;
                for (int p = 0; p < na; p++) {
                    const double g = L[p * GL + p], nrm = sqrt(fmax(g, 0.0));
                    const bool keep = !(nrm < (pass == 1 ? 1.0e-6 : 0.0)) && (pass == 2 || kept < dimFree);
                    const double ri = keep ? 1.0 / nrm : 0.0;
                    __syncwarp();
                    if (tid == p) L[p * GL + p] = ri;
                    double lqp = 0.0;
                    if (tid > p && tid < na) {
                        lqp = L[tid * GL + p] * ri;
                        L[tid * GL + p] = lqp;
                    }
                    __syncwarp();
                    if (tid > p && tid < na)
                        for (int q = p + 1; q <= tid; q++) L[tid * GL + q] -= lqp * L[q * GL + p];
                    __syncwarp();
                    kept += keep;
                }
                if (tid == 0) sm.nnew = kept;
            }
        }
        __syncthreads();
        // w_q <- (w_q - sum_i o_iq b_i - sum_{p<q} L(q, p) w_p) / L(q, q)
        const double *const L = sm.L;
        for (int q0 = 0; q0 < na; q0 += 8) {
            put_coefs(sm.cf, dimIter, q0, na, [&](int i, int q) { return sm.tot[i * na + q]; });
            for (int k = tid; k < nc; k += DT) {
                double x[8];
#pragma unroll
                for (int q = 0; q < 8; q++) x[q] = q0 + q < na ? W1[sm.act[q0 + q] * ld + k] : 0.0;
#pragma unroll 4
                for (int i = 0; i < dimIter; i++) {
                    const double v = Bl[i * ld + k];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const double2 f = sm.cf[i][q];
                        x[2 * q] -= f.x * v;
                        x[2 * q + 1] -= f.y * v;
                    }
                }
                if (pass > 0)
                    for (int p = 0; p < q0; p++) {
                        const double y = W1[sm.act[p] * ld + k];
#pragma unroll
                        for (int q = 0; q < 8; q++)
                            if (q0 + q < na) x[q] -= L[(q0 + q) * GL + p] * y;
                    }
#pragma unroll
                for (int q = 0; q < 8; q++)
                    if (q0 + q < na) {
                        if (pass > 0)
#pragma unroll
                            for (int p = 0; p < 8; p++)
                                if (p < q) x[q] -= L[(q0 + q) * GL + q0 + p] * x[p];
                        x[q] *= L[(q0 + q) * GL + q0 + q];
                        W1[sm.act[q0 + q] * ld + k] = x[q];
                    }
            }
        }
        __syncthreads();
        if (pass == 1) {  // leave the dropped vectors out
            nNew = sm.nnew;
            if (nNew < na) {
                if (tid == 0) {
                    int m = 0;
                    for (int q = 0; q < na; q++)
                        if (L[q * GL + q] != 0.0) sm.act[m++] = sm.act[q];
                }
                na = nNew;
                __syncthreads();
            }
        }
    }
    // the new basis vectors, and their staged copies (zero beyond nNew) for a
    // sigma launch whose size does not depend on nNew
    for (int q = 0; q < nroot; q++)
        for (int k = tid; k < nc; k += DT) {
            const double x = q < nNew ? W1[sm.act[q] * ld + k] : 0.0;
            if (q < nNew) b.B[cur][(size_t)(dimIter + q) * n + lo + k] = x;
            b.W[(size_t)q * n + lo + k] = x;
        }
    if (t.rank == 0) {
        if (tid < dimIter) {
            s.valR[tid] = vR[tid];
            s.lowestE[tid] = lw[tid];
        }
        if (tid < nroot) {
            s.eigenVal[tid] = sm.ev[tid];
            s.conv[tid] = sm.cvd[tid];
            b.fileEV[(size_t)tid * (n + 1)] = sm.ev[tid];
        }
        if (tid == 0) {
            dimFree -= nNew;
            s.iterations = iterations;
            s.cur = cur;
            s.dimIter = dimIter;
            s.dimFree = dimFree;
            s.newpos = dimIter;
            s.nNew = nNew;
            s.nonsym_steps += general;
            s.warn_imag += warn;
            s.pending = 1;
            if (nconv == nroot) {
                s.done = 1;
                s.converged = 1;
                s.pending = 0;
            } else {
                s.dim_exceed = 0;
                if (dimFree == 0) {
                    s.dim_exceed = 1;
                    s.ndimIter = D - s.dimDel;
                    if (s.ndimIter < nroot) {
                        s.ndimIter = nroot;
                        s.ndimFree = D - s.ndimIter;
                    } else {
                        s.ndimFree = s.dimDel;
                    }
                }
            }
            if (b.mailbox) b.mailbox[0] = s.done ? 0 : 1;
        }
    }
    t.leave();
}

// Ritz-matrix update with the new vectors (mod_davidson.f90:460-496): the
// staged sigma vectors AW[0..nNew) are put in place in AB and their products
// with the basis formed, one CTA for the new vector blockIdx.x / ngroup and a
// group of ABAR_G basis vectors: Abar(i, j) = b_i . Ab_j of the new column
// j, and of the new row i for the older j (which hold no staged vector).
// dimIter is that before the step's vectors; the next step counts them in.
constexpr int ABAR_T = 256, ABAR_G = 4;
__global__ void __launch_bounds__(ABAR_T) k_dav_abar(DavState *st, DavBuffers b, int ngroup) {
    __shared__ double red[2 * ABAR_G][ABAR_T / 32];
    const DavState &s = *st;
    if (s.done) return;
    const int n = s.dimA, D = s.D, dimIter = s.dimIter, nNew = s.nNew, cur = s.cur;
    const int q = blockIdx.x / ngroup, g = blockIdx.x % ngroup;
    const int i0 = g * ABAR_G, tot = dimIter + nNew;
    if (q >= nNew || i0 >= tot) return;
    const double *B = b.B[cur];
    double *AB = b.AB[cur];
    const double *aw = b.AW + (size_t)q * n, *bq = B + (size_t)(dimIter + q) * n;
    double *ab = AB + (size_t)(dimIter + q) * n;
    double col[ABAR_G], row[ABAR_G];
#pragma unroll
    for (int u = 0; u < ABAR_G; u++) col[u] = row[u] = 0.0;
#pragma unroll 2
    for (int k = threadIdx.x; k < n; k += ABAR_T) {
        const double a = aw[k], x = bq[k];
        if (g == 0) ab[k] = a;
#pragma unroll
        for (int u = 0; u < ABAR_G; u++) {
            const int i = i0 + u;
            if (i < tot) col[u] = fma(B[(size_t)i * n + k], a, col[u]);
            if (i < dimIter) row[u] = fma(x, AB[(size_t)i * n + k], row[u]);
        }
    }
    const int w = threadIdx.x >> 5;
#pragma unroll
    for (int u = 0; u < ABAR_G; u++) {
        col[u] = warp_allsum(col[u]);
        row[u] = warp_allsum(row[u]);
        if ((threadIdx.x & 31) == 0) {
            red[u][w] = col[u];
            red[ABAR_G + u][w] = row[u];
        }
    }
    __syncthreads();
    if (threadIdx.x < 2 * ABAR_G) {
        double v = 0.0;
        for (int i = 0; i < ABAR_T / 32; i++) v += red[threadIdx.x][i];
        const int i = i0 + (int)threadIdx.x % ABAR_G;
        if (threadIdx.x < ABAR_G) {
            if (i < tot) st->Abar[i + (dimIter + q) * D] = v;
        } else if (i < dimIter) {
            st->Abar[(dimIter + q) + i * D] = v;
        }
    }
}

// eigen test of the final roots (mod_davidson.f90:525-542): AR in w-buffer
__global__ void __launch_bounds__(DT) k_dav_final(DavState *st, DavBuffers b, const double *AR) {
    __shared__ double sh[DT / 32 + 1];
    __shared__ int shi[DT / 32 + 1];
    DavState &s = *st;
    const int n = s.dimA;
    double worst = 0.0;
    for (int ir = 0; ir < s.nroot; ir++) {
        const double *R = b.fileEV + (size_t)ir * (n + 1);
        double w = R[0];
        for (int k = threadIdx.x; k < n; k += DT) b.w0[k] = AR[(size_t)ir * n + k] - w * R[1 + k];
        __syncthreads();
        double e = fabs(block_amax(b.w0, n, sh, shi));
        if (e > worst) worst = e;
    }
    if (threadIdx.x == 0) s.max_resid = worst;
}

// ------------------------------------------------------------------- DIIS
// LINPACK dgefa / dgesl (as MINV, src/libsrint/minv.f, calls them) by one
// warp on a matrix in shared memory (n <= 32): lane i owns row i.  Pivot =
// first row of largest magnitude, NaN counting as the largest (compared as it
// is, it would leave the lanes with different rows and some with none); every
// element sees the same operations in the same order as the sequential LINPACK
// loops.
__device__ void warp_dgefa(double *a, int lda, int n, int *ipvt) {
    const int i = threadIdx.x & 31;
    for (int k = 0; k < n - 1; k++) {
        double m = (i >= k && i < n) ? fabs(a[i + k * lda]) : -1.0;
        if (!(m >= -1.0)) m = HUGE_VAL;
        int l = (i >= k && i < n) ? i : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1) {
            double om = __shfl_xor_sync(0xffffffffu, m, o);
            int ol = __shfl_xor_sync(0xffffffffu, l, o);
            if (om > m || (om == m && ol < l)) {
                m = om;
                l = ol;
            }
        }
        if (i == 0) ipvt[k] = l;
        __syncwarp();
        if (a[l + k * lda] == 0.0) continue;
        if (l != k && i >= k && i < n) {  // swap rows l and k in columns >= k (lane i: column i)
            double t = a[l + i * lda];
            a[l + i * lda] = a[k + i * lda];
            a[k + i * lda] = t;
        }
        __syncwarp();
        const double t = -1.0 / a[k + k * lda];
        if (i > k && i < n) {
            double aik = a[i + k * lda] * t;
            a[i + k * lda] = aik;
            for (int j = k + 1; j < n; j++) a[i + j * lda] += a[k + j * lda] * aik;
        }
        __syncwarp();
    }
    if (i == 0) ipvt[n - 1] = n - 1;
    __syncwarp();
}
__device__ void warp_dgesl(const double *a, int lda, int n, const int *ipvt, double *bv) {
    const int i = threadIdx.x & 31;
    for (int k = 0; k < n - 1; k++) {
        const int l = ipvt[k];
        const double t = bv[l];
        __syncwarp();
        if (i == 0 && l != k) {
            bv[l] = bv[k];
            bv[k] = t;
        }
        __syncwarp();
        if (i > k && i < n) bv[i] += t * a[i + k * lda];
        __syncwarp();
    }
    for (int kb = 0; kb < n; kb++) {
        const int k = n - 1 - kb;
        if (i == 0) bv[k] /= a[k + k * lda];
        __syncwarp();
        const double t = -bv[k];
        if (i < k) bv[i] += t * a[i + k * lda];
        __syncwarp();
    }
}

// block sums of v[0..M) (and block maxima with MAX) of every thread, entry j
// to out[j]; every thread calls it, the caller's barrier publishes out
template <int M, bool MAX = false>
__device__ void block_reduce(const double (&v)[M], double (*red)[DT / 32], double *out) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double x[M];
#pragma unroll
    for (int j = 0; j < M; j++) x[j] = MAX ? warp_allmax(v[j]) : warp_allsum(v[j]);
    if (lane == 0)
#pragma unroll
        for (int j = 0; j < M; j++) red[j][w] = x[j];
    __syncthreads();
    if (threadIdx.x < M) {
        double t = MAX ? -1.0 : 0.0;
        for (int i = 0; i < DT / 32; i++) t = MAX ? fmax(t, red[threadIdx.x][i]) : t + red[threadIdx.x][i];
        out[threadIdx.x] = t;
    }
    __syncthreads();
}

// One step of the device-driven solver (see solvers.cuh) for the root of this
// cluster.  Short R1 vectors are latency-bound (one CTA; up to three
// exchanges a step), the (R1, R2) vectors of the grCPS(D) programs
// bandwidth-bound: 2 x diis_dim stored vectors are read a step, by 16 SMs
// (26 k elements: 230 us a step on one SM, 33 on 16).
//   1. R1 = pr / den and the sums of orthogonalR2L (R -= (<L|R> / ||L||) L:
//      the reference divides by the norm, not its square) or <R1|nrmv>;
//   2. that correction, the DIIS error vector and its overlaps;
//   3. the bordered system (every CTA for itself), the extrapolated vector,
//      its residual and the sums of the second correction;
//   4. the second correction.
__global__ void __launch_bounds__(DT) k_solver_step(SolverArgs a) {
    __shared__ double red[DIIS_MAXDIM][DT / 32], ex[2][DIIS_MAXDIM], tot[DIIS_MAXDIM];
    __shared__ double Bm[DIIS_MAXDIM * DIIS_MAXDIM], row[DIIS_MAXDIM];
    __shared__ double coef[DIIS_MAXDIM + 1];
    __shared__ double aug[(DIIS_MAXDIM + 1) * (DIIS_MAXDIM + 1)], rhs[DIIS_MAXDIM + 1];
    __shared__ int ipvt[DIIS_MAXDIM + 1];
    const int len = a.len, tid = threadIdx.x;
    Team t(len);
    const int r = blockIdx.x / t.size;
    SolverState &ss = a.ss[r];
    DiisState &ds = a.ds[r];
    const bool active = ss.active;
    const int iter = ss.iter + 1, maxdim = ds.maxdim, id = ds.idimr - 1, nd = ds.ndimr;
    for (int e = tid; e < DIIS_MAXDIM * DIIS_MAXDIM; e += DT) Bm[e] = ds.Bm[e];
    t.sync();  // every CTA has read the state
    if (!active) return;
    const size_t o = (size_t)r * len;
    double *pr = a.pr + o, *R1 = a.R1 + o;
    const double *cc = a.cc + o, *S = a.S + o;
    const double *L = a.L ? a.L + o : nullptr, *NV = a.nrmv ? a.nrmv + o : nullptr;
    double *prev = a.db.prev + (size_t)r * a.sprev, *err = a.db.err + (size_t)r * a.serr;
    double *amp = a.db.amp + (size_t)r * a.serr;
    const double *U = L ? L : NV;  // the vector of the two corrections
    double ll = 0.0;               // ||L||
    // ---- 1
    double s2[2] = {0.0, 0.0};
    const double mw0 = a.w0 ? -a.w0[r] : 0.0;
    for (int k = t.lo + tid; k < t.hi; k += DT) {
        double x;
        if (iter > 1) {  // pr = cc; pr += (-w0) R1; pr += sigma  (the reference's updates, in order)
            x = (a.w0 ? fma(mw0, R1[k], cc[k]) : cc[k]) + S[k];
            pr[k] = x;
        } else {
            x = pr[k];
        }
        double v = (iter > 1 || !a.keep_first) ? x / a.den[k] : R1[k];
        R1[k] = v;
        if (U) {
            const double u = U[k];
            s2[0] = fma(u, u, s2[0]);
            s2[1] = fma(u, v, s2[1]);
        }
    }
    double f = 0.0, g = 1.0;  // the correction R1 = g (R1 + f U)
    if (U) {
        double *part = t.next(ex[0], DIIS_MAXDIM);
        block_reduce(s2, red, part);
        t.sync();
        const double uu = t.sum(part, 0), ur = t.sum(part, 1);
        if (L) {
            ll = sqrt(uu);
            f = -ur / ll;
        } else {
            g = 1.0 / ur;
        }
    }
    // ---- 2
    if (iter == 1) {
        double s1[2] = {0.0, 0.0};
        for (int k = t.lo + tid; k < t.hi; k += DT) {
            double v = R1[k];
            if (L) v += f * L[k];
            v *= g;
            R1[k] = v;
            prev[k] = v;
            if (U) s1[1] = fma(U[k], v, s1[1]);
        }
        if (U) {
            double *part = t.next(ex[0], DIIS_MAXDIM);
            block_reduce(s1, red, part);
            t.sync();
            const double ur = t.sum(part, 1);
            if (L) f = -ur / ll;
            else g = 1.0 / ur;
        }
    } else {
        double dt[DIIS_MAXDIM];
#pragma unroll
        for (int j = 0; j < DIIS_MAXDIM; j++) dt[j] = 0.0;
        for (int k = t.lo + tid; k < t.hi; k += DT) {
            double v = R1[k];
            if (L) v += f * L[k];
            v *= g;
            const double p = prev[k], e = v - p;
            amp[(size_t)id * len + k] = p;
            err[(size_t)id * len + k] = e;
#pragma unroll
            for (int j = 0; j < DIIS_MAXDIM; j++)
                if (j < nd) dt[j] = fma(e, j == id ? e : err[(size_t)j * len + k], dt[j]);
        }
        double *part = t.next(ex[0], DIIS_MAXDIM);
        block_reduce(dt, red, part);
        t.sync();
        // only the row of the error vector stored now changes; the others
        // are kept in the state from earlier steps
        if (tid < nd) {
            const double x = t.sum(part, tid);
            row[tid] = x;
            Bm[id + tid * DIIS_MAXDIM] = x;
            Bm[tid + id * DIIS_MAXDIM] = x;
        }
        __syncthreads();
        // ---- 3
        if (tid < 32) {  // dodiis (src/libsrint/dodiis.f): bordered system with -1e-4
            const int n1 = nd + 1;
            for (int e = tid; e < n1 * n1; e += 32) {
                const int i = e % n1, j = e / n1;
                aug[e] = (i == 0 && j == 0) ? 0.0
                         : (i == 0 || j == 0) ? -1.0e-4
                                              : Bm[(i - 1) + (j - 1) * DIIS_MAXDIM];
            }
            if (tid < n1) rhs[tid] = (tid == 0) ? -1.0e-4 : 0.0;
            __syncwarp();
            warp_dgefa(aug, n1, n1, ipvt);
            warp_dgesl(aug, n1, n1, ipvt, rhs);
            if (tid < nd) coef[tid] = rhs[tid + 1];
        }
        __syncthreads();
        double s1[1] = {0.0}, big[1] = {-1.0};
        for (int k = t.lo + tid; k < t.hi; k += DT) {
            double v = 0.0, p = 0.0;
#pragma unroll 4
            for (int i = 0; i < nd; i++) {
                v += coef[i] * err[(size_t)i * len + k];
                p += coef[i] * amp[(size_t)i * len + k];
            }
            if (fabs(v) > big[0]) big[0] = fabs(v);
            v += p;
            prev[k] = v;
            R1[k] = v;
            if (U) s1[0] = fma(U[k], v, s1[0]);
        }
        part = t.next(ex[0], DIIS_MAXDIM);
        block_reduce<1, true>(big, red, part);
        block_reduce(s1, red, part + 1);
        t.sync();
        const double res = fmax(t.amax(part, 0), 0.0), ur = t.sum(part, 1);
        if (tid == 0) tot[0] = res;
        f = 0.0;
        g = 1.0;
        if (L) f = -ur / ll;
        else if (NV) g = 1.0 / ur;
    }
    // ---- 4
    if (U)
        for (int k = t.lo + tid; k < t.hi; k += DT) {
            double v = R1[k];
            if (L) v += f * L[k];
            R1[k] = v * g;
        }
    if (t.rank == 0) {
        if (iter > 1 && tid < nd) {
            ds.Bm[id + tid * DIIS_MAXDIM] = row[tid];
            ds.Bm[tid + id * DIIS_MAXDIM] = row[tid];
        }
        if (tid == 0) {
            const double res = iter > 1 ? tot[0] : 1.0;
            ds.res = res;
            ds.ndimr = iter > 1 ? ((nd + 1 < maxdim) ? nd + 1 : maxdim) : 1;
            ds.idimr = iter > 1 ? (id + 2 > maxdim ? 1 : id + 2) : 1;
            ss.iter = iter;
            ss.res = res;
            const int go = !((iter > 1 && fabs(res) < a.tol) || iter > a.cyc);
            ss.active = go;
            a.mailbox[r] = go;
        }
    }
    t.leave();
}

// the general eigen-solve of the Davidson step on one given matrix
// (row-major, n <= DAV_MAXD), for verification against LAPACK
__global__ void __launch_bounds__(32) k_geev_probe(const double *A, int n, double *wr, double *wi, double *V,
                                                    int *sweeps) {
    __shared__ double H[DAV_MAXD * GL], Z[DAV_MAXD * GL], X[DAV_MAXD * GL], r[DAV_MAXD], im[DAV_MAXD];
    for (int e = threadIdx.x; e < n * n; e += 32) H[(e / n) * GL + e % n] = A[e];
    __syncwarp();
    const int sw = warp_geev(H, Z, X, Z, r, im, n);
    if (threadIdx.x < n) {
        wr[threadIdx.x] = r[threadIdx.x];
        wi[threadIdx.x] = im[threadIdx.x];
    }
    for (int e = threadIdx.x; e < n * n; e += 32) V[e] = Z[(e / n) * GL + e % n];
    if (threadIdx.x == 0) *sweeps = sw;
}

// the symmetric eigen-solve of the Davidson step on one given matrix
__global__ void __launch_bounds__(DT) k_syev_probe(const double *A, int n, double *wr, double *V) {
    __shared__ double S[DAV_MAXD * GL], S2[DAV_MAXD * GL], U[DAV_MAXD * GL], U2[DAV_MAXD * GL], w[DAV_MAXD];
    __shared__ int place[DAV_MAXD];
    jacobi_place(S, n, [&](int i, int j) { return A[i * n + j]; });
    const double *const E = block_jacobi(S, U, S2, U2, n, w, place);
    if ((int)threadIdx.x < n) wr[threadIdx.x] = w[threadIdx.x];
    for (int e = threadIdx.x; e < n * n; e += DT) V[e] = E[(e / n) * GL + place[e % n]];
}

}  // namespace

int syev_probe(const double *A_dev, int n, double *w, double *V) {
    if (n < 1 || n > DAV_MAXD) return set_error(CPSD_EARG, "syev: n must be 1..32");
    k_syev_probe<<<1, DT, 0, stream()>>>(A_dev, n, w, V);
    count_launch();
    return cuda_check(cudaGetLastError(), "k_syev_probe");
}

int geev_probe(const double *A_dev, int n, double *wr, double *wi, double *V, int *sweeps) {
    if (n < 1 || n > DAV_MAXD) return set_error(CPSD_EARG, "geev: n must be 1..32");
    k_geev_probe<<<1, 32, 0, stream()>>>(A_dev, n, wr, wi, V, sweeps);
    count_launch();
    return cuda_check(cudaGetLastError(), "k_geev_probe");
}

int dav_init_launch(DavState *st, const DavBuffers &b) {
    k_dav_init<<<1, DT, 0, stream()>>>(st, b);
    count_launch();
    return cuda_check(cudaGetLastError(), "k_dav_init");
}
int dav_step_launch(DavState *st, const DavBuffers &b, i64 n, int nroot, int D) {
    constexpr size_t base = (sizeof(DavShared) + 15) / 16 * 16, most = base + sizeof(double) * DAV_LOCAL;
    static_assert(most + 1024 <= 227 * 1024, "shared memory of a Davidson step");
    static std::atomic<int> fits[TEAM_MAXDEV];
    int ctas;
    CPSD_TRY(team_most(k_dav_step, most, fits, &ctas));
    cudaEvent_t end;
    CPSD_TRY(timing_begin(0.0, 0, 0, 0, 30, &end));
    const int size = team_size(n, DAV_PER, ctas);
    const int nc = (int)(((n + size - 1) / size + 31) & ~(i64)31);
    const i64 need = (i64)2 * (D + nroot) * dav_ld(nc);
    const int local = need <= DAV_LOCAL;
    CPSD_TRY(launch_team(k_dav_step, 1, size, base + (local ? sizeof(double) * (size_t)need : 0), "k_dav_step", st, b,
                         local));
    count_launch();
    return timing_end(end);
}
int dav_abar_launch(DavState *st, const DavBuffers &b, int nroot, int D) {
    cudaEvent_t end;
    CPSD_TRY(timing_begin(0.0, 0, 0, 0, 31, &end));
    const int ngroup = (D + ABAR_G - 1) / ABAR_G;
    k_dav_abar<<<nroot * ngroup, ABAR_T, 0, stream()>>>(st, b, ngroup);
    count_launch();
    CPSD_TRY(cuda_check(cudaGetLastError(), "k_dav_abar"));
    return timing_end(end);
}
int dav_final_launch(DavState *st, const DavBuffers &b) {
    // AR of the final roots was written to b.AB[0] by the caller
    k_dav_final<<<1, DT, 0, stream()>>>(st, b, b.AB[0]);
    count_launch();
    return cuda_check(cudaGetLastError(), "k_dav_final");
}
int solver_step_launch(const SolverArgs &a) {
    if (a.nb <= 0) return CPSD_OK;
    static std::atomic<int> fits[TEAM_MAXDEV];
    int ctas;
    CPSD_TRY(team_most(k_solver_step, 0, fits, &ctas));
    cudaEvent_t end;
    CPSD_TRY(timing_begin(0.0, a.nb, 0, 0, 32, &end));
    CPSD_TRY(launch_team(k_solver_step, a.nb, team_size(a.len, DT, ctas), 0, "k_solver_step", a));
    count_launch();
    return timing_end(end);
}

}  // namespace cpsd
