// Symmetric eigen-decomposition of the FO overlap on the GPU: the role of
// DIAGGE_FO / EWEVGE_FO (diagon_sic.f:45-232, Householder tridiagonalisation
// and implicit QL) in LOWSIC (lowden_files.f:2-172), done here by the cyclic
// Jacobi method with the round-robin (tournament) ordering, which rotates
// n/2 disjoint index pairs at once.  One CTA holds the matrix (N_o is at most a few
// hundred), in shared memory when it fits; the rotations reach the eigenvectors in
// a kernel of their own, or beyond that size in the same CTA.
//
// Each round: every pair (p, q) gets the rotation that zeroes A(p,q) (the
// symmetric Schur decomposition with t = sign(tau)/(|tau| + sqrt(1 + tau^2))),
// then all row updates A <- J^T A, then all column updates A <- A J and
// V <- V J.  An off-diagonal entry below eps/2 sqrt|A(p,p) A(q,q)| is not
// rotated; a sweep (m - 1 rounds, m = n rounded up to even) without any
// rotation ends the iteration.  Eigenvalues are returned in ascending order,
// as EWEVGE_FO returns them with IORD = -1 (diagon_sic.f:64), with their
// eigenvectors in the same order.  Everything is FP64.
#include <cfloat>

#include "kernels.cuh"

namespace flosic {

constexpr int EIG_THREADS = 1024;
constexpr int EIG_MAX_N = 1024;          // pairs held in shared memory: EIG_MAX_N / 2
constexpr int EIG_SMEM_MAX_N = 160;      // matrix in shared memory up to 160 x 161 doubles (206 KB)
constexpr int EIG_MAX_SWEEPS = 60;

// More than EIG_SMEM_MAX_N FOs.  A(i, j) at A[i * (n + 1) + j].  The rotations are
// accumulated transposed, Vt(m, k) = component k of vector m, so that a column
// update of V is a row update of Vt (contiguous in memory).
__global__ void __launch_bounds__(EIG_THREADS, 1)
k_sym_eigen(int n, const double* __restrict__ ain, double* __restrict__ aglob, double* __restrict__ vt,
            double* __restrict__ wout, double* __restrict__ vout, int* __restrict__ info) {
  __shared__ double rc[EIG_MAX_N / 2], rs[EIG_MAX_N / 2];
  __shared__ int rp[EIG_MAX_N / 2], rq[EIG_MAX_N / 2];
  __shared__ int nrot;
  double* A = aglob;
  const int ld = n + 1;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    A[i * ld + j] = ain[e];
    vt[e] = (i == j) ? 1.0 : 0.0;
  }
  __syncthreads();
  const int m = n + (n & 1), half = m / 2;
  bool converged = (n <= 1);
  for (int sweep = 0; sweep < EIG_MAX_SWEEPS && !converged; ++sweep) {
    if (tid == 0) nrot = 0;
    __syncthreads();
    for (int r = 0; r < m - 1; ++r) {
      for (int k = tid; k < half; k += nt) {
        const int a = (k == 0) ? 0 : ((k - 1 + r) % (m - 1)) + 1;
        const int b = ((m - 2 - k + r) % (m - 1)) + 1;
        const int p = min(a, b), q = max(a, b);
        double c = 1.0, s = 0.0;
        if (q < n) {
          const double apq = A[p * ld + q];
          const double app = A[p * ld + p], aqq = A[q * ld + q];
          if (apq != 0.0 && fabs(apq) > 0.5 * DBL_EPSILON * sqrt(fabs(app * aqq))) {
            const double tau = (aqq - app) / (2.0 * apq);
            const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
            c = 1.0 / sqrt(1.0 + t * t);
            s = t * c;
            atomicAdd(&nrot, 1);
          }
        }
        rp[k] = p;
        rq[k] = q;
        rc[k] = c;
        rs[k] = s;
      }
      __syncthreads();
      // rows p, q of A (A <- J^T A) and of Vt (V <- V J)
      for (int e = tid; e < half * n; e += nt) {
        const int k = e / n, j = e - k * n;
        const double s = rs[k];
        if (s == 0.0) continue;
        const double c = rc[k];
        const int p = rp[k], q = rq[k];
        double x = A[p * ld + j], y = A[q * ld + j];
        A[p * ld + j] = c * x - s * y;
        A[q * ld + j] = s * x + c * y;
        x = vt[p * n + j];
        y = vt[q * n + j];
        vt[p * n + j] = c * x - s * y;
        vt[q * n + j] = s * x + c * y;
      }
      __syncthreads();
      // columns p, q of A (A <- A J); lanes run over rows i
      for (int e = tid; e < half * n; e += nt) {
        const int k = e / n, i = e - k * n;
        const double s = rs[k];
        if (s == 0.0) continue;
        const double c = rc[k];
        const int p = rp[k], q = rq[k];
        const double x = A[i * ld + p], y = A[i * ld + q];
        A[i * ld + p] = c * x - s * y;
        A[i * ld + q] = s * x + c * y;
      }
      __syncthreads();
    }
    converged = (nrot == 0);
    __syncthreads();  // every thread has read nrot before it is reset
  }
  // ascending order (ties by index): rank of each eigenvalue, then scatter
  for (int i = tid; i < n; i += nt) {
    const double d = A[i * ld + i];
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double dj = A[j * ld + j];
      rank += (dj < d || (dj == d && j < i)) ? 1 : 0;
    }
    wout[rank] = d;
    for (int k = 0; k < n; ++k) vout[(size_t)k * n + rank] = vt[(size_t)i * n + k];
  }
  if (tid == 0) *info = converged ? 0 : 1;
}

// Up to EIG_SMEM_MAX_N the work is split in two.  k_sym_eigen_rot rotates A alone:
// a thread takes 2 x 2 blocks (rows of pair i, columns of pair j) through the row
// and then the column rotation, the same operations on the same operands as the
// two passes above with one barrier fewer, and records (c, s).  The eigenvectors
// do not feed back, so k_sym_eigen_vec applies the recorded rotations to each
// component (a column of Vt) in a warp of its own, all components at once.
// Bound by latency (a barrier pair and one division chain per round).  N_o = 128:
// 7.9 -> 4.3 ms (the one-CTA form also updated Vt in L2 in every round).
__device__ __forceinline__ void eig_pair(int k, int r, int m, int& p, int& q) {
  const int a = (k == 0) ? 0 : ((k - 1 + r) % (m - 1)) + 1;
  const int b = ((m - 2 - k + r) % (m - 1)) + 1;
  p = min(a, b);
  q = max(a, b);
}

__global__ void __launch_bounds__(EIG_THREADS, 1)
k_sym_eigen_rot(int n, const double* __restrict__ ain, double2* __restrict__ rot, double* __restrict__ wout,
                int* __restrict__ meta) {
  extern __shared__ __align__(16) double eig_sm[];
  __shared__ double rc[EIG_SMEM_MAX_N / 2], rs[EIG_SMEM_MAX_N / 2];
  __shared__ int rp[EIG_SMEM_MAX_N / 2], rq[EIG_SMEM_MAX_N / 2];
  __shared__ int nrot;
  double* A = eig_sm;
  const int ld = n + 1, tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < n * n; e += nt) A[(e / n) * ld + e % n] = ain[e];
  __syncthreads();
  const int m = n + (n & 1), half = m / 2, jw = (half + 31) / 32;
  bool converged = (n <= 1);
  int rounds = 0;
  for (int sweep = 0; sweep < EIG_MAX_SWEEPS && !converged; ++sweep) {
    if (tid == 0) nrot = 0;
    __syncthreads();
    for (int r = 0; r < m - 1; ++r, ++rounds) {
      for (int k = tid; k < half; k += nt) {
        int p, q;
        eig_pair(k, r, m, p, q);
        double c = 1.0, s = 0.0;
        if (q < n) {
          const double apq = A[p * ld + q];
          const double app = A[p * ld + p], aqq = A[q * ld + q];
          if (apq != 0.0 && fabs(apq) > 0.5 * DBL_EPSILON * sqrt(fabs(app * aqq))) {
            const double tau = (aqq - app) / (2.0 * apq);
            const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
            c = 1.0 / sqrt(1.0 + t * t);
            s = t * c;
            atomicAdd(&nrot, 1);
          }
        }
        rp[k] = p;
        rq[k] = q;
        rc[k] = c;
        rs[k] = s;
        rot[(size_t)rounds * half + k] = make_double2(c, s);
      }
      __syncthreads();
      // a warp takes rows of pair i, its lanes the columns of the pairs j
      for (int e = tid >> 5; e < half * jw; e += nt >> 5) {
        const int i = jw == 1 ? e : e / jw, j = (e - i * jw) * 32 + (tid & 31);
        if (j >= half) continue;
        const double si = rs[i], sj = rs[j];
        if (si == 0.0 && sj == 0.0) continue;
        const double ci = rc[i], cj = rc[j];
        const int p = rp[i], q = rq[i], u = rp[j], v = rq[j];
        const bool hq = q < n, hv = v < n;  // the padding index of an odd n is not rotated
        double apu = A[p * ld + u], apv = hv ? A[p * ld + v] : 0.0;
        double aqu = hq ? A[q * ld + u] : 0.0, aqv = hq && hv ? A[q * ld + v] : 0.0;
        if (si != 0.0) {
          double x = apu, y = aqu;
          apu = ci * x - si * y;
          aqu = si * x + ci * y;
          x = apv;
          y = aqv;
          apv = ci * x - si * y;
          aqv = si * x + ci * y;
        }
        if (sj != 0.0) {
          double x = apu, y = apv;
          apu = cj * x - sj * y;
          apv = sj * x + cj * y;
          x = aqu;
          y = aqv;
          aqu = cj * x - sj * y;
          aqv = sj * x + cj * y;
        }
        A[p * ld + u] = apu;
        if (hv) A[p * ld + v] = apv;
        if (hq) A[q * ld + u] = aqu;
        if (hq && hv) A[q * ld + v] = aqv;
      }
      __syncthreads();
    }
    converged = (nrot == 0);
    __syncthreads();  // every thread has read nrot before it is reset
  }
  // ascending order (ties by index): rank of each eigenvalue
  for (int i = tid; i < n; i += nt) {
    const double d = A[i * ld + i];
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double dj = A[j * ld + j];
      rank += (dj < d || (dj == d && j < i)) ? 1 : 0;
    }
    wout[rank] = d;
    meta[2 + i] = rank;
  }
  if (tid == 0) {
    meta[0] = converged ? 0 : 1;
    meta[1] = rounds;
  }
}

__global__ void __launch_bounds__(32) k_sym_eigen_vec(int n, const double2* __restrict__ rot,
                                                      const int* __restrict__ meta, double* __restrict__ vout) {
  __shared__ double col[EIG_SMEM_MAX_N];  // component k of every vector
  constexpr int PER = EIG_SMEM_MAX_N / 64;  // pairs per lane, rounded up below
  const int k = blockIdx.x, lane = threadIdx.x, rounds = meta[1];
  for (int i = lane; i < n; i += 32) col[i] = (i == k) ? 1.0 : 0.0;
  __syncwarp();
  const int m = n + (n & 1), half = m / 2;
  double2 cs[PER + 1], nx[PER + 1];
  auto fetch = [&](int round, double2 (&o)[PER + 1]) {
#pragma unroll
    for (int j = 0; j <= PER; ++j) {
      const int pr = lane + 32 * j;
      o[j] = pr < half && round < rounds ? __ldg(rot + (size_t)round * half + pr) : make_double2(1.0, 0.0);
    }
  };
  // the pairs of round 0; every index but 0 then moves on by one in each round
  int ia[PER + 1], ib[PER + 1];
#pragma unroll
  for (int j = 0; j <= PER; ++j) {
    const int pr = lane + 32 * j;
    ia[j] = pr == 0 ? 0 : pr;
    ib[j] = m - 1 - pr;
  }
  fetch(0, cs);
  for (int round = 0; round < rounds; ++round) {
    fetch(round + 1, nx);
#pragma unroll
    for (int j = 0; j <= PER; ++j) {
      if (cs[j].y != 0.0) {
        const int p = min(ia[j], ib[j]), q = max(ia[j], ib[j]);
        const double c = cs[j].x, s = cs[j].y, x = col[p], y = col[q];
        col[p] = c * x - s * y;
        col[q] = s * x + c * y;
      }
      cs[j] = nx[j];
      if (ia[j] != 0 && ++ia[j] == m) ia[j] = 1;
      if (++ib[j] == m) ib[j] = 1;
    }
    __syncwarp();
  }
  for (int i = lane; i < n; i += 32) vout[(size_t)k * n + meta[2 + i]] = col[i];
}

cudaError_t init_sym_eigen() {
  return cudaFuncSetAttribute(k_sym_eigen_rot, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(sizeof(double) * EIG_SMEM_MAX_N * (EIG_SMEM_MAX_N + 1)));
}

static size_t eig_rotations(int n) {
  const size_t m = n + (n & 1);
  return (size_t)EIG_MAX_SWEEPS * (m > 0 ? m - 1 : 0) * (m / 2);
}

// n <= EIG_SMEM_MAX_N: the recorded rotations; beyond: the matrix and Vt.
size_t sym_eigen_work(int n) {
  return n <= EIG_SMEM_MAX_N ? 2 * eig_rotations(n) + 2 : (size_t)n * (n + 1) + (size_t)n * n;
}
size_t sym_eigen_info(int n) { return (size_t)n + 2; }

int launch_sym_eigen(int n, const double* a, double* work, double* w, double* v, int* info, cudaStream_t st) {
  if (n < 1 || n > EIG_MAX_N) return 0;
  if (n <= EIG_SMEM_MAX_N) {
    double2* rot = reinterpret_cast<double2*>(work);
    k_sym_eigen_rot<<<1, EIG_THREADS, sizeof(double) * n * (n + 1), st>>>(n, a, rot, w, info);
    k_sym_eigen_vec<<<n, 32, 0, st>>>(n, rot, info, v);
    return 2;
  }
  k_sym_eigen<<<1, EIG_THREADS, 0, st>>>(n, a, work, work + (size_t)n * (n + 1), w, v, info);
  return 1;
}

}  // namespace flosic
