// FO densities by the reference's route (sm_100a, FP64).
//
// POISSON1 builds the density of each FO, for the SIC exchange-correlation,
// from the Gaussian-pair polynomials of the Poisson calls: at the points inside
// a call's RCUT sphere (every point when NPOT = 1) it adds, pair by pair,
//   rho_p(r) = exp(-ARG) POLY(r - C) . RHOC  exp(-delta |r - C|^2)
// and, for gradient corrections, the derivative polynomials RHOD of the
// gradient and second-derivative channels (poisson1.f:849-948, coefficients
// from gtdncf.F:5-1113).  Coefficients of magnitude <= 1e-14 are skipped and
// the points outside RCUT receive nothing from the call's pairs, so this
// density is the reference's truncated one rather than phi^2.
//
//   k_pair_dens_coef   RHOC (35) per (pair, FO), thresholded as the reference
//                      skips its entries.  Every RHOD entry is a power f times one
//                      RHOC entry (gtdncf.F), so the derivative channels are the
//                      derivatives of the one polynomial, except where RHOC is
//                      between 1e-14 / f and 1e-14: the entry is then kept in the
//                      channels of those f alone, and listed apart.
//   k_pair_density     all pairs of one FO over one mesh tile: near test per
//                      point, the polynomial with its derivatives, channel sums
//                      in call order
#include <cstddef>

#include "coulomb_common.cuh"
#include "kernels.cuh"

namespace flosic {

namespace {

// Cartesian powers of the ten s/p/d components (x, y, z order).
__constant__ int c_dens_pow[10][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {2, 0, 0},
                                      {0, 2, 0}, {0, 0, 2}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}};

constexpr double DENS_EPS = 1.0e-14;  // poisson1.f:860,870,880
constexpr int DENS_THREADS = TILE;    // one mesh point per thread

// A coefficient row: 35 entries in the order pair_channels reads them (x power
// descending, then y, then z), then a bit per monomial m that only derivative
// channels keep.  The values of those are in a second array of rows, at m.
constexpr int DENS_LD = 36;
__device__ __forceinline__ int dens_pos(int px, int py, int pz) {
  const int n = 4 - px, u = n - py, s = u - pz;
  return n * (n + 1) * (n + 2) / 6 + u * (u + 1) / 2 + s;
}

__device__ __forceinline__ double dens_keep(double v) { return fabs(v) > DENS_EPS ? v : 0.0; }

// Powers (px, py, pz) of monomial m in the POLY order (degree, then x power
// ascending, then y power ascending).
__device__ __forceinline__ void mono_powers(int m, int& px, int& py, int& pz) {
  const int d = (m == 0) ? 0 : (m < 4) ? 1 : (m < 10) ? 2 : (m < 20) ? 3 : 4;
  const int base = (d == 0) ? 0 : (d == 1) ? 1 : (d == 2) ? 4 : (d == 3) ? 10 : 20;
  int off = m - base, x = 0;
  while (off >= d - x + 1) {
    off -= d - x + 1;
    ++x;
  }
  px = x;
  py = off;
  pz = d - x - off;
}

__global__ void __launch_bounds__(128) k_pair_dens_coef(const PairGeo* __restrict__ pairs, int nfo, int nprim,
                                                        const double* __restrict__ u, int nch,
                                                        double* __restrict__ dc, double* __restrict__ dronly) {
  __shared__ double P1[10][10][3][5];
  const int ip = blockIdx.x, tid = threadIdx.x;
  const PairGeo g = pairs[ip];
  // gtdncf.F:9-16: the product centre and exponent argument of the pair
  const double dlt = g.a + g.b;
  double C[3], arg = 0.0;
  for (int d = 0; d < 3; ++d) {
    C[d] = (g.a * g.A[d] + g.b * g.B[d]) / dlt;
    arg = arg + (g.A[d] - g.B[d]) * (g.A[d] - g.B[d]);
  }
  arg = arg * g.a * g.b / dlt;
  // 1-D factors (rho + C - A)^na (rho + C - B)^nb as polynomials in rho
  for (int q = tid; q < 300; q += blockDim.x) {
    const int mu = q / 30, nu = (q / 3) % 10, d = q % 3;
    const double ca = C[d] - g.A[d], cb = C[d] - g.B[d];
    const int na = c_dens_pow[mu][d], nb = c_dens_pow[nu][d];
    double pa[3] = {0, 0, 0}, pb[3] = {0, 0, 0};
    if (na == 0) pa[0] = 1;
    else if (na == 1) { pa[0] = ca; pa[1] = 1; }
    else { pa[0] = ca * ca; pa[1] = 2 * ca; pa[2] = 1; }
    if (nb == 0) pb[0] = 1;
    else if (nb == 1) { pb[0] = cb; pb[1] = 1; }
    else { pb[0] = cb * cb; pb[1] = 2 * cb; pb[2] = 1; }
    double e[5] = {0, 0, 0, 0, 0};
    for (int x = 0; x <= na; ++x)
      for (int y = 0; y <= nb; ++y) e[x + y] += pa[x] * pb[y];
    for (int j = 0; j < 5; ++j) P1[mu][nu][d][j] = e[j];
  }
  for (int k = tid; k < nfo; k += blockDim.x) dc[((size_t)ip * nfo + k) * DENS_LD + 35] = 0.0;  // no bit set
  __syncthreads();
  const double ex = exp(-arg);
  for (int q = tid; q < nfo * 35; q += blockDim.x) {
    const int k = q / 35, m = q % 35;
    int px, py, pz;
    mono_powers(m, px, py, pz);
    const double* pu = u + ((size_t)k * nprim + g.pi) * 10;
    const double* pv = u + ((size_t)k * nprim + g.pj) * 10;
    // RHOC(m) = exp(-ARG) sum_{mu,nu} GAM(mu,nu) x-factor y-factor z-factor, with
    // GAM the pair block of the FO's density matrix (coupot_sic.F:366-482)
    double s = 0.0;
    for (int mu = 0; mu < 10; ++mu) {
      const double ui = pu[mu];
      if (ui == 0.0) continue;
      for (int nu = 0; nu < 10; ++nu) {
        const double gm = ui * pv[nu] * g.times;
        if (gm == 0.0) continue;
        const double fx = P1[mu][nu][0][px], fy = P1[mu][nu][1][py], fz = P1[mu][nu][2][pz];
        if (fx == 0.0 || fy == 0.0 || fz == 0.0) continue;
        s += gm * fx * fy * fz;
      }
    }
    const double rc = s * ex;
    const size_t r0 = ((size_t)ip * nfo + k) * DENS_LD;
    dc[r0 + dens_pos(px, py, pz)] = dens_keep(rc);
    // the largest factor of the monomial's RHOD entries
    const int lo = min(px, min(py, pz)), hi = max(px, max(py, pz)), mid = px + py + pz - lo - hi;
    const int f = nch == 1 ? 0 : (nch == 4 ? hi : max(hi, max(hi * (hi - 1), hi * mid)));
    if (dens_keep(rc) == 0.0 && dens_keep(f * rc) != 0.0) {
      dronly[r0 + m] = rc;
      atomicOr(reinterpret_cast<unsigned long long*>(dc + r0 + 35), 1ull << m);
    }
  }
}

// Value, first derivative and half the second derivative of a polynomial by
// Horner's scheme, coefficients highest first; t counts them from 0 (a compile-
// time constant after unrolling), ND the derivatives kept.
template <int ND>
struct Horner {
  double v, d1, d2;
  __device__ __forceinline__ void add(int t, double x, double c) {
    if (ND >= 2 && t >= 2) d2 = t == 2 ? d1 : fma(d2, x, d1);
    if (ND >= 1 && t >= 1) d1 = t == 1 ? v : fma(d1, x, v);
    v = t == 0 ? c : fma(v, x, c);
  }
};

// x^e for e <= 3 (1 for e < 0, where the factor is zero).
__device__ __forceinline__ double power3(double x, int e) {
  const double x2 = x * x;
  return e <= 0 ? 1.0 : (e == 1 ? x : (e == 2 ? x2 : x2 * x));
}

// Channels 1.. of the monomials that only derivative channels keep, before the
// Gaussian factor: every RHOD entry f c above the threshold, with its product-rule
// terms.  of: their values.  Out of line, since a row with such an entry is the
// exception (20 atoms, 64 FOs, 50,021 points, PBE: k_pair_density 26.6 ms without
// these entries, 27.5 with them; 28.3 with the first value loaded ahead).
template <int NCH>
__device__ __noinline__ void derivative_only(unsigned long long bits, const double* __restrict__ of, double x,
                                             double y, double z, double delta, double* a) {
  double g[3] = {0.0, 0.0, 0.0}, h[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (; bits; bits &= bits - 1) {
    const int m = __ffsll((long long)bits) - 1;
    const double c = of[m];
    int px, py, pz;
    mono_powers(m, px, py, pz);
    const double X = px == 4 ? x * power3(x, 3) : power3(x, px), Y = py == 4 ? y * power3(y, 3) : power3(y, py),
                 Z = pz == 4 ? z * power3(z, 3) : power3(z, pz);
    const double X1 = power3(x, px - 1), Y1 = power3(y, py - 1), Z1 = power3(z, pz - 1);
    g[0] += dens_keep(px * c) * (X1 * Y * Z);
    g[1] += dens_keep(py * c) * (X * Y1 * Z);
    g[2] += dens_keep(pz * c) * (X * Y * Z1);
    if constexpr (NCH == 10) {
      h[0] += dens_keep(px * (px - 1) * c) * (power3(x, px - 2) * Y * Z);
      h[1] += dens_keep(py * (py - 1) * c) * (X * power3(y, py - 2) * Z);
      h[2] += dens_keep(pz * (pz - 1) * c) * (X * Y * power3(z, pz - 2));
      h[3] += dens_keep(px * py * c) * (X1 * Y1 * Z);
      h[4] += dens_keep(px * pz * c) * (X1 * Y * Z1);
      h[5] += dens_keep(py * pz * c) * (X * Y1 * Z1);
    }
  }
  const double d2 = 2.0 * delta;
  a[0] = g[0];
  a[1] = g[1];
  a[2] = g[2];
  if constexpr (NCH == 10) {
    a[3] = h[0] - 2.0 * d2 * x * g[0];
    a[4] = h[1] - 2.0 * d2 * y * g[1];
    a[5] = h[2] - 2.0 * d2 * z * g[2];
    a[6] = h[3] - d2 * (y * g[0] + x * g[1]);
    a[7] = h[4] - d2 * (z * g[0] + x * g[2]);
    a[8] = h[5] - d2 * (z * g[1] + y * g[2]);
  }
}

// Channels of one pair and one FO at offset (x, y, z) before the Gaussian
// factor: the polynomial RHOC and its derivatives by nested Horner schemes (z
// inside y inside x, 90 multiply-adds for all ten channels against 155 with the
// monomials and RHOD tables), then the product-rule terms of the Gaussian's
// derivatives (poisson1.f:849-940).  row: its 35 coefficients in shared memory,
// read in order.
template <int NCH>
__device__ __forceinline__ void pair_channels(double x, double y, double z, double delta,
                                              const double* __restrict__ row, double (&a)[NCH]) {
  constexpr int ND = NCH == 1 ? 0 : (NCH == 4 ? 1 : 2);
  const double2* r2 = reinterpret_cast<const double2*>(row);
  Horner<ND> X;                                  // the polynomial in x
  Horner<(ND > 1 ? 1 : 0)> XY, XZ;               // its y and z derivatives
  Horner<0> XYY, XZZ, XYZ;
  double2 two = r2[0];
  int at = 0;
#pragma unroll
  for (int n = 0; n <= 4; ++n) {                 // x power 4 - n
    Horner<ND> Y;
    Horner<(ND > 1 ? 1 : 0)> YZ;
    Horner<0> YZZ;
#pragma unroll
    for (int u = 0; u <= n; ++u) {               // y power n - u
      Horner<ND> Z;
#pragma unroll
      for (int s = 0; s <= u; ++s, ++at) {       // z power u - s
        if (at > 0 && (at & 1) == 0) two = r2[at >> 1];
        Z.add(s, z, (at & 1) ? two.y : two.x);
      }
      Y.add(u, y, Z.v);
      if (ND >= 1 && u >= 1) YZ.add(u - 1, y, Z.d1);
      if (ND >= 2 && u >= 2) YZZ.add(u - 2, y, Z.d2);
    }
    X.add(n, x, Y.v);
    if (ND >= 1 && n >= 1) {
      XY.add(n - 1, x, Y.d1);
      XZ.add(n - 1, x, YZ.v);
    }
    if (ND >= 2 && n >= 2) {
      XYY.add(n - 2, x, Y.d2);
      XYZ.add(n - 2, x, YZ.d1);
      XZZ.add(n - 2, x, YZZ.v);
    }
  }
  a[0] = X.v;
  if constexpr (NCH > 1) {
    const double d1x2 = delta * 2.0, px = X.d1, py = XY.v, pz = XZ.v;
    if constexpr (NCH == 10) {
      const double d1x4 = delta * 4.0, d2x4 = delta * delta * 4.0;
      a[4] = 2.0 * X.d2 - d1x4 * x * px + (d2x4 * (x * x) - d1x2) * a[0];
      a[5] = 2.0 * XYY.v - d1x4 * y * py + (d2x4 * (y * y) - d1x2) * a[0];
      a[6] = 2.0 * XZZ.v - d1x4 * z * pz + (d2x4 * (z * z) - d1x2) * a[0];
      a[7] = XY.d1 - d1x2 * y * px - d1x2 * x * py + d2x4 * (x * y) * a[0];
      a[8] = XZ.d1 - d1x2 * z * px - d1x2 * x * pz + d2x4 * (x * z) * a[0];
      a[9] = XYZ.v - d1x2 * y * pz - d1x2 * z * py + d2x4 * (y * z) * a[0];
    }
    a[1] = px - d1x2 * x * a[0];
    a[2] = py - d1x2 * y * a[0];
    a[3] = pz - d1x2 * z * a[0];
  }
}

// Block = (mesh tile, FO k), one point per thread.  The pairs are taken 128 at a
// time: those whose call's sphere reaches the tile are queued in order with
// their sphere and centre, their coefficient rows stream through two shared
// buffers of DENS_CHUNK rows (cp.async one chunk ahead, one barrier per chunk),
// and each is added at the points inside its sphere, so every point sums its
// contributions in the reference's order.  Bounded by the FP64 pipe (~180
// operations per (pair, point, FO) with ten channels) and its chains at 16 warps per SM.
// Measured, 40 atoms, 128 FOs, 37,888 points, PBE: 288 -> 164 ms (before: one barrier
// per pair and rows of 156 entries, 78 16-byte shared-memory loads each).
constexpr int DENS_CHUNK = 16;
// resident blocks per SM that the registers of the sums allow (the function called
// out of line would take more: 152, 30.3 ms)
constexpr int dens_blocks(int nch) { return nch == 10 ? 4 : (nch == 4 ? 7 : 8); }
template <int NCH>
__global__ void __launch_bounds__(DENS_THREADS, dens_blocks(NCH)) k_pair_density(MeshDev M, int npairs,
                                                               const PairGeo* __restrict__ pairs,
                                                               const CallFO* __restrict__ cfo, int cfo_ld, int nfo,
                                                               const double* __restrict__ dc,
                                                               const double* __restrict__ dronly,
                                                               double* __restrict__ rhog, size_t ldr) {
  __shared__ __align__(16) double s_row[2][DENS_CHUNK][DENS_LD];
  __shared__ double s_geo[DENS_THREADS][4];  // queue: C[3], delta
  __shared__ double s_cg[DENS_THREADS][4];   // queue: CG, RCUT^2
  __shared__ int s_pair[DENS_THREADS];
  __shared__ int s_cnt[DENS_THREADS / 32];
  const int tile = blockIdx.x, k = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = M.tile_lo[3 * tile + d];
    hi[d] = M.tile_hi[3 * tile + d];
  }
  const int pt = tile * TILE + tid;
  const bool valid = pt < M.n;
  const double x = valid ? M.x[pt] : 0.0, y = valid ? M.y[pt] : 0.0, z = valid ? M.z[pt] : 0.0;
  double acc[NCH];
#pragma unroll
  for (int c = 0; c < NCH; ++c) acc[c] = 0.0;
  for (int q0 = 0; q0 < npairs; q0 += DENS_THREADS) {
    const int q = q0 + tid;
    bool hit = false;
    int c = 0;
    if (q < npairs) {
      c = pairs[q].call;
      const CallFO& f = cfo[(size_t)c * cfo_ld + k];
      hit = f.npot == 1 || tile_class(lo, hi, f.cg[0], f.cg[1], f.cg[2], f.rcut2) != 1;
    }
    const unsigned b = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) s_cnt[warp] = __popc(b);
    __syncthreads();  // and every thread is done with the previous window
    int before = 0, qn = 0;
#pragma unroll
    for (int w = 0; w < DENS_THREADS / 32; ++w) {
      before += (w < warp) ? s_cnt[w] : 0;
      qn += s_cnt[w];
    }
    if (hit) {
      const int i = before + __popc(b & ((1u << lane) - 1u));
      const CallFO& f = cfo[(size_t)c * cfo_ld + k];
      const PairGeo& g = pairs[q];
      s_pair[i] = q;
      for (int d = 0; d < 3; ++d) {
        s_cg[i][d] = f.cg[d];
        s_geo[i][d] = g.C[d];
      }
      s_cg[i][3] = f.rcut2;
      s_geo[i][3] = g.delta;
    }
    __syncthreads();
    auto copy = [&](int e0, int buf) {
      const int ne = min(DENS_CHUNK, qn - e0);
      for (int i = tid; i < ne * (DENS_LD / 2); i += DENS_THREADS) {
        const int e = i / (DENS_LD / 2), o = i - e * (DENS_LD / 2);
        cp_async16(&s_row[buf][e][2 * o], dc + ((size_t)s_pair[e0 + e] * nfo + k) * DENS_LD + 2 * o);
      }
      cp_async_commit();
    };
    if (qn > 0) copy(0, 0);
    for (int e0 = 0, buf = 0; e0 < qn; e0 += DENS_CHUNK, buf ^= 1) {
      cp_async_wait_all();
      __syncthreads();  // this chunk has arrived and the other buffer is free
      if (e0 + DENS_CHUNK < qn) copy(e0 + DENS_CHUNK, buf ^ 1);
      const int ne = min(DENS_CHUNK, qn - e0);
      for (int i = 0; i < ne; ++i) {
        const double* cg = s_cg[e0 + i];
        const bool near = valid && !(sqdist_rn2(x, y, z, cg[0], cg[1], cg[2]) > cg[3]);
        if (!near) continue;
        const double* g = s_geo[e0 + i];
        const double rx = x - g[0], ry = y - g[1], rz = z - g[2], delta = g[3];
        const double chgd = exp(-(delta * (rz * rz + ry * ry + rx * rx)));
        double a[NCH];
        pair_channels<NCH>(rx, ry, rz, delta, s_row[buf][i], a);
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) acc[ch] += chgd * a[ch];
        if constexpr (NCH > 1) {
          const unsigned long long bits = (unsigned long long)__double_as_longlong(s_row[buf][i][35]);
          if (bits) {
            double e[NCH - 1];
            derivative_only<NCH>(bits, dronly + ((size_t)s_pair[e0 + i] * nfo + k) * DENS_LD, rx, ry, rz, delta, e);
#pragma unroll
            for (int ch = 1; ch < NCH; ++ch) acc[ch] += chgd * e[ch - 1];
          }
        }
      }
    }
  }
  if (valid) {
#pragma unroll
    for (int c = 0; c < NCH; ++c) rhog[((size_t)c * nfo + k) * ldr + pt] = acc[c];
  }
}

}  // namespace

// The rows, and with derivative channels as many again for the entries that only those keep.
int pair_density_ld(int nch) { return nch > 1 ? 2 * DENS_LD : DENS_LD; }

void launch_pair_density(int npairs, const PairGeo* pairs, const CallFO* cfo, int cfo_ld, int nfo, int nprim,
                         const double* u, int nch, const MeshDev& M, double* dc, double* rhog, size_t ldr,
                         cudaStream_t st) {
  if (nfo <= 0 || M.ntiles <= 0) return;
  double* dronly = dc + (size_t)npairs * nfo * DENS_LD;
  if (npairs > 0) k_pair_dens_coef<<<npairs, 128, 0, st>>>(pairs, nfo, nprim, u, nch, dc, dronly);
  const dim3 grid(M.ntiles, nfo);
#define PD(n) k_pair_density<n><<<grid, DENS_THREADS, 0, st>>>(M, npairs, pairs, cfo, cfo_ld, nfo, dc, dronly, rhog, ldr)
  if (nch == 1) PD(1);
  else if (nch == 4) PD(4);
  else PD(10);
#undef PD
}

}  // namespace flosic
