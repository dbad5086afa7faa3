// Coulomb potential of the calls whose near/far geometry differs per FO
// (every call with more than one POISSON1 slot: its CG is charge weighted,
// poisson1.f:503-520).  Near field and far field are two kernels.
//
//   k_perfo_near  A CTA owns 64 mesh points (8 warps x 8) and up to 32, 64 or
//                 128 FOs and walks the pairs of the calls in order, 128 at a
//                 time: it drops the calls with no near point of any FO in its
//                 box, lists the FOs that have some, and streams those FOs'
//                 coefficient rows through two shared-memory buffers.  A warp
//                 forms the G columns of its points in registers, directly as B
//                 fragments of mma.sync m8n8k4 .f64 (lane 4 n + q holds row q of
//                 each k-step at point n; one column per (pair, point), the Boys
//                 values of four pairs at once over the four lanes of a point),
//                 and multiplies the listed FOs' coefficient rows into FP64
//                 accumulators, added call by call, masked point by
//                 point where a sphere cuts the warp's box.
//   k_perfo_far   One warp owns 64 points (two per lane) and one FO and adds
//                 the L <= 6 multipole expansions of the far calls as Clenshaw
//                 sums.
//
// What bounds it: the FP64 pipe (tensor and FMA path share ~37 TF/s), 92 flops
// per near (pair, point, FO), ~100-260 per far (call, point, FO), and beside it
// the instructions that form a column (~150 per warp and pair).  The form before,
// one 384-thread CTA per 128 points with producer and consumer warps, spent 9-14
// us per (call, tile) in CTA barriers, stage hand-overs and per-call FO status,
// whatever the call's size; with NSPN=2 most calls are one 16-48-row pair.
// Measured, FP64, both kernels: benzene (37,843 points, 21 + 21 FOs) 85.9 -> 24.5
// ms (near 16.9, far 11.5 when alone; far on a side stream), the 40-atom system
// (100,003 points, 128 FOs) 108 -> 62 ms, water (3,942 points) 2.0 -> 0.13 ms.
#include <algorithm>

#include "coulomb_common.cuh"

namespace flosic {

// Columns of one pair in MMA order: k-step s (0..11), lane residue q.  Row of
// COEFICIENT order at position 4 s + q (-1: zero).  Residues 1, 2, 3 hold the
// monomials of one cyclic permutation (a,b,c) of (x,y,z) each, so their values
// have one formula; residue 0, with (a,b,c) = (x,y,z), holds the rest:
//   F_0..F_2 group   a F1 | a F2 | aa F2 | ab F2      (0: F0, F1, F2, none)
//   F_3 group        aa | ab | aaa | aab              (0: xyz, xxz, xyy, yzz)
//   F_4 group        aaaa | aaab | aaac | aabb        (0: xxyz, xyyz, xyzz, none)
// The first 4, 8 and 12 k-steps are the pairs of Boys variant 3, 4 and 5.
__constant__ int8_t c_mma_row[NEAR_K] = {0,  5,  4,  3,  1,  8,  7,  6,  2,  14, 11, 9,  -1, 13, 10, 12,
                                         26, 20, 17, 15, 28, 19, 16, 18, 27, 30, 24, 21, 22, 29, 23, 25,
                                         41, 45, 35, 31, 38, 44, 34, 36, 37, 43, 39, 32, -1, 42, 33, 40};

// Brings the coefficient rows of the per-FO calls' pairs into the order the lanes
// read them, in place: nothing reads the former order after the call set-up, and a
// second array would be as large as the coefficients.  A row is [group g of four
// k-steps][16]; the 16-byte piece that holds k-steps 4 g + 2 h and 4 g + 2 h + 1 of
// residue q is number 4 h + q of its group.  A warp takes a row at a time.
__global__ void __launch_bounds__(256) k_perfo_pack(int nfo, const PairGeo* __restrict__ pairs,
                                                    const CallShare* __restrict__ share, int per_fo_only,
                                                    double* __restrict__ coef) {
  const int pr = blockIdx.x, lane = threadIdx.x & 31;
  if (!per_fo_only && share[pairs[pr].call].shared) return;
  auto from = [](int e) { return (int)c_mma_row[4 * (4 * (e >> 4) + 2 * ((e >> 3) & 1) + (e & 1)) + ((e >> 1) & 3)]; };
  const int r0 = from(lane), r1 = lane < NEAR_K - 32 ? from(lane + 32) : -1;
  for (int k = threadIdx.x >> 5; k < nfo; k += blockDim.x >> 5) {
    double* row = coef + ((size_t)pr * nfo + k) * COEF_LD;
    const double v0 = r0 >= 0 ? row[r0] : 0.0, v1 = r1 >= 0 ? row[r1] : 0.0;
    __syncwarp();
    row[lane] = v0;
    if (lane < NEAR_K - 32) row[lane + 32] = v1;
  }
}

// Spheres around the mean pair centre c of each call: a point within rin is
// near for every FO, a point beyond rout for none.  One warp per call.
__global__ void __launch_bounds__(256) k_perfo_bounds(int ncalls, int nfo, const CallInfo* __restrict__ calls,
                                                      const PairGeo* __restrict__ pairs,
                                                      const CallFO* __restrict__ cfo, CallBound* __restrict__ out) {
  const int c = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= ncalls) return;
  const CallInfo ci = calls[c];
  double s[3] = {0.0, 0.0, 0.0};
  for (int q = lane; q < ci.np; q += 32)
    for (int d = 0; d < 3; ++d) s[d] += pairs[ci.p0 + q].C[d];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    for (int o = 16; o > 0; o >>= 1) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
    s[d] /= ci.np;
  }
  double rin = DBL_MAX, rout = 0.0;
  for (int k = lane; k < nfo; k += 32) {
    const CallFO& f = cfo[(size_t)c * nfo + k];
    if (f.npot == 1) {
      rout = DBL_MAX;
      continue;
    }
    const double dx = f.cg[0] - s[0], dy = f.cg[1] - s[1], dz = f.cg[2] - s[2];
    const double d = sqrt(dx * dx + dy * dy + dz * dz);
    rin = fmin(rin, f.rcut * (1.0 - 1e-12) - d * (1.0 + 1e-12));
    rout = fmax(rout, (f.rcut + d) * (1.0 + 1e-12));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    rin = fmin(rin, __shfl_xor_sync(0xffffffffu, rin, o));
    rout = fmax(rout, __shfl_xor_sync(0xffffffffu, rout, o));
  }
  if (lane == 0) {
    CallBound b;
    for (int d = 0; d < 3; ++d) b.c[d] = s[d];
    rin = fmax(rin, 0.0);
    b.rin2 = rin < 1e150 ? rin * rin : DBL_MAX;
    b.rout2 = rout < 1e150 ? rout * rout : DBL_MAX;
    b.p0 = ci.p0;
    b.np = ci.np;
    out[c] = b;
  }
}

// Box of a warp's points (each lane gives one point that exists).
__device__ __forceinline__ void warp_box(double x, double y, double z, double lo[3], double hi[3]) {
  lo[0] = hi[0] = x;
  lo[1] = hi[1] = y;
  lo[2] = hi[2] = z;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
}

// 0: every point near for every FO; 1: no point near for any FO; 2: neither.
__device__ __forceinline__ int bound_class(const double lo[3], const double hi[3], const CallBound& b) {
  const int in = tile_class(lo, hi, b.c[0], b.c[1], b.c[2], b.rin2);
  if (in == 0) return 0;
  return tile_class(lo, hi, b.c[0], b.c[1], b.c[2], b.rout2) == 1 ? 1 : 2;
}

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// ---------------------------------------------------------------------------
// Near field
// ---------------------------------------------------------------------------
constexpr int NEAR_WARPS = 8;                  // warps per CTA
constexpr int NEAR_PTS = 8;                    // points per warp
constexpr int NEAR_THREADS = 32 * NEAR_WARPS;
constexpr int NEAR_CTA_PTS = NEAR_WARPS * NEAR_PTS;
constexpr int NEAR_PER_TILE = TILE / NEAR_CTA_PTS;
constexpr int NEAR_WIN = 128;                  // pairs classified at once
constexpr int near_rows_cap(int mt) { return mt <= 4 ? 192 : (mt <= 8 ? 224 : 448); }

struct __align__(16) NearEntry {
  int pre;                                     // coefficient rows of the entries before it
  int call, pair;
  uint8_t lead, nl, fmt, flags;                // index into lead, listed FOs, Boys variant, NEAR_FIRST ...
};
constexpr int NEAR_FIRST = 1, NEAR_LAST = 2;   // of its call
constexpr int NEAR_CUT = 4;                    // last of a call some sphere of which cuts the CTA's box: after its
                                               // coefficient rows come the listed FOs' CallFO records, two per row

template <int MT>
struct NearSmem {
  static constexpr int ROWS = near_rows_cap(MT);  // coefficient rows (16 doubles) per buffer
  static_assert(ROWS >= 3 * 8 * MT + 4 * MT, "a pair's rows of all FOs and their spheres fit");
  double A[2][ROWS * 16];
  double V[NEAR_WARPS][8 * MT * NEAR_PTS];     // the warps' potentials, [FO][point]
  double p[NEAR_CTA_PTS][3];
  double box[NEAR_WARPS + 1][6];               // of each warp's points, and of all
  double geo[NEAR_WIN][6];                     // queue: pair centre x y z x y, exponent sum
  NearEntry queue[NEAR_WIN + 1];               // the window's pairs with near points in this CTA
  int lead[NEAR_WIN];                          // the window's calls; + (1 << 30) when all FOs are near
  int cnt[NEAR_WIN];                           // FOs of the block with near points in the CTA's box
  int wcount[NEAR_WIN / 32][2];
  uint8_t list[NEAR_WIN][8 * MT];              // those FOs, ascending
};

// The column values of one (pair, point) for lane residue q: four k-steps of
// group g, products in the association of poisson1.f:925-959.  Positions whose
// coefficient row is padding hold any finite value.
template <typename T>
struct NearLane {
  T a, b, c, aa, ab, bb;
  __device__ __forceinline__ NearLane(T a_, T b_, T c_) : a(a_), b(b_), c(c_), aa(a_ * a_), ab(a_ * b_), bb(b_ * b_) {}
};
template <typename T, int g>
__device__ __forceinline__ void near_group(const NearLane<T>& L, const T (&F)[5], bool q0, double (&o)[4]) {
  if constexpr (g == 0) {
    o[0] = (double)(q0 ? F[0] : F[1] * L.a);
    o[1] = (double)(q0 ? F[1] : F[2] * L.a);
    o[2] = (double)(q0 ? F[2] : F[2] * L.aa);
    o[3] = (double)(F[2] * L.ab);
  } else if constexpr (g == 1) {
    o[0] = (double)(F[3] * (q0 ? L.a * (L.b * L.c) : L.aa));
    o[1] = (double)(F[3] * (q0 ? L.c * L.aa : L.ab));
    o[2] = (double)(F[3] * (L.a * (q0 ? L.bb : L.aa)));
    o[3] = (double)(F[3] * (L.b * (q0 ? L.c * L.c : L.aa)));
  } else {
    const T t = q0 ? L.b * L.c : L.aa;
    o[0] = (double)(F[4] * (L.aa * t));
    o[1] = (double)(F[4] * (L.ab * t));
    o[2] = (double)(F[4] * (q0 ? L.ab * (L.c * L.c) : (L.a * L.c) * L.aa));
    o[3] = (double)(F[4] * (L.aa * L.bb));
  }
}

// Boys values F_0..F_{fmt-1} (absent orders zero) by the steps of boys_fmt, with
// the variant chosen by selection: the lanes of a warp hold different pairs.
template <typename T>
__device__ __forceinline__ void near_boys(const double* __restrict__ tab, T x, T ex, int fmt, T (&F)[5]) {
  if (x > T(16)) {
    if constexpr (sizeof(T) == 8) {  // as boys_fmt, from one reciprocal square root
      const double h = rsqrt(x), r = 0.5 * h * h;
      F[0] = r * (x * h * 1.77245385090551602728 - ex);
      F[1] = r * (F[0] - ex);
      F[2] = r * (3.0 * F[1] - ex);
      F[3] = r * (5.0 * F[2] - ex);
      F[4] = r * (7.0 * F[3] - ex);
    } else {
      boys_fmt<T>(tab, x, ex, fmt, F);
    }
    return;
  }
  const int it = (int)(T(100) * x + T(1.5));
  const T rect1 = T(2) * x, dt = T(1.0e-2) * T(it - 1) - x;
  const double* f = tab + (size_t)(it - 1) * BOYS_NC + (fmt - 3);
  const T o7 = T(1) / T(7), o5 = T(1) / T(5), o3 = T(1) / T(3);
  const T top = T(f[0]) + dt * (T(f[1]) + dt * (T(f[4]) + dt * T(f[7])));
  F[4] = fmt == 5 ? top : T(0);
  F[3] = fmt == 5 ? (top * rect1 + ex) * o7 : (fmt == 4 ? top : T(0));
  F[2] = fmt == 3 ? top : (F[3] * rect1 + ex) * o5;
  F[1] = (F[2] * rect1 + ex) * o3;
  F[0] = F[1] * rect1 + ex;
}

// Four k-steps of one group: two 16-byte fragment loads and four MMAs per eight
// listed FOs.  A0, A1: the lane's two pieces of the first rows.  An entry lists at
// least one FO, so the first eight need no test (benzene: 24.8 -> 24.5 ms, 128 FOs
// and 100,003 points: 63.3 -> 62.2).
template <int MT, typename T, int g>
__device__ __forceinline__ void near_mma(double (&acc)[MT][2], const double* __restrict__ A0,
                                         const double* __restrict__ A1, int nmt, const NearLane<T>& L,
                                         const T (&F)[5], bool q0) {
  double b[4];
  near_group<T, g>(L, F, q0, b);
  auto step = [&](int mt) {
    const double2 a0 = *reinterpret_cast<const double2*>(A0 + mt * 128);
    const double2 a1 = *reinterpret_cast<const double2*>(A1 + mt * 128);
    dmma(acc[mt], a0.x, b[0]);
    dmma(acc[mt], a0.y, b[1]);
    dmma(acc[mt], a1.x, b[2]);
    dmma(acc[mt], a1.y, b[3]);
  };
  step(0);
#pragma unroll
  for (int mt = 1; mt < MT; ++mt) {
    if (mt >= nmt) break;
    step(mt);
  }
}

// delta |r|^2 (poisson1.f:640-650); the single-precision form fixes its roundings
template <typename T>
__device__ __forceinline__ T near_arg(T delta, T x, T y, T z) {
  if constexpr (sizeof(T) == 4) return delta * __fadd_rn(__fadd_rn(__fmul_rn(z, z), __fmul_rn(y, y)), __fmul_rn(x, x));
  else return delta * (z * z + y * y + x * x);
}

template <int MT, bool MIXED>
__device__ __forceinline__ void near_block(const CoulombJob& J, int blk, int fob, int part,
                                           const double* __restrict__ tab) {
  using PT = typename std::conditional<MIXED, float, double>::type;
  constexpr int FOB = 8 * MT;
  extern __shared__ __align__(128) unsigned char smraw[];
  NearSmem<MT>& S = *reinterpret_cast<NearSmem<MT>*>(smraw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = lane >> 2, q = lane & 3;
  const int k0 = fob * FOB, nk = min(FOB, J.nfo - k0);
  const int cta0 = blk * NEAR_CTA_PTS;
  if (cta0 >= J.M.n) return;  // whole CTA
  const int npairs = J.lists[2 * J.ncalls + 2];
  if (npairs == 0) return;
  // this part's pairs; a call cut by the part's ends begins and ends there
  const int pl0 = (int)((long long)npairs * part / J.nseg), npl = (int)((long long)npairs * (part + 1) / J.nseg);
  const int pb = cta0 + warp * NEAR_PTS;
  const int npt = min(NEAR_PTS, J.M.n - pb);  // <= 0: this warp only helps with the copies
  double* V = S.V[warp];
  for (int e = lane; e < nk * NEAR_PTS; e += 32) V[e] = 0.0;
  {
    // points past the end repeat the last one and are not stored
    const int p = min(pb + (lane & 7), J.M.n - 1);
    const double x = J.M.x[p], y = J.M.y[p], z = J.M.z[p];
    double lo[3], hi[3];
    warp_box(x, y, z, lo, hi);
    if (lane < NEAR_PTS) {
      S.p[warp * NEAR_PTS + lane][0] = x;
      S.p[warp * NEAR_PTS + lane][1] = y;
      S.p[warp * NEAR_PTS + lane][2] = z;
    }
    if (lane == 0)
      for (int d = 0; d < 3; ++d) {
        S.box[warp][d] = lo[d];
        S.box[warp][3 + d] = hi[d];
      }
  }
  __syncthreads();
  if (tid < 6) {
    double v = S.box[0][tid];
    for (int w = 1; w < NEAR_WARPS; ++w) v = tid < 3 ? fmin(v, S.box[w][tid]) : fmax(v, S.box[w][tid]);
    S.box[NEAR_WARPS][tid] = v;
  }
  __syncthreads();
  const double(*pts)[3] = &S.p[warp * NEAR_PTS];
  const double* box = S.box[warp];
  double T[MT][2];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) T[mt][0] = T[mt][1] = 0.0;
  int np = 0;  // pairs of the open call
  const int piece = n * 16 + 2 * (q ^ ((n & 1) << 2));  // of the lane's coefficient rows
  PT Fq[5] = {};  // Boys values of one pair of the current four
  const int cyc = max(q - 1, 0);  // the lane's coordinates: (x,y,z), (x,y,z), (y,z,x), (z,x,y)
  const double pa = pts[n][cyc], pb_ = pts[n][cyc == 2 ? 0 : cyc + 1], pc = pts[n][cyc == 0 ? 2 : cyc - 1];
  unsigned long long near = 0;
  // asynchronous copy of the coefficient rows of queue entries [e0, e1) into
  // buffer b, one warp per entry: [group][listed FO][16], the halves of odd rows
  // exchanged so that the eight lanes of two rows read all 32 banks
  auto copy = [&](int e0, int e1, int b) {
    for (int e = e0 + warp; e < e1; e += NEAR_WARPS) {
      const NearEntry w = S.queue[e];
      const int nl = w.nl;
      const uint8_t* list = S.list[w.lead];
      double* dst = S.A[b] + (w.pre - S.queue[e0].pre) * 16;
      for (int g = 0; g < w.fmt - 2; ++g, dst += nl * 16) {
        const double* src = J.coef + ((size_t)w.pair * J.nfo + k0) * COEF_LD + g * 16;
        for (int i = lane; i < nl * 8; i += 32) {
          const int r = i >> 3, pc = i & 7;
          cp_async16(dst + r * 16 + 2 * (pc ^ ((r & 1) << 2)), src + (int)list[r] * COEF_LD + 2 * pc);
        }
      }
      if (w.flags & NEAR_CUT) {
        const CallFO* cf = J.cfo + (size_t)w.call * J.nfo + k0;
        for (int i = lane; i < nl * 4; i += 32)
          cp_async16(dst + 2 * i, reinterpret_cast<const double*>(cf + list[i >> 2]) + 2 * (i & 3));
      }
    }
    cp_async_commit();
  };

  for (int w0 = pl0; w0 < npl; w0 += NEAR_WIN) {
    // 1. the window's calls with near points of some FO in the CTA's box
    bool act = false, leads = false;
    int cls = 1;
    PerfoPair my{};
    const double* bx = S.box[NEAR_WARPS];
    const double clo[3] = {bx[0], bx[1], bx[2]}, chi[3] = {bx[3], bx[4], bx[5]};
    if (tid < NEAR_WIN && w0 + tid < npl) {
      my = J.plist[w0 + tid];
      if (w0 + tid == pl0) my.first = 1;
      if (w0 + tid == npl - 1) my.last = 1;
      cls = bound_class(clo, chi, J.bound[my.call]);
      act = cls != 1;
      leads = act && (tid == 0 || my.first);
    }
    unsigned bal = __ballot_sync(0xffffffffu, leads);
    if (lane == 0 && warp < NEAR_WIN / 32) S.wcount[warp][0] = __popc(bal);
    __syncthreads();  // and every warp is done with the previous window
    int before = 0, nlead = 0;
#pragma unroll
    for (int w = 0; w < NEAR_WIN / 32; ++w) {
      const int cw = S.wcount[w][0];
      before += w < warp ? cw : 0;
      nlead += cw;
    }
    const int mycall = before + __popc(bal & (lane == 31 ? 0xffffffffu : (2u << lane) - 1u)) - 1;
    if (leads) S.lead[mycall] = my.call | (cls == 0 ? 1 << 30 : 0);
    __syncthreads();
    // 2. per call, the block's FOs with near points in the CTA's box
    for (int u = warp; u < nlead; u += NEAR_WARPS) {
      const int cc = S.lead[u];
      const bool allnear = cc >> 30;
      const CallFO* cf = J.cfo + (size_t)(cc & ((1 << 30) - 1)) * J.nfo + k0;
      int n1 = 0;
#pragma unroll
      for (int kb = 0; kb < FOB; kb += 32) {
        const int k = kb + lane;
        bool on = k < nk;
        if (on && !allnear) {
          const CallFO& f = cf[k];
          on = f.npot == 1 || tile_class(clo, chi, f.cg[0], f.cg[1], f.cg[2], f.rcut2) != 1;
        }
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) S.list[u][n1 + __popc(m & ((1u << lane) - 1u))] = (uint8_t)k;
        n1 += __popc(m);
      }
      if (lane == 0) S.cnt[u] = n1;
    }
    __syncthreads();
    // 3. the queue: the pairs of the calls that keep an FO
    act = act && S.cnt[mycall] > 0;
    bal = __ballot_sync(0xffffffffu, act);
    const bool cut = act && my.last && !(S.lead[mycall] >> 30);
    int rows = act ? S.cnt[mycall] * (my.fmt - 2) + (cut ? (S.cnt[mycall] + 1) / 2 : 0) : 0;
    const int mine = rows;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, rows, o);
      if (lane >= o) rows += v;
    }
    if (lane == 31 && warp < NEAR_WIN / 32) {
      S.wcount[warp][0] = __popc(bal);
      S.wcount[warp][1] = rows;
    }
    __syncthreads();
    before = 0;
    int qn = 0, rbefore = 0, rtotal = 0;
#pragma unroll
    for (int w = 0; w < NEAR_WIN / 32; ++w) {
      const int cw = S.wcount[w][0], rw = S.wcount[w][1];
      before += w < warp ? cw : 0;
      rbefore += w < warp ? rw : 0;
      qn += cw;
      rtotal += rw;
    }
    if (act) {
      const int e = before + __popc(bal & ((1u << lane) - 1u));
      S.queue[e] = NearEntry{rbefore + rows - mine, my.call, my.pair, (uint8_t)mycall, (uint8_t)S.cnt[mycall],
                             (uint8_t)my.fmt,
                             (uint8_t)(my.first * NEAR_FIRST + my.last * NEAR_LAST + (cut ? NEAR_CUT : 0))};
      const PairGeo& g = J.pairs[my.pair];
      S.geo[e][0] = S.geo[e][3] = g.C[0];
      S.geo[e][1] = S.geo[e][4] = g.C[1];
      S.geo[e][2] = g.C[2];
      S.geo[e][5] = g.delta;
    }
    if (tid == 0) S.queue[qn].pre = rtotal;
    __syncthreads();
    // 4. chunks of at most 32 entries whose rows fill a buffer
    auto chunk_end = [&](int e0) {
      int e = e0;
      while (e < qn && e - e0 < 32 && S.queue[e + 1].pre - S.queue[e0].pre <= NearSmem<MT>::ROWS) ++e;
      return e;
    };
    int e0 = 0, e1 = chunk_end(0), b = 0, fquad = -1;
    if (e1 > 0) copy(0, e1, 0);
    while (e0 < qn) {
      const int e2 = chunk_end(e1);
      cp_async_wait_all();
      __syncthreads();  // this chunk has arrived and the other buffer is free
      if (e1 < qn) copy(e1, e2, b ^ 1);
      if (npt > 0) {
        int wc = 1;
        if (lane < e1 - e0) {
          const double lo[3] = {box[0], box[1], box[2]}, hi[3] = {box[3], box[4], box[5]};
          wc = bound_class(lo, hi, J.bound[S.queue[e0 + lane].call]);
        }
        const double* A = S.A[b] - S.queue[e0].pre * 16;
        unsigned todo = __ballot_sync(0xffffffffu, wc != 1);
        const unsigned full = __ballot_sync(0xffffffffu, wc == 0);
        while (todo) {
          const int i = __ffs(todo) - 1, e = e0 + i;
          todo &= todo - 1;
          const NearEntry w = S.queue[e];
          const int nl = w.nl, nmt = (nl + 7) >> 3;
          const double* Ae = A + w.pre * 16;
          if (w.flags & NEAR_FIRST) np = 0;
          ++np;
          if ((e >> 2) != fquad) {
            // Boys values of four pairs at once: lane residue q takes pair 4 fquad + q
            fquad = e >> 2;
            const int eq = min(4 * fquad + q, qn - 1);
            const double* gq = S.geo[eq];
            const double* pp = pts[n];
            const PT arg = near_arg<PT>(PT(gq[5]), PT(pp[0] - gq[0]), PT(pp[1] - gq[1]), PT(pp[2] - gq[2]));
            PT ex;
            if constexpr (MIXED) ex = expf(-arg);
            else ex = exp(-arg);
            near_boys<PT>(tab, arg, ex, S.queue[eq].fmt, Fq);
          }
          const double* gq = S.geo[e] + cyc;
          const NearLane<PT> L(PT(pa - gq[0]), PT(pb_ - gq[1]), PT(pc - gq[2]));
          const int src = (lane & 28) | (e & 3);
          PT F[5];
#pragma unroll
          for (int j = 0; j < 3; ++j) F[j] = __shfl_sync(0xffffffffu, Fq[j], src);
          const double *A0 = Ae + piece, *A1 = Ae + (piece ^ 8);
          near_mma<MT, PT, 0>(T, A0, A1, nmt, L, F, q == 0);
          if (w.fmt >= 4) {
            F[3] = __shfl_sync(0xffffffffu, Fq[3], src);
            near_mma<MT, PT, 1>(T, A0 + nl * 16, A1 + nl * 16, nmt, L, F, q == 0);
          }
          if (w.fmt >= 5) {
            F[4] = __shfl_sync(0xffffffffu, Fq[4], src);
            near_mma<MT, PT, 2>(T, A0 + 2 * nl * 16, A1 + 2 * nl * 16, nmt, L, F, q == 0);
          }
          if (!(w.flags & NEAR_LAST)) continue;
          // the call's sum goes to V (call by call, so that no sum depends on how
          // FOs are blocked); a point counts for an FO when it is inside the FO's sphere
          const uint8_t* list = S.list[w.lead];
          const CallFO* sph = reinterpret_cast<const CallFO*>(Ae + (w.fmt - 2) * nl * 16);
          const bool isfull = (full >> i) & 1u;  // then every FO is listed
          const double *p0 = pts[2 * q], *p1 = pts[2 * q + 1];
          if (isfull && lane == 0) near += (unsigned long long)(nk * npt) * np;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            if (mt >= nmt) break;
            const int s = mt * 8 + n;
            if (s < nl) {
              bool n0 = true, n1 = true;  // points past the end: never stored
              if (!isfull) {
                const CallFO& f = sph[s];
                const double cx = f.cg[0], cy = f.cg[1], cz = f.cg[2], rc2 = f.rcut2;
                n0 = 2 * q < npt && !(sqdist_rn2(p0[0], p0[1], p0[2], cx, cy, cz) > rc2);
                n1 = 2 * q + 1 < npt && !(sqdist_rn2(p1[0], p1[1], p1[2], cx, cy, cz) > rc2);
                near += (unsigned)(((int)n0 + (int)n1) * np);
              }
              double2* ch = reinterpret_cast<double2*>(V + (int)list[s] * NEAR_PTS + 2 * q);
              double2 v = *ch;
              if (n0) v.x += T[mt][0];
              if (n1) v.y += T[mt][1];
              *ch = v;
            }
            T[mt][0] = T[mt][1] = 0.0;
          }
        }
      }
      e0 = e1;
      e1 = e2;
      b ^= 1;
    }
  }
  if (npt > 0) {
    __syncwarp();
    for (int e = lane; e < nk * NEAR_PTS; e += 32) {
      const int k = e / NEAR_PTS, p = e - k * NEAR_PTS;
      if (p >= npt) continue;
      if (J.nseg > 1) J.seg[((size_t)part * J.nfo + k0 + k) * J.ldv + pb + p] = V[e];
      else J.vh[(size_t)(k0 + k) * J.ldv + pb + p] += V[e];
    }
    count_add(J.cnt_perfo, near, 0, 0);
  }
}

// resident CTAs per SM the registers are limited for
template <int MT>
constexpr int near_ctas() { return MT <= 8 ? 2 : 1; }

template <int MT, bool MIXED>
__global__ void __launch_bounds__(NEAR_THREADS, near_ctas<MT>())
k_perfo_near(const __grid_constant__ CoulombJob J, const double* __restrict__ tab) {
  near_block<MT, MIXED>(J, blockIdx.x, blockIdx.y, blockIdx.z, tab);
}

// Many (molecule, spin) jobs: items[i] = {job, 128-point tile, FO block, 0}; blockIdx.y: part.
template <int MT, bool MIXED>
__global__ void __launch_bounds__(NEAR_THREADS, near_ctas<MT>())
k_perfo_near_batch(const CoulombJob* __restrict__ jobs, const int4* __restrict__ items,
                   const double* __restrict__ tab) {
  __shared__ CoulombJob J;
  const int4 w = items[blockIdx.x / NEAR_PER_TILE];
  if (threadIdx.x == 0) J = jobs[w.x];
  __syncthreads();
  if ((int)blockIdx.y >= J.nseg) return;
  near_block<MT, MIXED>(J, w.y * NEAR_PER_TILE + blockIdx.x % NEAR_PER_TILE, w.z, blockIdx.y, tab);
}

// ---------------------------------------------------------------------------
// Far field
// ---------------------------------------------------------------------------
// Potential of one FO at one point, sum_lm MV[lm] Y_lm(u) / r^(l+1), degree LMX
// at compile time.
//
// FP64: Clenshaw sums.  With w = d / r^2 and s = 1/r^2 the terms are solid
// harmonics of w over r; per order m, Q_l = z Q_{l-1} - c_lm s Q_{l-2} once the
// moments carry the recursion's leading factors (k_perfo_pack_mom), so a term
// costs two fused multiply-adds instead of the four operations of forming the
// harmonic and adding it (131 against ~250 FP64 operations at LMX = 6).
// Moments: mv[l] for m = 0, then per m the (cos, sin) pairs of l = m..6.
__host__ __device__ constexpr int far_pos(int l, int m) { return m == 0 ? l : 8 + 2 * ((m - 1) * 6 - (m - 1) * (m - 2) / 2 + l - m); }
// c_lm = B_lm / (A_lm A_{l-1,m}), A = (2l-1)/(l-m), B = (l+m-1)/(l-m)
__host__ __device__ constexpr double far_c(int l, int m) {
  return (double)((l + m - 1) * (l - 1 - m)) / (double)((2 * l - 1) * (2 * l - 3));
}

template <int LMX>
__device__ __forceinline__ double far_sum(const double* __restrict__ mv, double wx, double wy, double wz, double s) {
  double pot;
  {
    double b1 = mv[LMX], b2 = 0.0;
#pragma unroll
    for (int l = LMX - 1; l >= 0; --l) {
      double b = fma(wz, b1, mv[l]);
      if (l + 2 <= LMX) b = fma(-far_c(l + 2, 0) * s, b2, b);
      b2 = b1;
      b1 = b;
    }
    pot = b1;
  }
  double c = wx, t = wy;
#pragma unroll
  for (int m = 1; m <= LMX; ++m) {
    const double2 top = *reinterpret_cast<const double2*>(mv + far_pos(LMX, m));
    double b1 = top.x, b2 = 0.0, d1 = top.y, d2 = 0.0;
#pragma unroll
    for (int l = LMX - 1; l >= m; --l) {
      const double2 a = *reinterpret_cast<const double2*>(mv + far_pos(l, m));
      double b = fma(wz, b1, a.x), d = fma(wz, d1, a.y);
      if (l + 2 <= LMX) {
        const double cs = -far_c(l + 2, m) * s;
        b = fma(cs, b2, b);
        d = fma(cs, d2, d);
      }
      b2 = b1;
      b1 = b;
      d2 = d1;
      d1 = d;
    }
    pot = fma(c, b1, pot);
    pot = fma(t, d1, pot);
    const double nc = c * wx - t * wy;
    t = c * wy + t * wx;
    c = nc;
  }
  return pot;
}

// FP32: the harmonics of harmonics.f, summed per degree and scaled once per degree.
template <int LMX>
__device__ __forceinline__ float far_sum(const float* __restrict__ mv, float ux, float uy, float uz, float hn) {
  float acc[LMX + 1];
#pragma unroll
  for (int l = 0; l <= LMX; ++l) acc[l] = 0.f;
  harmonics_mmajor(ux, uy, uz, LMX, [&](int row, int l, float v) { acc[l] += mv[row] * v; });
  float pot = 0.f, rec = hn;
#pragma unroll
  for (int l = 0; l <= LMX; ++l) {
    pot += acc[l] * rec;
    rec *= hn;
  }
  return pot;
}

// Brings the moments of the per-FO calls into the form k_perfo_far reads, in place,
// rows of MOM_LD doubles: in FP64 times the leading factors of far_sum's recursion,
// prod_{i=m+1..l} (2i-1)/(i-m) and prod_{i=2..m} (2i-1), in its order; in the mixed
// path rounded to FP32 in the order of the moments (MOM_LD floats, then unused space).
__global__ void __launch_bounds__(64) k_perfo_pack_mom(int nfo, int mixed, int per_fo_only,
                                                       const CallShare* __restrict__ share,
                                                       double* __restrict__ momv) {
  const int c = blockIdx.x, j = threadIdx.x;
  if (!per_fo_only && share[c].shared) return;
  int pos = j;
  double f = j < NMOM ? 1.0 : 0.0;
  if (!mixed && j < NMOM) {
    int l = 0;
    while ((l + 1) * (l + 1) <= j) ++l;
    const int m = (j - l * l + 1) / 2;
    pos = far_pos(l, m) + (m > 0 && j == l * l + 2 * m);
    for (int i = m + 1; i <= l; ++i) f *= (double)(2 * i - 1) / (double)(i - m);
    for (int i = 2; i <= m; ++i) f *= (double)(2 * i - 1);
  } else if (!mixed) {
    pos = j == NMOM ? 7 : j;  // the positions far_pos leaves out
  }
  for (int k = blockIdx.y; k < nfo; k += gridDim.y) {
    double* row = momv + ((size_t)c * nfo + k) * MOM_LD;
    const double v = j < NMOM ? row[j] * f : 0.0;
    __syncthreads();
    if (j >= MOM_LD) continue;
    if (mixed) reinterpret_cast<float*>(row)[j] = (float)v;
    else row[pos] = v;
  }
}

constexpr int FAR_FOS = 4;             // FOs per CTA (1 for one density): a warp has one FO and 64 points, two per lane
constexpr int far_threads(int fos) { return 2 * 32 * fos; }
constexpr int FAR_CALLS = 8;           // calls per buffer
static_assert(sizeof(CallFO) == 64 && MOM_LD % 4 == 0, "copied in 16-byte pieces");
static_assert(far_pos(6, 6) + 1 < MOM_LD, "moment positions");

template <int FOS, bool MIXED>
struct FarSmem {
  using PT = typename std::conditional<MIXED, float, double>::type;
  CallFO f[2][FAR_CALLS][FOS];
  PT mv[2][FAR_CALLS][FOS][MOM_LD];
  double box[far_threads(FOS) / 32 + 1][6];
  int queue[far_threads(FOS)];
  int wcount[far_threads(FOS) / 32];
};

template <int FOS, bool MIXED>
__device__ __forceinline__ void far_block(const CoulombJob& J, int tile, int grp, int part) {
  using PT = typename std::conditional<MIXED, float, double>::type;
  __shared__ __align__(16) FarSmem<FOS, MIXED> S;
  constexpr int NT = far_threads(FOS), NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k0 = grp * FOS, nk = min(FOS, J.nfo - k0);
  const int p0 = tile * TILE, npt = min(TILE, J.M.n - p0);
  const int* list = J.lists + J.ncalls;
  const int ncall = J.lists[2 * J.ncalls + 1];
  if (ncall == 0) return;
  const int first = (int)((long long)ncall * part / J.nseg), nl = (int)((long long)ncall * (part + 1) / J.nseg);
  const int k = warp >> 1;                       // this warp's FO
  const int pl = (warp & 1) * 64 + lane;         // and points pl, pl + 32
  double x[2], y[2], z[2], V[2] = {0.0, 0.0};
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int p = p0 + min(pl + 32 * j, npt - 1);
    x[j] = J.M.x[p];
    y[j] = J.M.y[p];
    z[j] = J.M.z[p];
  }
  {
    double lo[3], hi[3], lo1[3], hi1[3];
    warp_box(x[0], y[0], z[0], lo, hi);
    warp_box(x[1], y[1], z[1], lo1, hi1);
    if (lane == 0)
      for (int d = 0; d < 3; ++d) {
        S.box[warp][d] = fmin(lo[d], lo1[d]);
        S.box[warp][3 + d] = fmax(hi[d], hi1[d]);
      }
  }
  __syncthreads();
  if (tid < 6) {
    double v = S.box[0][tid];
    for (int w = 1; w < NW; ++w) v = tid < 3 ? fmin(v, S.box[w][tid]) : fmax(v, S.box[w][tid]);
    S.box[NW][tid] = v;
  }
  __syncthreads();
  unsigned long long far = 0, terms = 0;
  auto copy = [&](int e0, int e1, int b) {
    constexpr int MP = MOM_LD * sizeof(PT) / 16;  // 16-byte pieces of one FO's moments
    const int per = nk * (MP + 4);
    for (int e = tid; e < (e1 - e0) * per; e += NT) {
      const int i = e / per, r = e - i * per;
      const size_t ck = (size_t)S.queue[e0 + i] * J.nfo + k0;
      if (r < nk * MP) {
        const int kk = r / MP, o = r - kk * MP;
        cp_async16(reinterpret_cast<char*>(S.mv[b][i][kk]) + 16 * o,
                   reinterpret_cast<const char*>(J.momv + (ck + kk) * MOM_LD) + 16 * o);
      } else {
        cp_async16(reinterpret_cast<char*>(S.f[b][i]) + 16 * (r - nk * MP),
                   reinterpret_cast<const char*>(J.cfo + ck) + 16 * (r - nk * MP));
      }
    }
    cp_async_commit();
  };
  for (int l0 = first; l0 < nl; l0 += NT) {
    // the window's calls with far points in the tile, in order
    bool act = false;
    int c = 0;
    if (l0 + tid < nl) {
      c = list[l0 + tid];
      const double* bx = S.box[NW];
      const double lo[3] = {bx[0], bx[1], bx[2]}, hi[3] = {bx[3], bx[4], bx[5]};
      const CallBound& b = J.bound[c];
      act = tile_class(lo, hi, b.c[0], b.c[1], b.c[2], b.rin2) != 0;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, act);
    if (lane == 0) S.wcount[warp] = __popc(bal);
    __syncthreads();  // and every warp is done with the previous window
    int before = 0, qn = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const int cw = S.wcount[w];
      before += w < warp ? cw : 0;
      qn += cw;
    }
    if (act) S.queue[before + __popc(bal & ((1u << lane) - 1u))] = c;
    __syncthreads();
    if (qn > 0) copy(0, min(FAR_CALLS, qn), 0);
    for (int e0 = 0, b = 0; e0 < qn; e0 += FAR_CALLS, b ^= 1) {
      const int ne = min(FAR_CALLS, qn - e0);
      cp_async_wait_all();
      __syncthreads();  // this chunk has arrived and the other buffer is free
      if (e0 + FAR_CALLS < qn) copy(e0 + FAR_CALLS, min(e0 + 2 * FAR_CALLS, qn), b ^ 1);
      if (k >= nk) continue;
#pragma unroll 1
      for (int i = 0; i < ne; ++i) {
        const CallFO& f = S.f[b][i][k];
        if (f.npot == 1) continue;
        const double cx = f.cg[0], cy = f.cg[1], cz = f.cg[2], rc2 = f.rcut2;
        double r2[2];
        bool isfar[2];
        int nf = 0;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          r2[j] = sqdist_rn2(x[j], y[j], z[j], cx, cy, cz);
          isfar[j] = pl + 32 * j < npt && r2[j] > rc2;
          nf += __popc(__ballot_sync(0xffffffffu, isfar[j]));
        }
        if (nf == 0) continue;
        const PT* mv = S.mv[b][i][k];
        PT a[2][4], pot[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const PT dx = PT(x[j] - cx), dy = PT(y[j] - cy), dz = PT(z[j] - cz);
          if constexpr (MIXED) {
            const float hn = rsqrtf(isfar[j] ? (float)r2[j] : 1.f);
            a[j][0] = hn * dx;
            a[j][1] = hn * dy;
            a[j][2] = hn * dz;
            a[j][3] = hn;
          } else {
            const double hn = rsqrt(isfar[j] ? r2[j] : 1.0), s = hn * hn;
            a[j][0] = s * dx;
            a[j][1] = s * dy;
            a[j][2] = s * dz;
            a[j][3] = s;
            r2[j] = hn;
          }
        }
        switch (f.lmax) {
#define FAR_CASE(L)                                                              \
  {                                                                              \
    pot[0] = far_sum<L>(mv, a[0][0], a[0][1], a[0][2], a[0][3]);                 \
    pot[1] = far_sum<L>(mv, a[1][0], a[1][1], a[1][2], a[1][3]);                 \
    break;                                                                       \
  }
          case 0: FAR_CASE(0)
          case 1: FAR_CASE(1)
          case 2: FAR_CASE(2)
          case 3: FAR_CASE(3)
          case 4: FAR_CASE(4)
          case 5: FAR_CASE(5)
          default: FAR_CASE(6)
#undef FAR_CASE
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          double v;
          if constexpr (MIXED) v = (double)pot[j];
          else v = r2[j] * pot[j];
          if (isfar[j]) V[j] += v;
        }
        if (lane == 0) {
          far += (unsigned long long)nf;
          terms += (unsigned long long)nf * (unsigned long long)__popcll(f.keep);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (k < nk && pl + 32 * j < npt) {
      const int p = p0 + pl + 32 * j;
      J.seg[((size_t)(perfo_near_parts(J.nseg) + part) * J.nfo + k0 + k) * J.ldv + p] = V[j];
    }
  count_add(J.cnt_perfo, 0, far, terms);
}

// Three CTAs per SM in FP32 (80 registers; benzene beside the near field 22.9 -> 21.6
// ms); in FP64 that limit spills and slows both fields (24.8 -> 31.4 ms).
template <int FOS, bool MIXED>
__global__ void __launch_bounds__(far_threads(FOS), MIXED ? 3 : 2) k_perfo_far(const __grid_constant__ CoulombJob J) {
  far_block<FOS, MIXED>(J, blockIdx.x, blockIdx.y, blockIdx.z);
}

// items[i] = {job, tile, FO block of fob FOs, 0}; blockIdx.y: group of FAR_FOS FOs of the block,
// blockIdx.z: part.
template <bool MIXED>
__global__ void __launch_bounds__(far_threads(FAR_FOS), MIXED ? 3 : 2)
k_perfo_far_batch(const CoulombJob* __restrict__ jobs, const int4* __restrict__ items, int fob) {
  __shared__ CoulombJob J;
  const int4 w = items[blockIdx.x];
  if (threadIdx.x == 0) J = jobs[w.x];
  __syncthreads();
  const int grp = w.z * (fob / FAR_FOS) + blockIdx.y;
  if (grp * FAR_FOS >= J.nfo || (int)blockIdx.z >= J.nseg) return;
  far_block<FAR_FOS, MIXED>(J, w.y, grp, blockIdx.z);
}

// vh += the parts' sums in order: near parts (one part has been added already),
// then far parts.  FOs [k0, k0 + nk) of one tile.
__device__ __forceinline__ void add_parts(const CoulombJob& J, int tile, int k0, int nk) {
  if (J.lists[2 * J.ncalls + 1] == 0) return;
  const int parts = perfo_near_parts(J.nseg) + J.nseg;
  const int p = tile * TILE + (int)threadIdx.x;
  if (threadIdx.x >= TILE || p >= J.M.n) return;
  for (int k = k0; k < k0 + nk; ++k) {
    double v = 0.0;
    for (int s = 0; s < parts; ++s) v += J.seg[((size_t)s * J.nfo + k) * J.ldv + p];
    J.vh[(size_t)k * J.ldv + p] += v;
  }
}
__global__ void __launch_bounds__(TILE) k_perfo_add(const __grid_constant__ CoulombJob J) {
  add_parts(J, blockIdx.x, blockIdx.y, 1);
}
__global__ void __launch_bounds__(TILE) k_perfo_add_batch(const CoulombJob* __restrict__ jobs,
                                                          const int4* __restrict__ items, int fob) {
  const int4 w = items[blockIdx.x];
  __shared__ CoulombJob J;
  if (threadIdx.x == 0) J = jobs[w.x];
  __syncthreads();
  add_parts(J, w.y, w.z * fob, min(fob, J.nfo - w.z * fob));
}

// ---------------------------------------------------------------------------
// One density
// ---------------------------------------------------------------------------
// Near field of one density (COUPOT1): with a single row the tensor cores would
// multiply seven rows of padding, so each thread evaluates the pairs at its own
// point from coefficient rows staged in shared memory, and the pair list is cut
// into parts until the chip is full.  ~200 FP64 operations per (pair, point).
// C60 (17,520 points, 53,460 pairs, 19,020 calls), whole evaluation: 84 ms with
// the shared-geometry kernel (137 CTAs, each walking every pair), now near 3.8 and far 2.1 ms.
constexpr int ONE_CHUNK = 16;  // pairs per buffer

__global__ void __launch_bounds__(TILE) k_one_near(const __grid_constant__ CoulombJob J,
                                                   const double* __restrict__ tab) {
  __shared__ __align__(16) double A[2][ONE_CHUNK][COEF_LD];
  __shared__ double geo[TILE][4], sph[TILE][4];
  __shared__ PerfoPair queue[TILE];
  __shared__ double box[TILE / 32 + 1][6];
  __shared__ int wcount[TILE / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = blockIdx.y;
  const int p0 = blockIdx.x * TILE, npt = min(TILE, J.M.n - p0);
  const int npairs = J.lists[2 * J.ncalls + 2];
  const int pl0 = (int)((long long)npairs * part / J.nseg), npl = (int)((long long)npairs * (part + 1) / J.nseg);
  const int p = p0 + min(tid, npt - 1);
  const double x = J.M.x[p], y = J.M.y[p], z = J.M.z[p];
  {
    double lo[3], hi[3];
    warp_box(x, y, z, lo, hi);
    if (lane == 0)
      for (int d = 0; d < 3; ++d) {
        box[warp][d] = lo[d];
        box[warp][3 + d] = hi[d];
      }
  }
  __syncthreads();
  double clo[3], chi[3];
  for (int d = 0; d < 3; ++d) {
    clo[d] = box[0][d];
    chi[d] = box[0][3 + d];
    for (int w = 1; w < TILE / 32; ++w) {
      clo[d] = fmin(clo[d], box[w][d]);
      chi[d] = fmax(chi[d], box[w][3 + d]);
    }
  }
  double V = 0.0;
  unsigned long long near = 0;
  for (int w0 = pl0; w0 < npl; w0 += TILE) {
    bool act = false;
    PerfoPair my{};
    if (w0 + tid < npl) {
      my = J.plist[w0 + tid];
      act = bound_class(clo, chi, J.bound[my.call]) != 1;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, act);
    if (lane == 0) wcount[warp] = __popc(bal);
    __syncthreads();  // and every thread is done with the previous window
    int before = 0, qn = 0;
#pragma unroll
    for (int w = 0; w < TILE / 32; ++w) {
      const int cw = wcount[w];
      before += w < warp ? cw : 0;
      qn += cw;
    }
    if (act) {
      const int e = before + __popc(bal & ((1u << lane) - 1u));
      queue[e] = my;
      const PairGeo& g = J.pairs[my.pair];
      geo[e][0] = g.C[0];
      geo[e][1] = g.C[1];
      geo[e][2] = g.C[2];
      geo[e][3] = g.delta;
      const CallFO& f = J.cfo[my.call];
      sph[e][0] = f.cg[0];
      sph[e][1] = f.cg[1];
      sph[e][2] = f.cg[2];
      sph[e][3] = f.rcut2;
    }
    __syncthreads();
    auto copy = [&](int e0, int b) {
      const int ne = min(ONE_CHUNK, qn - e0);
      for (int i = tid; i < ne * (COEF_LD / 2); i += TILE) {
        const int e = i / (COEF_LD / 2), o = i - e * (COEF_LD / 2);
        cp_async16(&A[b][e][2 * o], J.coef + (size_t)queue[e0 + e].pair * COEF_LD + 2 * o);
      }
      cp_async_commit();
    };
    if (qn > 0) copy(0, 0);
    for (int e0 = 0, b = 0; e0 < qn; e0 += ONE_CHUNK, b ^= 1) {
      cp_async_wait_all();
      __syncthreads();  // this chunk has arrived and the other buffer is free
      if (e0 + ONE_CHUNK < qn) copy(e0 + ONE_CHUNK, b ^ 1);
      const int ne = min(ONE_CHUNK, qn - e0);
      for (int i = 0; i < ne; ++i) {
        const double* s = sph[e0 + i];
        const bool nr = tid < npt && !(sqdist_rn2(x, y, z, s[0], s[1], s[2]) > s[3]);
        if (!__any_sync(0xffffffffu, nr)) continue;
        const double* g = geo[e0 + i];
        const int fmt = queue[e0 + i].fmt;
        const double rx = x - g[0], ry = y - g[1], rz = z - g[2];
        const double arg = near_arg<double>(g[3], rx, ry, rz);
        double F[5], mono[35];
        near_boys<double>(tab, arg, exp(-arg), fmt, F);
        monomials(rx, ry, rz, mono);
        const double v = pair_potential(A[b][i], mono, fmt, F, F, F);
        if (nr) {
          V += v;
          ++near;
        }
      }
    }
  }
  if (tid < npt) J.seg[(size_t)part * J.ldv + p0 + tid] = V;
  count_add(J.cnt_perfo, near, 0, 0);
}

// ---------------------------------------------------------------------------
// Launches
// ---------------------------------------------------------------------------
template <int MT>
static cudaError_t near_attr() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* f) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(NearSmem<MT>));
  };
  set(k_perfo_near<MT, false>);
  set(k_perfo_near<MT, true>);
  set(k_perfo_near_batch<MT, false>);
  set(k_perfo_near_batch<MT, true>);
  return e;
}

cudaError_t init_coulomb_perfo() {
  cudaError_t e = near_attr<4>();
  if (e == cudaSuccess) e = near_attr<8>();
  if (e == cudaSuccess) e = near_attr<16>();
  return e;
}

int launch_perfo_setup(int ncalls, int npairs, int nfo, const CallInfo* calls, const PairGeo* pairs,
                       const CallFO* cfo, const CallShare* share, bool per_fo_only, bool mixed, bool one_density,
                       double* coef, double* momv, CallBound* bound, cudaStream_t st) {
  if (ncalls <= 0 || npairs <= 0) return 0;
  k_perfo_bounds<<<(ncalls + 7) / 8, 256, 0, st>>>(ncalls, nfo, calls, pairs, cfo, bound);
  if (!one_density)  // k_one_near reads the coefficients in their first order
    k_perfo_pack<<<npairs, 256, 0, st>>>(nfo, pairs, share, per_fo_only ? 1 : 0, coef);
  k_perfo_pack_mom<<<dim3(ncalls, std::min(nfo, 32)), 64, 0, st>>>(nfo, mixed ? 1 : 0, per_fo_only ? 1 : 0, share, momv);
  return one_density ? 2 : 3;
}

template <int MT>
static void launch_near(const CoulombJob& J, bool mixed, const double* tab, cudaStream_t st) {
  const dim3 grid(J.M.ntiles * NEAR_PER_TILE, (J.nfo + 8 * MT - 1) / (8 * MT), J.nseg);
  if (mixed) k_perfo_near<MT, true><<<grid, NEAR_THREADS, sizeof(NearSmem<MT>), st>>>(J, tab);
  else k_perfo_near<MT, false><<<grid, NEAR_THREADS, sizeof(NearSmem<MT>), st>>>(J, tab);
}

// The near field starts on st, the far field on the side stream: its small CTAs
// fill the SMs as the near field's uneven ones end (benzene, 296 tiles: 28.6 ->
// 24.7 ms both).
int launch_perfo(const CoulombJob& J, int wm, bool mixed, const double* tab, const SideStream& side,
                 cudaStream_t st) {
  if (J.M.ntiles <= 0 || J.nfo <= 0) return 0;
  cudaEventRecord(side.fork, st);
  cudaStreamWaitEvent(side.st, side.fork, 0);
  if (wm == 4) launch_near<16>(J, mixed, tab, st);
  else if (wm == 2) launch_near<8>(J, mixed, tab, st);
  else launch_near<4>(J, mixed, tab, st);
  const dim3 grid(J.M.ntiles, (J.nfo + FAR_FOS - 1) / FAR_FOS, J.nseg);
  if (mixed) k_perfo_far<FAR_FOS, true><<<grid, far_threads(FAR_FOS), 0, side.st>>>(J);
  else k_perfo_far<FAR_FOS, false><<<grid, far_threads(FAR_FOS), 0, side.st>>>(J);
  cudaEventRecord(side.join, side.st);
  cudaStreamWaitEvent(st, side.join, 0);
  k_perfo_add<<<dim3(J.M.ntiles, J.nfo), TILE, 0, st>>>(J);
  return 3;
}

// Enough CTAs for eight per SM, from the mesh alone (a short pair list leaves some of
// the parts without a pair).
int one_density_parts(int ntiles) { return std::max(2, std::min(32, 8 * 148 / std::max(ntiles, 1))); }

int launch_one_density(const CoulombJob& J, const double* tab, cudaStream_t st) {
  if (J.M.ntiles <= 0) return 0;
  k_perfo_far<1, false><<<dim3(J.M.ntiles, 1, J.nseg), far_threads(1), 0, st>>>(J);
  k_one_near<<<dim3(J.M.ntiles, J.nseg), TILE, 0, st>>>(J, tab);
  k_perfo_add<<<dim3(J.M.ntiles, 1), TILE, 0, st>>>(J);
  return 3;
}

template <int MT>
static void launch_near_batch(const CoulombJob* jobs, const int4* items, int nitems, int parts, bool mixed,
                              const double* tab, cudaStream_t st) {
  const dim3 grid(nitems * NEAR_PER_TILE, parts);
  if (mixed) k_perfo_near_batch<MT, true><<<grid, NEAR_THREADS, sizeof(NearSmem<MT>), st>>>(jobs, items, tab);
  else k_perfo_near_batch<MT, false><<<grid, NEAR_THREADS, sizeof(NearSmem<MT>), st>>>(jobs, items, tab);
}

int launch_perfo_batch(const CoulombJob* jobs, const int4* items, int nitems, int parts, int wm, bool mixed,
                       const double* tab, cudaStream_t st) {
  if (nitems <= 0) return 0;
  const dim3 grid(nitems, 32 * wm / FAR_FOS, parts);
  if (mixed) k_perfo_far_batch<true><<<grid, far_threads(FAR_FOS), 0, st>>>(jobs, items, 32 * wm);
  else k_perfo_far_batch<false><<<grid, far_threads(FAR_FOS), 0, st>>>(jobs, items, 32 * wm);
  if (wm == 4) launch_near_batch<16>(jobs, items, nitems, parts, mixed, tab, st);
  else if (wm == 2) launch_near_batch<8>(jobs, items, nitems, parts, mixed, tab, st);
  else launch_near_batch<4>(jobs, items, nitems, parts, mixed, tab, st);
  k_perfo_add_batch<<<nitems, TILE, 0, st>>>(jobs, items, 32 * wm);
  return 3;
}

}  // namespace flosic
