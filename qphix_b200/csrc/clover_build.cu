// Clover term construction and inversion on the device.
//
// QPhiX takes the clover term and its inverse as inputs (its callers build
// them with Chroma's QDPCloverTerm); these kernels produce the same packed
// arrays on the GPU from a resident gauge field, so that a solve never has to
// leave the device:
//   clover_build   A = diag_mass + sigma.F in the clover-leaf normalisation
//                  of tests/mesfield.cc:25-64 (F = (Q - Q^+)/8, Q the four
//                  plaquette leaves) and the packing of
//                  tests/clover_term_qdp_w.h:114-200,325-442 (coefficients
//                  x 1/2), two 6x6 Hermitian blocks (diag[6], offd[15])
//   clover_invert  packed A^-1 (exact 6x6 inverse per block)
//   clover_invert_twisted  full (A + i mu g5)^-1 and (A - i mu g5)^-1 for
//                  the twisted-mass clover operator (g5 = +1 on block 0)
//   clover_invert_ndtm  the inverse of the two-flavour diagonal block
//                  [[A + i mu g5, -eps], [-eps, A - i mu g5]]: with
//                  Q = (A^2 + mu^2 - eps^2)^-1 (A commutes with g5) it is
//                  [[Q (A - i mu g5), eps Q], [eps Q, Q (A + i mu g5)]]; the
//                  flavour-diagonal blocks as full clover fields, eps Q packed
//                  (the fields include/qphix/ndtm_reuse_operator_clover.h:38-50
//                   takes, tm_clov_dslash_def.h:96-104)
// All arithmetic in FP64; results are stored in the destination field's
// precision.
#include "qpx_finalize.cuh"
#include "qpx_host.h"

namespace qpx {

typedef cx<double> zd;

struct M3 {
  zd m[3][3];
};

__device__ __forceinline__ M3 mm(const M3 &a, const M3 &b)
{
  M3 c;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      c.m[i][j] = cmad(a.m[i][2], b.m[2][j], cmad(a.m[i][1], b.m[1][j], cmul(a.m[i][0], b.m[0][j])));
  return c;
}

__device__ __forceinline__ M3 dag(const M3 &a)
{
  M3 c;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) c.m[i][j] = conj(a.m[j][i]);
  return c;
}

__device__ __forceinline__ M3 minus(const M3 &a, const M3 &b)
{
  M3 c;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) c.m[i][j] = a.m[i][j] - b.m[i][j];
  return c;
}

// U_dir at x + a mu + b nu, a and b in {-1, 0, 1}
template <int RECON>
__device__ __forceinline__ M3 link_at(const GaugeArg &g, const Geom &geo, const int x[4], int mu, int a, int nu, int b,
                                      int dir)
{
  const int n[4] = {geo.nx, geo.ny, geo.nz, geo.nt};
  int c[4];
#pragma unroll
  for (int d = 0; d < 4; d++) {
    c[d] = x[d] + (d == mu ? a : 0) + (d == nu ? b : 0);
    c[d] += c[d] < 0 ? n[d] : (c[d] >= n[d] ? -n[d] : 0);
  }
  const int cb = (c[0] + c[1] + c[2] + c[3]) & 1;
  const int s = ((c[3] * geo.nz + c[2]) * geo.ny + c[1]) * geo.nxh + (c[0] >> 1);
  M3 u;
  GaugeIO<F64, RECON>::load(g, cb, dir, s, u.m);
  return u;
}

// reals k, k + 1 of a site (k even: one chunk holds both, every chunk length is even)
template <typename Q>
__device__ __forceinline__ void dev_store_pair(void *base, long long stride, int vpc, int s, int k, double v0, double v1)
{
  const long long e = ((long long)(k / vpc) * stride + s) * vpc + k % vpc;
  if constexpr (Q::prec == PREC_F64) {
    *reinterpret_cast<double2 *>(reinterpret_cast<double *>(base) + e) = make_double2(v0, v1);
  } else if constexpr (Q::prec == PREC_F32) {
    *reinterpret_cast<float2 *>(reinterpret_cast<float *>(base) + e) = make_float2((float)v0, (float)v1);
  } else {
    const float v[2] = {(float)v0, (float)v1};
    *reinterpret_cast<uint32_t *>(reinterpret_cast<uint16_t *>(base) + e) = pack2(v, Q());
  }
}

// Clover leaf F and the packed term, a block per 32 sites: lane = site, one
// warp per plane (0,1),(0,2),(0,3),(1,2),(1,3),(2,3); the planes' F meet in
// shared memory, then the six warps share the packing.  Only the
// anti-Hermitian part of the leaf sum Q enters, so a leaf may be replaced by
// minus its adjoint, which lets pairs of leaves share a product:
//   Q - Q^+ = G - G^+,  G = U_mu(x) (S1 - S4) + (S2 - S3) U_mu(x-mu)
// with the two-link completions S of the four leaves: 10 products of 3 x 3
// matrices a plane instead of 12.
// What bounds it: the latency of the link loads and product chains at the
// occupancy the registers leave (24^3x48, 18-real links: FP64 pipe 22 % busy
// and 591 us at 182 registers and one block of 6 warps per multiprocessor;
// two blocks of at most 168 registers, with 52 bytes spilled, 364 us; the
// pipe's own time is 120 us).  One thread per site over all planes kept six
// F's, spilled to a 928-byte stack and took 666 us there; both checkerboards'
// terms and one inverse (below) went from 2254 to 927 us.
constexpr int kPlanes = 6, kLeafSites = 32;

template <int RECON, typename Q>
__global__ void __launch_bounds__(kPlanes *kLeafSites, 2)
    clover_build_kernel(Geom geo, GaugeArg g, void *out, long long stride, int vpc, int cb, double diag_mass,
                        double coeff_r, double coeff_t)
{
  __shared__ double f[kPlanes][9][kLeafSites];  // Im F_ii, then F_10, F_20, F_21
  const int lane = threadIdx.x & 31, plane = threadIdx.x >> 5;
  const int site = blockIdx.x * kLeafSites + lane;
  const int s = site < geo.vh ? site : geo.vh - 1;
  int xh, y, z, t, par;
  site_coords(geo, s, cb, xh, y, z, t, par);
  const int x[4] = {2 * xh + par, y, z, t};
  const int mu = plane < 3 ? 0 : (plane < 5 ? 1 : 2), nu = plane < 3 ? plane + 1 : (plane < 5 ? plane - 1 : 3);
#define AT(a, b, dir) link_at<RECON>(g, geo, x, mu, a, nu, b, dir)
  M3 q;
  {
    // U_mu(x) U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+ and the adjoint of U_nu(x-nu)^+ U_mu(x-nu) U_nu(x-nu+mu) U_mu(x)^+
    const M3 s1 = mm(mm(AT(1, 0, nu), dag(AT(0, 1, mu))), dag(AT(0, 0, nu)));
    const M3 s4 = mm(mm(dag(AT(1, -1, nu)), dag(AT(0, -1, mu))), AT(0, -1, nu));
    q = mm(AT(0, 0, mu), minus(s1, s4));
  }
  {
    // U_nu(x) U_mu(x-mu+nu)^+ U_nu(x-mu)^+ U_mu(x-mu) and the adjoint of
    // U_mu(x-mu)^+ U_nu(x-mu-nu)^+ U_mu(x-mu-nu) U_nu(x-nu)
    const M3 s2 = mm(mm(AT(0, 0, nu), dag(AT(-1, 1, mu))), dag(AT(-1, 0, nu)));
    const M3 s3 = mm(mm(dag(AT(0, -1, nu)), dag(AT(-1, -1, mu))), AT(-1, -1, nu));
    const M3 p = mm(minus(s2, s3), AT(-1, 0, mu));
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) q.m[i][j] = q.m[i][j] + p.m[i][j];
  }
#undef AT
  const double cf = 0.125 * (nu == 3 ? coeff_t : coeff_r);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    f[plane][i][lane] = cf * (q.m[i][i].im + q.m[i][i].im);
#pragma unroll
    for (int j = 0; j < i; j++) {
      const zd v = cf * (q.m[i][j] - conj(q.m[j][i]));
      f[plane][3 + 2 * (i + j - 1)][lane] = v.re;
      f[plane][4 + 2 * (i + j - 1)][lane] = v.im;
    }
  }
  __syncthreads();
  // F_ij of a plane; F is anti-Hermitian
  auto at = [&](int k, int i, int j) -> zd {
    if (i == j) return {0.0, f[k][i][lane]};
    const int o = 3 + 2 * (i + j - 1);
    const zd v = {f[k][o][lane], f[k][o + 1][lane]};
    return i > j ? v : zd{-v.re, v.im};
  };
  if (site >= geo.vh) return;
  // 36 pairs of reals: per block 3 of the diagonal and 15 complex numbers below it
  for (int e = plane; e < 36; e += kPlanes) {
    const int b = e / 18, o = e % 18 - 3;
    double v0, v1;
    if (o < 0) {
      auto diag = [&](int i) {
        const double r = b == 0 ? f[5][i % 3][lane] - f[0][i % 3][lane] : -(f[5][i % 3][lane] + f[0][i % 3][lane]);
        return i < 3 ? diag_mass + r : diag_mass - r;
      };
      v0 = diag(2 * (o + 3));
      v1 = diag(2 * (o + 3) + 1);
    } else {
      int i = 1;
      while ((i + 1) * i / 2 <= o) i++;
      const int j = o - i * (i - 1) / 2;
      zd v;
      if (i < 3 || j >= 3) {  // within a spin: +- i (F_xy -+ F_zt)
        const zd f0 = at(0, i % 3, j % 3), f5 = at(5, i % 3, j % 3);
        v = b == 0 ? itimes(f0 - f5) : itimes(f5 + f0);
        if (i >= 3) v = zd{-v.re, -v.im};
      } else {
        const zd em = itimes(at(2, i - 3, j)) + at(4, i - 3, j), bm = itimes(at(3, i - 3, j)) - at(1, i - 3, j);
        v = b == 0 ? bm - em : em + bm;
      }
      v0 = v.re;
      v1 = v.im;
    }
    dev_store_pair<Q>(out, stride, vpc, s, 36 * b + (o < 0 ? 2 * (o + 3) : 6 + 2 * o), v0, v1);
  }
}

// Gauss-Jordan inverse in place of a 6 x 6 complex matrix with partial
// pivoting, a thread per column: a[i] is row i of this thread's column
// `col`; the six columns of a site's block sit in six warps at the same lane.  In
// step c the owner of column c picks the pivot row, swaps it up and leaves
// its column, the pivot's reciprocal and the row in shared memory (two
// buffers, one barrier a step); every column then eliminates with it.
// Returns which column of the inverse this thread ends up with.
struct PivotBuf {
  double v[2][2][15][32];  // [buffer][block][6 complex, reciprocal, pivot row][lane]
};
// rows c and p >= c of a column exchanged, by selects: the column stays in registers
__device__ __forceinline__ void swap_rows(zd a[6], int c, int p)
{
  double re = a[c].re, im = a[c].im;
#pragma unroll
  for (int r = 1; r < 6; r++) {
    if (r <= c) continue;
    const bool hit = r == p;
    const double vr = a[r].re, vi = a[r].im;
    a[r].re = hit ? a[c].re : vr;
    a[r].im = hit ? a[c].im : vi;
    re = hit ? vr : re;
    im = hit ? vi : im;
  }
  a[c] = {re, im};
}
__device__ __forceinline__ int invert6(zd a[6], int col, int b, int lane, PivotBuf &buf)
{
  int dest = col;
  int piv[6];
#pragma unroll
  for (int c = 0; c < 6; c++) {
    double(*pb)[32] = buf.v[c & 1][b];
    if (col == c) {
      int p = c;
      double best = a[c].re * a[c].re + a[c].im * a[c].im;
#pragma unroll
      for (int r = c + 1; r < 6; r++) {
        const double v = a[r].re * a[r].re + a[r].im * a[r].im;
        if (v > best) {
          best = v;
          p = r;
        }
      }
      swap_rows(a, c, p);
#pragma unroll
      for (int r = 0; r < 6; r++) {
        pb[2 * r][lane] = a[r].re;
        pb[2 * r + 1][lane] = a[r].im;
      }
      pb[12][lane] = a[c].re / best;
      pb[13][lane] = -a[c].im / best;
      pb[14][lane] = (double)p;
    }
    __syncthreads();
    const zd rp = {pb[12][lane], pb[13][lane]};
    piv[c] = (int)pb[14][lane];
    if (col == c) {
      // the pivot column becomes a column of the inverse
#pragma unroll
      for (int r = 0; r < 6; r++) a[r] = r == c ? rp : zd{-a[r].re, -a[r].im} * rp;
    } else {
      swap_rows(a, c, piv[c]);
      a[c] = a[c] * rp;
#pragma unroll
      for (int r = 0; r < 6; r++)
        if (r != c) a[r] = cmad(zd{-pb[2 * r][lane], -pb[2 * r + 1][lane]}, a[c], a[r]);
    }
  }
  // undo the row swaps as column swaps, last first
#pragma unroll
  for (int c = 5; c >= 0; c--) dest = dest == c ? piv[c] : (dest == piv[c] ? c : dest);
  return dest;
}

// column j of block b of the packed term (diag[6], offd[15] below the diagonal)
template <typename Pin>
__device__ __forceinline__ zd packed_at(const void *in, long long stride, int vpc, int s, int b, int i, int j)
{
  if (i == j) return {dev_load_real<Pin>(in, stride, vpc, s, 36 * b + i), 0.0};
  const int hi = i > j ? i : j, lo = i > j ? j : i, k = 36 * b + 6 + hi * (hi - 1) + 2 * lo;
  const zd v = {dev_load_real<Pin>(in, stride, vpc, s, k), dev_load_real<Pin>(in, stride, vpc, s, k + 1)};
  return i > j ? v : conj(v);
}

// mode 0: packed Hermitian inverse of A; mode 1: full inverses of A +/- i mu g5;
// mode 2: the two-flavour inverses (full out0 = up, out1 = down, packed out2)
// A block per 32 sites, lane = site, a warp per (block of A, column): the
// matrix is 24 registers a thread and every access is coalesced.  One thread
// per site with the matrices and their inverses in local memory (3.6 KB of
// stack) took 1025 us at 24^3x48 (FP64, mode 0), 18 times the term's and its
// inverse's bytes; this takes 222 us.
constexpr int kInvertThreads = 12 * 32;

// rows below the diagonal, and the diagonal, of column j of a packed block
template <typename Q>
__device__ __forceinline__ void store_packed(void *o, long long stride, int vpc, int s, int b, int j, const zd v[6],
                                             double scale)
{
#pragma unroll
  for (int i = 0; i < 6; i++) {
    if (i == j) dev_store_real<Q>(o, stride, vpc, s, 36 * b + i, scale * v[i].re);
    if (i > j) dev_store_pair<Q>(o, stride, vpc, s, 36 * b + 6 + i * (i - 1) + 2 * j, scale * v[i].re, scale * v[i].im);
  }
}
template <typename Q>
__device__ __forceinline__ void store_full(void *o, long long stride, int vpc, int s, int b, int j, const zd v[6])
{
#pragma unroll
  for (int i = 0; i < 6; i++) dev_store_pair<Q>(o, stride, vpc, s, 72 * b + (i * 6 + j) * 2, v[i].re, v[i].im);
}

template <typename Pin, typename Q, int MODE>
__global__ void __launch_bounds__(kInvertThreads)
    clover_invert_kernel(Geom geo, const void *in, long long stride, int vpc_in, void *out0, void *out1, int vpc_out,
                         double mu, void *out2, int vpc_out2, double eps)
{
  __shared__ PivotBuf buf;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = w / 6, col = w % 6;
  const int site = blockIdx.x * 32 + lane;
  const int s = site < geo.vh ? site : geo.vh - 1;
  const bool live = site < geo.vh;
  const double g5 = b == 0 ? 1.0 : -1.0;
  zd a[6];
#pragma unroll
  for (int i = 0; i < 6; i++) a[i] = packed_at<Pin>(in, stride, vpc_in, s, b, i, col);
  if (MODE == 0) {
    const int j = invert6(a, col, b, lane, buf);
    if (live) store_packed<Q>(out0, stride, vpc_out, s, b, j, a, 1.0);
  } else if (MODE == 1) {
#pragma unroll 1
    for (int sgn = 0; sgn < 2; sgn++) {
      zd m[6];
#pragma unroll
      for (int i = 0; i < 6; i++) m[i] = {a[i].re, a[i].im + (i == col ? (sgn == 0 ? mu * g5 : -(mu * g5)) : 0.0)};
      if (sgn) __syncthreads();  // the buffers of the inverse before
      const int j = invert6(m, col, b, lane, buf);
      if (live) store_full<Q>(sgn == 0 ? out0 : out1, stride, vpc_out, s, b, j, m);
    }
  } else {
    zd q[6];
#pragma unroll
    for (int i = 0; i < 6; i++) {
      zd v = {i == col ? mu * mu - eps * eps : 0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 6; k++) v = cmad(packed_at<Pin>(in, stride, vpc_in, s, b, i, k), a[k], v);
      q[i] = v;
    }
    const int j = invert6(q, col, b, lane, buf);
    if (!live) return;
    // up: Q (A - i mu g5), down: Q (A + i mu g5); Q and A commute
    zd up[6], dn[6];
    const double tw = mu * g5;
#pragma unroll
    for (int i = 0; i < 6; i++) {
      zd v = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 6; k++) v = cmad(packed_at<Pin>(in, stride, vpc_in, s, b, i, k), q[k], v);
      up[i] = {v.re + tw * q[i].im, v.im - tw * q[i].re};
      dn[i] = {v.re - tw * q[i].im, v.im + tw * q[i].re};
    }
    store_full<Q>(out0, stride, vpc_out, s, b, j, up);
    store_full<Q>(out1, stride, vpc_out, s, b, j, dn);
    store_packed<Q>(out2, stride, vpc_out2, s, b, j, q, eps);
  }
}

// The two-flavour inverse clover term on its own (no hop), one (up, down)
// pair per thread: out_up = Fa psi_up + C psi_dn, out_dn = Fb psi_dn + C psi_up
// (TMClovDslash::two_flav_inverse_clover_term, tm_clov_dslash_body.h:1184-1343;
// per-site form codegen/dslash_common.cc:1198-1341), FP64 arithmetic
template <typename P>
__global__ void two_flav_clover_kernel(int vh, int npairs, SpinorArg out, SpinorArg in, CloverArg fa, CloverArg fb,
                                       CloverArg c)
{
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y;
  if (s >= vh || k >= npairs) return;
  using T = typename P::real;
  T up[24], dn[24], f[72], cl[36];
  SpinorIO<P>::load(in, 2 * k, s, up);
  SpinorIO<P>::load(in, 2 * k + 1, s, dn);
  double ou[24], od[24];
  for (int b = 0; b < 2; b++) {
    // one 6-vector block: index i = 3 (spin - 2b) + colour
    zd xu[6], xd[6];
    for (int i = 0; i < 6; i++) {
      const int e = ((2 * b + i / 3) * 3 + i % 3) * 2;
      xu[i] = zd{(double)up[e], (double)up[e + 1]};
      xd[i] = zd{(double)dn[e], (double)dn[e + 1]};
    }
    zd yu[6], yd[6];
    CloverIO<P, 144>::load(fa, s, 72 * b, 72, f);
    for (int i = 0; i < 6; i++) {
      zd v = {0.0, 0.0};
      for (int j = 0; j < 6; j++) v = v + zd{(double)f[(i * 6 + j) * 2], (double)f[(i * 6 + j) * 2 + 1]} * xu[j];
      yu[i] = v;
    }
    CloverIO<P, 144>::load(fb, s, 72 * b, 72, f);
    for (int i = 0; i < 6; i++) {
      zd v = {0.0, 0.0};
      for (int j = 0; j < 6; j++) v = v + zd{(double)f[(i * 6 + j) * 2], (double)f[(i * 6 + j) * 2 + 1]} * xd[j];
      yd[i] = v;
    }
    // packed Hermitian C: up += C dn, dn += C up
    CloverIO<P, 72>::load(c, s, 36 * b, 36, cl);
    for (int i = 0; i < 6; i++) {
      yu[i] = yu[i] + zd{(double)cl[i], 0.0} * xd[i];
      yd[i] = yd[i] + zd{(double)cl[i], 0.0} * xu[i];
    }
    for (int i = 1; i < 6; i++)
      for (int j = 0; j < i; j++) {
        const int od = i * (i - 1) / 2 + j;
        const zd a = {(double)cl[6 + 2 * od], (double)cl[7 + 2 * od]};
        yu[i] = yu[i] + a * xd[j];
        yu[j] = yu[j] + conj(a) * xd[i];
        yd[i] = yd[i] + a * xu[j];
        yd[j] = yd[j] + conj(a) * xu[i];
      }
    for (int i = 0; i < 6; i++) {
      const int e = ((2 * b + i / 3) * 3 + i % 3) * 2;
      ou[e] = yu[i].re;
      ou[e + 1] = yu[i].im;
      od[e] = yd[i].re;
      od[e + 1] = yd[i].im;
    }
  }
  for (int e = 0; e < 24; e++) {
    up[e] = (T)ou[e];
    dn[e] = (T)od[e];
  }
  SpinorIO<P>::store(out, 2 * k, s, up);
  SpinorIO<P>::store(out, 2 * k + 1, s, dn);
}

template <typename Pin, typename Q>
__global__ void clover_convert_kernel(Geom geo, const void *in, int vpc_in, void *out, int vpc_out, long long stride,
                                      int nr)
{
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= geo.vh) return;
  for (int k = 0; k < nr; k++)
    dev_store_real<Q>(out, stride, vpc_out, s, k, dev_load_real<Pin>(in, stride, vpc_in, s, k));
}

#define QPX_OUT_SWITCH(prec, CALL)                          \
  switch (prec) {                                           \
  case PREC_F64: { using Q = F64; CALL; } break;            \
  case PREC_F32: { using Q = F32; CALL; } break;            \
  case PREC_F16: { using Q = F16; CALL; } break;            \
  case PREC_BF16: { using Q = BF16; CALL; } break;          \
  case PREC_Q16: { using Q = F16; CALL; } break;            \
  case PREC_Q16F32: { using Q = F32; CALL; } break;         \
  default: throw Error(QPHIX_GPU_EINVAL, "bad precision");  \
  }
#define QPX_IN_SWITCH(prec, CALL)                           \
  switch (prec) {                                           \
  case PREC_F64: { using Pin = F64; CALL; } break;          \
  case PREC_F32: { using Pin = F32; CALL; } break;          \
  case PREC_F16: { using Pin = F16; CALL; } break;          \
  case PREC_BF16: { using Pin = BF16; CALL; } break;        \
  case PREC_Q16: { using Pin = F16; CALL; } break;          \
  case PREC_Q16F32: { using Pin = F32; CALL; } break;       \
  default: throw Error(QPHIX_GPU_EINVAL, "bad precision");  \
  }

void launch_clover_build(int recon, int prec_out, Geom geo, GaugeArg g, void *out, long long stride, int vpc, int cb,
                         double diag_mass, double cr, double ct, dim3 grid, cudaStream_t st)
{
  if (recon == 12) {
    QPX_OUT_SWITCH(prec_out, (clover_build_kernel<12, Q><<<grid, kPlanes * kLeafSites, 0, st>>>(geo, g, out, stride, vpc, cb, diag_mass,
                                                                                cr, ct)));
  } else {
    QPX_OUT_SWITCH(prec_out, (clover_build_kernel<18, Q><<<grid, kPlanes * kLeafSites, 0, st>>>(geo, g, out, stride, vpc, cb, diag_mass,
                                                                                cr, ct)));
  }
}

void launch_clover_invert(int prec_in, int prec_out, Geom geo, const void *in, long long stride, int vpc_in, void *o0,
                          void *o1, int vpc_out, int mode, double mu, dim3 grid, cudaStream_t st, void *o2,
                          int vpc_out2, double eps)
{
#define QPX_INVERT(MODE)                                                                                       \
  QPX_IN_SWITCH(prec_in, QPX_OUT_SWITCH(prec_out, (clover_invert_kernel<Pin, Q, MODE><<<grid, kInvertThreads, 0, st>>>( \
                                                       geo, in, stride, vpc_in, o0, o1, vpc_out, mu, o2, vpc_out2, eps))))
  if (mode == 0) {
    QPX_INVERT(0)
  } else if (mode == 1) {
    QPX_INVERT(1)
  } else {
    QPX_INVERT(2)
  }
#undef QPX_INVERT
}

void launch_two_flav_clover(int prec, int vh, int npairs, SpinorArg out, SpinorArg in, CloverArg fa, CloverArg fb,
                            CloverArg c, cudaStream_t st)
{
  dim3 grid((unsigned)((vh + 63) / 64), (unsigned)npairs);
  switch (prec) {
  case PREC_F64: two_flav_clover_kernel<F64><<<grid, 64, 0, st>>>(vh, npairs, out, in, fa, fb, c); break;
  case PREC_F32: two_flav_clover_kernel<F32><<<grid, 64, 0, st>>>(vh, npairs, out, in, fa, fb, c); break;
  case PREC_F16: two_flav_clover_kernel<F16><<<grid, 64, 0, st>>>(vh, npairs, out, in, fa, fb, c); break;
  case PREC_BF16: two_flav_clover_kernel<BF16><<<grid, 64, 0, st>>>(vh, npairs, out, in, fa, fb, c); break;
  case PREC_Q16: two_flav_clover_kernel<Q16><<<grid, 64, 0, st>>>(vh, npairs, out, in, fa, fb, c); break;
  case PREC_Q16F32: two_flav_clover_kernel<Q16F32><<<grid, 64, 0, st>>>(vh, npairs, out, in, fa, fb, c); break;
  default: throw Error(QPHIX_GPU_EINVAL, "bad precision");
  }
}

void launch_clover_convert(int prec_in, int prec_out, Geom geo, const void *in, int vpc_in, void *out, int vpc_out,
                           long long stride, int nr, dim3 grid, cudaStream_t st)
{
  QPX_IN_SWITCH(prec_in, QPX_OUT_SWITCH(prec_out, (clover_convert_kernel<Pin, Q><<<grid, QPX_BLOCK, 0, st>>>(
                                                       geo, in, vpc_in, out, vpc_out, stride, nr))));
}

}  // namespace qpx
