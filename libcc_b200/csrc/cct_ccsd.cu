// CCSD T1-dressing terms of the reference's OpenACC CCSD port
// (src/triples-ijk/ccsd_acc.f: terms_29_30_31, lines 1-60, and
// terms_32_33_34_35, lines 64-160), on one GPU holding every occupied index.
// They contract the same expanded VVVO slices (ab|c j) as the triples W build,
// here with T1 (O1) and T2 (O2) into CCSD residual intermediates.
//
// terms_29_30_31, per occupied j, as the reference's DGEMM / TRANMD / INSITU
// sequence composes (the oracle restates the literal sequence):
//   T2(i,y,z,j) += sum_x O1(i,x) G_j(x,y,z),
//   G_j(x,y,z) = (z x|y j) - sum_k O1(k,z) VL(k,x,y,j) - sum_k O1(k,y) VR(z,k,x,j).
// The O1 contraction is moved inside the two correction terms, so no nu^3 G_j
// is formed:
//   T2(i,y,z,j) += X_j(y,z,i) - sum_k O1(k,z) P_j(i,k,y) - sum_k O1(k,y) Q_j(i,z,k),
//   X_j(p,q,i) = sum_x (x q|p j) O1(i,x),   P_j(i,k,y) = sum_x O1(i,x) VL(k,x,y,j),
//   Q_j(i,z,k) = sum_x O1(i,x) VR(z,k,x,j).
// X_j is 2 no^2 nu^3 flops on the tensor pipe instead of 6 no^2 nu^3, read from
// the packed slices without expanding them.  For no <= 32 one kernel forms
// X_j and P_j for a (y, j) and adds both to T2 (f4_x_kernel), a second one Q_j
// and its product for eight z (f4_qt_kernel); larger no runs the W-build tile on
// gathered rows and element-wise kernels.
//
// terms_32_33_34_35:
//   t2 <- t2^T as an (nou x nou) matrix                            (TRANSQ)
//   o2(x,y,k,l) <- o2(k,x,y,l)                                     (INSITU 12, 23)
//   RL_pre(i,y,z,j) = sum_x O1(i,x) (x y|z j) = X_j(z,y,i);  rl <- RL_pre^T
//                                                                  (DGEMM, TRANSQ)
//   vm(x,y,z,a) <- vm(y,x,z,a) + T((x,z), (a,y)),                  (TRANMD 312, update, TRANMD 23)
//   T((k,l), (a,j)) = sum_{x,y} o2(k,x,y,l) (a y|x j)
// T is one GEMM of M = no^2, N = nu no, K = nu^2 for all j at once: the FP64
// tensor-core W-build tile (cct_wbuild_tile.cuh) on row operands laid out
// for it.  The reference's VM update loop (ccsd_acc.f:136-144) adds tmp at
// an offset of one element; this follows the evident intent, VM(k,l,j,a) +=
// tmp((k,l),a).
#include "cct_internal.cuh"
#include "cct_wbuild_tile.cuh"

#include <map>
#include <mutex>

namespace cct {
namespace {


int grid_of(int64_t n) {
  int64_t b = (n + 255) / 256;
  return (int)(b > 148 * 32 ? 148 * 32 : (b < 1 ? 1 : b));
}

// O1 as the W-build tile's column operand: o1pad[i][x] = O1(i,x), rows of kp
// doubles, zero past (no, nu)
__global__ void f4_o1pad_kernel(int no, int nu, int64_t kp, int64_t np, const double *__restrict__ o1,
                                double *__restrict__ o1pad) {
  const int64_t n = np * kp;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / kp, x = e - i * kp;
    o1pad[e] = (i < no && x < nu) ? o1[i + (int64_t)no * x] : 0.0;
  }
}

// P[j][y][k][i] = sum_x O1(i,x) VL(k,x,y,j) and Q[j][z][k][i] = sum_x O1(i,x) VR(z,k,x,j)
__global__ void f4_pq_kernel(int no, int nu, const double *__restrict__ o1, const double *__restrict__ vl,
                             const double *__restrict__ vr, double *__restrict__ P, double *__restrict__ Q) {
  const int64_t n = (int64_t)no * no * nu * no;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < 2 * n; e += (int64_t)gridDim.x * blockDim.x) {
    const int which = e >= n;
    const int64_t r = e - which * n;
    const int64_t i = r % no, k = (r / no) % no, y = (r / ((int64_t)no * no)) % nu, j = r / ((int64_t)no * no * nu);
    double s = 0.0;
    if (!which) {
      const double *v = vl + k + (int64_t)no * (int64_t)nu * (y + (int64_t)nu * j);  // VL(k, x, y, j), x stride no
      for (int x = 0; x < nu; x++) s += o1[i + (int64_t)no * x] * v[(int64_t)no * x];
      P[r] = s;
    } else {
      const double *v = vr + y + (int64_t)nu * (k + (int64_t)no * (int64_t)nu * j);  // VR(z=y, k, x, j), x stride nu no
      for (int x = 0; x < nu; x++) s += o1[i + (int64_t)no * x] * v[(int64_t)nu * no * x];
      Q[r] = s;
    }
  }
}

// ---- no <= kNoTile: the products with O1 on the FP64 tensor pipe
// (mma.sync.m16n8k4), NT = ceil(no / 8) column fragments.
constexpr int kNoTile = 32;

__device__ __forceinline__ void cp8(double *smem, const double *gmem, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(ok ? 8 : 0));
}

// O1 in fragment order, so a warp's fragment is one contiguous 256-byte load:
//   ob[x / 4][j][lane] = O1(8 j + lane / 4, x + lane % 4)      column operand, K = x
//   oa[y / 16][k / 4][h][lane] = O1(k + lane % 4, y + 8 h + lane / 4)  row operand, K = k
// zero past (no, nu); x runs to a multiple of 16.
__global__ void f4_o1frag_kernel(int no, int nu, int nt, int k4, int64_t nob, int64_t noa,
                                 const double *__restrict__ o1, double *__restrict__ ob, double *__restrict__ oa) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nob + noa;
       e += (int64_t)gridDim.x * blockDim.x) {
    const bool b = e < nob;
    const int64_t r = b ? e : e - nob;
    const int lane = (int)(r & 31), g = lane >> 2, t = lane & 3;
    const int64_t f = r >> 5;
    int64_t i, x;
    if (b) {
      i = 8 * (f % nt) + g;
      x = 4 * (f / nt) + t;
    } else {
      i = 4 * ((f / 2) % k4) + t;
      x = 16 * (f / 2 / k4) + 8 * (f & 1) + g;
    }
    const double v = i < no && x < nu ? o1[i + (int64_t)no * x] : 0.0;
    (b ? ob : oa)[r] = v;
  }
}

// X_j(p, q, i) = sum_x (x q|p j) O1(i, x) for one (p, j) per CTA; T2 form (t2
// set): T2(i,p,q,j) += X_j(p,q,i) - sum_k O1(k,q) P(i,k), P(i,k) = sum_x O1(i,x)
// VL(k,x,p,j); else X goes to X[(j nu^2 + p nu + q) np + i].
//
// The packed triangle of (p, j) holds (x q) once, row max(x,q).  A warp owns 32
// rows q, two 16-row blocks; per 16 x each block is 16 rows of the triangle's
// 128-byte runs whichever side of the diagonal it lies on (rows q right of
// it, rows x left of it, kept transposed in shared memory), so every global read
// is coalesced; blocks on the diagonal are read element by element.  Element
// (r, c) of a block lies at 16 r + (c ^ 4 (r & 3)), r the triangle row: the
// fragment reads hit sixteen bank pairs either way.  Runs start on any 8-byte
// boundary, hence 8-byte copies.  Warps share nothing in the main loop, so there is no
// barrier in it; ten warps and two CTAs on an SM keep the packed slices of a
// whole wave (2 x 148 of 0.4 MB at nu = 320) near the size of L2, where the second
// of an element's two reads finds it.
// Bound: the FP64 tensor pipe (3.8e10 flop at no24-nu320: 1.0 ms).  There the
// X GEMM on rows gathered through the triangle index, P and the T2 pass took 4.07 ms, this
// kernel 1.99 ms.
constexpr int kXW = 10;        // warps
constexpr int kXStages = 2;    // 16-x chunks in flight per warp
constexpr int kXSmem = kXW * kXStages * 2 * 256 * 8;
static_assert(kXStages * 2 * 256 >= kNoTile * kNoTile, "the warps' sums of P fit");
template <int NT>
__global__ void __launch_bounds__(kXW * 32, 2)
    f4_x_kernel(int no, uint32_t nu, int k4, const double *__restrict__ vvvo, const double *__restrict__ ob,
                const double *__restrict__ oa, const double *__restrict__ vl, double *__restrict__ t2,
                double *__restrict__ X, int64_t np) {
  extern __shared__ __align__(16) double xsm[];
  __shared__ double ps[kNoTile][NT * 8];  // -P(i, k) at [k][i]
  const int p = blockIdx.x, j = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nk = (nu + 15) / 16;  // x chunks
  const double *tri = vvvo + ((int64_t)j * nu + p) * ((int64_t)nu * (nu + 1) / 2);
  if (t2) {
    // P: every warp takes each tenth four of the x, all (k, i); the warps'
    // sums are added in order.  (A (16 k, 8 i) tile per warp over every x
    // left ten warps waiting on six chains of loads: 0.6 ms of the launch.)
    const double *slab = vl + (int64_t)no * nu * (p + (int64_t)nu * j);  // VL(k, x, p, j) = slab[k + no x]
    double acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int n = 0; n < NT; n++)
#pragma unroll
        for (int r = 0; r < 4; r++) acc[m][n][r] = 0.0;
#pragma unroll 2
    for (int ks = warp; ks < 4 * nk; ks += kXW) {
      const int x = 4 * ks + t;
      double a[4], bf[NT];
#pragma unroll
      for (int q = 0; q < 4; q++) a[q] = 8 * q + g < no && x < nu ? slab[8 * q + g + (int64_t)no * x] : 0.0;
#pragma unroll
      for (int n = 0; n < NT; n++) bf[n] = __ldg(ob + ((int64_t)ks * NT + n) * 32 + lane);
#pragma unroll
      for (int n = 0; n < NT; n++) {
        wb::dmma_16x8x4(acc[0][n], a[0], a[1], bf[n]);
        if (NT > 2) wb::dmma_16x8x4(acc[1][n], a[2], a[3], bf[n]);
      }
    }
    double *part = xsm + warp * (kNoTile * NT * 8);
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int n = 0; n < NT; n++)
#pragma unroll
        for (int r = 0; r < 4; r++)
          part[(16 * m + g + 8 * (r >> 1)) * (NT * 8) + 8 * n + 2 * t + (r & 1)] = acc[m][n][r];
    __syncthreads();
    for (int e = threadIdx.x; e < kNoTile * NT * 8; e += kXW * 32) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kXW; w++) v += xsm[w * (kNoTile * NT * 8) + e];
      (&ps[0][0])[e] = e < no * NT * 8 ? -v : 0.0;  // (a row k >= no is 0 x O1: NaN where O1 is infinite)
    }
    __syncthreads();
  }
  double *mine = xsm + warp * (kXStages * 2 * 256);
  const int lr = lane >> 4, lc = lane & 15;
  for (int qb = 32 * warp; qb < nu; qb += 32 * kXW) {
    double acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int n = 0; n < NT; n++)
#pragma unroll
        for (int r = 0; r < 4; r++) acc[m][n][r] = 0.0;
    auto load = [&](int c) {  // chunk c into its ring slot
      const int x0 = 16 * c;
#pragma unroll
      for (int m = 0; m < 2; m++) {
        double *dst = mine + ((c & (kXStages - 1)) * 2 + m) * 256;
        const int q0 = qb + 16 * m;
        if (x0 == q0) {  // the diagonal block, rows q
#pragma unroll
          for (int it = 0; it < 8; it++) {
            const int r = lr + 2 * it, q = q0 + r, x = x0 + lc;
            const uint32_t hi = max(q, x), lo = min(q, x);  // nu <= 4096: triangle offsets below 2^24
            cp8(dst + 16 * r + (lc ^ ((r & 3) << 2)), tri + (hi < nu ? hi * (hi + 1) / 2 + lo : 0), hi < nu);
          }
        } else {  // rows of the triangle R0 .., columns C0 .. < R0
          const int R0 = max(x0, q0), C = min(x0, q0) + lc;
#pragma unroll
          for (int it = 0; it < 8; it++) {
            const uint32_t r = lr + 2 * it, row = R0 + r;
            cp8(dst + 16 * r + (lc ^ ((r & 3) << 2)), tri + (row < nu ? row * (row + 1) / 2 + C : 0), row < nu);
          }
        }
      }
    };
#pragma unroll
    for (int c = 0; c < kXStages - 1; c++) {
      if (c < nk) load(c);
      wb::cp_async_commit();
    }
    for (int c = 0; c < nk; c++) {
      if (c + kXStages - 1 < nk) load(c + kXStages - 1);
      wb::cp_async_commit();
      wb::cp_async_wait<kXStages - 1>();
      __syncwarp();
      const double *src = mine + (c & (kXStages - 1)) * 512;
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        double b[NT];
#pragma unroll
        for (int n = 0; n < NT; n++) b[n] = __ldg(ob + ((int64_t)(4 * c + kk) * NT + n) * 32 + lane);
#pragma unroll
        for (int m = 0; m < 2; m++) {
          const double *blk = src + m * 256;
          const int x = 4 * kk + t;
          double a0, a1;
          if (16 * c > qb + 16 * m) {  // rows x: the block is kept transposed
            a0 = blk[16 * x + (g ^ ((x & 3) << 2))];
            a1 = blk[16 * x + ((g + 8) ^ ((x & 3) << 2))];
          } else {
            a0 = blk[16 * g + (x ^ ((g & 3) << 2))];
            a1 = blk[16 * (g + 8) + (x ^ ((g & 3) << 2))];
          }
#pragma unroll
          for (int n = 0; n < NT; n++) wb::dmma_16x8x4(acc[m][n], a0, a1, b[n]);
        }
      }
      __syncwarp();  // the slot is refilled by the next iteration's load
    }
    wb::cp_async_wait<0>();
    if (t2) {
      for (int kk = 0; kk < k4; kk++) {
        double b[NT];
#pragma unroll
        for (int n = 0; n < NT; n++) b[n] = ps[4 * kk + t][8 * n + g];
#pragma unroll
        for (int m = 0; m < 2; m++) {
          const int64_t yt = qb / 16 + m;
          if (16 * yt >= nu) continue;
          const double *a = oa + ((yt * k4 + kk) * 2) * 32 + lane;
          const double a0 = __ldg(a), a1 = __ldg(a + 32);
#pragma unroll
          for (int n = 0; n < NT; n++) wb::dmma_16x8x4(acc[m][n], a0, a1, b[n]);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int q = qb + 16 * m + g + 8 * h;
        if (q >= nu) continue;
        double *row = t2 ? t2 + (int64_t)no * (p + (int64_t)nu * (q + (int64_t)nu * j))
                         : X + (((int64_t)j * nu + p) * nu + q) * np;
        double old[NT][2];
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int r = 0; r < 2; r++) {
            const int i = 8 * n + 2 * t + r;
            old[n][r] = t2 && i < no ? row[i] : 0.0;
          }
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int r = 0; r < 2; r++) {
            const int i = 8 * n + 2 * t + r;
            if (i < no) row[i] = old[n][r] + acc[m][n][2 * h + r];
          }
      }
  }
}

// T2(i,y,z,j) -= sum_k O1(k,y) Q(i,z,k), Q(i,z,k) = sum_x O1(i,x) VR(z,k,x,j),
// for eight z and one j per CTA, one z per warp: VR(z .. z+7, k, x, j) are
// 64-byte runs, staged 8 x at a time; the warp's Q then is the column operand
// of its z's T2 slab, which is one contiguous run over (i, y).  Element (z, k)
// of an x lies at 33 z + k, an x every 268 doubles: fragment reads (k = 0..3 by x
// = 0..3) hit sixteen bank pairs, the copies at most two to a pair.
// Bound: HBM, VR once and T2 read and written (1.4 GB at no24-nu320: 0.21 ms).  0.52 ms
// there; Q and the T2 pass as two kernels took 1.91 ms.
constexpr int kQX = 8, kQPitch = 268, kQStages = 3;
constexpr int kQSmem = 8 * kNoTile * kNoTile * 8;  // the ring, later the warps' Q
static_assert(kQStages * kQX * kQPitch <= 8 * kNoTile * kNoTile, "the ring fits");
template <int NT>
__global__ void __launch_bounds__(256, 2)
    f4_qt_kernel(int no, int nu, int k4, const double *__restrict__ ob, const double *__restrict__ oa,
                 const double *__restrict__ vr, double *__restrict__ t2) {
  extern __shared__ __align__(16) double qsm[];
  const int z0 = blockIdx.x * 8, j = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nc = (nu + kQX - 1) / kQX;
  const int64_t nuno = (int64_t)nu * no;
  const double *src = vr + nuno * nu * j;
  auto load = [&](int c) {
    double *dst = qsm + (c % kQStages) * (kQX * kQPitch);
    for (int e = threadIdx.x; e < kQX * kNoTile * 8; e += 256) {
      const int z = e & 7, k = (e >> 3) & (kNoTile - 1), xl = e >> 8, x = c * kQX + xl;
      if (k >= no) continue;  // (rows past no of a fragment are never stored)
      const bool ok = x < nu && z0 + z < nu;
      cp8(dst + xl * kQPitch + 33 * z + k, src + (ok ? (z0 + z) + (int64_t)nu * k + nuno * x : 0), ok);
    }
  };
  double acc[2][NT][4];
#pragma unroll
  for (int m = 0; m < 2; m++)
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
      for (int r = 0; r < 4; r++) acc[m][n][r] = 0.0;
  for (int e = threadIdx.x; e < kQStages * kQX * kQPitch; e += 256) qsm[e] = 0.0;  // k >= no
  __syncthreads();
#pragma unroll
  for (int c = 0; c < kQStages - 1; c++) {
    if (c < nc) load(c);
    wb::cp_async_commit();
  }
  for (int c = 0; c < nc; c++) {
    wb::cp_async_wait<kQStages - 2>();
    __syncthreads();
    if (c + kQStages - 1 < nc) load(c + kQStages - 1);
    wb::cp_async_commit();
    const double *buf = qsm + (c % kQStages) * (kQX * kQPitch) + 33 * warp;
#pragma unroll
    for (int kk = 0; kk < kQX / 4; kk++) {
      double b[NT];
#pragma unroll
      for (int n = 0; n < NT; n++) b[n] = __ldg(ob + ((int64_t)(c * (kQX / 4) + kk) * NT + n) * 32 + lane);
#pragma unroll
      for (int m = 0; m < 2; m++) {
        if (m == 1 && NT <= 2) continue;  // no <= 16
        const double *a = buf + (4 * kk + t) * kQPitch + 16 * m + g;
        const double a0 = a[0], a1 = a[8];
#pragma unroll
        for (int n = 0; n < NT; n++) wb::dmma_16x8x4(acc[m][n], a0, a1, b[n]);
      }
    }
  }
  wb::cp_async_wait<0>();
  __syncthreads();  // every warp is done with the ring
  const int z = z0 + warp;
  if (z >= nu) return;
  // -Q(i, z, k) at [k][i], the warp's own
  double *qz = qsm + warp * (kNoTile * kNoTile);
#pragma unroll
  for (int m = 0; m < 2; m++)
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
      for (int r = 0; r < 4; r++)
        qz[(16 * m + g + 8 * (r >> 1)) * kNoTile + 8 * n + 2 * t + (r & 1)] =
            16 * m + g + 8 * (r >> 1) < no ? -acc[m][n][r] : 0.0;
  __syncwarp();
  double b[2 * NT][NT];
#pragma unroll
  for (int kk = 0; kk < 2 * NT; kk++)
#pragma unroll
    for (int n = 0; n < NT; n++) b[kk][n] = qz[(4 * kk + t) * kNoTile + 8 * n + g];
  double *slab = t2 + nuno * (z + (int64_t)nu * j);
  const int ny = (nu + 15) / 16;
  for (int yt = 0; yt < ny; yt++) {
    // the product is summed on its own and T2 rounded once
    double c[NT][4], old[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int y = 16 * yt + g + 8 * (r >> 1), i = 8 * n + 2 * t + (r & 1);
        old[n][r] = y < nu && i < no ? slab[i + (int64_t)no * y] : 0.0;
        c[n][r] = 0.0;
      }
#pragma unroll
    for (int kk = 0; kk < 2 * NT; kk++) {
      if (kk >= k4) break;
      const double *a = oa + (((int64_t)yt * k4 + kk) * 2) * 32 + lane;
      const double a0 = __ldg(a), a1 = __ldg(a + 32);
#pragma unroll
      for (int n = 0; n < NT; n++) wb::dmma_16x8x4(c[n], a0, a1, b[kk][n]);
    }
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int y = 16 * yt + g + 8 * (r >> 1), i = 8 * n + 2 * t + (r & 1);
        if (y < nu && i < no) slab[i + (int64_t)no * y] = old[n][r] + c[n][r];
      }
  }
}

// T2(i,y,z,j) += X_j(y,z,i) - sum_k O1(k,z) P[j][y][k][i] - sum_k O1(k,y) Q[j][z][k][i]
__global__ void f4_t2_kernel(int no, int nu, int64_t np, const double *__restrict__ o1, const double *__restrict__ X,
                             const double *__restrict__ P, const double *__restrict__ Q, double *__restrict__ t2) {
  const int64_t nu2 = (int64_t)nu * nu, n = (int64_t)no * nu2 * no;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % no, y = (e / no) % nu, z = (e / ((int64_t)no * nu)) % nu, j = e / ((int64_t)no * nu2);
    double v = X[(j * nu2 + y * nu + z) * np + i];
    const double *pj = P + (j * nu + y) * no * no + i, *qj = Q + (j * nu + z) * no * no + i;
    for (int k = 0; k < no; k++) v -= o1[k + (int64_t)no * z] * pj[(int64_t)k * no];
    for (int k = 0; k < no; k++) v -= o1[k + (int64_t)no * y] * qj[(int64_t)k * no];
    t2[e] += v;
  }
}

// rl = RL_pre^T as (nou x nou) matrices: rl[(z + nu j) + nou (i + no y)] = X_j(z,y,i)
// (written in order; the X reads are strided)
__global__ void f4_rl_kernel(int no, int nu, int64_t np, const double *__restrict__ X, double *__restrict__ rl) {
  const int64_t nu2 = (int64_t)nu * nu, nou = (int64_t)no * nu, n = nou * nou;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t zj = e % nou, iy = e / nou, z = zj % nu, j = zj / nu, i = iy % no, y = iy / no;
    rl[e] = X[(j * nu2 + z * nu + y) * np + i];
  }
}

// dst = src^T for an n x n column-major matrix
__global__ void f4_transq_kernel(int64_t n, const double *__restrict__ src, double *__restrict__ dst) {
  const int64_t nn = n * n;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nn; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e % n, c = e / n;
    dst[e] = src[c + n * r];
  }
}

// Zeroes the padding of the T GEMM's operands: the columns of a split past nu^2
// (na rows of apad, np of bpad a split), the rows of bpad past nb.  One launch:
// clearing both operands whole took 0.18 of 3.7 ms at no16-nu200, a memset per
// split 20 of 157 us at the smallest sizes.
__global__ void f4_pad_kernel(int64_t nu2, int64_t kp, int64_t na, int64_t nb, int64_t np, double *__restrict__ apad,
                              double *__restrict__ bpad) {
  const int64_t z = blockIdx.y, left = nu2 - z * kp, used = left < 0 ? 0 : (left < kp ? left : kp), cols = kp - used;
  const int64_t step = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t e = first; e < cols * (na + nb); e += step) {
    const int64_t r = e / cols, c = used + e - r * cols;
    if (r < na)
      apad[(z * na + r) * kp + c] = 0.0;
    else
      bpad[(z * np + r - na) * kp + c] = 0.0;
  }
  for (int64_t e = first; e < (np - nb) * kp; e += step) bpad[(z * np + nb) * kp + e] = 0.0;
}

// o2 (no,nu,nu,no) -> o2b (nu,nu,no,no), o2b(x,y,k,l) = o2(k,x,y,l); also the
// GEMM's row operand apad[(k + no l)][x + nu y] with rows of kp doubles
__global__ void f4_o2_kernel(int no, int nu, int64_t kp, const double *__restrict__ o2, double *__restrict__ o2b,
                             double *__restrict__ apad) {
  const int64_t nu2 = (int64_t)nu * nu, n = nu2 * no * no, no2 = (int64_t)no * no;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t xy = e % nu2, kl = e / nu2;
    const int64_t x = xy % nu, y = xy / nu, k = kl % no, l = kl / no;
    const double v = o2[k + no * (x + nu * (y + nu * l))];
    o2b[e] = v;
    const int64_t z = xy / kp;  // K split
    apad[(z * no2 + kl) * kp + (xy - z * kp)] = v;
  }
}

// the GEMM's column operand: bpad[split][(a + nu j)][x + nu y] = (a y|x j), rows
// of kp doubles per split (np rows per split).  A transpose through shared
// memory: a CTA reads 32 packed columns (j, x0..x0+31) x 32 consecutive
// triangle entries t0..t0+31 along the columns, and writes each entry (a, y),
// a >= y, as 32 consecutive x of rows (a, j) and (y, j).  HBM-bound by its two
// writes and one read an element; where an entry's two runs begin, and after
// how many x they go on in the next split, is worked out once an entry, by one
// warp while the loads are in flight.  With the square root and the divisions by
// kp done for every element it took 0.576 ms at no16-nu200, 0.274 ms now (0.23 at
// the HBM rate).
constexpr int kTT = 32;
__global__ void __launch_bounds__(256) f4_b_kernel(int no, int nu, int64_t kp, int64_t np,
                                                   const double *__restrict__ vvvo, double *__restrict__ bpad) {
  __shared__ double tile[kTT][kTT + 1];
  __shared__ int64_t s_run[2][kTT];  // where the run of x0 begins in rows (a, j), (y, j); -1: no run
  __shared__ int s_left[2][kTT];     // columns of its split from x0 on (at most kTT)
  const int64_t nutr = (int64_t)nu * (nu + 1) / 2;
  const int64_t x0 = (int64_t)blockIdx.y * kTT, t0 = (int64_t)blockIdx.x * kTT;
  const int j = blockIdx.z;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double v[kTT / 8];
#pragma unroll
  for (int i = 0; i < kTT / 8; i++) {
    const int64_t x = x0 + ty + 8 * i, t = t0 + tx;
    v[i] = (x < nu && t < nutr) ? __ldg(vvvo + ((int64_t)j * nu + x) * nutr + t) : 0.0;
  }
  if (threadIdx.x < kTT) {
    const int64_t t = t0 + threadIdx.x;
    // t = a (a + 1) / 2 + y with 0 <= y <= a
    int64_t a = (int64_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while (a * (a + 1) / 2 > t) a--;
    while ((a + 1) * (a + 2) / 2 <= t) a++;
    const int64_t y = t - a * (a + 1) / 2;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t row = h ? y : a, c = x0 + (int64_t)nu * (h ? a : y);
      const int64_t z = c / kp, r = c - z * kp, left = kp - r;
      s_run[h][threadIdx.x] = t < nutr && (h == 0 || a != y) ? (z * np + row + (int64_t)nu * j) * kp + r : -1;
      s_left[h][threadIdx.x] = (int)(left < kTT ? left : kTT);
    }
  }
#pragma unroll
  for (int i = 0; i < kTT / 8; i++) tile[ty + 8 * i][tx] = v[i];
  __syncthreads();
  if (x0 + tx >= nu) return;
  const int64_t jump = (np - 1) * kp;  // from the end of a split's row to the next split's
#pragma unroll
  for (int i = 0; i < kTT / 8; i++) {
    const int ti = ty + 8 * i;
    const double e = tile[tx][ti];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      int64_t at = s_run[h][ti];
      if (at < 0) continue;
      at += tx;
      for (int64_t left = s_left[h][ti]; tx >= left; left += kp) at += jump;
      bpad[at] = e;
    }
  }
}

// vm_out(x,y,z,a) = vm_in(y,x,z,a) + sum over the K splits of T[(x + no z) np + (a + nu y)]
__global__ void f4_vm_kernel(int no, int nu, int64_t np, int nsplit, int64_t tsplit, const double *__restrict__ vm_in,
                             const double *__restrict__ t, double *__restrict__ vm_out) {
  const int64_t n = (int64_t)no * no * no * nu;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = e % no, y = (e / no) % no, z = (e / ((int64_t)no * no)) % no, a = e / ((int64_t)no * no * no);
    const double *tz = t + (x + no * z) * np + (a + nu * y);
    double v = tz[0];
    for (int sp = 1; sp < nsplit; sp++) v += tz[sp * tsplit];
    vm_out[e] = vm_in[y + no * (x + no * (z + no * a))] + v;
  }
}

// Device workspace of the two entry points, kept between calls: a call asks
// for the same sequence of buffers every time, so slot k of entry point e on
// device d (the k-th buffer of the call) is reused, and grown when a call
// needs more; after the first call of a shape nothing is allocated.  The
// entry points are synchronous and serialised by a mutex;
// ccT_ccsd_release_workspace frees the workspace.
struct Workspace {
  std::vector<std::pair<void *, size_t>> slot;
};
std::mutex g_ws_mutex;
std::map<std::pair<int, int>, Workspace> g_ws;

struct DevBuf {  // device copies of host arrays (or the caller's device arrays) and scratch
  std::lock_guard<std::mutex> lock{g_ws_mutex};
  Workspace *ws = nullptr;
  size_t next = 0;
  explicit DevBuf(int entry) {
    int dev = 0;
    cudaGetDevice(&dev);
    ws = &g_ws[{dev, entry}];
  }
  int alloc(void **dst, size_t bytes) {
    if (bytes < 8) bytes = 8;
    if (next == ws->slot.size()) ws->slot.push_back({nullptr, 0});
    std::pair<void *, size_t> &sl = ws->slot[next++];
    if (sl.second < bytes) {
      if (sl.first) CCT_CUDA(cudaFree(sl.first));
      sl = {nullptr, 0};
      CCT_CUDA(cudaMalloc(&sl.first, bytes));
      sl.second = bytes;
    }
    *dst = sl.first;
    return CCT_OK;
  }
  int get(double **dst, const double *src, int64_t n, int32_t mem, bool upload, cudaStream_t s) {
    if (mem == CCT_MEM_DEVICE) {
      *dst = const_cast<double *>(src);
      return CCT_OK;
    }
    CCT_TRY(alloc(reinterpret_cast<void **>(dst), (size_t)n * 8));
    if (upload) CCT_CUDA(cudaMemcpyAsync(*dst, src, (size_t)n * 8, cudaMemcpyHostToDevice, s));
    return CCT_OK;
  }
  int tmp(double **dst, int64_t n) { return alloc(reinterpret_cast<void **>(dst), (size_t)n * 8); }
};

// O1 in fragment order (f4_o1frag_kernel), no <= kNoTile.
struct O1Frag {
  int nt, k4;
  double *ob, *oa;
};
int o1_fragments(int64_t no, int64_t nu, const double *d_o1, DevBuf &b, O1Frag *f, cudaStream_t s) {
  f->nt = (int)((no + 7) / 8);
  f->k4 = (int)((no + 3) / 4);
  const int64_t chunks = (nu + 15) / 16, nob = 4 * chunks * f->nt * 32, noa = chunks * f->k4 * 64;
  CCT_TRY(b.tmp(&f->ob, nob));
  CCT_TRY(b.tmp(&f->oa, noa));
  f4_o1frag_kernel<<<grid_of(nob + noa), 256, 0, s>>>((int)no, (int)nu, f->nt, f->k4, nob, noa, d_o1, f->ob, f->oa);
  CCT_CUDA(cudaGetLastError());
  return CCT_OK;
}

template <int NT>
int launch_x(int64_t no, int64_t nu, const O1Frag &f, const double *vvvo, const double *vl, double *t2, double *X,
             int64_t np, cudaStream_t s) {
  static int configured_device = -1;  // (the entry points are serialised)
  int dev = 0;
  CCT_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    CCT_CUDA(cudaFuncSetAttribute(f4_x_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kXSmem));
    configured_device = dev;
  }
  f4_x_kernel<NT><<<dim3((unsigned)nu, (unsigned)no), kXW * 32, kXSmem, s>>>((int)no, (int)nu, f.k4, vvvo, f.ob, f.oa,
                                                                            vl, t2, X, np);
  CCT_CUDA(cudaGetLastError());
  return CCT_OK;
}
// vl and t2 set: the T2 update; else X (rows of np doubles).
int launch_x(int64_t no, int64_t nu, const O1Frag &f, const double *vvvo, const double *vl, double *t2, double *X,
             int64_t np, cudaStream_t s) {
  switch (f.nt) {
    case 1: return launch_x<1>(no, nu, f, vvvo, vl, t2, X, np, s);
    case 2: return launch_x<2>(no, nu, f, vvvo, vl, t2, X, np, s);
    case 3: return launch_x<3>(no, nu, f, vvvo, vl, t2, X, np, s);
    default: return launch_x<4>(no, nu, f, vvvo, vl, t2, X, np, s);
  }
}
template <int NT>
int launch_qt(int64_t no, int64_t nu, const O1Frag &f, const double *vr, double *t2, cudaStream_t s) {
  static int configured_device = -1;
  int dev = 0;
  CCT_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    CCT_CUDA(cudaFuncSetAttribute(f4_qt_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kQSmem));
    configured_device = dev;
  }
  f4_qt_kernel<NT><<<dim3((unsigned)((nu + 7) / 8), (unsigned)no), 256, kQSmem, s>>>((int)no, (int)nu, f.k4, f.ob,
                                                                                     f.oa, vr, t2);
  CCT_CUDA(cudaGetLastError());
  return CCT_OK;
}

// X_j(p,q,i) = sum_x (x q|p j) O1(i,x) for every occupied j, X_j at x + j nu^2 np,
// row (p,q) at (p nu + q) np: f4_x_kernel, or for no > kNoTile the W-build
// tile, one packed-row job per j.
int packed_o1_gemm(int64_t no, int64_t nu, const double *d_o1, const double *d_vvvo, DevBuf &b, double **X,
                   int64_t *np_out, cudaStream_t s) {
  const int64_t nutr = nu * (nu + 1) / 2;
  if (no <= kNoTile) {
    O1Frag f;
    CCT_TRY(o1_fragments(no, nu, d_o1, b, &f, s));
    *np_out = 8 * f.nt;
    CCT_TRY(b.tmp(X, no * nu * nu * *np_out));
    return launch_x(no, nu, f, d_vvvo, nullptr, nullptr, *X, *np_out, s);
  }
  Dims g{};
  g.nu = (int)nu;                  // M = nu^2 rows (p, q)
  g.no = 0;                        // K = nu (the packed part of a row alone)
  g.KP = round_up(nu, kKB);
  g.BN = choose_bn((int)no);
  g.NP = round_up(no, g.BN);
  double *o1pad;
  CCT_TRY(b.tmp(&o1pad, g.NP * g.KP));
  CCT_TRY(b.tmp(X, no * nu * nu * g.NP));
  f4_o1pad_kernel<<<grid_of(g.NP * g.KP), 256, 0, s>>>((int)no, (int)nu, g.KP, g.NP, d_o1, o1pad);
  CCT_CUDA(cudaGetLastError());
  std::vector<GemmJob> jobs((size_t)no);
  for (int64_t j = 0; j < no; j++) {
    const double *pj = d_vvvo + j * nu * nutr;  // the nu packed columns of occupied j
    jobs[j] = GemmJob{pj, pj, o1pad, o1pad, *X + j * nu * nu * g.NP, 1, 1, pj, pj};
  }
  GemmJob *d_jobs;
  CCT_TRY(b.alloc(reinterpret_cast<void **>(&d_jobs), jobs.size() * sizeof(GemmJob)));
  CCT_CUDA(cudaMemcpyAsync(d_jobs, jobs.data(), jobs.size() * sizeof(GemmJob), cudaMemcpyHostToDevice, s));
  CCT_TRY(launch_wbuild_f64(g, d_jobs, (int)no, s));
  *np_out = g.NP;
  return CCT_OK;
}

int check_args(int64_t no, int64_t nu, int32_t mem) {
  if (no < 1 || nu < 1 || no > 4096 || nu > 4096 || (mem != CCT_MEM_HOST && mem != CCT_MEM_DEVICE)) {
    set_error("need 1 <= no, nu <= 4096 and mem CCT_MEM_HOST or CCT_MEM_DEVICE");
    return CCT_ERR_INVALID;
  }
  return CCT_OK;
}

}  // namespace
}  // namespace cct

using namespace cct;

extern "C" int ccT_ccsd_terms_29_31(int64_t no, int64_t nu, const double *o1, double *t2, const double *vl,
                                    const double *vr, const double *vvvo, int32_t mem) {
  CCT_TRY(check_args(no, nu, mem));
  if (!o1 || !t2 || !vl || !vr || !vvvo) {
    set_error("an array pointer is NULL");
    return CCT_ERR_INVALID;
  }
  const cudaStream_t s = nullptr;
  const int64_t nu2 = nu * nu, nutr = nu * (nu + 1) / 2;
  DevBuf b(0);
  double *d_o1, *d_t2, *d_vl, *d_vr, *d_vvvo;
  CCT_TRY(b.get(&d_o1, o1, no * nu, mem, true, s));
  CCT_TRY(b.get(&d_t2, t2, no * nu2 * no, mem, true, s));
  CCT_TRY(b.get(&d_vl, vl, no * nu2 * no, mem, true, s));
  CCT_TRY(b.get(&d_vr, vr, nu * no * nu * no, mem, true, s));
  CCT_TRY(b.get(&d_vvvo, vvvo, nutr * nu * no, mem, true, s));
  if (no <= kNoTile) {
    O1Frag f;
    CCT_TRY(o1_fragments(no, nu, d_o1, b, &f, s));
    CCT_TRY(launch_x(no, nu, f, d_vvvo, d_vl, d_t2, nullptr, 0, s));
    switch (f.nt) {
      case 1: CCT_TRY(launch_qt<1>(no, nu, f, d_vr, d_t2, s)); break;
      case 2: CCT_TRY(launch_qt<2>(no, nu, f, d_vr, d_t2, s)); break;
      case 3: CCT_TRY(launch_qt<3>(no, nu, f, d_vr, d_t2, s)); break;
      default: CCT_TRY(launch_qt<4>(no, nu, f, d_vr, d_t2, s)); break;
    }
  } else {
    double *X, *P, *Q;
    int64_t np = 0;
    CCT_TRY(packed_o1_gemm(no, nu, d_o1, d_vvvo, b, &X, &np, s));
    CCT_TRY(b.tmp(&P, no * no * nu * no));
    CCT_TRY(b.tmp(&Q, no * no * nu * no));
    f4_pq_kernel<<<grid_of(2 * no * no * nu * no), 256, 0, s>>>((int)no, (int)nu, d_o1, d_vl, d_vr, P, Q);
    CCT_CUDA(cudaGetLastError());
    f4_t2_kernel<<<grid_of(no * nu2 * no), 256, 0, s>>>((int)no, (int)nu, np, d_o1, X, P, Q, d_t2);
    CCT_CUDA(cudaGetLastError());
  }
  if (mem == CCT_MEM_HOST) CCT_CUDA(cudaMemcpyAsync(t2, d_t2, (size_t)no * nu2 * no * 8, cudaMemcpyDeviceToHost, s));
  CCT_CUDA(cudaStreamSynchronize(s));
  return CCT_OK;
}

extern "C" int ccT_ccsd_terms_32_35(int64_t no, int64_t nu, const double *o1, double *o2, double *t2, double *vm,
                                    double *rl, const double *vvvo, int32_t mem) {
  CCT_TRY(check_args(no, nu, mem));
  if (!o1 || !o2 || !t2 || !vm || !rl || !vvvo) {
    set_error("an array pointer is NULL");
    return CCT_ERR_INVALID;
  }
  if (nu * nu < no) {
    set_error("terms_32_35 needs nu^2 >= no");
    return CCT_ERR_INVALID;
  }
  const cudaStream_t s = nullptr;
  const int64_t nu2 = nu * nu, nou = no * nu, n4 = nou * nou, nutr = nu * (nu + 1) / 2;
  DevBuf b(1);
  double *d_o1, *d_o2, *d_t2, *d_vm, *d_rl, *d_vvvo;
  CCT_TRY(b.get(&d_o1, o1, no * nu, mem, true, s));
  CCT_TRY(b.get(&d_o2, o2, n4, mem, true, s));
  CCT_TRY(b.get(&d_t2, t2, n4, mem, true, s));
  CCT_TRY(b.get(&d_vm, vm, no * no * no * nu, mem, true, s));
  CCT_TRY(b.get(&d_rl, rl, n4, mem, false, s));
  CCT_TRY(b.get(&d_vvvo, vvvo, nutr * nu * no, mem, true, s));
  // TRANSQ(T2) (ccsd_acc.f:83)
  double *tmp;
  CCT_TRY(b.tmp(&tmp, n4));
  CCT_CUDA(cudaMemcpyAsync(tmp, d_t2, (size_t)n4 * 8, cudaMemcpyDeviceToDevice, s));
  f4_transq_kernel<<<grid_of(n4), 256, 0, s>>>(nou, tmp, d_t2);
  CCT_CUDA(cudaGetLastError());
  // RL_pre(i,y,z,j) = sum_x O1(i,x) (x y|z j) = X_j(z,y,i) (line 109), then TRANSQ into rl (line 151)
  {
    double *X;
    int64_t np = 0;
    CCT_TRY(packed_o1_gemm(no, nu, d_o1, d_vvvo, b, &X, &np, s));
    f4_rl_kernel<<<grid_of(n4), 256, 0, s>>>((int)no, (int)nu, np, X, d_rl);
    CCT_CUDA(cudaGetLastError());
  }
  // INSITU 12, 23 of O2 (lines 84-85) and the GEMM operands.  T has few
  // output tiles (M = no^2) and a long contraction (K = nu^2), so K is split
  // into nsplit ranges, each a job of its own (the operands stored split by
  // split), for whole waves of CTAs; f4_vm_kernel sums the splits in order.
  Dims g{};
  g.nu = (int)no;                        // M = no^2 rows (k + no l)
  g.BN = choose_bn(nou);
  g.NP = round_up(nou, g.BN);            // N = nu no (a + nu j)
  int nsplit = 1;
  {
    int dev = 0, nsm = 148;
    CCT_CUDA(cudaGetDevice(&dev));
    CCT_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int64_t slots = 3 * (int64_t)nsm;  // W-build tile: three CTAs per SM
    const int64_t tiles = ((int64_t)no * no + wb::BM - 1) / wb::BM * (g.NP / g.BN);
    double best = 0.0;
    for (int sp = 1; sp <= 16 && (int64_t)sp * kKB <= nu2; sp++) {
      const int64_t ctas = tiles * sp, waves = (ctas + slots - 1) / slots;
      const double fill = (double)ctas / (double)(waves * slots);
      if (fill > best + 0.02) {
        best = fill;
        nsplit = sp;
      }
    }
  }
  g.KP = round_up((nu2 + nsplit - 1) / nsplit, kKB);  // K per split (x + nu y), zero past nu^2
  g.no = (int)(g.KP - no);                            // every column of a split counts as valid
  double *o2in, *apad, *bpad, *t;
  CCT_TRY(b.tmp(&o2in, n4));
  CCT_TRY(b.tmp(&apad, nsplit * no * no * g.KP));
  CCT_TRY(b.tmp(&bpad, nsplit * g.NP * g.KP));
  CCT_TRY(b.tmp(&t, nsplit * no * no * g.NP));
  CCT_CUDA(cudaMemcpyAsync(o2in, d_o2, (size_t)n4 * 8, cudaMemcpyDeviceToDevice, s));
  const int64_t pad_blocks = std::min<int64_t>(64, (g.KP * (no * no + g.NP) + 8191) / 8192);
  f4_pad_kernel<<<dim3((unsigned)pad_blocks, nsplit), 256, 0, s>>>(nu2, g.KP, no * no, nou, g.NP, apad, bpad);
  CCT_CUDA(cudaGetLastError());
  f4_o2_kernel<<<grid_of(n4), 256, 0, s>>>((int)no, (int)nu, g.KP, o2in, d_o2, apad);
  CCT_CUDA(cudaGetLastError());
  {
    const int64_t nutr = nu * (nu + 1) / 2;
    const dim3 grid((unsigned)((nutr + kTT - 1) / kTT), (unsigned)((nu + kTT - 1) / kTT), (unsigned)no);
    f4_b_kernel<<<grid, 256, 0, s>>>((int)no, (int)nu, g.KP, g.NP, d_vvvo, bpad);
  }
  CCT_CUDA(cudaGetLastError());
  // T((k,l),(a,j)) = sum_{x,y} o2b(x,y,k,l) (a y|x j) (line 119 for every j) on the FP64 tensor cores
  std::vector<GemmJob> jobs(nsplit);
  for (int z = 0; z < nsplit; z++) {
    const double *az = apad + (int64_t)z * no * no * g.KP, *bz = bpad + (int64_t)z * g.NP * g.KP;
    jobs[z] = GemmJob{az, az, bz, bz, t + (int64_t)z * no * no * g.NP, 1, 0};
  }
  GemmJob *d_job;
  CCT_TRY(b.alloc(reinterpret_cast<void **>(&d_job), nsplit * sizeof(GemmJob)));
  CCT_CUDA(cudaMemcpyAsync(d_job, jobs.data(), nsplit * sizeof(GemmJob), cudaMemcpyHostToDevice, s));
  CCT_TRY(launch_wbuild_f64(g, d_job, nsplit, s));
  // VM: TRANMD 312, the update of lines 125-131, TRANMD 23 (lines 86, 154)
  double *vmin;
  CCT_TRY(b.tmp(&vmin, no * no * no * nu));
  CCT_CUDA(cudaMemcpyAsync(vmin, d_vm, (size_t)no * no * no * nu * 8, cudaMemcpyDeviceToDevice, s));
  f4_vm_kernel<<<grid_of(no * no * no * nu), 256, 0, s>>>((int)no, (int)nu, g.NP, nsplit, no * no * g.NP, vmin, t,
                                                          d_vm);
  CCT_CUDA(cudaGetLastError());
  if (mem == CCT_MEM_HOST) {
    CCT_CUDA(cudaMemcpyAsync(t2, d_t2, (size_t)n4 * 8, cudaMemcpyDeviceToHost, s));
    CCT_CUDA(cudaMemcpyAsync(o2, d_o2, (size_t)n4 * 8, cudaMemcpyDeviceToHost, s));
    CCT_CUDA(cudaMemcpyAsync(vm, d_vm, (size_t)no * no * no * nu * 8, cudaMemcpyDeviceToHost, s));
    CCT_CUDA(cudaMemcpyAsync(rl, d_rl, (size_t)n4 * 8, cudaMemcpyDeviceToHost, s));
  }
  CCT_CUDA(cudaStreamSynchronize(s));
  return CCT_OK;
}

extern "C" int ccT_ccsd_release_workspace(void) {
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  int prev = 0;
  cudaGetDevice(&prev);
  for (auto &e : g_ws) {
    cudaSetDevice(e.first.first);
    for (auto &sl : e.second.slot)
      if (sl.first) cudaFree(sl.first);
  }
  g_ws.clear();
  cudaSetDevice(prev);
  return CCT_OK;
}
