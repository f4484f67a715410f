// Per-tuple E[4] (etd) and E[5] v1 reduction.
//
// Reference: t1wt3_ijk (src/triples-ijk/t1wt3.f90:18-109), T3SQUA_SMP
// (src/triples-abc/t3squa.f:1-113), ADT3DEN + DRT1WT3IJK/IJ/JK
// (src/triples-abc/ddcc_aux.f:97-238).  Per tuple (i,j,k) with W_aaa = 0:
//
//   x3 = sum_abc W_abc (8 W_abc - 4(W_acb + W_cba + W_bac) + 2(W_bca + W_cab)) / D_abc
//   v1(a,i) += sum_bc [Z1 VOE(b,c,j,k) + Z2 VOE(b,c,k,j)] / D_abc      (Z1..Z6 as in
//   v1(a,j) += sum_bc [Z3 VOE(b,c,i,k) + Z5 VOE(b,c,k,i)] / D_abc       t1wt3.f90:80-85,
//   v1(a,k) += sum_bc [Z4 VOE(b,c,i,j) + Z6 VOE(b,c,j,i)] / D_abc       summed over all b)
//   etd += w x3,  v1 += w (...),  w = 1 (i>j>k) or 1/2 (i=j or j=k)
//
// The twelve terms arrive as the three GEMM outputs X_g (cct_wbuild_f64.cu),
// so W at all six index permutations is assembled on chip: one CTA owns an
// unordered triple of 8-wide index blocks {A<=B<=C}, brings the X blocks of
// its orbit into shared memory, and evaluates every element of those blocks
// once.  Per-CTA partials are summed by
// tuple_sum_kernel and group_add_kernel in a fixed order, so results are bitwise reproducible.
#include <algorithm>
#include <type_traits>

#include "cct_internal.cuh"
#include "cct_reduce_block.cuh"

namespace cct {
namespace {

using namespace red;

// Block triples of every tuple of the group, blockIdx.x-th and each
// gridDim.x-th after it; a group may mix tuple kinds, the branch is uniform over
// a CTA.
template <Fill FILL>
__global__ void __launch_bounds__(RT, 2) reduce_kernel(int nu, int no, int64_t NP, int ncta, int64_t vsize,
                                                      const __grid_constant__ TupleGroup grp,
                                                      const double *__restrict__ eh, const double *__restrict__ ep,
                                                      const double *__restrict__ vb,
                                                      const int16_t *__restrict__ table, double *__restrict__ xpart,
                                                      double *__restrict__ vpart, int *err, int wait_limit) {
  extern __shared__ __align__(16) double dyn_smem[];
  const Smem m(dyn_smem);
  int u = blockIdx.x / ncta, c = blockIdx.x - u * ncta;
  if (u >= grp.n) return;
  int S0 = table[3 * c], S1 = table[3 * c + 1], S2 = table[3 * c + 2];
  auto start = [&](const TupleDev &t, int A, int B, int C) {
    if (FILL == kBulk)
      start_copies(nu, no, NP, t, vb, A, B, C, m);
    else
      start_rows(nu, no, NP, t, vb, A, B, C, m);
  };
  if (FILL == kBulk) init_copies(m);
  start(grp.t[u], S0, S1, S2);
  for (uint32_t round = 0;; round ^= 1) {
    int u1 = u, c1 = c + gridDim.x;
    while (c1 >= ncta) {
      c1 -= ncta;
      u1++;
    }
    const bool more = u1 < grp.n;
    int T0 = 0, T1 = 0, T2 = 0;
    if (more) {
      T0 = table[3 * c1];
      T1 = table[3 * c1 + 1];
      T2 = table[3 * c1 + 2];
    }
    if (FILL == kRows)
      rows_landed();
    else if (!copies_landed(m, round, err, wait_limit))
      return;
    auto next = [&]() {
      if (!more) return;
      __syncthreads();
      start(grp.t[u1], T0, T1, T2);
    };
    const TupleDev &t = grp.t[u];
    double *xp = xpart + (int64_t)u * ncta + c, *vp = vpart + u * vsize;
    auto block = [&](auto kind) {
      constexpr int KIND = decltype(kind)::value;
      reduce_compute<KIND>(nu, t, eh, ep, S0, S1, S2, xp, vp, m, next);
    };
    if (t.kind == kIJK)
      block(std::integral_constant<int, kIJK>{});
    else if (t.kind == kIJJ)
      block(std::integral_constant<int, kIJJ>{});
    else
      block(std::integral_constant<int, kIIJ>{});
    if (!more) break;
    u = u1;
    c = c1;
    S0 = T0;
    S1 = T1;
    S2 = T2;
  }
}

// Sums of one tuple's partials, weighted: tsum[0] = its E[4], then the v1
// columns of i, j and k (nu each).  Grid (1 + ceil(nu / kFinA), tuple of the
// group).  Block 0 sums the per-CTA x3 partials (sum t takes partials t, t+256, ...
// in order, then a tree over the 256 sums); every other block
// owns kFinA virtual indices a, one warp per (a, column), each summing the
// column's v1 partials over all block triples containing a (lane-strided,
// then a shuffle tree).  The loads of a thread's partials are issued eight at
// a time ahead of its (ordered) adds.
// Two virtual indices: 192 threads at 40 registers fit beside a CTA of the
// emulated W build (576 threads at 96), under which these sums run.
constexpr int kFinA = 2;
constexpr int kFinThreads = 32 * 3 * kFinA;
__global__ void __launch_bounds__(kFinThreads) tuple_sum_kernel(int nu, int nb, int64_t ncta, int64_t vsize,
                                                                const __grid_constant__ TupleGroup grp,
                                                                const double *__restrict__ xpart_all,
                                                                const double *__restrict__ vpart_all,
                                                                double *__restrict__ tsum_all) {
  constexpr int U = 8;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const double weight = grp.t[blockIdx.y].weight;
  const double *xpart = xpart_all + (int64_t)blockIdx.y * ncta, *vpart = vpart_all + (int64_t)blockIdx.y * vsize;
  double *tsum = tsum_all + (int64_t)blockIdx.y * (1 + 3 * nu);
  if (blockIdx.x == 0) {
    __shared__ double red[256];
    for (int q = tid; q < 256; q += kFinThreads) {  // 256 partial sums, whatever the threads
      double s = 0.0;
      for (int64_t c0 = q; c0 < ncta; c0 += 256 * U) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = c0 + 256 * u < ncta ? xpart[c0 + 256 * u] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++)
          if (c0 + 256 * u < ncta) s += v[u];
      }
      red[q] = s;
    }
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
      for (int q = tid; q < st; q += kFinThreads) red[q] += red[q + st];
      __syncthreads();
    }
    if (tid == 0) tsum[0] = weight * red[0];
    return;
  }
  const int warp = tid >> 5, la8 = warp / 3, col = warp - 3 * (warp / 3);
  const int a = (blockIdx.x - 1) * kFinA + la8;
  if (a < nu) {
    const int X = a / RB, la = a - (a / RB) * RB;
    const int64_t npairs = (int64_t)nb * (nb + 1) / 2;
    const double *slab = vpart + (((int64_t)X * RB + la) * 3 + col) * npairs;
    double v = 0.0;
    for (int64_t q0 = lane; q0 < npairs; q0 += 32 * U) {
      double x[U];
#pragma unroll
      for (int u = 0; u < U; u++) x[u] = q0 + 32 * u < npairs ? slab[q0 + 32 * u] : 0.0;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (q0 + 32 * u < npairs) v += x[u];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) tsum[1 + col * nu + a] = weight * v;
  }
}

// Adds the group's tuple sums to the accumulators in tuple order, each tuple's
// columns in the order i, j, k: etd_acc[0..1] is a Neumaier (sum,
// compensation) pair, v1_acc(nu, no) takes one thread per element.
__global__ void __launch_bounds__(256) group_add_kernel(int nu, int no, const __grid_constant__ TupleGroup grp,
                                                        const double *__restrict__ tsum, double *__restrict__ etd_acc,
                                                        double *__restrict__ v1_acc) {
  const int64_t stride = 1 + 3 * (int64_t)nu;
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      double sum = etd_acc[0], comp = etd_acc[1];
      for (int u = 0; u < grp.n; u++) {
        const double v = tsum[u * stride];
        const double nsum = sum + v;
        comp += fabs(sum) >= fabs(v) ? (sum - nsum) + v : (v - nsum) + sum;
        sum = nsum;
      }
      etd_acc[0] = sum;
      etd_acc[1] = comp;
    }
    return;
  }
  const int64_t e = (int64_t)(blockIdx.x - 1) * 256 + threadIdx.x;
  if (e >= (int64_t)nu * no) return;
  const int x = (int)(e / nu), a = (int)(e - (int64_t)x * nu);
  double v = v1_acc[e];
  constexpr int U = 4;  // tuples whose loads are in flight together
  for (int u0 = 0; u0 < grp.n; u0 += U) {
    double c[U][3];
#pragma unroll
    for (int q = 0; q < U; q++) {
      const TupleDev &t = grp.t[u0 + q < grp.n ? u0 + q : u0];
      const double *s = tsum + (u0 + q) * stride + 1 + a;
      const bool live = u0 + q < grp.n;
      c[q][0] = live && t.i == x ? s[0] : 0.0;
      c[q][1] = live && t.j == x ? s[nu] : 0.0;
      c[q][2] = live && t.k == x ? s[2 * (int64_t)nu] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < U; q++) v = ((v + c[q][0]) + c[q][1]) + c[q][2];
  }
  v1_acc[e] = v;
}

// out3 = {ets, etd, ets+etd}; ets = 2 sum_{i,a} t1(i,a) v1(a,i) (triples.F90:311-316)
__global__ void ets_kernel(int no, int nu, const double *__restrict__ t1, const double *__restrict__ v1,
                           const double *__restrict__ etd_acc, double *__restrict__ out3) {
  __shared__ double red[256];
  const int tid = threadIdx.x;
  double s = 0.0;
  const int64_t n = (int64_t)no * nu;
  for (int64_t e = tid; e < n; e += 256) {
    const int64_t i = e / nu, a = e - (e / nu) * nu;
    s += t1[i + (int64_t)no * a] * v1[a + (int64_t)nu * i];
  }
  red[tid] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (tid < st) red[tid] += red[tid + st];
    __syncthreads();
  }
  if (tid == 0) {
    const double ets = 2.0 * red[0];
    const double etd = etd_acc[0] + etd_acc[1];
    out3[0] = ets;
    out3[1] = etd;
    out3[2] = ets + etd;
  }
}

// One thread per entry of a tile (launch_build_vb).
__global__ void build_vb_kernel(int no, int nu, int nb, const double *__restrict__ voe, double *__restrict__ vb) {
  const int64_t n = (int64_t)no * no * nb * nb * VTILE, nu2 = (int64_t)nu * nu;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t tile = e / VTILE, yz = tile / ((int64_t)nb * nb), AB = tile - yz * nb * nb;
    const int64_t A = AB / nb, B = AB - A * nb, y = yz / no, z = yz - y * no;
    const int64_t f = RB * A + (e & 7), s = RB * B + ((e >> 3) & 7);
    double v = 0.0;
    if (f < nu && s < nu)
      v = fma(2.0, voe[(z * no + y) * nu2 + f + nu * s], -voe[(y * no + z) * nu2 + f + nu * s]);
    vb[e] = v;
  }
}

}  // namespace

int launch_build_vb(const Dims &d, const double *voe, double *vb, cudaStream_t s) {
  const int64_t blocks = (vb_size(d) + 255) / 256;
  build_vb_kernel<<<(unsigned)std::min<int64_t>(blocks, 148 * 64), 256, 0, s>>>(d.no, d.nu, d.nb, voe, vb);
  CCT_CUDA(cudaGetLastError());
  return CCT_OK;
}

template <Fill FILL>
int launch_reduce_fill(const Dims &d, const TupleGroup &g, const double *eh, const double *ep, const double *vb,
                       const int16_t *cta_table, double *xpart, double *vpart, int *err, cudaStream_t s,
                       int wait_limit) {
  constexpr int smem = REDUCE_SMEM;
  static int configured_device = -1;
  int dev = 0;
  CCT_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    CCT_CUDA(cudaFuncSetAttribute(reduce_kernel<FILL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    CCT_CUDA(cudaFuncSetAttribute(reduce_kernel<FILL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                  cudaSharedmemCarveoutMaxShared));
    configured_device = dev;
  }
  static int nsm = 0;
  if (nsm == 0) CCT_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  // up to two rounds of two CTAs per SM: a CTA per triple (no4-nu36: 79 us a
  // forward, 80 with every CTA taking two)
  const int64_t total = d.ncta * g.n, blocks = total <= 4 * nsm ? total : 2 * nsm;
  reduce_kernel<FILL><<<(unsigned)blocks, RT, smem, s>>>(d.nu, d.no, d.NP, (int)d.ncta, vpart_size(d), g, eh, ep, vb,
                                                         cta_table, xpart, vpart, err, wait_limit);
  CCT_CUDA(cudaGetLastError());
  return CCT_OK;
}

int launch_reduce(const Dims &d, const TupleGroup &g, bool blocked, const double *eh, const double *ep,
                  const double *vb, const int16_t *cta_table, double *xpart, double *vpart, int *err, cudaStream_t s,
                  int wait_limit) {
  if (d.NP % RB) {
    set_error("the reduction needs NP a multiple of 8 (NP = " + std::to_string(d.NP) + ")");
    return CCT_ERR_INVALID;
  }
  if (blocked) return launch_reduce_fill<kBulk>(d, g, eh, ep, vb, cta_table, xpart, vpart, err, s, wait_limit);
  return launch_reduce_fill<kRows>(d, g, eh, ep, vb, cta_table, xpart, vpart, err, s, wait_limit);
}

int launch_finalize(const Dims &d, const TupleGroup &g, const double *xpart, const double *vpart, double *tsum,
                    double *etd_acc, double *v1_acc, cudaStream_t s) {
  static int configured_device = -1;
  int dev = 0;
  CCT_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    // the W builds' and reductions' carveout: an SM that would have to change
    // it first drains
    CCT_CUDA(cudaFuncSetAttribute(tuple_sum_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                  cudaSharedmemCarveoutMaxShared));
    CCT_CUDA(cudaFuncSetAttribute(group_add_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                  cudaSharedmemCarveoutMaxShared));
    configured_device = dev;
  }
  const int vblocks = (d.nu + kFinA - 1) / kFinA;  // one warp per (virtual index, column)
  tuple_sum_kernel<<<dim3(1 + vblocks, g.n), kFinThreads, 0, s>>>(d.nu, d.nb, d.ncta, vpart_size(d), g, xpart, vpart,
                                                                  tsum);
  CCT_CUDA(cudaGetLastError());
  const int ablocks = (int)(((int64_t)d.nu * d.no + 255) / 256);
  group_add_kernel<<<1 + ablocks, 256, 0, s>>>(d.nu, d.no, g, tsum, etd_acc, v1_acc);
  CCT_CUDA(cudaGetLastError());
  return CCT_OK;
}

int launch_ets(const Dims &d, const double *t1, const double *v1_acc, const double *etd_acc, double *out3,
               cudaStream_t s) {
  ets_kernel<<<1, 256, 0, s>>>(d.no, d.nu, t1, v1_acc, etd_acc, out3);
  CCT_CUDA(cudaGetLastError());
  return CCT_OK;
}

}  // namespace cct
