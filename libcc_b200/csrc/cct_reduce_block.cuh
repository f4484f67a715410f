// One block triple of the per-tuple E[4] / v1 reduction as a device function,
// shared by the per-tuple reduction kernel (cct_reduce.cu) and the persistent
// batch kernel (cct_batch.cu).  See cct_reduce.cu for the algorithm and the
// reference lines it follows.
#pragma once
#include "cct_internal.cuh"

namespace cct {
namespace red {


constexpr int RB = kRB;  // 8
constexpr int RT = 256;  // threads per reduction CTA
constexpr int SL = 512;  // doubles per 8x8x8 block

// The six permutations of three positions, in a fixed order:
// 0:(0,1,2)=abc 1:(0,2,1)=acb 2:(1,0,2)=bac 3:(1,2,0)=bca 4:(2,0,1)=cab 5:(2,1,0)=cba
__host__ __device__ constexpr int pm(int p, int m) {
  return p == 0 ? m : p == 1 ? (m == 0 ? 0 : m == 1 ? 2 : 1) : p == 2 ? (m == 0 ? 1 : m == 1 ? 0 : 2)
       : p == 3 ? (m == 0 ? 1 : m == 1 ? 2 : 0) : p == 4 ? (m == 0 ? 2 : m == 1 ? 0 : 1)
                : (m == 0 ? 2 : m == 1 ? 1 : 0);
}
__host__ __device__ constexpr int pidx(int p0, int p1) { return p0 * 2 + (p1 > p0 ? p1 - 1 : p1); }
// perm value of role r for element pi(x): W(x_{pi(r(0))}, ...) -> index of pi o r
__host__ __device__ constexpr int compose(int pi, int r) { return pidx(pm(pi, pm(r, 0)), pm(pi, pm(r, 1))); }

// W assembly per tuple kind: W(x0,x1,x2) += X_g(x_al0, x_al1, x_al2); {g, al0, al1, al2}
//   i>j>k : X0(a,b,c) + X1(a,c,b) + X2(b,c,a)
//   (i,j,j): X0(a,b,c) + X0(a,c,b) + X1(b,c,a) + X1(c,b,a)
//   (i,i,k): X0(a,b,c) + X0(b,a,c) + X1(a,c,b) + X1(b,c,a)
__host__ __device__ constexpr int term_entry(int kind, int term, int f) {
  constexpr int tab[3][4][4] = {{{0, 0, 1, 2}, {1, 0, 2, 1}, {2, 1, 2, 0}, {0, 0, 0, 0}},
                                {{0, 0, 1, 2}, {0, 0, 2, 1}, {1, 1, 2, 0}, {1, 2, 1, 0}},
                                {{0, 0, 1, 2}, {0, 1, 0, 2}, {1, 0, 2, 1}, {1, 1, 2, 0}}};
  return tab[kind][term][f];
}

template <typename T>
__device__ __forceinline__ T sel3(int m, T v0, T v1, T v2) {
  return m == 0 ? v0 : (m == 1 ? v1 : v2);
}

// Shared memory of a CTA, every block in its plain order (a bulk copy lands as
// it lies in memory):
//   X: block q of GEMM output g at (6 g + q) SL, element (u0,u1,u2) at 64 u0 + 8 u1 + u2,
//      q = the permutation of (A,B,C) it lies at: blocks (S_q0, S_q1, S_q2);
//   V: 8 x 8 tiles of the combined VOE planes (launch_build_vb), 64 doubles
//      each: pair 0 (b,c), 1 (a,c), 2 (a,b) x orientation (0: lower, higher
//      coordinate; 1: higher, lower) x planes jk kj ik ki ij ji;
//   the phase-C partials, and one mbarrier.
constexpr int kXBlocks = 18;
constexpr int VTILE = 64, VORI = 6 * VTILE, VPAIR = 2 * VORI, kVTiles = 36;
constexpr int kPartDoubles = 3 * (RT / 32) * RB * 3 + RT / 32;
constexpr int REDUCE_SMEM = (kXBlocks * SL + 3 * VPAIR + kPartDoubles + 1) * 8;

// Where the X blocks come from: kBulk, 8 x 8 x 8 blocks (xblock_base), each one
// contiguous 4 KB bulk copy; kRows, rows of NP (a forward that keeps W for the
// backward, the backward itself).
enum Fill { kBulk, kRows };

__device__ __forceinline__ int nb_of(int nu) { return (nu + RB - 1) / RB; }

// Element coordinates of a thread within block (A,B,C), packed 3 bits each
// (l0 lowest); the thread's second element (e = 1) is l2 ^ 4.  The map is
// linear over GF(2) and one to one on (tid, e).  A half-warp reads 64-bit
// words, so its sixteen lanes must fall on sixteen bank pairs, (64 u0 + 8 u1 +
// u2) mod 16 = u2 and the low bit of u1, for u any permutation of l: on every
// ordered pair of axes the three bits of one and the low bit of the other are
// independent in the four half-warp bits.  The same holds for the VOE tiles
// (u + 8 v).  Lanes with equal l0 differ by lane bits 1 and 16, with equal l1
// by 2 and 24, with equal l2 by 4 and 16; lane ^ 8 has l2 ^ 4.
__host__ __device__ __forceinline__ int orbit_coords(int t) {
  const int b0 = t & 1, b1 = (t >> 1) & 1, b2 = (t >> 2) & 1, b3 = (t >> 3) & 1, b4 = (t >> 4) & 1;
  const int w0 = (t >> 5) & 1, w1 = (t >> 6) & 1, w2 = (t >> 7) & 1;
  return (b1 ^ b2 ^ w0) | b2 << 1 | b3 << 2 | (b0 ^ b2) << 3 | (b0 ^ w1) << 4 | (b3 ^ b4) << 5 | (b0 ^ b1) << 6 |
         (b1 ^ w2) << 7 | b3 << 8;
}

// slot[p]: the first permutation whose ordered block triple equals O_p (so
// equal blocks of a degenerate orbit are loaded once).
__device__ __forceinline__ void orbit_slots(int S0, int S1, int S2, int slot[6]) {
  auto Sm = [&](int m) { return sel3(m, S0, S1, S2); };
#pragma unroll
  for (int p = 0; p < 6; p++) {
    slot[p] = p;
#pragma unroll
    for (int q = 5; q >= 0; q--)
      if (q < p && Sm(pm(q, 0)) == Sm(pm(p, 0)) && Sm(pm(q, 1)) == Sm(pm(p, 1)) && Sm(pm(q, 2)) == Sm(pm(p, 2)))
        slot[p] = q;
  }
}

// Tile c of the 36 VOE tiles of a CTA: source in vb, [y][z][nb][nb][64].
__device__ __forceinline__ int64_t voe_tile(int c, int no, int nb, const TupleDev &t, int S0, int S1, int S2) {
  const int pr = c / 12, ori = (c / 6) & 1, pl = c % 6, k = pl >> 1;
  const int lo = pr == 0 ? S1 : S0, hi = pr == 2 ? S1 : S2;
  const int y = k == 0 ? t.j : t.i, z = k == 2 ? t.j : t.k;  // planes 2k: (y,z), 2k + 1: (z,y)
  const int B1 = ori ? hi : lo, B2 = ori ? lo : hi;
  return ((((int64_t)(pl & 1 ? z : y) * no + (pl & 1 ? y : z)) * nb + B1) * nb + B2) * VTILE;
}

__device__ __forceinline__ bool wait_landed(uint32_t bar, uint32_t parity, int *err, int limit) {
  for (int it = 0; it < limit; it++) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  atomicExch(err, 1);
  return false;
}

// Shared memory of a reduction CTA.
struct Smem {
  double *Xs, *Vs;
  double (*part)[RT / 32][RB][3];  // [axis][warp][l][col]
  double *red;
  uint64_t *bar;
  __device__ __forceinline__ explicit Smem(double *dyn) {
    Xs = dyn;
    Vs = Xs + kXBlocks * SL;
    part = reinterpret_cast<double (*)[RT / 32][RB][3]>(Vs + 3 * VPAIR);
    red = Vs + 3 * VPAIR + 3 * (RT / 32) * RB * 3;
    bar = reinterpret_cast<uint64_t *>(red + RT / 32);
  }
};

// kBulk: the barrier of the copies, once per CTA (ends with a block barrier).
__device__ __forceinline__ void init_copies(const Smem &m) {
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(m.bar)));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncthreads();
}
// kBulk: starts the copies of a block triple into X and V.  Every thread has read
// what it needs of the blocks before (a block barrier lies between).  One
// copy per thread, spread over the warps: X block c = 6 g + q, then the VOE
// tiles.
__device__ __forceinline__ void start_copies(int nu, int no, int64_t NP, const TupleDev &t,
                                             const double *__restrict__ vb, int S0, int S1, int S2, const Smem &m) {
  const int tid = threadIdx.x, nb = nb_of(nu);
  const int nx = t.kind == kIJK ? 18 : 12;  // X blocks: three GEMM outputs, or a degenerate tuple's two
  const uint32_t sbar = (uint32_t)__cvta_generic_to_shared(m.bar);
  int slot[6];
  orbit_slots(S0, S1, S2, slot);
  auto Sm = [&](int q) { return sel3(q, S0, S1, S2); };
  if (tid == 0) {
    int nq = 0;
#pragma unroll
    for (int q = 0; q < 6; q++) nq += slot[q] == q;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sbar),
                 "r"((uint32_t)(nx / 6 * nq * SL * 8 + kVTiles * VTILE * 8))
                 : "memory");
  }
  const int c = (tid >> 5) + (tid & 31) * (RT / 32);
  if (c < nx) {
    const int q = c % 6;
    int sq = 0, O0 = 0, O1 = 0, O2 = 0;
#pragma unroll
    for (int p = 0; p < 6; p++)
      if (p == q) {
        sq = slot[p];
        O0 = Sm(pm(p, 0));
        O1 = Sm(pm(p, 1));
        O2 = Sm(pm(p, 2));
      }
    if (sq == q) {
      const double *src = sel3(c / 6, t.x[0], t.x[1], t.x[2]) + xblock_base(O0, O1, O2, nu, NP);
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              (uint32_t)__cvta_generic_to_shared(m.Xs + c * SL)),
          "l"(src), "r"(SL * 8), "r"(sbar)
          : "memory");
    }
  } else if (c < nx + kVTiles) {
    const int v = c - nx;
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            (uint32_t)__cvta_generic_to_shared(m.Vs + v * VTILE)),
        "l"(vb + voe_tile(v, no, nb, t, S0, S1, S2)), "r"(VTILE * 8), "r"(sbar)
        : "memory");
  }
}
// kBulk: waits for the copies of the parity's round.  False (for the whole CTA)
// when `limit` polls ran out: the error word is set, the copies have had the
// full limit to land, and the CTA must return.
__device__ __forceinline__ bool copies_landed(const Smem &m, uint32_t parity, int *err, int limit) {
  const uint32_t sbar = (uint32_t)__cvta_generic_to_shared(m.bar);
  const bool ok = wait_landed(sbar, parity, err, limit);
  if (__syncthreads_and(ok)) return true;
  wait_landed(sbar, parity, err, kReduceWaitLimit);
  return false;
}

// kRows: starts the copies of a block triple into X and V, 16 bytes a thread at a
// time: a row (p,q) of an X block is 64 contiguous bytes (NP is a multiple of 8),
// so an X block is one copy of every thread.  Rows of indices >= nu become zero.
// The barriers as for start_copies; rows_landed waits.  With one plain load a thread
// and element before each triple's arithmetic a kept-W forward took 33.2 ms at
// no12-nu120 and 54.0 at no10-nu160, 28.0 and 47.4 so.
__device__ __forceinline__ void start_rows(int nu, int no, int64_t NP, const TupleDev &t,
                                           const double *__restrict__ vb, int S0, int S1, int S2, const Smem &m) {
  static_assert(RT == 4 * RB * RB, "a thread per 16 bytes of an X block");
  const int tid = threadIdx.x, nb = nb_of(nu), ng = t.kind == kIJK ? 3 : 2;
  const int u0 = tid >> 5, u1 = (tid >> 2) & 7, off = 8 * (tid >> 2) + 2 * (tid & 3);
  auto cp16 = [](double *dst, const double *src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(ok ? 16 : 0)
                 : "memory");
  };
  int slot[6];
  orbit_slots(S0, S1, S2, slot);
#pragma unroll
  for (int q = 0; q < 6; q++) {
    if (slot[q] != q) continue;
    const int O0 = sel3(pm(q, 0), S0, S1, S2), O1 = sel3(pm(q, 1), S0, S1, S2), O2 = sel3(pm(q, 2), S0, S1, S2);
    const int xp = RB * O0 + u0, xq = RB * O1 + u1;
    const bool ok = xp < nu && xq < nu;
    const int64_t e = ok ? ((int64_t)xp * nu + xq) * NP + RB * O2 + 2 * (tid & 3) : 0;
    for (int g = 0; g < ng; g++) cp16(m.Xs + (6 * g + q) * SL + off, t.x[g] + e, ok);
  }
  for (int c = tid; c < kVTiles * VTILE / 2; c += RT)
    cp16(m.Vs + 2 * c, vb + voe_tile(c / (VTILE / 2), no, nb, t, S0, S1, S2) + 2 * (c % (VTILE / 2)), true);
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void rows_landed() {
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}

// One unordered block triple {A<=B<=C}, its X and V in shared memory.  Each thread
// evaluates two orbits -- the six index permutations of one (a,b,c) of block
// (A,B,C) share six W values and one denominator -- and accumulates E[4] and
// the v1 updates of all six elements; next() runs once every read of X and V
// is done (it may hold block barriers), then the fixed-order sums over the CTA.
//
// Entries of indices >= nu are whatever lies in the padding of the X blocks:
// only elements whose three indices are < nu are evaluated.
//
// What bounds it: the X traffic (3 nu^3 doubles a tuple).  The blocks reach
// shared memory by bulk copies in the order they lie in memory, so no thread
// spends an instruction on them; W is summed from them in registers as it is
// used.  Two CTAs per SM (97 KB each) walk over the block triples, the next
// triple's copies started before the sums of the last.  At no24-nu320 (3-digit X)
// a launch took 245 us when threads staged W through registers term by term
// (four CTAs per SM, 1740 instructions a warp), 203 us with one CTA per block
// triple on bulk copies, 181 us now.
template <int KIND, class Next>
__device__ __forceinline__ void reduce_compute(int nu, const TupleDev &t, const double *__restrict__ eh,
                                               const double *__restrict__ ep, const int S0, const int S1,
                                               const int S2, double *__restrict__ xpart_slot,
                                               double *__restrict__ vpart, const Smem &m, Next next) {
  constexpr int NTERM = KIND == kIJK ? 3 : 4, NG = KIND == kIJK ? 3 : 2;
  double *Xs = m.Xs, *Vs = m.Vs, *red = m.red;
  auto part = m.part;
  const int tid = threadIdx.x;
  int slot[6];
  orbit_slots(S0, S1, S2, slot);

  const double dijk = eh[t.i] + eh[t.j] + eh[t.k];
  double x3 = 0.0;
  double accA[3] = {0.0, 0.0, 0.0}, accB[3] = {0.0, 0.0, 0.0}, accC[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
  const int lc0 = orbit_coords(tid);
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int lc[3] = {lc0 & 7, (lc0 >> 3) & 7, (lc0 >> 6) ^ (4 * e)};
    const int l0 = lc[0], l1 = lc[1], l2 = lc[2];
    const int a = RB * S0 + l0, b = RB * S1 + l1, c = RB * S2 + l2;
    bool take = a < nu && b < nu && c < nu && !(a == b && b == c);  // W_aaa = 0 (ZEROT3)
    if (S0 == S1 && l0 > l1) take = false;  // the orbit is counted from its a<=b member
    if (S1 == S2 && l1 > l2) take = false;  // ... and from its b<=c member
    if (!take) continue;
    const double mult = (a == b || b == c) ? 0.5 : 1.0;  // three distinct elements, each met twice
    // W at permutation p of the element: X_g(y_al0, y_al1, y_al2) of y = x o p
    // is the entry of X_g at permutation p o al
    double w[6];
    {
      double xv[NG][6];
#pragma unroll
      for (int g = 0; g < NG; g++)
#pragma unroll
        for (int q = 0; q < 6; q++)
          xv[g][q] = Xs[(6 * g + slot[q]) * SL + 64 * lc[pm(q, 0)] + 8 * lc[pm(q, 1)] + lc[pm(q, 2)]];
#pragma unroll
      for (int p = 0; p < 6; p++) {
        double s = 0.0;
#pragma unroll
        for (int term = 0; term < NTERM; term++) {
          const int q = pidx(pm(p, term_entry(KIND, term, 1)), pm(p, term_entry(KIND, term, 2)));
          const double v = xv[term_entry(KIND, term, 0)][q];
          s = term == 0 ? v : s + v;
        }
        w[p] = s;
      }
    }
    const double dinv = mult * __drcp_rn(dijk - (ep[a] + ep[b] + ep[c]));
    // E[4] of the six elements: sum_pi W_pi (8 W_pi - 4 (sum over the three
    // transposed roles) + 2 (the two cyclic roles)).  Transpositions flip the
    // parity of the permutation, cycles keep it, so with Ev / Od the sums of
    // W over the even / odd permutations this is
    //   6 sum_even (W - Ev/3)^2 + 6 sum_odd (W - Od/3)^2 + 4 (Ev - Od)^2.
    const double Ev = w[0] + w[3] + w[4], Od = w[1] + w[2] + w[5];
    const double e3 = Ev * (1.0 / 3.0), o3 = Od * (1.0 / 3.0);
    const double r0 = w[0] - e3, r3 = w[3] - e3, r4 = w[4] - e3;
    const double r1 = w[1] - o3, r2 = w[2] - o3, r5 = w[5] - o3;
    const double sq = fma(r5, r5, fma(r4, r4, fma(r3, r3, fma(r2, r2, fma(r1, r1, r0 * r0)))));
    const double g = Ev - Od;
    x3 = fma(fma(6.0, sq, 4.0 * (g * g)), dinv, x3);
    // v1: with d1 = W_abc - W_bac, d2 = W_bca - W_acb, d3 = W_cba - W_cab of
    // the element (each an even minus an odd permutation, D below) and the
    // combined planes V[yz] = 2 VOE(.,.,y,z) - VOE(.,.,z,y), the Z1..Z6 sums
    // of t1wt3.f90:80-85 are
    //   d1 V[jk] - d2 V[kj],   -d1 V[ik] - d3 V[ki],   d2 V[ij] + d3 V[ji];
    // every element reads the VOE entries those lines name, so no symmetry of
    // VOE is assumed.
    double D[3][3];  // D[e][o] = W(even perm e) - W(odd perm o), evens 0 3 4, odds 1 2 5
#pragma unroll
    for (int ie = 0; ie < 3; ie++)
#pragma unroll
      for (int io = 0; io < 3; io++) D[ie][io] = w[ie == 0 ? 0 : ie + 2] - w[io == 2 ? 5 : io + 1];
    auto diff = [&](int x, int y) {  // W_x - W_y for permutations of opposite parity
      const bool xe = x == 0 || x == 3 || x == 4;
      const int ev = xe ? x : y, od = xe ? y : x;
      const double v = D[ev == 0 ? 0 : ev - 2][od == 5 ? 2 : od - 1];
      return xe ? v : -v;
    };
    // tile entries of the three index pairs: (lo, hi) in orientation 0, (hi, lo) in 1
    const int rp[3] = {l1 + 8 * l2, l0 + 8 * l2, l0 + 8 * l1};
    const int rpT[3] = {l2 + 8 * l1, l2 + 8 * l0, l1 + 8 * l0};
#pragma unroll
    for (int first = 0; first < 3; first++) {
      // the two elements whose first index is x_first: pi = 2 first (second <
      // third, orientation 0) and 2 first + 1 (orientation 1); their VOE pair is
      // the other two coordinates
      double ci = 0.0, cj = 0.0, ck = 0.0;
#pragma unroll
      for (int flip = 0; flip < 2; flip++) {
        const int pi = 2 * first + flip;
        const double d1 = diff(compose(pi, 0), compose(pi, 2));
        const double d2 = diff(compose(pi, 3), compose(pi, 1));
        const double d3 = diff(compose(pi, 5), compose(pi, 4));
        const double *v = Vs + first * VPAIR + flip * VORI + (flip ? rpT[first] : rp[first]);
        ci = fma(d1, v[0 * VTILE], fma(-d2, v[1 * VTILE], ci));
        cj = fma(-d1, v[2 * VTILE], fma(-d3, v[3 * VTILE], cj));
        ck = fma(d2, v[4 * VTILE], fma(d3, v[5 * VTILE], ck));
      }
      if (first == 0) {
        accA[0] = fma(ci, dinv, accA[0]); accA[1] = fma(cj, dinv, accA[1]); accA[2] = fma(ck, dinv, accA[2]);
      } else if (first == 1) {
        accB[0] = fma(ci, dinv, accB[0]); accB[1] = fma(cj, dinv, accB[1]); accB[2] = fma(ck, dinv, accB[2]);
      } else {
        accC[e][0] = fma(ci, dinv, accC[e][0]); accC[e][1] = fma(cj, dinv, accC[e][1]);
        accC[e][2] = fma(ck, dinv, accC[e][2]);
      }
    }
  }
  next();
  // ---- fixed-order sums: over the lanes of equal l0 / l1 / l2 (orbit_coords),
  // then over the warps, each of which holds all eight values of every axis
  const int warp = tid >> 5, lane = tid & 31;
  const int l0 = lc0 & 7, l1 = (lc0 >> 3) & 7, l2 = lc0 >> 6;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    double va = accA[q], vbq = accB[q];
    double vc = accC[0][q] + __shfl_xor_sync(0xffffffffu, accC[1][q], 8);
    va += __shfl_xor_sync(0xffffffffu, va, 1);
    va += __shfl_xor_sync(0xffffffffu, va, 16);
    vbq += __shfl_xor_sync(0xffffffffu, vbq, 2);
    vbq += __shfl_xor_sync(0xffffffffu, vbq, 24);
    vc += __shfl_xor_sync(0xffffffffu, vc, 4);
    vc += __shfl_xor_sync(0xffffffffu, vc, 16);
    if ((lane & 17) == 0) part[0][warp][l0][q] = va;
    if ((lane & 18) == 0) part[1][warp][l1][q] = vbq;
    if ((lane & 20) == 0) part[2][warp][l2][q] = vc;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) x3 += __shfl_down_sync(0xffffffffu, x3, off);
  if (lane == 0) red[warp] = x3;
  __syncthreads();

  if (tid == RT - 1) {
    double sum = 0.0;
#pragma unroll
    for (int w2 = 0; w2 < RT / 32; w2++) sum += red[w2];
    *xpart_slot = sum;
  }
  // v1 partials: position pos (first of equal blocks) collects every coordinate m
  // whose block equals it; written to vslab[X][l][col][q], q = the pair of the
  // other two blocks, so every (block, pair) slot has exactly one writer.
  if (tid < 72) {
    const int pos = tid / 24, l = (tid / 3) % 8, col = tid % 3;
    const int posm[3] = {0, S1 == S0 ? 0 : 1, S2 == S0 ? 0 : (S2 == S1 ? 1 : 2)};
    if (sel3(pos, posm[0], posm[1], posm[2]) == pos) {
      double v = 0.0;
#pragma unroll
      for (int m = 0; m < 3; m++) {
        if (posm[m] != pos) continue;
#pragma unroll
        for (int w2 = 0; w2 < RT / 32; w2++) v += part[m][w2][l][col];
      }
      const int X = pos == 0 ? S0 : (pos == 1 ? S1 : S2);
      const int Y = pos == 0 ? S1 : S0, Z = pos == 2 ? S1 : S2;  // the other two, Y <= Z
      const int64_t npairs = (int64_t)nb_of(nu) * (nb_of(nu) + 1) / 2;
      const int64_t q = (int64_t)Z * (Z + 1) / 2 + Y;
      vpart[(((int64_t)X * RB + l) * 3 + col) * npairs + q] = v;
    }
  }
}

}  // namespace red
}  // namespace cct
