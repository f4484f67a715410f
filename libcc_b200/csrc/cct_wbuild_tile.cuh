// The FP64 W-build GEMM tile as a device function, shared by the per-tuple
// kernel (cct_wbuild_f64.cu) and the persistent batch kernel (cct_batch.cu).
// See cct_wbuild_f64.cu for the formulation and the reference lines.
#pragma once
#include <type_traits>

#include "cct_internal.cuh"

namespace cct {
namespace wb {

constexpr int BM = 128, BK = kKB;
constexpr int WM = 32;
constexpr int NWARP = BM / WM;
constexpr int NT = NWARP * 32;
constexpr int STAGES = 3;
// Shared tiles are unpadded (16 doubles a row) with column c of row r stored
// at c ^ 4 (r & 3): the 64-bit fragment loads of a half-warp (rows g = 0..3,
// columns t = 0..3) then hit four disjoint 32-byte bank groups, and a CTA
// needs 64-75 KB, so three fit on an SM.
constexpr int LDS = BK;
__device__ __forceinline__ int swz(int r, int c) { return r * LDS + (c ^ ((r & 3) << 2)); }
constexpr int MF = WM / 16;

template <int BN, int TM = BM>
constexpr int smem_bytes() {
  return STAGES * (TM + BN) * LDS * 8 + TM * 2 * 4 + TM * 2 * 2 * 2;  // tiles, row offsets, packed (p, q)
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int src_bytes) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, int src_bytes) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// cp.async of 16 bytes (zero-filled when !live) to a shared address plus a constant.
template <int OFF>
__device__ __forceinline__ void cp_async16_at(uint32_t smem, const void *gmem, bool live) {
  asm volatile("cp.async.cg.shared.global [%0+%1], [%2], 16, %3;\n" ::"r"(smem), "n"(OFF), "l"(gmem),
               "r"(live ? 16 : 0));
}
template <int OFF>
__device__ __forceinline__ double lds_at(uint32_t smem) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1+%2];\n" : "=d"(v) : "r"(smem), "n"(OFF));
  return v;
}

__device__ __forceinline__ void dmma_16x8x4(double *d, double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// One TM x BN output tile (tile_m, tile_n) of one W-build GEMM job, TM/32
// warps of 32 rows each; every thread of the TM-thread CTA calls it.  Each
// KP-long half of the contraction holds KV = nu + no columns and zero
// padding, whose k4 steps are skipped.  smem_raw holds smem_bytes<BN, TM>().
// It starts with a barrier, so a persistent CTA can call it for consecutive
// tiles on the same shared memory.  blocked: X in 8 x 8 x 8 blocks
// (xblock_base; four lanes write one 64-byte row of a block, as in rows of NP).
template <int BN, int TM = BM>
__device__ __forceinline__ void wbuild_tile(const GemmJob &job, int nu, int64_t KP, int64_t KV, int64_t NP,
                                            int tile_m, int tile_n, bool blocked, unsigned char *smem_raw) {
  constexpr int BM = TM, NT = TM;
  constexpr int NF = BN / 8;
  double *As = reinterpret_cast<double *>(smem_raw);
  double *Bs = As + STAGES * BM * LDS;
  int *rowoff = reinterpret_cast<int *>(Bs + STAGES * BN * LDS);  // [2][BM] row index into E (or -1)
  int16_t *rowpq = reinterpret_cast<int16_t *>(rowoff + 2 * BM);   // [2][BM][2] (p, q) of the row (packed jobs)

  const int64_t M = (int64_t)nu * nu;
  const int64_t m0 = (int64_t)tile_m * BM;
  const int n0 = tile_n * BN;
  const int tid = threadIdx.x;

  __syncthreads();
  for (int r = tid; r < BM; r += NT) {
    const int64_t m = m0 + r;
    if (m < M) {
      const int p = (int)(m / nu), q = (int)(m - (int64_t)(m / nu) * nu);
      rowoff[r] = p * nu + q;
      rowoff[BM + r] = q * nu + p;
      rowpq[2 * r] = (int16_t)p;
      rowpq[2 * r + 1] = (int16_t)q;
      rowpq[2 * (BM + r)] = (int16_t)q;
      rowpq[2 * (BM + r) + 1] = (int16_t)p;
    } else {
      rowoff[r] = -1;
      rowoff[BM + r] = -1;
    }
  }
  __syncthreads();

  const int ktiles_half = (int)(KP / BK);
  const int ktiles = ktiles_half * job.nhalves;
  // Shared addresses are a per-thread base plus constants: the rows a thread
  // copies are NT/8 apart and the rows of a fragment 8 apart, multiples of 4, so
  // the XOR of a row (r & 3) is the same for all of them.  (Indexing the tiles
  // through swz() for every copy and fragment, with a K check per step, took
  // 464 instructions a warp and k-tile beside its 40 MMAs and kept the FP64 pipe
  // at 0.84: one tuple took 708 us at no16-nu200 and 4.11 ms at no24-nu320, 631 us
  // and 3.95 ms now.)
  constexpr int RS = LDS * 8;               // bytes of a row
  constexpr int A_ST = BM * RS, B_ST = BN * RS;  // bytes of a stage
  const uint32_t sA = (uint32_t)__cvta_generic_to_shared(As), sB = (uint32_t)__cvta_generic_to_shared(Bs);
  const int cr = tid >> 3, chunk = tid & 7;  // a thread copies 16-byte chunk `chunk` of rows cr, cr + NT/8, ...
  const uint32_t cdst = (uint32_t)swz(cr, chunk * 2) * 8;
  const uint32_t kp8 = (uint32_t)KP * 8;

  auto load_stage = [&](int stage, int kt) {
    const int h = kt >= ktiles_half;
    const int64_t k0 = (int64_t)(kt - h * ktiles_half) * BK;
    const double *abase = h ? job.a1 : job.a0;
    const double *bbase = h ? job.b1 : job.b0;
    if (!job.packed) {
      const uint32_t dst = sA + stage * A_ST + cdst;
      const char *src0 = reinterpret_cast<const char *>(abase + k0 + chunk * 2);
      const int *ro = rowoff + h * BM + cr;
      auto rows = [&](auto self, auto ic) {
        constexpr int I = decltype(ic)::value;
        if constexpr (I < 8) {
          const int r = ro[I * (NT / 8)];
          cp_async16_at<I *(NT / 8) * RS>(dst, src0 + (uint64_t)(uint32_t)max(r, 0) * kp8, r >= 0);
          self(self, std::integral_constant<int, I + 1>{});
        }
      };
      static_assert(BM == NT, "eight passes of NT/8 rows");
      rows(rows, std::integral_constant<int, 0>{});
    } else {
      double *as = As + stage * BM * LDS;
      // the row's E values gathered one double at a time: the packed
      // triangle holds (k q | p x) at tri(k, q) of column p, the -T2 rows the
      // k >= nu part; past nu + no the row is zero
      const double *tbase = h ? job.t1 : job.t0;
      const int64_t nutr = (int64_t)nu * (nu + 1) / 2;
      const int nov = (int)(KV - nu);
#pragma unroll
      for (int rr = tid >> 3; rr < BM; rr += NT / 8) {
        const int ro = rowoff[h * BM + rr];
        const int pr = rowpq[2 * (h * BM + rr)], qr = rowpq[2 * (h * BM + rr) + 1];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int64_t k = k0 + chunk * 2 + e;
          const double *src = abase;
          int bytes = 0;
          if (ro >= 0 && k < nu) {
            src = abase + (int64_t)pr * nutr + (k >= qr ? k * (k + 1) / 2 + qr : (int64_t)qr * (qr + 1) / 2 + k);
            bytes = 8;
          } else if (ro >= 0 && k < KV) {
            src = tbase + (int64_t)ro * nov + (k - nu);
            bytes = 8;
          }
          cp_async8(as + swz(rr, chunk * 2 + e), src, bytes);
        }
      }
    }
    {
      const uint32_t dst = sB + stage * B_ST + cdst;
      const char *src = reinterpret_cast<const char *>(bbase + (int64_t)(n0 + cr) * KP + k0 + chunk * 2);
      const int64_t step = (int64_t)(NT / 8) * kp8;
      auto rows = [&](auto self, auto ic) {
        constexpr int I = decltype(ic)::value;
        if constexpr (I * (NT / 8) < BN) {
          if (I * (NT / 8) + NT / 8 <= BN || cr < BN - I * (NT / 8))
            cp_async16_at<I *(NT / 8) * RS>(dst, src + I * step, true);
          self(self, std::integral_constant<int, I + 1>{});
        }
      };
      rows(rows, std::integral_constant<int, 0>{});
    }
  };

  const int warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;

  double acc[MF][NF][4];
#pragma unroll
  for (int i = 0; i < MF; i++)
#pragma unroll
    for (int j = 0; j < NF; j++)
#pragma unroll
      for (int r = 0; r < 4; r++) acc[i][j][r] = 0.0;

#pragma unroll
  for (int s = 0; s < STAGES - 1; s++) {
    if (s < ktiles) load_stage(s, s);
    cp_async_commit();
  }

  // fragment bases of the four k4 steps: row g, column (4 s) ^ 4 (g & 3) + t
  const uint32_t fA = sA + ((warp * WM + g) * LDS + t) * 8, fB = sB + (g * LDS + t) * 8;
  const uint32_t gx = (uint32_t)(g & 3) * 32;
  int stage = 0, fill = STAGES - 1;
  for (int kt = 0; kt < ktiles; kt++) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    {
      const int nk = kt + STAGES - 1;
      if (nk < ktiles) load_stage(fill, nk);
      cp_async_commit();
      if (++fill == STAGES) fill = 0;
    }
    auto step = [&](int s) {
      const uint32_t pa = fA + stage * A_ST + ((uint32_t)(32 * s) ^ gx);
      const uint32_t pb = fB + stage * B_ST + ((uint32_t)(32 * s) ^ gx);
      double af[MF][2], bf[NF];
      auto fa = [&](auto self, auto ic) {
        constexpr int I = decltype(ic)::value;
        if constexpr (I < MF) {
          af[I][0] = lds_at<I * 16 * RS>(pa);
          af[I][1] = lds_at<(I * 16 + 8) * RS>(pa);
          self(self, std::integral_constant<int, I + 1>{});
        }
      };
      auto fb = [&](auto self, auto ic) {
        constexpr int J = decltype(ic)::value;
        if constexpr (J < NF) {
          bf[J] = lds_at<J * 8 * RS>(pb);
          self(self, std::integral_constant<int, J + 1>{});
        }
      };
      fa(fa, std::integral_constant<int, 0>{});
      fb(fb, std::integral_constant<int, 0>{});
#pragma unroll
      for (int i = 0; i < MF; i++)
#pragma unroll
        for (int j = 0; j < NF; j++) dmma_16x8x4(acc[i][j], af[i][0], af[i][1], bf[j]);
    };
    // columns of this k-tile below nu + no; the k4 steps past them multiply zero padding
    const int kv = (int)(KV - (int64_t)(kt < ktiles_half ? kt : kt - ktiles_half) * BK);
    if (kv > BK - 4) {
#pragma unroll
      for (int s = 0; s < BK / 4; s++) step(s);
    } else {
#pragma unroll 1
      for (int s = 0; 4 * s < kv; s++) step(s);
    }
    if (++stage == STAGES) stage = 0;
  }
  cp_async_wait<0>();

  // epilogue: X[(p*nu+q)*NP + s], or its place in the blocks
#pragma unroll
  for (int i = 0; i < MF; i++) {
#pragma unroll
    for (int half = 0; half < 2; half++) {
      const int64_t m = m0 + warp * WM + i * 16 + g + half * 8;
      if (m >= M) continue;
      double *orow = job.out + m * NP + n0 + 2 * t;
      int64_t step = 8;
      if (blocked) {
        const int r = warp * WM + i * 16 + g + half * 8, p = rowpq[2 * r], q = rowpq[2 * r + 1];
        orow = job.out + xblock_base(p >> 3, q >> 3, n0 >> 3, nu, NP) + ((p & 7) * 8 + (q & 7)) * 8 + 2 * t;
        step = 512;
      }
#pragma unroll
      for (int j = 0; j < NF; j++) {
        double2 v = make_double2(acc[i][j][2 * half], acc[i][j][2 * half + 1]);
        *reinterpret_cast<double2 *>(orow + j * step) = v;
      }
    }
  }
}

}  // namespace wb
}  // namespace cct
