// Alpha-single x beta-single terms of sigma on densely connected string sets, one small FP64
// tensor-core product per alpha row.
//
//   sigma[Ia, Ib] += sum_{(Ja, pq, sa) in S_a(Ia)} sum_{(Jb, rs, sb) in S_b(Ib)} sa sb (pq|rs) C[Ja, Jb]
//
// (MultTPBThrust::run, tpb/mult_thrust.h:1172-1582; sbd::mult, tpb/mult.h:625-881.)  For one alpha
// row the inner sum over its K singles does not depend on Ib but only on the pair rs and on Jb:
//
//   P[rs, Jb] = sum_i (sa_i (pq_i|rs)) C[Ja_i, Jb],      sigma[Ia, Ib] += sum sb P[rs, Jb],
//
// a product of an M x K by a K x nb matrix, M the distinct unordered pairs {r,s} of the beta singles
// ((pq|rs) = (pq|sr): 153 at 18 orbitals), followed by one gather per beta single instead of one
// multiply-add per pair of singles.  The product computes M values per Jb of which as many as Jb has
// singles are used (39 of 153 on an 18-orbital molecular set of 4,041 strings), so it does
// M / (singles per string) times the multiply-adds of the direct loop, in registers and on the FP64
// tensor pipe instead of through two shared-memory reads each.
#include <algorithm>
#include <bitset>
#include <cmath>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "tc_util.cuh"
#include "tpb_common.cuh"

namespace sbdtpb {
namespace {

constexpr int kCols = 32;        // ket columns Jb per step
constexpr int kGemmWarps = 12;   // warps 0..11: the product
constexpr int kLoadWarp = 12;    // warp 12: C into shared memory
constexpr int kGatherWarps = 3;  // warps 13..15: the beta singles
constexpr int kThreads = 32 * (kGemmWarps + 1 + kGatherWarps);
constexpr int kStages = 3;       // ring of C blocks
constexpr int kMaxPBufs = 4;     // buffers of P: as many as fit, at least 2
constexpr int kMaxK = 64;        // alpha singles per group (8 double k-steps of 8)
constexpr int kWarpBlocks = 2;   // 8-row blocks of P per product warp
constexpr int kMaxBlocks = kGemmWarps * kWarpBlocks;
constexpr int kRounds = 4;       // entries of a group of beta singles read side by side
constexpr int kIlp = 3;          // groups per lane read side by side
constexpr uint32_t kNoEntry = 0xffffffffu;

// Column n of row k of a staged C block, and of row m of P: rows are 32 elements without padding, the
// columns permuted so that the B fragments of a half warp (4 rows x 4 columns; of a warp, 4 x 8, in
// FP32) and the stores of a quarter warp's accumulators (2 rows x 8 columns; 4 x 8 in FP32) touch
// every bank once.
template <typename T>
__device__ __forceinline__ int b_pos(int k, int n) {
  return k * kCols + (n ^ ((k & 3) << (sizeof(T) == 8 ? 2 : 3)));
}
__host__ __device__ __forceinline__ int p_pos(int m, int n) { return m * kCols + (n ^ ((m & 3) << 3)); }

struct RowArgs {
  const uint32_t *rows;   // alpha rows with singles, most singles first
  const uint32_t *a_off;  // [na + 1] alpha singles
  const uint2 *a_ent;     // (ket Ja, +-(pq + 1)), per row ascending by the row of P of their pair
  const int32_t *pair_m;  // pair pq -> row of P of its unordered pair, -1 when no beta single has it
  const int32_t *m_pair;  // row of P -> pair
  const uint4 *hdr;       // per (pass, chunk, gather warp): (byte offset of its program, groups, rounds, byte offset of its entries)
  const unsigned char *prog;  // first entry of each round, Ib of each group, entries (see build_program)
  const double *eri;
  int L2, M;
  int passes, bpp;        // passes over the rows of P, 8-row blocks per pass
  uint32_t nchunks, nb;
  uint32_t pbufs;         // buffers of P
  uint32_t kcap;          // rows of the staged C block (a multiple of 8, at most kMaxK)
  uint32_t prog_cap;      // bytes of one program buffer
  int *err;               // pinned host memory: set when a wait expired
};

// Sums of rows that do not fit in shared memory (not kSig).
struct RowScratch {
  void *rows;       // [slots][nb]
  uint32_t *taken;  // [slots] whether a CTA has the row
  uint32_t slots;   // as many as CTAs are resident at a time
};

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};" : "+d"(c0), "+d"(c1) : "d"(a), "d"(b));
}
// v, its sign flipped when bit 15 of s is set
__device__ __forceinline__ double flip(double v, uint32_t s) {
  return __hiloint2double(__double2hiint(v) ^ (int)(s << 16), __double2loint(v));
}
__device__ __forceinline__ float flip(float v, uint32_t s) { return __int_as_float(__float_as_int(v) ^ (int)(s << 16)); }
// one element global -> shared, zero where !in
template <typename T>
__device__ __forceinline__ void cp_elem(T *dst, const T *src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"((int)sizeof(T)),
               "r"(in ? (int)sizeof(T) : 0)
               : "memory");
}
__device__ __forceinline__ void cp16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// arrives on the mbarrier once this thread's copies so far have landed
__device__ __forceinline__ void cp_arrive(uint32_t mbar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(mbar) : "memory");
}

struct Bars {
  uint64_t c_full[kStages], c_free[kStages], p_full[kMaxPBufs], p_free[kMaxPBufs];
};

// What bounds it: the FP64 tensor pipe (m8n8k4, 16 cycles each per quarter SM).  The warps run in
// three roles coupled only by mbarriers, so that the product warps drift apart and one's stores and
// waits lie under another's products (one barrier of all product warps per step: 16.0 ms where this
// takes 12.6).  The integral rows stay in registers for a whole pass over the columns.  The direct
// kernel took (ms, before -> here): 18 orbitals, 4,041 strings FP64 50.9 -> 12.6 (the products alone need
// 6.1 at the 36.5 TFLOP/s a register-only loop of these instructions reaches; product warps without
// the gather 8.4, gather without the products 6.8); 1,387 strings symmetric 2.10 -> 1.07; 24 orbitals,
// 5,514 strings FP32 symmetric 73.1 -> 31.6; 12-orbital full CI FP64 1.40 -> 0.43.  The error against
// 64-bit sums in another order went down (FP64 2.5e-16 -> 1.4e-16, FP32 6.8e-8 -> 4.1e-8 of sigma's norm).
//
// Shared memory: Bars, [kStages][kcap][32] of C, [pbufs][8 bpp][32] of P, per gather warp
// [2][prog_cap] of its program, and (kSig) one row of sums.  Rows of sums that do not fit (FP64 from about 10,000
// columns, FP32 35,000) lie in scratch rows, one per resident CTA, which stay in L2.  They are summed from zero
// too: added to sigma one by one, each term rounded at sigma's size (FP64 3.0e-16 of sigma's norm where this
// gives 1.4e-16, FP32 1.7e-7 and 4.4e-8).  Three scratch sums are loaded before the first is stored (20 orbitals,
// 14,000 strings FP64 263 -> 201 ms; 22 orbitals, 16,000 216 -> 172).
template <typename T, bool kSym, bool kSig>
__global__ void __launch_bounds__(kThreads, 1) ab_rows_kernel(RowArgs a, const T *__restrict__ C, T *__restrict__ sigma,
                                                              RowScratch sc) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t slot;
  Bars *bars = reinterpret_cast<Bars *>(smem);
  T *Bs = reinterpret_cast<T *>(smem + sizeof(Bars));
  T *Ps = Bs + (size_t)kStages * a.kcap * kCols;
  const uint32_t pbuf = 8 * a.bpp * kCols;
  unsigned char *prog_s = reinterpret_cast<unsigned char *>(Ps + a.pbufs * pbuf);
  T *sig_s = reinterpret_cast<T *>(prog_s + 2 * kGatherWarps * a.prog_cap);

  const uint32_t ia = a.rows[blockIdx.x];
  const uint32_t e0 = a.a_off[ia], K = a.a_off[ia + 1] - e0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ngroups = (K + kMaxK - 1) / kMaxK;
  auto addr = [](const uint64_t &b) { return tc::smem_addr(&b); };
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; i++) {
      tc::mbar_init(addr(bars->c_full[i]), 32);
      tc::mbar_init(addr(bars->c_free[i]), kGemmWarps);
    }
    for (int i = 0; i < kMaxPBufs; i++) {
      tc::mbar_init(addr(bars->p_full[i]), kGemmWarps);
      tc::mbar_init(addr(bars->p_free[i]), kGatherWarps);
    }
    tc::fence_mbar_init();
    if constexpr (!kSig) {
      // there are as many scratch rows as CTAs at a time, so one is free; give up after some rounds all the same
      uint32_t k = blockIdx.x % sc.slots, tries = 64 * sc.slots;
      while (atomicCAS(&sc.taken[k], 0u, 1u) != 0u && --tries) k = k + 1 < sc.slots ? k + 1 : 0;
      __threadfence();
      slot = tries ? k : sc.slots;
    }
  }
  __syncthreads();
  if constexpr (!kSig) {
    if (slot == sc.slots) {
      if (threadIdx.x == 0) *reinterpret_cast<volatile int *>(a.err) = 5;
      return;
    }
  }
  // every wait is bounded; an expired one is recorded and its warp leaves (the others' waits for it
  // then expire too)
  auto wait = [&](const uint64_t &b, uint32_t parity, int code) {
    if (tc::mbar_wait(addr(b), parity)) return true;
    *reinterpret_cast<volatile int *>(a.err) = code;
    return false;
  };

  if (warp < kGemmWarps) {
    double A[kWarpBlocks][kMaxK / 4];
    int kend[kWarpBlocks], kmax = 0;  // double k-steps of each block
    const int row = lane >> 2, q = lane & 3;
    // step; its stage of the ring and buffer of P, with their phases
    uint32_t s = 0, st = 0, ph = 0, pb = 0, pp = 0;
    for (uint32_t g = 0; g < ngroups; g++) {
      const uint32_t ge = e0 + g * kMaxK, kg = min((uint32_t)kMaxK, K - g * kMaxK);
      for (int pass = 0; pass < a.passes; pass++) {
        // this pass's rows of the integral matrix, as A fragments: block warp + 12 j holds rows
        // 8 (bpp pass + warp + 12 j) .. + 8 of P
        bool in[kWarpBlocks];
        int m[kWarpBlocks], used[kWarpBlocks];
        const double *erow[kWarpBlocks];
#pragma unroll
        for (int j = 0; j < kWarpBlocks; j++) {
          const int blk = warp + kGemmWarps * j;
          m[j] = 8 * (a.bpp * pass + blk) + row;
          in[j] = blk < a.bpp && m[j] < a.M;
          erow[j] = a.eri + (in[j] ? a.m_pair[m[j]] : 0);
          used[j] = 0;
        }
#pragma unroll
        for (int kk = 0; kk < kMaxK / 4; kk++) {
          const uint32_t i = 4 * kk + q;
          const int32_t ps = i < kg ? (int32_t)a.a_ent[ge + i].y : 0;
          const int pq = (ps > 0 ? ps : -ps) - 1;
          const int mi = kSym && ps ? a.pair_m[pq] : 0;
#pragma unroll
          for (int j = 0; j < kWarpBlocks; j++) {
            double v = 0.0;
            // symmetric: the half of the terms whose transposes are the other half, pairs rs above
            // pq and rs = pq at half weight (entries ascend by pair_m, so a block's later ones are
            // all zero)
            if (in[j] && ps && (!kSym || mi <= m[j])) {
              v = erow[j][(size_t)pq * a.L2];
              if (ps < 0) v = -v;
              if (kSym && mi == m[j]) v *= 0.5;
              used[j] = kk / 2 + 1;
            }
            A[j][kk] = v;
          }
        }
        kmax = 0;
#pragma unroll
        for (int j = 0; j < kWarpBlocks; j++) {
          kend[j] = (int)__reduce_max_sync(0xffffffffu, (unsigned)used[j]);
          kmax = max(kmax, kend[j]);
        }
        for (uint32_t chunk = 0; chunk < a.nchunks; chunk++, s++) {
          if (!wait(bars->c_full[st], ph, 1)) return;
          double acc[kWarpBlocks][kCols / 8][2];
#pragma unroll
          for (int j = 0; j < kWarpBlocks; j++)
#pragma unroll
            for (int n = 0; n < kCols / 8; n++) acc[j][n][0] = acc[j][n][1] = 0.0;
          // B fragment (k = 4 kk + q, n = 8 nt + row) at b_pos: the permutation is one of the 8-column
          // tiles (tile ^ h), in FP64 also of the columns within a tile
          const int h = sizeof(T) == 8 ? q >> 1 : q;
          const T *b = Bs + (size_t)st * a.kcap * kCols + q * kCols + (sizeof(T) == 8 ? row ^ ((q & 1) << 2) : row);
          const T *bt[kCols / 8];
#pragma unroll
          for (int n = 0; n < kCols / 8; n++) bt[n] = b + 8 * (n ^ h);
#pragma unroll
          for (int kp = 0; kp < kMaxK / 8; kp++) {
            if (kp < kmax) {
              double bf[2][kCols / 8];
#pragma unroll
              for (int i = 0; i < 2; i++)
#pragma unroll
                for (int n = 0; n < kCols / 8; n++)
                  bf[i][n] = (double)bt[n][(8 * kp + 4 * i) * kCols];
#pragma unroll
              for (int j = 0; j < kWarpBlocks; j++)
                if (kp < kend[j]) {
#pragma unroll
                  for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int n = 0; n < kCols / 8; n++) dmma(acc[j][n][0], acc[j][n][1], A[j][2 * kp + i], bf[i][n]);
                }
            }
          }
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(addr(bars->c_free[st]));
          if (++st == kStages) st = 0, ph ^= 1;
          if (s >= a.pbufs && !wait(bars->p_free[pb], pp ^ 1, 2)) return;
          T *p = Ps + pb * pbuf;
#pragma unroll
          for (int j = 0; j < kWarpBlocks; j++) {
            const int blk = warp + kGemmWarps * j;
            if (blk < a.bpp) {
#pragma unroll
              for (int n = 0; n < kCols / 8; n++) {
                T *d = p + p_pos(8 * blk + row, 8 * n + 2 * q);
                if constexpr (sizeof(T) == 8) *reinterpret_cast<double2 *>(d) = make_double2(acc[j][n][0], acc[j][n][1]);
                else *reinterpret_cast<float2 *>(d) = make_float2((float)acc[j][n][0], (float)acc[j][n][1]);
              }
            }
          }
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(addr(bars->p_full[pb]));
          if (++pb == a.pbufs) pb = 0, pp ^= 1;
        }
      }
    }
  } else if (warp == kLoadWarp) {
    // C[Ja_i, chunk] -> row i of the stage, lane n the column n; zero past the row's end and from K up
    // to a multiple of 8
    uint32_t st = 0, ph = 0, s = 0;
    for (uint32_t g = 0; g < ngroups; g++) {
      const uint32_t ge = e0 + g * kMaxK, kg = min((uint32_t)kMaxK, K - g * kMaxK), kpad = (kg + 7) & ~7u;
      const uint32_t ket0 = lane < kg ? a.a_ent[ge + lane].x : 0, ket1 = lane + 32 < kg ? a.a_ent[ge + 32 + lane].x : 0;
      for (int pass = 0; pass < a.passes; pass++)
        for (uint32_t chunk = 0; chunk < a.nchunks; chunk++, s++) {
          if (s >= kStages && !wait(bars->c_free[st], ph ^ 1, 3)) {
            cp_wait<0>();  // the copies in flight
            return;
          }
          T *dst = Bs + (size_t)st * a.kcap * kCols;
          const uint32_t col = chunk * kCols + lane;
          const bool cin = col < a.nb;
          const T *src = C + (cin ? col : 0);
#pragma unroll 4
          for (uint32_t i = 0; i < kpad; i++) {
            const uint32_t ket = __shfl_sync(0xffffffffu, i < 32 ? ket0 : ket1, i & 31);
            const bool in = cin && i < kg;
            cp_elem(dst + b_pos<T>(i, lane), src + (size_t)(in ? ket : 0) * a.nb, in);
          }
          cp_arrive(addr(bars->c_full[st]));
          if (++st == kStages) st = 0, ph ^= 1;
        }
    }
    cp_wait<0>();
  } else {
    // gather warp gw owns the columns Ib with (Ib / 32) % 3 == gw: its own program, no other warp
    // touches its part of the sigma row
    const int gw = warp - kLoadWarp - 1;
    const uint32_t per_group = (uint32_t)a.passes * a.nchunks, steps = ngroups * per_group;
    T *srow = sigma + (size_t)ia * a.nb;
    T *scr = nullptr;
    if constexpr (kSig) {
      for (uint32_t c = 32 * gw + lane; c < a.nb; c += 32 * kGatherWarps) sig_s[c] = T(0);
    } else {
      scr = reinterpret_cast<T *>(sc.rows) + (size_t)slot * a.nb;
      for (uint32_t c = 32 * gw + lane; c < a.nb; c += 32 * kGatherWarps) scr[c] = T(0);
    }
    unsigned char *own = prog_s + 2 * gw * a.prog_cap;
    auto fetch = [&](uint32_t cell, uint32_t s) {
      const uint4 h = a.hdr[cell * kGatherWarps + gw];
      const uint32_t bytes = a.hdr[cell * kGatherWarps + gw + 1].x - h.x;  // multiples of 16
      unsigned char *dst = own + (s & 1) * a.prog_cap;
      for (uint32_t o = lane * 16; o < bytes; o += 32 * 16) cp16(dst + o, a.prog + (size_t)h.x + o);
      cp_commit();
      return h;
    };
    uint32_t cell = 0, pb = 0, pp = 0;
    uint4 h = fetch(0, 0);
    for (uint32_t s = 0; s < steps; s++) {
      const uint4 cur = h;
      cell = cell + 1 < per_group ? cell + 1 : 0;
      __syncwarp();
      if (s + 1 < steps) {
        h = fetch(cell, s + 1);
        cp_wait<1>();
      } else {
        cp_wait<0>();
      }
      __syncwarp();
      if (!wait(bars->p_full[pb], pp, 4)) break;
      const uint32_t ng = cur.y, rounds = cur.z;  // rounds: a multiple of kRounds
      const unsigned char *pr = own + (s & 1) * a.prog_cap;
      const uint16_t *first = reinterpret_cast<const uint16_t *>(pr);  // [rounds + kRounds]
      const uint32_t *ibs = reinterpret_cast<const uint32_t *>(first + rounds + kRounds);
      const uint16_t *ent = reinterpret_cast<const uint16_t *>(pr + cur.w);
      const T *p = Ps + pb * pbuf;
      // the first kRounds entries of kIlp groups side by side: twelve chains of two dependent reads
      uint32_t f[kRounds + 1];
#pragma unroll
      for (int i = 0; i <= kRounds; i++) f[i] = first[i];
      for (uint32_t t = lane; t < ng; t += 32 * kIlp) {
        uint32_t e[kIlp][kRounds];
        T v[kIlp][kRounds];
        uint32_t gib[kIlp];
        T gs[kIlp];
        if constexpr (!kSig) {
          // (the Ib of a cell's groups are distinct)
#pragma unroll
          for (int j = 0; j < kIlp; j++) {
            gib[j] = t + 32 * j < ng ? ibs[t + 32 * j] : ibs[0];
            gs[j] = scr[gib[j]];
          }
        }
#pragma unroll
        for (int j = 0; j < kIlp; j++)
#pragma unroll
          for (int i = 0; i < kRounds; i++)
            e[j][i] = t + 32 * j < f[i + 1] - f[i] ? ent[f[i] + t + 32 * j] : kNoEntry;
#pragma unroll
        for (int j = 0; j < kIlp; j++)
#pragma unroll
          for (int i = 0; i < kRounds; i++)
            v[j][i] = e[j][i] != kNoEntry ? flip(p[e[j][i] & 0x7fffu], e[j][i] & 0x8000u) : T(0);
#pragma unroll
        for (int j = 0; j < kIlp; j++)
          if (t + 32 * j < ng) {
            const uint32_t ib = ibs[t + 32 * j];
            const T sum = (v[j][0] + v[j][1]) + (v[j][2] + v[j][3]);
            if constexpr (kSig) sig_s[ib] += sum;
            else scr[gib[j]] = gs[j] + sum;
          }
      }
      // the few groups with more entries (the same lane has them)
      for (uint32_t rd = kRounds; rd < rounds; rd += kRounds) {
#pragma unroll
        for (int i = 0; i <= kRounds; i++) f[i] = first[rd + i];
        for (uint32_t t = lane; t < f[1] - f[0]; t += 32) {
          T v[kRounds];
#pragma unroll
          for (int i = 0; i < kRounds; i++) {
            const uint32_t e = t < f[i + 1] - f[i] ? ent[f[i] + t] : kNoEntry;
            v[i] = e != kNoEntry ? flip(p[e & 0x7fffu], e & 0x8000u) : T(0);
          }
          const uint32_t ib = ibs[t];
          const T sum = (v[0] + v[1]) + (v[2] + v[3]);
          if constexpr (kSig) sig_s[ib] += sum;
          else scr[ib] += sum;
        }
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(addr(bars->p_free[pb]));
      if (++pb == a.pbufs) pb = 0, pp ^= 1;
    }
    cp_wait<0>();
    __syncwarp();
    if constexpr (kSig) {
      for (uint32_t c = 32 * gw + lane; c < a.nb; c += 32 * kGatherWarps)
        srow[c] = (T)((double)srow[c] + (double)sig_s[c]);
    } else {
      for (uint32_t c0 = 32 * gw + lane; c0 < a.nb; c0 += 8 * 32 * kGatherWarps) {
        T o[8], v[8];  // eight columns' loads side by side
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const uint32_t c = c0 + i * 32 * kGatherWarps;
          o[i] = c < a.nb ? srow[c] : T(0);
          v[i] = c < a.nb ? scr[c] : T(0);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const uint32_t c = c0 + i * 32 * kGatherWarps;
          if (c < a.nb) srow[c] = (T)((double)o[i] + (double)v[i]);
        }
      }
      // the three warps are done with the scratch row
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kGatherWarps) : "memory");
      if (threadIdx.x == 32 * (kLoadWarp + 1)) {
        __threadfence();
        atomicExch(&sc.taken[slot], 0u);
      }
    }
  }
}

size_t rows_smem(const ABRows &r, size_t size, size_t nb, bool sig, uint32_t pbufs) {
  return sizeof(Bars) + size * kStages * r.kcap * kCols + size * pbufs * 8 * r.bpp * kCols +
         2 * kGatherWarps * (size_t)r.prog_cap + (sig ? size * nb : 0);
}

template <typename T, bool kSym, bool kSig>
int launch_rows(sbd_tpb_handle *h, RowArgs a, const T *C, T *sigma) {
  a.pbufs = 2;
  while (a.pbufs < kMaxPBufs && rows_smem(h->abr, sizeof(T), a.nb, kSig, a.pbufs + 1) <= h->smem_optin) a.pbufs++;
  const size_t smem = rows_smem(h->abr, sizeof(T), a.nb, kSig, a.pbufs);
  const auto kern = ab_rows_kernel<T, kSym, kSig>;
  TPB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if constexpr (!kSig) {
    int ctas = 0;
    TPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, kern, kThreads, smem));
    if ((uint32_t)(ctas * h->num_sms) > h->abr.slots) return fail(SBD_TPB_ERR_CUDA, "alpha-beta row kernel: scratch rows");
  }
  kern<<<h->abr.nrows, kThreads, smem, h->stream>>>(a, C, sigma, RowScratch{h->abr.scratch, h->abr.taken, h->abr.slots});
  TPB_LAUNCHED(h);
  return SBD_TPB_OK;
}

// Status words of the kernel's bounded waits, from one pinned page per device: pinning memory takes 1.3 ms
// (and unpinning 0.4), as long as twenty sigmas of a small problem.  A word belongs to one handle from its
// first program to its end; when all 1,024 of a page are taken a handle pins its own.
class StatusPage {
 public:
  int *get() {
    std::lock_guard<std::mutex> lock(m_);
    cudaPointerAttributes at;
    if (page_ && (cudaPointerGetAttributes(&at, page_) != cudaSuccess || at.type != cudaMemoryTypeHost))
      page_ = nullptr;  // the program reset the device: the page went with its context
    if (!page_ && cudaHostAlloc(&page_, sizeof(int) * kWords, cudaHostAllocMapped) == cudaSuccess) taken_.reset();
    size_t k = 0;
    while (k < kWords && taken_[k]) k++;
    int *w = nullptr;
    if (page_ && k < kWords) {
      taken_[k] = true;
      w = page_ + k;
    } else if (cudaHostAlloc(&w, sizeof(int), cudaHostAllocMapped) != cudaSuccess) {
      w = nullptr;
    }
    cudaGetLastError();
    if (w) *w = 0;
    return w;
  }
  void put(int *w) {
    std::lock_guard<std::mutex> lock(m_);
    if (page_ && w >= page_ && w < page_ + kWords) taken_[w - page_] = false;
    else cudaFreeHost(w);
  }

 private:
  static constexpr size_t kWords = 1024;
  std::mutex m_;
  int *page_ = nullptr;
  std::bitset<kWords> taken_;
};
constexpr int kMaxDevices = 64;
StatusPage g_status[kMaxDevices];

}  // namespace

void ab_rows_free(sbd_tpb_handle *h) {
  ABRows &r = h->abr;
  if (r.block) cudaFree(r.block);
  if (r.err) g_status[h->device % kMaxDevices].put(r.err);
  r = ABRows();
}

// Which kernel: the multiply-adds of the products (padded) over those of the direct loop, which does each of
// them through two shared-memory reads.  The rows kernel runs up to these ratios.  Direct / rows time, FP64
// general, symmetric, FP32 general, symmetric: 26 orbitals, 120 molecular strings (ratio 10) 4.1, 4.1, 3.4, 3.8; 18
// orbitals, 4,041 (4) 4.1, 3.9, 3.2, 3.1; sampled strings: 20 orbitals, 6,000 (10) 2.6, 2.4, 2.1, 1.9; 21, 6,000 (14.9)
// 1.8, 1.6, 1.1, 1.0; 20, 3,500 (16.7) 1.37, 1.32, 1.10, 1.06; 22, 13,000 (17.1) 1.93, 1.64, 1.21, 1.07; 22, 11,000
// (19.8) 1.57, 1.34, 1.04, 0.92; 20, 3,000 (19.9) 1.14, 1.06, 0.94, 0.88; 20, 2,700 (22.6) 0.92, 0.87, 0.78, 0.73; 22,
// 8,000 (26.6) 1.07, 0.92, 0.71, 0.63.  Sets with one or two singles a string lie above 100, where the padded
// products lose tenfold.  FP32 has the lower line: its vectors pay FP64 products.
constexpr double kMostRatio64 = 20.0, kMostRatio32 = 17.0;

// The row program where the ratio is at most `most`; ready stays false where it is not or the program does not fit.
static int build_program(sbd_tpb_handle *h, SinglesHost &host, double most) {
  ABRows &r = h->abr;
  r.ratio = HUGE_VAL;
  const size_t na = h->astr.size(), nb = h->bstr.size(), L2 = (size_t)h->L * h->L;
  const size_t nnza = h->ta_s.nnz, nnzb = h->tb_s.nnz;
  if (!nnza || !nnzb) return SBD_TPB_OK;
  TPB_CHECK(host.fetch(h));
  const std::vector<uint32_t> &ao = host.ao, &bo = host.bo, &bket = host.bket;
  const std::vector<int32_t> &bpair = host.bpair;
  auto pair_of = [](int32_t ps) { return (ps > 0 ? ps : -ps) - 1; };
  // rows of P: the unordered pairs of the beta singles, ascending
  std::vector<int32_t> pair_m(L2, -1), m_pair;
  std::vector<char> seen(L2, 0);
  for (int32_t ps : bpair) seen[pair_of(ps)] = 1;
  for (int x = 0; x < h->L; x++)
    for (int y = x; y < h->L; y++)
      if (seen[x * h->L + y] || seen[y * h->L + x]) {
        pair_m[x * h->L + y] = pair_m[y * h->L + x] = (int32_t)m_pair.size();
        m_pair.push_back(x * h->L + y);
      }
  const int M = (int)m_pair.size(), blocks = (M + 7) / 8;
  r.M = M;
  r.passes = (blocks + kMaxBlocks - 1) / kMaxBlocks;
  r.bpp = (blocks + r.passes - 1) / r.passes;
  r.nchunks = (uint32_t)((nb + kCols - 1) / kCols);
  double gemm = 0.0;
  uint32_t kmax = 0;
  for (size_t i = 0; i < na; i++) {
    const uint32_t k = ao[i + 1] - ao[i];
    kmax = std::max(kmax, k);
    gemm += (double)((k + 7) / 8 * 8);
  }
  r.ratio = gemm * 8.0 * r.bpp * r.passes * (double)nb / ((double)nnza * (double)nnzb);
  if (r.ratio > most) return SBD_TPB_OK;
  std::vector<uint32_t> rows;
  for (size_t i = 0; i < na; i++)
    if (ao[i + 1] > ao[i]) rows.push_back((uint32_t)i);
  std::stable_sort(rows.begin(), rows.end(),
                   [&](uint32_t x, uint32_t y) { return ao[x + 1] - ao[x] > ao[y + 1] - ao[y]; });
  r.nrows = (uint32_t)rows.size();
  r.kcap = (std::min<uint32_t>(kmax, kMaxK) + 7) & ~7u;
  // alpha singles, per row ascending by the row of P of their own pair
  std::vector<uint32_t> aket(nnza);
  std::vector<int32_t> apair(nnza);
  TPB_CUDA(cudaMemcpy(aket.data(), h->ta_s.ket, sizeof(uint32_t) * nnza, cudaMemcpyDeviceToHost));
  TPB_CUDA(cudaMemcpy(apair.data(), h->pa.s_pair, sizeof(int32_t) * nnza, cudaMemcpyDeviceToHost));
  std::vector<uint2> ent(nnza);
  for (size_t e = 0; e < nnza; e++) ent[e] = make_uint2(aket[e], (uint32_t)apair[e]);
  for (size_t i = 0; i < na; i++)
    std::stable_sort(ent.begin() + ao[i], ent.begin() + ao[i + 1], [&](const uint2 &x, const uint2 &y) {
      return pair_m[pair_of((int32_t)x.y)] < pair_m[pair_of((int32_t)y.y)];
    });
  // beta singles by (pass, chunk of their ket, gather warp of their bra), each cell by bra Ib; then
  // grouped by Ib, groups with the most entries first, entries round by round so that consecutive
  // lanes read consecutive ones
  const size_t ncell = (size_t)r.passes * r.nchunks * kGatherWarps;
  auto cell_of = [&](size_t f, size_t ib) {
    const size_t pass = pair_m[pair_of(bpair[f])] / (8 * r.bpp);
    return (pass * r.nchunks + bket[f] / kCols) * kGatherWarps + ib / 32 % kGatherWarps;
  };
  std::vector<uint32_t> start(ncell + 1, 0), order(nnzb), bra(nnzb);
  for (size_t i = 0; i < nb; i++)
    for (uint32_t f = bo[i]; f < bo[i + 1]; f++) start[cell_of(f, i) + 1]++;
  for (size_t c = 0; c < ncell; c++) start[c + 1] += start[c];
  {
    std::vector<uint32_t> at(start.begin(), start.end() - 1);
    for (size_t i = 0; i < nb; i++)
      for (uint32_t f = bo[i]; f < bo[i + 1]; f++) {
        bra[f] = (uint32_t)i;
        order[at[cell_of(f, i)]++] = f;
      }
  }
  std::vector<uint4> hdr(ncell + 1);
  std::vector<unsigned char> prog;
  std::vector<std::pair<uint32_t, uint32_t>> grp, sorted;  // (first entry, entries)
  size_t cap = 16;
  for (size_t c = 0; c < ncell; c++) {
    grp.clear();
    uint32_t most = 0;
    for (uint32_t f = start[c]; f < start[c + 1]; f++) {
      if (grp.empty() || bra[order[f]] != bra[order[grp.back().first]]) grp.emplace_back(f, 0u);
      most = std::max(most, ++grp.back().second);
    }
    sorted.clear();
    for (uint32_t k = most; k > 0; k--)
      for (const auto &g : grp)
        if (g.second == k) sorted.push_back(g);
    // program of the cell: the first entry of each round (rounds padded to a multiple of kRounds),
    // Ib of each group, then, 16-byte aligned, the entries round by round: entry k of the groups
    // that have more than k
    const size_t rounds = ((size_t)most + kRounds - 1) / kRounds * kRounds, nent = start[c + 1] - start[c];
    const size_t head = ((rounds + kRounds) * 2 + grp.size() * 4 + 15) & ~(size_t)15;
    const size_t bytes = head + ((nent * 2 + 15) & ~(size_t)15);
    if (prog.size() + bytes > 0xffffffffull || nent > 0xffff) return SBD_TPB_OK;
    hdr[c] = make_uint4((uint32_t)prog.size(), (uint32_t)grp.size(), (uint32_t)rounds, (uint32_t)head);
    prog.resize(prog.size() + bytes);
    unsigned char *pc = prog.data() + hdr[c].x;
    uint16_t *first = reinterpret_cast<uint16_t *>(pc), *en = reinterpret_cast<uint16_t *>(pc + head);
    uint32_t *ibs = reinterpret_cast<uint32_t *>(first + rounds + kRounds);
    for (size_t t = 0; t < sorted.size(); t++) ibs[t] = bra[order[sorted[t].first]];
    size_t w = 0;
    for (size_t k = 0; k < rounds + kRounds; k++) {
      first[k] = (uint16_t)w;
      for (size_t t = 0; t < sorted.size() && sorted[t].second > k; t++) {
        const uint32_t f = order[sorted[t].first + k];
        const int m = pair_m[pair_of(bpair[f])] % (8 * r.bpp);
        en[w++] = (uint16_t)(p_pos(m, (int)(bket[f] % kCols)) | (bpair[f] < 0 ? 0x8000 : 0));
      }
    }
    cap = std::max(cap, bytes);
  }
  hdr[ncell] = make_uint4((uint32_t)prog.size(), 0, 0, 0);
  r.prog_cap = (uint32_t)cap;
  if (rows_smem(r, sizeof(double), nb, false, 2) > h->smem_optin) return SBD_TPB_OK;
  // one allocation holds all of it
  size_t bytes = 0;
  auto part = [&](const auto &v) {
    const size_t at = bytes;
    bytes = (bytes + sizeof(v[0]) * v.size() + 15) & ~(size_t)15;
    return at;
  };
  const size_t o_rows = part(rows), o_ent = part(ent), o_pair = part(pair_m), o_m = part(m_pair), o_hdr = part(hdr),
               o_prog = part(prog);
  // scratch rows where an FP64 row of sums does not fit in shared memory: one CTA of the kernel fills an SM's
  // registers (512 threads of 128)
  r.slots = rows_smem(r, sizeof(double), nb, true, 2) > h->smem_optin ? h->num_sms : 0;
  const std::vector<uint32_t> taken(r.slots, 0);
  const size_t o_taken = part(taken), o_scratch = bytes;
  bytes += sizeof(double) * nb * r.slots;
  size_t free_b = 0, total_b = 0;
  TPB_CUDA(cudaMemGetInfo(&free_b, &total_b));
  if (bytes > free_b / 8) return SBD_TPB_OK;
  TPB_CUDA(cudaMalloc(&r.block, bytes));
  unsigned char *d = r.block;
  auto place = [&](size_t at, const auto &v) { return h2d(h, d + at, v.data(), sizeof(v[0]) * v.size()); };
  TPB_CUDA(place(o_rows, rows));
  TPB_CUDA(place(o_ent, ent));
  TPB_CUDA(place(o_pair, pair_m));
  TPB_CUDA(place(o_m, m_pair));
  TPB_CUDA(place(o_hdr, hdr));
  TPB_CUDA(place(o_prog, prog));
  TPB_CUDA(place(o_taken, taken));
  TPB_CUDA(cudaStreamSynchronize(h->stream));
  r.rows = reinterpret_cast<uint32_t *>(d + o_rows);
  r.ent = reinterpret_cast<uint2 *>(d + o_ent);
  r.pair_m = reinterpret_cast<int32_t *>(d + o_pair);
  r.m_pair = reinterpret_cast<int32_t *>(d + o_m);
  r.hdr = reinterpret_cast<uint4 *>(d + o_hdr);
  r.prog = d + o_prog;
  r.taken = reinterpret_cast<uint32_t *>(d + o_taken);
  r.scratch = d + o_scratch;
  r.err = g_status[h->device % kMaxDevices].get();
  if (!r.err) return fail(SBD_TPB_ERR_OOM, "alpha-beta row program: pinned status word");
  r.ready = true;
  return SBD_TPB_OK;
}

// Whether the term of this type's vectors takes the rows kernel; the program is built once per problem, when the
// first type takes it.  Memory that runs short, the host's or the device's, leaves the direct kernel to do the term.
int ab_rows_prepare(sbd_tpb_handle *h, SinglesHost &host, bool f32, bool *use) {
  const double most = f32 ? kMostRatio32 : kMostRatio64;
  *use = h->abr.ready && h->abr.ratio <= most;
  if (h->abr.tried || h->abr.ratio > most) return SBD_TPB_OK;  // (ratio 0: not counted yet)
  int rc;
  try {
    rc = build_program(h, host, most);
  } catch (const std::bad_alloc &) {
    rc = SBD_TPB_ERR_OOM;
  }
  const double ratio = h->abr.ratio;
  if (!h->abr.ready) ab_rows_free(h);
  h->abr.ratio = ratio;
  h->abr.tried = ratio <= most;
  *use = h->abr.ready;
  if (rc != SBD_TPB_ERR_OOM) return rc;
  cudaGetLastError();
  return SBD_TPB_OK;
}

int ab_rows_check(sbd_tpb_handle *h) {
  int *err = h->abr.err;
  if (!err || !*err) return SBD_TPB_OK;
  const int e = *err;
  *err = 0;
  return fail(SBD_TPB_ERR_CUDA, "alpha-beta row kernel: bounded wait expired (code " + std::to_string(e) + ")");
}

// sigma += the alpha-beta terms.  sym (identical string lists, C = C^T): only the half B of the terms
// whose transposes are the others, so that B + B^T is the whole term.
template <typename T>
int ab_rows_apply(sbd_tpb_handle *h, const T *C, T *sigma, bool sym) {
  const ABRows &r = h->abr;
  RowArgs a{};
  a.rows = r.rows;
  a.a_off = h->ta_s.off;
  a.a_ent = r.ent;
  a.pair_m = r.pair_m;
  a.m_pair = r.m_pair;
  a.hdr = r.hdr;
  a.prog = r.prog;
  a.eri = h->d_eri;
  a.L2 = h->L * h->L;
  a.M = r.M;
  a.passes = r.passes;
  a.bpp = r.bpp;
  a.nchunks = r.nchunks;
  a.nb = (uint32_t)h->bstr.size();
  a.kcap = r.kcap;
  a.prog_cap = r.prog_cap;
  a.err = r.err;  // unified addressing: the same pointer on the device
  // the row is summed in shared memory where it fits, else in a scratch row
  if (rows_smem(r, sizeof(T), a.nb, true, 2) <= h->smem_optin)
    return sym ? launch_rows<T, true, true>(h, a, C, sigma) : launch_rows<T, false, true>(h, a, C, sigma);
  return sym ? launch_rows<T, true, false>(h, a, C, sigma) : launch_rows<T, false, false>(h, a, C, sigma);
}

template int ab_rows_apply<double>(sbd_tpb_handle *, const double *, double *, bool);
template int ab_rows_apply<float>(sbd_tpb_handle *, const float *, float *, bool);

}  // namespace sbdtpb
