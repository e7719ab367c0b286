// Same-spin passes of sigma on densely connected string sets: the doubles of 8 neighbouring bra
// strings as one list of their distinct kets (included by sigma.cu).
//
// Neighbouring strings of a molecular set share half of their kets (8 rows of a 4,041-string N2 set:
// 3,240 doubles over 1,470 kets), so a thread that holds all 8 rows of its columns loads each ket's
// elements once and multiplies them into the rows that have it: half the gathered bytes, and eight
// independent sums per load instead of one.  Each row still adds its doubles in ascending ket order,
// then its singles, with sigma_block_kernel's arithmetic: the same bits.
//
// A thread's VW columns lie 128 apart, so every access of a warp is one contiguous run whatever the
// row length; VW is chosen by the number of CTAs (launch_union).  Bound by the gathers' round trips to L2: half
// of a warp's cycles between two issues, with 19 warps an SM (88 registers in FP64); L1/TEX is 66 % busy, the
// issue slots 53 %, the FP64 pipe 36 %, L2 36 %.  When these passes are taken: union_ahead.
// ms per pass, per-row kernels -> here: 18 orbitals, 4,041 strings (odd rows) FP64 alpha 11.9 -> 4.3, beta
// 12.5 -> 4.3; 24 orbitals, 5,514 strings FP32 one-pass 19.8 -> 8.0; 18 orbitals, 1,387 strings FP64 0.86 /
// 0.91 -> 0.47 / 0.49, FP32 0.72 / 0.76 -> 0.33 / 0.35.
#pragma once

constexpr int kUnionThreads = 128;
constexpr int kUnionChunk = 64;  // kets staged at a time, two buffers

__device__ __forceinline__ void union_cp16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <typename T, bool kAlpha, bool kSym, int VW, int M>
__global__ void __launch_bounds__(kUnionThreads, M)
    sigma_union_kernel(BlockArgs a, UnionArgs u, const T *__restrict__ X, T *__restrict__ out, T *__restrict__ XT) {
  constexpr uint32_t W = kUnionThreads * VW;
  __shared__ __align__(16) uint32_t u_ket[2][kUnionChunk];
  __shared__ __align__(16) T u_val[2][kUnionChunk][kBlkRows];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t *ss_ket = reinterpret_cast<uint32_t *>(smem_raw);
  int32_t *ss_row = reinterpret_cast<int32_t *>(ss_ket + a.max_s);  // +-(row of jtab + 1)
  double *ss_val = reinterpret_cast<double *>(smem_raw + ((a.max_s * 8 + 15) & ~15u));

  const uint32_t nrb = (a.nrows + kBlkRows - 1) / kBlkRows;
  const uint32_t rb = blockIdx.x % nrb, slab = blockIdx.x / nrb;
  const uint32_t r0 = rb * kBlkRows, ncols = a.ncols;
  const int nr = (int)min((uint32_t)kBlkRows, a.nrows - r0);
  const uint32_t c0 = slab * W + threadIdx.x;
  bool ok[VW];
#pragma unroll
  for (int i = 0; i < VW; i++) ok[i] = c0 + i * kUnionThreads < ncols;

  const uint32_t u0 = __ldg(&u.off[rb]), u1 = __ldg(&u.off[rb + 1]);
  const T *uval = reinterpret_cast<const T *>(u.val);
  auto stage = [&](uint32_t e, int b) {  // 16-byte copies: 4 kets; 16 / sizeof(T) values
    const uint32_t n = min((uint32_t)kUnionChunk, u1 - e);
    constexpr uint32_t per = kBlkRows * sizeof(T) / 16;
    for (uint32_t t = threadIdx.x; t < n * per; t += kUnionThreads)
      union_cp16(reinterpret_cast<unsigned char *>(u_val[b]) + t * 16,
                 reinterpret_cast<const unsigned char *>(uval + (size_t)e * kBlkRows) + t * 16);
    if (threadIdx.x < n / 4) union_cp16(&u_ket[b][4 * threadIdx.x], u.ket + e + 4 * threadIdx.x);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (u0 < u1) stage(u0, 0);
  const uint32_t slo = __ldg(&a.s_off[r0]), shi = __ldg(&a.s_off[r0 + nr]);
  for (uint32_t e = slo + threadIdx.x; e < shi; e += kUnionThreads) {
    const int32_t ps = __ldg(&a.s_pair[e]), jr = __ldg(&a.pmap[(ps > 0 ? ps : -ps) - 1]) + 1;
    ss_ket[e - slo] = __ldg(&a.s_ket[e]);
    ss_row[e - slo] = ps > 0 ? jr : -jr;
    ss_val[e - slo] = (double)val_of<T>(a.s_val, a.s_valf, e);
  }

  T acc[kBlkRows][VW];
#pragma unroll
  for (int r = 0; r < kBlkRows; r++)
#pragma unroll
    for (int i = 0; i < VW; i++) acc[r][i] = T(0);
  int b = 0;
  for (uint32_t e0 = u0; e0 < u1; e0 += kUnionChunk, b ^= 1) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (e0 + kUnionChunk < u1) stage(e0 + kUnionChunk, b ^ 1);
    const uint32_t n = min((uint32_t)kUnionChunk, u1 - e0);
    for (uint32_t e = 0; e < n; e += 4) {
      T x[4][VW];
      uint32_t km[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        km[k] = u_ket[b][e + k];
        const T *xr = X + (size_t)(km[k] & 0xffffffu) * ncols + c0;
#pragma unroll
        for (int i = 0; i < VW; i++) x[k][i] = ok[i] ? __ldg(xr + i * kUnionThreads) : T(0);
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int r = 0; r < kBlkRows; r++) {
          const T v = u_val[b][e + k][r];
          if (km[k] >> (24 + r) & 1) {
#pragma unroll
            for (int i = 0; i < VW; i++) acc[r][i] = madd(acc[r][i], v, x[k][i]);
          }
        }
      }
    }
  }
  __syncthreads();  // the singles are staged (also when the block has no doubles)

  T own[kAlpha && !kSym ? kBlkRows : 1][VW];
#pragma unroll
  for (int r = 0; r < kBlkRows; r++) {
    if (r >= nr) continue;
    const uint32_t row = r0 + r;
    const uint32_t s0 = __ldg(&a.s_off[row]) - slo, s1 = __ldg(&a.s_off[row + 1]) - slo;
    for (uint32_t e = s0; e < s1; e += 4) {
      // four singles' loads before their sums
      T x[4][VW];
      double j[4][VW];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t ee = min(e + k, s1 - 1);
        const int32_t jr = ss_row[ee];
        const T *xr = X + (size_t)ss_ket[ee] * ncols + c0;
        const double *jp = a.jtab + (size_t)((jr > 0 ? jr : -jr) - 1) * ncols + c0;
#pragma unroll
        for (int i = 0; i < VW; i++) {
          x[k][i] = ok[i] ? __ldg(xr + i * kUnionThreads) : T(0);
          j[k][i] = ok[i] ? __ldg(jp + i * kUnionThreads) : 0.0;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (e + k < s1) {
          const double v = ss_val[e + k], sg = ss_row[e + k] > 0 ? 1.0 : -1.0;
#pragma unroll
          for (int i = 0; i < VW; i++) acc[r][i] += (T)__dmul_rn(v + sg * j[k][i], (double)x[k][i]);
        }
    }
    if constexpr (kAlpha) {
      const T *hsrc = sizeof(T) == 8 ? reinterpret_cast<const T *>(a.hii) : reinterpret_cast<const T *>(a.hii32);
      const double hshift = sizeof(T) == 8 ? -a.core_shift : a.core_shift;
#pragma unroll
      for (int i = 0; i < VW; i++) {
        if (!ok[i]) continue;
        const size_t idx = (size_t)row * ncols + c0 + i * kUnionThreads;
        const T xo = __ldg(X + idx);
        const double hd = __dmul_rn((double)__ldg(hsrc + idx) + hshift, (double)xo);
        double res;
        if constexpr (kSym) {
          res = (double)acc[r][i] + 0.5 * hd;
        } else {
          own[r][i] = xo;
          res = (double)acc[r][i] + hd;
        }
        if (a.accumulate) res += (double)out[idx];
        out[idx] = (T)res;
      }
    }
  }
  if constexpr (kSym) return;
  // transposed: column c's 8 rows are contiguous in C^T (alpha) or sigma (beta)
  const bool runs = nr == kBlkRows && a.nrows % (16 / sizeof(T)) == 0 &&
                    reinterpret_cast<uintptr_t>(kAlpha ? XT : out) % 16 == 0;
#pragma unroll
  for (int i = 0; i < VW; i++) {
    if (!ok[i]) continue;
    const size_t o = (size_t)(c0 + i * kUnionThreads) * a.nrows + r0;
    if (runs) {
      constexpr int RW = 16 / sizeof(T);
#pragma unroll
      for (int r = 0; r < kBlkRows; r += RW) {
        Vec<T, RW, true> v;
        if constexpr (kAlpha) {
#pragma unroll
          for (int q = 0; q < RW; q++) v.v[q] = own[r + q][i];
          v.store(XT + o + r);
        } else {
          v.load_rw(out + o + r);
#pragma unroll
          for (int q = 0; q < RW; q++) v.v[q] += acc[r + q][i];
          v.store(out + o + r);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < kBlkRows; r++)
        if (r < nr) {
          if constexpr (kAlpha) XT[o + r] = own[r][i];
          else out[o + r] += acc[r][i];
        }
    }
  }
}
