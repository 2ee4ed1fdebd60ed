// edm_readout.cu — lifetime readouts of TCSPC stacks on the device.
//
// For every pixel of a uint32 stack [n_px][n_bins] (the engine's FLIM stacks
// or the batched acquisition's histograms), in float64:
//   intensity = sum_k n_k;
//   tau_mean  = sum_k n_k t_k / intensity, t_k = (k + 0.5) T / n_bins in ns,
//               NaN below min_counts_mean           (analysis.py:87-150);
//   g, s      = sum_k n_k cos(phi_k) / intensity, sum_k n_k sin(phi_k) / intensity,
//               phi_k = 2 pi h (k + 0.5) / n_bins, 0 below min_counts_phasor;
//   tau_phi   = (s / g) / omega, omega = 2 pi h / T in 1/ns, where g > 1e-10;
//   tau_mod   = sqrt(1 / m^2 - 1) / omega, m^2 = g^2 + s^2 in (1e-10, 1 - 1e-10)
//               (analysis.py:497-566); NaN elsewhere.
// The kernel streams the stack once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>

#include "../../include/edm_b200.h"
#include "edm_error.h"

namespace {

// The float64 2^52 + v of a 32-bit v: its bits are 2^52's with v in the low word.
__device__ __forceinline__ double two52_plus(uint32_t v) { return __hiloint2double(0x43300000, (int)v); }

// Bins k and K-1-k share |cos| and |sin| of their phases (phi_{K-1-k} =
// 2 pi h - phi_k), so a pair adds (n_k + n_{K-1-k}) cos(phi_k) to G and
// (n_k - n_{K-1-k}) sin(phi_k) to S.  The same sum and difference give the
// intensity and the first moment sum_k n_k k = (K-1)/2 I - sum_pairs (n_k -
// n_{K-1-k}) ((K-1)/2 - k), both exact: integers and half-integers below 2^53.
struct Sums {
  double I = 0.0, M = 0.0, G = 0.0, S = 0.0;
};
__device__ __forceinline__ void readout_pair(uint32_t na, uint32_t nb, double c, double s, double w, Sums& t) {
  // counts to float64 without a conversion, every step exact
  const double a = two52_plus(na), b = two52_plus(nb);
  const double dif = a - b, sum = a + (b - 9007199254740992.0);
  t.I += sum;
  t.M = fma(dif, w, t.M);
  t.G = fma(sum, c, t.G);
  t.S = fma(dif, s, t.S);
}

// The six readouts of pixel px from its intensity, sum of n_k k and phasor sums.
struct Readout {
  double width, omega, nan;
  int min_mean, min_phasor;
  int64_t n_px;
  double* out;
  __device__ __forceinline__ void write(int64_t px, double In, double KW, double G, double S) const {
    const double tau = In >= min_mean ? width * (KW + 0.5 * In) / In : nan;
    const bool mask = In >= min_phasor;
    const double g = mask ? G / In : 0.0, s = mask ? S / In : 0.0;
    const bool valid = mask && g > 1e-10;
    const double m2 = g * g + s * s;
    out[0 * n_px + px] = In;
    out[1 * n_px + px] = tau;
    out[2 * n_px + px] = g;
    out[3 * n_px + px] = s;
    out[4 * n_px + px] = valid ? (s / g) / omega : nan;
    out[5 * n_px + px] = (valid && m2 > 1e-10 && m2 < 1.0 - 1e-10) ? sqrt(1.0 / m2 - 1.0) / omega : nan;
  }
};

// Exact float64 value of an integer v < 2^52: the double whose bits are
// 2^52 + v, minus 2^52 (one add instead of an integer-to-double conversion).
__device__ __forceinline__ double u52_to_f64(uint64_t v) {
  const double d = __hiloint2double(0x43300000 | (int)(uint32_t)(v >> 32), (int)(uint32_t)v);
  return __dsub_rn(d, 4503599627370496.0);
}
__device__ __forceinline__ void readout_pair(uint32_t na, uint32_t nb, int k, int kb, const double* c_k,
                                             const double* s_k, uint64_t& I, uint64_t& KW, double& G, double& S) {
  I += (uint64_t)na + nb;
  KW += (uint64_t)na * (uint32_t)k + (uint64_t)nb * (uint32_t)kb;
  G = fma(u52_to_f64((uint64_t)na + nb), c_k[k], G);
  S = fma(__dsub_rn(u52_to_f64((uint64_t)na + 4294967296ull - nb), 4294967296.0), s_k[k], S);
}

// Short rows: a thread per pixel reads its row from both ends in 16-byte words, the
// lanes of a warp 32 rows side by side.  Intensity and sum n_k k are integer sums.
__global__ void __launch_bounds__(256) k_readout_rows(const uint32_t* __restrict__ stack, int64_t n_px, int n_bins,
                                                      double T_ns, int harmonic, int min_mean, int min_phasor,
                                                      double* __restrict__ out) {
  __shared__ double c_k[256], s_k[256];
  for (int k = threadIdx.x; k < n_bins; k += blockDim.x) {
    const double phi = 2.0 * M_PI * harmonic * (k + 0.5) / n_bins;
    c_k[k] = cos(phi);
    s_k[k] = sin(phi);
  }
  __syncthreads();
  const int nq = n_bins / 4;  // uint4 per pixel
  const Readout R{T_ns / n_bins, 2.0 * M_PI * harmonic / T_ns, __longlong_as_double(0x7FF8000000000000ll),
                  min_mean,      min_phasor,                   n_px,
                  out};
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t px = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; px < n_px; px += step) {
    const uint4* row = reinterpret_cast<const uint4*>(stack + px * (int64_t)n_bins);
    uint64_t I = 0, KW = 0;
    double G = 0.0, S = 0.0;
    int q = 0;
    for (; q < nq - 1 - q; ++q) {  // word q (bins 4q..4q+3) against word nq-1-q, reversed
      const int qb = nq - 1 - q;
      const uint4 a = __ldg(row + q), b = __ldg(row + qb);
      readout_pair(a.x, b.w, 4 * q, 4 * qb + 3, c_k, s_k, I, KW, G, S);
      readout_pair(a.y, b.z, 4 * q + 1, 4 * qb + 2, c_k, s_k, I, KW, G, S);
      readout_pair(a.z, b.y, 4 * q + 2, 4 * qb + 1, c_k, s_k, I, KW, G, S);
      readout_pair(a.w, b.x, 4 * q + 3, 4 * qb, c_k, s_k, I, KW, G, S);
    }
    if (q == nq - 1 - q) {  // odd word count: the middle word pairs within itself
      const uint4 a = __ldg(row + q);
      readout_pair(a.x, a.w, 4 * q, 4 * q + 3, c_k, s_k, I, KW, G, S);
      readout_pair(a.y, a.z, 4 * q + 1, 4 * q + 2, c_k, s_k, I, KW, G, S);
    }
    R.write(px, (double)I, (double)KW, G, S);
  }
}

__device__ __forceinline__ void copy16_async(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Long rows.  Bound: the stack's bytes from DRAM (4.19M pixels of 256 bins in 703 us,
// 687 at the copy's rate; 1,090 by k_readout_rows).  A warp takes groups of kGroup
// pixels, four lanes per pixel, and keeps kStages groups' rows on the way into its own
// part of shared memory by 16-byte asynchronous copies: consecutive lanes copy
// consecutive words of the rows, four 128-byte lines per instruction.  (A
// thread per pixel reading its row from both ends touched 32 lines per
// instruction, which held the L1's tag stage at 0.63 of the HBM rate.)  Twelve
// warps with two stages each: with eight and three the arithmetic of a stage was
// no longer hidden (1,354 us).  Rows
// are padded to an odd multiple of 64 bytes, so that the two rows of a
// shared-memory phase lie in different banks.  The four lanes' float64 sums are
// a quarter as long as one lane's: g's relative error (rms, against 80-bit
// arithmetic, 64 to 256 bins) 2.6e-16..4.2e-16 before, 1.3e-16..1.5e-16 now.
constexpr int kReadoutWarps = 12, kGroup = 8, kStages = 2;

__device__ __host__ constexpr int row_words(int nq) { return nq + (12 - nq % 8) % 8; }  // = 4 mod 8, at least nq
constexpr size_t stage_bytes(int nq) { return sizeof(uint4) * kReadoutWarps * kStages * kGroup * row_words(nq); }

// NQ: n_bins / 4 when known to the compiler (128 and 256 bins), else 0.
template <int NQ>
__global__ void __launch_bounds__(32 * kReadoutWarps) k_readout(const uint32_t* __restrict__ stack, int64_t n_px,
                                                              int n_bins_arg, double T_ns, int harmonic, int min_mean,
                                                              int min_phasor, double* __restrict__ out) {
  extern __shared__ __align__(16) uint4 stage_mem[];
  __shared__ __align__(16) double c_k[128], s_k[128], w_k[128];
  const int n_bins = NQ ? 4 * NQ : n_bins_arg;
  for (int k = threadIdx.x; k < n_bins / 2; k += blockDim.x) {
    const double phi = 2.0 * M_PI * harmonic * (k + 0.5) / n_bins;
    c_k[k] = cos(phi);
    s_k[k] = sin(phi);
    w_k[k] = 0.5 * (n_bins - 1) - k;
  }
  __syncthreads();
  const int nq = n_bins / 4, ld = row_words(nq);  // uint4 per pixel, and per row in shared memory
  const int lane = threadIdx.x & 31, sub = lane & 3, warp = threadIdx.x >> 5;
  uint4* mine = stage_mem + (size_t)warp * kStages * kGroup * ld;
  const Readout R{T_ns / n_bins, 2.0 * M_PI * harmonic / T_ns, __longlong_as_double(0x7FF8000000000000ll),
                  min_mean,      min_phasor,                   n_px,
                  out};
  const int64_t groups = (n_px + kGroup - 1) / kGroup;
  const int64_t step = (int64_t)gridDim.x * kReadoutWarps;
  const uint4* words = reinterpret_cast<const uint4*>(stack);
  auto fetch = [&](int64_t g, int stage) {  // a group's rows are contiguous; past the last one, nothing
    if (g < groups) {
      const int64_t px0 = g * kGroup;
      const int n = (int)(n_px - px0 < kGroup ? n_px - px0 : kGroup) * nq;
      uint4* dst = mine + stage * kGroup * ld;
      const uint4* src = words + px0 * nq;
      if (NQ && n == kGroup * nq) {
#pragma unroll
        for (int i = 0; i < kGroup * NQ / 32; ++i) {
          const int k = lane + 32 * i;
          copy16_async(dst + (k / (NQ ? NQ : 1)) * ld + k % (NQ ? NQ : 1), src + k);
        }
      } else {
        int row = 0, col = lane;
        for (int i = lane; i < n; i += 32, col += 32) {
          while (col >= nq) {
            col -= nq;
            ++row;
          }
          copy16_async(dst + row * ld + col, src + i);
        }
      }
    }
    copies_commit();
  };
  int64_t g = (int64_t)blockIdx.x * kReadoutWarps + warp;
  for (int k = 0; k < kStages - 1; ++k) fetch(g + k * step, k);
  for (int stage = 0; g < groups; g += step, stage = stage + 1 == kStages ? 0 : stage + 1) {
    fetch(g + (kStages - 1) * step, (stage + kStages - 1) % kStages);
    copies_wait<kStages - 1>();
    __syncwarp();
    const uint4* row = mine + (stage * kGroup + (lane >> 2)) * ld;
    Sums t;
    int q = sub;
#pragma unroll 4
    for (; q < nq - 1 - q; q += 4) {  // word q (bins 4q..4q+3) against word nq-1-q, reversed
      const uint4 a = row[q], b = row[nq - 1 - q];
      const double2 c0 = *(const double2*)(c_k + 4 * q), c1 = *(const double2*)(c_k + 4 * q + 2);
      const double2 s0 = *(const double2*)(s_k + 4 * q), s1 = *(const double2*)(s_k + 4 * q + 2);
      const double2 w0 = *(const double2*)(w_k + 4 * q), w1 = *(const double2*)(w_k + 4 * q + 2);
      readout_pair(a.x, b.w, c0.x, s0.x, w0.x, t);
      readout_pair(a.y, b.z, c0.y, s0.y, w0.y, t);
      readout_pair(a.z, b.y, c1.x, s1.x, w1.x, t);
      readout_pair(a.w, b.x, c1.y, s1.y, w1.y, t);
    }
    if (q == nq - 1 - q) {  // odd word count: the middle word pairs within itself
      const uint4 a = row[q];
      readout_pair(a.x, a.w, c_k[4 * q], s_k[4 * q], w_k[4 * q], t);
      readout_pair(a.y, a.z, c_k[4 * q + 1], s_k[4 * q + 1], w_k[4 * q + 1], t);
    }
    __syncwarp();  // the stage is read: the next fetch may overwrite it
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      t.I += __shfl_xor_sync(0xffffffffu, t.I, o);
      t.M += __shfl_xor_sync(0xffffffffu, t.M, o);
      t.G += __shfl_xor_sync(0xffffffffu, t.G, o);
      t.S += __shfl_xor_sync(0xffffffffu, t.S, o);
    }
    const int64_t px = g * kGroup + (lane >> 2);
    if (sub != 0 || px >= n_px) continue;
    R.write(px, t.I, 0.5 * (n_bins - 1) * t.I - t.M, t.G, t.S);
  }
}

// Pixels from which k_readout_rows is the faster.  k_readout spends a latency on
// every eight pixels however short their rows, and unless it knows the row's length
// (128 and 256 bins) the copies' index arithmetic is not hidden; k_readout_rows needs
// many threads.  Rows / staged, us: 16 bins 7.4 / 7.4 at 10,000 pixels, 7.3 / 8.3 at
// 30,000, 91 / 303 at 4.2M; 64 bins 7.6 / 7.3, 8.4 / 9.3, 303 / 389; 100 bins 39.9 /
// 36.6 at 262,144, 68.6 / 68.6 at 524,288, 124.7 / 127.4 at 1.05M; 160 bins 111 / 109
// at 524,288, 195 / 208 at 1.05M; 252 bins 29.8 / 27.7 at 65,536, 45.8 / 49.3 at
// 131,072, 272 / 321 at 1.05M; 256 bins 290 / 221 there.
int64_t rows_from(int n_bins) {
  if (n_bins == 128 || n_bins == 256) return INT64_MAX;
  return n_bins <= 96 ? 1 << 14 : (n_bins <= 176 ? 1 << 20 : 1 << 17);
}

}  // namespace

extern "C" int edm_readout_lifetimes(const uint32_t* stack_dev, int64_t n_px, int32_t n_bins, double time_range_s,
                                     int32_t harmonic, int32_t min_counts_mean, int32_t min_counts_phasor,
                                     double* out_dev, void* stream) {
  if (!stack_dev || !out_dev || n_px < 0 || n_bins <= 0 || n_bins > 256 || n_bins % 4 != 0 || !(time_range_s > 0.0) ||
      harmonic < 1)
    return edm::report_error(EDM_EINVAL,
                             "edm_readout_lifetimes: bad argument (n_bins must be a multiple of 4 up to 256)");
  if (((uintptr_t)stack_dev & 15u) != 0)
    return edm::report_error(EDM_EINVAL, "edm_readout_lifetimes: stack must be 16-byte aligned");
  if (n_px == 0) return EDM_OK;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const cudaStream_t s = (cudaStream_t)stream;
  if (n_px >= rows_from(n_bins)) {
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_readout_rows, 256, 0);
    const int64_t want = (n_px + 255) / 256, cap = (int64_t)sms * std::max(1, per_sm);
    k_readout_rows<<<(unsigned)std::min(want, cap), 256, 0, s>>>(stack_dev, n_px, n_bins, time_range_s * 1e9, harmonic,
                                                                   min_counts_mean, min_counts_phasor, out_dev);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return edm::report_error(EDM_ECUDA, std::string("edm_readout_lifetimes: ") + cudaGetErrorString(e));
    return EDM_OK;
  }
  const size_t smem = stage_bytes(n_bins / 4);
  const auto kernel = n_bins == 256 ? k_readout<64> : (n_bins == 128 ? k_readout<32> : k_readout<0>);
  // the limit is the kernel's, not the call's: always the same, so that another
  // thread's call with fewer bins cannot lower it before this launch
  constexpr int most = (int)stage_bytes(64);
  if (const cudaError_t a = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      a != cudaSuccess)
    return edm::report_error(EDM_ECUDA, std::string("edm_readout_lifetimes: ") + cudaGetErrorString(a));
  // blocks that fit an SM's 227 KB of shared memory
  const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(5, (227 * 1024) / (smem + 4096)));
  const int64_t want = (n_px + kGroup * kReadoutWarps - 1) / (kGroup * kReadoutWarps), cap = (int64_t)sms * per_sm;
  const unsigned blocks = (unsigned)(want < cap ? want : cap);
  kernel<<<blocks, 32 * kReadoutWarps, smem, s>>>(stack_dev, n_px, n_bins, time_range_s * 1e9, harmonic, min_counts_mean,
                                                  min_counts_phasor, out_dev);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return edm::report_error(EDM_ECUDA, std::string("edm_readout_lifetimes: ") + cudaGetErrorString(e));
  return EDM_OK;
}
