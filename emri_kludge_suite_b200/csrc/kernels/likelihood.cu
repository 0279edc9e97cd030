// likelihood.cu -- see likelihood.cuh.
//
// After cuFFT has turned each template channel into its half spectrum H_j,
// the reference multiplies by the weights (likelihood_prep) and calls
// cublasZdotc four times per template with a device sync after each.  Here one
// kernel reads every template bin once and produces both products for both
// channels: per thread a strided FP64 accumulation over bins, warp-shuffle
// and shared-memory reduction to one partial per CTA, then a second tiny
// kernel adds the partials of each template in a fixed order (deterministic,
// no atomics).  Data and weights (77 MB for N = 3.2e6) stay L2-resident
// across templates; the template spectra stream from HBM once.  The rows of
// FP64 batches of even length are packed transforms: a real transform of N
// samples is a complex one of N / 2 and a pass that separates the even and odd
// samples' spectra, and that pass is arithmetic on two bins the reduction
// reads anyway, so the transform's own packing and separating passes over the
// rows (a third of its time) are not made.  An FP32
// variant reads FP32 spectra, data and weights and accumulates with Kahan
// compensation.
#include "likelihood.cuh"

#include <algorithm>

namespace aak {
namespace {

__global__ void __launch_bounds__(kIpThreads) k_inner_partial(InnerProductArgs a) {
  const int k = blockIdx.y;
  const int tid = threadIdx.x;
  double dh = 0.0, hh = 0.0;
  const int64_t stride = (int64_t)gridDim.x * kIpThreads;
  for (int ch = 0; ch < 2; ++ch) {
    const double2 *H = reinterpret_cast<const double2 *>(a.H[ch] + (int64_t)k * a.row_doubles);
    const double2 *D = reinterpret_cast<const double2 *>(a.D[ch]);
    const double *w = a.w[ch];
    for (int64_t j = (int64_t)blockIdx.x * kIpThreads + tid; j < a.nbins; j += stride) {
      const double2 h = H[j];
      const double2 d = __ldg(&D[j]);
      const double wj = __ldg(&w[j]);
      const double hr = wj * h.x, hi = wj * h.y;
      dh = fma(hr, d.x, fma(hi, d.y, dh));
      hh = fma(hr, hr, fma(hi, hi, hh));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    dh += __shfl_xor_sync(0xffffffffu, dh, o);
    hh += __shfl_xor_sync(0xffffffffu, hh, o);
  }
  __shared__ double s[2][kIpThreads / 32];
  const int w = tid >> 5, l = tid & 31;
  if (l == 0) {
    s[0][w] = dh;
    s[1][w] = hh;
  }
  __syncthreads();
  if (tid == 0) {
    double a0 = 0.0, a1 = 0.0;
    for (int i = 0; i < kIpThreads / 32; ++i) {
      a0 += s[0][i];
      a1 += s[1][i];
    }
    a.partial[((int64_t)k * gridDim.x + blockIdx.x) * 2 + 0] = a0;
    a.partial[((int64_t)k * gridDim.x + blockIdx.x) * 2 + 1] = a1;
  }
}

// Bins k and M - k of a real transform of length 2 M from its packed transform
// Z: with E, O the spectra of the even and odd samples and tw = exp(-i pi k /
// M), H[k] = E + tw O and H[M - k] = conj(E - tw O), where E = (Z[k] + conj
// Z[M - k]) / 2 and O = -i (Z[k] - conj Z[M - k]) / 2.
__device__ __forceinline__ void unpack_pair(double2 z1, double2 z2, double2 tw, double2 &h1, double2 &h2) {
  const double ex = 0.5 * (z1.x + z2.x), ey = 0.5 * (z1.y - z2.y);
  const double ox = 0.5 * (z1.y + z2.y), oy = -0.5 * (z1.x - z2.x);
  const double px = tw.x * ox - tw.y * oy, py = tw.x * oy + tw.y * ox;
  h1 = make_double2(ex + px, ey + py);
  h2 = make_double2(ex - px, py - ey);
}
__device__ __forceinline__ double2 pair_twiddle(int64_t k, double inv_m) {
  double s, c;
  sincospi((double)k * inv_m, &s, &c);
  return make_double2(c, -s);
}

// Products from packed rows: a thread takes the bins k and M - k of both
// channels together, for kIpPackedTemplates templates that share the twiddle,
// data and weights.  Bound by HBM (the packed rows, read once).
constexpr int kIpPackedTemplates = 4;
__global__ void __launch_bounds__(kIpThreads) k_inner_packed(InnerProductArgs a) {
  constexpr int NT = kIpPackedTemplates;
  const int t0 = blockIdx.y * NT;
  const int tid = threadIdx.x;
  const int64_t M = a.nbins - 1, pairs = M / 2 + 1;
  const double inv_m = 1.0 / (double)M;
  int64_t row[NT];  // past the last template: the last one again, not written
#pragma unroll
  for (int t = 0; t < NT; ++t) row[t] = (int64_t)min(t0 + t, a.ntemplates - 1) * a.row_doubles;
  double dh[NT], hh[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) dh[t] = hh[t] = 0.0;
  const int64_t stride = (int64_t)gridDim.x * kIpThreads;
  for (int64_t k = (int64_t)blockIdx.x * kIpThreads + tid; k < pairs; k += stride) {
    const double2 tw = pair_twiddle(k, inv_m);
    const int64_t k2 = M - k, kz = (k == 0) ? 0 : k2;
    const double both = (k2 == k) ? 0.0 : 1.0;  // the middle bin of an even M is its own partner
#pragma unroll
    for (int ch = 0; ch < 2; ++ch) {
      const double2 *D = reinterpret_cast<const double2 *>(a.D[ch]);
      const double2 d1 = __ldg(&D[k]), d2 = __ldg(&D[k2]);
      const double w1 = __ldg(&a.w[ch][k]), w2 = __ldg(&a.w[ch][k2]) * both;
      double2 z1[NT], z2[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const double2 *Z = reinterpret_cast<const double2 *>(a.H[ch] + row[t]);
        z1[t] = Z[k];
        z2[t] = Z[kz];
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        double2 h1, h2;
        unpack_pair(z1[t], z2[t], tw, h1, h2);
        const double ar = w1 * h1.x, ai = w1 * h1.y, br = w2 * h2.x, bi = w2 * h2.y;
        dh[t] = fma(ar, d1.x, fma(ai, d1.y, dh[t]));
        hh[t] = fma(ar, ar, fma(ai, ai, hh[t]));
        dh[t] = fma(br, d2.x, fma(bi, d2.y, dh[t]));
        hh[t] = fma(br, br, fma(bi, bi, hh[t]));
      }
    }
  }
  __shared__ double s[2 * NT][kIpThreads / 32];
  const int w = tid >> 5, l = tid & 31;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dh[t] += __shfl_xor_sync(0xffffffffu, dh[t], o);
      hh[t] += __shfl_xor_sync(0xffffffffu, hh[t], o);
    }
    if (l == 0) {
      s[2 * t][w] = dh[t];
      s[2 * t + 1][w] = hh[t];
    }
  }
  __syncthreads();
  if (tid < 2 * NT && t0 + tid / 2 < a.ntemplates) {
    double x = 0.0;
    for (int i = 0; i < kIpThreads / 32; ++i) x += s[tid][i];
    a.partial[((int64_t)(t0 + tid / 2) * gridDim.x + blockIdx.x) * 2 + (tid & 1)] = x;
  }
}

__global__ void __launch_bounds__(kIpThreads) k_unpack_rows(double *H, int64_t row_doubles) {
  const int64_t M = row_doubles / 2 - 1, pairs = M / 2 + 1;
  const double inv_m = 1.0 / (double)M;
  double2 *Z = reinterpret_cast<double2 *>(H + (int64_t)blockIdx.y * row_doubles);
  for (int64_t k = (int64_t)blockIdx.x * kIpThreads + threadIdx.x; k < pairs; k += (int64_t)gridDim.x * kIpThreads) {
    const double2 z1 = Z[k], z2 = Z[k == 0 ? 0 : M - k];
    double2 h1, h2;
    unpack_pair(z1, z2, pair_twiddle(k, inv_m), h1, h2);
    Z[k] = h1;
    if (M - k != k) Z[M - k] = h2;
  }
}

// FP32 spectra: per-thread Kahan sums (the compensation c carries the low
// part each addition loses), then the warp's pairwise shuffle tree in FP32
// and the warps of the CTA in FP64.
__device__ __forceinline__ void kahan_add(float &sum, float &c, float x) {
  const float y = x - c;
  const float t = sum + y;
  c = (t - sum) - y;
  sum = t;
}

__global__ void __launch_bounds__(kIpThreads) k_inner_partial_f32(InnerProductArgs32 a) {
  const int k = blockIdx.y;
  const int tid = threadIdx.x;
  float dh = 0.f, hh = 0.f, cdh = 0.f, chh = 0.f;
  const int64_t stride = (int64_t)gridDim.x * kIpThreads;
  for (int ch = 0; ch < 2; ++ch) {
    const float2 *H = reinterpret_cast<const float2 *>(a.H[ch] + (int64_t)k * a.row_floats);
    const float2 *D = reinterpret_cast<const float2 *>(a.D[ch]);
    const float *w = a.w[ch];
    for (int64_t j = (int64_t)blockIdx.x * kIpThreads + tid; j < a.nbins; j += stride) {
      const float2 h = H[j];
      const float2 d = __ldg(&D[j]);
      const float wj = __ldg(&w[j]);
      const float hr = wj * h.x, hi = wj * h.y;
      kahan_add(dh, cdh, fmaf(hr, d.x, hi * d.y));
      kahan_add(hh, chh, fmaf(hr, hr, hi * hi));
    }
  }
  dh -= cdh;
  hh -= chh;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    dh += __shfl_xor_sync(0xffffffffu, dh, o);
    hh += __shfl_xor_sync(0xffffffffu, hh, o);
  }
  __shared__ double s[2][kIpThreads / 32];
  const int w = tid >> 5, l = tid & 31;
  if (l == 0) {
    s[0][w] = (double)dh;
    s[1][w] = (double)hh;
  }
  __syncthreads();
  if (tid == 0) {
    double a0 = 0.0, a1 = 0.0;
    for (int i = 0; i < kIpThreads / 32; ++i) {
      a0 += s[0][i];
      a1 += s[1][i];
    }
    a.partial[((int64_t)k * gridDim.x + blockIdx.x) * 2 + 0] = a0;
    a.partial[((int64_t)k * gridDim.x + blockIdx.x) * 2 + 1] = a1;
  }
}

__global__ void k_inner_final(const double *partial, int nblocks, int ntemplates, double *out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ntemplates) return;
  double a0 = 0.0, a1 = 0.0;
  for (int b = 0; b < nblocks; ++b) {
    a0 += partial[((int64_t)k * nblocks + b) * 2 + 0];
    a1 += partial[((int64_t)k * nblocks + b) * 2 + 1];
  }
  out[2 * k + 0] = 4.0 * a0;
  out[2 * k + 1] = 4.0 * a1;
}

// Each CTA stages the weighted differences of kFisherBins bins of every
// derivative and both channels in shared memory (bins major, the derivative
// index padded to kFisherMaxDim + 1 so that the staging stores spread over
// the banks), then each thread adds the products of its one or two (channel,
// i <= j) pairs over the staged bins.  Each template row streams from HBM once.
// Packed rows: a chunk is kFisherBins / 2 bins k and their partners M - k, their
// twiddles computed once for all rows.
template <bool kPacked>
__global__ void __launch_bounds__(kFisherThreads) k_fisher_partial(FisherArgs a) {
  __shared__ double2 sD[2][kFisherBins][kFisherMaxDim + 1];
  __shared__ double2 s_tw[kFisherBins / 2];
  const int64_t M = a.nbins - 1;
  const double inv_m = 1.0 / (double)M;
  const int nd = a.nd, tid = threadIdx.x;
  const int npair = nd * (nd + 1) / 2, ncombo = 2 * npair;
  int cc[2] = {0, 0}, ii[2] = {0, 0}, jj[2] = {0, 0};
  double acc[2] = {0.0, 0.0};
  bool has[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {  // this thread's pairs q = tid, tid + kFisherThreads
    const int q = tid + m * kFisherThreads;
    has[m] = q < ncombo;
    if (!has[m]) continue;
    const int c = q / npair;
    int r = q - c * npair, i = 0;
    while (r >= nd - i) {  // row-major upper triangle: row i holds nd - i pairs
      r -= nd - i;
      ++i;
    }
    cc[m] = c;
    ii[m] = i;
    jj[m] = i + r;
  }
  constexpr int kStep = kPacked ? kFisherBins / 2 : kFisherBins;
  const int64_t span = kPacked ? M / 2 + 1 : a.nbins;
  const int64_t nchunks = (span + kStep - 1) / kStep;
  for (int64_t ck = blockIdx.x; ck < nchunks; ck += gridDim.x) {
    const int64_t b0 = ck * kStep;
    if (kPacked && tid < kStep) s_tw[tid] = pair_twiddle(b0 + tid, inv_m);
    __syncthreads();  // the previous chunk's products are done
    if constexpr (kPacked) {
#pragma unroll 2
      for (int idx = tid; idx < 2 * nd * kStep; idx += kFisherThreads) {
        const int b = idx % kStep, rest = idx / kStep;
        const int i = rest % nd, c = rest / nd;
        const int64_t k = b0 + b, k2 = M - k;
        double2 h1 = make_double2(0.0, 0.0), h2 = h1;
        if (k < span) {
          const double *Hc = c ? a.H[1] : a.H[0];
          const double2 *Zu = reinterpret_cast<const double2 *>(Hc + (int64_t)(2 * i + 1) * a.row_doubles);
          const double2 *Zd = reinterpret_cast<const double2 *>(Hc + (int64_t)(2 * i) * a.row_doubles);
          const int64_t kz = (k == 0) ? 0 : k2;
          const double2 u1 = Zu[k], v1 = Zd[k], u2 = Zu[kz], v2 = Zd[kz];
          const double *w = c ? a.w[1] : a.w[0];
          const double w1 = __ldg(w + k) * a.scale, w2 = (k2 == k) ? 0.0 : __ldg(w + k2) * a.scale;
          unpack_pair(make_double2(u1.x - v1.x, u1.y - v1.y), make_double2(u2.x - v2.x, u2.y - v2.y), s_tw[b], h1, h2);
          h1 = make_double2(w1 * h1.x, w1 * h1.y);
          h2 = make_double2(w2 * h2.x, w2 * h2.y);
        }
        sD[c][b][i] = h1;
        sD[c][kStep + b][i] = h2;
      }
    } else {
#pragma unroll 4
      for (int idx = tid; idx < 2 * nd * kFisherBins; idx += kFisherThreads) {
        const int b = idx % kFisherBins, rest = idx / kFisherBins;
        const int i = rest % nd, c = rest / nd;
        const int64_t bin = b0 + b;
        double2 d = make_double2(0.0, 0.0);
        if (bin < a.nbins) {
          const double *Hc = c ? a.H[1] : a.H[0];  // selected, not indexed: the arguments stay in registers
          const double2 *Hu = reinterpret_cast<const double2 *>(Hc + (int64_t)(2 * i + 1) * a.row_doubles);
          const double2 *Hd = reinterpret_cast<const double2 *>(Hc + (int64_t)(2 * i) * a.row_doubles);
          const double2 u = Hu[bin], v = Hd[bin];
          const double wv = __ldg((c ? a.w[1] : a.w[0]) + bin) * a.scale;
          d = make_double2(wv * (u.x - v.x), wv * (u.y - v.y));
        }
        sD[c][b][i] = d;
      }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      if (!has[m]) continue;
      const int c = cc[m], i = ii[m], j = jj[m];
      double s = acc[m];
#pragma unroll 8
      for (int b = 0; b < kFisherBins; ++b) {
        const double2 x = sD[c][b][i], y = sD[c][b][j];
        s = fma(x.x, y.x, fma(x.y, y.y, s));
      }
      acc[m] = s;
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
    if (has[m]) a.partial[(int64_t)blockIdx.x * ncombo + tid + m * kFisherThreads] = acc[m];
}

// One warp per (channel, i <= j) pair: lane l adds the partials of CTAs
// l, l + 32, ... in order, then a fixed shuffle tree (deterministic).
__global__ void __launch_bounds__(kFisherThreads) k_fisher_final(FisherArgs a, int nblocks) {
  const int nd = a.nd, npair = nd * (nd + 1) / 2, ncombo = 2 * npair;
  const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (q >= ncombo) return;
  double s = 0.0;
  for (int b = lane; b < nblocks; b += 32) s += a.partial[(int64_t)b * ncombo + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane != 0) return;
  const int c = q / npair;
  int r = q - c * npair, i = 0;
  while (r >= nd - i) {
    r -= nd - i;
    ++i;
  }
  const int j = i + r;
  a.out[(c * nd + i) * nd + j] = 4.0 * s;
  a.out[(c * nd + j) * nd + i] = 4.0 * s;
}

}  // namespace

int fisher_grid(int num_sms, int64_t nbins) {
  const int64_t nchunks = (nbins + kFisherBins - 1) / kFisherBins;
  return (int)std::max<int64_t>(1, std::min<int64_t>(nchunks, (int64_t)num_sms * 4));
}

void launch_fisher_gram(const FisherArgs &a, int num_sms, cudaStream_t stream) {
  if (a.nd <= 0 || a.nd > kFisherMaxDim) return;
  const int grid = fisher_grid(num_sms, a.nbins);
  if (a.packed) k_fisher_partial<true><<<grid, kFisherThreads, 0, stream>>>(a);
  else k_fisher_partial<false><<<grid, kFisherThreads, 0, stream>>>(a);
  const int ncombo = a.nd * (a.nd + 1), warps = kFisherThreads / 32;
  k_fisher_final<<<(ncombo + warps - 1) / warps, kFisherThreads, 0, stream>>>(a, grid);
}

void launch_inner_products_f32(const InnerProductArgs32 &a, cudaStream_t stream) {
  if (a.ntemplates <= 0) return;
  dim3 grid(kIpBlocksPerTemplate, a.ntemplates);
  k_inner_partial_f32<<<grid, kIpThreads, 0, stream>>>(a);
  k_inner_final<<<(a.ntemplates + 127) / 128, 128, 0, stream>>>(a.partial, kIpBlocksPerTemplate, a.ntemplates, a.out);
}

void launch_inner_products_packed(const InnerProductArgs &a, cudaStream_t stream) {
  if (a.ntemplates <= 0) return;
  dim3 grid(kIpBlocksPerTemplate, (a.ntemplates + kIpPackedTemplates - 1) / kIpPackedTemplates);
  k_inner_packed<<<grid, kIpThreads, 0, stream>>>(a);
  k_inner_final<<<(a.ntemplates + 127) / 128, 128, 0, stream>>>(a.partial, kIpBlocksPerTemplate, a.ntemplates, a.out);
}

void launch_unpack_rows(double *H, int64_t row_doubles, int rows, cudaStream_t stream) {
  if (rows <= 0) return;
  k_unpack_rows<<<dim3(256, rows), kIpThreads, 0, stream>>>(H, row_doubles);
}

void launch_inner_products(const InnerProductArgs &a, cudaStream_t stream) {
  if (a.ntemplates <= 0) return;
  dim3 grid(kIpBlocksPerTemplate, a.ntemplates);
  k_inner_partial<<<grid, kIpThreads, 0, stream>>>(a);
  k_inner_final<<<(a.ntemplates + 127) / 128, 128, 0, stream>>>(a.partial, kIpBlocksPerTemplate, a.ntemplates, a.out);
}

}  // namespace aak
