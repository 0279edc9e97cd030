// aak_segments.cuh -- FP64 dense stage from polynomial segments (included by
// aak_dense.cu inside its namespace).
//
// Over 256 samples the trajectory, the AB2 rates and the antenna response
// change by 1e-4 of themselves: to FP64 rounding they are polynomials of
// degree 4 (7 in the last days before a plunge) in the sample index, and the
// AB2 phase sums, being sums of polynomials, are polynomials of one degree
// more.  So the spline, the PN rates, the amplitude's power and the response
// are evaluated at eight Chebyshev points of each segment instead of at its
// 256 samples, and a sample costs a few Horner chains; and since a tile's
// phase increments are known before the samples are visited, the chain of
// carries is summed ahead of the waveform kernel, whose tiles no longer wait
// for one another.
//
// k_tile_segments (one warp a tile, a lane a node) tests the cut by the
// Chebyshev coefficients it drops: they must lie at the rounding noise of the
// node values (kSegTol).  A tile that fails -- a frozen or clamped trajectory,
// the end of a plunge, an irregular sample time, an end of the spline -- is marked
// direct and goes through k_waveform's per-sample phase pass with its carry given.
#pragma once

// quantities sampled at the nodes: gamma~dot, Phidot, alphadot, then (waveform)
// amplitude, sqrt(1 - e^2), e, F+_I, Fx_I, F+_II, Fx_II (times the response
// constant), Doppler lever arm; or (phase product) e
constexpr int kNodeQ = 11, kNodeQPhase = 4;
// polynomials kept a segment beside the three phases: all but alphadot; the phase product keeps all four
constexpr int kPolyQ = 10, kPolyQPhase = 4;
// A dropped coefficient counts as noise below this fraction of its quantity:
// the node values' own rounding (spline, PN rates) reaches 2e-15 in the sources
// of the benchmark batch, and the truncated terms oscillate over a segment, so
// that they add less than 1e-14 rad a segment to a phase.
constexpr double kSegTol = 4e-15;
constexpr int kSegWarps = 8;  // tiles of one CTA of k_tile_segments

__device__ __forceinline__ TileHead *tile_head(const BatchView &bv, int64_t g) {
  return reinterpret_cast<TileHead *>(bv.tile_seg + g * (bv.phase_out ? kSegSlotBytesPhase : kSegSlotBytes));
}

// doubles of one segment's coefficients
__host__ __device__ constexpr int seg_doubles(int D, bool phase) {
  return (3 * (D + 2) + (phase ? kPolyQPhase : kPolyQ) * (D + 1) + 1) / 2 * 2;
}

static_assert(kSegSlotBytes == sizeof(TileHead) + 4 * sizeof(double) * seg_doubles(7, false), "a slot of the waveform");
static_assert(kSegSlotBytesPhase == sizeof(TileHead) + 4 * sizeof(double) * seg_doubles(7, true), "a slot of the phase product");

struct SegTables {
  double fit4t[kSegNodes][kSegNodes];  // five rows of the cut fit, then the three dropped Chebyshev coefficients
  double fit7[kSegNodes][kSegNodes];
  double sum4[2][6][kSegNodes], sum7[2][9][kSegNodes];  // forward, backward
};
constexpr SegTables make_seg_tables() {
  SegTables t{};
  for (int j = 0; j < kSegNodes; ++j) {
    for (int k = 0; k < 5; ++k) t.fit4t[k][j] = kSegFit4[k][j];
    for (int k = 0; k < 3; ++k) t.fit4t[5 + k][j] = kSegTail[k][j];
    for (int k = 0; k < 8; ++k) t.fit7[k][j] = kSegFit7[k][j];
    for (int k = 0; k < 6; ++k) {
      t.sum4[0][k][j] = kSegFwd4[k][j];
      t.sum4[1][k][j] = kSegBwd4[k][j];
    }
    for (int k = 0; k < 9; ++k) {
      t.sum7[0][k][j] = kSegFwd7[k][j];
      t.sum7[1][k][j] = kSegBwd7[k][j];
    }
  }
  return t;
}
__constant__ SegTables c_seg = make_seg_tables();
__constant__ double c_node[kSegNodes] = {kSegNode[0], kSegNode[1], kSegNode[2], kSegNode[3],
                                         kSegNode[4], kSegNode[5], kSegNode[6], kSegNode[7]};

// LISA response of one instant (AAK.cc:441-462): F+_I, Fx_I, F+_II, Fx_II times
// the response constant, and cos(orbital phase - phi_S).
__device__ __forceinline__ void lisa_response(const SourceDesc &d, double co, double so, double F[4], double &cosorb_S) {
  const double cS = d.cosqS, sS = d.sinqS, cK = d.cosqK, sK = d.sinqK;
  cosorb_S = co * d.cphiS + so * d.sphiS;
  const double sinorb_S = so * d.cphiS - co * d.sphiS;
  const double cosorb_K = co * d.cosphiK + so * d.sinphiK;
  const double cosq = .5 * cS - kHalfSqrt3 * sS * cosorb_S;
  double c2w, s2w, cos2psi, sin2psi;
  double_angle<double>(kHalfSqrt3 * cS + .5 * sS * cosorb_S, sS * sinorb_S, c2w, s2w);
  const double c2o = co * co - so * so, s2o = 2. * so * co;
  const double cos2phi = c2o * c2w - s2o * s2w, sin2phi = s2o * c2w + c2o * s2w;
  double_angle<double>(.5 * cK - kHalfSqrt3 * sK * cosorb_K - cosq * d.Sdotn, d.psd0 - d.psd1 * co - d.psd2 * so, cos2psi,
                       sin2psi);
  const double cosq1 = .5 * (1. + cosq * cosq);
  F[0] = kHalfSqrt3 * (cosq1 * cos2phi * cos2psi - cosq * sin2phi * sin2psi);
  F[1] = kHalfSqrt3 * (cosq1 * cos2phi * sin2psi + cosq * sin2phi * cos2psi);
  F[2] = kHalfSqrt3 * (cosq1 * sin2phi * cos2psi + cosq * cos2phi * sin2psi);
  F[3] = kHalfSqrt3 * (cosq1 * sin2phi * sin2psi - cosq * cos2phi * cos2psi);
}

// Block-wide sum of N values of every thread (in every thread), for blocks of kSegWarps warps.
template <int N>
__device__ __forceinline__ void block_sum(double *v, double (*red)[8]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0)
    for (int q = 0; q < N; ++q) red[q][threadIdx.x >> 5] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < N; ++q) {
    double x = 0.0;
    for (int k = 0; k < kSegWarps; ++k) x += red[q][k];
    v[q] = x;
  }
}

// Shared scratch of a CTA that sums direct tiles and scans carries.
struct CarryShared {
  double red[8][8];
  double last[kTileChunks * kSegWarps];  // per 32 samples, their last positive Phidot (-1: none)
  double side[2][3];                     // the rates of the samples either side of the tile
  double lastP;
  int before[kSegWarps];
  int is_last;
};

// Phase increments of the samples [start, lim) of a direct tile, by the whole
// CTA: forward sums with the clamped Phidot (the last positive raw one; before
// any in the tile that of the sample before, or C where haveC) and backward
// ones, as the phase pass of k_waveform forms them, a rate's weights in its own
// and its neighbour's AB2 step taken together.  Where the value before the tile
// is not known, f[1] lacks C wC.
//
// Bound by latency: a sample's chain is a search, loads of the piece's knots and
// the rates.  A thread's four samples, and the two either side, go through it
// side by side.  Where the clamp acts over whole tiles (eight sources of 293 tiles
// past their plunge) the phase product takes 0.23 ms; with one warp a tile, each
// waiting for the tiles before it, 3.07.
__device__ void direct_sums(const BatchView &bv, const SourceDesc &d, const KnotWin &w, int start, int end, int lim,
                            bool haveC, double C, SegAgg &A, CarryShared &sh) {
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  double r[kTileChunks + 1][3];
  {
    // spline4w's search, the pieces of all of them found before any is evaluated
    const double *kt = bv.knot_t + d.knot_offset;
    const int last = w.k0 + w.n - 2;
    double t[kTileChunks + 1];
    int k[kTileChunks + 1];
    bool miss = false;
#pragma unroll
    for (int ch = 0; ch <= kTileChunks; ++ch) {  // the last one: warp 0 the sample before the tile, the others the one after
      const int i = (ch < kTileChunks) ? min(start + ch * kTileThreads + tid, lim - 1) : (wp == 0) ? start - 1 : end;
      t[ch] = sample_time(d, min(max(i, 0), d.vlength - 1));
      k[ch] = min(max(w.k0 + __double2int_rd((t[ch] - kt[w.k0]) * w.inv_h), w.k0), last);
    }
#pragma unroll
    for (int ch = 0; ch <= kTileChunks; ++ch)
      miss = miss || (k[ch] < last && kt[k[ch] + 1] <= t[ch]) || (k[ch] > w.k0 && kt[k[ch]] > t[ch]);
    if (miss) {
#pragma unroll
      for (int ch = 0; ch <= kTileChunks; ++ch) {
        while (k[ch] < last && kt[k[ch] + 1] <= t[ch]) ++k[ch];
        while (k[ch] > w.k0 && kt[k[ch]] > t[ch]) --k[ch];
      }
    }
#pragma unroll
    for (int ch = 0; ch <= kTileChunks; ++ch) {
      const int64_t o = d.knot_offset + k[ch];
      phase_rates(d, eval_piece(bv.knot_y[o], bv.knot_y[o + 1], bv.knot_c[o], bv.knot_c[o + 1], kt[k[ch]], kt[k[ch] + 1], t[ch]),
                  r[ch]);
    }
  }
  if (lane == 0 && wp < 2) {
    const bool ok = (wp == 0) ? start >= 1 : (end - 1 < d.i0 && end < d.vlength);
    for (int q = 0; q < 3; ++q) sh.side[wp][q] = ok ? r[kTileChunks][q] : (wp == 0 && q == 1) ? -1.0 : 0.0;
  }
  int clamp = 0;
#pragma unroll
  for (int ch = 0; ch < kTileChunks; ++ch) {
    const int i = start + ch * kTileThreads + tid;
    if (i >= d.i0 && i < lim && !(r[ch][1] > 0.0)) clamp = 1;
  }
  clamp = __syncthreads_or(clamp);
  const double *rb = sh.side[0], *ra = sh.side[1];
  const double P0 = (rb[1] > 0.0) ? rb[1] : haveC ? C : -1.0;  // clamped Phidot before the tile (-1: not known)
  double P[kTileChunks];  // clamped Phidot of the forward samples (-1: that of before the tile, not known)
#pragma unroll
  for (int ch = 0; ch < kTileChunks; ++ch) P[ch] = r[ch][1];
  if (clamp) {
    unsigned pos[kTileChunks];
#pragma unroll
    for (int ch = 0; ch < kTileChunks; ++ch) {
      const int i = start + ch * kTileThreads + tid;
      pos[ch] = __ballot_sync(0xffffffffu, i >= d.i0 && i < lim && r[ch][1] > 0.0);
      const double x = __shfl_sync(0xffffffffu, r[ch][1], pos[ch] ? 31 - __clz(pos[ch]) : 0);
      if (lane == 0) sh.last[ch * kSegWarps + wp] = pos[ch] ? x : -1.0;
    }
    __syncthreads();
#pragma unroll
    for (int ch = 0; ch < kTileChunks; ++ch) {
      const unsigned below = pos[ch] & (0xffffffffu >> (31 - lane));
      const double up = __shfl_sync(0xffffffffu, r[ch][1], below ? 31 - __clz(below) : 0);
      P[ch] = P0;
      for (int k = ch * kSegWarps + wp - 1; k >= 0; --k)
        if (sh.last[k] > 0.0) {
          P[ch] = sh.last[k];
          break;
        }
      if (below) P[ch] = up;
    }
  }
  double v[7] = {0, 0, 0, 0, 0, 0, 0};  // forward sums, backward sums, weight of the Phidot before the tile
#pragma unroll
  for (int ch = 0; ch < kTileChunks; ++ch) {
    const int i = start + ch * kTileThreads + tid;
    if (i < lim && i >= d.i0) {
      const double wt = (i == d.i0 ? 1.0 : 1.5) - ((i + 1 < lim) ? .5 : 0.0);
      v[0] = fma(wt, r[ch][0], v[0]);
      if (clamp && P[ch] < 0.0) v[6] += wt;
      else v[1] = fma(wt, P[ch], v[1]);
      v[2] = fma(wt, r[ch][2], v[2]);
    }
    if (i < lim && i <= d.i0) {
      const double wt = (i >= 1 ? (i == d.i0 ? 1.0 : 1.5) : 0.0) - ((i - 1 >= start && i - 1 >= 1) ? .5 : 0.0);
      for (int q = 0; q < 3; ++q) v[3 + q] = fma(wt, r[ch][q], v[3 + q]);
    }
    if (i == lim - 1) sh.lastP = P[ch];
  }
  block_sum<7>(v, sh.red);
  if (start > d.i0 && start < lim) {
    v[0] -= .5 * rb[0];
    v[2] -= .5 * rb[2];
    if (P0 < 0.0) v[6] -= .5;
    else v[1] -= .5 * P0;
  }
  if (end - 1 < d.i0 && end - 1 >= max(start, 1) && end - 1 < lim)
    for (int q = 0; q < 3; ++q) v[3 + q] -= .5 * ra[q];
  for (int q = 0; q < 3; ++q) {
    A.f[q] = v[q] * d.dt;
    A.b[q] = v[3 + q] * d.dt;
  }
  A.wC = v[6] * d.dt;
  A.lastP = sh.lastP;
  A.hasP = lim - 1 >= max(start, d.i0) && !(clamp && sh.lastP < 0.0);
  A.needC = P0 < 0.0;
}

// The window of tile g in global memory.
__device__ __forceinline__ KnotWin tile_window(const BatchView &bv, const SourceDesc &d, int k0, int nk) {
  KnotWin w{nullptr, nullptr, nullptr, nullptr, nullptr, k0, nk, 0, 0.0};
  const double *kt = bv.knot_t + d.knot_offset;
  const double span = kt[k0 + nk - 1] - kt[k0];
  w.inv_h = (span > 0.0) ? (double)(nk - 1) / span : 0.0;
  return w;
}

// A direct tile by the whole CTA: the rates either side of it, and its sums.
__device__ void direct_tile(const BatchView &bv, const QueueItem &it, int lim, CarryShared &sh) {
  const SourceDesc &d = bv.src[it.s];
  const int start = it.lt * kTileSamples, end = min(start + kTileSamples, d.vlength);
  const int head = (d.i0 <= 0) ? 0 : min(d.i0 / kTileSamples, d.n_tiles - 1);
  SegAgg A;
  direct_sums(bv, d, tile_window(bv, d, it.k0, it.nk), start, end, lim, it.lt <= head, 0.0, A, sh);
  if (threadIdx.x == 0) {
    TilePrep &P = bv.tile_prep[it.g];
    for (int q = 0; q < 3; ++q) {
      P.rb[q] = sh.side[0][q];
      P.ra[q] = sh.side[1][q];
    }
    bv.tile_agg[it.g] = A;
  }
  __syncthreads();  // sh is free again
}

// The phase at a tile's head modulo 2 pi, x0 + (h, l) as a double-double: the
// samples add their tile-local part to it, so that a phase of 1e5 rad loses
// none of its digits to its turns.
__device__ __forceinline__ void reduced_base(double x0, double &h, double &l) {
  double s, e;
  two_sum(x0, h, s, e);
  const double k = rint(s * (1.0 / kTwoPi));
  const double r = fma(-k, 6.283185307179586, s);
  two_sum(r, fma(-k, 2.4492935982947064e-16, e + l), h, l);
}

// The phases that GenPhase keeps after the plunge buffer, those of sample
// i_plunge (AAKPhase.cc:253-257), into the source's slot of frozen (the whole CTA,
// after the carries).  first_frozen: the first sample that takes them.
__device__ __forceinline__ long long first_frozen(const SourceDesc &d) {
  if (d.status != 0 || d.i_plunge < 0 || d.i_plunge >= d.vlength) return (long long)d.vlength;
  return max((long long)d.i_plunge + (long long)d.i_buffer + 2, (long long)d.i0 + 1);
}
// Whether sample i takes the frozen phases (sample i_plunge itself too, so that the two stay equal to the last bit).
__device__ __forceinline__ bool is_frozen(const SourceDesc &d, int i) {
  const long long first = first_frozen(d);
  return first < d.vlength && (i >= first || i == d.i_plunge);
}
__device__ void frozen_phases(const BatchView &bv, int s, const SourceDesc &d, CarryShared &sh) {
  if (first_frozen(d) >= d.vlength) return;
  const int i = d.i_plunge, lt = i / kTileSamples;
  const int64_t g = bv.tile_start[s] + lt;
  const TileHead *H = tile_head(bv, g);
  const int mode = __ldcg(&H->mode);
  double v[3] = {0, 0, 0};
  if (i != d.i0) {
    if (mode > 0) {
      const int seg = (i % kTileSamples) / 256, D = mode;
      const double x = ((double)(i % 256) - kSegMid) * (1.0 / kSegHalf);
      const double *c = reinterpret_cast<const double *>(H + 1) + seg * seg_doubles(D == 4 ? 4 : 7, true);
      for (int q = 0; q < 3; ++q) {
        double p = __ldcg(c + q * (D + 2) + D + 1);
        for (int k = D; k >= 0; --k) p = fma(p, x, __ldcg(c + q * (D + 2) + k));
        v[q] = (i < d.i0) ? -p : p;
      }
    } else {
      const KnotWin w = tile_window(bv, d, bv.tile_knot[2 * g], bv.tile_knot[2 * g + 1]);
      const int start = lt * kTileSamples, end = min(start + kTileSamples, d.vlength);
      SegAgg A;
      if (i > d.i0) {  // the forward sum of the tile's samples before i
        direct_sums(bv, d, w, start, end, i, true, __ldcg(&H->C), A, sh);
        for (int q = 0; q < 3; ++q) v[q] = A.f[q];
      } else {  // the backward sum of those after i
        direct_sums(bv, d, w, i + 1, end, end, true, 0.0, A, sh);
        for (int q = 0; q < 3; ++q) v[q] = -A.b[q];
      }
    }
  }
  if (threadIdx.x == 0) {
    const double X0[3] = {d.gim0, d.Phi0, d.alp0};
    for (int q = 0; q < 3; ++q)
      bv.frozen[3 * s + q] = (i == d.i0) ? X0[q] : X0[q] + (__ldcg(&H->hi[q]) + (__ldcg(&H->lo[q]) + v[q]));
  }
}

// The carries of one source's tiles (the whole CTA): every tile's aggregates of the
// tiles between it and the head, in double-double, forward and backward; a
// forward tile whose Phidot clamp reaches back past its first sample gets the
// value that the tiles before it leave, the last one known, times its weight.
// The waveform gets the phases at the tile's head modulo 2 pi, the phase product
// the signed sums.
__device__ void scan_source(const BatchView &bv, int s, CarryShared &sh) {
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const SourceDesc &d = bv.src[s];
  const int64_t t0 = bv.tile_start[s];
  const int T = d.n_tiles, i0 = d.i0;
  const int head = (i0 <= 0) ? 0 : min(i0 / kTileSamples, T - 1);
  const SegAgg *A = bv.tile_agg + t0;  // written in this launch by other CTAs
  __syncthreads();
#pragma unroll 1
  for (int dir = 1; dir >= -1; dir -= 2) {
    const int n = (dir > 0) ? T - head : head + 1;  // tiles of the chain, the head first
    if (dir < 0 && n == 1) break;
    const int per = (n + kSegWarps * 32 - 1) / (kSegWarps * 32), k0 = min(tid * per, n), k1 = min(k0 + per, n);
    // of the thread's first tile (its only one in a chain of up to 256): loaded once, all together
    const SegAgg &a0 = A[(dir > 0) ? head + min(k0, n - 1) : head - min(k0, n - 1)];
    double x0[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) x0[q] = __ldcg(((dir > 0) ? a0.f : a0.b) + q);
    bool clamp = false;
    double C0 = 0.0;  // the clamped Phidot that the tiles before the thread's leave
    if (dir > 0) {
      bool need = false;
      int last = -1;  // the thread's last tile that leaves one
#pragma unroll 8
      for (int k = k0; k < k1; ++k) {
        const int2 f = __ldcg(reinterpret_cast<const int2 *>(&A[head + k].hasP));
        if (f.x) last = k;
        need = need || f.y;
      }
      clamp = __syncthreads_or(need);
      if (clamp) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int b = __shfl_up_sync(0xffffffffu, last, o);
          if (lane >= o) last = max(last, b);
        }
        if (lane == 31) sh.before[wp] = last;
        int before = __shfl_up_sync(0xffffffffu, last, 1);
        if (lane == 0) before = -1;
        __syncthreads();
        for (int k = 0; k < wp; ++k) before = max(before, sh.before[k]);
        if (before >= 0) C0 = __ldcg(&A[head + before].lastP);
      }
    }
    double C = C0;
    // the increments of tile k of the chain, C the clamped Phidot before it and then after it
    const auto increments = [&](int k, double x[3]) {
      const SegAgg &a = A[(dir > 0) ? head + k : head - k];
#pragma unroll
      for (int q = 0; q < 3; ++q) x[q] = (k == k0) ? x0[q] : __ldcg(((dir > 0) ? a.f : a.b) + q);
      if (clamp) {
        if (__ldcg(&a.needC)) x[1] = fma(C, __ldcg(&a.wC), x[1]);
        if (__ldcg(&a.hasP)) C = __ldcg(&a.lastP);
      }
    };
    double hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0};
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      double x[3];
      increments(k, x);
#pragma unroll
      for (int q = 0; q < 3; ++q) dd_add(hi[q], lo[q], x[q]);
    }
    // exclusive scan of the threads' sums: inside the warp, then over the warps before
    double ph[3], pl[3];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double h = hi[q], l = lo[q];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double bh = __shfl_up_sync(0xffffffffu, h, o), bl = __shfl_up_sync(0xffffffffu, l, o);
        if (lane >= o) dd_add_dd(h, l, bh, bl);
      }
      ph[q] = __shfl_up_sync(0xffffffffu, h, 1);
      pl[q] = __shfl_up_sync(0xffffffffu, l, 1);
      if (lane == 0) ph[q] = pl[q] = 0.0;
      if (lane == 31) {
        sh.red[q][wp] = h;
        sh.red[3 + q][wp] = l;
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double h = 0.0, l = 0.0;
      for (int k = 0; k < wp && k0 < k1; ++k) dd_add_dd(h, l, sh.red[q][k], sh.red[3 + q][k]);
      dd_add_dd(h, l, ph[q], pl[q]);
      ph[q] = h;
      pl[q] = l;
    }
    C = C0;
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      TileHead *H = tile_head(bv, t0 + head + dir * k);
      if (dir > 0 || k > 0) {  // the head's own, of sum 0, is set once
        const double X0[3] = {d.gim0, d.Phi0, d.alp0};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          double h = dir * ph[q], l = dir * pl[q];
          if (!bv.phase_out) reduced_base(X0[q], h, l);
          H->hi[q] = h;
          H->lo[q] = l;
        }
        if (clamp) H->C = C;
      }
      double x[3];
      increments(k, x);
#pragma unroll
      for (int q = 0; q < 3; ++q) dd_add(ph[q], pl[q], x[q]);
    }
  }
  if (bv.phase_out) {
    __syncthreads();
    frozen_phases(bv, s, d, sh);
  }
}

// A matrix row times a quantity's eight node differences (16-byte loads).
__device__ __forceinline__ void seg_row(const double *row, double r[kSegNodes]) {
  const double2 *p = reinterpret_cast<const double2 *>(row);
#pragma unroll
  for (int j = 0; j < kSegNodes / 2; ++j) {
    const double2 v = p[j];
    r[2 * j] = v.x;
    r[2 * j + 1] = v.y;
  }
}
__device__ __forceinline__ double seg_dot(const double r[kSegNodes], const double *dv) {
  const double2 *p = reinterpret_cast<const double2 *>(dv);
  double a = 0.0, b = 0.0;
#pragma unroll
  for (int j = 0; j < kSegNodes / 2; ++j) {
    const double2 v = p[j];
    a = fma(r[2 * j], v.x, a);
    b = fma(r[2 * j + 1], v.y, b);
  }
  return a + b;
}

// The phases' polynomials of a tile (one warp, eight lanes a segment, a lane a
// coefficient) with the tile-local offsets of their segments; returns the
// tile's increment of each phase in tot[].
template <int D, int SD>
__device__ __forceinline__ void phase_segments(const SegTables &tb, const double (*dv)[32], const double *ref, double *out,
                                               int nseg, int bwd, bool head, double dt, double tot[3]) {
  const int lane = threadIdx.x & 31, seg = lane >> 3, k = lane & 7;
  double row[kSegNodes], row8[kSegNodes], fit[kSegNodes];
  const bool on = k < D + 2, used = seg < nseg;
  if constexpr (D == 4) {
    seg_row(tb.sum4[bwd][on ? k : 0], row);
    seg_row(tb.fit4t[k], fit);
  } else {
    seg_row(tb.sum7[bwd][k], row);
    seg_row(tb.sum7[bwd][8], row8);
    seg_row(tb.fit7[k], fit);
  }
  const double sg = (bwd && (k & 1)) ? -1.0 : 1.0;  // x^k at the end of the sum: x = 1 (forward) or -1
  // x^k at the first sample less x^k at the sample before it (the head tile's Euler step)
  double xd = 0.0;
  if (head) {
    double a = 1.0;
    for (int p = 0; p < k; ++p) a *= -kSegMid / kSegHalf;
    xd = (k <= D) ? a - ((k & 1) ? -1.0 : 1.0) : 0.0;
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double *x = dv[q] + 8 * seg;
    double c = seg_dot(row, x), c8 = 0.0;
    if (k == 0) c = fma(kSegMid, ref[q], c);
    else if (k == 1) c = fma(bwd ? -kSegHalf : kSegHalf, ref[q], c);
    c *= dt;
    if constexpr (D == 7) c8 = (k == 0) ? seg_dot(row8, x) * dt : 0.0;
    double T = (on && used) ? sg * c + c8 : 0.0;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) T += __shfl_xor_sync(0xffffffffu, T, o, 8);
    double before = 0.0, all = 0.0;
    if (head) {
      // the first step from t = 0 is an Euler step (AAK.cc:250): r_0 dt instead of (3 r_0 - r_{-1}) dt / 2
      double dr = xd * seg_dot(fit, x);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) dr += __shfl_xor_sync(0xffffffffu, dr, o, 8);
      before = all = -.5 * dt * __shfl_sync(0xffffffffu, dr, 0);
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const double Tg = __shfl_sync(0xffffffffu, T, 8 * g);
      if (bwd ? g > seg : g < seg) before += Tg;
      all += Tg;
    }
    tot[q] = all;
    if (used && on) out[seg * SD + q * (D + 2) + k] = (k == 0) ? c + before : c;
    if (D == 7 && used && k == 0) out[seg * SD + q * (D + 2) + 8] = c8;
  }
}

template <bool kPhase>
__global__ void __launch_bounds__(kSegWarps * 32, 3) k_tile_segments(BatchView bv) {
  constexpr int NQ = kPhase ? kNodeQPhase : kNodeQ, NP = kPhase ? kPolyQPhase : kPolyQ;
  __shared__ __align__(16) SegTables tb;
  __shared__ __align__(16) double s_dv[kSegWarps][NQ][32];
  {
    const double *src = reinterpret_cast<const double *>(&c_seg);
    double *dst = reinterpret_cast<double *>(&tb);
    for (int k = threadIdx.x; k < (int)(sizeof(SegTables) / sizeof(double)); k += blockDim.x) dst[k] = src[k];
  }
  __syncthreads();
  const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
#pragma unroll 1
  for (int64_t jq = (int64_t)blockIdx.x * warps + wp; jq < bv.total_tiles; jq += (int64_t)gridDim.x * warps) {
    const QueueItem it = bv.queue[jq];
    const SourceDesc &d = bv.src[it.s];
    TileHead *H = tile_head(bv, it.g);
    TilePrep P;
    P.ec = 0.0;
    P.K = -1;
    P.stride = 0;
    P.src = it.s;
    for (int q = 0; q < 3; ++q) P.rb[q] = P.ra[q] = 0.0;
    P.rb[1] = -1.0;
    int mode = -1;
    SegAgg A{};
    const int start = it.lt * kTileSamples, end = min(start + kTileSamples, d.vlength);
    const int lim = kPhase ? end : min(end, n_eff(d));
    const int i0 = d.i0, T = d.n_tiles;
    const int head = (i0 <= 0) ? 0 : min(i0 / kTileSamples, T - 1);
    const int dir = (it.lt > head) ? 1 : (it.lt < head) ? -1 : 0;
    if ((it.flags & (kPhase ? kQueueFailed : kQueueNoWave)) == 0) {
      KnotWin w{nullptr, nullptr, nullptr, nullptr, nullptr, it.k0, it.nk, 0, 0.0};
      const double *kt = bv.knot_t + d.knot_offset;
      const double span = kt[w.k0 + w.n - 1] - kt[w.k0];
      w.inv_h = (span > 0.0) ? (double)(w.n - 1) / span : 0.0;
      // ---- node values
      const int seg = lane >> 3, k = lane & 7, nseg = (lim - start + 255) / 256;
      const bool used = seg < nseg;
      double v[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[q] = 0.0;
      if (used) {
        const double t = ((double)(start + 256 * seg - i0) + fma(kSegHalf, c_node[k], kSegMid)) * d.dt;
        const Traj4 q = spline4w(bv, d, t, w);
        double om;
        phase_rates(d, q, v, &om);
        if constexpr (kPhase) {
          v[3] = q.e;
        } else {
          v[3] = pow(om * d.M_phys_sec, 2. / 3.) * d.zeta;
          v[4] = sqrt(1. - q.e * q.e);
          v[5] = q.e;
          if (d.mich) {
            double so, co, cosorb;
            sincos(kTwoPi * t / kYear, &so, &co);
            lisa_response(d, co, so, v + 6, cosorb);
            v[10] = kAUsec * d.sinqS * cosorb;
          } else {
            for (int q4 = 0; q4 < 4; ++q4) v[6 + q4] = d.F0[q4];
          }
        }
      }
      // a forward tile's Phidot is positive throughout, and its sample times are evenly spaced
      const bool even = (start > 0 || (i0 == 0 && d.t_first == 0.0)) && (dir != 0 || (i0 == 0 && start == 0));
      // The source's first and last samples lie outside the nodes.  The boundary layer of the natural spline there falls
      // to 0.27 of itself a knot: with knots no closer than the samples the nodes see it (1.5 samples further in) if it
      // matters; where they are closer (a fast inspiral), the tiles at either end are direct.
      const bool ends = (it.lt == 0 || it.lt == T - 1) && it.nk > end - start;
      bool bad7 = !even || ends || (used && dir >= 0 && !(v[1] > 0.0)), bad4 = false;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {  // v becomes the value at the segment's reference node
        const double r = __shfl_sync(0xffffffffu, v[q], (lane & 24) | kSegRef);
        s_dv[wp][q][lane] = v[q] - r;
        v[q] = r;
      }
      __syncwarp();
      // ---- lanes 0-4 of a segment: the cut fit's coefficients, 5-7: the dropped ones
      double *out = reinterpret_cast<double *>(H + 1);
      constexpr int SD4 = seg_doubles(4, kPhase), SD7 = seg_doubles(7, kPhase);
      const int bwd = dir < 0;
      {
        double row[kSegNodes];
        seg_row(tb.fit4t[k], row);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          const double c = seg_dot(row, s_dv[wp][q] + 8 * seg);
          const double scale = (kPhase || q < 6) ? fabs(v[q]) : (q == 10) ? kAUsec : 1.0;
          if (k >= 5) {
            const bool ok = fabs(c) <= kSegTol * scale;
            if (used && !ok) (k == 5 ? bad4 : bad7) = true;
          }
          const int p = (kPhase || q < 2) ? q : q - 1;  // the waveform keeps no alphadot
          if ((kPhase || q != 2) && k < 5 && used) out[seg * SD4 + 18 + p * 5 + k] = (k == 0) ? c + v[q] : c;
        }
      }
      const bool fail = __any_sync(0xffffffffu, bad7);
      mode = fail ? 0 : (__any_sync(0xffffffffu, bad4) ? 7 : 4);
      if (mode != 0) {
        double tot[3];
        if (mode == 4) {
          phase_segments<4, SD4>(tb, s_dv[wp], v, out, nseg, bwd, dir == 0, d.dt, tot);
        } else {
          double row[kSegNodes];
          seg_row(tb.fit7[k], row);
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            const double c = seg_dot(row, s_dv[wp][q] + 8 * seg);
            const int p = (kPhase || q < 2) ? q : q - 1;
            if ((kPhase || q != 2) && used) out[seg * SD7 + 27 + p * 8 + k] = (k == 0) ? c + v[q] : c;
          }
          phase_segments<7, SD7>(tb, s_dv[wp], v, out, nseg, bwd, dir == 0, d.dt, tot);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) (bwd ? A.b : A.f)[q] = tot[q];
        A.lastP = __shfl_sync(0xffffffffu, v[1], 8 * (nseg - 1));
        A.hasP = !bwd;
      }
      // ---- Taylor table of the tile, about e near its middle; the nodes reach within 2.5 samples of its ends, and the
      // factor 1.25 covers what they leave
      if constexpr (!kPhase) {
        if (d.nmodes <= kTabModes) {
          const double ec = __shfl_sync(0xffffffffu, v[5], 8 * ((nseg - 1) >> 1));
          double de = used ? fabs(v[5] + s_dv[wp][5][lane] - ec) : 0.0;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) de = fmax(de, __shfl_xor_sync(0xffffffffu, de, o));
          int K = 0;
          if (ec > 1e-6) K = taylor_terms_fp64(d.nmodes * (1.25 * de + 1e-15), d.nmodes);  // bounds n |e - e_c| over the tile
          P.ec = ec;
          P.K = (int16_t)K;
          P.stride = (int16_t)(K > 0 ? row_stride<double>(K) : 0);
        }
      }
    }
    if (lane == 0) {
      if (mode == 0) {  // direct tiles from the list's front; those whose sums have no table, and take longest, from its end
        if (!kPhase && P.K <= 0) bv.direct_list[bv.total_tiles - 1 - atomicAdd(bv.seg_ctl + kCtlDirectSlow, 1)] = (int32_t)jq;
        else bv.direct_list[atomicAdd(bv.seg_ctl + kCtlDirectCount, 1)] = (int32_t)jq;
        atomicAdd(bv.seg_ctl + kCtlSource + it.s, 1);
      }
      bv.tile_prep[it.g] = P;
      if (mode != 0) bv.tile_agg[it.g] = A;
      H->C = 0.0;
      H->sgn = (dir < 0) ? -1.0 : 1.0;
      H->ec = P.ec;
      H->mode = mode;
      H->K = max((int)P.K, 0);
      H->stride = P.stride;
      H->nmodes = d.nmodes;
    }
    __syncwarp();  // the node values are read: the next tile's may be written
  }
}

// Between the segments and the waveform: blocks below `carry_blocks` sum the
// direct tiles and then each source's carries (a source without direct tiles
// at once, another by the CTA that finishes its last one); the next ones
// build the tiles' Taylor tables, one thread a (tile, harmonic); the last ones
// help with the direct tiles where there are more of those than carry blocks
// (they come last so that the tables need not wait for them: 2344 direct tiles
// 0.24 -> 0.15 ms).  The small sources are not the segments'.
__global__ void __launch_bounds__(kSegWarps * 32, 2) k_tile_carries(BatchView bv, int carry_blocks, int table_blocks, int rows) {
  __shared__ CarryShared sh;
  const int blk = blockIdx.x, carriers = gridDim.x - table_blocks;
  if (blk >= carry_blocks && blk < carry_blocks + table_blocks) {
    table_row<false>(bv, rows, (int64_t)(blk - carry_blocks) * blockDim.x + threadIdx.x);
    return;
  }
  for (int s = blk; s < bv.nsrc && blk < carry_blocks; s += carry_blocks)
    if (bv.seg_ctl[kCtlSource + s] == 0 && bv.src[s].n_tiles > kSmallTiles) scan_source(bv, s, sh);
  const int n = bv.seg_ctl[kCtlDirectCount], slow = bv.seg_ctl[kCtlDirectSlow];
  for (int m = blk < carry_blocks ? blk : blk - table_blocks; m < n + slow; m += carriers) {
    const QueueItem it = bv.queue[bv.direct_list[m < n ? m : bv.total_tiles - 1 - (m - n)]];
    const SourceDesc &d = bv.src[it.s];
    const int end = min((it.lt + 1) * kTileSamples, d.vlength);
    direct_tile(bv, it, bv.phase_out ? end : min(end, n_eff(d)), sh);
    if (threadIdx.x == 0) {
      __threadfence();
      sh.is_last = atomicAdd(bv.seg_ctl + kCtlSource + bv.nsrc + it.s, 1) == bv.seg_ctl[kCtlSource + it.s] - 1;
      __threadfence();
    }
    __syncthreads();
    if (sh.is_last) scan_source(bv, it.s, sh);
    __syncthreads();
  }
}

// Horner evaluation of coefficients at index OFF .. OFF + N - 1 of a segment (16-byte loads)
template <int OFF, int N>
__device__ __forceinline__ double seg_poly(const double2 *c, double x) {
  auto el = [&](int i) { return (i & 1) ? c[i >> 1].y : c[i >> 1].x; };
  double v = el(OFF + N - 1);
#pragma unroll
  for (int k = N - 2; k >= 0; --k) v = fma(v, x, el(OFF + k));
  return v;
}

// ------------------------------------------------------------------ waveform kernel of the segments
// What a sample needs before its mode sums, and after them.  w: the chain's
// sign, 0 for the sample at t = 0, whose phases are the initial ones.  The
// phases are those of the tile's head modulo 2 pi plus at most 1024 samples', so
// that sincos stays in its fast range (below 1e5 rad).
struct SegRotor {
  double c1, s1, cD, sD, dl;
};
template <int D>
__device__ __forceinline__ SegRotor seg_rotor(const double2 *c, double x, double w, const TileHead &H) {
  constexpr int Q = 3 * (D + 2);
  SegRotor R;
  const double Phi = H.hi[1] + fma(w, seg_poly<D + 2, D + 2>(c, x), H.lo[1]);
  const double gd = seg_poly<Q, D + 1>(c, x), Pd = seg_poly<Q + (D + 1), D + 1>(c, x);
  const double e = seg_poly<Q + 4 * (D + 1), D + 1>(c, x), arm = seg_poly<Q + 9 * (D + 1), D + 1>(c, x);
  R.dl = e - H.ec;
  sincos(fma(Pd, arm, Phi), &R.s1, &R.c1);
  sincos(2.0 * gd * arm, &R.sD, &R.cD);
  return R;
}
// h_I, h_II from the mode sums: the orientation (AAK.cc:425-440, RotCoeff
// KSParMap.cc:532-574) from alpha, the response from its polynomials; every
// quotient of the sample goes through one reciprocal.
template <int D>
__device__ __forceinline__ void seg_output(const double2 *c, double x, double w, const SourceDesc &d, const TileHead &H,
                                           double Sa, double Sb, double Sc, double &hI, double &hII) {
  constexpr int Q = 3 * (D + 2);
  const double gim = H.hi[0] + fma(w, seg_poly<0, D + 2>(c, x), H.lo[0]);
  const double alp = H.hi[2] + fma(w, seg_poly<2 * (D + 2), D + 2>(c, x), H.lo[2]);
  double sa, ca, s2g, c2g;
  sincos(alp, &sa, &ca);
  sincos(2.0 * gim, &s2g, &c2g);
  const double L0 = d.Lc[0] + sa * d.Ls[0] + ca * d.Lq[0];
  const double L1 = d.Lc[1] + sa * d.Ls[1] + ca * d.Lq[1];
  const double L2 = d.Lc[2] + ca * d.Lq[2];
  const double n0 = d.nv[0], n1 = d.nv[1], n2 = d.nv[2];
  const double Ln = L0 * n0 + L1 * n1 + L2 * n2;
  // beta = atan2(by, bx): cos and sin of twice it over by^2 + bx^2
  const double by = -d.Sdotn + d.coslam * Ln, bx = d.beta_c * ca + d.beta_s * sa;
  const double b2 = bx * bx + by * by;
  const double nL0 = n1 * L2 - n2 * L1, nL1 = n2 * L0 - n0 * L2, nL2 = n0 * L1 - n1 * L0;
  const double X = nL0 * d.nxS[0] + nL1 * d.nxS[1] + nL2 * d.nxS[2];
  const double Y = (L0 * d.nxS[0] + L1 * d.nxS[1] + L2 * d.nxS[2]) - (d.Sv[0] * nL0 + d.Sv[1] * nL1 + d.Sv[2] * nL2);
  const double N2 = (nL0 * nL0 + nL1 * nL1 + nL2 * nL2) * (d.nxS_norm * d.nxS_norm);
  double c2b = 1.0, s2b = 0.0, r0, r1;  // atan2(0, 0) = 0
  const double both = b2 * N2;
  if (both > 1e-200) {
    const double inv = 1.0 / both, ib = inv * N2, in = inv * b2;
    c2b = (bx * bx - by * by) * ib;
    s2b = 2.0 * bx * by * ib;
    r0 = 2.0 * X * X * in - 1.0;
    r1 = X * Y * in;
  } else {  // a direction at rounding distance of a singular one: each quotient by itself
    if (b2 > 0.0) {
      c2b = (bx * bx - by * by) / b2;
      s2b = 2.0 * bx * by / b2;
    }
    const double norm = sqrt(nL0 * nL0 + nL1 * nL1 + nL2 * nL2) * d.nxS_norm;
    const double cr = X / norm, sr = Y / norm;
    r0 = 2.0 * cr * cr - 1.0;
    r1 = cr * sr;
  }
  const double cg = c2g * c2b - s2g * s2b, sg = s2g * c2b + c2g * s2b;  // 2 (gamma~ + beta)
  const double Amp = seg_poly<Q + 2 * (D + 1), D + 1>(c, x), se = seg_poly<Q + 3 * (D + 1), D + 1>(c, x);
  const double a = -Amp * Sa, b = -Amp * se * Sb, cc = 2.0 * Amp * Sc;
  const double Ln2 = Ln * Ln;
  // A+ and Ax in the wave frame, rotated to the NK frame
  const double Ap0 = (1.0 + Ln2) * (b * sg - a * cg) + cc * (1.0 - Ln2), Ac0 = 2.0 * Ln * (b * cg + a * sg);
  const double Ap = Ap0 * r0 + Ac0 * r1, Ac = Ac0 * r0 - Ap0 * r1;
  hI = seg_poly<Q + 5 * (D + 1), D + 1>(c, x) * Ap + seg_poly<Q + 6 * (D + 1), D + 1>(c, x) * Ac;
  hII = seg_poly<Q + 7 * (D + 1), D + 1>(c, x) * Ap + seg_poly<Q + 8 * (D + 1), D + 1>(c, x) * Ac;
}

// Bytes of shared memory of one staged tile: source record, head and
// coefficients, Taylor table.
constexpr size_t kSegStageBase = sizeof(SourceDesc) + (size_t)kSegSlotBytes;

// One thread requests queue item j's record, head with coefficients, and
// table into a stage (every size a multiple of 16 bytes); nothing for a
// direct tile, no coefficients for a tile without output.  Returns the tile's
// place in its source and its mode.
__device__ __forceinline__ int2 seg_stage(const BatchView &bv, int64_t j, unsigned char *st, uint64_t *bar) {
  const QueueItem q = bv.queue[j];
  const TileHead *H = tile_head(bv, q.g);
  const int mode = H->mode, K = H->K, nm = H->nmodes;
  const int2 what = make_int2(q.lt, mode);
  if (mode == 0) return what;
  fence_proxy_async_smem();
  const uint32_t nd = (uint32_t)sizeof(SourceDesc);
  const uint32_t nc = (uint32_t)sizeof(TileHead) + (mode > 0 ? 4u * (uint32_t)seg_doubles(mode == 4 ? 4 : 7, false) * 8u : 0u);
  const uint32_t nt = (mode > 0 && K > 0) ? (uint32_t)(nm * H->stride * (int)sizeof(double)) : 0u;
  mbar_arrive_expect_tx(bar, nd + nc + nt);
  bulk_copy_g2s(st, bv.src + q.s, nd, bar);
  bulk_copy_g2s(st + nd, H, nc, bar);
  if (nt) bulk_copy_g2s(st + kSegStageBase, static_cast<const unsigned char *>(bv.tile_tab) + q.g * bv.tab_slot, nt, bar);
  return what;
}

// Persistent CTAs over the queue; a tile's inputs arrive by bulk copies while
// the tile before it runs, and a thread needs no other barrier: its slot m is
// the same in every segment, so x is a constant of the thread.  Bound by FP64
// issue: at 30 harmonics (K = 5) 20 of 29 instructions of a sample are the mode
// sums, J samples a thread share their table loads.  parts (1, or 2 where J
// divides half a tile): queue entries a tile, each with its share of the
// segments, so that a small batch fills the chip.
template <int J, int kMinB>
__global__ void __launch_bounds__(kTileThreads, kMinB) k_wave_segments(BatchView bv, int stage_bytes, int parts) {
  extern __shared__ __align__(16) unsigned char s_stage[];
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ long long s_next[2];
  __shared__ int2 s_what[2];  // place in the source, mode
  const int tid = threadIdx.x;
  const double x = ((double)tid - kSegMid) * (1.0 / kSegHalf);
  const long long units = (long long)bv.total_tiles * parts;
  if (tid == 0) {
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    mbar_init_fence();
    const long long j = (long long)atomicAdd(bv.seg_ctl + kCtlQueue, 1);
    s_next[0] = j;
    if (j < units) s_what[0] = seg_stage(bv, j / parts, s_stage, &s_bar[0]);
  }
  __syncthreads();
  uint32_t parity = 0u;  // bit b: phase of barrier b
  for (int b = 0;; b ^= 1) {
    const long long j = s_next[b];
    if (j >= units) break;
    if (tid == 0) {
      const long long jn = (long long)atomicAdd(bv.seg_ctl + kCtlQueue, 1);
      s_next[b ^ 1] = jn;
      if (jn < units) s_what[b ^ 1] = seg_stage(bv, jn / parts, s_stage + (b ^ 1) * stage_bytes, &s_bar[b ^ 1]);
    }
    const int mode = s_what[b].y;
    const int start = s_what[b].x * kTileSamples;
    if (mode == 0) {  // a direct tile: not this kernel's
      __syncthreads();
      continue;
    }
    unsigned char *st = s_stage + b * stage_bytes;
    const bool ok = mbar_wait_bounded(&s_bar[b], (parity >> b) & 1u);
    parity ^= 1u << b;
    if (!ok) {
      atomicExch(bv.device_status, 1u);
      if (bv.status_report) atomicExch(bv.status_report, 1u);
    }
    const SourceDesc &d = *reinterpret_cast<const SourceDesc *>(st);
    const TileHead &H = *reinterpret_cast<const TileHead *>(st + sizeof(SourceDesc));
    const double2 *co = reinterpret_cast<const double2 *>(st + sizeof(SourceDesc) + sizeof(TileHead));
    const double *tab = reinterpret_cast<const double *>(st + kSegStageBase);
    const int end = ok ? min(start + kTileSamples, d.vlength) : start;  // a copy that did not land: no output
    const int lim = (mode > 0) ? min(end, n_eff(d)) : start;
    const int K = H.K;
    const int sd2 = seg_doubles(mode == 4 ? 4 : 7, false) / 2;
    const int first = (int)(j % parts) * (kTileChunks / parts), past = first + kTileChunks / parts;
#pragma unroll 1
    for (int g0 = first; g0 < past; g0 += J) {
      if (start + 256 * g0 >= end) break;
      double dl[J], c1[J], s1[J], cD[J], sD[J], Sa[J], Sb[J], Sc[J];
#pragma unroll
      for (int m = 0; m < J; ++m) {
        Sa[m] = Sb[m] = Sc[m] = 0.0;
        c1[m] = cD[m] = 1.0;
        s1[m] = sD[m] = dl[m] = 0.0;
        if (start + 256 * (g0 + m) < lim) {
          const double2 *c = co + (g0 + m) * sd2;
          const double w = (start + 256 * (g0 + m) + tid == d.i0) ? 0.0 : H.sgn;
          const SegRotor R = (mode == 4) ? seg_rotor<4>(c, x, w, H) : seg_rotor<7>(c, x, w, H);
          dl[m] = R.dl;
          c1[m] = R.c1;
          s1[m] = R.s1;
          cD[m] = R.cD;
          sD[m] = R.sD;
        }
      }
      switch (K) {
        case 4: mode_sums_fp64<4, J>(tab, d.nmodes, H.stride, dl, c1, s1, cD, sD, Sa, Sb, Sc); break;
        case 5: mode_sums_fp64<5, J>(tab, d.nmodes, H.stride, dl, c1, s1, cD, sD, Sa, Sb, Sc); break;
        case 6: mode_sums_fp64<6, J>(tab, d.nmodes, H.stride, dl, c1, s1, cD, sD, Sa, Sb, Sc); break;
        case 8: mode_sums_fp64<8, J>(tab, d.nmodes, H.stride, dl, c1, s1, cD, sD, Sa, Sb, Sc); break;
        case 10: mode_sums_fp64<10, J>(tab, d.nmodes, H.stride, dl, c1, s1, cD, sD, Sa, Sb, Sc); break;
        default: break;
      }
#pragma unroll
      for (int m = 0; m < J; ++m) {
        const int i = start + 256 * (g0 + m) + tid;
        if (i >= end) continue;
        const double t = sample_time(d, i);
        double hI = 0.0, hII = 0.0;
        if (i < lim) {
          const double2 *c = co + (g0 + m) * sd2;
          if (K == 0)  // no table for this tile: per-sample Miller recurrence
            mode_sums_miller(bv.bessel_start + d.bessel_offset, d.nmodes, dl[m] + H.ec, c1[m], s1[m], cD[m], sD[m],
                             Sa[m], Sb[m], Sc[m]);
          const double w = (i == d.i0) ? 0.0 : H.sgn;
          if (mode == 4) seg_output<4>(c, x, w, d, H, Sa[m], Sb[m], Sc[m], hI, hII);
          else seg_output<7>(c, x, w, d, H, Sa[m], Sb[m], Sc[m], hI, hII);
          if (i > d.i_plunge) {
            const double t_plunge = sample_time(d, d.i_plunge);
            const double t_zero = t_plunge + d.dt * d.i_buffer;
            const double wgt = exp((t_plunge - t_zero) / (t - t_plunge) + (t_plunge - t_zero) / (t - t_zero)) + 1.;
            hI = hI / wgt;
            hII = hII / wgt;
          }
        }
        store_h(bv, d.out_offset + i, hI, hII);
        if (bv.t_out) bv.t_out[d.out_offset + i] = (d.status != 0) ? 0.0 : t;
      }
    }
    __syncthreads();  // the stage is free, and the next item known
  }
}

// The phase product of a tile of polynomial segments: the eight rows of
// GenPhase's packing, sums in its order (AAKPhase.cc:347-354).
template <int D>
__device__ __forceinline__ void phase_rows(const BatchView &bv, const SourceDesc &d, const TileHead &H, const double2 *co,
                                           int start, int end, const double *frozen) {
  constexpr int Q = 3 * (D + 2);
  const int tid = threadIdx.x;
  const double x = ((double)tid - kSegMid) * (1.0 / kSegHalf);
  const int64_t sr = bv.phase_stride;
#pragma unroll
  for (int sg = 0; sg < kTileChunks; ++sg) {
    const int i = start + 256 * sg + tid;
    if (i >= end) break;
    const double2 *c = co + sg * (seg_doubles(D, true) / 2);
    const double w = (i == d.i0) ? 0.0 : H.sgn;  // t = 0: the initial phases
    double X[3] = {d.gim0 + (H.hi[0] + fma(w, seg_poly<0, D + 2>(c, x), H.lo[0])),
                   d.Phi0 + (H.hi[1] + fma(w, seg_poly<D + 2, D + 2>(c, x), H.lo[1])),
                   d.alp0 + (H.hi[2] + fma(w, seg_poly<2 * (D + 2), D + 2>(c, x), H.lo[2]))};
    if (is_frozen(d, i))
      for (int q = 0; q < 3; ++q) X[q] = frozen[q];
    const double gd = seg_poly<Q, D + 1>(c, x), Pd = seg_poly<Q + (D + 1), D + 1>(c, x);
    const double ad = seg_poly<Q + 2 * (D + 1), D + 1>(c, x);
    double *o = bv.phase_out + d.out_offset + i;
    o[0] = sample_time(d, i);
    o[sr] = X[1];
    o[2 * sr] = X[1] + X[0];
    o[3 * sr] = X[1] + X[0] + X[2];
    o[4 * sr] = Pd;
    o[5 * sr] = Pd + gd;
    o[6 * sr] = Pd + gd + ad;
    o[7 * sr] = seg_poly<Q + 3 * (D + 1), D + 1>(c, x);
  }
}
