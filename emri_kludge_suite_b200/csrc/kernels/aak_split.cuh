// The split-precision waveform of a batch (with the tile pre-pass): FP64
// spline, rates, AB2 phase sums and angle reductions, FP32 response, Bessel
// tables and harmonic recurrence.  Included in aak_dense.cu.
//
// A CTA takes one tile at a time from the work queue, in the passes of the
// kernel that does everything inside the tile (the same operations and sums in
// the same order), arranged for what bounds it: waits.  No pipe is saturated
// (issue 64 % of the cycles, FMA 32, FP64 21, LSU 33); the barriers and the copies
// at a tile's start were 30 % of that kernel's time.  So
// - the next tile's record, parameters and knot window are requested while the
//   last quarter of this tile's sums runs, and five barriers a tile stand for
//   the ten of before;
// - the next item is taken there and not in the middle of the tile.  A CTA that
//   holds an item while it still sums another one keeps that item's successors
//   waiting in their look-back: with few sources, most of the time of the
//   kernel;
// - what stays in registers over the harmonic sums is kept small: at 80
//   registers (three CTAs an SM) every spilled one is loaded in their loop.
// Measured: 64 sources, 1.1e8 samples, 30 harmonics 8.06 -> 7.41 ms; 12 sources
// integrated backwards with 11 to 61 harmonics 2.11 -> 1.36 ms.  Slower: a
// thread's four samples consecutive in both passes with the rates in registers
// (+5 %: more instructions), a fourth CTA at 64 registers (+17 %), two samples
// side by side (+6 %), two iterations of the phase pass side by side (+1 %).

struct alignas(16) SplitShared {
  SourceDesc desc, next_desc;  // this tile's, and the next one's on its way
  TilePrep prep, next_prep;
  QueueItem item;
  double4 wy[kWin], wc[kWin], wb[kWin], wd[kWin];
  double wt[kWin + 2];
  double red[2][3][kTileThreads / 32];
  double cy[7], lastP;
  Geom<float> geom;
  uint64_t mbar[2];  // record + parameters + window; table
  int win[3];        // first knot, knots, offset in wt
  int have;          // item holds a tile (0: the queue is empty)
};

template <int kJoint, int kMinB>
__global__ void __launch_bounds__(kTileThreads, kMinB) k_wave_split(BatchView bv) {
  static_assert(kTileChunks == 4 && kTileThreads == 256, "four slots a thread");
  static_assert(kTileChunks % kJoint == 0, "joint samples must divide the chunks");
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ SplitShared sh;
  double *const sv_e = reinterpret_cast<double *>(s_raw), *const sv_om = sv_e + kTileSamples, *const sv_gim = sv_e + 2 * kTileSamples,
               *const sv_Phi = sv_e + 3 * kTileSamples, *const sv_alp = sv_e + 4 * kTileSamples,
               *const sv_nu = sv_e + 5 * kTileSamples, *const sv_gd = sv_e + 6 * kTileSamples;
  float *const tab = reinterpret_cast<float *>(sv_e + kDynVals * kTileSamples);
  const int tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(&sh.mbar[0], 1);
    mbar_init(&sh.mbar[1], 1);
    mbar_init_fence();
  }
  __syncthreads();
  // One thread takes the queue's next item and requests its record, parameters
  // and knot window (their last readers are behind a barrier).  Items leave the queue in chain order and a CTA's next item
  // comes after its current one, whose sums are published before it can wait
  // for anything of the next: one item ahead cannot stall the chains.
  const auto fetch = [&]() {
    const long long j = (long long)atomicAdd(bv.work_counter, 1ull);
    sh.have = (j < bv.total_tiles) ? 1 : 0;
    if (j < bv.total_tiles) {
      const QueueItem q = bv.queue[j];
      sh.item = q;
      if (!(q.flags & kQueueNoWave))
        issue_stage(bv, q, &sh.next_desc, &sh.next_prep, sh.win, sh.wt, sh.wy, sh.wc, &sh.mbar[0]);
    }
  };
  if (tid == 32) fetch();
  __syncthreads();
  uint32_t ph0 = 0u, ph1 = 0u;  // phase parity of the two barriers
  bool bad = false;             // a copy did not land
  const auto report = [&]() {
    atomicExch(bv.device_status, 1u);
    if (bv.status_report) atomicExch(bv.status_report, 1u);
  };
#pragma unroll 1
  while (sh.have) {
    TileCtx c;
    c.s = sh.item.s;
    c.lt = sh.item.lt;
    c.g = sh.item.g;
    c.start = c.lt * kTileSamples;
    if (sh.item.flags & kQueueNoWave) {
      // failed source, or a tile entirely after the taper: zeros, and an empty aggregate for the chain
      const SourceDesc &dz = bv.src[c.s];
      c.end = min(c.start + kTileSamples, dz.vlength);
      for (int ch = 0; ch < kTileChunks; ++ch) {
        const int i = c.start + ch * kTileThreads + tid;
        if (i < c.end) {
          store_h(bv, dz.out_offset + i, 0.0, 0.0);
          if (bv.t_out) bv.t_out[dz.out_offset + i] = (dz.status != 0) ? 0.0 : sample_time(dz, i);
        }
      }
      __syncthreads();  // the item's readers
      if (tid == 0) {
        const double zero[3] = {0.0, 0.0, 0.0};
        publish_aggregate(bv, c.g, zero, 0.0, false);
      }
      if (tid == 32) fetch();
      __syncthreads();
      continue;
    }
    const SourceDesc &d = sh.desc;
    const TilePrep &pr = sh.prep;
    if (!mbar_wait_bounded(&sh.mbar[0], ph0)) bad = true;
    ph0 ^= 1u;
    KnotWin w{sh.wt + sh.win[2], sh.wy, sh.wc, sh.wb, sh.wd, sh.win[0], sh.win[1], 0, 0.0};
    w.staged = w.n > 0 && w.n <= kWin;
    if (!bad) {
      constexpr int kDescWords = (int)(sizeof(SourceDesc) / 16), kPrepWords = (int)(sizeof(TilePrep) / 16);
      static_assert(kDescWords + kPrepWords < kTileThreads - 1, "a thread a word, the last one makes the response constants");
      if (tid < kDescWords) reinterpret_cast<uint4 *>(&sh.desc)[tid] = reinterpret_cast<const uint4 *>(&sh.next_desc)[tid];
      else if (tid < kDescWords + kPrepWords)
        reinterpret_cast<uint4 *>(&sh.prep)[tid - kDescWords] = reinterpret_cast<const uint4 *>(&sh.next_prep)[tid - kDescWords];
      if (tid == kTileThreads - 1) make_geom(sh.next_desc, sh.geom);
      window_pieces(bv, sh.next_desc, w);
    }
    if (__syncthreads_or(bad)) {  // report it and stop this CTA
      if (tid == 0) report();
      return;
    }
    const bool has_tab = pr.K > 0 && d.nmodes <= kTabModes;
    if (tid == 0 && has_tab) {  // the tile's Taylor table, one row a pair of harmonics
      fence_proxy_async_smem();
      const uint32_t bytes = (uint32_t)((d.nmodes + 1) >> 1) * (uint32_t)pr.stride * (uint32_t)sizeof(float);
      mbar_arrive_expect_tx(&sh.mbar[1], bytes);
      bulk_copy_g2s(tab, static_cast<const unsigned char *>(bv.tile_tab) + c.g * bv.tab_slot, bytes, &sh.mbar[1]);
    }
    c.end = min(c.start + kTileSamples, d.vlength);
    c.neff = n_eff(d);
    c.head = (d.i0 <= 0) ? 0 : min(d.i0 / kTileSamples, d.n_tiles - 1);
    const int lim = min(c.end, c.neff);  // samples [start, lim) feed the output
    // chain direction: +1 after the head tile, -1 before it, 0 the head
    const int dir = (c.lt > c.head) ? 1 : (c.lt < c.head) ? -1 : 0;
    // A forward tile whose Phidot clamp reaches back past its first sample
    // needs the chain's clamped Phidot first.
    const bool needC = dir > 0 && !(pr.rb[1] > 0.0);
    if (needC) {
      if (tid < 32) {
        double hi[3], lo[3], C;
        look_back_warp(bv, c, 1, hi, lo, C);
        if (tid == 0) {
          for (int q = 0; q < 3; ++q) {
            sh.cy[q] = hi[q];
            sh.cy[3 + q] = lo[q];
          }
          sh.cy[6] = C;
        }
      }
      __syncthreads();
    }
    const double Pin = (pr.rb[1] > 0.0) ? pr.rb[1] : (needC ? sh.cy[6] : 0.0);  // clamped Phidot just before the tile
    // ---------------- (A) spline and rates of every sample, four a thread
    // (slots tid + 256 ch); the rates sit in the phase slots until (D)
    int nonpos = 0;  // a forward sample whose raw Phidot is not positive
#pragma unroll 1
    for (int ch = 0; ch < kTileChunks; ++ch) {
      const int sl = ch * kTileThreads + tid, i = c.start + sl;
      Traj4 q = {0, 0, 0, 0};
      double r[3] = {0, 0, 0}, om = 0.0;
      if (i < lim) {
        q = spline4w(bv, d, sample_time(d, i), w);
        phase_rates(d, q, r, &om);
        if (i >= d.i0 && !(r[1] > 0.0)) nonpos = 1;
      }
      sv_e[sl] = q.e;
      sv_om[sl] = om * d.M_phys_sec;
      sv_gim[sl] = r[0];
      sv_Phi[sl] = r[1];
      sv_alp[sl] = r[2];
      sv_gd[sl] = r[0];
    }
    nonpos = __syncthreads_or(nonpos);
    // (B) the clamped Phidot (AAK.cc:254: the raw rate if positive, else the
    //     previous clamped value) where the clamp acts: one thread walks the
    //     tile and parks it in the nu slots
    if (nonpos) {
      if (tid == 0) {
        double P = Pin;
        for (int sl = 0; sl < lim - c.start; ++sl)
          if (c.start + sl >= d.i0) {
            const double raw = sv_Phi[sl];
            if (raw > 0.0) P = raw;
            sv_nu[sl] = P;
          }
      }
      __syncthreads();
    }
    // ---------------- (C) AB2 increments of the thread's four consecutive
    // slots, their running sums, and one block scan of the thread totals
    const int j0 = 4 * tid;
    const bool back = d.i0 > 0 && c.start <= d.i0;  // the tile has a backward region
    double incF[4][3], incB[4][3], nuv[4];
    double tF[3] = {0, 0, 0}, tB[3] = {0, 0, 0};
    {
      double rm[3], Pm;  // rates and clamped Phidot of the slot before
      if (j0 == 0) {
        rm[0] = pr.rb[0];
        rm[2] = pr.rb[2];
        Pm = Pin;
      } else {
        rm[0] = sv_gim[j0 - 1];
        rm[2] = sv_alp[j0 - 1];
        Pm = nonpos ? sv_nu[j0 - 1] : sv_Phi[j0 - 1];
      }
      double rc[3] = {sv_gim[j0], sv_Phi[j0], sv_alp[j0]};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = c.start + j0 + k;
        const bool in = i < lim, vf = in && i >= d.i0, vb = in && i >= 1 && i <= d.i0;
        double rn[3];  // rates of the slot after (the tile's last slot: the sample after the tile)
        if (k < 3 || j0 + 4 < kTileSamples) {
          rn[0] = sv_gim[j0 + k + 1];
          rn[1] = sv_Phi[j0 + k + 1];
          rn[2] = sv_alp[j0 + k + 1];
        } else {
          rn[0] = pr.ra[0];
          rn[1] = pr.ra[1];
          rn[2] = pr.ra[2];
        }
        const double P = (vf && nonpos) ? sv_nu[j0 + k] : rc[1];
        for (int q = 0; q < 3; ++q) incF[k][q] = incB[k][q] = 0.0;
        if (vf) {
          if (i == d.i0) {
            incF[k][0] = rc[0] * d.dt;
            incF[k][1] = P * d.dt;
            incF[k][2] = rc[2] * d.dt;
          } else {
            incF[k][0] = (1.5 * rc[0] - .5 * rm[0]) * d.dt;
            incF[k][1] = (1.5 * P - .5 * Pm) * d.dt;
            incF[k][2] = (1.5 * rc[2] - .5 * rm[2]) * d.dt;
          }
        }
        if (vb) {
          if (i == d.i0) {
            incB[k][0] = rc[0] * d.dt;
            incB[k][1] = rc[1] * d.dt;
            incB[k][2] = rc[2] * d.dt;
          } else {
            incB[k][0] = (1.5 * rc[0] - .5 * rn[0]) * d.dt;
            incB[k][1] = (1.5 * rc[1] - .5 * rn[1]) * d.dt;
            incB[k][2] = (1.5 * rc[2] - .5 * rn[2]) * d.dt;
          }
        }
        nuv[k] = ((i > d.i0) ? P : rc[1]) / 2. / kPi;
        // the owner of the tile's last output sample records its clamped Phidot (forward samples)
        if (vf && i == lim - 1) sh.lastP = P;
        rm[0] = rc[0];
        rm[2] = rc[2];
        Pm = P;
        rc[0] = rn[0];
        rc[1] = rn[1];
        rc[2] = rn[2];
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        tF[q] += incF[k][q];
        tB[q] += incB[k][q];
      }
    double runF[3], runB[3] = {0.0, 0.0, 0.0}, eF[3], eB[3] = {0.0, 0.0, 0.0};
    // (its barrier orders every read of (C) before the writes of (D))
    block_exscan3x2(tF, tB, back, sh.red, eF, runF, eB, runB);
    const double X0[3] = {d.gim0, d.Phi0, d.alp0};
    // ---------------- (D) tile-local phases: forward, the increments of the
    // tile's samples before i; backward, those of its samples up to i
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int sl = j0 + k, i = c.start + sl;
      double *const svq[3] = {sv_gim, sv_Phi, sv_alp};
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        svq[q][sl] = (i > d.i0) ? eF[q] : eB[q] + incB[k][q];
        eF[q] += incF[k][q];
        eB[q] += incB[k][q];
      }
      sv_nu[sl] = nuv[k];
    }
    // chain carry: warp 0 publishes this tile's aggregate, looks back for the
    // exclusive prefix and publishes the inclusive record
    if (tid < 32) {
      const bool hasF = lim - 1 >= max(c.start, d.i0);  // forward output samples in the tile
      double hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0}, C = 0.0;
      if (needC) {
        for (int q = 0; q < 3; ++q) {
          hi[q] = sh.cy[q];
          lo[q] = sh.cy[3 + q];
        }
        C = sh.cy[6];
      } else if (dir != 0) {
        const TileAgg agg{{(dir > 0) ? runF[0] : runB[0], (dir > 0) ? runF[1] : runB[1], (dir > 0) ? runF[2] : runB[2]},
                          hasF ? sh.lastP : 0.0, hasF, true};
        look_back_warp(bv, c, dir, hi, lo, C, agg);
      }
      if (tid == 0) {
        double fh[3] = {0, 0, 0}, fl[3] = {0, 0, 0}, bh[3] = {0, 0, 0}, bl[3] = {0, 0, 0};
        for (int q = 0; q < 3; ++q) {
          sh.cy[q] = hi[q];
          sh.cy[3 + q] = lo[q];
          if (dir >= 0) {
            fh[q] = hi[q];
            fl[q] = lo[q];
            dd_add(fh[q], fl[q], runF[q]);
          }
          if (dir <= 0) {
            bh[q] = hi[q];
            bl[q] = lo[q];
            dd_add(bh[q], bl[q], runB[q]);
          }
        }
        publish_inclusive(bv, c.g, fh, fl, bh, bl, hasF ? sh.lastP : C);
      }
    }
    __syncthreads();
    // the phases of this thread's own samples: X0 + carry + local part
    // (forward), X0 - (carry + increments after the sample) (backward)
    {
      const double hi[3] = {sh.cy[0], sh.cy[1], sh.cy[2]}, lo[3] = {sh.cy[3], sh.cy[4], sh.cy[5]};
#pragma unroll 1
      for (int sl = tid; sl < lim - c.start; sl += kTileThreads) {
        const int i = c.start + sl;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          double *const sv = sv_gim + q * kTileSamples;
          const double v = sv[sl];
          sv[sl] = (i > d.i0) ? X0[q] + (hi[q] + (lo[q] + v))
                   : (i == d.i0) ? X0[q] : X0[q] - (hi[q] + (lo[q] + (runB[q] - v)));
        }
      }
    }
    // ---------------- harmonic sums, kJoint samples a thread at a time
    const int K = max((int)pr.K, 0), rs = (int)pr.stride;
    if (has_tab) {
      if (!mbar_wait_bounded(&sh.mbar[1], ph1)) {
        bad = true;  // the CTA stops at its next tile
        report();
      }
      ph1 ^= 1u;
    }
#pragma unroll 1
    for (int g0 = 0; g0 < 4; g0 += kJoint) {
      if (tid == 32 && g0 + kJoint == 4) fetch();
      SamplePrep<float> S[kJoint];
      float dl[kJoint], c1[kJoint], s1[kJoint], cD[kJoint], sD[kJoint], Sa[kJoint], Sb[kJoint], Sc[kJoint], d0[kJoint];
      double ph[kJoint];
#pragma unroll
      for (int m = 0; m < kJoint; ++m) {
        const int sl = (g0 + m) * kTileThreads + tid, i = c.start + sl;
        if (i < lim) {
          S[m] = prep_split(d, sh.geom, pr.ec, sample_time(d, i), sv_e[sl], sv_om[sl], sv_gim[sl], sv_Phi[sl],
                            sv_alp[sl], sv_nu[sl], sv_gd[sl]);
        } else {
          S[m] = SamplePrep<float>{};
          S[m].c1 = S[m].cD = 1.f;
        }
        dl[m] = S[m].dl;
        ph[m] = S[m].ph;
        d0[m] = S[m].d0;
        c1[m] = S[m].c1;
        s1[m] = S[m].s1;
        cD[m] = S[m].cD;
        sD[m] = S[m].sD;
      }
      switch (K) {
        case 2: mode_sums_split<2, kJoint>(tab, d.nmodes, rs, dl, c1, s1, cD, sD, ph, d0, Sa, Sb, Sc); break;
        case 3: mode_sums_split<3, kJoint>(tab, d.nmodes, rs, dl, c1, s1, cD, sD, ph, d0, Sa, Sb, Sc); break;
        case 4: mode_sums_split<4, kJoint>(tab, d.nmodes, rs, dl, c1, s1, cD, sD, ph, d0, Sa, Sb, Sc); break;
        case 6: mode_sums_split<6, kJoint>(tab, d.nmodes, rs, dl, c1, s1, cD, sD, ph, d0, Sa, Sb, Sc); break;
        default: break;
      }
#pragma unroll
      for (int m = 0; m < kJoint; ++m) {
        const int sl = (g0 + m) * kTileThreads + tid, i = c.start + sl;
        if (i >= c.end) continue;
        const double t = sample_time(d, i);
        double hI = 0.0, hII = 0.0;
        if (i < c.neff) {
          if (K == 0) {  // no table for this tile: per-sample Miller recurrence in FP64
            double a64, b64, c64;
            mode_sums_miller(bv.bessel_start + d.bessel_offset, d.nmodes, sv_e[sl], (double)c1[m], (double)s1[m], (double)cD[m],
                             (double)sD[m], a64, b64, c64);
            Sa[m] = (float)a64;
            Sb[m] = (float)b64;
            Sc[m] = (float)c64;
          }
          finish<float>(S[m], Sa[m], Sb[m], Sc[m], hI, hII);
          if (i > d.i_plunge) {
            const double t_plunge = sample_time(d, d.i_plunge), t_zero = t_plunge + d.dt * d.i_buffer;
            const double wgt = exp((t_plunge - t_zero) / (t - t_plunge) + (t_plunge - t_zero) / (t - t_zero)) + 1.;
            hI = hI / wgt;
            hII = hII / wgt;
          }
        }
        store_h(bv, d.out_offset + i, hI, hII);
        if (bv.t_out) bv.t_out[d.out_offset + i] = t;
      }
    }
    __syncthreads();
  }
}
