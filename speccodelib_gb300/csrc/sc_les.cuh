// Passes of the LES right-hand side in gradient form.
//
// smag.f90:21-32 transforms u, the vorticity and the six S_ij back (12
// fields); all of them are combinations of u and its nine derivatives, and a
// derivative costs nothing before the transform along its own axis.  So u and
// d/dz u leave the z-inverse (6 fields), the y-inverse adds d/dy u (9), the
// x-pass forms d/dx u from the rows of u and every product in physical space.
// Forward, the stress divergence -i k_j tau_ij (spectral_les.f90:232-234) is
// taken axis by axis the same way: the x-pass returns L_i - i kx tau_i1 and
// the five stresses still needed (8 fields), the y-forward leaves
// L_i - i kx tau_i1 - i ky tau_i2 and tau_i3 (6), which the z-forward
// combines.  71 field passes per right-hand side instead of 97, and 29
// strided-axis transforms instead of 38: the Smagorinsky step at 256^3 FP32
// 7.01 -> 5.22 ms, at 128^3 (dynamic) 1.51 -> 1.09 ms, at 128^3 FP64 17.7 -> 11.3 ms.
// The rows that it serves: les_gradient_rows (sc_xgroup.cuh); others keep the
// twelve fields.
#pragma once
#include "sc_tma_passes.cuh"

namespace sc {

// Slots of the LES work fields, in the order of each pass.
//   after the z-inverse: u (0-2), d/dz u (3-5)
//   after the y-inverse: u (0-2), d/dz u (3-5), d/dy u (6-8)
//   after the x-pass:    A_i = L_i - i kx tau_i1 (0-2), tau_12, tau_22, tau_23
//                        (3-5), tau_13 (6), tau_33 (7)
//   after the y-forward: B_i = A_i - i ky tau_i2 (0-2), tau_13 (6), tau_23
//                        (5), tau_33 (7)
__host__ __device__ constexpr int les_t3(int i) { return i == 0 ? 6 : (i == 1 ? 5 : 7); }   // tau_i3

// Shared memory of the y passes below: two or three tiles (one of work, or
// the ring of pairs), so that two CTAs share an SM.
template <typename T, int LOGN> struct LesYCfg {
  using Cfg = TmaCfg<T, LOGN>;
  static constexpr size_t SMEM = 3 * Cfg::TILE_BYTES + kSmemAlignPad;
};

// y-inverse of six fields in place (u, d/dz u), with d/dy u of the first three
// as fields 6-8 from the same tiles: 15 field passes, where transforming nine
// fields takes 18.  Persistent, two tiles in flight and one of work; bound by
// DRAM and the transforms' barriers as pencil_tma_kernel.
template <typename T, int LOGN>
__global__ void __launch_bounds__(TmaCfg<T, LOGN>::NT, 2)
les_yinv_kernel(const __grid_constant__ CUtensorMap map, TmaPass<T> tp, Geom g, const C2<T>* __restrict__ tw) {
  pdl_wait();
  using Cfg = TmaCfg<T, LOGN>;
  using E = typename Cfg::Engine;
  using C = C2<T>;
  constexpr int P = Cfg::P;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  __shared__ __align__(8) uint64_t bars[2];
  if (launch_failed(tp.err)) return;
  auto buf = [&](int b) { return reinterpret_cast<C*>(smraw + (size_t)b * Cfg::TILE_BYTES); };
  C* const work = buf(2);
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  __syncthreads();
  const int per = tp.ntx * tp.nouter, total = per * 6, step = gridDim.x;
  auto decode = [&](int job, int& kx0, int& outer, int& f) { tile_of(tp, job, P, kx0, outer, f); };
  auto issue = [&](int job, int b) {
    int kx0, outer, f;
    decode(job, kx0, outer, f);
    tma_issue_tile<Cfg>(buf(b), &map, &bars[b], 1, kx0, outer, f, P, Cfg::TILE_BYTES);
  };
  int job = blockIdx.x;
  if (threadIdx.x == 0 && job < total) issue(job, 0);
  for (int it = 0; job < total; job += step, ++it) {
    const int b = it & 1;
    if (threadIdx.x == 0 && job + step < total) {
      fence_proxy_async();
      issue(job + step, b ^ 1);
    }
    if (!mbar_wait_bounded(&bars[b], (it >> 1) & 1, tp.err)) {
      // the copy into the other buffer still has to land
      if (threadIdx.x == 0 && job + step < total) mbar_wait_bounded(&bars[b ^ 1], ((it + 1) >> 1) & 1, nullptr);
      return;
    }
    int kx0, outer, f;
    decode(job, kx0, outer, f);
    const int nvalid = min(P, g.nxh - kx0);
    C* __restrict__ fp = tp.base + f * tp.field + outer * tp.outer_stride + kx0;
    C out[E::JL][E::RL];
    auto store = [&](C* __restrict__ q) {
#pragma unroll
      for (int a = 0; a < E::JL; ++a)
#pragma unroll
        for (int r = 0; r < E::RL; ++r) {
          int p, n;
          if (E::out_pos(a, r, p, n) && p < nvalid) q[n * tp.axis_stride + p] = out[a][r];
        }
    };
    if (f < 3) {
      E::template run_map<true>(out, buf(b), work, tw,
                                [](C x, int, int n) { return cmuli(cscale(x, (T)wavenum(n, Cfg::N))); });
      store(fp + 6 * tp.field);
    }
    E::template run_smem<true>(out, buf(b), tw);
    store(fp);
  }
}

// y-forward of the x-pass's eight fields with the ky part of the stress
// divergence: the pairs (A_i, tau_i2) leave as B_i = A_i - i ky tau_i2 (tau_23
// as itself too), tau_13 and tau_33 alone.  14 field passes.  Persistent; the
// tiles of all pairs and singles stream through one three-deep ring, tau_i2
// before its A_i, its transformed values waiting in its tile.
template <typename T, int LOGN>
__global__ void __launch_bounds__(TmaCfg<T, LOGN>::NT, 2)
les_yfwd_kernel(const __grid_constant__ CUtensorMap map, TmaPass<T> tp, Geom g, const C2<T>* __restrict__ tw) {
  pdl_wait();
  using Cfg = TmaCfg<T, LOGN>;
  using E = FFTEngine<T, LOGN, Cfg::P, Cfg::P, Cfg::NT, true, 0, true>;
  using C = C2<T>;
  constexpr int P = Cfg::P;
  constexpr int NS = 3;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  __shared__ __align__(8) uint64_t bars[NS];
  if (launch_failed(tp.err)) return;
  auto buf = [&](int b) { return reinterpret_cast<C*>(smraw + (size_t)b * Cfg::TILE_BYTES); };
  if (threadIdx.x == 0) {
    for (int b = 0; b < NS; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  __syncthreads();
  // units of this CTA: u = blockIdx.x + i gridDim.x over [pairs | singles]
  const int per = tp.ntx * tp.nouter, pairs = 3 * per, units = 5 * per, first = blockIdx.x, step = gridDim.x;
  auto count = [&](int n) { return n > first ? (n - first - 1) / step + 1 : 0; };
  const int npair = count(pairs), nunit = count(units);
  const int nstream = nunit + npair;   // tiles: two per pair
  auto decode = [&](int s, int& kx0, int& outer, int& type, bool& tau) {
    const bool pr = s < 2 * npair;
    const int i = pr ? s / 2 : s - npair;
    tau = pr && !(s & 1);
    tile_of(tp, first + i * step, P, kx0, outer, type);
  };
  // field of a stream tile: tau_i2 (3 + i) or A_i (i) of pair i; singles 6, 7
  auto field_of = [](int type, bool tau) { return type < 3 ? (tau ? 3 + type : type) : 3 + type; };
  auto issue = [&](int s) {
    int kx0, outer, type;
    bool tau;
    decode(s, kx0, outer, type, tau);
    tma_issue_tile<Cfg>(buf(s % NS), &map, &bars[s % NS], 1, kx0, outer, field_of(type, tau), P, Cfg::TILE_BYTES);
  };
  if (threadIdx.x == 0)
    for (int s = 0; s < NS && s < nstream; ++s) issue(s);
  for (int s = 0; s < nstream; ++s) {
    const int b = s % NS;
    if (!mbar_wait_bounded(&bars[b], (s / NS) & 1, tp.err)) {
      if (threadIdx.x == 0)   // copies in flight into the other buffers
        for (int k = 1; k < NS && s + k < nstream; ++k)
          mbar_wait_bounded(&bars[(s + k) % NS], ((s + k) / NS) & 1, nullptr);
      return;
    }
    int kx0, outer, type;
    bool tau;
    decode(s, kx0, outer, type, tau);
    const int nvalid = min(P, g.nxh - kx0);
    C out[E::JL][E::RL];
    E::template run_smem<false>(out, buf(b), tw);
    C* __restrict__ fp =
        tp.base + (long long)field_of(type, tau) * tp.field + outer * tp.outer_stride + kx0;
    C* const held = buf(tau ? b : (s + NS - 1) % NS);   // tau_i2 transformed, at (p, n): n P + p
#pragma unroll
    for (int a = 0; a < E::JL; ++a)
#pragma unroll
      for (int r = 0; r < E::RL; ++r) {
        int p, n;
        if (!E::out_pos(a, r, p, n)) continue;
        C x = out[a][r];
        if (tau) {
          held[n * P + p] = x;
          if (type != 2) continue;
        } else if (type < 3) {
          x = csub(x, cmuli(cscale(held[n * P + p], (T)wavenum(n, g.ny))));
        }
        if (p < nvalid) fp[n * tp.axis_stride + p] = x;
      }
    // refill: a single's buffer, or both of a finished pair.  The barrier puts
    // every thread's reads of the held values before the copies.
    if (!tau) {
      __syncthreads();
      if (threadIdx.x == 0) {
        fence_proxy_async();
        if (type < 3 && s - 1 + NS < nstream) issue(s - 1 + NS);
        if (s + NS < nstream) issue(s + NS);
      }
    }
  }
}

// z-forward of B_i and tau_i3 (w_i = B_i - i kz tau_i3) + the spectral update,
// with symmetrize's kx = 0 copy (hermitian_column).  The B tiles are
// transformed in place; the three tau tiles stream through a fourth buffer
// into registers and are subtracted.  Tiles of 64-byte rows, so that three
// CTAs share an SM at 256-point FP32 pencils.  (Nine tiles streamed through a
// ring into register accumulators, one CTA per SM, took 466 us at 256^3.)
template <typename T, int LOGN> struct LesZCfg {
  using Cfg = TmaCfg<T, LOGN>;
  static constexpr int N = Cfg::N;
  static constexpr int P0 = Cfg::P * sizeof(C2<T>) >= 128 ? Cfg::P / 2 : Cfg::P;
  static constexpr int P = sizeof(C2<T>) * (size_t)N * P0 > 48 * 1024 ? P0 / 2 : P0;
  static constexpr int NT_RAW = P * N / 8;
  static constexpr int NT = NT_RAW > 512 ? 512 : (NT_RAW < 32 ? 32 : NT_RAW);
  using Engine = FFTEngine<T, LOGN, P, P, NT, true>;
  static constexpr size_t TILE = sizeof(C2<T>) * (size_t)N * P;
  static constexpr size_t SMEM = 4 * TILE + kSmemAlignPad;
  static constexpr int FIT = (int)(233472 / (SMEM + 1024));
  static constexpr int REGS = 65536 / (NT * 80);           // CTAs that leave 80 registers a thread
  static constexpr int MIN = FIT < REGS ? FIT : REGS;
  static constexpr int MINB = MIN > 8 ? 8 : (MIN < 1 ? 1 : MIN);
};

template <typename T, int LOGN, int MODE>
__global__ void __cluster_dims__(1, 2, 1) __launch_bounds__(LesZCfg<T, LOGN>::NT, LesZCfg<T, LOGN>::MINB)
les_zfwd_kernel(const __grid_constant__ CUtensorMap fmap, StageArgs<T> st, Geom g, const C2<T>* __restrict__ tw,
                int* err) {
  pdl_wait();
  using Z = LesZCfg<T, LOGN>;
  using Cfg = TmaCfg<T, LOGN>;
  using E = typename Z::Engine;
  using C = C2<T>;
  constexpr int P = Z::P, N = Z::N, NT = Z::NT;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  C* w[3];
  for (int c = 0; c < 3; ++c) w[c] = reinterpret_cast<C*>(smraw + c * Z::TILE);
  C* const tau = reinterpret_cast<C*>(smraw + 3 * Z::TILE);
  __shared__ __align__(8) uint64_t bars[4];
  __shared__ T s_coef;
  const int kx0 = blockIdx.x * P;
  const int iy = paired_row(blockIdx.y, g.ny);
  const int nvalid = min(P, g.nxh - kx0);
  const long long zstride = (long long)g.ny * g.nxp;
  const long long base = (long long)iy * g.nxp + kx0;
  const T ky = (T)wavenum(iy, g.ny);
  const bool paired = st.symmetrize && kx0 == 0;   // meets its partner: both CTAs stay until then
  if (!paired && launch_failed(err)) return;
  const int kyi = wavenum(iy, g.ny), fk_b = st.fkmax2.b;
  const bool fblock = st.forced && kx0 * kx0 + kyi * kyi < fk_b;
  if (threadIdx.x == 0) {
    for (int c = 0; c < 4; ++c) mbar_init(&bars[c], 1);
    fence_mbar_init();
    fence_proxy_async();
    tma_issue_tile<Cfg>(w[0], &fmap, &bars[0], 2, kx0, iy, 0, P, Z::TILE);
    tma_issue_tile<Cfg>(tau, &fmap, &bars[3], 2, kx0, iy, les_t3(0), P, Z::TILE);
    tma_issue_tile<Cfg>(w[1], &fmap, &bars[1], 2, kx0, iy, 1, P, Z::TILE);
    tma_issue_tile<Cfg>(w[2], &fmap, &bars[2], 2, kx0, iy, 2, P, Z::TILE);
  }
  // one warp finds the forcing coefficient
  if (fblock && threadIdx.x >= NT - 32) {
    const double kf = warp_sum(forcing_energy_lane(st.kf_partial, st.kf_tiles, st.kf_ptile, g.ny, fk_b));
    if (threadIdx.x == NT - 32) s_coef = (T)(st.eps / (2.0 * kf));
  }
  __syncthreads();
  bool ok = true;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    ok = mbar_wait_bounded(&bars[c], 0, err) && ok;
    if (!ok && !paired) return;
    C* const wc = reinterpret_cast<C*>(smraw + c * Z::TILE);
    E::template run_inplace<false>(wc, tw);
    ok = mbar_wait_bounded(&bars[3], c & 1, err) && ok;
    if (!ok && !paired) return;
    C o[E::JL][E::RL];
    E::template run_smem<false>(o, tau, tw);   // every read of the tile precedes its last barrier
    if (threadIdx.x == 0 && c < 2 && ok) {
      fence_proxy_async();
      tma_issue_tile<Cfg>(tau, &fmap, &bars[3], 2, kx0, iy, les_t3(c + 1), P, Z::TILE);
    }
#pragma unroll
    for (int a = 0; a < E::JL; ++a)
#pragma unroll
      for (int r = 0; r < E::RL; ++r) {
        int p, n;
        if (E::out_pos(a, r, p, n))
          wc[n * P + p] = csub(wc[n * P + p], cmuli(cscale(o[a][r], (T)wavenum(n, g.nz))));
      }
  }
  __syncthreads();
  if (paired) {
    cluster_arrive();   // tau is free for the partner's column
    hermitian_column<T, P, N, NT, true>(w, tau, st, g, iy, base, zstride, fblock, fblock ? s_coef : T(0), 0, fk_b);
    if (!ok) return;
  }
  zfwd_update<T, P, N, NT, 2, MODE>(w, st, g, kx0, iy, nvalid, base, zstride, fblock, fblock ? s_coef : T(0), 0, fk_b,
                                    paired, false);
}

}  // namespace sc
