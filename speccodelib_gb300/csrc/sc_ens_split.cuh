// 2D ensembles, one launch per pass: the form of a stage in which each pass
// has the tiles, registers and CTAs per SM that suit it.
//
// The cooperative stage kernel (sc_ens.cuh) runs its three phases with one
// register budget (16 warps per SM, that of the x phase) and loads, transforms
// and stores a tile in turn; with work fields larger than L2 it reached a third
// of the copy bandwidth.  Here the members of one size form a class whose
// fields lie at equal distances, so that a tensor map spans it, and a step of
// a class is one y-inverse, then per stage an x-pass and a y-pass that ends the
// stage and begins the next:
//
//   ens_yinv  (first stage)  s^ -> u, v, w along y, three transforms from one
//                            TMA-fed tile
//   ens_x     c2r of u, v, w, the products u w and v w, r2c
//   ens_yfwd  both products forward along y, N^, symmetrize2d, mask, the RK
//             stage; then the next stage's u, v, w from the new stage input
//             still in the tile, which never goes to memory
//
// 51 field passes per step instead of 60.  Classes are independent within a
// step and run on streams of their own (branches of the captured graph), so
// that one fills the tail of another.  Values do not depend on what is
// batched together.
#pragma once
#include "sc_ens.cuh"
#include "sc_tma_passes.cuh"
#include "sc_xgroup.cuh"

namespace sc {

template <typename T> struct EnsParam { T dt, alpha, nu8; };

// The members of one size: member m's field f (w, s, acc, u, v, w in physical
// space) at base + (6 m + f) field, rows of nxp.
template <typename T> struct EnsClass {
  int n, logn, nxh, nxp;
  long long field;
  C2<T>* base;
  const EnsParam<T>* par;
  T scale;            // 1/N^2
  const C2<T>* tw;    // twiddle tables (length L at offset L)
  int* err;
  int nsm;
  int m0, count;      // members of this launch
  int stage;          // 1 .. 4
};

template <typename T, int LOGN> struct EnsSplitCfg {
  static constexpr int N = 1 << LOGN;
  static constexpr int U = sizeof(T) / 4;
  // rows of 64 bytes or more: 32 KB tiles and two CTAs per SM up to N = 512,
  // 64 KB and one at 1024 (16 points per thread; its ens_yfwd 185 us for 16
  // members, 213 with 32-byte rows and two CTAs)
  static constexpr int P4 = LOGN <= 8 ? 16 : 8;
  static constexpr int P = sizeof(T) == 4 ? P4 : P4 / 2;
  static constexpr int MINB = LOGN <= 9 ? 2 : 1;
  static constexpr int NT_RAW = P * N / 8;
  static constexpr int NT = NT_RAW > 512 ? 512 : (NT_RAW < 32 ? 32 : NT_RAW);
  static constexpr int BOX = N < 256 ? N : 256;
  static constexpr int NBOX = N / BOX;
  using Engine = FFTEngine<T, LOGN, P, P, NT, true>;
  static constexpr size_t TILE = sizeof(C2<T>) * (size_t)N * P;
  static constexpr size_t SMEM_INV = 3 * TILE + kSmemAlignPad;
  static constexpr size_t SMEM_FWD = 2 * TILE + kSmemAlignPad;
};

// u^ = i ky w^/k^2 (f = 0), v^ = -i kx w^/k^2 (f = 1) at (kx, ky)
template <typename C, typename T> __device__ __forceinline__ C ens_vel(C x, int f, T kx, T ky) {
  const T k2 = kx * kx + ky * ky;
  const T ik2 = k2 > T(0) ? T(1) / k2 : T(0);
  return f == 0 ? cmuli(cscale(x, ky * ik2)) : cmulmi(cscale(x, kx * ik2));
}

// u, v, w of a stage input held in the tile `s` (kept until w is transformed
// in place), through `work`, to the fields q, q + field, q + 2 field
template <typename T, int LOGN>
__device__ __forceinline__ void ens_uvw(C2<T>* s, C2<T>* work, const C2<T>* __restrict__ tw, int kx0, int nvalid,
                                        C2<T>* q, long long field, int nxp) {
  using Cfg = EnsSplitCfg<T, LOGN>;
  using E = typename Cfg::Engine;
  using C = C2<T>;
  C out[E::JL][E::RL];
  auto store = [&](C* __restrict__ d) {
#pragma unroll
    for (int a = 0; a < E::JL; ++a)
#pragma unroll
      for (int r = 0; r < E::RL; ++r) {
        int p, n;
        if (E::out_pos(a, r, p, n) && p < nvalid) d[(long long)n * nxp + p] = out[a][r];
      }
  };
  E::template run_map<true>(out, s, work, tw,
                            [&](C x, int p, int n) { return ens_vel<C, T>(x, 0, (T)(kx0 + p), (T)wavenum(n, Cfg::N)); });
  store(q);
  E::template run_map<true>(out, s, work, tw,
                            [&](C x, int p, int n) { return ens_vel<C, T>(x, 1, (T)(kx0 + p), (T)wavenum(n, Cfg::N)); });
  store(q + field);
  E::template run_smem<true>(out, s, tw);
  store(q + 2 * field);
}

// First stage's operands from the state.  Persistent, two tiles in flight.
template <typename T, int LOGN>
__global__ void __launch_bounds__(EnsSplitCfg<T, LOGN>::NT, EnsSplitCfg<T, LOGN>::MINB)
ens_yinv_kernel(const __grid_constant__ CUtensorMap map, EnsClass<T> ec) {
  pdl_wait();
  using Cfg = EnsSplitCfg<T, LOGN>;
  using C = C2<T>;
  constexpr int P = Cfg::P;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  __shared__ __align__(8) uint64_t bars[2];
  if (launch_failed(ec.err)) return;
  auto buf = [&](int b) { return reinterpret_cast<C*>(smraw + (size_t)b * Cfg::TILE); };
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  __syncthreads();
  const int ntx = (ec.nxh + P - 1) / P, total = ntx * ec.count;
  auto issue = [&](int job, int b) {
    tma_issue_tile<Cfg>(buf(b), &map, &bars[b], 1, (job % ntx) * P, ec.m0 + job / ntx, 0, P, Cfg::TILE);
  };
  int job = blockIdx.x;
  const int step = gridDim.x;
  if (threadIdx.x == 0 && job < total) issue(job, 0);
  for (int it = 0; job < total; job += step, ++it) {
    const int b = it & 1;
    if (threadIdx.x == 0 && job + step < total) {
      fence_proxy_async();
      issue(job + step, b ^ 1);
    }
    if (!mbar_wait_bounded(&bars[b], (it >> 1) & 1, ec.err)) {
      if (threadIdx.x == 0 && job + step < total) mbar_wait_bounded(&bars[b ^ 1], ((it + 1) >> 1) & 1, nullptr);
      return;
    }
    const int kx0 = (job % ntx) * P;
    C* q = ec.base + (6LL * (ec.m0 + job / ntx) + 3) * ec.field + kx0;
    ens_uvw<T, LOGN>(buf(b), buf(2), ec.tw + Cfg::N, kx0, min(P, ec.nxh - kx0), q, ec.field, ec.nxp);
  }
}

// End of a stage (see the head of this file).  A block per kx tile and member, in
// one dimension: a class may have more members than the other two admit.
template <typename T, int LOGN>
__global__ void __launch_bounds__(EnsSplitCfg<T, LOGN>::NT, EnsSplitCfg<T, LOGN>::MINB)
ens_yfwd_kernel(const __grid_constant__ CUtensorMap map, EnsClass<T> ec) {
  pdl_wait();
  using Cfg = EnsSplitCfg<T, LOGN>;
  using E = typename Cfg::Engine;
  using C = C2<T>;
  constexpr int P = Cfg::P, N = Cfg::N, NT = Cfg::NT;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  C* const t0 = reinterpret_cast<C*>(smraw);
  C* const t1 = reinterpret_cast<C*>(smraw + Cfg::TILE);
  __shared__ __align__(8) uint64_t bars[2];
  const int ntx = (ec.nxh + P - 1) / P;
  const int kx0 = blockIdx.x % ntx * P, m = ec.m0 + blockIdx.x / ntx;
  const int nvalid = min(P, ec.nxh - kx0);
  const C* __restrict__ tw = ec.tw + N;
  if (launch_failed(ec.err)) return;
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
    fence_proxy_async();
    tma_issue_tile<Cfg>(t0, &map, &bars[0], 1, kx0, m, 3, P, Cfg::TILE);
    tma_issue_tile<Cfg>(t1, &map, &bars[1], 1, kx0, m, 4, P, Cfg::TILE);
  }
  __syncthreads();
  const EnsParam<T> par = ec.par[m];
  if (!mbar_wait_bounded(&bars[0], 0, ec.err)) {
    if (threadIdx.x == 0) mbar_wait_bounded(&bars[1], 0, nullptr);
    return;
  }
  E::template run_inplace<false>(t0, tw);
  if (!mbar_wait_bounded(&bars[1], 0, ec.err)) return;
  E::template run_inplace<false>(t1, tw);
  // N^ = -i (kx (u w)^ + ky (v w)^) into t0
  for (int e = threadIdx.x; e < P * N; e += NT) {
    const C a = cmulmi(cscale(t0[e], (T)(kx0 + e % P))), b = cmulmi(cscale(t1[e], (T)wavenum(e / P, N)));
    t0[e] = cadd(a, b);
  }
  __syncthreads();
  if (kx0 == 0) {
    // symmetrize2d's conjugate copies lie in this pencil
    for (int n = N / 2 + 1 + threadIdx.x; n < N; n += NT) t0[n * P] = cconj(t0[(N - n) * P]);
    __syncthreads();
  }
  const double kc = 2.0 * (N / 2) / 3.0;
  const int kc_b = k2_lt(kc * kc);
  const int stage = ec.stage;
  C* const fw = ec.base + 6LL * m * ec.field + kx0;
  C* const facc = fw + 2 * ec.field;
  constexpr int EB = 4;
  const T dt = par.dt, hdt = T(0.5) * par.dt;
  for (int e0 = threadIdx.x; e0 < P * N; e0 += NT * EB) {
    C v[EB], ac[EB];
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      const int e = e0 + i * NT;
      v[i] = ac[i] = czero<C>();
      if (e >= P * N || e % P >= nvalid) continue;
      const long long idx = (long long)(e / P) * ec.nxp + e % P;
      if (stage < 4) v[i] = fw[idx];
      if (stage > 1) ac[i] = facc[idx];
    }
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      const int e = e0 + i * NT;
      if (e >= P * N) continue;
      const int p = e % P, n = e / P, ix = kx0 + p;
      const int ky = wavenum(n, N);
      const int k2i = ix * ix + ky * ky;
      C w = t0[e];
      if (n == N / 2 || ix >= ec.nxh - 1 || (ix == 0 && n == 0) || k2i >= kc_b) w = czero<C>();
      const T k2 = (T)k2i, k4 = k2 * k2;   // exact: k2 < 2^24
      const T Ef = exp(-((par.alpha + par.nu8 * (k4 * k4)) * dt * T(0.5)));
      const T E2 = Ef * Ef;
      C sn = czero<C>(), an = czero<C>();
      switch (stage) {
        case 1:
          an = cscale(w, E2 * dt);
          sn = cscale(cadd(v[i], cscale(w, hdt)), Ef);
          break;
        case 2:
          an = cadd(ac[i], cscale(w, T(2) * Ef * dt));
          sn = cadd(cscale(v[i], Ef), cscale(w, hdt));
          break;
        case 3:   // stage 3 leaves E^2 v + (acc + 2 E dt w3)/6 in acc, so stage 4 reads no v
          an = cadd(cscale(v[i], E2), cscale(cadd(ac[i], cscale(w, T(2) * Ef * dt)), T(1) / T(6)));
          sn = cadd(cscale(v[i], E2), cscale(w, Ef * dt));
          break;
        default:
          an = cadd(ac[i], cscale(cscale(w, dt), T(1) / T(6)));
          break;
      }
      if (p < nvalid) {
        const long long idx = (long long)n * ec.nxp + p;
        if (stage < 4) facc[idx] = an;
        else fw[idx] = an;
      }
      t0[e] = sn;
    }
  }
  if (stage == 4) return;
  __syncthreads();
  ens_uvw<T, LOGN>(t0, t1, tw, kx0, nvalid, fw + 3 * ec.field, ec.field, ec.nxp);
}

// Rows of a class: u w and v w over u and v.  Lane groups up to M = 256.
template <typename T, int LOGM> struct EnsXCfg {
  using GF = GroupFFT<T, LOGM>;
  static constexpr int WARPS = 4, NT = 32 * WARPS;
  static constexpr size_t SMEM = sizeof(C2<T>) * (size_t)GF::RW * GF::BUF * WARPS;
};
template <typename T, int LOGM>
__global__ void __launch_bounds__(EnsXCfg<T, LOGM>::NT, sizeof(T) == 4 ? 4 : 2) ens_xgroup_kernel(EnsClass<T> ec) {
  pdl_wait();
  using C = C2<T>;
  using Cfg = EnsXCfg<T, LOGM>;
  using GF = GroupFFT<T, LOGM>;
  constexpr int E = GF::E, M = GF::M;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int warp = threadIdx.x >> 5;
  Geom g{};
  auto R = xg_row<T, LOGM>(reinterpret_cast<C*>(smraw) + warp * GF::RW * GF::BUF, 0, 0, g, ec.tw + M, ec.tw + 2 * M, 1);
  const long long rows = (long long)ec.count * ec.n;
  long long row = ((long long)blockIdx.x * Cfg::WARPS + warp) * GF::RW + R.lane / GF::L;
  R.live = row < rows;
  if (!R.live) row = rows - 1;
  R.off = 6 * (ec.m0 + row / ec.n) * ec.field + (row % ec.n) * ec.nxp;
  C b[E];
  R.load_phys(ec.base + 5 * ec.field, b);
#pragma unroll 1
  for (int f = 3; f < 5; ++f) {
    C x[E];
    R.load_phys(ec.base + f * ec.field, x);
#pragma unroll
    for (int i = 0; i < E; ++i) x[i] = mk<C>(x[i].x * b[i].x, x[i].y * b[i].y);
    R.store_r2c(x, ec.base + f * ec.field, ec.scale);
  }
}
// M = 512: a warp per row (ens_xrow)
template <typename T> __global__ void __launch_bounds__(256, 2) ens_xwarp_kernel(EnsClass<T> ec) {
  pdl_wait();
  using C = C2<T>;
  using WF = WarpFFT<T, 9>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int warp = threadIdx.x >> 5;
  const long long rows = (long long)ec.count * ec.n, row = (long long)blockIdx.x * 8 + warp;
  if (row >= rows) return;
  EnsMember<T> mb{};
  mb.nxp = ec.nxp;
  mb.field = ec.field;
  mb.scale = ec.scale;
  mb.work = ec.base + (6 * (ec.m0 + row / ec.n) + 3) * ec.field;
  ens_xrow<T, 9>(mb, (int)(row % ec.n), reinterpret_cast<C*>(smraw) + warp * (WF::SMEM + WF::M), ec.tw);
}

// Host side: the kernels of one class on `s`.
template <typename T, int LOGN> cudaError_t ens_split_stage_n(const CUtensorMap& map, const EnsClass<T>& ec, cudaStream_t s) {
  using Cfg = EnsSplitCfg<T, LOGN>;
  using C = C2<T>;
  constexpr size_t sx9 = sizeof(C) * 8 * (WarpFFT<T, 9>::SMEM + WarpFFT<T, 9>::M);
  static cudaError_t attr = [] {
    cudaError_t e = cudaFuncSetAttribute(ens_yinv_kernel<T, LOGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM_INV);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ens_yfwd_kernel<T, LOGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM_FWD);
    if constexpr (LOGN == 10) {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(ens_xwarp_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx9);
    } else {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(ens_xgroup_kernel<T, LOGN - 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)EnsXCfg<T, LOGN - 1>::SMEM);
    }
    return e;
  }();
  if (attr != cudaSuccess) return attr;
  const int ntx = (ec.nxh + Cfg::P - 1) / Cfg::P;
  if (ec.stage == 1) {
    const int total = ntx * ec.count, most = 2 * ec.nsm;
    const cudaError_t e = launch_pdl(ens_yinv_kernel<T, LOGN>, dim3(total < most ? total : most), dim3(Cfg::NT), Cfg::SMEM_INV, s, map, ec);
    if (e != cudaSuccess) return e;
  }
  const long long rows = (long long)ec.count * ec.n;
  if constexpr (LOGN == 10) {
    const cudaError_t e = launch_pdl(ens_xwarp_kernel<T>, dim3((unsigned)((rows + 7) / 8)), dim3(256), sx9, s, ec);
    if (e != cudaSuccess) return e;
  } else {
    using X = EnsXCfg<T, LOGN - 1>;
    const int per = X::WARPS * GroupFFT<T, LOGN - 1>::RW;
    const cudaError_t e =
        launch_pdl(ens_xgroup_kernel<T, LOGN - 1>, dim3((unsigned)((rows + per - 1) / per)), dim3(X::NT), X::SMEM, s, ec);
    if (e != cudaSuccess) return e;
  }
  return launch_pdl(ens_yfwd_kernel<T, LOGN>, dim3(ntx * ec.count), dim3(Cfg::NT), Cfg::SMEM_FWD, s, map, ec);
}

// sc_ens_split_*.cu
template <typename T> cudaError_t ens_split_stage(const CUtensorMap& map, const EnsClass<T>& ec, cudaStream_t s);
template <typename T> int ens_split_tile(int logn);   // tile width of the maps

}  // namespace sc
