// TMA-fed strided-axis passes (y and z).
//
// A pencil tile -- P consecutive kx columns by the N points of the pencil --
// is one box of a 4D tensor map (x = kx, y, z, field), so one thread issues
// the whole tile as one or two cp.async.bulk.tensor loads that land in shared
// memory already in the FFT engine's layout sm[n*P + p].  Loads complete on
// an mbarrier; the CTA transforms one buffer while the next tile streams into
// the other, so HBM stays busy while the FFT stages run.
//
//   pencil_tma_kernel : plain y / z pass over nf fields, persistent over
//                       (tile, outer, field) jobs, double-buffered.
//   zinv_tma_kernel   : z-inverse pass of the right-hand side: v^ tile (3
//                       fields) by TMA, the 6 outputs v^, i k x v^ generated
//                       from shared memory, transformed, stored.
//   zfwd_tma_kernel   : z-forward pass of the Lamb vector (3 fields by TMA,
//                       transformed in place) + the spectral update.
#pragma once
#include "sc_passes.cuh"
#include "sc_tma.cuh"

namespace sc {

template <typename T, int LOGN> struct TmaCfg {
  static constexpr int N = 1 << LOGN;
  static constexpr int U = sizeof(T) / 4;   // 8-byte units per complex element
  // tile width: 64-byte rows for long pencils (two buffers fit twice per SM)
  static constexpr int P = sizeof(T) == 4 ? (LOGN <= 8 ? 16 : 8) : (LOGN <= 8 ? 8 : 4);
  static constexpr int NT_RAW = P * N / 8;
  static constexpr int NT = NT_RAW > 512 ? 512 : (NT_RAW < 32 ? 32 : NT_RAW);
  static constexpr int BOX = N < 256 ? N : 256;   // TMA box extent limit
  static constexpr int NBOX = N / BOX;
  using Engine = FFTEngine<T, LOGN, P, P, NT, true>;
  static constexpr size_t TILE_BYTES = sizeof(C2<T>) * N * P;
  // pipeline depth of pencil_tma_kernel: tiles in flight per CTA
  static constexpr int STAGES = TILE_BYTES <= 8192 ? 3 : (TILE_BYTES <= 16384 ? 4 : 3);
  // its CTAs per SM: eight for tiles of 8 KB and less (128 threads or fewer; the
  // 512 x 64 x 256 FP32 step 7.73 -> 7.02 ms per five), else two (four CTAs of
  // 16 KB tiles took 34 us against 29 for nine fields at 128^3)
  static constexpr int PB = TILE_BYTES <= 8192 ? 8 : 2;
  // zinv uses a narrower tile: 3 inputs + 1 work buffer
  static constexpr int PZ = P >= 8 ? P / 2 : P;
  static constexpr int NTZ_RAW = PZ * N / 8;
  static constexpr int NTZ = NTZ_RAW > 512 ? 512 : (NTZ_RAW < 32 ? 32 : NTZ_RAW);
  // work buffer padded one slot per 8 points: conflict-free first-stage scatter
  using EngineZ = FFTEngine<T, LOGN, PZ, PZ, NTZ, true, 3>;
  static constexpr size_t TILEZ_BYTES = sizeof(C2<T>) * N * PZ;
  static constexpr size_t WORKZ_BYTES = sizeof(C2<T>) * EngineZ::SMEM_ELEMS;
};

// L2 prefetch of the update's operands for a z tile (thread 0; `fmap` is the
// whole field slab with tiles P wide and BOX long in z).
template <typename Cfg, typename T>
__device__ __forceinline__ void prefetch_update_tile(const CUtensorMap* fmap, const StageArgs<T>& st, int kx0,
                                                     int iy) {
#pragma unroll
  for (int i = 0; i < 6; ++i)
    if (i < st.pf_n)
      for (int h = 0; h < Cfg::NBOX; ++h) tma_prefetch_4d(fmap, kx0 * Cfg::U, iy, h * Cfg::BOX, st.pf_slot[i]);
}

// The z-forward kernels run as clusters of two CTAs that hold the pencils ky
// and -ky of one kx tile (ky = 0 is paired with ky = -ny/2): block row b works
// on this ky index.
__device__ __forceinline__ int paired_row(int b, int ny) {
  const int m = b >> 1;
  return !(b & 1) ? m : (m == 0 ? ny / 2 : ny - m);
}
// Hermitian copy of symmetrize.f90:52-62 on the kx = 0 column (p = 0) of the
// NF tiles w: the targets (kz index over nz/2, and ky index over ny/2 at kz = 0)
// take the conjugates of w(-ky, -kz) from the partner CTA (from the own tiles at
// ky = 0), pushed through distributed shared memory.  src(c, n, w) gives the
// column's value from the tile's (and may change the tile).  This replaces a side
// buffer, a fix-up launch after every z-forward and, in the fused RK stages, a
// one-tile z-inverse launch: three dependent launches per stage become one (256^3
// FP32 step 3.08 -> 2.97 ms, 64^3 178 -> 145 us, 512^3 24.0 -> 23.5 ms).
// Where the values go: with COL into `col` (NF N/2 values of shared memory), from
// which the partner fills its tiles, and the caller has arrived (cluster_arrive)
// once its col is free; without COL straight into the partner's targets, which are
// no sources, and the caller arrives after its barrier on the tiles.
// Every thread of both CTAs calls it, after a barrier on the tiles; it ends with
// a barrier.
template <int NF, int P, int N, int NT, bool COL, typename C, class F>
__device__ __forceinline__ void column_copy(C* const w[], C* col, int iy, int ny, F&& src) {
  cluster_wait();
  const uint32_t to = iy == 0 ? cluster_rank() : (cluster_rank() ^ 1u);
  for (int n = threadIdx.x; n < N / 2; n += NT) {
    if (n == 0 && iy > ny / 2) continue;   // a target
#pragma unroll
    for (int c = 0; c < NF; ++c) {
      const C v = cconj(src(c, n, w[c][n * P]));
      if (iy != ny / 2 && (n > 0 || iy > 0)) cluster_store(COL ? &col[c * (N / 2) + n] : &w[c][(N - n) % N * P], v, to);
    }
  }
  cluster_sync();
  if (COL || iy == ny / 2) {
    for (int n = threadIdx.x; n < N / 2; n += NT) {
      if (n == 0 && iy <= ny / 2) continue;
#pragma unroll
      for (int c = 0; c < NF; ++c) w[c][(N - n) % N * P] = iy == ny / 2 ? czero<C>() : col[c * (N / 2) + n];
    }
    __syncthreads();
  }
}

// The same after the z-forward transform of the right-hand side and before the
// spectral update, which treats the column like any other: forcing is added to
// the column first.
template <typename T, int P, int N, int NT, bool COL>
__device__ __forceinline__ void hermitian_column(C2<T>* const w[3], C2<T>* col, const StageArgs<T>& st, const Geom& g,
                                                 int iy, long long base, long long zstride, bool fblock, T coef,
                                                 int flo_b, int fk_b) {
  using C = C2<T>;
  const int kyi = wavenum(iy, g.ny);
  column_copy<3, P, N, NT, COL>(w, col, iy, g.ny, [&](int c, int n, C& v) {
    const int k2 = kyi * kyi + n * n;
    if (fblock && k2 < fk_b && k2 >= flo_b) v = cadd(v, cscale(st.sin[c][base + n * zstride], coef));
    return v;
  });
}

// Where a pencil lies: element (p, n) of tile (kx0, outer) of field f is
// base + f*field + outer*outer_stride + n*axis_stride + kx0 + p.
template <typename T> struct TmaPass {
  C2<T>* base;            // field 0 of the group
  long long field;        // elements between fields
  long long axis_stride;
  long long outer_stride;
  int axis;               // 1 = y, 2 = z
  int nouter;             // number of outer slabs (nz for y, ny for z)
  int ntx;                // kx tiles
  int nf;                 // fields
  int* err;               // device error word
};

// Job `job` of a pass (kx tile fastest, field slowest), in 32-bit arithmetic: the
// jobs of every grid size stay below 2^31, and 64-bit divisions here made a 64^3
// FP32 step 104 us instead of 102, 128^3 396 instead of 380, 256^3 2.91 ms instead of 2.85.
template <typename T>
__device__ __forceinline__ void tile_of(const TmaPass<T>& tp, int job, int P, int& kx0, int& outer, int& f) {
  const int per = tp.ntx * tp.nouter;
  f = job / per;
  const int t = job - f * per;
  outer = t / tp.ntx;
  kx0 = (t - outer * tp.ntx) * P;
}

// Issue the loads of one field tile: box (P, BOX, 1) along y or (P, 1, BOX) along z.
template <typename Cfg>
__device__ __forceinline__ void tma_issue_tile(void* dst, const CUtensorMap* map, uint64_t* bar, int axis,
                                               int kx0, int outer, int f, int P, size_t bytes) {
  mbar_arrive_expect_tx(bar, (uint32_t)bytes);
  for (int h = 0; h < Cfg::NBOX; ++h) {
    char* d = static_cast<char*>(dst) + (size_t)h * Cfg::BOX * P * sizeof(C2<float>) * Cfg::U;
    if (axis == 1) tma_load_4d(d, map, bar, kx0 * Cfg::U, h * Cfg::BOX, outer, f);
    else tma_load_4d(d, map, bar, kx0 * Cfg::U, outer, h * Cfg::BOX, f);
  }
}

template <typename T, int LOGN, bool INV>
__global__ void __launch_bounds__(TmaCfg<T, LOGN>::NT, TmaCfg<T, LOGN>::PB)
pencil_tma_kernel(const __grid_constant__ CUtensorMap map, TmaPass<T> tp, Geom g, const C2<T>* __restrict__ tw) {
  pdl_wait();
  using Cfg = TmaCfg<T, LOGN>;
  // stage-0 writes XOR-rotated (conflict-free 64-byte rows) in the forward
  // pass only: measured 4% faster there, 3% slower in the inverse pass
  using E = FFTEngine<T, LOGN, Cfg::P, Cfg::P, Cfg::NT, true, 0, !INV>;
  using C = C2<T>;
  constexpr int P = Cfg::P;
  constexpr int NS = Cfg::STAGES;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  __shared__ __align__(8) uint64_t bars[NS];
  const int total = tp.ntx * tp.nouter * tp.nf;
  const bool failed = launch_failed(tp.err);
  if (threadIdx.x == 0) {
    for (int b = 0; b < NS; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  __syncthreads();
  auto buf = [&](int b) { return reinterpret_cast<C*>(smraw + (size_t)b * Cfg::TILE_BYTES); };
  // field slowest: the CTAs in flight work on neighbouring tiles of one
  // field (field fastest, six fields at the same offset, measured 12%
  // slower for the six-field inverse y-pass)
  auto decode = [&](int job, int& kx0, int& outer, int& f) { tile_of(tp, job, P, kx0, outer, f); };
  auto issue = [&](int job, int b) {
    int kx0, outer, f;
    decode(job, kx0, outer, f);
    tma_issue_tile<Cfg>(buf(b), &map, &bars[b], tp.axis, kx0, outer, f, P, Cfg::TILE_BYTES);
  };
  if (failed) return;
  // prologue: the first NS-1 jobs of this CTA in flight
  if (threadIdx.x == 0) {
    for (int k = 0; k < NS - 1; ++k) {
      const int jk = blockIdx.x + k * gridDim.x;
      if (jk < total) issue(jk, k);
    }
  }
  int job = blockIdx.x;
  for (int it = 0; job < total; job += gridDim.x, ++it) {
    const int b = it % NS;
    const int ahead = job + (NS - 1) * gridDim.x;
    if (threadIdx.x == 0 && ahead < total) {
      fence_proxy_async();
      issue(ahead, (it + NS - 1) % NS);
    }
    if (!mbar_wait_bounded(&bars[b], (it / NS) & 1, tp.err)) return;
    // the tile's destination before the transform (its address arithmetic
    // then overlaps the FFT; measured 1.41 -> 1.27 ms for the six-field
    // inverse pass at 512^3)
    int kx0, outer, f;
    decode(job, kx0, outer, f);
    const int nvalid = min(P, g.nxh - kx0);
    C* __restrict__ fp = tp.base + f * tp.field + outer * tp.outer_stride + kx0;
    C out[E::JL][E::RL];
    E::template run_smem<INV>(out, buf(b), tw);
#pragma unroll
    for (int a = 0; a < E::JL; ++a)
#pragma unroll
      for (int r = 0; r < E::RL; ++r) {
        int p, n;
        if (E::out_pos(a, r, p, n) && p < nvalid) fp[n * tp.axis_stride + p] = out[a][r];
      }
  }
}

// z-inverse pass of one right-hand side (DNS): outputs v (3) and w = i k x v (3).
template <typename T, int LOGN>
__global__ void __launch_bounds__(TmaCfg<T, LOGN>::NTZ, 3)
zinv_tma_kernel(const __grid_constant__ CUtensorMap vmap, ZvArgs<T> za, FieldList<T> out, Geom g,
                const C2<T>* __restrict__ tw, int* err) {
  using Cfg = TmaCfg<T, LOGN>;
  using E = typename Cfg::EngineZ;
  using C = C2<T>;
  constexpr int P = Cfg::PZ;
  constexpr int N = Cfg::N;
  constexpr int NT = Cfg::NTZ;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  C* in[3];
  for (int c = 0; c < 3; ++c) in[c] = reinterpret_cast<C*>(smraw + c * Cfg::TILEZ_BYTES);
  C* work = reinterpret_cast<C*>(smraw + 3 * Cfg::TILEZ_BYTES);
  __shared__ __align__(8) uint64_t bar;
  __shared__ double red[NT / 32 + 1];
  const int kx0 = blockIdx.x * P;
  const int iy = blockIdx.y;
  const int nvalid = min(P, g.nxh - kx0);
  const long long zstride = (long long)g.ny * g.nxp;
  const long long base = (long long)iy * g.nxp + kx0;
  const T ky = (T)wavenum(iy, g.ny);
  if (launch_failed(err)) return;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    fence_proxy_async();
    mbar_arrive_expect_tx(&bar, (uint32_t)(3 * Cfg::TILEZ_BYTES));
    for (int c = 0; c < 3; ++c)
      for (int h = 0; h < Cfg::NBOX; ++h)
        tma_load_4d(reinterpret_cast<char*>(in[c]) + (size_t)h * Cfg::BOX * P * sizeof(C), &vmap, &bar,
                    kx0 * Cfg::U, iy, h * Cfg::BOX, c);
  }
  __syncthreads();
  if (!mbar_wait_bounded(&bar, 0, err)) return;
  // forcing band energy of the stage input (force.f90:16-22), FP64
  const int kyi = wavenum(iy, g.ny), fk_b = za.fs.fkmax2.b;
  const bool fsum = za.fs.enabled && kx0 * kx0 + kyi * kyi < fk_b;
  if (fsum) {
    double q = 0.0;
    for (int e = threadIdx.x; e < P * N; e += NT) {
      const int p = e % P, n = e / P;
      const int kx = kx0 + p, kz = wavenum(n, g.nz);
      if (p < nvalid && kx * kx + kyi * kyi + kz * kz < fk_b) {
        double s = 0.0;
        for (int c = 0; c < 3; ++c) s += (double)in[c][e].x * in[c][e].x + (double)in[c][e].y * in[c][e].y;
        q += (kx0 + p == 0) ? 0.5 * s : s;
      }
    }
    double sum = block_sum<NT>(q, red);
    if (threadIdx.x == 0) za.fs.partial[(long long)blockIdx.x * g.ny + iy] = sum;
  }
  for (int f = 0; f < 6; ++f) {
    C x[E::J1][E::R1], o[E::JL][E::RL];
#pragma unroll
    for (int a = 0; a < E::J1; ++a)
#pragma unroll
      for (int r = 0; r < E::R1; ++r) {
        int p, n;
        E::in_pos(a, r, p, n);
        const int e = n * P + p;
        const T kx = (T)(kx0 + p), kz = (T)wavenum(n, g.nz);
        x[a][r] = zv_gen<ZV_DNS>(f, in[0][e], in[1][e], in[2][e], kx, ky, kz, true);
      }
    E::template run<true>(x, o, work, tw);
    C* __restrict__ fp = out.f[f] + base;
#pragma unroll
    for (int a = 0; a < E::JL; ++a)
#pragma unroll
      for (int r = 0; r < E::RL; ++r) {
        int p, n;
        if (E::out_pos(a, r, p, n) && p < nvalid) fp[n * zstride + p] = o[a][r];
      }
  }
}

// z-forward pass of NIN fields (LES: the Lamb vector and tau_ij, NIN = 9)
// + the spectral update: the fields' tiles stream through a three-deep TMA
// ring, each transformed from shared memory into registers and accumulated
// into w (zfwd_accumulate); a buffer is refilled once its transform has read
// it.  fmap: the NIN fields, tiles P wide along z.
template <typename T, int LOGN, int NIN>
__global__ void __launch_bounds__(TmaCfg<T, LOGN>::NT, 1)
zfwd_fields_tma_kernel(const __grid_constant__ CUtensorMap fmap, StageArgs<T> st, Geom g,
                       const C2<T>* __restrict__ tw, int* err) {
  using Cfg = TmaCfg<T, LOGN>;
  using E = typename Cfg::Engine;
  using C = C2<T>;
  constexpr int P = Cfg::P;
  constexpr int NB = 3;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  __shared__ __align__(8) uint64_t bars[NB];
  __shared__ double s_coef;
  auto buf = [&](int b) { return reinterpret_cast<C*>(smraw + (size_t)b * Cfg::TILE_BYTES); };
  const int kx0 = blockIdx.x * P;
  const int iy = blockIdx.y;
  const int nvalid = min(P, g.nxh - kx0);
  const long long zstride = (long long)g.ny * g.nxp;
  const long long base = (long long)iy * g.nxp + kx0;
  const T ky = (T)wavenum(iy, g.ny);
  if (launch_failed(err)) return;
  if (threadIdx.x == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&bars[b], 1);
    fence_mbar_init();
    fence_proxy_async();
    for (int f = 0; f < NB && f < NIN; ++f)
      tma_issue_tile<Cfg>(buf(f), &fmap, &bars[f], 2, kx0, iy, f, P, Cfg::TILE_BYTES);
  }
  __syncthreads();
  C w[E::JL][E::RL][3];
  for (int f = 0; f < NIN; ++f) {
    const int b = f % NB;
    if (!mbar_wait_bounded(&bars[b], (f / NB) & 1, err)) return;
    C o[E::JL][E::RL];
    E::template run_smem<false>(o, buf(b), tw);   // every read of buf(b) precedes its last barrier
    if (threadIdx.x == 0 && f + NB < NIN) {
      fence_proxy_async();
      tma_issue_tile<Cfg>(buf(b), &fmap, &bars[b], 2, kx0, iy, f + NB, P, Cfg::TILE_BYTES);
    }
    zfwd_accumulate<E, T>(w, o, f, kx0, ky, g);
  }
  zfwd_finish<E, T>(w, st, g, kx0, iy, nvalid, base, zstride, s_coef);
}

// State, accumulator and integrating factor ez of EB points n0 + i RS of a z
// pencil (those below N); p0 is the pencil's first point.  The factor comes with
// the state: loaded at its use it waited for the stores of the point before.
template <typename T, int EB> struct UpdateBatch {
  C2<T> v[EB][3], a[EB][3];
  T ez[EB];
  template <int MODE, int N, int RS>
  __device__ __forceinline__ void load(const StageArgs<T>& st, int n0, long long p0, long long zstride, bool factor) {
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      const int iz = n0 + i * RS;
      if (iz >= N) continue;
      load_state<T, MODE>(st, p0 + iz * zstride, v[i], a[i]);
      ez[i] = factor ? st.ez[iz] : T(1);
    }
  }
};

// The z-forward's spectral update of tile (kx0, iy) from the transformed
// right-hand side in the tiles w (element (p, n) at n P + p; forcing and
// symmetrize's copy of the kx = 0 column already in them when `paired`), in
// batches of EB points per thread: all state loads of a batch are issued
// before any of them is used (the next batch's before this one is worked on, as
// zfwd_zinv does, gained nothing here).  fblock: the tile meets the forcing band, whose
// coefficient is coef.  tstore (RK stage 4): the new state goes back into the
// tiles.
template <typename T, int P, int N, int NT, int EB, int MODE>
__device__ __forceinline__ void zfwd_update(C2<T>* const w[3], const StageArgs<T>& st, const Geom& g, int kx0, int iy,
                                            int nvalid, long long base, long long zstride, bool fblock, T coef,
                                            int flo_b, int fk_b, bool paired, bool tstore) {
  using C = C2<T>;
  static_assert(NT % P == 0, "a thread keeps its kx");
  constexpr int RS = NT / P;
  const int kyi = wavenum(iy, g.ny), kc_b = st.kcut2.b;
  const int p = threadIdx.x % P, ix = kx0 + p;
  if (p >= nvalid) return;
  const bool factor = mode_reads_factor(MODE >= 0 ? MODE : st.mode);
  const T exy = factor ? st.ex[ix] * st.ey[iy] : T(1);
#pragma unroll 1
  for (int n0 = threadIdx.x / P; n0 < N; n0 += RS * EB) {
    UpdateBatch<T, EB> cur;
    cur.template load<MODE, N, RS>(st, n0, base + p, zstride, factor);
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      const int iz = n0 + i * RS;
      if (iz >= N) continue;
      const long long idx = base + iz * zstride + p;
      C wp[3] = {w[0][iz * P + p], w[1][iz * P + p], w[2][iz * P + p]};
      if (fblock && !(paired && ix == 0)) {
        const int kz = wavenum(iz, g.nz);
        const int k2 = ix * ix + kyi * kyi + kz * kz;
        if (k2 < fk_b && k2 >= flo_b) {
          const T ac = coef;
#pragma unroll
          for (int c = 0; c < 3; ++c) wp[c] = cadd(wp[c], cscale(st.sin[c][idx], ac));
        }
      }
      if (st.symmetrize) {
        if (iy == g.ny / 2 || iz == g.nz / 2 || ix == g.nxh - 1 || (ix == 0 && iy == 0 && iz == 0))
          wp[0] = wp[1] = wp[2] = czero<C>();
      }
      if (tstore) {
        C vn[3];
        finish_point_pre<T, MODE>(st, g, idx, ix, iy, iz, kc_b, wp, cur.v[i], cur.a[i], vn, exy * cur.ez[i]);
#pragma unroll
        for (int c = 0; c < 3; ++c) w[c][iz * P + p] = vn[c];
      } else {
        finish_point_pre<T, MODE>(st, g, idx, ix, iy, iz, kc_b, wp, cur.v[i], cur.a[i], nullptr, exy * cur.ez[i]);
      }
    }
  }
}

// z-forward pass of the Lamb vector + the spectral update (DNS).  MODE: the
// update mode as a compile-time constant (-1: st.mode at run time).  With
// MODE == SM_RK4 and vstore, the new state goes back into the tiles and
// leaves by bulk tensor stores through vmap (st.vout, tiles as lmap).
// Short pencils: a z kernel at 64^3 is one CTA or two per SM and its time a
// chain of latencies, so three groups of threads transform the three tiles at
// once instead of one group in turn.  FP32 pencils to 128 points and FP64 to 64.
// A group's threads take one radix-8 job each to 64 points, two at 128.  Step
// times, groups against in turn: FP32 64^3 137 -> 112 us, 128^3 430 -> 396 us;
// FP64 32^3 417 -> 267 us, 64^3 933 -> 862 us, but 128^3 5.66 -> 5.79 ms (bound by
// FP64 issue, and fewer CTAs per SM).  Two jobs per thread at 32 points: 68 -> 74
// us; one at 128: 396 -> 445 us.
template <typename T, int LOGN> struct ZgCfg {
  using Cfg = TmaCfg<T, LOGN>;
  static constexpr bool ON = LOGN <= (sizeof(T) == 4 ? 7 : 6);
  static constexpr int NTG_RAW = Cfg::P * Cfg::N / (LOGN <= 6 ? 8 : 16);
  static constexpr int NTG = NTG_RAW < 32 ? 32 : NTG_RAW;
  static constexpr int NT = 3 * NTG;
  using Engine = FFTEngine<T, LOGN, Cfg::P, Cfg::P, NTG, true, 0, true, 8, true>;
};

// Thread count of zfwd_tma_kernel: for 512- and 256-point pencils 16 points
// per thread, which gives its in-place transforms the two-pass form
// (SC_ZFWD_NT8: 8 points per thread, the radix-8 stages).
template <typename T, int LOGN> struct ZfCfg {
  using Cfg = TmaCfg<T, LOGN>;
#ifdef SC_ZFWD_NT8
  static constexpr int NT = Cfg::NT;
#else
  static constexpr int NT = (LOGN == 9 || LOGN == 8) ? Cfg::P * Cfg::N / 16 : Cfg::NT;
#endif
  using Engine = FFTEngine<T, LOGN, Cfg::P, Cfg::P, NT, true>;
  using G = ZgCfg<T, LOGN>;
  static constexpr bool GROUPED = G::ON;
  static constexpr int NTF = GROUPED ? G::NT : NT;   // threads of zfwd_tma_kernel
};

template <typename T, int LOGN, int MODE>
__global__ void __cluster_dims__(1, 2, 1) __launch_bounds__(ZfCfg<T, LOGN>::NTF, 2)
zfwd_tma_kernel(const __grid_constant__ CUtensorMap lmap, const __grid_constant__ CUtensorMap vmap, int vstore,
                StageArgs<T> st, Geom g, const C2<T>* __restrict__ tw, int* err) {
  pdl_wait();
  using Cfg = TmaCfg<T, LOGN>;
  using E = typename ZfCfg<T, LOGN>::Engine;
  using C = C2<T>;
  constexpr int P = Cfg::P;
  constexpr int N = Cfg::N;
  constexpr int NT = ZfCfg<T, LOGN>::NTF;
  using ZG = ZgCfg<T, LOGN>;
  constexpr bool GROUPED = ZfCfg<T, LOGN>::GROUPED;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  C* w[3];
  for (int c = 0; c < 3; ++c) w[c] = reinterpret_cast<C*>(smraw + c * Cfg::TILE_BYTES);
  __shared__ __align__(8) uint64_t bars[3];
  __shared__ T s_coef;
  const int kx0 = blockIdx.x * P;
  const int iy = paired_row(blockIdx.y, g.ny);
  const int nvalid = min(P, g.nxh - kx0);
  const long long zstride = (long long)g.ny * g.nxp;
  const long long base = (long long)iy * g.nxp + kx0;
  const T ky = (T)wavenum(iy, g.ny);
  // the kx = 0 tiles meet their partner: both CTAs stay until then
  const bool paired = st.symmetrize && kx0 == 0;
  // The exchanged column: a buffer of its own on short pencils (the pair then
  // waits once), else straight into the partner's tiles, which leaves the L1 to
  // the update's loads (6 KB more per CTA of the 512-point tiles: 512^3 FP32
  // stage 4 1.09 -> 1.24 ms, variable-step pass 2.14 -> 2.29 ms).
  constexpr bool COL = GROUPED;
  __shared__ C s_col[COL ? 3 * N / 2 : 1];
  if (paired && COL) cluster_arrive();
  const bool failed = !paired && launch_failed(err);
  if (!GROUPED && failed) return;
  if (threadIdx.x == 0) {
    for (int c = 0; c < 3; ++c) mbar_init(&bars[c], 1);
    fence_mbar_init();
    fence_proxy_async();
    for (int c = 0; c < 3; ++c) {
      mbar_arrive_expect_tx(&bars[c], (uint32_t)Cfg::TILE_BYTES);
      for (int h = 0; h < Cfg::NBOX; ++h)
        tma_load_4d(reinterpret_cast<char*>(w[c]) + (size_t)h * Cfg::BOX * P * sizeof(C), &lmap, &bars[c],
                    kx0 * Cfg::U, iy, h * Cfg::BOX, c);
    }
  }
  const int kyi = wavenum(iy, g.ny), fk_b = st.fkmax2.b;
  const bool fblock = st.forced && kx0 * kx0 + kyi * kyi < fk_b;
  // lower edge of the forcing band (0 for force.f90's k2 < fkmax^2)
  const int flo_b = st.fband_lo2.b;
  if (fblock && threadIdx.x >= NT - 32) {   // one warp finds the forcing coefficient
    double coef = 0.0;
    if (st.fcoef) coef = *st.fcoef;
    else coef = st.eps / (2.0 * warp_sum(forcing_energy_lane(st.kf_partial, st.kf_tiles, st.kf_ptile, g.ny, fk_b)));
    if (threadIdx.x == NT - 32) s_coef = (T)coef;
  }
  __syncthreads();
  bool ok = !failed;
  if constexpr (GROUPED) {
    const int grp = threadIdx.x / ZG::NTG;
    ok = mbar_wait_bounded(&bars[grp], 0, err) && ok;
    ZG::Engine::template run_inplace<false>(w[0] + (size_t)grp * P * N, tw);
  } else {
    for (int c = 0; c < 3; ++c) {
      ok = mbar_wait_bounded(&bars[c], 0, err) && ok;
      if (!ok && !paired) return;
      E::template run_inplace<false>(w[c], tw);
    }
  }
  ok = __syncthreads_and(ok);
  if (!ok && !paired) return;
  if (paired) {
    if (!COL) cluster_arrive();
    hermitian_column<T, P, N, NT, COL>(w, s_col, st, g, iy, base, zstride, fblock, fblock ? s_coef : T(0), flo_b, fk_b);
    if (!ok) return;
  }
  constexpr int EB = GROUPED ? 3 : (NT >= 512 ? 2 : 4);
  const bool tstore = MODE == SM_RK4 && vstore;
  zfwd_update<T, P, N, NT, EB, MODE>(w, st, g, kx0, iy, nvalid, base, zstride, fblock, fblock ? s_coef : T(0), flo_b,
                                     fk_b, paired, tstore);
  if (tstore) {
    fence_proxy_async();
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int c = 0; c < 3; ++c)
        for (int h = 0; h < Cfg::NBOX; ++h)
          tma_store_4d(&vmap, reinterpret_cast<char*>(w[c]) + (size_t)h * Cfg::BOX * P * sizeof(C), kx0 * Cfg::U,
                       iy, h * Cfg::BOX, c);
      tma_store_commit();
      tma_store_wait_read<0>();
    }
  }
}

// z-forward pass of a passive scalar's flux u phi (three fields, scaled by
// 1/N^3 in the x-pass): w_phi = i k . (u phi)^ (convecphi_dns.f90:25-47), plus
// the scalar's forcing, symmetrize and the dealiasing mask, leaving by bulk
// tensor stores.  Three forward passes, a divergence pass, up to two forcing
// passes, two symmetrize passes and the mask over whole fields become the
// flux read once and w_phi written once (4 F); latency-bound at 2 CTAs per SM
// as the other z-forward passes (86 us at 256^3 FP32, 3.1 TB/s).
template <typename T> struct DivArgs {
  const C2<T>* phi;       // band forcing: += (*fcoef) phi on flo2 <= k2 < fhi2 (fcoef may be null)
  const double* fcoef;
  K2Lt flo2, fhi2;
  const C2<T>* vz;        // mean gradient: -= meangrad vz (vz may be null)
  T meangrad;
  int mask;               // zero k2 >= kcut2 (k2 > 0)
  K2Lt kcut2;
};

template <typename T, int LOGN>
__global__ void __cluster_dims__(1, 2, 1) __launch_bounds__(ZfCfg<T, LOGN>::NT, 2)
zfwd_div_tma_kernel(const __grid_constant__ CUtensorMap fmap, const __grid_constant__ CUtensorMap omap, DivArgs<T> da,
                    Geom g, const C2<T>* __restrict__ tw, int* err) {
  pdl_wait();
  using Cfg = TmaCfg<T, LOGN>;
  using E = typename ZfCfg<T, LOGN>::Engine;
  using C = C2<T>;
  constexpr int P = Cfg::P;
  constexpr int N = Cfg::N;
  constexpr int NT = ZfCfg<T, LOGN>::NT;
  extern __shared__ __align__(128) unsigned char smdyn[];
  unsigned char* smraw = align128(smdyn);
  C* w[3];
  for (int c = 0; c < 3; ++c) w[c] = reinterpret_cast<C*>(smraw + c * Cfg::TILE_BYTES);
  __shared__ __align__(8) uint64_t bars[3];
  const int kx0 = blockIdx.x * P;
  const int iy = paired_row(blockIdx.y, g.ny);
  const int nvalid = min(P, g.nxh - kx0);
  const long long zstride = (long long)g.ny * g.nxp;
  const long long base = (long long)iy * g.nxp + kx0;
  const bool paired = kx0 == 0;   // meets its partner: both CTAs stay until then
  constexpr bool COL = ZfCfg<T, LOGN>::GROUPED;   // as zfwd_tma_kernel
  __shared__ C s_col[COL ? N / 2 : 1];
  if (paired && COL) cluster_arrive();
  if (!paired && launch_failed(err)) return;
  if (threadIdx.x == 0) {
    for (int c = 0; c < 3; ++c) mbar_init(&bars[c], 1);
    fence_mbar_init();
    fence_proxy_async();
    for (int c = 0; c < 3; ++c)
      tma_issue_tile<Cfg>(w[c], &fmap, &bars[c], 2, kx0, iy, c, P, Cfg::TILE_BYTES);
  }
  __syncthreads();
  bool ok = true;
  for (int c = 0; c < 3; ++c) {
    ok = mbar_wait_bounded(&bars[c], 0, err) && ok;
    if (!ok && !paired) return;
    E::template run_inplace<false>(w[c], tw);
  }
  const int kyi = wavenum(iy, g.ny);
  const int lo_b = da.flo2.b, hi_b = da.fhi2.b, kc_b = da.kcut2.b;
  const bool fblock = da.fcoef && kx0 * kx0 + kyi * kyi < hi_b;
  const T fc = fblock ? (T)*da.fcoef : T(0);
  constexpr int EB = NT >= 512 ? 2 : 4;
  for (int e0 = threadIdx.x; e0 < P * N; e0 += NT * EB) {
    C vz[EB];
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      const int e = e0 + i * NT;
      const int p = e % P, iz = e / P;
      vz[i] = czero<C>();
      if (da.vz && e < P * N && p < nvalid) vz[i] = da.vz[base + iz * zstride + p];
    }
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      const int e = e0 + i * NT;
      if (e >= P * N) continue;
      const int p = e % P, iz = e / P, ix = kx0 + p;
      const int kzi = wavenum(iz, g.nz), k2 = ix * ix + kyi * kyi + kzi * kzi;
      C d = cadd(cadd(cscale(w[0][e], (T)ix), cscale(w[1][e], (T)kyi)), cscale(w[2][e], (T)kzi));
      d = cmuli(d);
      if (fblock && k2 >= lo_b && k2 < hi_b && p < nvalid) d = cadd(d, cscale(da.phi[base + iz * zstride + p], fc));
      if (da.vz) d = csub(d, cscale(vz[i], da.meangrad));
      if (iy == g.ny / 2 || iz == g.nz / 2 || ix == g.nxh - 1 || k2 == 0 || (da.mask && k2 >= kc_b)) d = czero<C>();
      w[0][e] = d;
    }
  }
  if (paired) {
    // the kx = 0 copy: zeroing and mask are the same at k and -k
    __syncthreads();
    if (!COL) cluster_arrive();
    column_copy<1, P, N, NT, COL>(w, s_col, iy, g.ny, [](int, int, const C& v) { return v; });
    if (!ok) return;
  }
  fence_proxy_async();
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int h = 0; h < Cfg::NBOX; ++h)
      tma_store_4d(&omap, reinterpret_cast<char*>(w[0]) + (size_t)h * Cfg::BOX * P * sizeof(C), kx0 * Cfg::U, iy,
                   h * Cfg::BOX, 0);
    tma_store_commit();
    tma_store_wait_read<0>();
  }
}

}  // namespace sc
