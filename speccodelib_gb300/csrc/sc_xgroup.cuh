// Lane-group x-axis pass (c2r, physical-space products, r2c): a group of L
// lanes owns one grid row, 32 / L rows per warp.
//
// An M-point complex transform (M = nx/2 = L E, L <= E) is two register DFTs:
// lane l holds the points l + L r, an E-point DFT over r, twiddles W_M^{l k1},
// a transpose inside the group through a padded shared buffer after which
// lane l holds the E / L columns k1 = l + L b, and an L-point DFT over each.
// The inverse leaves every field in the same scrambled order (register b L +
// k2 of lane l: point l + L b + E k2), the products are formed there, and the
// forward transform is the transposed network back to natural order.
//
// Why next to the warp-per-row pass (sc_xwarp.cuh): that one finishes its
// transforms across 32 / E lanes with shuffle butterflies, in which both
// sides of a pair are computed by every lane.  In FP64 the pass is bound by
// the double-precision pipe (two lanes per SM), so operations are what counts:
// here every lane only computes values it keeps, and the half-length c2r /
// r2c steps handle the pair (k, M - k), whose sums, differences and twiddled
// products are conjugates of each other, once instead of twice (12 operations
// per pair, not 20); the final scale rides on fused multiply-adds.  About 225
// operations per complex point of a Lamb product instead of 565.  At 128^3
// FP64 a launch takes 448 us (the warp pass 940), near the pipe's 375.  In FP32
// it serves the short rows (M = 16, 32) that leave a whole warp per row no
// points to work on, in place of the block kernel (64^3 step 212 -> 201 us).
#pragma once
#include "sc_passes.cuh"
#include "sc_xwarp.cuh"

namespace sc {

template <typename T, int LOGM> struct GroupFFT {
  using C = C2<T>;
  static constexpr int M = 1 << LOGM;
  static constexpr int E = LOGM <= 4 ? 4 : (LOGM <= 6 ? 8 : 16);   // points per lane
  static constexpr int L = M / E;                                   // lanes per row
  static constexpr int B = E / L;
  static constexpr int RW = 32 / L;                                 // rows per warp
  static_assert(L >= 4 && L <= E && L <= 16, "group sizes");
  // Transpose buffer of a group: E rows of L + 1, so that a phase of the
  // banks (8 lanes of 16 bytes, 16 of 8) reads down a column without
  // conflicts; the groups that share a phase start L slots apart in it.
  static constexpr int ROW = L + 1;
  static constexpr int PH = sizeof(C) == 16 ? 8 : 16;
  static constexpr int PAD = L < PH ? ((L - E * ROW) % PH + PH) % PH : 0;
  static constexpr int BUF = E * ROW + PAD;

  template <bool INV> __device__ static __forceinline__ void twiddle(C (&x)[E], const C* __restrict__ tw, int l) {
#pragma unroll
    for (int k1 = 1; k1 < E; ++k1) {
      const C w = __ldg(&tw[l * k1]);
      x[k1] = INV ? cmulc(x[k1], w) : cmul(x[k1], w);
    }
  }
  template <bool INV>
  __device__ static __forceinline__ void nat_to_scr(C (&x)[E], C* buf, const C* __restrict__ tw, int l) {
    dftE<E, INV>(x);
    twiddle<INV>(x, tw, l);
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) buf[k1 * ROW + l] = x[k1];
    __syncwarp();
#pragma unroll
    for (int b = 0; b < B; ++b)
#pragma unroll
      for (int t = 0; t < L; ++t) x[b * L + t] = buf[(l + L * b) * ROW + t];
    __syncwarp();
#pragma unroll
    for (int b = 0; b < B; ++b) dftE<L, INV>(x + b * L);
  }
  template <bool INV>
  __device__ static __forceinline__ void scr_to_nat(C (&x)[E], C* buf, const C* __restrict__ tw, int l) {
#pragma unroll
    for (int b = 0; b < B; ++b) dftE<L, INV>(x + b * L);
#pragma unroll
    for (int b = 0; b < B; ++b)
#pragma unroll
      for (int t = 0; t < L; ++t) buf[(l + L * b) * ROW + t] = x[b * L + t];
    __syncwarp();
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) x[k1] = buf[k1 * ROW + l];
    __syncwarp();
    twiddle<INV>(x, tw, l);
    dftE<E, INV>(x);
  }
};

// One lane's view of its group's row at element offset `off` of every field.
template <typename T, int LOGM> struct XgRow {
  using GF = GroupFFT<T, LOGM>;
  using C = C2<T>;
  static constexpr int M = GF::M, E = GF::E, L = GF::L, H = GF::E / 2;
  C* buf;          // the group's transpose buffer
  C* keep;         // kept rows in scrambled order, lane-private: row c at [(c E + i) 32 + lane]
  const C* twM;
  const C* twN;
  long long off;
  int l, lane, mate;   // lane in the group, lane in the warp, lane that holds the mirrored columns
  bool live;           // the row exists (its results are stored)

  __device__ __forceinline__ C shfl(C v, int src) const {
    C r;
    r.x = __shfl_sync(0xffffffffu, v.x, src);
    r.y = __shfl_sync(0xffffffffu, v.y, src);
    return r;
  }
  __device__ __forceinline__ C& kept(int c, int i) const { return keep[(c * E + i) * 32 + lane]; }

  // Z of the half-length c2r in natural order.  A lane forms the pairs
  // (k, M - k) of its first E/2 points; Z_{M-k} belongs to the mate lane's
  // register E-1-r (lane 0: to its own register E-r, and Z_{M/2} = 2 conj X).
  // DX: of the x derivative i k X instead.
  template <bool DX = false> __device__ __forceinline__ void load_z(const C* f, C (&x)[E]) const {
    const C* rp = f + off;
    auto at = [&](int k) {
      const C v = rp[k];
      return DX ? cmuli(cscale(v, (T)k)) : v;
    };
    C zp[H];
#pragma unroll
    for (int r = 0; r < H; ++r) {
      const int k = l + L * r;
      C xk = at(k), xm = at(M - k);
      if (r == 0 && l == 0) { xk.y = 0; xm.y = 0; }   // DC and Nyquist are real
      const C e = cadd(xk, cconj(xm));
      const C o = cmulc(csub(xk, cconj(xm)), __ldg(&twN[k]));
      x[r] = mk<C>(e.x - o.y, e.y + o.x);      // e + i o
      zp[r] = mk<C>(e.x + o.y, o.x - e.y);     // conj(e) + i conj(o)
    }
    if (l == 0) {
      const C h = at(M / 2);
#pragma unroll
      for (int r = 0; r < H - 1; ++r) zp[r] = zp[r + 1];
      zp[H - 1] = mk<C>(h.x + h.x, -(h.y + h.y));
    }
#pragma unroll
    for (int r = 0; r < H; ++r) x[E - 1 - r] = shfl(zp[r], mate);
  }
  template <bool DX = false> __device__ __forceinline__ void load_phys(const C* f, C (&x)[E]) const {
    load_z<DX>(f, x);
    GF::template nat_to_scr<true>(x, buf, twM, l);
  }

  // The row's values from natural-order Z: X_k = s/2 (e - i d) in lo, X_{M-k} =
  // s/2 (conj e - i conj d) in hi (k = l + L r, r < E/2), X_{M/2} in mid (lane
  // 0), with e = Z_k + conj Z_{M-k}, d = W_N^k (Z_k - conj Z_{M-k})
  __device__ __forceinline__ void r2c_vals(C (&x)[E], C (&lo)[H], C (&hi)[H], C& mid, T s) const {
    GF::template scr_to_nat<false>(x, buf, twM, l);
    const T c = T(0.5) * s;
#pragma unroll
    for (int r = 0; r < H; ++r) {
      const C snd = l == 0 ? x[(E - r) % E] : x[E - 1 - r];
      const C zm = shfl(snd, mate), zk = x[r];
      const C e = cadd(zk, cconj(zm));
      const C d = cmul(csub(zk, cconj(zm)), cscale(__ldg(&twN[l + L * r]), c));
      lo[r] = mk<C>(c * e.x + d.y, c * e.y - d.x);
      hi[r] = mk<C>(c * e.x - d.y, -(c * e.y) - d.x);
    }
    mid = mk<C>(s * x[H].x, -(s * x[H].y));
  }
  __device__ __forceinline__ void store_vals(C* f, const C (&lo)[H], const C (&hi)[H], const C& mid) const {
    if (!live) return;
    C* op = f + off;
#pragma unroll
    for (int r = 0; r < H; ++r) {
      op[l + L * r] = lo[r];
      op[M - l - L * r] = hi[r];
    }
    if (l == 0) op[M / 2] = mid;
  }
  __device__ __forceinline__ void store_r2c(C (&x)[E], C* f, T s) const {
    C lo[H], hi[H], mid;
    r2c_vals(x, lo, hi, mid, s);
    store_vals(f, lo, hi, mid);
  }

  __device__ __forceinline__ void load_a(const C* const f[3]) const {
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      C x[E];
      load_phys(f[c], x);
#pragma unroll
      for (int i = 0; i < E; ++i) kept(c, i) = x[i];
    }
  }

  // out = r2c(sc (a x b)): b_x and b_y kept in rows 3 and 4, b_z in registers;
  // L_z leaves before b_z is read, as in the warp pass
  __device__ __forceinline__ void cross_store(const C* const bf[3], C* const of[3], T sc) const {
    C b[E], x[E];
    load_phys(bf[0], b);
#pragma unroll
    for (int i = 0; i < E; ++i) kept(3, i) = b[i];
    load_phys(bf[1], b);
#pragma unroll
    for (int i = 0; i < E; ++i) {
      kept(4, i) = b[i];
      const C ax = kept(0, i), ay = kept(1, i), bx = kept(3, i);
      x[i] = mk<C>(ax.x * b[i].x - ay.x * bx.x, ax.y * b[i].y - ay.y * bx.y);
    }
    store_r2c(x, of[2], sc);
    load_phys(bf[2], b);
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const C ay = kept(1, i), az = kept(2, i), by = kept(4, i);
      x[i] = mk<C>(ay.x * b[i].x - az.x * by.x, ay.y * b[i].y - az.y * by.y);
    }
    store_r2c(x, of[0], sc);
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const C ax = kept(0, i), az = kept(2, i), bx = kept(3, i);
      x[i] = mk<C>(az.x * bx.x - ax.x * b[i].x, az.y * bx.y - ax.y * b[i].y);
    }
    store_r2c(x, of[1], sc);
  }

  // XW_GRAD: rows 0-2 = u_c, 3 + 3 j + c = d_j u_c kept, then the products as
  // XwRow::les_store
  __device__ __forceinline__ void les_rows(const C* const f[9], C* const of[8], T sc, T tcoef) const {
    auto put = [&](int q, const C (&x)[E]) {
#pragma unroll
      for (int i = 0; i < E; ++i) kept(q, i) = x[i];
    };
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      C x[E];
      load_phys(f[c], x);
      put(c, x);
      load_phys<true>(f[c], x);
      put(3 + c, x);
    }
#pragma unroll 1
    for (int q = 3; q < 9; ++q) {
      C x[E];
      load_phys(f[q], x);
      put(3 + q, x);
    }
    auto S = [&](int p, int q, int i) {   // S_pq = (d_p u_q + d_q u_p) / 2
      const C a = kept(3 + 3 * p + q, i), b = kept(3 + 3 * q + p, i);
      return mk<C>(T(0.5) * (a.x + b.x), T(0.5) * (a.y + b.y));
    };
    C s[E];
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const C s11 = kept(3, i), s22 = kept(7, i), s33 = kept(11, i), s12 = S(0, 1, i), s13 = S(0, 2, i), s23 = S(1, 2, i);
      s[i].x = tcoef * sqrt(T(2) * (s11.x * s11.x + s22.x * s22.x + s33.x * s33.x +
                                    T(2) * (s12.x * s12.x + s13.x * s13.x + s23.x * s23.x)));
      s[i].y = tcoef * sqrt(T(2) * (s11.y * s11.y + s22.y * s22.y + s33.y * s33.y +
                                    T(2) * (s12.y * s12.y + s13.y * s13.y + s23.y * s23.y)));
    }
    C lo[H], hi[H], mid;
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
      C x[E], tl[H], th[H], tm;
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const C t = S(0, c, i);
        x[i] = mk<C>(s[i].x * t.x, s[i].y * t.y);
      }
      r2c_vals(x, tl, th, tm, T(1));
      if (c > 0) store_vals(of[c == 1 ? 3 : 6], tl, th, tm);   // tau_12, tau_13
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const C u1 = kept(c1, i), u2 = kept(c2, i);
        const C a = kept(3 + 3 * c + c1, i), b = kept(3 + 3 * c1 + c, i);
        const C d = kept(3 + 3 * c2 + c, i), e = kept(3 + 3 * c + c2, i);
        x[i] = mk<C>(u1.x * (a.x - b.x) - u2.x * (d.x - e.x), u1.y * (a.y - b.y) - u2.y * (d.y - e.y));
      }
      r2c_vals(x, lo, hi, mid, sc);
#pragma unroll
      for (int r = 0; r < H; ++r) {
        const int k = l + L * r;
        lo[r] = csub(lo[r], cmuli(cscale(tl[r], (T)k)));
        hi[r] = csub(hi[r], cmuli(cscale(th[r], (T)(M - k))));
      }
      mid = csub(mid, cmuli(cscale(tm, (T)(M / 2))));
      store_vals(of[c], lo, hi, mid);
    }
#pragma unroll 1
    for (int q = 0; q < 3; ++q) {   // tau_22, tau_23, tau_33
      C x[E];
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const C t = S(q == 2 ? 2 : 1, q == 0 ? 1 : 2, i);
        x[i] = mk<C>(s[i].x * t.x, s[i].y * t.y);
      }
      store_r2c(x, of[q == 2 ? 7 : 4 + q], T(1));
    }
  }

  // of[c] = r2c(sc a_c phi) (convecphi_dns.f90:20-23)
  __device__ __forceinline__ void flux_store(const C* pf, C* const of[3], T sc) const {
    C b[E];
    load_phys(pf, b);
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      C x[E];
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const C a = kept(c, i);
        x[i] = mk<C>(a.x * b[i].x, a.y * b[i].y);
      }
      store_r2c(x, of[c], sc);
    }
  }

  // tau_ij = tcoef |S| S_ij (smag.f90:41-64) of the S_ij rows sf (order 11 12
  // 13 22 23 33), kept in rows 0..5
  __device__ __forceinline__ void tau_store(const C* const sf[6], C* const of[6], T tcoef) const {
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
      C x[E];
      load_phys(sf[q], x);
#pragma unroll
      for (int i = 0; i < E; ++i) kept(q, i) = x[i];
    }
    C a[E];
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const C s11 = kept(0, i), s12 = kept(1, i), s13 = kept(2, i), s22 = kept(3, i), s23 = kept(4, i), s33 = kept(5, i);
      a[i].x = sqrt(T(2) * (s11.x * s11.x + s22.x * s22.x + s33.x * s33.x +
                            T(2) * (s12.x * s12.x + s13.x * s13.x + s23.x * s23.x)));
      a[i].y = sqrt(T(2) * (s11.y * s11.y + s22.y * s22.y + s33.y * s33.y +
                            T(2) * (s12.y * s12.y + s13.y * s13.y + s23.y * s23.y)));
    }
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
      C x[E];
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const C s = kept(q, i);
        x[i] = mk<C>(a[i].x * s.x, a[i].y * s.y);
      }
      store_r2c(x, of[q], tcoef);
    }
  }
};

template <typename T, int LOGM, int MODE> struct XgCfg {
  using GF = GroupFFT<T, LOGM>;
  static constexpr int KEPT = MODE == XW_GRAD ? 12 : (MODE == XW_SMAG ? 6 : 5);
  static constexpr int PER_WARP = GF::RW * (KEPT * GF::M + GF::BUF);
  // four warps, fewer where their kept rows pass the 227 KB of a CTA
  static constexpr int FIT = (int)(227 * 1024 / (sizeof(C2<T>) * PER_WARP));
  static constexpr int WARPS = FIT < 4 ? FIT : 4, NT = 32 * WARPS;
  static constexpr size_t SMEM = sizeof(C2<T>) * (size_t)PER_WARP * WARPS;
  static constexpr int MINB = SMEM * 2 <= 220 * 1024 ? 2 : 1;
};

template <typename T, int LOGM>
__device__ __forceinline__ XgRow<T, LOGM> xg_row(C2<T>* warp_smem, int kept, long long warp, const Geom& g,
                                                 const C2<T>* twM, const C2<T>* twN, long long rows) {
  using GF = GroupFFT<T, LOGM>;
  XgRow<T, LOGM> R;
  R.lane = threadIdx.x & 31;
  R.l = R.lane % GF::L;
  const int q = R.lane / GF::L;
  R.mate = q * GF::L + (GF::L - R.l) % GF::L;
  R.keep = warp_smem;
  R.buf = warp_smem + kept * GF::M * GF::RW + q * GF::BUF;
  const long long row = warp * GF::RW + q;
  R.live = row < rows;
  R.off = (R.live ? row : rows - 1) * g.nxp;
  R.twM = twM;
  R.twN = twN;
  return R;
}

// Modes, operands and aliasing as xpass_warp_kernel (sc_xwarp.cuh); XW_SMAG
// reads u and w before its first output and S_ij before it writes tau_ij.
template <typename T, int LOGM, int MODE>
__global__ void __launch_bounds__(XgCfg<T, LOGM, MODE>::NT, XgCfg<T, LOGM, MODE>::MINB)
xpass_group_kernel(FieldList<T> fin, FieldList<T> fout, Geom g, const C2<T>* __restrict__ twM,
                   const C2<T>* __restrict__ twN, XArgs<T> xa) {
  using C = C2<T>;
  using Cfg = XgCfg<T, LOGM, MODE>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int warp = threadIdx.x >> 5;
  const XgRow<T, LOGM> R = xg_row<T, LOGM>(reinterpret_cast<C*>(smraw) + warp * Cfg::PER_WARP, Cfg::KEPT,
                                           (long long)blockIdx.x * Cfg::WARPS + warp, g, twM, twN, xa.rows);
  const C* u[3] = {fin.f[0], fin.f[1], fin.f[2]};
  const C* w[3] = {fin.f[3], fin.f[4], fin.f[5]};
  C* o[3] = {fout.f[0], fout.f[1], fout.f[2]};
  if constexpr (MODE == XW_DNS || MODE == XW_SCALAR) {
    R.load_a(u);
    R.cross_store(w, o, xa.scale);
    if constexpr (MODE == XW_SCALAR) {
      C* of[3] = {fout.f[3], fout.f[4], fout.f[5]};
      R.flux_store(fin.f[6], of, xa.scale);
    }
  } else if constexpr (MODE == XW_GRAD) {
    const C* f[9] = {u[0], u[1], u[2], fin.f[6], fin.f[7], fin.f[8], w[0], w[1], w[2]};
    C* of[8] = {o[0], o[1], o[2], fout.f[3], fout.f[4], fout.f[5], fout.f[6], fout.f[7]};
    R.les_rows(f, of, xa.scale, (T)(-2.0 * (*xa.c1) * xa.delta2) * xa.scale);
  } else if constexpr (MODE == XW_SMAG) {
    const C* s[6] = {fin.f[6], fin.f[7], fin.f[8], fin.f[9], fin.f[10], fin.f[11]};
    C* ot[6] = {fout.f[3], fout.f[4], fout.f[5], fout.f[6], fout.f[7], fout.f[8]};
    R.load_a(u);
    R.cross_store(w, o, xa.scale);
    R.tau_store(s, ot, (T)(-2.0 * (*xa.c1) * xa.delta2) * xa.scale);
  } else {
    const C* phi[3] = {fin.f[6], fin.f[7], fin.f[8]};
    C* o2[3] = {fout.f[3], fout.f[4], fout.f[5]};
    R.load_a(phi);
    R.cross_store(w, o, T(-1));
    R.cross_store(u, o2, T(1));
  }
}

// max |u|^2 and the non-finite count of three velocity fields, as
// xpass_umax_kernel.
template <typename T, int LOGM> struct XgUmaxCfg {
  using GF = GroupFFT<T, LOGM>;
  static constexpr int PER_WARP = GF::RW * GF::BUF;
  static constexpr int WARPS = 8, NT = 32 * WARPS;
  static constexpr size_t SMEM = sizeof(C2<T>) * (size_t)PER_WARP * WARPS;
};
template <typename T, int LOGM>
__global__ void __launch_bounds__(XgUmaxCfg<T, LOGM>::NT)
xgroup_umax_kernel(FieldList<T> fin, Geom g, const C2<T>* __restrict__ twM, const C2<T>* __restrict__ twN, XArgs<T> xa,
                   unsigned long long* out) {
  using C = C2<T>;
  using Cfg = XgUmaxCfg<T, LOGM>;
  constexpr int E = GroupFFT<T, LOGM>::E;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int warp = threadIdx.x >> 5;
  const XgRow<T, LOGM> R = xg_row<T, LOGM>(reinterpret_cast<C*>(smraw) + warp * Cfg::PER_WARP, 0,
                                           (long long)blockIdx.x * Cfg::WARPS + warp, g, twM, twN, xa.rows);
  C u2[E];
#pragma unroll
  for (int i = 0; i < E; ++i) u2[i] = czero<C>();
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    C x[E];
    R.load_phys(fin.f[c], x);
#pragma unroll
    for (int i = 0; i < E; ++i) u2[i] = mk<C>(x[i].x * x[i].x + u2[i].x, x[i].y * x[i].y + u2[i].y);
  }
  T m = T(0);
  int nf = 0;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    m = fmax(m, fmax(u2[i].x, u2[i].y));
    nf += (!isfinite(u2[i].x) || !isfinite(u2[i].y)) ? 1 : 0;
  }
  umax_block_out<Cfg::WARPS>(R.live ? (double)m : 0.0, R.live ? nf : 0, out);
}

}  // namespace sc
