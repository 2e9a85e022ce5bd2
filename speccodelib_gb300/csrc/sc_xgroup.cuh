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
// FP64 a launch takes 448 us (the warp pass 940), near the pipe's 375.
//
// In FP32 it serves rows of M = 16 to 64, where a whole warp per row has one
// or two points per lane (block kernel at 16 and 32): Lamb product at 128^3
// 34.9 -> 18.0 us, its adjoint 56 -> 29, the LES products 92 -> 58; 64^3 step
// 212 -> 201.  At M = 128 both forms take the same time (181 us at 256^3; the
// LES products 458 in the warp pass, 684 here) and at M = 256 the warp pass
// with its staged rows is faster (1.20 ms at 512^3, 1.33 here): the line lies
// between 64 and 128.
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
// KT: the first KT kept rows wait in tensor memory (FP32), the others in
// shared memory; both are lane-private, read four points at a time.
template <typename T, int LOGM, int KT = 0> struct XgRow {
  using GF = GroupFFT<T, LOGM>;
  using C = C2<T>;
  static constexpr int M = GF::M, E = GF::E, L = GF::L, H = GF::E / 2;
  C* buf;          // the group's transpose buffer
  C* keep;         // kept rows in scrambled order: row c >= KT at [((c - KT) E + i) 32 + lane]
  uint32_t ta = 0; // row c < KT at columns ta + 2 E c .. of the warp's lanes
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
  __device__ __forceinline__ void put(int c, const C (&x)[E]) const {
    if (c < KT) {
      if constexpr (KT > 0 && sizeof(T) == 4) {
#pragma unroll
        for (int i0 = 0; i0 < E; i0 += 8) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            w[2 * i] = __float_as_uint(x[i0 + i].x);
            w[2 * i + 1] = __float_as_uint(x[i0 + i].y);
          }
          tmem_store16(ta + (uint32_t)(2 * E * c + 2 * i0), w);
        }
        tmem_wait_store();
      }
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i) keep[((c - KT) * E + i) * 32 + lane] = x[i];
    }
  }
  // row c at points i0 .. i0 + 3
  __device__ __forceinline__ void get(int c, int i0, C (&a)[4]) const {
    if (c < KT) {
      if constexpr (KT > 0 && sizeof(T) == 4) {
        uint32_t w[8];
        tmem_load8(ta + (uint32_t)(2 * E * c + 2 * i0), w);
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = mk<C>(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = keep[((c - KT) * E + i0 + i) * 32 + lane];
    }
  }

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
    C* op = f + off;
    if (live) {
#pragma unroll
      for (int r = 0; r < H; ++r) {
        op[l + L * r] = lo[r];
        op[M - l - L * r] = hi[r];
      }
      if (l == 0) op[M / 2] = mid;
    }
    __syncwarp();   // tensor-memory accesses are warp-collective
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
      put(c, x);
    }
  }

  // out = r2c(sc (a x b)): b_x and b_y kept in rows 3 and 4, b_z in registers;
  // L_z leaves before b_z is read, as in the warp pass
  __device__ __forceinline__ void cross_store(const C* const bf[3], C* const of[3], T sc) const {
    C b[E], x[E];
    load_phys(bf[0], b);
    put(3, b);
    load_phys(bf[1], b);
    put(4, b);
#pragma unroll
    for (int i0 = 0; i0 < E; i0 += 4) {
      C ax[4], ay[4], bx[4];
      get(0, i0, ax);
      get(1, i0, ay);
      get(3, i0, bx);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        x[i0 + i] = mk<C>(ax[i].x * b[i0 + i].x - ay[i].x * bx[i].x, ax[i].y * b[i0 + i].y - ay[i].y * bx[i].y);
    }
    store_r2c(x, of[2], sc);
    load_phys(bf[2], b);
#pragma unroll
    for (int i0 = 0; i0 < E; i0 += 4) {
      C ay[4], az[4], by[4];
      get(1, i0, ay);
      get(2, i0, az);
      get(4, i0, by);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        x[i0 + i] = mk<C>(ay[i].x * b[i0 + i].x - az[i].x * by[i].x, ay[i].y * b[i0 + i].y - az[i].y * by[i].y);
    }
    store_r2c(x, of[0], sc);
#pragma unroll
    for (int i0 = 0; i0 < E; i0 += 4) {
      C ax[4], az[4], bx[4];
      get(0, i0, ax);
      get(2, i0, az);
      get(3, i0, bx);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        x[i0 + i] = mk<C>(az[i].x * bx[i].x - ax[i].x * b[i0 + i].x, az[i].y * bx[i].y - ax[i].y * b[i0 + i].y);
    }
    store_r2c(x, of[1], sc);
  }

  // t[0..3] = S_pq = (d_p u_q + d_q u_p) / 2 at points i0 .. from the kept
  // gradient rows of les_rows
  __device__ __forceinline__ void strain(int p, int q, int i0, C (&t)[4]) const {
    get(3 + 3 * p + q, i0, t);
    if (p == q) return;
    C b[4];
    get(3 + 3 * q + p, i0, b);
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = mk<C>(T(0.5) * (t[i].x + b[i].x), T(0.5) * (t[i].y + b[i].y));
  }

  // XW_GRAD: rows 0-2 = u_c, 3 + 3 j + c = d_j u_c kept, then the products as
  // XwRow::les_store
  __device__ __forceinline__ void les_rows(const C* const f[9], C* const of[8], T sc, T tcoef) const {
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
    C s[E];
#pragma unroll
    for (int i0 = 0; i0 < E; i0 += 4) {
      C d[4], o[4], t[4];
      auto add = [&](C (&acc)[4], bool first) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          acc[i] = first ? mk<C>(t[i].x * t[i].x, t[i].y * t[i].y)
                         : mk<C>(t[i].x * t[i].x + acc[i].x, t[i].y * t[i].y + acc[i].y);
      };
      strain(0, 0, i0, t);
      add(d, true);
      strain(1, 1, i0, t);
      add(d, false);
      strain(2, 2, i0, t);
      add(d, false);
      strain(0, 1, i0, t);
      add(o, true);
      strain(0, 2, i0, t);
      add(o, false);
      strain(1, 2, i0, t);
      add(o, false);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        s[i0 + i] = mk<C>(tcoef * sqrt(T(2) * (d[i].x + T(2) * o[i].x)), tcoef * sqrt(T(2) * (d[i].y + T(2) * o[i].y)));
    }
    auto tau = [&](int p, int q, C (&x)[E]) {
#pragma unroll
      for (int i0 = 0; i0 < E; i0 += 4) {
        C t[4];
        strain(p, q, i0, t);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i0 + i] = mk<C>(s[i0 + i].x * t[i].x, s[i0 + i].y * t[i].y);
      }
    };
    C lo[H], hi[H], mid;
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
      C x[E], tl[H], th[H], tm;
      tau(0, c, x);
      r2c_vals(x, tl, th, tm, T(1));
      if (c > 0) store_vals(of[c == 1 ? 3 : 6], tl, th, tm);   // tau_12, tau_13
#pragma unroll
      for (int i0 = 0; i0 < E; i0 += 4) {
        // L_c = u_c1 (d_c u_c1 - d_c1 u_c) - u_c2 (d_c2 u_c - d_c u_c2)
        C u[4], a[4], b[4];
        get(c1, i0, u);
        get(3 + 3 * c + c1, i0, a);
        get(3 + 3 * c1 + c, i0, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i0 + i] = mk<C>(u[i].x * (a[i].x - b[i].x), u[i].y * (a[i].y - b[i].y));
        get(c2, i0, u);
        get(3 + 3 * c2 + c, i0, a);
        get(3 + 3 * c + c2, i0, b);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          x[i0 + i] = mk<C>(x[i0 + i].x - u[i].x * (a[i].x - b[i].x), x[i0 + i].y - u[i].y * (a[i].y - b[i].y));
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
      tau(q == 2 ? 2 : 1, q == 0 ? 1 : 2, x);
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
      for (int i0 = 0; i0 < E; i0 += 4) {
        C a[4];
        get(c, i0, a);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i0 + i] = mk<C>(a[i].x * b[i0 + i].x, a[i].y * b[i0 + i].y);
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
      put(q, x);
    }
    C a[E];
#pragma unroll
    for (int i0 = 0; i0 < E; i0 += 4) {
      C s[6][4];
#pragma unroll
      for (int q = 0; q < 6; ++q) get(q, i0, s[q]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i0 + i].x = sqrt(T(2) * (s[0][i].x * s[0][i].x + s[3][i].x * s[3][i].x + s[5][i].x * s[5][i].x +
                                   T(2) * (s[1][i].x * s[1][i].x + s[2][i].x * s[2][i].x + s[4][i].x * s[4][i].x)));
        a[i0 + i].y = sqrt(T(2) * (s[0][i].y * s[0][i].y + s[3][i].y * s[3][i].y + s[5][i].y * s[5][i].y +
                                   T(2) * (s[1][i].y * s[1][i].y + s[2][i].y * s[2][i].y + s[4][i].y * s[4][i].y)));
      }
    }
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
      C x[E];
#pragma unroll
      for (int i0 = 0; i0 < E; i0 += 4) {
        C s[4];
        get(q, i0, s);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i0 + i] = mk<C>(a[i0 + i].x * s[i].x, a[i0 + i].y * s[i].y);
      }
      store_r2c(x, of[q], tcoef);
    }
  }
};

template <typename T, int LOGM, int MODE> struct XgCfg {
  using GF = GroupFFT<T, LOGM>;
  static constexpr int KEPT = MODE == XW_GRAD ? 12 : (MODE == XW_SMAG ? 6 : 5);
  // FP32 rows of 64 points: three (XW_GRAD: six) kept rows in tensor memory,
  // which leaves shared memory for four CTAs per SM (LES products at 128^3 71
  // -> 58 us); a warp per lane quarter
  static constexpr int KT = sizeof(T) == 4 && LOGM >= 6 ? (MODE == XW_GRAD ? 6 : 3) : 0;
  static constexpr int TM_COLS = 2 * GF::E * KT <= 64 ? 64 : 128;
  static_assert(2 * GF::E * KT <= TM_COLS, "tensor-memory rows");
  static constexpr int PER_WARP = GF::RW * ((KEPT - KT) * GF::M + GF::BUF);
  // Warps per CTA: four (fewer where their kept rows pass the 227 KB of a CTA).
  // FP64 rows of up to 128 points one: the warps need nothing of each other, and
  // few rows then reach more SMs (four steps, FP64: LES at 64 x 32 x 32 4.30 -> 4.06
  // ms, DNS at 256 x 32 x 32 4.06 -> 3.80; 128^3 unchanged).  At 256 points it is slower
  // (512 x 32 x 32 LES 12.8 -> 18.0 ms).
  static constexpr int FIT = (int)(227 * 1024 / (sizeof(C2<T>) * PER_WARP));
  static constexpr int WMAX = sizeof(T) == 8 && LOGM < 8 ? 1 : 4;
  static constexpr int WARPS = FIT < WMAX ? FIT : WMAX, NT = 32 * WARPS;
  static constexpr size_t SMEM = sizeof(C2<T>) * (size_t)PER_WARP * WARPS;
  static constexpr int FITB = (int)(220 * 1024 / SMEM), MAXB = sizeof(T) == 4 ? 4 : 8 / WARPS;
  static constexpr int MINB = FITB < 1 ? 1 : (FITB > MAXB ? MAXB : FITB);
};

template <typename T, int LOGM, int KT = 0>
__device__ __forceinline__ XgRow<T, LOGM, KT> xg_row(C2<T>* warp_smem, int kept, long long warp, const Geom& g,
                                                     const C2<T>* twM, const C2<T>* twN, long long rows) {
  using GF = GroupFFT<T, LOGM>;
  XgRow<T, LOGM, KT> R;
  R.lane = threadIdx.x & 31;
  R.l = R.lane % GF::L;
  const int q = R.lane / GF::L;
  R.mate = q * GF::L + (GF::L - R.l) % GF::L;
  R.keep = warp_smem;
  R.buf = warp_smem + (kept - KT) * GF::M * GF::RW + q * GF::BUF;
  const long long row = warp * GF::RW + q;
  R.live = row < rows;
  R.off = (R.live ? row : rows - 1) * g.nxp;
  R.twM = twM;
  R.twN = twN;
  return R;
}

// Few rows.  A warp here works on its 32 / L rows for as long with one warp per SM
// as with a full one (FP64, Lamb product: 57 us at M = 32, 63 at 64, 137 at 128, 171
// at 256), so FP64 grids of few rows leave most of the chip idle, and the block
// kernel, a CTA per row, is faster: at 512 rows 39, 45, 48 and 101 us, the S_ij
// products 61, 70, 136 and 292 (here 138, 151, 329, 411).  At 1024 rows it is 39,
// 45, 91 and 198 us, and from 2048 on slower; the S_ij products at M = 128 stay
// faster there to 4096 rows (922 us, here 1019; 8192: 1769, 1707), three warps per
// SM filling this kernel's rounds badly.  The line: 6 rows per SM, 27 for the latter.
// FP32 rows (a Lamb product of 64 rows in 5 to 6 us) have no such case; M = 16
// neither (27 us, block 33).
template <typename T, int LOGM, int MODE> inline bool xg_few_rows(long long rows, int nsm) {
  if (sizeof(T) == 4 || LOGM < 5 || MODE == XW_SCALAR) return false;   // XW_SCALAR: no block kernel
  return rows <= (MODE == XW_SMAG && LOGM == 7 ? 27LL : 6LL) * nsm;
}

// The gradient form of the LES right-hand side: where XW_GRAD has the row length,
// except in FP64 where few rows would go to the block kernel (Smagorinsky step at 256
// rows, M = 32 / 64: 786 / 869 us, with the block kernel's S_ij products 573 / 629;
// at 1024: 1004 / 1173 and 900 / 1225) and at M = 128 and 256, where twelve kept rows
// leave two warps per SM (256 x 128 x 128 32.0 ms, with S_ij 27.8; 512 x 64 x 64 16.1
// and 13.1; 128^3 11.3 and 13.0).
template <typename T> inline bool les_gradient_rows(int logm, long long rows, int nsm) {
  if (logm < 4 || logm > (sizeof(T) == 4 ? 8 : 6)) return false;
  return logm == 5   ? !xg_few_rows<T, 5, XW_GRAD>(rows, nsm)
         : logm == 6 ? !xg_few_rows<T, 6, XW_GRAD>(rows, nsm)
                     : true;
}

// Modes, operands and aliasing as xpass_warp_kernel (sc_xwarp.cuh); XW_SMAG
// reads u and w before its first output and S_ij before it writes tau_ij.
template <typename T, int LOGM, int MODE>
__global__ void __launch_bounds__(XgCfg<T, LOGM, MODE>::NT, XgCfg<T, LOGM, MODE>::MINB)
xpass_group_kernel(FieldList<T> fin, FieldList<T> fout, Geom g, const C2<T>* __restrict__ twM,
                   const C2<T>* __restrict__ twN, XArgs<T> xa) {
  pdl_wait();
  using C = C2<T>;
  using Cfg = XgCfg<T, LOGM, MODE>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int warp = threadIdx.x >> 5;
  auto R = xg_row<T, LOGM, Cfg::KT>(reinterpret_cast<C*>(smraw) + warp * Cfg::PER_WARP, Cfg::KEPT,
                                    (long long)blockIdx.x * Cfg::WARPS + warp, g, twM, twN, xa.rows);
  __shared__ uint32_t s_tmem;
  if constexpr (Cfg::KT > 0) {
    static_assert(Cfg::KT == 0 || Cfg::WARPS == 4, "a warp per lane quarter of tensor memory");
    if (warp == 0) tmem_alloc(&s_tmem, Cfg::TM_COLS);
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    R.ta = s_tmem + ((uint32_t)(32 * warp) << 16);
  }
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
  if constexpr (Cfg::KT > 0) {
    // every warp's tensor-memory reads are complete before the release
    tmem_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      tmem_fence_after_sync();
      tmem_dealloc(s_tmem, Cfg::TM_COLS);
    }
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
  const auto R = xg_row<T, LOGM>(reinterpret_cast<C*>(smraw) + warp * Cfg::PER_WARP, 0,
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
