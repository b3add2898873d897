// stage2d.cuh -- fused 2D stage kernel, included by stage2d.cu,
// stage2d_tma.cu, batch.cu and batch16.cu (each with its tile constants).
//
// One launch evaluates the reference's whole spatial operator for a TX x TY
// tile of interior cells and writes the stage result, its ghost images and
// the per-dimension fast-speed maxima.  The terms are those of the
// reference's step (src/iosmaug.c:631-835); sums are regrouped at rounding
// level (agreement with the reference stays ~1e-16 relative):
//   - divisions by rho_t and by the cell width are multiplications with
//     reciprocals;
//   - the source of a hyperdiffusion pass is a difference of face fluxes: with
//     R(i) = max|D3| / max|D1| the reference's coefficients are nu_r(i) = c(i)
//     R(i), nu_l(i) = c(i) R(i-1), c = dl cmax chyp, so that the pass adds dt
//     cmax/dl (G(i) - G(i-1)) with G(i) = chyp R(i) (q(i+1) - q(i)) x face mean;
//   - increments are summed from zero and added to the base state.
//
// Two precision forms share the code (template MIX):
//   FP64   every value and every operation in double;
//   mixed  perturbation fields stored in float (stage buffers, and the base
//          state as a float high/low pair), backgrounds in double; fluxes,
//          the pressure recovery p_t = (g-1)(e - m^2/2rho_t) - ..., the
//          CFL speeds, the stage sums and the RK4 accumulator in double;
//          the hyperdiffusion ratios and face fluxes in float, with q itself
//          formed in double and every pass's increment summed in double.
//
// A block works in phases over the tile, all fields and both directions per
// phase, so that it meets five block barriers:
//   0  staging: q of the six hyperdiffusion fields on the tile + 3-cell halo
//   1  centred fluxes of both directions on the tile +-2
//   2  own cell: divergence of the fluxes, background coupling, gravity
//   3  nu ratios of all ten passes; one thread takes a line of a field (11
//      faces along x, the tile's height along y; ratio_line): 14 to 16 loads
//      per line instead of six per face
//   4  own cell: diffusive terms; cross-term arrays of the four passes that
//      have them
//   5  own cell: cross terms, driver, stage sum, stores, ghost images, CFL
//      maxima
// The arrays of phases 1-2 and 3-5 share their memory (66 KB in FP64 without
// background fields: three blocks of 256 threads at 80 registers).
//
// Bound by issue and latency, not by HBM: 57 warp instructions per cell and
// stage at 49 % issue.  With every pass on its own the kernel took 109 at 60 %.
// RK4 per step then and now: 4096^2 FP64 10.50 and 6.43 ms (2.3 ms at the
// measured copy bandwidth), 64^2 0.092 and 0.049, 2048^2 mixed 2.46 and 1.40.
#pragma once

// (included inside namespace smaug)
namespace s2 {
// rows of the staged arrays: an odd pitch, so that lines along x taken by
// neighbouring threads fall on different banks
constexpr int QX = RX | 1;
constexpr int QC = QX * RY;
// staged fields: q of rho, e, v1, v2, b1, b2; the mixed form also keeps the
// momenta and the energy as stored (floats), which products with 1/rho_t would
// round again
enum { QR = 0, QE = 1, QV1 = 2, QV2 = 3, QB1 = 4, QB2 = 5, QM1 = 6, QM2 = 7, QEN = 8 };
template <bool BG, bool MIX, bool O6>
struct Lay {
  using H = typename Form<MIX>::H;
  static constexpr int NQ = MIX ? 9 : 6;
  static constexpr int NC = MIX ? 4 : 3;     // cross arrays: m, B, energy (v and b parts)
  // flux arrays: the tile +-2 along the direction (+-3 along dim 0 for the
  // 6th-order derivative, which a 2D build of the reference applies along
  // dim 0 only: its dir-1 USE_DORDER3 branch is overwritten by the 4th-order
  // form, src/gradops.cu:536-544)
  static constexpr int FH = O6 ? 3 : 2;
  static constexpr int FXW = TX + 2 * FH, FXN = FXW * TY, FYN = TX * (TY + 4);
  // ratio arrays of the five passes along x (faces -1 .. TX-1, rows -1 .. TY)
  // and along y (columns -1 .. TX, faces -1 .. TY-1); cross arrays on the tile
  // +-1 across
  static constexpr int RXW = TX + 1, RXN = RXW * (TY + 2), RYW = TX + 2, RYN = RYW * (TY + 1);
  static constexpr int CXN = TX * (TY + 2), CYW = TX + 2, CYN = CYW * TY;
  // byte offsets; double arrays first
  static constexpr int RT = 0;                                  // rho_t (background fields only)
  static constexpr int RI = RT + (BG ? QC * 8 : 0);             // 1/rho_t (mixed only)
  static constexpr int RD = RI + (MIX ? QC * 8 : 0);            // 1/dl of the region's columns and rows
  static constexpr int U = RD + (RX + RY) * 8;                  // union
  static constexpr int FB = 5 * (FXN + FYN) * 8;
  static constexpr int HB = (5 * (RXN + RYN) + NC * (CXN + CYN)) * (int)sizeof(H);
  static constexpr int Q = U + ((FB > HB ? FB : HB) + 15) / 16 * 16;
  static constexpr int BYTES = Q + NQ * QC * (int)sizeof(H);
};
template <bool BG, bool MIX, bool O6 = false>
__host__ __device__ constexpr size_t smem_bytes() {
  return Lay<BG, MIX, O6>::BYTES;
}

// derived values of one region cell (r: its index in the staged arrays)
template <bool BG, bool MIX, bool O6, typename ST>
__device__ __forceinline__ void derive(char* sm, int r, bool ok, const ST* w, double rhob) {
  using L = Lay<BG, MIX, O6>;
  using HT = typename L::H;
  HT* const Q = reinterpret_cast<HT*>(sm + L::Q);
  const double m1 = (double)w[M1], m2 = (double)w[M2], b1 = (double)w[B1], b2 = (double)w[B2];
  double rt = BG ? (double)w[RHO] + rhob : (double)w[RHO];
  if (!ok) rt = 1.0;
  const double ri = recip(rt);
  const double v1 = mulr(m1, ri), v2 = mulr(m2, ri);
  Q[QR * QC + r] = (HT)w[RHO];
  Q[QE * QC + r] = (HT)fma(-0.5, fma(b1, b1, fma(b2, b2, fma(m1, v1, mulr(m2, v2)))), (double)w[EN]);
  Q[QV1 * QC + r] = (HT)v1;
  Q[QV2 * QC + r] = (HT)v2;
  Q[QB1 * QC + r] = (HT)w[B1];
  Q[QB2 * QC + r] = (HT)w[B2];
  if constexpr (MIX) {
    Q[QM1 * QC + r] = (HT)w[M1];
    Q[QM2 * QC + r] = (HT)w[M2];
    Q[QEN * QC + r] = (HT)w[EN];
    reinterpret_cast<double*>(sm + L::RI)[r] = ri;
  }
  if (BG) reinterpret_cast<double*>(sm + L::RT)[r] = rt;
}

// fluxes of rho, m1, m2, e and the B component across at region cell r, along
// dim 0 (X) into fx[k * sx] and along dim 1 (Y) into fy[k * sy]
// (src/centdiff1.cu:51-197, src/centdiff2.cu:203-323):
//   F_rho = m_D (= m_D rho'/rho_t + rho_b m_D/rho_t)
//   F_m_c = v_D m_c + delta_cD p_t - (B'_c Bb_D + Bb_c B'_D) - B'_c B'_D
//   F_e   = v_D (e + p_t + e_b) - (B'_D (Bb.m) + Bb_D (B'.m) + B'_D (B'.m)) / rho_t
//   F_B_c = v_D (B'_c + Bb_c) - v_c (B'_D + Bb_D)
// The momentum flux across is symmetric and the induction flux antisymmetric.
// In the FP64 form e and p_t come from the staged q_e = e - (B'^2 + m.v)/2:
// p_t = (g-1)(q_e + B'^2/2) - (g-2)(B'.Bb + B'^2/2).
template <bool BG, bool MIX, bool O6, bool X, bool Y>
__device__ __forceinline__ void flux_at(const char* sm, double gamma, int r, const double* g, double* fx, int sx,
                                        double* fy, int sy) {
  using L = Lay<BG, MIX, O6>;
  using HT = typename L::H;
  const HT* const Q = reinterpret_cast<const HT*>(sm + L::Q);
  const double b1 = (double)Q[QB1 * QC + r], b2 = (double)Q[QB2 * QC + r];
  double m1, m2, v1, v2, e, msr;
  const double hb = 0.5 * fma(b1, b1, mulr(b2, b2));
  if constexpr (MIX) {
    const double ri = reinterpret_cast<const double*>(sm + L::RI)[r];
    m1 = (double)Q[QM1 * QC + r];
    m2 = (double)Q[QM2 * QC + r];
    v1 = mulr(m1, ri);
    v2 = mulr(m2, ri);
    msr = 0.5 * fma(m1, v1, mulr(m2, v2));
    e = (double)Q[QEN * QC + r] - msr;
  } else {
    const double rt = BG ? reinterpret_cast<const double*>(sm + L::RT)[r] : (double)Q[QR * QC + r];
    v1 = (double)Q[QV1 * QC + r];
    v2 = (double)Q[QV2 * QC + r];
    m1 = mulr(v1, rt);
    m2 = mulr(v2, rt);
    msr = 0.5 * fma(m1, v1, mulr(m2, v2));
    e = (double)Q[QE * QC + r] + hb;
  }
  const double bb1 = BG ? g[2] : 0.0, bb2 = BG ? g[3] : 0.0;
  // computept3 (src/dervfields.cu:107-153); e holds the energy without m.v/2
  const double pt =
      fma(gamma - 1.0, e, -mulr(gamma - 2.0, BG ? fma(b1, bb1, fma(b2, bb2, hb)) : hb));
  const double t1 = BG ? b1 + bb1 : b1, t2 = BG ? b2 + bb2 : b2;
  const double bv = fma(b1, v1, mulr(b2, v2));
  const double tv = BG ? fma(bb1, v1, fma(bb2, v2, bv)) : bv;  // (B' + B_b) . v
  const double h = (e + msr) + (BG ? pt + g[0] : pt);
  const double s12 = fma(v1, m2, -(BG ? fma(b1, t2, mulr(bb1, b2)) : mulr(b1, b2)));
  const double ind = fma(v1, t2, -mulr(v2, t1));
  if (X) {
    fx[0] = m1;
    fx[sx] = fma(v1, m1, pt) - (BG ? fma(b1, t1, mulr(bb1, b1)) : mulr(b1, b1));
    fx[2 * sx] = s12;
    fx[3 * sx] = fma(v1, h, -(BG ? fma(b1, tv, mulr(bb1, bv)) : mulr(b1, bv)));
    fx[4 * sx] = ind;
  }
  if (Y) {
    fy[0] = m2;
    fy[sy] = s12;
    fy[2 * sy] = fma(v2, m2, pt) - (BG ? fma(b2, t2, mulr(bb2, b2)) : mulr(b2, b2));
    fy[3 * sy] = fma(v2, h, -(BG ? fma(b2, tv, mulr(bb2, bv)) : mulr(b2, bv)));
    fy[4 * sy] = -ind;
  }
}

// The diffusive terms of the five passes along D at the tile cell r.
// p: the passes' ratio arrays at faces i and i-1 -- rho, e and the momentum
// along D hold R dq, the momentum and B across D hold R.
template <bool BG, bool MIX, bool O6, int D>
__device__ __forceinline__ void diffuse(const char* sm, const double* chyp, int r, double k,
                                        const typename Form<MIX>::H* p, int pn, int ps, double* out) {
  using L = Lay<BG, MIX, O6>;
  using HT = typename L::H;
  constexpr int S = D == 0 ? 1 : QX;
  constexpr int QA = D == 0 ? QV2 : QV1, QB = D == 0 ? QB2 : QB1;  // across
  constexpr int FA = D == 0 ? M2 : M1, FD = D == 0 ? M1 : M2, FB = D == 0 ? B2 : B1;
  const HT* const q = reinterpret_cast<const HT*>(sm + L::Q) + r;
  HT rp, rm, mdp, mdm, map, mam;  // sums over the two cells of faces i, i-1: rho_t, m along, m across
  if constexpr (MIX) {
    if (BG) {
      const double* t = reinterpret_cast<const double*>(sm + L::RT) + r;
      rp = (HT)(t[0] + t[S]);
      rm = (HT)(t[-S] + t[0]);
    } else {
      rp = q[QR * QC] + q[QR * QC + S];
      rm = q[QR * QC - S] + q[QR * QC];
    }
    constexpr int MD = D == 0 ? QM1 : QM2, MA = D == 0 ? QM2 : QM1;
    mdp = q[MD * QC] + q[MD * QC + S];
    mdm = q[MD * QC - S] + q[MD * QC];
    map = q[MA * QC] + q[MA * QC + S];
    mam = q[MA * QC - S] + q[MA * QC];
  } else {
    const HT* t = BG ? reinterpret_cast<const HT*>(sm + L::RT) + r : q + QR * QC;
    constexpr int QD = D == 0 ? QV1 : QV2;
    const HT tm = t[-S], t0 = t[0], tp = t[S];
    rp = t0 + tp;
    rm = tm + t0;
    const HT md = mulr(q[QD * QC], t0), ma = mulr(q[QA * QC], t0);
    mdp = fma(q[QD * QC + S], tp, md);
    mdm = fma(q[QD * QC - S], tm, md);
    map = fma(q[QA * QC + S], tp, ma);
    mam = fma(q[QA * QC - S], tm, ma);
  }
  const HT va0 = q[QA * QC], b0 = q[QB * QC], bp = q[QB * QC + S], bm = q[QB * QC - S];
  const HT vp = p[2 * pn], vm = p[2 * pn - ps];
  const HT ap = mulr(p[3 * pn], q[QA * QC + S] - va0), am = mulr(p[3 * pn - ps], va0 - q[QA * QC - S]);
  const HT fp = mulr(p[4 * pn], bp - b0), fm = mulr(p[4 * pn - ps], b0 - bm);
  // the momentum pass along D counts twice (COMP == DIM); face means carry 1/2
  const double kd = 0.5 * k * chyp[FD], ka = 0.25 * k * chyp[FA], kb = k * chyp[FB];
  out[RHO] = fma(k * chyp[RHO], (double)(p[0] - p[-ps]), out[RHO]);
  out[FD] = fma(kd, (double)fma(vp, rp, -mulr(vm, rm)), out[FD]);
  out[FA] = fma(ka, (double)fma(ap, rp, -mulr(am, rm)), out[FA]);
  out[FB] = fma(kb, (double)(fp - fm), out[FB]);
  double e = fma(k * chyp[EN], (double)(p[pn] - p[pn - ps]), out[EN]);
  e = fma(kd, (double)fma(vp, mdp, -mulr(vm, mdm)), e);
  e = fma(ka, (double)fma(ap, map, -mulr(am, mam)), e);
  out[EN] = fma(0.5 * kb, (double)fma(fp, b0 + bp, -mulr(fm, bm + b0)), e);
}

// Cross arrays along D at region cell r (hyperdifmomsourcene2-4,
// hyperdifbsourcene1b-4): tau = (q+ - q-) (R + R-) cmax chyp / 8 of the
// momentum across D, t: / 4 of B; rho_t tau, t, and the energy's tau m_D - t
// B_D (two arrays in the mixed form, whose sums are double).  p: the ratios.
template <bool BG, bool MIX, bool O6, int D>
__device__ __forceinline__ void cross_at(const char* sm, const double* chyp, double cmax, bool zero, int r,
                                         const typename Form<MIX>::H* p, int pn, int ps,
                                         typename Form<MIX>::H* c, int cn) {
  using L = Lay<BG, MIX, O6>;
  using HT = typename L::H;
  constexpr int S = D == 0 ? 1 : QX;
  constexpr int QA = D == 0 ? QV2 : QV1, QB = D == 0 ? QB2 : QB1;
  const HT* const q = reinterpret_cast<const HT*>(sm + L::Q) + r;
  const HT kv = zero ? (HT)0 : (HT)(0.125 * cmax * chyp[D == 0 ? M2 : M1]);
  const HT kb = zero ? (HT)0 : (HT)(0.25 * cmax * chyp[D == 0 ? B2 : B1]);
  const HT tau = (q[QA * QC + S] - q[QA * QC - S]) * (p[3 * pn] + p[3 * pn - ps]) * kv;
  const HT t = (q[QB * QC + S] - q[QB * QC - S]) * (p[4 * pn] + p[4 * pn - ps]) * kb;
  const HT rt = BG ? (HT) reinterpret_cast<const double*>(sm + L::RT)[r] : q[QR * QC];
  const HT m = MIX ? q[(D == 0 ? QM1 : QM2) * QC] : q[(D == 0 ? QV1 : QV2) * QC] * rt;
  const HT b = q[(D == 0 ? QB1 : QB2) * QC];
  c[0] = rt * tau;
  c[cn] = t;
  if constexpr (MIX) {
    c[2 * cn] = tau * m;
    c[3 * cn] = t * b;
  } else {
    c[2 * cn] = fma(tau, m, -mulr(t, b));
  }
}
}  // namespace s2

// The base state and the accumulator of a tile row, which its last phase
// reads, into L2, a block's lifetime ahead of their use: lane k of the row
// takes field k of the twelve.
template <int MODE, bool MIX>
__device__ __forceinline__ void prefetch_row(const KBufs& B, long nc, int x0, int gj, int n0, int n1, int tx) {
  using ST = typename Form<MIX>::S;
  if (tx >= 12 || gj > n1 - 3) return;
  const bool base = tx < 6;
  if (base ? !(MODE == SMAUG_INT_EULER || B.stage < 3) : !(MODE != SMAUG_INT_EULER && B.stage > 0)) return;
  const long c = (base ? tx : tx - 6) * nc + (long)gj * n0;
  const int a = x0 < 2 ? 2 : x0, b = x0 + TX - 1 > n0 - 3 ? n0 - 3 : x0 + TX - 1;
#pragma unroll
  for (int k = 0; k < TX * 8 / 128 + 1; k++) {
    const int x = a + 16 * k < b ? a + 16 * k : b;
    const void* p = base ? static_cast<const void*>(static_cast<const ST*>(B.un) + c + x)
                         : static_cast<const void*>(B.acc + c + x);
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
  }
}

// Bulk tensor copy of the staged state of tile (bx, by) -- the 6 fields in
// the storage type into s, and (background fields) rho_b into gdst --
// completing on tt.bar.  Cells outside the grid read 0.  The region starts at
// column x0 - HALO = XORG - HALO + bx TX, which the TMA-staged kernel's tile
// origin makes a multiple of 32 cells (the copy's x offset must be 16-byte
// aligned).
template <bool BG, bool MIX>
__device__ __forceinline__ void tma_stage_issue(void* s, void* gdst, const TmaTile& tt, int bx, int by) {
  using ST = typename Form<MIX>::S;
  const unsigned bytes = 6 * RC * sizeof(ST) + (BG ? RC * sizeof(double) : 0);
  const int x = XORG - HALO + bx * TX, y = 2 - HALO + by * TY;
  fence_proxy_async_smem();
  mbar_expect_tx(tt.bar, bytes);
  tma_load_3d(s, tt.ms, x, y, 0, tt.bar);
  if (BG) tma_load_3d(gdst, tt.mg, x, y, 1, tt.bar);
}

// The stage for tile (bx, by) of one grid; the single-run kernels below and
// in stage2d_tma.cu and the batched kernel (batch_kernel.cuh) call it.  TMA:
// the state arrives by bulk tensor copy (tt: the block's copy schedule) in
// buffers ahead of the arrays above, and the copy of the block's next tile
// is issued as soon as this tile's values have been derived from them.
// Returns false when a copy did not complete in time (FLAG_TMA_TIMEOUT set;
// the block must stop).
template <int MODE, bool BG, bool MIX, bool O6 = false, bool CG = false, bool TMA = false>
__device__ __forceinline__ bool stage2d_body(const KParams& P, const KBufs& B, int bx, int by,
                                             const TmaTile* tt = nullptr) {
  using ST = typename Form<MIX>::S;
  using L = s2::Lay<BG, MIX, O6>;
  using HT = typename L::H;
  using s2::QC;
  using s2::QX;
  constexpr bool rk = MODE != SMAUG_INT_EULER;
  extern __shared__ double smem[];
  char* sm = reinterpret_cast<char*>(smem);
  ST* raw = nullptr;
  double* rawb = nullptr;
  if constexpr (TMA) {
    // the copy boxes land on 128-byte boundaries (the launch adds the slack);
    // an offset added to the shared array itself, so that the compiler still
    // addresses the tile arrays as shared memory
    sm += (128u - (smem_u32(sm) & 127u)) & 127u;
    raw = reinterpret_cast<ST*>(sm);
    rawb = reinterpret_cast<double*>(sm + 6 * RC * sizeof(ST));
    sm += 6 * RC * sizeof(ST) + (BG ? RC * sizeof(double) : 0);
  }
  double* const RD0 = reinterpret_cast<double*>(sm + L::RD);
  double* const RD1 = RD0 + RX;
  double* const F = reinterpret_cast<double*>(sm + L::U);
  HT* const RR = reinterpret_cast<HT*>(sm + L::U);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int x0 = XORG + bx * TX, y0 = 2 + by * TY;
  const int n0 = P.n0, n1 = P.n1;
  const long nc = P.ncell;
  const ST* const uin = static_cast<const ST*>(B.uin);
  const bool hyper = P.hyperdif == 1;
  // the region inside the grid: no source redirection in the staging
  const bool inner = x0 - HALO >= 0 && by >= 1 && x0 - HALO + RX <= n0 && y0 + TY + HALO <= n1;
  // running CFL maxima of the grid when the block starts
  double seen[2];
  __shared__ unsigned long long red[2];
  __shared__ int arrived;
  {
    const unsigned long long* cm = B.cmax_out;
    seen[0] = __longlong_as_double(__ldcg(cm));
    seen[1] = __longlong_as_double(__ldcg(cm + 1));
  }

  // ---- phase 0: staging ----------------------------------------------------
  // Source cell of a region cell: the cell itself; index -1 along an axis the
  // copy of index 5 (bc_hyperdifl); index n the stray store's source
  // (B.padsrc); -1 for the rest (zeros).
  auto source = [&](int gi, int gj) -> int {
    const bool ix = gi >= 0 && gi < n0, iy = gj >= 0 && gj < n1;
    if (ix && iy) return gj * n0 + gi;
    if (iy) return gi == -1 ? gj * n0 + 5 : (gi == n0 ? B.padsrc[0][gj] : -1);
    if (ix) return gj == -1 ? 5 * n0 + gi : (gj == n1 ? B.padsrc[1][gi] : -1);
    return -1;
  };
  if constexpr (TMA) {
    // every thread waits on the barrier
    if (tt->issue_self && tid == 0) tma_stage_issue<BG, MIX>(raw, rawb, *tt, bx, by);
    const bool ok = mbar_wait(tt->bar, tt->parity, TMA_WAIT_NS);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        atomicOr(B.flags, FLAG_TMA_TIMEOUT);
        mbar_wait(tt->bar, tt->parity, TMA_WAIT_NS);  // the copy in flight
      }
      __syncthreads();
      return false;
    }
  }
  {
    // all loads of a thread's region cells first, then their use
    constexpr int NI = (RX * RY + NTHREADS - 1) / NTHREADS;
    ST w[NI][6];
    double rhob[NI];
    int c[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int u = tid + i * NTHREADS;
      const int lx = u % RX, ly = u / RX;
      const int gi = x0 - HALO + lx, gj = y0 - HALO + ly;
      const bool in = inner || (gi >= 0 && gi < n0 && gj >= 0 && gj < n1);
      c[i] = u >= RX * RY ? -1 : in ? gj * n0 + gi : source(gi, gj);
      rhob[i] = 0.0;
      if (TMA && in && u < RX * RY) {
#pragma unroll
        for (int f = 0; f < 6; f++) w[i][f] = raw[f * RC + u];
        if (BG) rhob[i] = rawb[u];
      } else {
#pragma unroll
        for (int f = 0; f < 6; f++) w[i][f] = c[i] >= 0 ? ldin<CG>(uin + f * nc + c[i]) : (ST)0;
        if (BG) rhob[i] = c[i] >= 0 ? __ldg(B.bg + nc + c[i]) : 0.0;
      }
    }
    prefetch_row<MODE, MIX>(B, nc, x0, y0 + ty, n0, n1, tx);
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int u = tid + i * NTHREADS;
      if (u < RX * RY) s2::derive<BG, MIX, O6>(sm, u / RX * QX + u % RX, c[i] >= 0, w[i], rhob[i]);
    }
  }
  for (int r = tid; r < RX + RY; r += NTHREADS) {
    const int d = r < RX ? 0 : 1, g = d == 0 ? x0 - HALO + r : y0 - HALO + (r - RX);
    RD0[r] = (g >= 0 && g < (d == 0 ? n0 : n1)) ? 1.0 / B.delx[d][g] : 1.0;
  }

  // ---- dt of this step and stage time ----------------------------------
  const double cin[2] = {ldsc<CG>(B.cmax_in), ldsc<CG>(B.cmax_in + 1)};
  double dt, tstage;
  {
    const bool first = bx == 0 && by == 0 && tid == 0;
    if (B.stage == 0) {
      dt = device_dt(P, cin, ldsc<CG>(B.dt_prev), 2);
      tstage = ldsc<CG>(B.t_prev);
      if (first) {
        *B.dt_new = dt;
        *B.t_new = tstage + dt;
      }
    } else {
      dt = ldsc<CG>(B.dt_new);
      tstage = ldsc<CG>(B.t_prev) + (B.stage == 3 ? dt : 0.5 * dt);
    }
    if (first) B.cmax_clear[0] = B.cmax_clear[1] = B.cmax_clear[2] = 0ull;
  }
  __syncthreads();
  if (tid == 0) {
    // after the barrier: every warp is done with the block's previous tile
    red[0] = red[1] = 0ull;
    arrived = 0;
  }
  if constexpr (TMA) {
    if (tid == 0 && tt->nbx >= 0) tma_stage_issue<BG, MIX>(raw, rawb, *tt, tt->nbx, tt->nby);
  }

  const int lxo = tx + HALO, lyo = ty + HALO, ro = lyo * QX + lxo;
  const int gi = x0 + tx, gj = y0 + ty;
  const bool active = (XORG >= 2 || gi >= 2) && gi <= n0 - 3 && gj <= n1 - 3;
  const long co = active ? (long)gj * n0 + gi : 0;
  double gb[4] = {0, 0, 0, 0};  // background fields at the tile cell

  // ---- phase 1: centred fluxes: both directions at the own cell, then the
  // cells beside the tile, one direction each -------------------------------
  auto back = [&](int lx, int ly, double* g) {
    const int ci = x0 - HALO + lx, cj = y0 - HALO + ly;
    if (inner || (ci >= 0 && ci < n0 && cj >= 0 && cj < n1)) {
      const long c = (long)cj * n0 + ci;
      g[0] = __ldg(B.bg + c);
      g[2] = __ldg(B.bg + 2 * nc + c);
      g[3] = __ldg(B.bg + 3 * nc + c);
    }
  };
  if (BG) {
    back(lxo, lyo, gb);
    if (active) gb[1] = __ldg(B.bg + nc + co);
  }
  s2::flux_at<BG, MIX, O6, true, true>(sm, P.gamma, ro, gb, F + ty * L::FXW + tx + L::FH, L::FXN,
                                       F + 5 * L::FXN + (ty + 2) * TX + tx, L::FYN);
  constexpr int NHY = 4 * TX, NHX = 2 * L::FH * TY;
  for (int u = tid; u < NHY + NHX; u += NTHREADS) {
    double g[4] = {0, 0, 0, 0};
    if (u < NHY) {
      const int row = u / TX, fr = row < 2 ? row : row + TY, col = u % TX;  // flux row 0, 1, TY+2, TY+3
      if (BG) back(HALO + col, HALO - 2 + fr, g);
      s2::flux_at<BG, MIX, O6, false, true>(sm, P.gamma, (HALO - 2 + fr) * QX + HALO + col, g, nullptr, 0,
                                            F + 5 * L::FXN + fr * TX + col, L::FYN);
    } else {
      const int v = u - NHY, c = v % (2 * L::FH), fc = c < L::FH ? c : c + TX, row = v / (2 * L::FH);
      if (BG) back(HALO - L::FH + fc, HALO + row, g);
      s2::flux_at<BG, MIX, O6, true, false>(sm, P.gamma, (HALO + row) * QX + HALO - L::FH + fc, g,
                                            F + row * L::FXW + fc, L::FXN, nullptr, 0);
    }
  }
  __syncthreads();

  // ---- phase 2: divergence at the own cell --------------------------------
  const HT* const qo = reinterpret_cast<const HT*>(sm + L::Q) + ro;
  const double rd0 = RD0[lxo], rd1 = RD1[lyo];
  const bool z0 = (P.bt[0] != 0) && zero1n(gi, n0), z1 = (P.bt[1] != 0) && zero1n(gj, n1);
  double out[6];
  {
    const double kx = ((P.bt[0] != 0) && zero3dn(gi, n0)) || (O6 && edge6(gi, n0)) ? 0.0
                                                                                  : dt * rd0 * (O6 ? 0.25 : 1.0 / 12.0);
    const double ky = (P.bt[1] != 0) && zero3dn(gj, n1) ? 0.0 : dt * rd1 * (1.0 / 12.0);
    // 12 h times the 4th-order derivative; 4 h times the 6th-order one
    auto dx = [&](auto a) -> double {
      const double u1 = (double)a(1) - (double)a(-1), u2 = (double)a(-2) - (double)a(2);
      if constexpr (O6) return fma(3.0, u1, fma(0.6, u2, mulr((double)a(3) - (double)a(-3), 1.0 / 15.0)));
      return fma(8.0, u1, u2);
    };
    auto dy = [&](auto a) -> double {
      return fma(8.0, (double)a(1) - (double)a(-1), (double)a(-2) - (double)a(2));
    };
    const double* const fx = F + ty * L::FXW + tx + L::FH;
    const double* const fy = F + 5 * L::FXN + (ty + 2) * TX + tx;
    auto ddx = [&](int k) { return dx([&](int s) { return fx[k * L::FXN + s]; }); };
    auto ddy = [&](int k) { return dy([&](int s) { return fy[k * L::FYN + s * TX]; }); };
    out[RHO] = fma(-ky, ddy(0), -mulr(kx, ddx(0)));
    out[M1] = fma(-ky, ddy(1), -mulr(kx, ddx(1)));
    out[M2] = fma(-ky, ddy(2), -mulr(kx, ddx(2)));
    out[EN] = fma(-ky, ddy(3), -mulr(kx, ddx(3)));
    out[B2] = -mulr(kx, ddx(4));
    out[B1] = -mulr(ky, ddy(4));
    if (BG) {
      // addenergyterms_cd2 (src/centdiff2.cu:80-115)
      auto vel = [&](int c, int s) -> double {
        if constexpr (MIX)
          return mulr((double)qo[(s2::QM1 + c) * QC + s], reinterpret_cast<const double*>(sm + L::RI)[ro + s]);
        else
          return (double)qo[(s2::QV1 + c) * QC + s];
      };
      const double v1x = mulr(kx, dx([&](int s) { return vel(0, s); }));
      const double v2x = mulr(kx, dx([&](int s) { return vel(1, s); }));
      const double v1y = mulr(ky, dy([&](int s) { return vel(0, s * QX); }));
      const double v2y = mulr(ky, dy([&](int s) { return vel(1, s * QX); }));
      const double ptb =
          fma(P.gamma - 1, gb[0], -mulr(0.5 * (P.gamma - 2), fma(gb[2], gb[2], mulr(gb[3], gb[3]))));
      out[EN] = fma(-ptb, v1x + v2y, out[EN]);
      out[EN] = fma(gb[2], fma(gb[2], v1x, mulr(gb[3], v2x)), out[EN]);
      out[EN] = fma(gb[3], fma(gb[2], v1y, mulr(gb[3], v2y)), out[EN]);
    }
    if (P.has_grav) {
      // addgrav_cd2 (src/centdiff2.cu:118-154); m rho / rho_t = v rho
      const double rho = (double)qo[s2::QR * QC];
      double v1, v2;
      if constexpr (MIX) {
        const double ri = reinterpret_cast<const double*>(sm + L::RI)[ro];
        v1 = mulr((double)qo[s2::QM1 * QC], ri);
        v2 = mulr((double)qo[s2::QM2 * QC], ri);
      } else {
        v1 = (double)qo[s2::QV1 * QC];
        v2 = (double)qo[s2::QV2 * QC];
      }
      out[M1] = fma(dt * P.g[0], rho, out[M1]);
      out[M2] = fma(dt * P.g[1], rho, out[M2]);
      out[EN] = fma(dt * fma(P.g[0], v1, mulr(P.g[1], v2)), rho, out[EN]);
    }
  }

  // base state and accumulator of the own cell, all loaded before the first
  // store (a load after a store to the accumulator would wait for its own
  // round trip) and before the last phase's arithmetic
  double ub[6], ac[6];
  auto load_base = [&] {
    if (!active) return;
    if (!rk || B.stage < 3) {
#pragma unroll
      for (int f = 0; f < 6; f++) ub[f] = base_value<MIX, CG>(B, f * nc + co);
    }
    if (rk && B.stage > 0) {
#pragma unroll
      for (int f = 0; f < 6; f++) ac[f] = ldsc<CG>(B.acc + f * nc + co);
    }
  };
  if (!hyper) {
    load_base();
  } else {
    __syncthreads();
    // ---- phase 3: nu ratios ------------------------------------------------
    // pieces of rows: 11 faces (three to a 32-cell row), 9 for a 16-cell one
    constexpr int NS = (TX + 11) / 11, SL = (TX + NS) / NS;
    constexpr int NXT = (3 * TY + 2 * (TY + 2)) * NS, NYT = 3 * TX + 2 * (TX + 2);
    for (int u = tid; u < NXT + NYT; u += NTHREADS) {
      if (u < NXT) {
        // rows of rho, e, v1 on the tile, of v2, b2 one more on each side
        const int s = u % NS, v = u / NS;
        const bool cr = v >= 3 * TY;
        const int k = cr ? 3 + (v - 3 * TY) / (TY + 2) : v / TY;
        const int row = cr ? (v - 3 * TY) % (TY + 2) : 1 + v % TY;  // 0 .. TY+1
        const int fld = k == 0 ? s2::QR : k == 1 ? s2::QE : k == 2 ? s2::QV1 : k == 3 ? s2::QV2 : s2::QB2;
        const int f0 = s * SL, n = TX + 1 - f0 < SL ? TX + 1 - f0 : SL;
        const HT* q = reinterpret_cast<const HT*>(sm + L::Q) + fld * QC + (row + HALO - 1) * QX + HALO - 1 + f0;
        HT* o = RR + k * L::RXN + row * L::RXW + f0;
        ratio_line<SL, 1, (TX + 1) % SL == 0>(q, n, [&](int i, HT r, HT dq) { o[i] = cr ? r : r * dq; });
      } else {
        // columns of rho, e, v2 on the tile, of v1, b1 one more on each side
        const int v = u - NXT;
        const bool cr = v >= 3 * TX;
        const int k = cr ? 3 + (v - 3 * TX) / (TX + 2) : v / TX;
        const int col = cr ? (v - 3 * TX) % (TX + 2) : 1 + v % TX;  // 0 .. TX+1
        const int fld = k == 0 ? s2::QR : k == 1 ? s2::QE : k == 2 ? s2::QV2 : k == 3 ? s2::QV1 : s2::QB1;
        const HT* q = reinterpret_cast<const HT*>(sm + L::Q) + fld * QC + (HALO - 1) * QX + col + HALO - 1;
        HT* o = RR + 5 * L::RXN + k * L::RYN + col;
        ratio_line<TY + 1, QX, true>(q, TY + 1, [&](int i, HT r, HT dq) { o[i * L::RYW] = cr ? r : r * dq; });
      }
    }
    __syncthreads();
    // ---- phase 4: diffusive terms; cross arrays (zero outside [2, n-3] and
    // next to the edges) of the own cell and of the cells beside the tile ------
    HT* const CX = RR + 5 * (L::RXN + L::RYN);
    HT* const CY = CX + L::NC * L::CXN;
    const HT* const px = RR + (ty + 1) * L::RXW + tx + 1;
    const HT* const py = RR + 5 * L::RXN + (ty + 1) * L::RYW + tx + 1;
    s2::diffuse<BG, MIX, O6, 0>(sm, P.chyp, ro, z0 ? 0.0 : dt * cin[0] * rd0, px, L::RXN, 1, out);
    s2::cross_at<BG, MIX, O6, 0>(sm, P.chyp, cin[0], z0 || !active, ro, px, L::RXN, 1, CX + (ty + 1) * TX + tx,
                                 L::CXN);
    s2::diffuse<BG, MIX, O6, 1>(sm, P.chyp, ro, z1 ? 0.0 : dt * cin[1] * rd1, py, L::RYN, L::RYW, out);
    s2::cross_at<BG, MIX, O6, 1>(sm, P.chyp, cin[1], z1 || !active, ro, py, L::RYN, L::RYW,
                                 CY + ty * L::CYW + tx + 1, L::CYN);
    for (int u = tid; u < 2 * TX + 2 * TY; u += NTHREADS) {
      const bool xd = u < 2 * TX;
      // tile cell + 1: rows 0 and TY+1 of the x passes, columns 0 and TX+1 of the y passes
      const int v = u - 2 * TX;
      const int cx = xd ? u % TX + 1 : (v & 1) * (TX + 1), cy = xd ? u / TX * (TY + 1) : v / 2 + 1;
      const int ci = x0 - 1 + cx, cj = y0 - 1 + cy;
      const int r = (cy + HALO - 1) * QX + cx + HALO - 1;
      const bool out2 = ci < 2 || ci > n0 - 3 || cj < 2 || cj > n1 - 3;
      if (xd)
        s2::cross_at<BG, MIX, O6, 0>(sm, P.chyp, cin[0], out2 || ((P.bt[0] != 0) && zero1n(ci, n0)), r,
                                     RR + cy * L::RXW + cx, L::RXN, 1, CX + cy * TX + cx - 1, L::CXN);
      else
        s2::cross_at<BG, MIX, O6, 1>(sm, P.chyp, cin[1], out2 || ((P.bt[1] != 0) && zero1n(cj, n1)), r,
                                     RR + 5 * L::RXN + cy * L::RYW + cx, L::RYN, L::RYW,
                                     CY + (cy - 1) * L::CYW + cx, L::CYN);
    }
    load_base();
    __syncthreads();
    // ---- phase 5: cross terms --------------------------------------------------
    {
      // d/dy of the x passes' arrays, d/dx of the y passes'
      const double ky = z1 ? 0.0 : 0.5 * dt * rd1, kx = z0 ? 0.0 : 0.5 * dt * rd0;
      const HT* const c = CX + (ty + 1) * TX + tx;
      auto dc = [&](int k) -> double { return (double)(c[k * L::CXN + TX] - c[k * L::CXN - TX]); };
      out[M1] = fma(ky, dc(0), out[M1]);
      out[B1] = fma(-ky, dc(1), out[B1]);
      out[EN] = fma(ky, dc(2), out[EN]);
      if constexpr (MIX) out[EN] = fma(-ky, dc(3), out[EN]);
      const HT* const d = CY + ty * L::CYW + tx + 1;
      auto dd = [&](int k) -> double { return (double)(d[k * L::CYN + 1] - d[k * L::CYN - 1]); };
      out[M2] = fma(kx, dd(0), out[M2]);
      out[B2] = fma(-kx, dd(1), out[B2]);
      out[EN] = fma(kx, dd(2), out[EN]);
      if constexpr (MIX) out[EN] = fma(-kx, dd(3), out[EN]);
    }
  }

  // ---- driver, stage sum, stores, ghost images, CFL maxima ------------------
  double cm[2] = {seen[0], seen[1]};
  if (P.cmax_floor[0] > cm[0]) cm[0] = P.cmax_floor[0];
  if (P.cmax_floor[1] > cm[1]) cm[1] = P.cmax_floor[1];
  if (active) {
    double res[6];
    const bool is_base = !rk || B.stage == 3;
    const double wgt = (B.stage == 0 || B.stage == 3) ? 1.0 / 6.0 : 1.0 / 3.0;
    const double cst = (B.stage == 2) ? 1.0 : 0.5;
    if (P.driver == SMAUG_DRIVER_GAUSS) {
      // source_parallel + addsourceterms2
      double v = P.drv_amp;
      if (P.drv_period > 0) v *= sin(tstage * 2.0 * M_PI / P.drv_period);
      if (P.drv_sigma[0] > 0) {
        const double x = B.pos[0][gi] - P.drv_x0[0];
        v *= exp(-x * x / (P.drv_sigma[0] * P.drv_sigma[0]));
      }
      if (P.drv_sigma[1] > 0) {
        const double x = B.pos[1][gj] - P.drv_x0[1];
        v *= exp(-x * x / (P.drv_sigma[1] * P.drv_sigma[1]));
      }
      const double rr = rk ? (double)qo[s2::QR * QC] : ub[RHO] + out[RHO];
      out[M1] = fma(dt * v, rr + gb[1], out[M1]);
    }
#pragma unroll
    for (int f = 0; f < 6; f++) {
      if (!rk) {
        res[f] = ub[f] + out[f];
      } else if (B.stage == 3) {
        res[f] = fma(wgt, out[f], ac[f]);
      } else {
        B.acc[f * nc + co] = fma(wgt, out[f], B.stage == 0 ? ub[f] : ac[f]);
        res[f] = fma(cst, out[f], ub[f]);
      }
    }
    int hmax = 0;  // largest exponent word: infinities and NaN have 0x7ff
#pragma unroll
    for (int f = 0; f < 6; f++) hmax = max(hmax, __double2hiint(res[f]) & 0x7fffffff);
    if (hmax >= 0x7ff00000) atomicOr(B.flags, 1);
    auto speeds = [&](const double* g) {
      if (may_exceed<2, BG>(P.gamma, res, g, cm)) {
        const double2 c =
            cfast2_call(P.gamma, res[RHO], res[M1], res[M2], res[EN], res[B1], res[B2], g[0], g[1], g[2], g[3]);
        cm[0] = dmax0(cm[0], c.x);
        cm[1] = dmax0(cm[1], c.y);
      }
    };
#pragma unroll
    for (int f = 0; f < 6; f++) store_value<MIX>(B, f * nc + co, res[f], is_base);
    speeds(gb);
    // tiles that hold cells within 4 of an end of the interior have images
    if (x0 < 6 || y0 < 6 || x0 + TX > n0 - 6 || y0 + TY > n1 - 6) {
      int ix[3], iy[3];
      ix[0] = gi;
      iy[0] = gj;
      const int nx = 1 + ghost_images(gi, n0, P.bc[0], ix + 1);
      const int ny = 1 + ghost_images(gj, n1, P.bc[1], iy + 1);
      bool negated = false;  // res holds the negated values
      for (int b = 0; b < ny; b++)
        for (int a = b == 0 ? 1 : 0; a < nx; a++) {
          const long cc = (long)iy[b] * n0 + ix[a];
          // antisymmetric images carry the opposite sign (negation is exact)
          const bool neg = ((a > 0) && P.gneg[0]) != ((b > 0) && P.gneg[1]);
          if (neg != negated) {
#pragma unroll
            for (int f = 0; f < 6; f++) res[f] = -res[f];
            negated = neg;
          }
#pragma unroll
          for (int f = 0; f < 6; f++) store_value<MIX>(B, f * nc + cc, res[f], is_base);
          // without background fields an image has its source's fast speeds
          // unless its sign changed
          if (BG || neg) {
            double g[4] = {0, 0, 0, 0};
            if (BG) {
#pragma unroll
              for (int f = 0; f < 4; f++) g[f] = __ldg(B.bg + f * nc + cc);
            }
            speeds(g);
          }
        }
    }
  }
  // Maxima of the block, without a barrier: every warp adds its own to a shared
  // pair, and the last one hands the pair on if it exceeds what the grid had
  // when the block started.
  if (__any_sync(0xffffffffu, cm[0] > seen[0] || cm[1] > seen[1])) {
#pragma unroll
    for (int d = 0; d < 2; d++) {
      for (int o = 16; o > 0; o >>= 1) cm[d] = dmax0(cm[d], __shfl_xor_sync(0xffffffffu, cm[d], o));
      if ((tid & 31) == 0) atomicMax(&red[d], (unsigned long long)__double_as_longlong(cm[d]));
    }
  }
  if ((tid & 31) == 0) {
    __threadfence_block();
    if (atomicAdd(&arrived, 1) == NTHREADS / 32 - 1) {
#pragma unroll
      for (int d = 0; d < 2; d++) {
        const unsigned long long m = atomicMax(&red[d], 0ull);
        if (__longlong_as_double(m) > seen[d]) atomicMax(&B.cmax_out[d], m);
      }
    }
  }
  return true;
}

template <int MODE, bool BG, bool MIX, bool O6>
__global__ void __launch_bounds__(NTHREADS, MIX ? SMAUG_MINB2D_MIX : SMAUG_MINB2D)
    stage2d_fast(const KParams P, const KBufs B) {
  stage2d_body<MODE, BG, MIX, O6>(P, B, blockIdx.x, blockIdx.y);
}

// launch helper: picks the background and stencil-order specialisations
template <int MODE, bool MIX, bool O6>
static cudaError_t launch_stage2d_o(const KParams& K, const KBufs& B, cudaStream_t st) {
  dim3 block(TX, TY);
  dim3 grid((K.n0 - 4 + TX - 1) / TX, (K.n1 - 4 + TY - 1) / TY);
  if (K.has_bg) {
    stage2d_fast<MODE, true, MIX, O6><<<grid, block, s2::smem_bytes<true, MIX, O6>(), st>>>(K, B);
  } else {
    stage2d_fast<MODE, false, MIX, O6><<<grid, block, s2::smem_bytes<false, MIX, O6>(), st>>>(K, B);
  }
  return cudaGetLastError();
}
template <int MODE, bool MIX>
static cudaError_t launch_stage2d(const KParams& K, const KBufs& B, cudaStream_t st) {
  return K.order6 ? launch_stage2d_o<MODE, MIX, true>(K, B, st) : launch_stage2d_o<MODE, MIX, false>(K, B, st);
}

template <int MODE, bool BG, bool MIX, bool O6>
static cudaError_t stage2d_attr() {
  return cudaFuncSetAttribute(stage2d_fast<MODE, BG, MIX, O6>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)s2::smem_bytes<BG, MIX, O6>());
}
