// stage3d.cuh -- fused 3D stage kernel, included by stage3d.cu.
//
// One launch evaluates the reference's whole spatial operator (the 3D build,
// -DUSE_SAC_3D, of src/iosmaug.c:631-835) for an 8x8x8 tile of interior
// cells and writes the stage result, its ghost images and the per-dimension
// fast-speed maxima.  The terms and their arithmetic are those of the 2D
// kernel (stage2d.cuh) with three momentum and field components:
//   fluxes along each dimension and their 4th-order divergence
//     (src/centdiff1.cu:51-197, src/centdiff2.cu:203-323, grad3dn)
//   background energy coupling e -= dt p_tb dv_d/dx_d,
//     e += dt Bb_i Bb_d dv_d/dx_i (src/centdiff2.cu:80-115); the second sum
//     is evaluated in the pass of the derivative's direction i
//   gravity (src/centdiff2.cu:118-154)
//   hyperdiffusion of rho, e, m_c, B_c along every dimension
//     (src/hyperdifvisc1{r,l}.cu, src/hyperdif*source*.cu); the passes of
//     one field share one staging of q
//   user driver, stage combine, ghost images, CFL maxima.
// Sums per cell are reordered against the reference (per field instead of
// per dimension); agreement stays at rounding level.  The mixed precision
// form (template MIX) is the one of stage2d.cuh: float perturbation storage
// and hyperdiffusion arithmetic, double everywhere else.
//
// The state is read from global memory (L1/L2 resident across the phases of
// a block).  Shared memory holds 1/rho_t on the tile's 3-cell box, rho_t on the
// tile +-1, the per-axis metric, the box cells' sources, and one union of phase
// scratch:
//   flux phase:  7 flux arrays + 3 velocity arrays on the tile +-2 along the
//                direction
//   hyperdiffusion, field by field: q on the box, the nu ratios of the field's
//                passes (tile +-1 along the field's component only, which is
//                where its cross terms are differentiated), three cross arrays
// Bound by loads of the state from L2 and the barriers between the phases: 235
// warp instructions per cell and stage at 35 % issue (494 at 48 % with 8x8x4
// tiles and every pass on its own).  RK4 per step at 256^3 then and now: FP64
// 61.1 and 37.5 ms, mixed 54 and 38.  Other tiles now: 16x8x4 40.5, 8x8x4 45.8.
//
// A field takes three block barriers: q staged | ratios of all directions, one
// thread per piece of a line (ratio_line) | diffusive terms and cross arrays |
// cross terms beside the staging of the next field.
#pragma once

// (included inside namespace smaug)
namespace s3 {
#ifndef SMAUG_T3X
#define SMAUG_T3X 8
#endif
#ifndef SMAUG_T3Y
#define SMAUG_T3Y 8
#endif
#ifndef SMAUG_T3Z
#define SMAUG_T3Z 8
#endif
#ifndef SMAUG_MINB3D
#define SMAUG_MINB3D 2  // resident blocks per SM the 3D stage is compiled for
#endif
#ifndef SMAUG_NB3
#define SMAUG_NB3 3  // box cells of a thread whose loads are issued together
#endif
constexpr int T0 = SMAUG_T3X, T1 = SMAUG_T3Y, T2 = SMAUG_T3Z;  // tile (x fastest)
constexpr int NT = T0 * T1 * T2;       // threads per block, one cell each
constexpr int H = 3;                   // box halo
constexpr int BX = T0 + 2 * H, BY = T1 + 2 * H, BZ = T2 + 2 * H;
// row pitch of the box arrays: odd, so that lines along x taken by
// neighbouring threads fall on different banks
constexpr int BP = BX | 1;
constexpr int BC = BP * BY * BZ;
constexpr int BS1 = BP, BS2 = BP * BY;  // box strides
__host__ __device__ constexpr int max3(int a, int b, int c) {
  return a > b ? (a > c ? a : c) : (b > c ? b : c);
}
// flux arrays: the tile +-2 (+-3 for the 6th-order derivative) along the direction
template <bool O6>
__host__ __device__ constexpr int fa() {
  return max3((T0 + (O6 ? 6 : 4)) * T1 * T2, T0 * (T1 + (O6 ? 6 : 4)) * T2, T0 * T1 * (T2 + (O6 ? 6 : 4)));
}
// tile +-1 (rho_t), strides
constexpr int EX = T0 + 2, EY = T1 + 2, EZ = T2 + 2, EC = EX * EY * EZ;
// ratio areas: faces -1 .. T-1 along the direction, the tile across, one cell
// more on each side along the field's component; cross arrays: the tile +-1
// along the component
constexpr int RA = max3((T0 + 1) * (T1 + 2) * T2, (T0 + 1) * T1 * (T2 + 2),
                        max3((T0 + 2) * (T1 + 1) * T2, T0 * (T1 + 1) * (T2 + 2),
                             max3((T0 + 2) * T1 * (T2 + 1), T0 * (T1 + 2) * (T2 + 1), 0)));
constexpr int CA = max3((T0 + 2) * T1 * T2, T0 * (T1 + 2) * T2, T0 * T1 * (T2 + 2));
constexpr int NMET = BX + BY + BZ;
// cross arrays of one field: the two passes' momentum (or B) arrays and the
// energy's, summed over the passes in double (the mixed form keeps both float
// parts)
template <bool MIX>
__host__ __device__ constexpr int nca() { return MIX ? 4 : 3; }
template <bool MIX, bool O6 = false>
__host__ __device__ constexpr size_t union_bytes() {
  constexpr size_t h = ((MIX ? 2 : 1) * BC + 3 * RA + nca<MIX>() * CA) * sizeof(typename Form<MIX>::H);
  constexpr size_t f = 10 * fa<O6>() * sizeof(double);
  return ((f > h ? f : h) + 7) / 8 * 8;
}
template <bool MIX, bool O6 = false>
__host__ __device__ constexpr size_t smem_bytes() {
  return sizeof(double) * (BC + EC + NMET) + union_bytes<MIX, O6>() + sizeof(int) * BC;
}
__host__ __device__ constexpr int tdim(int d) { return d == 0 ? T0 : (d == 1 ? T1 : T2); }
__host__ __device__ constexpr int bstride(int d) { return d == 0 ? 1 : (d == 1 ? BS1 : BS2); }
}  // namespace s3

struct Box3 {
  double* R;       // [BC] 1/rho_t on the box
  double* T;       // [EC] rho_t on the tile +-1
  double* rd[3];   // 1/dl over the box extent of each axis
  void* U;         // union scratch
  int* C;          // [BC] q source code per box cell (box_code)
  int o[3];        // global coordinate of box index 0 per axis
  bool inner;      // the box lies inside the grid and off its pads
};
// index into Box3::T of box cell (lx, ly, lz)
__device__ __forceinline__ int eidx(int lx, int ly, int lz) {
  return ((lz - s3::H + 1) * s3::EY + (ly - s3::H + 1)) * s3::EX + (lx - s3::H + 1);
}

// q of a hyperdiffusion field from global memory (src/hyperdifvisc1r.cu:1225-1253)
template <typename ST, int KIND, int COMP>
__device__ __forceinline__ double hq3_global(const ST* u, const KBufs& B, long nc, long c) {
  const double rho = __ldg(u + c);
  if (KIND == 0) return rho;
  if (KIND == 3) return __ldg(u + (B3 + COMP) * nc + c);
  const double r = recip(rho + __ldg(B.bg + GRB * nc + c));
  if (KIND == 2) return (double)__ldg(u + (M3 + COMP) * nc + c) * r;
  double m2 = 0, b2 = 0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double m = __ldg(u + (M3 + a) * nc + c), b = __ldg(u + (B3 + a) * nc + c);
    m2 += m * m;
    b2 += b * b;
  }
  return (double)__ldg(u + E3 * nc + c) - 0.5 * (b2 + m2 * r);
}

// distance of box index l outside the tile range [H, H+T)
__device__ __forceinline__ int outside(int l, int T) {
  return l < s3::H ? s3::H - l : (l >= s3::H + T ? l - (s3::H + T - 1) : 0);
}

// (A) q of one field on the box: every cell within 1 of the tile on all
// axes but one, and within 3 on that one.  Pads: index -1 along an axis is
// the copy of index 5 (bc_hyperdifl), index n the stray tmp6 store of
// hyperdifvisc1r_parallel (source table B.padsrc).
template <bool MIX, int KIND, int COMP>
__device__ __forceinline__ void stage_q(const Box3& X, const KParams& P, const KBufs& B, int tid) {
  using HT = typename Form<MIX>::H;
  using ST = typename Form<MIX>::S;
  const ST* u = static_cast<const ST*>(B.uin);
  HT* Q = static_cast<HT*>(X.U);
  const long nc = P.ncell;
  // a thread's cells in groups whose loads are all issued before their use; six
  // at once (a whole thread) spill at 64 registers: 47.1 against 37.5 ms per RK4
  // step at 256^3
  constexpr int NI = (s3::BC + s3::NT - 1) / s3::NT, NB = KIND == 1 ? 1 : SMAUG_NB3, NF = KIND == 1 ? 7 : 1;
  constexpr int F0 = KIND == 0 ? R3 : KIND == 1 ? M3 : KIND == 2 ? M3 + COMP : B3 + COMP;
#pragma unroll 1
  for (int i0 = 0; i0 < NI; i0 += NB) {
    int code[NB];
    ST w[NB][NF];
#pragma unroll
    for (int i = 0; i < NB; i++) {
      const int r = tid + (i0 + i) * s3::NT;
      code[i] = r < s3::BC ? X.C[r] : -1;
#pragma unroll
      for (int f = 0; f < NF; f++) w[i][f] = code[i] >= 0 ? __ldg(u + (F0 + f) * nc + code[i]) : (ST)0;
    }
#pragma unroll
    for (int i = 0; i < NB; i++) {
      const int r = tid + (i0 + i) * s3::NT;
      if (r >= s3::BC) continue;
      double q = (double)w[i][0];
      if (KIND == 2) q = mulr(q, X.R[r]);
      if (KIND == 1) {
        // m1 m2 m3 e b1 b2 b3
        double m2 = 0, b2 = 0;
#pragma unroll
        for (int a = 0; a < 3; a++) {
          const double m = (double)w[i][a], b = (double)w[i][NF - 3 + a];
          m2 = fma(m, m, m2);
          b2 = fma(b, b, b2);
        }
        q = fma(-0.5, fma(m2, X.R[r], b2), (double)w[i][NF / 2]);
      }
      if (code[i] <= -2) q = hq3_global<ST, KIND, COMP>(u, B, nc, (long)(-2 - code[i]));
      Q[r] = (HT)q;
      if (MIX && KIND == 2) Q[s3::BC + r] = (HT)w[i][0];
    }
  }
}

// Source code of box cell r for the q stagings (computed once per block):
// the cell index when the cell is in the grid and read by some pass, -2 - src
// for a pad (index -1 along an axis: the cell with that coordinate 5,
// bc_hyperdifl; index n: the stray tmp6 store of hyperdifvisc1r_parallel,
// source table B.padsrc), -1 for a zero.  The passes read the cells within 1
// of the tile on all axes but one and within 3 on that one.
__device__ __forceinline__ int box_code(const Box3& X, const KParams& P, const KBufs& B, int lx, int ly,
                                        int lz) {
  const int ox = outside(lx, s3::T0), oy = outside(ly, s3::T1), oz = outside(lz, s3::T2);
  if ((ox > 1) + (oy > 1) + (oz > 1) > 1) return -1;
  const int n0 = P.n0, n1 = P.n1, n2 = P.n2;
  const int g0 = X.o[0] + lx, g1 = X.o[1] + ly, g2 = X.o[2] + lz;
  const bool i0 = g0 >= 0 && g0 < n0, i1 = g1 >= 0 && g1 < n1, i2 = g2 >= 0 && g2 < n2;
  if (i0 && i1 && i2) return (int)(((long)g2 * n1 + g1) * n0 + g0);
  int src = -1;
  if (!i0 && i1 && i2) {
    if (g0 == -1) src = (int)(((long)g2 * n1 + g1) * n0 + 5);
    else if (g0 == n0) src = B.padsrc[0][(long)g2 * n1 + g1];
  } else if (i0 && !i1 && i2) {
    if (g1 == -1) src = (int)(((long)g2 * n1 + 5) * n0 + g0);
    else if (g1 == n1) src = B.padsrc[1][(long)g2 * n0 + g0];
  } else if (i0 && i1 && !i2) {
    if (g2 == -1) src = (int)(((long)5 * n1 + g1) * n0 + g0);
    else if (g2 == n2) src = B.padsrc[2][(long)g1 * n0 + g0];
  }
  return src >= 0 ? -2 - src : -1;
}

// Geometry of the passes of field (KIND, COMP) along DIM.
template <int KIND, int COMP, int DIM>
struct Pass3 {
  static constexpr bool CROSS = (KIND == 2 && COMP != DIM) || KIND == 3;
  static constexpr bool ON = !(KIND == 3 && COMP == DIM);  // B is not diffused along itself
  static constexpr int X0 = CROSS && COMP == 0, X1 = CROSS && COMP == 1, X2 = CROSS && COMP == 2;
  // ratio area: extents and box coordinates of its first cell
  static constexpr int E0 = s3::T0 + (DIM == 0) + 2 * X0, E1 = s3::T1 + (DIM == 1) + 2 * X1;
  static constexpr int E2 = s3::T2 + (DIM == 2) + 2 * X2;
  static constexpr int G0 = s3::H - (DIM == 0) - X0, G1 = s3::H - (DIM == 1) - X1, G2 = s3::H - (DIM == 2) - X2;
  static constexpr int RS = DIM == 0 ? 1 : (DIM == 1 ? E0 : E0 * E1);  // stride along DIM
  static constexpr int SD = s3::bstride(DIM);
  // lines along DIM, cut into two pieces of SL faces (the last may be shorter)
  static constexpr int N = s3::tdim(DIM) + 1, SL = (N + 1) / 2;
  static constexpr int A1 = DIM == 0 ? E1 : E0, A2 = DIM == 2 ? E1 : E2, NL = ON ? A1 * A2 * 2 : 0;
  __device__ __forceinline__ static int ridx(int lx, int ly, int lz) {
    return ((lz - G2) * E1 + (ly - G1)) * E0 + (lx - G0);
  }
};
// cross arrays of component COMP: the tile +-1 along it
template <int COMP>
__device__ __forceinline__ int cidx3(int lx, int ly, int lz) {
  constexpr int X0 = COMP == 0, X1 = COMP == 1, X2 = COMP == 2;
  return ((lz - s3::H + X2) * (s3::T1 + 2 * X1) + (ly - s3::H + X1)) * (s3::T0 + 2 * X0) + (lx - s3::H + X0);
}

// piece u of the ratio lines of one pass: R where the pass has cross terms,
// R (q(l+1) - q(l)) where it has none
template <bool MIX, int KIND, int COMP, int DIM>
__device__ __forceinline__ void ratio_piece(const Box3& X, int u) {
  using HT = typename Form<MIX>::H;
  using G = Pass3<KIND, COMP, DIM>;
  const int a = u % G::A1, v = u / G::A1, b = v % G::A2, f0 = v / G::A2 * G::SL;
  int e[3];  // first face of the piece in the ratio area
  e[DIM] = f0;
  e[DIM == 0 ? 1 : 0] = a;
  e[DIM == 2 ? 1 : 2] = b;
  const int n = G::N - f0 < G::SL ? G::N - f0 : G::SL;
  const HT* q = static_cast<const HT*>(X.U) + ((G::G2 + e[2]) * s3::BY + G::G1 + e[1]) * s3::BP + G::G0 + e[0];
  HT* o = static_cast<HT*>(X.U) + (MIX ? 2 : 1) * s3::BC + DIM * s3::RA + (e[2] * G::E1 + e[1]) * G::E0 + e[0];
  ratio_line<G::SL, G::SD, G::N % G::SL == 0>(q, n,
                                              [&](int i, HT r, HT dq) { o[i * G::RS] = G::CROSS ? r : mulr(r, dq); });
}
template <bool MIX, int KIND, int COMP>
__device__ __forceinline__ void ratios3(const Box3& X, int tid) {
  constexpr int N0 = Pass3<KIND, COMP, 0>::NL, N1 = Pass3<KIND, COMP, 1>::NL, N2 = Pass3<KIND, COMP, 2>::NL;
  // each direction's pieces start at a warp of their own where that takes no
  // more rounds of the block
  constexpr int P0 = (N0 + 31) / 32 * 32, P1 = P0 + (N1 + 31) / 32 * 32;
  for (int u = tid; u < P1 + N2; u += s3::NT) {
    if (u < P0) {
      if (N0 > 0 && u < N0) ratio_piece<MIX, KIND, COMP, 0>(X, u);
    } else if (u < P1) {
      if (N1 > 0 && u - P0 < N1) ratio_piece<MIX, KIND, COMP, 1>(X, u - P0);
    } else {
      if (N2 > 0) ratio_piece<MIX, KIND, COMP, 2>(X, u - P1);
    }
  }
}

// Diffusive terms of one pass at the tile cell (hyperdif*source1):
// dt cmax/dl (G(i) - G(i-1)), G = chyp R dq times the face mean
template <bool BG, bool MIX, int KIND, int COMP, int DIM>
__device__ __forceinline__ void diffuse3(const Box3& X, const KParams& P, const int* lt, double k, double* out) {
  using HT = typename Form<MIX>::H;
  using G = Pass3<KIND, COMP, DIM>;
  if constexpr (G::ON) {
    constexpr int S = G::SD;
    const HT* q = static_cast<const HT*>(X.U) + (lt[2] * s3::BY + lt[1]) * s3::BP + lt[0];
    const HT* r = static_cast<const HT*>(X.U) + (MIX ? 2 : 1) * s3::BC + DIM * s3::RA + G::ridx(lt[0], lt[1], lt[2]);
    HT fp = r[0], fm = r[-G::RS];
    if constexpr (G::CROSS) {
      fp = mulr(fp, q[S] - q[0]);
      fm = mulr(fm, q[0] - q[-S]);
    }
    if constexpr (KIND == 0) {
      out[R3] = fma(k * P.chyp[R3], (double)(fp - fm), out[R3]);
    } else if constexpr (KIND == 1) {
      out[E3] = fma(k * P.chyp[E3], (double)(fp - fm), out[E3]);
    } else if constexpr (KIND == 2) {
      // the pass along the own component counts twice; face means carry 1/2
      constexpr int ES = DIM == 0 ? 1 : (DIM == 1 ? s3::EX : s3::EX * s3::EY);
      const double* t = X.T + eidx(lt[0], lt[1], lt[2]);
      HT rp, rm, mp, mm;
      if constexpr (MIX) {
        rp = (HT)(t[0] + t[ES]);
        rm = (HT)(t[-ES] + t[0]);
        mp = q[s3::BC] + q[s3::BC + S];
        mm = q[s3::BC - S] + q[s3::BC];
      } else {
        rp = t[0] + t[ES];
        rm = t[-ES] + t[0];
        const HT m0 = mulr(q[0], t[0]);
        mp = fma(q[S], t[ES], m0);
        mm = fma(q[-S], t[-ES], m0);
      }
      const double kk = (COMP == DIM ? 0.5 : 0.25) * k * P.chyp[M3 + COMP];
      out[M3 + COMP] = fma(kk, (double)fma(fp, rp, -mulr(fm, rm)), out[M3 + COMP]);
      out[E3] = fma(kk, (double)fma(fp, mp, -mulr(fm, mm)), out[E3]);
    } else {
      const double kk = k * P.chyp[B3 + COMP];
      out[B3 + COMP] = fma(kk, (double)(fp - fm), out[B3 + COMP]);
      out[E3] = fma(0.5 * kk, (double)fma(fp, q[0] + q[S], -mulr(fm, q[-S] + q[0])), out[E3]);
    }
  }
}

// Cross arrays of field (KIND, COMP) at one box cell (hyperdifmomsourcene2-4,
// hyperdifbsourcene1b-4): for the passes along the two other dimensions a,
// momentum: rho_t tau_a, and tau_a m_a for the energy; B: t_a, and t_a b_a, with
// tau = (q+ - q-) (R + R-) cmax chyp / 8, t: / 4.  Zero outside [2, n-3] and, per
// pass, next to a non-periodic edge along it.
// ma: m or b of the two passes' dimensions at the cell.
template <bool MIX, int KIND, int COMP>
__device__ __forceinline__ void cross3(const Box3& X, const KParams& P, const KBufs& B, const int* l,
                                       const typename Form<MIX>::S* ma) {
  using HT = typename Form<MIX>::H;
  const int n[3] = {P.n0, P.n1, P.n2};
  const int g[3] = {X.o[0] + l[0], X.o[1] + l[1], X.o[2] + l[2]};
  const bool in = g[0] >= 2 && g[0] <= n[0] - 3 && g[1] >= 2 && g[1] <= n[1] - 3 && g[2] >= 2 && g[2] <= n[2] - 3;
  const HT* q = static_cast<const HT*>(X.U) + (l[2] * s3::BY + l[1]) * s3::BP + l[0];
  HT* c = static_cast<HT*>(X.U) + (MIX ? 2 : 1) * s3::BC + 3 * s3::RA + cidx3<COMP>(l[0], l[1], l[2]);
  HT v[4] = {0, 0, 0, 0};
  if (in) {
    constexpr int DA = COMP == 0 ? 1 : 0, DB = COMP == 2 ? 1 : 2;
    auto pass = [&](auto dim, HT m, HT& f, HT& e) {
      constexpr int D = decltype(dim)::value;
      using G = Pass3<KIND, COMP, D>;
      if ((P.bt[D] != 0) && zero1n(g[D], n[D])) return;
      const HT* r = static_cast<const HT*>(X.U) + (MIX ? 2 : 1) * s3::BC + D * s3::RA + G::ridx(l[0], l[1], l[2]);
      const HT k = (HT)((KIND == 2 ? 0.125 : 0.25) * B.cmax_in[D] * P.chyp[(KIND == 2 ? M3 : B3) + COMP]);
      const HT t = (q[G::SD] - q[-G::SD]) * (r[0] + r[-G::RS]) * k;
      f = KIND == 2 ? (HT)X.T[eidx(l[0], l[1], l[2])] * t : t;
      e = mulr(t, m);
    };
    pass(std::integral_constant<int, DA>{}, (HT)ma[0], v[0], v[2]);
    pass(std::integral_constant<int, DB>{}, (HT)ma[1], v[1], v[3]);
  }
  c[0] = v[0];
  c[s3::CA] = v[1];
  if constexpr (MIX) {
    c[2 * s3::CA] = v[2];
    c[3 * s3::CA] = v[3];
  } else {
    c[2 * s3::CA] = v[2] + v[3];
  }
}
// the cross terms at the tile cell: d/dx_COMP of the arrays (sign - for B)
template <bool MIX, int KIND, int COMP>
__device__ __forceinline__ void cross_terms3(const Box3& X, const int* lt, double k, double* out) {
  using HT = typename Form<MIX>::H;
  constexpr int DA = COMP == 0 ? 1 : 0, DB = COMP == 2 ? 1 : 2, F = KIND == 2 ? M3 : B3;
  constexpr int S = COMP == 0 ? 1 : (COMP == 1 ? s3::T0 : s3::T0 * s3::T1);
  const HT* c = static_cast<const HT*>(X.U) + (MIX ? 2 : 1) * s3::BC + 3 * s3::RA + cidx3<COMP>(lt[0], lt[1], lt[2]);
  auto d = [&](int i) -> double { return (double)(c[i * s3::CA + S] - c[i * s3::CA - S]); };
  const double s = KIND == 2 ? k : -k;
  out[F + DA] = fma(s, d(0), out[F + DA]);
  out[F + DB] = fma(s, d(1), out[F + DB]);
  out[E3] = fma(s, d(2), out[E3]);
  if constexpr (MIX) out[E3] = fma(s, d(3), out[E3]);
}

// All passes of one field whose q has been staged (and not yet synchronised);
// bit a of zero: the cell lies next to a non-periodic edge along a.  Leaves the cross terms to the caller (cross_terms3), so that they
// run beside the next field's staging.
template <bool BG, bool MIX, int KIND, int COMP>
__device__ __forceinline__ void field3(const Box3& X, const KParams& P, const KBufs& B, int tid, const int* lt,
                                       double dt, int zero, double* out) {
  using ST = typename Form<MIX>::S;
  const ST* u = static_cast<const ST*>(B.uin);
  constexpr int F = KIND == 2 ? M3 : B3, DA = COMP == 0 ? 1 : 0, DB = COMP == 2 ? 1 : 2;
  constexpr int T = s3::tdim(COMP), L = s3::NT / T;  // cells of a layer across the component
  static_assert(2 * L <= s3::NT, "the two layers beside the tile take one round");
  auto get = [&](const int* b, ST* m) {
    const int g0 = X.o[0] + b[0], g1 = X.o[1] + b[1], g2 = X.o[2] + b[2];
    if (g0 > P.n0 - 1 || g1 > P.n1 - 1 || g2 > P.n2 - 1) return;
    const long c = ((long)g2 * P.n1 + g1) * P.n0 + g0;
    m[0] = __ldg(u + (F + DA) * P.ncell + c);
    m[1] = __ldg(u + (F + DB) * P.ncell + c);
  };
  __syncthreads();
  ratios3<MIX, KIND, COMP>(X, tid);
  __syncthreads();
  diffuse3<BG, MIX, KIND, COMP, 0>(X, P, lt, (zero >> 0) & 1 ? 0.0 : dt * B.cmax_in[0] * X.rd[0][lt[0]], out);
  diffuse3<BG, MIX, KIND, COMP, 1>(X, P, lt, (zero >> 1) & 1 ? 0.0 : dt * B.cmax_in[1] * X.rd[1][lt[1]], out);
  diffuse3<BG, MIX, KIND, COMP, 2>(X, P, lt, (zero >> 2) & 1 ? 0.0 : dt * B.cmax_in[2] * X.rd[2][lt[2]], out);
  if constexpr (KIND >= 2) {
    ST m[2] = {0, 0};
    get(lt, m);
    cross3<MIX, KIND, COMP>(X, P, B, lt, m);
    if (tid < 2 * L) {
      // the two layers beside the tile along the component
      const int v = tid % L;
      constexpr int A = COMP == 0 ? 1 : 0, C = COMP == 2 ? 1 : 2;
      int l[3];
      l[COMP] = s3::H + (tid < L ? -1 : T);
      l[A] = s3::H + v % s3::tdim(A);
      l[C] = s3::H + v / s3::tdim(A);
      get(l, m);
      cross3<MIX, KIND, COMP>(X, P, B, l, m);
    }
  }
  __syncthreads();
}

// fluxes along D at one cell: rho, m0..2, e, and the two B components across
// D (in increasing order); velocities for the background energy terms
template <bool BG, int D>
__device__ __forceinline__ void flux3(const double* s, const double* g, double r, double gamma,
                                      double* F, double* v) {
  const double m[3] = {s[1], s[2], s[3]};
  const double b[3] = {s[5], s[6], s[7]};
  const double bb[3] = {BG ? g[2] : 0.0, BG ? g[3] : 0.0, BG ? g[4] : 0.0};
  const double e = s[4], eb = BG ? g[0] : 0.0;
  const double md = m[D], vd = md * r;
  // computept3 (src/dervfields.cu:107-153)
  const double pt = (gamma - 1.0) * (e - 0.5 * (m[0] * m[0] + m[1] * m[1] + m[2] * m[2]) * r) -
                    (gamma - 2.0) * ((b[0] * bb[0] + b[1] * bb[1] + b[2] * bb[2]) +
                                     0.5 * (b[0] * b[0] + b[1] * b[1] + b[2] * b[2]));
  const double bd = b[D], bbd = bb[D];
  F[0] = md;
#pragma unroll
  for (int c = 0; c < 3; c++) F[1 + c] = vd * m[c] + (c == D ? pt : 0.0) - (b[c] * bbd + bb[c] * bd) - b[c] * bd;
  const double bbm = bb[0] * m[0] + bb[1] * m[1] + bb[2] * m[2];
  const double bm = b[0] * m[0] + b[1] * m[1] + b[2] * m[2];
  F[4] = vd * (e + pt + eb) - (bd * bbm + bbd * bm + bd * bm) * r;
  constexpr int c1 = D == 0 ? 1 : 0, c2 = D == 2 ? 1 : 2;
  F[5] = vd * (b[c1] + bb[c1]) - (m[c1] * r) * (bd + bbd);
  F[6] = vd * (b[c2] + bb[c2]) - (m[c2] * r) * (bd + bbd);
  v[0] = m[0] * r;
  v[1] = m[1] * r;
  v[2] = m[2] * r;
}

// flux phase along D: fluxes on the tile +-2 along D (+-3 for the 6th-order
// derivative), divergence and the background energy terms at the tile cells
template <bool BG, bool MIX, int D, bool O6>
__device__ __forceinline__ void flux_pass3(const Box3& X, const KParams& P, const KBufs& B, int tid,
                                           bool active, const int* lt, const int* gt, double dt,
                                           double* out) {
  constexpr int FH = O6 ? 3 : 2, FA = s3::fa<O6>();
  constexpr int E0 = s3::T0 + (D == 0 ? 2 * FH : 0), E1 = s3::T1 + (D == 1 ? 2 * FH : 0);
  constexpr int E2 = s3::T2 + (D == 2 ? 2 * FH : 0);
  constexpr int G0 = s3::H - (D == 0 ? FH : 0), G1 = s3::H - (D == 1 ? FH : 0), G2 = s3::H - (D == 2 ? FH : 0);
  constexpr int NAREA = E0 * E1 * E2;
  constexpr int FS = D == 0 ? 1 : (D == 1 ? E0 : E0 * E1);
  using ST = typename Form<MIX>::S;
  const ST* u = static_cast<const ST*>(B.uin);
  const int n[3] = {P.n0, P.n1, P.n2};
  const long nc = P.ncell;
  double* F = static_cast<double*>(X.U);
  for (int r = tid; r < NAREA; r += s3::NT) {
    const int lx = G0 + r % E0, ly = G1 + (r / E0) % E1, lz = G2 + r / (E0 * E1);
    const int g0 = X.o[0] + lx, g1 = X.o[1] + ly, g2 = X.o[2] + lz;
    double f[7] = {0, 0, 0, 0, 0, 0, 0}, v[3] = {0, 0, 0};
    if (X.inner || (g0 >= 0 && g0 < n[0] && g1 >= 0 && g1 < n[1] && g2 >= 0 && g2 < n[2])) {
      const long c = ((long)g2 * n[1] + g1) * n[0] + g0;
      double s[8], g[5] = {0, 0, 0, 0, 0};
#pragma unroll
      for (int k = 0; k < 8; k++) s[k] = __ldg(u + k * nc + c);
      if (BG) {
#pragma unroll
        for (int k = 0; k < 5; k++) g[k] = __ldg(B.bg + k * nc + c);
      }
      flux3<BG, D>(s, g, X.R[(lz * s3::BY + ly) * s3::BP + lx], P.gamma, f, v);
    }
#pragma unroll
    for (int k = 0; k < 7; k++) F[k * FA + r] = f[k];
    if (BG) {
#pragma unroll
      for (int k = 0; k < 3; k++) F[(7 + k) * FA + r] = v[k];
    }
  }
  __syncthreads();
  const bool z = ((P.bt[D] != 0) && zero3dn(gt[D], n[D])) || (O6 && edge6(gt[D], n[D]));
  const double rdl2 = 0.5 * X.rd[D][lt[D]];
  const int fo = ((lt[2] - G2) * E1 + (lt[1] - G1)) * E0 + (lt[0] - G0);
  if (active) {
    constexpr int c1 = D == 0 ? 1 : 0, c2 = D == 2 ? 1 : 2;
    const int fld[7] = {R3, M3, M3 + 1, M3 + 2, E3, B3 + c1, B3 + c2};
#pragma unroll
    for (int k = 0; k < 7; k++) {
      double gk = dflux<O6>(F + k * FA, fo, FS, rdl2);
      if (z) gk = 0;
      out[fld[k]] = out[fld[k]] - dt * gk;
    }
    if (BG) {
      // addenergyterms_cd2 (src/centdiff2.cu:80-115): -p_tb dv_D/dx_D, and
      // the derivative-along-D part of sum_i Bb_i Bb_d dv_d/dx_i
      const long co = ((long)gt[2] * n[1] + gt[1]) * n[0] + gt[0];
      const double eb = __ldg(B.bg + GEB * nc + co);
      const double bb[3] = {__ldg(B.bg + 2 * nc + co), __ldg(B.bg + 3 * nc + co), __ldg(B.bg + 4 * nc + co)};
      const double ptb = (P.gamma - 1) * eb - 0.5 * (P.gamma - 2) * (bb[0] * bb[0] + bb[1] * bb[1] + bb[2] * bb[2]);
      double gv = dflux<O6>(F + (7 + D) * FA, fo, FS, rdl2);
      if (z) gv = 0;
      out[E3] -= dt * ptb * gv;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        double gk = dflux<O6>(F + (7 + k) * FA, fo, FS, rdl2);
        if (z) gk = 0;
        out[E3] += dt * bb[D] * bb[k] * gk;
      }
    }
  }
  __syncthreads();
}

template <int MODE, bool BG, bool MIX, bool O6>
__global__ void __launch_bounds__(s3::NT, SMAUG_MINB3D) stage3d_fast(const KParams P, const KBufs B) {
  using ST = typename Form<MIX>::S;
  const ST* u = static_cast<const ST*>(B.uin);
  extern __shared__ double smem[];
  Box3 X;
  X.R = smem;
  X.T = smem + s3::BC;
  X.rd[0] = X.T + s3::EC;
  X.rd[1] = X.rd[0] + s3::BX;
  X.rd[2] = X.rd[1] + s3::BY;
  X.U = X.rd[2] + s3::BZ;
  X.C = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(X.U) + s3::union_bytes<MIX, O6>());
  const int tid = threadIdx.x;
  const int tx = tid % s3::T0, ty = (tid / s3::T0) % s3::T1, tz = tid / (s3::T0 * s3::T1);
  const int n[3] = {P.n0, P.n1, P.n2};
  const long nc = P.ncell;
  X.o[0] = 2 + blockIdx.x * s3::T0 - s3::H;
  X.o[1] = 2 + blockIdx.y * s3::T1 - s3::H;
  X.o[2] = 2 + blockIdx.z * s3::T2 - s3::H;
  // box indices 0 .. B-1 of every axis inside [0, n-1]: no bounds or pad
  // checks in the staging, flux and cross-term loops
  X.inner = X.o[0] >= 0 && X.o[1] >= 0 && X.o[2] >= 0 && X.o[0] + s3::BX <= n[0] &&
            X.o[1] + s3::BY <= n[1] && X.o[2] + s3::BZ <= n[2];

  // running CFL maxima of the grid when the block starts
  double seen[3];
#pragma unroll
  for (int d = 0; d < 3; d++)
    seen[d] = __longlong_as_double(__ldcg(static_cast<const unsigned long long*>(B.cmax_out) + d));

  // ---- 1/rho_t on the box and the per-axis metric ----------------------
  {
    constexpr int NI = (s3::BC + s3::NT - 1) / s3::NT, NB = SMAUG_NB3;
#pragma unroll 1
    for (int i0 = 0; i0 < NI; i0 += NB) {
      ST rho[NB];
      double rhob[NB];
#pragma unroll
      for (int i = 0; i < NB; i++) {
        const int r = tid + (i0 + i) * s3::NT;
        const int lx = r % s3::BP, ly = (r / s3::BP) % s3::BY, lz = r / s3::BS2;
        const int g0 = X.o[0] + lx, g1 = X.o[1] + ly, g2 = X.o[2] + lz;
        const bool in = r < s3::BC && lx < s3::BX &&
                        (X.inner || (g0 >= 0 && g0 < n[0] && g1 >= 0 && g1 < n[1] && g2 >= 0 && g2 < n[2]));
        const long c = in ? ((long)g2 * n[1] + g1) * n[0] + g0 : 0;
        rho[i] = in ? __ldg(u + c) : (ST)1;
        rhob[i] = in ? __ldg(B.bg + GRB * nc + c) : 0.0;
        if (r < s3::BC) X.C[r] = lx < s3::BX ? box_code(X, P, B, lx, ly, lz) : -1;
      }
#pragma unroll
      for (int i = 0; i < NB; i++) {
        const int r = tid + (i0 + i) * s3::NT;
        if (r >= s3::BC) continue;
        const int lx = r % s3::BP, ly = (r / s3::BP) % s3::BY, lz = r / s3::BS2;
        const double rt = (double)rho[i] + rhob[i];
        X.R[r] = recip(rt);
        if (outside(lx, s3::T0) <= 1 && outside(ly, s3::T1) <= 1 && outside(lz, s3::T2) <= 1)
          X.T[eidx(lx, ly, lz)] = rt;
      }
    }
  }
  // the stage sum's operands into L2, a block's lifetime ahead: one thread per
  // row of the tile and array
  for (int r = tid; r < 16 * s3::T1 * s3::T2; r += s3::NT) {
    const int f = r % 16, v = r / 16;
    const int g1 = X.o[1] + s3::H + v % s3::T1, g2 = X.o[2] + s3::H + v / s3::T1;
    const bool base = f < 8;
    if (g1 <= n[1] - 3 && g2 <= n[2] - 3 &&
        (base ? (MODE == SMAUG_INT_EULER || B.stage < 3) : (MODE != SMAUG_INT_EULER && B.stage > 0))) {
      const long c = (f & 7) * nc + ((long)g2 * n[1] + g1) * n[0] + X.o[0] + s3::H;
      const void* q = base ? static_cast<const void*>(static_cast<const ST*>(B.un) + c)
                           : static_cast<const void*>(B.acc + c);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
    }
  }
  for (int r = tid; r < s3::BX + s3::BY + s3::BZ; r += s3::NT) {
    const int a = r < s3::BX ? 0 : (r < s3::BX + s3::BY ? 1 : 2);
    const int l = r - (a == 0 ? 0 : (a == 1 ? s3::BX : s3::BX + s3::BY));
    const int g = X.o[a] + l;
    const double d = (g >= 0 && g < n[a]) ? B.delx[a][g] : 1.0;
    X.rd[a][l] = 1.0 / d;
  }

  // ---- dt of this step and stage time ----------------------------------
  double dt, tstage;
  const bool first = blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && tid == 0;
  if (B.stage == 0) {
    dt = device_dt(P, B.cmax_in, *B.dt_prev, 3);
    if (first) {
      *B.dt_new = dt;
      *B.t_new = *B.t_prev + dt;
      B.cmax_clear[0] = B.cmax_clear[1] = B.cmax_clear[2] = 0ull;
    }
    tstage = *B.t_prev;
  } else {
    dt = *B.dt_new;
    tstage = *B.t_prev + (B.stage == 3 ? dt : 0.5 * dt);
    if (first) B.cmax_clear[0] = B.cmax_clear[1] = B.cmax_clear[2] = 0ull;
  }
  __syncthreads();

  const int lt[3] = {tx + s3::H, ty + s3::H, tz + s3::H};
  const int gt[3] = {X.o[0] + lt[0], X.o[1] + lt[1], X.o[2] + lt[2]};
  const bool active = gt[0] <= n[0] - 3 && gt[1] <= n[1] - 3 && gt[2] <= n[2] - 3;
  const long co = active ? ((long)gt[2] * n[1] + gt[1]) * n[0] + gt[0] : 0;

  double out[8];  // increments
#pragma unroll
  for (int f = 0; f < 8; f++) out[f] = 0.0;

  // ---- fluxes and divergence, direction 0, 1, 2 ----------------------------
  flux_pass3<BG, MIX, 0, O6>(X, P, B, tid, active, lt, gt, dt, out);
  flux_pass3<BG, MIX, 1, O6>(X, P, B, tid, active, lt, gt, dt, out);
  flux_pass3<BG, MIX, 2, O6>(X, P, B, tid, active, lt, gt, dt, out);

  // ---- gravity (addgrav_cd2, src/centdiff2.cu:118-154) --------------------
  if (P.has_grav && active) {
    const double rho = (double)__ldg(u + co);
    const double rr = rho * X.R[(lt[2] * s3::BY + lt[1]) * s3::BP + lt[0]];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      out[M3 + a] = fma(dt * P.g[a], rho, out[M3 + a]);
      out[E3] = fma(dt * P.g[a] * (double)__ldg(u + (M3 + a) * nc + co), rr, out[E3]);
    }
  }

  // ---- hyperdiffusion, field by field; a field's cross terms run beside the
  // staging of the next --------------------------------------------------
  if (P.hyperdif == 1) {
    int zero = 0;  // directions next to whose non-periodic edge the cell lies
#pragma unroll
    for (int a = 0; a < 3; a++) zero |= ((P.bt[a] != 0) && zero1n(gt[a], n[a])) << a;
#define FIELD(K, C)                      \
  stage_q<MIX, K, C>(X, P, B, tid);      \
  field3<BG, MIX, K, C>(X, P, B, tid, lt, dt, zero, out)
#define CROSS(K, C) cross_terms3<MIX, K, C>(X, lt, (zero >> C) & 1 ? 0.0 : 0.5 * dt * X.rd[C][lt[C]], out)
    FIELD(0, 0);
    FIELD(1, 0);
    FIELD(2, 0);
    CROSS(2, 0);
    FIELD(2, 1);
    CROSS(2, 1);
    FIELD(2, 2);
    CROSS(2, 2);
    FIELD(3, 0);
    CROSS(3, 0);
    FIELD(3, 1);
    CROSS(3, 1);
    FIELD(3, 2);
    CROSS(3, 2);
#undef FIELD
#undef CROSS
  }

  // ---- user driver (source_parallel + addsourceterms2) ---------------------
  if (P.driver == SMAUG_DRIVER_GAUSS && active) {
    double v = P.drv_amp;
    if (P.drv_period > 0) v *= sin(tstage * 2.0 * M_PI / P.drv_period);
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (P.drv_sigma[a] > 0) {
        const double x = B.pos[a][gt[a]] - P.drv_x0[a];
        v *= exp(-x * x / (P.drv_sigma[a] * P.drv_sigma[a]));
      }
    }
    const double rr = (double)__ldg(u + co) + (MODE == SMAUG_INT_EULER ? out[R3] : 0.0);
    out[M3] = fma(dt * v, rr + __ldg(B.bg + GRB * nc + co), out[M3]);
  }

  // ---- combine, write, ghost images, CFL maxima -----------------------------
  double cm[3];
#pragma unroll
  for (int d = 0; d < 3; d++) cm[d] = P.cmax_floor[d] > seen[d] ? P.cmax_floor[d] : seen[d];
  if (active) {
    double res[8];
    const bool is_base = (MODE == SMAUG_INT_EULER) || B.stage == 3;
    // all loads before the first store (a load after a store to the
    // accumulator would wait for its own round trip)
    double ub[8], ac[8];
    if (MODE == SMAUG_INT_EULER || B.stage < 3) {
#pragma unroll
      for (int f = 0; f < 8; f++) ub[f] = base_value<MIX>(B, f * nc + co);
    }
    if (MODE != SMAUG_INT_EULER && B.stage > 0) {
#pragma unroll
      for (int f = 0; f < 8; f++) ac[f] = B.acc[f * nc + co];
    }
    if (MODE == SMAUG_INT_EULER) {
#pragma unroll
      for (int f = 0; f < 8; f++) res[f] = ub[f] + out[f];
    } else {
      const double wgt = (B.stage == 0 || B.stage == 3) ? 1.0 / 6.0 : 1.0 / 3.0;
      const double cst = (B.stage == 2) ? 1.0 : 0.5;
#pragma unroll
      for (int f = 0; f < 8; f++) {
        if (B.stage == 3) {
          res[f] = fma(wgt, out[f], ac[f]);
        } else {
          B.acc[f * nc + co] = fma(wgt, out[f], B.stage == 0 ? ub[f] : ac[f]);
          res[f] = fma(cst, out[f], ub[f]);
        }
      }
    }
    int hmax = 0;  // largest exponent word: infinities and NaN have 0x7ff
#pragma unroll
    for (int f = 0; f < 8; f++) hmax = max(hmax, __double2hiint(res[f]) & 0x7fffffff);
    if (hmax >= 0x7ff00000) atomicOr(B.flags, 1);
    int ix[3], iy[3], iz[3];
    ix[0] = gt[0];
    iy[0] = gt[1];
    iz[0] = gt[2];
    const int nx = 1 + ghost_images(gt[0], n[0], P.bc[0], ix + 1);
    const int ny = 1 + ghost_images(gt[1], n[1], P.bc[1], iy + 1);
    const int nz = 1 + ghost_images(gt[2], n[2], P.bc[2], iz + 1);
    bool negated = false;  // res holds the negated values
    for (int cz = 0; cz < nz; cz++)
      for (int b = 0; b < ny; b++)
        for (int a2 = 0; a2 < nx; a2++) {
          const long cc = ((long)iz[cz] * n[1] + iy[b]) * n[0] + ix[a2];
          // antisymmetric images carry the opposite sign (negation is exact)
          const bool neg = (((a2 > 0) && P.gneg[0]) != ((b > 0) && P.gneg[1])) != ((cz > 0) && P.gneg[2]);
          if (neg != negated) {
#pragma unroll
            for (int f = 0; f < 8; f++) res[f] = -res[f];
            negated = neg;
          }
          const double* r = res;
#pragma unroll
          for (int f = 0; f < 8; f++) store_value<MIX>(B, f * nc + cc, r[f], is_base);
          // without background fields an image has its source's fast speeds
          // unless its sign changed
          if (!BG && (a2 > 0 || b > 0 || cz > 0) && !neg) continue;
          double gg[5] = {0, 0, 0, 0, 0};
          if (BG) {
#pragma unroll
            for (int f = 0; f < 5; f++) gg[f] = __ldg(B.bg + f * nc + cc);
          }
          if (may_exceed<3, BG>(P.gamma, r, gg, cm)) {
            const double3 cv = cfast3_call(P.gamma, r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7], gg[0], gg[1],
                                           gg[2], gg[3], gg[4]);
            cm[0] = dmax0(cm[0], cv.x);
            cm[1] = dmax0(cm[1], cv.y);
            cm[2] = dmax0(cm[2], cv.z);
          }
        }
  }
  // maxima above what the grid had when the block started
  __shared__ double red[s3::NT / 32][3];
  if (__syncthreads_or(cm[0] > seen[0] || cm[1] > seen[1] || cm[2] > seen[2])) {
#pragma unroll
    for (int d = 0; d < 3; d++)
      for (int o = 16; o > 0; o >>= 1) cm[d] = dmax0(cm[d], __shfl_xor_sync(0xffffffffu, cm[d], o));
    if ((tid & 31) == 0) {
      red[tid >> 5][0] = cm[0];
      red[tid >> 5][1] = cm[1];
      red[tid >> 5][2] = cm[2];
    }
    __syncthreads();
    if (tid < 3) {
      double v = 0.0;
      for (int w = 0; w < s3::NT / 32; w++) v = dmax0(v, red[w][tid]);
      atomicMax(&B.cmax_out[tid], (unsigned long long)__double_as_longlong(v));
    }
  }
}

template <int MODE, bool MIX, bool O6>
static cudaError_t launch_stage3d_o(const KParams& K, const KBufs& B, cudaStream_t st) {
  dim3 grid((K.n0 - 4 + s3::T0 - 1) / s3::T0, (K.n1 - 4 + s3::T1 - 1) / s3::T1,
            (K.n2 - 4 + s3::T2 - 1) / s3::T2);
  if (K.has_bg)
    stage3d_fast<MODE, true, MIX, O6><<<grid, s3::NT, s3::smem_bytes<MIX, O6>(), st>>>(K, B);
  else
    stage3d_fast<MODE, false, MIX, O6><<<grid, s3::NT, s3::smem_bytes<MIX, O6>(), st>>>(K, B);
  return cudaGetLastError();
}
template <int MODE, bool MIX>
static cudaError_t launch_stage3d(const KParams& K, const KBufs& B, cudaStream_t st) {
  return K.order6 ? launch_stage3d_o<MODE, MIX, true>(K, B, st) : launch_stage3d_o<MODE, MIX, false>(K, B, st);
}

template <int MODE, bool BG, bool MIX, bool O6>
static cudaError_t stage3d_attr() {
  return cudaFuncSetAttribute(stage3d_fast<MODE, BG, MIX, O6>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)s3::smem_bytes<MIX, O6>());
}
