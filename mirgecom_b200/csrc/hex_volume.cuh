// Right-hand side of tensor-product hexahedra in two kernels (float64, ideal
// gas), the counterpart of k_volume / k_face for the line operators:
//
// k_hex_volume   one node per thread, its fields and the neighbours' face
//                values in shared memory.  Per node: the BR1 gradients of q and
//                T by the three line operators (never written to HBM), state
//                and total flux F = F_V - F_I, G_a = sum_j rx[a][j] F_j into
//                shared memory, the face-node records {F.n, |v| + c, p, c,
//                gamma}, and the volume divergence -sum_a WH1 (G_a - G0_a).
// k_hex_face     per face node the numerical flux from the neighbour's record
//                and both q (as k_face does), per node the lift along its three
//                lines, added to the rhs.
//
// The 1-D operators act on a node as dot products with the rows of its three
// line positions, which a thread holds in registers for the whole kernel
// (7 values per axis): 21 shared-memory reads and fused multiply-adds per node
// and field, no products against zero padding and no accumulators in shared
// memory.  WH1 is W1 with the element's own half of the central face value
// folded in (dg_refops.cuh: the same identity along a line),
//   WH1 = W1 + FSR/2 (L1[:,0] e_0^T - L1[:,p] e_p^T),
// so faces contribute the neighbour's half only.
//
// Against gradient, node-flux and surface kernels (18 gradient values per node
// written and read, 20 flux values written and read per node) the two kernels
// move about 320 bytes per node instead of 800.  48^3 order-4 Taylor-Green
// right-hand side: 6.27 -> 2.83 ms (volume 2.01: shared-memory reads, 59 % of
// the L1 data peak, and latency at 18 % of the warps; face 0.83: latency of the
// gathers); 990 order-2 elements 30.5 -> 15.2 us on the device.
#pragma once
#include "hex_kernels.cuh"

namespace mgc {

template <int ORDER>
struct HexV {
  using H = Hex<ORDER>;
  static constexpr int N1 = H::N1, NP = H::NP, NFP = H::NFP, NFN = H::NFN;
  static constexpr int NC = 5, NU = 6, ND = NC * 3, TW = trace_width(NC);
  static constexpr int NT = 128, EPB = NT / NP;
  // doubles per element: fields and face values, later the fluxes G
  static constexpr int VOL = imax(NU * (NP + NFN), ND * NP);
  static constexpr int GEO = 9 + 3;                       // metric, 1 / |rx[a]|
  static size_t smem_volume(int nperm) {
    return (size_t)EPB * (VOL + ND + GEO) * 8 + EPB * 6 * 4 + (size_t)nperm * NFP + 16;
  }
  static size_t smem_face(int nperm) {
    return (size_t)EPB * NC * NFN * 8 + 2 * (size_t)nperm * NFP + 16;
  }
  // workspace: records, node-0 shifts, wave speeds, boundary records and plus
  // states, each 256-byte aligned
  struct Parts {
    size_t s0, lam, btrace, bplus, total;
  };
  static Parts parts(int64_t nelem, int64_t nbf) {
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t nb = (size_t)(nbf > 0 ? nbf : 1), ne = (size_t)nelem;
    Parts p;
    p.s0 = al(ne * NFN * TW * 8);
    p.lam = p.s0 + al(ne * 6 * NC * 8);
    p.btrace = p.lam + al(ne * NP * 8);
    p.bplus = p.btrace + al(nb * NFP * TW * 8);
    p.total = p.bplus + al(nb * NFP * NC * 8);
    return p;
  }
};

namespace {

// A thread's rows of the line operators at its node (x0, x1, x2): w[a][k] =
// -WH1[x_a][k], l[a][s] = L1[x_a][s].
template <int ORDER>
struct LineRows {
  using H = Hex<ORDER>;
  static constexpr int N1 = H::N1;
  double w[3][N1], l[3][2];
  __device__ __forceinline__ void init(int node) {
    const int x[3] = {node % N1, node / N1 % N1, node / (N1 * N1)};
    const double fsr = c_hex64[H::OFF_FSR];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int i = x[a] < N1 ? x[a] : 0;
      l[a][0] = c_hex64[H::OFF_L + i * 2];
      l[a][1] = c_hex64[H::OFF_L + i * 2 + 1];
#pragma unroll
      for (int k = 0; k < N1; ++k) w[a][k] = -c_hex64[H::OFF_W + i * N1 + k];
      w[a][0] -= 0.5 * fsr * l[a][0];
      w[a][N1 - 1] += 0.5 * fsr * l[a][1];
    }
  }
};

// first node and stride of the node's line along axis a
template <int N1>
__device__ __forceinline__ void line_of(int node, int a, int& base, int& stride, int& n) {
  const int x = node % N1, y = node / N1 % N1, z = node / (N1 * N1);
  stride = a == 0 ? 1 : a == 1 ? N1 : N1 * N1;
  n = a == 0 ? y + N1 * z : a == 1 ? x + N1 * z : x + N1 * y;
  base = a == 0 ? N1 * n : a == 1 ? x + N1 * N1 * z : n;
}

template <int ORDER, bool VISC>
__global__ void __launch_bounds__(128, 3) k_hex_volume(DGArgs<double> a, GasParams g) {
  using V = HexV<ORDER>;
  using H = Hex<ORDER>;
  using R = double;
  constexpr int N1 = V::N1, NP = V::NP, NFP = V::NFP, NFN = V::NFN, NC = V::NC, NU = V::NU;
  constexpr int EPB = V::EPB, ND = V::ND, GEO = V::GEO, TW = V::TW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* vol = reinterpret_cast<R*>(smem_raw);             // [EPB][VOL]
  R* g0_s = vol + EPB * V::VOL;                        // [EPB][ND]
  R* geo_s = g0_s + EPB * ND;                          // [EPB][GEO]
  int32_t* conn_s = reinterpret_cast<int32_t*>(geo_s + EPB * GEO);   // [EPB][6]
  uint8_t* perm_s = reinterpret_cast<uint8_t*>(conn_s + EPB * 6);

  const int E = a.nelem;
  const int64_t EN = (int64_t)E * NP;
  const R fsr = c_hex64[H::OFF_FSR];
  const int tid = threadIdx.x;
  const int e = tid / NP, k = tid % NP;                // this thread's node
  LineRows<ORDER> op;
  op.init(k);
  int lb[3], ls[3], ln[3];
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) line_of<N1>(k, ax, lb[ax], ls[ax], ln[ax]);
  for (int i = tid; i < a.nperm * NFP; i += V::NT) perm_s[i] = a.perm[i];
  const int64_t bstride = (int64_t)a.nbf * NFP;

  const int ntiles = (E + EPB - 1) / EPB;
  bool bad = false;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int e0 = tile * EPB;
    const int ne = imin(EPB, E - e0);
    const bool act = e < ne;
    const int64_t gn = (int64_t)(e0 + e) * NP + k;
    __syncthreads();   // the previous tile's divergence has read G
    for (int i = tid; i < ne * 6; i += V::NT) conn_s[i] = a.conn[(int64_t)e0 * 6 + i];
    for (int i = tid; i < ne * 3; i += V::NT) {
      const int ee = i / 3, ax = i % 3;
      R mag2 = R(0);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const R v = a.rx[((int64_t)e0 + ee) * 9 + ax * 3 + j];
        geo_s[ee * GEO + ax * 3 + j] = v;
        mag2 += v * v;
      }
      geo_s[ee * GEO + 9 + ax] = R(1) / sqrt(mag2);
    }
    R qq[NC];
    if (act) {
#pragma unroll
      for (int c = 0; c < NC; ++c) qq[c] = a.q[c * EN + gn];
      if constexpr (VISC) {
        // shifted by the element's node 0
        R q0[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) q0[c] = a.q[c * EN + (int64_t)(e0 + e) * NP];
        R* u = vol + e * V::VOL;
#pragma unroll
        for (int c = 0; c < NC; ++c) u[c * NP + k] = qq[c] - q0[c];
        u[NC * NP + k] = node_temperature<R, 3, 0>(qq, R(0), g) - node_temperature<R, 3, 0>(q0, R(0), g);
      }
    }
    if constexpr (VISC) {
      // face values -+FSR (u* - u0 - own half), one face node per item; the
      // pairing and (at boundaries) the own value come from global memory, so
      // that the gathers start with the tile
      for (int fnode = tid; fnode < ne * NFN; fnode += V::NT) {
        const int ee = fnode / NFN, fm = fnode % NFN, f = fm / NFP, m = fm % NFP;
        const int cn = a.conn[((int64_t)e0 + ee) * 6 + f];
        int mode = 2, bf = 0;   // 0 two-sided average, 1 prescribed exterior, 2 interior value
        const int64_t g0 = (int64_t)(e0 + ee) * NP;
        const int64_t gm = g0 + hex_node<N1>(f >> 1, m, (f & 1) ? N1 - 1 : 0);
        int64_t gi = gm;
        if (cn >= 0) {
          const int en = cn >> 8, pr = cn & 255;
          const int kn = (pr < a.nperm) ? perm_s[pr * NFP + m] : NP;
          if (en >= E || kn >= NP) {
            atomicOr(a.status, ST_BAD_INDEX);
          } else {
            gi = (int64_t)en * NP + kn;
            mode = 0;
          }
        } else {
          bf = -(cn + 1);
          const int kind = (bf < a.nbf) ? a.bkind[bf] : -1;
          if (kind == BK_PRESCRIBED && a.bext)
            mode = 1;
          else if (kind != BK_DUMMY)   // unknown, or a kind the hexahedra do not evaluate
            atomicOr(a.status, ST_BAD_INDEX);
        }
        const R sg = (f & 1) ? fsr : -fsr;
        R* pc = vol + ee * V::VOL + NU * NP + fm;
        // the neighbour's value, or the own one (its half is u* - own half)
        R up[NU], q0[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          up[c] = a.q[c * EN + gi];
          q0[c] = a.q[c * EN + g0];
        }
        const R t0 = node_temperature<R, 3, 0>(q0, R(0), g);
        up[NC] = node_temperature<R, 3, 0>(up, R(0), g) - t0;
#pragma unroll
        for (int c = 0; c < NC; ++c) up[c] -= q0[c];
        if (mode == 1) {
          // exterior value less the own half
          R ub[NU];
#pragma unroll
          for (int c = 0; c < NC; ++c) ub[c] = a.bext[c * bstride + (int64_t)bf * NFP + m];
          ub[NC] = node_temperature<R, 3, 0>(ub, R(0), g) - t0;
#pragma unroll
          for (int c = 0; c < NU; ++c)
            up[c] = R(2) * (c < NC ? ub[c] - q0[c < NC ? c : 0] : ub[c]) - up[c];
        }
#pragma unroll
        for (int c = 0; c < NU; ++c) pc[c * NFN] = sg * (R(0.5) * up[c]);
      }
    }
    __syncthreads();

    // gradients, flux and G of this thread's node
    R gr[NC][3];
    NodeState<R, 3, 0> st;
    if (act) {
      const R* rxe = geo_s + e * GEO;
      R gq[NU][3];
      if constexpr (VISC) {
        const R* ue = vol + e * V::VOL;
#pragma unroll
        for (int c = 0; c < NU; ++c) {
          const R* u = ue + c * NP;
          const R* p = ue + NU * NP + c * NFN;
#pragma unroll
          for (int j = 0; j < 3; ++j) gq[c][j] = R(0);
#pragma unroll
          for (int ax = 0; ax < 3; ++ax) {
            R v = op.l[ax][0] * p[(2 * ax) * NFP + ln[ax]] + op.l[ax][1] * p[(2 * ax + 1) * NFP + ln[ax]];
#pragma unroll
            for (int i = 0; i < N1; ++i) v += op.w[ax][i] * u[lb[ax] + i * ls[ax]];
#pragma unroll
            for (int j = 0; j < 3; ++j) gq[c][j] += rxe[ax * 3 + j] * v;
          }
        }
      }
      make_state<R, 3, 0>(qq, R(0), g, st);
      R fl[NC][3];
      inviscid_flux<R, 3, 0>(st, fl);
      if constexpr (VISC) {
        R fv[NC][3];
        viscous_flux<R, 3, 0, false>(st, gq, gq[NC], fv);
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < 3; ++j) fl[c][j] = fv[c][j] - fl[c][j];
      } else {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < 3; ++j) fl[c][j] = -fl[c][j];
      }
      bad |= !(st.p == st.p) || !(st.c == st.c);
      R v2 = R(0);
#pragma unroll
      for (int j = 0; j < 3; ++j) v2 += st.v[j] * st.v[j];
      const R lam = sqrt(v2) + st.c;
      a.lam[gn] = lam;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
          R acc = R(0);
#pragma unroll
          for (int j = 0; j < 3; ++j) acc += rxe[ax * 3 + j] * fl[c][j];
          gr[c][ax] = acc;
        }
      // records of the faces this node lies on: n = -+rx[ax] / |rx[ax]|
      const int x[3] = {k % N1, k / N1 % N1, k / (N1 * N1)};
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        if (x[ax] != 0 && x[ax] != N1 - 1) continue;
        const int f = 2 * ax + (x[ax] == 0 ? 0 : 1);
        const R im = x[ax] == 0 ? -rxe[9 + ax] : rxe[9 + ax];
        R rec[TW];
#pragma unroll
        for (int c = 0; c < NC; ++c) rec[c] = gr[c][ax] * im;
        rec[NC] = lam;
        rec[NC + 1] = st.p;
        rec[NC + 2] = st.c;
        rec[NC + 3] = st.gamma;
#pragma unroll
        for (int i = NC + 4; i < TW; ++i) rec[i] = R(0);
        const int fm = f * NFP + ln[ax];
        store_rec<R, TW>(a.trace + ((int64_t)(e0 + e) * NFN + fm) * TW, fm, rec);
        const int cn = conn_s[e * 6 + f];
        if (cn < 0) {
          const int bf = -(cn + 1);
          if (bf < a.nbf && a.bkind[bf] == BK_PRESCRIBED && a.bext) {
            R gb[NU * 3];
#pragma unroll
            for (int i = 0; i < NU * 3; ++i) gb[i] = VISC ? gq[i / 3][i % 3] : R(0);
            boundary_record<R, 3, 0, false, VISC>(
                a, g, bf, ln[ax], NFP, gb, 1, rxe[ax * 3] * im, rxe[ax * 3 + 1] * im,
                rxe[ax * 3 + 2] * im, a.btrace + ((int64_t)bf * NFP + ln[ax]) * TW);
          }
        }
      }
      if (k == 0) {
#pragma unroll
        for (int i = 0; i < ND; ++i) g0_s[e * ND + i] = gr[i / 3][i % 3];
      }
    }
    __syncthreads();   // fields and face values have been read; G0 is complete
    if (act) {
      R* gs = vol + e * V::VOL;
#pragma unroll
      for (int i = 0; i < ND; ++i) gs[i * NP + k] = gr[i / 3][i % 3] - g0_s[e * ND + i];
    }
    // element-constant shift of the face terms, F0 . n
    for (int i = tid; i < ne * 6 * NC; i += V::NT) {
      const int c = i % NC, f = i / NC % 6, ee = i / (NC * 6), ax = f >> 1;
      const R v = g0_s[ee * ND + c * 3 + ax] * geo_s[ee * GEO + 9 + ax];
      a.s0[(int64_t)e0 * 6 * NC + i] = (f & 1) ? v : -v;
    }
    __syncthreads();
    if (act) {
      const R* ge = vol + e * V::VOL;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        R v = R(0);
#pragma unroll
        for (int ax = 0; ax < 3; ++ax)
#pragma unroll
          for (int i = 0; i < N1; ++i) v += op.w[ax][i] * ge[(c * 3 + ax) * NP + lb[ax] + i * ls[ax]];
        a.out[c * EN + gn] = v;
      }
    }
  }
  if (bad) atomicOr(a.status, ST_NAN);
}

template <int ORDER, bool VISC>
__global__ void __launch_bounds__(128, 5) k_hex_face(DGArgs<double> a, GasParams g) {
  using V = HexV<ORDER>;
  using H = Hex<ORDER>;
  using R = double;
  constexpr int N1 = V::N1, NP = V::NP, NFP = V::NFP, NFN = V::NFN, NC = V::NC;
  constexpr int EPB = V::EPB, TW = V::TW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* s_s = reinterpret_cast<R*>(smem_raw);             // [EPB][NC][NFN]
  uint8_t* perm_s = reinterpret_cast<uint8_t*>(s_s + EPB * NC * NFN);
  uint8_t* fslot_s = perm_s + a.nperm * NFP;

  const int E = a.nelem;
  const int64_t EN = (int64_t)E * NP;
  const R fsr = c_hex64[H::OFF_FSR];
  const int tid = threadIdx.x;
  const int e = tid / NP, k = tid % NP;
  LineRows<ORDER> op;
  op.init(k);
  int ln[3];
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    int b, s;
    line_of<N1>(k, ax, b, s, ln[ax]);
  }
  for (int i = tid; i < a.nperm * NFP; i += V::NT) {
    perm_s[i] = a.perm[i];
    fslot_s[i] = a.fslot[i];
  }
  const int64_t bstride = (int64_t)a.nbf * NFP;

  const int ntiles = (E + EPB - 1) / EPB;
  bool bad = false;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int e0 = tile * EPB;
    const int ne = imin(EPB, E - e0);
    __syncthreads();   // the previous tile's lift has read s_s
    // this thread's rhs values, in flight during the face phase
    R rhs[NC];
    const int64_t gn = (int64_t)(e0 + e) * NP + k;
    if (e < ne) {
#pragma unroll
      for (int c = 0; c < NC; ++c) rhs[c] = a.out[c * EN + gn];
    }
    for (int fnode = tid; fnode < ne * NFN; fnode += V::NT) {
      const int ee = fnode / NFN, fm = fnode % NFN, f = fm / NFP, m = fm % NFP, ax = f >> 1;
      const int cn = a.conn[((int64_t)e0 + ee) * 6 + f];
      const R* rx = a.rx + ((int64_t)e0 + ee) * 9 + ax * 3;
      const R mag = sqrt(rx[0] * rx[0] + rx[1] * rx[1] + rx[2] * rx[2]);
      const R fsc = mag * fsr;
      const int64_t gm = (int64_t)(e0 + ee) * NP + hex_node<N1>(ax, m, (f & 1) ? N1 - 1 : 0);
      const R* recm = a.trace + ((int64_t)(e0 + ee) * NFN + fm) * TW;
      const R* s0 = a.s0 + ((int64_t)(e0 + ee) * 6 + f) * NC;
      R* bcol = s_s + ee * NC * NFN + fm;
      // 0 interior, 1 prescribed, 2 interior flux only (dummy boundary, or a
      // pairing that fails its index checks)
      int mode = 2, slp = 0;
      const R* recp = nullptr;
      const R* qp_g = nullptr;
      int64_t qstride = EN;
      if (cn >= 0) {
        const int en = cn >> 8, pr = cn & 255;
        int kn = NP, sl = NFN;
        if (pr < a.nperm) {
          kn = perm_s[pr * NFP + m];
          sl = fslot_s[pr * NFP + m];
        }
        if (en < E && kn < NP && sl < NFN) {
          recp = a.trace + ((int64_t)en * NFN + sl) * TW;
          slp = sl;
          qp_g = a.q + (int64_t)en * NP + kn;
          mode = 0;
        } else {
          atomicOr(a.status, ST_BAD_INDEX);
        }
      } else {
        const int bf = -(cn + 1);
        const int kind = (bf < a.nbf) ? a.bkind[bf] : -1;
        if (kind == BK_PRESCRIBED && a.bext) {
          recp = a.btrace + ((int64_t)bf * NFP + m) * TW;
          slp = m;
          qp_g = a.bplus + (int64_t)bf * NFP + m;
          qstride = bstride;
          mode = 1;
        } else if (kind != BK_DUMMY) {
          atomicOr(a.status, ST_BAD_INDEX);
        }
      }
      if (mode == 2) {
        R rm[TW];
        load_rec<R, TW>(recm, fm, rm);
#pragma unroll
        for (int c = 0; c < NC; ++c) bcol[c * NFN] = (fsc * R(0.5)) * (rm[c] - s0[c]);
        continue;
      }
      if (a.flux_kind == FLUX_HLL) {
        R n[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const R v = rx[j] / mag;
          n[j] = (f & 1) ? v : -v;
        }
        face_flux_general<R, 3, 0, VISC>(a, EN, gm, recm, fm, recp, slp, qp_g, qstride, n[0], n[1],
                                         n[2], fsc, s0, bcol, NFN);
        continue;
      }
      // F* . n - F0 . n less the own half that WH1 carries (k_face)
      R rp[6];
      static_assert(!RecLayout<R, TW>::ROT, "unrotated records");
      load_record<R, 6>(recp, rp);
      const R lam = (a.flux_kind == FLUX_RUSANOV) ? fmax(a.lam[gm], rp[NC]) : R(0);
      const R hf = fsc * R(-0.5);
#pragma unroll
      for (int c = 0; c < NC; ++c)
        bcol[c * NFN] = hf * ((rp[c] + s0[c]) + lam * (a.q[c * EN + gm] - qp_g[c * qstride]));
    }
    __syncthreads();
    if (e < ne) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const R* s = s_s + (e * NC + c) * NFN;
        R v = rhs[c];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax)
          v += op.l[ax][0] * s[(2 * ax) * NFP + ln[ax]] + op.l[ax][1] * s[(2 * ax + 1) * NFP + ln[ax]];
        a.out[c * EN + gn] = v;
        bad |= !(v == v);
      }
    }
  }
  if (bad) atomicOr(a.status, ST_NAN);
}

template <int ORDER, bool VISC>
inline int hex_rhs_order(DGArgs<double> a, const GasParams& g, char* ws, cudaStream_t s) {
  using V = HexV<ORDER>;
  const auto p = V::parts(a.nelem, a.nbf);
  a.trace = reinterpret_cast<double*>(ws);
  a.s0 = reinterpret_cast<double*>(ws + p.s0);
  a.lam = reinterpret_cast<double*>(ws + p.lam);
  a.btrace = reinterpret_cast<double*>(ws + p.btrace);
  a.bplus = reinterpret_cast<double*>(ws + p.bplus);
  const int ntiles = (a.nelem + V::EPB - 1) / V::EPB;
  int nblk = 0;
  size_t smem = V::smem_volume(a.nperm);
  auto k1 = k_hex_volume<ORDER, VISC>;
  int rc = prepare_kernel(k1, smem);
  if (rc) return rc;
  rc = persistent_grid(k1, V::NT, smem, ntiles, &nblk);
  if (rc) return rc;
  k1<<<nblk, V::NT, smem, s>>>(a, g);
  if (cudaGetLastError() != cudaSuccess) return MGC_E_CUDA;
  if (a.mid_event && cudaEventRecord(static_cast<cudaEvent_t>(a.mid_event), s) != cudaSuccess)
    return MGC_E_CUDA;
  smem = V::smem_face(a.nperm);
  auto k2 = k_hex_face<ORDER, VISC>;
  rc = prepare_kernel(k2, smem);
  if (rc) return rc;
  rc = persistent_grid(k2, V::NT, smem, ntiles, &nblk);
  if (rc) return rc;
  k2<<<nblk, V::NT, smem, s>>>(a, g);
  return cudaGetLastError() == cudaSuccess ? MGC_OK : MGC_E_CUDA;
}

inline size_t hex_rhs_workspace(int order, int64_t nelem, int64_t nbf) {
  switch (order) {
    case 1: return HexV<1>::parts(nelem, nbf).total;
    case 2: return HexV<2>::parts(nelem, nbf).total;
    case 3: return HexV<3>::parts(nelem, nbf).total;
    case 4: return HexV<4>::parts(nelem, nbf).total;
    default: return 0;
  }
}

inline int hex_rhs(int order, bool visc, const DGArgs<double>& a, const GasParams& g, char* ws,
                   cudaStream_t s) {
  switch (order) {
    case 1: return visc ? hex_rhs_order<1, true>(a, g, ws, s) : hex_rhs_order<1, false>(a, g, ws, s);
    case 2: return visc ? hex_rhs_order<2, true>(a, g, ws, s) : hex_rhs_order<2, false>(a, g, ws, s);
    case 3: return visc ? hex_rhs_order<3, true>(a, g, ws, s) : hex_rhs_order<3, false>(a, g, ws, s);
    case 4: return visc ? hex_rhs_order<4, true>(a, g, ws, s) : hex_rhs_order<4, false>(a, g, ws, s);
    default: return MGC_E_UNSUPPORTED;
  }
}

}  // namespace

}  // namespace mgc
