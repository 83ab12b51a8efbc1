// Two-kernel right-hand side for simplicial elements: a volume kernel and a
// face kernel.
//
// k_volume (one persistent CTA per SM slot, a loop over element tiles):
//   gradients  grad_cv_operator + grad_t_operator (navierstokes.py:129-347)
//              exactly as k_grad computes them, but kept in shared memory
//              (node-major); written to HBM only when the caller asks for
//              them (return_gradients, navierstokes.py:573-574)
//   pointwise  per node: state, total flux F = F_V - F_I (viscous.py:232-293,
//              inviscid.py:65-102), Arrhenius sources (eos.py:858-875); the
//              metric-combined volume flux G_r = sum_j (dr_r/dx_j) F_j into
//              shared memory; for each face the node lies on, a face-node
//              record {F.n, |v| + c, p, c, gamma} into HBM; the node-0 flux
//              F0.n per face (the element-constant shift) into HBM; at
//              prescribed boundary faces the exterior state's record
//   volume     rhs = -sum_r W_r (G_r - G0_r) + sources on the tensor cores,
//              written to HBM (float64: WH_r, the weak derivative with the
//              element's own half of the central face flux folded in,
//              dg_refops.cuh)
// k_face (persistent as well):
//   faces      per face node: the neighbour's record (through the face
//              pairing) and the own one (float64: its wave speed only, WH
//              having added the own half), q on both sides, and the numerical
//              flux F*_V - F*_I (Rusanov / central from the records alone, HLL
//              through the general path) minus F0.n, scaled by the face factor
//   lift       rhs += LIFT S on the tensor cores
//
// Against the three-pass split (gradients, per-node flux records, surface)
// this never writes the gradients to HBM, writes compact face-node records
// instead of full per-node flux records, and leaves the face kernel a small
// contraction (K = Nf * Nfp).  Subtracting the element-constant flux F0 from
// the volume terms (volume kernel) and from the face terms (face kernel)
// leaves the discrete divergence unchanged: -W c + LIFT (c.n) = 0 for a
// constant c, so -WH c + LIFT (c.n) / 2 = 0.
#pragma once
#include "async_copy.cuh"
#include "boundary.cuh"
#include "dg_kernels.cuh"

namespace mgc {

// Face-node record: F.n (NC values, n the element's own outward unit normal),
// then |v| + c, p, c, gamma, padded to 16 bytes.
__host__ __device__ constexpr int trace_width(int nc) { return round_up(nc + 4, 4); }

// The 16-byte chunks of a record are stored rotated by its slot (face slot
// f * NFP + m; m for boundary records): the threads of a warp read the same
// chunk of consecutive records, which would all start in the same few banks of
// L1 (64-byte records: 4 lanes on one bank; 128-byte ones: 8).  Face kernel of
// the reacting mixture, 32^3 p3: float32 430 -> 408 us (L1 data wavefronts 72 ->
// 62 % of peak), float64 1129 -> 835 us (with four resident blocks instead of
// three).
template <class R, int TW>
struct RecLayout {
  static constexpr int VEC = 16 / (int)sizeof(R), NCH = TW / VEC;
  static constexpr bool ROT = (NCH & (NCH - 1)) == 0;
  static constexpr int PER_LINE = imax(1, 128 / (TW * (int)sizeof(R)));
  // offset (values) of chunk t of the record in *slot*
  static __device__ __forceinline__ int chunk(int slot, int t) {
    return ROT ? ((t + slot / PER_LINE) & (NCH - 1)) * VEC : t * VEC;
  }
};

template <class R, int DIM, int ORDER, int NS, bool MIX>
struct VCfg {
  using G = Cfg<R, DIM, ORDER, NS, MIX>;
  static constexpr int RB = (int)sizeof(R);
  static constexpr bool TF32 = G::TF32;
  static constexpr int NP = G::NP, NF = G::NF, NFP = G::NFP, NFN = G::NFN;
  static constexpr int NC = G::NC, NU = G::NU;
  static constexpr int MP = G::MP, MT = G::MT, NAC = G::NAC, MROW = Tile<R>::MROW;
  static constexpr int KSTEP = Tile<R>::KSTEP;
  static constexpr int KU = G::KU, KS = G::KS, KL = G::KL, NFPK = G::NFPK, KUR = G::KUR;
  static constexpr int GEO = G::GEO;
  static constexpr int TW = trace_width(NC);
  // node-major staging rows (odd strides: a warp reading one row per lane,
  // or the tensor-core fragment pattern, hits distinct banks)
  static constexpr int GST = (NU * DIM) | 1;     // gradients of one node
  static constexpr int FST = (NC * DIM) | 1;     // metric-combined fluxes of one node

  // ---- volume kernel: threads, elements per tile, shared memory
  static constexpr int NT = TF32 ? 256 : 128;
  static constexpr int MINB = 2;
  static constexpr int BUDGET = 111 * 1024;
  static constexpr int A_VOL = NAC * (DIM * MP * KU + NF * MP * KL);
  static constexpr __host__ __device__ int nnode(int epb) { return epb * NP + (KUR - NP) + 4; }
  static constexpr __host__ __device__ int ncol_g(int epb) { return round_up(NU * epb, 8); }
  static constexpr __host__ __device__ int w1(int epb) {
    return imax(ncol_g(epb) * (KU + KS), nnode(epb) * FST + NS * epb * NP);
  }
  static constexpr __host__ __device__ int vol_reals(int epb) {
    return A_VOL + w1(epb) + nnode(epb) * GST + epb * GEO + NU * epb;
  }
  static constexpr __host__ __device__ size_t vol_bytes(int epb, int nperm) {
    return (size_t)vol_reals(epb) * RB + NFN * 4 + epb * NF * 4 + NP * NF * 2 +
           (size_t)nperm * NFP + 64;
  }
  // largest multiple of 4 elements (8 on the float32 path) within the budget
  // with up to 32 face-pairing permutations
  static constexpr __host__ __device__ int pick_epb() {
    int best = 4;
    for (int e = 4; e <= 32; e += (TF32 ? 4 : 4))
      if (vol_bytes(e, 32) <= (size_t)BUDGET && (!TF32 || e % 8 == 0 || e == 4)) best = e;
    return best;
  }
  static constexpr int EPB = pick_epb();
  static constexpr int NNODE = nnode(EPB);
  static constexpr int NCOL = ncol_g(EPB);
  static constexpr int W1 = w1(EPB);
  static constexpr int NCOLD = round_up(NC * EPB, 8);      // divergence columns

  // ---- flux-volume kernel (gradients from HBM): no gradient operands or
  // staging of its own gradients; element tiles sized so the pointwise phase
  // fills the block.  Where the rows allow it (STAGED below) the tile's inputs
  // are staged in shared memory: rows of the NC fields, the operator and source
  // temperatures, the gradients
  static constexpr int NT3 = TF32 ? 256 : 128;
  // operator rows: NP per r.  The last m-tile reads up to MP rows, on into the
  // next matrix or gfl (accumulator rows >= NP, never stored)
  static constexpr int A_FLUX = NAC * DIM * NP * KU;
  static constexpr int ROW_T = NC, ROW_G = NC + (MIX ? 2 : 0);
  static constexpr __host__ __device__ int rows3(bool visc) {
    return ROW_G + (visc ? NU * DIM : 0);
  }
  static constexpr int GEO3 = DIM * DIM + NF * DIM;        // metric, unit normals
  static constexpr __host__ __device__ int nnode3(int epb) { return epb * NP + (KUR - NP) + 4; }
  static constexpr __host__ __device__ size_t flux_bytes(int epb, bool visc, bool staged) {
    return (size_t)round_up(A_FLUX + nnode3(epb) * FST + NS * epb * NP + 2 * epb * GEO3 +
                                epb * NC * DIM, 4) * RB +
           (staged ? (size_t)round_up(epb * NP * RB, 16) * rows3(visc) : 0) + NFN * 4 +
           2 * epb * NF * 4 + NP * NF * 2 + 64;
  }
  // the largest tile with at most one node per thread and two blocks per SM;
  // staged rows of a tile start on 16 bytes
  static constexpr __host__ __device__ int epb3(bool staged) {
    int best = 1;
    for (int e = 1; e * NP <= NT3; ++e)
      if (flux_bytes(e, true, staged) <= (size_t)BUDGET && (!staged || e * NP * RB % 16 == 0))
        best = e;
    return best;
  }
  static_assert(epb3(true) * NP * RB % 16 == 0, "no tile of whole 16-byte pieces");

  // ---- face kernel
  // 8-element tiles (the face pass is bound by its gathers' latency: 8.7 ms
  // against 9.8 ms for four blocks of 16 elements at 80^3, float32), in 24 or
  // 25 resident warps.  160 threads where they take the tile's face nodes in
  // whole rounds (order-3 tetrahedra: 320 in two; with 128 the third round is
  // half empty, 64^3 float32 3.27 -> 3.10 ms); 128 elsewhere (order 2 in one
  // round of 192: 0.50 -> 0.62 ms at 40^3, four blocks hide less latency than
  // six).  The four fields of the 2-D ideal gas fit seven blocks (72 registers:
  // unbounded, order 1 takes 74 and six blocks, 600 x 600 cells 0.90 -> 0.85 ms)
  static constexpr int NT2 = TF32 && (8 * NFN) % 160 == 0 ? 160 : 128;
  static constexpr int MINB2 = TF32 ? (NC == 4 ? 7 : 800 / NT2) : 4;
  static constexpr int KFR = round_up(NFN, KSTEP);
  static constexpr int KF = Tile<R>::stride(KFR);
  static constexpr int A_FACE = NAC * MP * KF;
  static constexpr int EPB2 = 8;
  static constexpr int NCOL2 = round_up(NC * EPB2, 8);
  static size_t face_bytes(int nperm) {
    return (size_t)(A_FACE + NCOL2 * KF + EPB2 * GEO) * RB + NFN * 4 + EPB2 * NF * 4 +
           2 * (size_t)nperm * NFP + 64;
  }
};

namespace {

// 16-byte vector store / load of the record in *slot* (TW values, 16-byte
// aligned)
template <class R, int TW>
__device__ __forceinline__ void store_rec(R* dst, int slot, const R (&rec)[TW]) {
  using L = RecLayout<R, TW>;
#pragma unroll
  for (int t = 0; t < L::NCH; ++t) {
    R* p = dst + L::chunk(slot, t);
    if constexpr (sizeof(R) == 4)
      *reinterpret_cast<float4*>(p) =
          make_float4(rec[4 * t], rec[4 * t + 1], rec[4 * t + 2], rec[4 * t + 3]);
    else
      *reinterpret_cast<double2*>(p) = make_double2(rec[2 * t], rec[2 * t + 1]);
  }
}
template <class R, int TW>
__device__ __forceinline__ void load_rec(const R* src, int slot, R (&rec)[TW]) {
  using L = RecLayout<R, TW>;
#pragma unroll
  for (int t = 0; t < L::NCH; ++t) {
    R v[L::VEC];
    load_record<R, L::VEC>(src + L::chunk(slot, t), v);
#pragma unroll
    for (int i = 0; i < L::VEC; ++i) rec[t * L::VEC + i] = v[i];
  }
}

// The exterior state's record at face node m of prescribed boundary face bf
// (boundary.py:141-146 for the viscous part: the exterior state with the
// interior gradients *gq* [NU][DIM] of the face node), in the neighbour's
// convention: -F_ext.n with n the interior's outward normal.  Out of line,
// arguments by value, so that its state does not enter the register
// allocation of the pointwise phase.
template <class R, int DIM, int NS, bool MIX, bool VISC>
__device__ __noinline__ void boundary_record(const DGArgs<R> a, const GasParams g, int bf, int m,
                                             int nfp, const R* gq, int64_t gs, R n0, R n1, R n2,
                                             R* dst) {
  constexpr int NC = DIM + 2 + NS, TW = trace_width(NC);
  const R n[3] = {n0, n1, n2};
  const int64_t bstride = (int64_t)a.nbf * nfp, bo = (int64_t)bf * nfp + m;
  R qp[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) qp[c] = a.bext[c * bstride + bo];
  NodeState<R, DIM, NS> sp;
  make_state<R, DIM, NS>(qp, MIX ? a.bext[NC * bstride + bo] : R(0), g, sp);
  R fe[NC][DIM];
  inviscid_flux<R, DIM, NS>(sp, fe);
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int j = 0; j < DIM; ++j) fe[c][j] = -fe[c][j];
  if (VISC) {
    R gqv[NC][DIM], gt[DIM];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int j = 0; j < DIM; ++j) gqv[c][j] = gq[(c * DIM + j) * gs];
#pragma unroll
    for (int j = 0; j < DIM; ++j) gt[j] = gq[(NC * DIM + j) * gs];
    R fv[NC][DIM];
    viscous_flux<R, DIM, NS, MIX>(sp, gqv, gt, fv);
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int j = 0; j < DIM; ++j) fe[c][j] += fv[c][j];
  }
  R rec[TW];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    R acc = R(0);
#pragma unroll
    for (int j = 0; j < DIM; ++j) acc += fe[c][j] * n[j];
    rec[c] = -acc;
  }
  rec[NC] = wavespeed<R, DIM, NS>(sp);
  rec[NC + 1] = sp.p;
  rec[NC + 2] = sp.c;
  rec[NC + 3] = sp.gamma;
#pragma unroll
  for (int i = NC + 4; i < TW; ++i) rec[i] = R(0);
  store_rec<R, TW>(dst, m, rec);
#pragma unroll
  for (int c = 0; c < NC; ++c) a.bplus[c * bstride + bo] = qp[c];
}

// The exterior record of a Mengaldo boundary face node (neighbour
// convention) and its state_plus q into bplus.  The face kernel combines it
// with the interior record as for an interior face: central(F_V) from the
// pair gives F_V(state_bc, grad_cv_bc, grad_t_bc) . n when the exterior
// viscous part is 2 F_V,bc - F_V-; the inviscid part is the numerical flux
// between the interior state and state_plus (boundary.py:583-730).
template <class R, int DIM, int NS, bool MIX, bool VISC>
__device__ __noinline__ void mengaldo_record(const DGArgs<R> a, const GasParams g, int kind,
                                             int bf, int m, int nfp, int64_t EN, int64_t gm,
                                             const R* gq, int64_t gs, R n0, R n1, R n2, R* dst) {
  constexpr int NC = DIM + 2 + NS, TW = trace_width(NC);
  const R n[3] = {n0, n1, n2};
  R qm[NC];
  NodeState<R, DIM, NS> sm;
  boundary_minus<R, DIM, NS, MIX>(a, g, EN, gm, qm, sm);
  R par[NC + 1];
  const int64_t bstride = (int64_t)a.nbf * nfp, bo = (int64_t)bf * nfp + m;
#pragma unroll
  for (int c = 0; c <= NC; ++c) par[c] = bk_needs_bext(kind) ? a.bext[c * bstride + bo] : R(0);
  R qp[NC];
  bc_plus_cv<R, DIM, NS>(kind, g, qm, sm.t, sm.p, sm.c, sm.gamma, n, par, qp);
  // mixtures: the plus state's temperature re-solved from T- (the far field
  // state comes with its own)
  R tp = R(0);
  if (MIX) tp = (kind == BK_FARFIELD) ? par[NC] : node_temperature<R, DIM, NS>(qp, sm.t, g);
  NodeState<R, DIM, NS> sp;
  make_state<R, DIM, NS>(qp, tp, g, sp);
  R fip[NC];
  inviscid_flux_n<R, DIM, NS>(sp, n, fip);
  R rec[TW];
#pragma unroll
  for (int c = 0; c < NC; ++c) rec[c] = fip[c];
  if (VISC) {
    R qbc[NC];
    bc_state_cv<R, DIM, NS>(kind, g, qm, sm.t, sm.p, sm.c, sm.gamma, n, par, qbc);
    R tb = R(0);
    if (MIX) tb = (kind == BK_FARFIELD) ? par[NC] : node_temperature<R, DIM, NS>(qbc, sm.t, g);
    NodeState<R, DIM, NS> sb;
    make_state<R, DIM, NS>(qbc, tb, g, sb);
    R gqv[NC][DIM], gt[DIM];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int j = 0; j < DIM; ++j) gqv[c][j] = gq[(c * DIM + j) * gs];
#pragma unroll
    for (int j = 0; j < DIM; ++j) gt[j] = gq[(NC * DIM + j) * gs];
    R fvm[NC][DIM];
    viscous_flux<R, DIM, NS, MIX>(sm, gqv, gt, fvm);
    bc_gradients<R, DIM, NS>(kind, qm, qbc, n, gqv, gt);
    R fvb[NC][DIM];
    viscous_flux<R, DIM, NS, MIX>(sb, gqv, gt, fvb);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      R vb = R(0), vm = R(0);
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        vb += fvb[c][j] * n[j];
        vm += fvm[c][j] * n[j];
      }
      // -(F_V+ - F_I+) . n with F_V+ . n = 2 F_V,bc . n - F_V- . n
      rec[c] = -((R(2) * vb - vm) - fip[c]);
    }
  }
  rec[NC] = wavespeed<R, DIM, NS>(sp);
  rec[NC + 1] = sp.p;
  rec[NC + 2] = sp.c;
  rec[NC + 3] = sp.gamma;
#pragma unroll
  for (int i = NC + 4; i < TW; ++i) rec[i] = R(0);
  store_rec<R, TW>(dst, m, rec);
#pragma unroll
  for (int c = 0; c < NC; ++c) a.bplus[c * bstride + bo] = qp[c];
}

// Ask L2 for the 128-byte lines of [p, p + bytes), the work spread over the
// block's threads: the next tile's contiguous inputs are fetched while the
// current tile computes (prefetch.global.L2 does not block and takes no
// registers; a line already resident costs nothing).
__device__ __forceinline__ void prefetch_l2(const void* p, size_t bytes) {
  const uintptr_t a0 = reinterpret_cast<uintptr_t>(p) & ~uintptr_t(127);
  const uintptr_t a1 = reinterpret_cast<uintptr_t>(p) + bytes;
  for (uintptr_t a = a0 + (uintptr_t)threadIdx.x * 128; a < a1; a += (uintptr_t)blockDim.x * 128)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
}

// Face slots f * NFP + m of each volume node (-1: none), [NP][NF], in face
// order: one node per thread, every thread of a warp reading the same face
// node at a time.
template <int DIM, int ORDER>
__device__ __forceinline__ void fill_slots(int16_t* slot_s) {
  using S = Simplex<DIM, ORDER>;
  for (int k = threadIdx.x; k < S::NP; k += blockDim.x) {
    int n = 0;
    for (int fm = 0; fm < S::NF * S::NFP; ++fm)
      if (c_face_nodes<DIM, ORDER>(fm) == k) slot_s[k * S::NF + n++] = (int16_t)fm;
    for (; n < S::NF; ++n) slot_s[k * S::NF + n] = -1;
  }
}

// Volume kernel: gradients, pointwise fluxes, face-node records and the
// volume part of the divergence.  VISC false: the Euler operator (no
// gradient pass, F = -F_I).
template <class R, int DIM, int ORDER, int NS, bool MIX, bool VISC>
__global__ void __launch_bounds__((VCfg<R, DIM, ORDER, NS, MIX>::NT),
                                  (VCfg<R, DIM, ORDER, NS, MIX>::MINB))
    k_volume(DGArgs<R> a, GasParams g) {
  using V = VCfg<R, DIM, ORDER, NS, MIX>;
  using S = Simplex<DIM, ORDER>;
  constexpr int NP = V::NP, NF = V::NF, NFP = V::NFP, NFN = V::NFN, NC = V::NC, NU = V::NU;
  constexpr int EPB = V::EPB, MP = V::MP, MT = V::MT, NAC = V::NAC, MROW = V::MROW;
  constexpr int KU = V::KU, KS = V::KS, KL = V::KL, NFPK = V::NFPK, KUR = V::KUR;
  constexpr int NCOL = V::NCOL, NCOLD = V::NCOLD, NNODE = V::NNODE;
  constexpr int GST = V::GST, FST = V::FST, TW = V::TW;
  constexpr int AWN = DIM * MP * KU, ALN = NF * MP * KL;
  constexpr int ENP = EPB * NP;
  static_assert(NCOL * (KU + KS) <= V::W1 && NNODE * FST + NS * ENP <= V::W1, "work region");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* aw = reinterpret_cast<R*>(smem_raw);                  // [NAC][DIM][MP][KU]
  R* al = aw + NAC * AWN;                                  // [NAC][NF][MP][KL]
  R* w1 = al + NAC * ALN;                                  // work region
  R* bu = w1;                                              //   [NCOL][KU]  (gradient pass)
  R* bs = bu + NCOL * KU;                                  //   [NCOL][KS]  (gradient pass)
  R* gfl = w1;                                             //   [NNODE][FST] (after it)
  R* src_s = w1 + NNODE * FST;                             //   [NS][ENP]
  R* gn = w1 + V::W1;                                      // [NNODE][GST] gradients
  R* rx_s = gn + NNODE * GST;                              // [EPB][DIM][DIM]
  R* nrm_s = rx_s + EPB * DIM * DIM;                       // [EPB][NF][DIM]
  R* fs_s = nrm_s + EPB * NF * DIM;                        // [EPB][NF]
  R* u0_s = fs_s + EPB * NF;                               // [NU][EPB]
  int* fn_s = reinterpret_cast<int*>(u0_s + NU * EPB);     // [NFN]
  int32_t* conn_s = fn_s + NFN;                            // [EPB][NF]
  int16_t* slot_s = reinterpret_cast<int16_t*>(conn_s + EPB * NF);   // [NP][NF]
  uint8_t* perm_s = reinterpret_cast<uint8_t*>(slot_s + NP * NF);

  const int E = a.nelem;
  const int64_t EN = (int64_t)E * NP;
  const bool sources = MIX && a.add_sources;
  const bool rows16 =
      ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.t_op)) & 15) == 0 &&
      (KU * sizeof(R)) % 16 == 0;

  // operators W(H)_r (gradient and divergence) and LIFT_f (gradient), zero padded
  for (int i = threadIdx.x; i < AWN; i += blockDim.x) {
    const int r = i / (MP * KU), row = (i / KU) % MP, k = i % KU;
    put_a<R>(aw, AWN, i, (row < NP && k < NP) ? refop(S::template OFF_WDIV<R> + (r * NP + row) * NP + k) : 0.0);
  }
  if (VISC)
    for (int i = threadIdx.x; i < ALN; i += blockDim.x) {
      const int f = i / (MP * KL), row = (i / KL) % MP, m = i % KL;
      put_a<R>(al, ALN, i,
               (row < NP && m < NFP) ? refop(S::OFF_LIFT + row * NFN + f * NFP + m) : 0.0);
    }
  for (int i = threadIdx.x; i < V::W1 + NNODE * GST; i += blockDim.x) w1[i] = R(0);
  for (int i = threadIdx.x; i < NFN; i += blockDim.x) fn_s[i] = c_face_nodes<DIM, ORDER>(i);
  for (int i = threadIdx.x; i < a.nperm * NFP; i += blockDim.x) perm_s[i] = a.perm[i];
  fill_slots<DIM, ORDER>(slot_s);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int nwarps = blockDim.x >> 5;
  constexpr int NACC = V::TF32 ? 4 : 2;
  const int ntiles = (a.nowned + EPB - 1) / EPB;
  bool bad = false;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int e0 = tile * EPB;
    const int ne = imin(EPB, a.nowned - e0);
    // the previous tile's last phase reads the work region, src_s and the
    // geometry, which this tile overwrites
    __syncthreads();
    stage_conn<NF>(a.conn, e0, ne, conn_s);
    load_geometry<R, DIM, ORDER>(a.rx, e0, ne, rx_s, nrm_s, fs_s);
    // the normals and face factors load_geometry computes last are read by
    // other threads in every phase below (the Euler operator goes straight
    // to the pointwise phase)
    __syncthreads();

    if constexpr (VISC) {
      // ---- gradient pass (as k_grad), results into gn
      bool rows_done = false;
      if constexpr (MIX && NP % 4 == 0 && sizeof(R) == 4) {
        if (rows16) {
          for (int it = threadIdx.x; it < ne * NU; it += blockDim.x) {
            const int e = it % ne, c = it / ne;
            const float* src = (c < NC ? a.q + c * EN : a.t_op) + (int64_t)(e0 + e) * NP;
            float4 v[NP / 4];
#pragma unroll
            for (int i = 0; i < NP / 4; ++i) v[i] = reinterpret_cast<const float4*>(src)[i];
            const float u0 = v[0].x;
            float4* dst = reinterpret_cast<float4*>(bu + (c * EPB + e) * KU);
#pragma unroll
            for (int i = 0; i < NP / 4; ++i)
              dst[i] = make_float4(v[i].x - u0, v[i].y - u0, v[i].z - u0, v[i].w - u0);
            u0_s[c * EPB + e] = u0;
          }
          rows_done = true;
        }
      }
      if (!rows_done) {
        for (int idx = threadIdx.x; idx < ne * NP; idx += blockDim.x) {
          const int e = idx / NP, k = idx % NP;
          const int64_t gnd = (int64_t)e0 * NP + idx, g0 = (int64_t)(e0 + e) * NP;
          R qq[NC], q0[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            qq[c] = a.q[c * EN + gnd];
            q0[c] = a.q[c * EN + g0];
          }
          const R t = MIX ? a.t_op[gnd] : node_temperature<R, DIM, NS>(qq, R(0), g);
          const R t0 = MIX ? a.t_op[g0] : node_temperature<R, DIM, NS>(q0, R(0), g);
#pragma unroll
          for (int c = 0; c < NC; ++c) bu[(c * EPB + e) * KU + k] = qq[c] - q0[c];
          bu[(NC * EPB + e) * KU + k] = t - t0;
          if (k == 0) {
#pragma unroll
            for (int c = 0; c < NC; ++c) u0_s[c * EPB + e] = q0[c];
            u0_s[NC * EPB + e] = t0;
          }
        }
      }
      __syncthreads();

      // face values fscale * (u* - u0), one face node per item
      for (int fnode = threadIdx.x; fnode < ne * NFN; fnode += blockDim.x) {
        const int e = fnode / NFN, fm = fnode % NFN, f = fm / NFP, m = fm % NFP;
        const int k = fn_s[fm];
        const int cn = conn_s[e * NF + f];
        const R fsc = fs_s[e * NF + f];
        int mode = 2;      // 0 two-sided average, 1 prescribed exterior, 2 interior value
        int64_t gi = 0;
        int bf = 0;
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
          int kind = (bf < a.nbf) ? a.bkind[bf] : -1;
          if ((bk_needs_bext(kind) && !a.bext) || kind > BK_OUTFLOW) kind = -1;
          if (kind == BK_PRESCRIBED) {
            mode = 1;
          } else if (bk_mengaldo(kind)) {
            mode = 3;
          } else if (kind < 0) {
            atomicOr(a.status, ST_BAD_INDEX);
          }
        }
        R* bcol = bs + e * KS + f * NFPK + m;
        if (mode == 2) {
#pragma unroll
          for (int c = 0; c < NU; ++c)
            bcol[c * EPB * KS] = (folds<R>() ? fsc * R(0.5) : fsc) * bu[(c * EPB + e) * KU + k];
          continue;
        }
        const int64_t bstride = (int64_t)a.nbf * NFP, bo = (int64_t)bf * NFP + m;
        R up[NU];
        if (mode == 3) {
          const R* nf = nrm_s + (e * NF + f) * DIM;
          mengaldo_grad_value<R, DIM, NS, MIX>(a, g, a.bkind[bf], bf, m, NFP, EN,
                                               (int64_t)(e0 + e) * NP + k, nf[0], nf[1],
                                               DIM > 2 ? nf[DIM - 1] : R(0), up);
          mode = 1;
        } else {
#pragma unroll
          for (int c = 0; c < NC; ++c)
            up[c] = (mode == 0) ? a.q[c * EN + gi] : a.bext[c * bstride + bo];
          if (MIX)
            up[NC] = (mode == 0) ? a.t_op[gi] : a.bext[NC * bstride + bo];
          else
            up[NC] = node_temperature<R, DIM, NS>(up, R(0), g);
        }
#pragma unroll
        for (int c = 0; c < NU; ++c) {
          const R um = bu[(c * EPB + e) * KU + k];
          const R du = up[c] - u0_s[c * EPB + e];
          R v;
          if constexpr (folds<R>())
            v = (mode == 0) ? du * R(0.5) : du - um * R(0.5);
          else
            v = (mode == 0) ? (du + um) * R(0.5) : du;
          bcol[c * EPB * KS] = fsc * v;
        }
      }
      __syncthreads();

      // the next tile's rows of q and the temperatures, its geometry and
      // face pairing, into L2 while this tile computes
      {
        const int tn = tile + gridDim.x;
        if (tn < ntiles) {
          const int e1 = tn * EPB, n1 = imin(EPB, a.nowned - e1);
          const size_t row = (size_t)n1 * NP * sizeof(R);
          for (int c = 0; c < NC; ++c) prefetch_l2(a.q + c * EN + (int64_t)e1 * NP, row);
          if (MIX) prefetch_l2(a.t_op + (int64_t)e1 * NP, row);
          if (MIX && a.add_sources) prefetch_l2(a.t_src + (int64_t)e1 * NP, row);
          prefetch_l2(a.rx + (int64_t)e1 * DIM * DIM, (size_t)n1 * DIM * DIM * sizeof(R));
          prefetch_l2(a.conn + (int64_t)e1 * NF, (size_t)n1 * NF * 4);
        }
      }

      // contraction and metric combination into gn[node][c * DIM + j]
      for (int w = warp; w < (NCOL / 8) * MT; w += nwarps) {
        const int nt = w / MT, t = w % MT;
        R du[DIM][NACC], lf[NF][NACC];
#pragma unroll
        for (int v = 0; v < NACC; ++v) {
#pragma unroll
          for (int r = 0; r < DIM; ++r) du[r][v] = R(0);
#pragma unroll
          for (int f = 0; f < NF; ++f) lf[f][v] = R(0);
        }
        const R* bcol = bu + (nt * 8 + gq) * KU + tq;
        const R* scol = bs + (nt * 8 + gq) * KS + tq;
        if constexpr (!V::TF32) {
#pragma unroll
          for (int ks = 0; ks < KUR / 4; ++ks) {
            const double b = bcol[ks * 4];
#pragma unroll
            for (int r = 0; r < DIM; ++r)
              dmma884(du[r], aw[(r * MP + t * 8 + gq) * KU + ks * 4 + tq], b);
          }
#pragma unroll
          for (int f = 0; f < NF; ++f)
#pragma unroll
            for (int ks = 0; ks < NFPK / 4; ++ks)
              dmma884(lf[f], al[(f * MP + t * 8 + gq) * KL + ks * 4 + tq], scol[f * NFPK + ks * 4]);
        } else {
#pragma unroll
          for (int ks = 0; ks < KUR / 8; ++ks) {
            const SplitB b(bcol[ks * 8], bcol[ks * 8 + 4]);
#pragma unroll
            for (int r = 0; r < DIM; ++r) {
              uint32_t ah[4], alo[4];
              load_a_tf32_ldsm(ah, aw + r * MP * KU, KU, t * 16, ks * 8, lane);
              load_a_tf32_ldsm(alo, aw + AWN + r * MP * KU, KU, t * 16, ks * 8, lane);
              mma_tf32x3(du[r], ah, alo, b);
            }
          }
#pragma unroll
          for (int f = 0; f < NF; ++f)
#pragma unroll
            for (int ks = 0; ks < NFPK / 8; ++ks) {
              const SplitB b(scol[f * NFPK + ks * 8], scol[f * NFPK + ks * 8 + 4]);
              uint32_t ah[4], alo[4];
              load_a_tf32_ldsm(ah, al + f * MP * KL, KL, t * 16, ks * 8, lane);
              load_a_tf32_ldsm(alo, al + ALN + f * MP * KL, KL, t * 16, ks * 8, lane);
              mma_tf32x3(lf[f], ah, alo, b);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = nt * 8 + 2 * tq + h;
          const int c = col / EPB, e = col % EPB;
          if (c >= NU || e >= ne) continue;
          R rxe[DIM][DIM], nre[NF][DIM];
#pragma unroll
          for (int r = 0; r < DIM; ++r)
#pragma unroll
            for (int j = 0; j < DIM; ++j) rxe[r][j] = rx_s[e * DIM * DIM + r * DIM + j];
#pragma unroll
          for (int f = 0; f < NF; ++f)
#pragma unroll
            for (int j = 0; j < DIM; ++j) nre[f][j] = nrm_s[(e * NF + f) * DIM + j];
#pragma unroll
          for (int half = 0; half < NACC / 2; ++half) {
            const int i = t * MROW + gq + 8 * half;
            if (i >= NP) continue;
            const int v = 2 * half + h;
#pragma unroll
            for (int j = 0; j < DIM; ++j) {
              R gsum = R(0);
#pragma unroll
              for (int f = 0; f < NF; ++f) gsum += nre[f][j] * lf[f][v];
#pragma unroll
              for (int r = 0; r < DIM; ++r) gsum -= rxe[r][j] * du[r][v];
              gn[(e * NP + i) * GST + c * DIM + j] = gsum;
              if (a.grad_out)
                a.grad_out[((int64_t)c * DIM + j) * EN + (int64_t)(e0 + e) * NP + i] = gsum;
            }
          }
        }
      }
      // every contraction has read bu/bs (the region gfl and src_s reuse)
      // and every gradient is in gn
      __syncthreads();
    }

    // ---- pointwise: fluxes, records, sources; G_r into gfl[node][c * DIM + r]
    for (int n = threadIdx.x; n < ne * NP; n += blockDim.x) {
      const int e = n / NP, k = n % NP;
      const int64_t gnd = (int64_t)(e0 + e) * NP + k;
      R qq[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) qq[c] = a.q[c * EN + gnd];
      NodeState<R, DIM, NS> st;
      make_state<R, DIM, NS>(qq, MIX ? a.t_op[gnd] : R(0), g, st);
      R fl[NC][DIM];
      inviscid_flux<R, DIM, NS>(st, fl);
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int j = 0; j < DIM; ++j) fl[c][j] = -fl[c][j];
      if constexpr (VISC) {
        // the gradients are read from the node's shared-memory row where the
        // viscous flux uses them (no register copy of all (NC+1) DIM values)
        const R* gr = gn + n * GST;
        R fv[NC][DIM];
        viscous_flux<R, DIM, NS, MIX>(st, reinterpret_cast<const R(*)[DIM]>(gr), gr + NC * DIM,
                                      fv);
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < DIM; ++j) fl[c][j] = fv[c][j] + fl[c][j];
      }
      bad |= !(st.p == st.p) || !(st.c == st.c);
      const R* rxe = rx_s + e * DIM * DIM;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          R acc = R(0);
#pragma unroll
          for (int j = 0; j < DIM; ++j) acc += rxe[r * DIM + j] * fl[c][j];
          gfl[n * FST + c * DIM + r] = acc;
        }
      if constexpr (MIX && NS > 0) {
        if (sources) {
          R om[NS];
          production_rates<R, NS>(st.rho, a.t_src[gnd], st.y, (R)g.zero_level, om);
#pragma unroll
          for (int s = 0; s < NS; ++s) src_s[s * ENP + n] = mech<R>().mw[s] * om[s];
        }
      }
      R v2 = R(0);
#pragma unroll
      for (int j = 0; j < DIM; ++j) v2 += st.v[j] * st.v[j];
      const R lam = sqrt(v2) + st.c;
      if constexpr (folds<R>()) a.lam[gnd] = lam;
      // one record per face slot of this node
#pragma unroll 1
      for (int sl = 0; sl < NF; ++sl) {
        const int fm = slot_s[k * NF + sl];
        if (fm < 0) break;
        const int f = fm / NFP;
        const R* nf = nrm_s + (e * NF + f) * DIM;
        R rec[TW];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          R acc = R(0);
#pragma unroll
          for (int j = 0; j < DIM; ++j) acc += fl[c][j] * nf[j];
          rec[c] = acc;
        }
        rec[NC] = lam;
        rec[NC + 1] = st.p;
        rec[NC + 2] = st.c;
        rec[NC + 3] = st.gamma;
#pragma unroll
        for (int i = NC + 4; i < TW; ++i) rec[i] = R(0);
        store_rec<R, TW>(a.trace + ((int64_t)(e0 + e) * NFN + fm) * TW, fm, rec);
      }
      if (k == 0) {
        // element-constant shift of the face terms: F0 . n_f, every face
        R* s0e = a.s0 + (int64_t)(e0 + e) * NF * NC;
#pragma unroll 1
        for (int f = 0; f < NF; ++f) {
          const R* nf = nrm_s + (e * NF + f) * DIM;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            R acc = R(0);
#pragma unroll
            for (int j = 0; j < DIM; ++j) acc += fl[c][j] * nf[j];
            s0e[f * NC + c] = acc;
          }
        }
      }
    }
    // exterior records of the tile's boundary face nodes, in a loop of their
    // own: out of line calls inside the pointwise loop would make the
    // compiler spill that loop's registers around them for every node
    for (int fnode = threadIdx.x; fnode < ne * NFN; fnode += blockDim.x) {
      const int e = fnode / NFN, fm = fnode % NFN, f = fm / NFP, m = fm % NFP;
      const int cn = conn_s[e * NF + f];
      if (cn >= 0) continue;
      const int bf = -(cn + 1);
      const int kind = (bf < a.nbf) ? a.bkind[bf] : -1;
      if ((bk_needs_bext(kind) && !a.bext) || (kind != BK_PRESCRIBED && !bk_mengaldo(kind)))
        continue;
      const int k = fn_s[fm];
      const int n = e * NP + k;
      const R* nf = nrm_s + (e * NF + f) * DIM;
      R* dst = a.btrace + ((int64_t)bf * NFP + m) * TW;
      if (kind == BK_PRESCRIBED)
        boundary_record<R, DIM, NS, MIX, VISC>(a, g, bf, m, NFP, VISC ? gn + n * GST : nullptr,
                                               1, nf[0], nf[1], DIM > 2 ? nf[DIM - 1] : R(0),
                                               dst);
      else
        mengaldo_record<R, DIM, NS, MIX, VISC>(a, g, kind, bf, m, NFP, EN,
                                               (int64_t)(e0 + e) * NP + k,
                                               VISC ? gn + n * GST : nullptr, 1, nf[0], nf[1],
                                               DIM > 2 ? nf[DIM - 1] : R(0), dst);
    }
    __syncthreads();

    // ---- volume divergence: rhs = -sum_r W_r (G_r - G0_r) (+ sources); one
    // m-tile and NTG n-tiles per warp item.  Column col = c * EPB + e reads
    // node rows of element e; rows k >= NP of the operator are zero, so the
    // padded k reach into the next rows harmlessly (finite, zero-filled).
    constexpr int NNT = NCOLD / 8;
    constexpr int NTG = (NNT % 3 == 0) ? 3 : ((NNT % 2 == 0) ? 2 : 1);
    for (int w = warp; w < (NNT / NTG) * MT; w += nwarps) {
      const int ngp = w / MT, t = w % MT;
      R d[NTG][NACC];
#pragma unroll
      for (int u = 0; u < NTG; ++u)
#pragma unroll
        for (int v = 0; v < NACC; ++v) d[u][v] = R(0);
      // this lane's B column per n-tile: element row base and field offset
      int cbase[NTG];
#pragma unroll
      for (int u = 0; u < NTG; ++u) {
        const int col = (ngp * NTG + u) * 8 + gq;
        const int c = col / EPB, e = col % EPB;
        cbase[u] = (c < NC) ? (e * NP) * FST + c * DIM : -1;
      }
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
        R g0[NTG];
#pragma unroll
        for (int u = 0; u < NTG; ++u) g0[u] = cbase[u] >= 0 ? gfl[cbase[u] + r] : R(0);
        if constexpr (!V::TF32) {
#pragma unroll
          for (int ks = 0; ks < KUR / 4; ++ks) {
            const double av = aw[(r * MP + t * 8 + gq) * KU + ks * 4 + tq];
            const int kk = ks * 4 + tq;
#pragma unroll
            for (int u = 0; u < NTG; ++u) {
              const double b = cbase[u] >= 0 ? gfl[cbase[u] + kk * FST + r] - g0[u] : 0.0;
              dmma884(d[u], av, b);
            }
          }
        } else {
#pragma unroll
          for (int ks = 0; ks < KUR / 8; ++ks) {
            uint32_t ah[4], alo[4];
            load_a_tf32_ldsm(ah, aw + r * MP * KU, KU, t * 16, ks * 8, lane);
            load_a_tf32_ldsm(alo, aw + AWN + r * MP * KU, KU, t * 16, ks * 8, lane);
            const int k0 = ks * 8 + tq;
#pragma unroll
            for (int u = 0; u < NTG; ++u) {
              float b0 = 0.f, b1 = 0.f;
              if (cbase[u] >= 0) {
                b0 = gfl[cbase[u] + k0 * FST + r] - g0[u];
                b1 = gfl[cbase[u] + (k0 + 4) * FST + r] - g0[u];
              }
              mma_tf32x3(d[u], ah, alo, b0, b1);
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < NTG; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = (ngp * NTG + u) * 8 + 2 * tq + h;
          const int c = col / EPB, e = col % EPB;
          if (c >= NC || e >= ne) continue;
          R* outp = a.out + (int64_t)c * EN + (int64_t)(e0 + e) * NP;
#pragma unroll
          for (int half = 0; half < NACC / 2; ++half) {
            const int i = t * MROW + gq + 8 * half;
            if (i >= NP) continue;
            R v = -d[u][2 * half + h];
            if (sources && c >= 2 + DIM) v += src_s[(c - 2 - DIM) * ENP + e * NP + i];
            outp[i] = v;
          }
        }
    }
  }
  if (bad) atomicOr(a.status, ST_NAN);
}

// Flux-volume kernel: the pointwise phase and the volume divergence of
// k_volume with the gradients read from HBM (written by the gradient kernel),
// for the three-kernel pass gradient -> flux-volume -> face.
//
// STAGED: the tile's inputs (NC fields, temperatures, (NC+1) DIM gradients: one
// contiguous row of EPB * NP values each) are brought into shared memory by
// bulk copies (cp.async.bulk), issued as soon as the previous tile's pointwise
// phase has read its own and running under that tile's divergence; its
// geometry is computed in the same window into a second buffer.  A node's
// thread then reads them where the flux needs them: no address arithmetic, no
// registers held for loads in flight, no wait for DRAM at the start of a tile.
// Measured: float64 32^3 p3 2.57 -> 2.46 ms, float32 1260 tetrahedra 23.5 ->
// 20.2 us; float32 64^3 p3 is the same with and without (7.46 ms).
// Not STAGED: rows that bulk copies cannot move (flux_rows_aligned: a row start
// off 16 bytes, as with an unaligned caller's pointer, an odd number of float32
// order-2 elements, 2-D float32 orders 1 and 4) are read from global memory by
// the node's thread.  Right-hand side of the 7-species mixture, float32, threads
// copying such rows into shared memory -> direct reads: 2-D order 4, 301 x 299
// cells 1.83 -> 0.99 ms; order 2, 27 x 25 x 25 cells, offset by one value 1.15 ->
// 0.66 ms.
template <class R, int DIM, int ORDER, int NS, bool MIX, bool VISC, bool STAGED>
__global__ void __launch_bounds__((VCfg<R, DIM, ORDER, NS, MIX>::NT3), 2)
    k_flux_volume(DGArgs<R> a, GasParams g) {
  using V = VCfg<R, DIM, ORDER, NS, MIX>;
  using S = Simplex<DIM, ORDER>;
  constexpr int NP = V::NP, NF = V::NF, NFP = V::NFP, NFN = V::NFN, NC = V::NC;
  constexpr int EPB = V::epb3(STAGED), MT = V::MT, MROW = V::MROW;
  constexpr int KU = V::KU, KUR = V::KUR, NCOLD = round_up(NC * EPB, 8), NNODE = V::nnode3(EPB);
  constexpr int FST = V::FST, TW = V::TW, GEO = V::GEO3, DD = DIM * DIM;
  constexpr int AWN = DIM * NP * KU;
  constexpr int ENP = EPB * NP;
  constexpr int NROW = STAGED ? V::rows3(VISC) : 0, RST = round_up(ENP * (int)sizeof(R), 16) / (int)sizeof(R);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* aw = reinterpret_cast<R*>(smem_raw);                  // [NAC][DIM][NP][KU]
  R* gfl = aw + V::A_FLUX;                                 // [NNODE][FST]
  R* src_s = gfl + NNODE * FST;                            // [NS][ENP]
  R* geo_s = src_s + NS * ENP;                             // [2][EPB][GEO]
  R* f0_s = geo_s + 2 * EPB * GEO;                         // [EPB][NC * DIM] node-0 fluxes
  R* row_s = aw + round_up(V::A_FLUX + NNODE * FST + NS * ENP + 2 * EPB * GEO + EPB * NC * DIM,
                           4);                             // [NROW][RST]
  int* fn_s = reinterpret_cast<int*>(row_s + NROW * RST);  // [NFN]
  int32_t* conn_s = fn_s + NFN;                            // [2][EPB][NF]
  int16_t* slot_s = reinterpret_cast<int16_t*>(conn_s + 2 * EPB * NF);   // [NP][NF]
  __shared__ __align__(8) uint64_t staged;                 // the tile's rows have landed

  const int64_t EN = (int64_t)a.nelem * NP;
  const bool sources = MIX && a.add_sources;
  // float32 drivers pass one temperature for both uses
  const bool own_src = sources && a.t_src != a.t_op;
  auto row_ptr = [&](int i) -> const R* {
    if (i < NC) return a.q + i * EN;
    if (MIX && i < V::ROW_G) return i == V::ROW_T ? a.t_op : (own_src ? a.t_src : nullptr);
    return a.grad + (i - V::ROW_G) * EN;
  };
  // input *i* of node *gnd*, the tile's node *n*
  auto value = [&](int i, int n, int64_t gnd) -> R {
    if constexpr (STAGED)
      return row_s[i * RST + n];
    else
      return row_ptr(i)[gnd];
  };
  const int ntiles = (a.nowned + EPB - 1) / EPB;
  // rows of tile *tl*: bulk copies by warp 0, what is left of a last tile's rows
  // (less than 16 bytes each) by all threads
  auto stage_rows = [&](int tl) {
    const int64_t n0 = (int64_t)tl * ENP;
    const int n = imin(ENP, (int)((int64_t)a.nowned * NP - n0));
    const uint32_t bytes = (uint32_t)(n * sizeof(R)) & ~15u;
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0)
        mbar_expect(&staged, bytes * (uint32_t)(NROW - (MIX && !own_src ? 1 : 0)));
      __syncwarp();
      for (int i = threadIdx.x; i < NROW; i += 32) {
        const R* p = row_ptr(i);
        if (p && bytes) bulk_load(row_s + i * RST, p + n0, bytes, &staged);
      }
    }
    const int done_n = bytes / (int)sizeof(R);
    if (done_n < n) {
      const int m = n - done_n;
      for (int i = threadIdx.x; i < NROW * m; i += blockDim.x) {
        const R* p = row_ptr(i / m);
        if (p) row_s[(i / m) * RST + done_n + i % m] = p[n0 + done_n + i % m];
      }
    }
  };
  // geometry and face pairing of tile *tl* into buffer *b*, by the threads
  // [t0, t0 + nt): metric and unit normals as load_geometry computes them
  auto geometry = [&](int tl, int b, int t0, int nt) {
    const int e1 = tl * EPB, n1 = imin(EPB, a.nowned - e1);
    R* gb = geo_s + b * EPB * GEO;
    for (int i = (int)threadIdx.x - t0; i < n1 * NF; i += nt) {
      if (i < 0) break;
      const int e = i / NF, f = i % NF;
      conn_s[b * EPB * NF + i] = a.conn[(int64_t)e1 * NF + i];
      const R* rxg = a.rx + (int64_t)(e1 + e) * DD;
      R rx[DD];
#pragma unroll
      for (int k = 0; k < DD; ++k) rx[k] = rxg[k];
      R nv[DIM], mag2 = 0;
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        R s = 0;
#pragma unroll
        for (int r = 0; r < DIM; ++r)
          s += rx[r * DIM + j] * RefBank<R>::get(S::OFF_NREF + f * DIM + r);
        nv[j] = s;
        mag2 += s * s;
      }
      const R mag = sqrt(mag2);
#pragma unroll
      for (int j = 0; j < DIM; ++j) gb[e * GEO + DD + f * DIM + j] = nv[j] / mag;
      if (f == 0) {
#pragma unroll
        for (int k = 0; k < DD; ++k) gb[e * GEO + k] = rx[k];
      }
    }
  };

  if (STAGED && threadIdx.x == 0) {
    mbar_init(&staged, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < AWN; i += blockDim.x) {
    const int k = i % KU, row = i / KU;                    // row = r * NP + output node
    put_a<R>(aw, AWN, i, k < NP ? refop(S::template OFF_WDIV<R> + row * NP + k) : 0.0);
  }
  for (int i = threadIdx.x; i < NNODE * FST + NS * ENP; i += blockDim.x) gfl[i] = R(0);
  for (int i = threadIdx.x; i < NFN; i += blockDim.x) fn_s[i] = c_face_nodes<DIM, ORDER>(i);
  fill_slots<DIM, ORDER>(slot_s);
  __syncthreads();
  if ((int)blockIdx.x < ntiles) {
    if constexpr (STAGED) stage_rows(blockIdx.x);
    geometry(blockIdx.x, 0, 0, blockDim.x);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int nwarps = blockDim.x >> 5;
  constexpr int NACC = V::TF32 ? 4 : 2;
  bool bad = false;
  int it = 0;
  bool timeout = false;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
    const int b = it & 1;
    const int e0 = tile * EPB;
    const int ne = imin(EPB, a.nowned - e0);
    const R* gb = geo_s + b * EPB * GEO;
    // the previous tile's divergence has read gfl and src_s; this tile's
    // geometry is complete
    __syncthreads();
    const bool ok = !STAGED || mbar_wait(&staged, it & 1, nullptr);

    // one node per thread (as a loop: 1 % of the float32 order-3 right-hand side
    // slower, 2 % of the order-2 one)
    static_assert(ENP <= V::NT3, "one node per thread");
    if (const int n = threadIdx.x; n < ne * NP && ok) {
      const int e = n / NP, k = n % NP;
      const int64_t gnd = (int64_t)(e0 + e) * NP + k;
      R qq[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) qq[c] = value(c, n, gnd);
      NodeState<R, DIM, NS> st;
      make_state<R, DIM, NS>(qq, MIX ? value(V::ROW_T, n, gnd) : R(0), g, st);
      R fl[NC][DIM];
      inviscid_flux<R, DIM, NS>(st, fl);
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int j = 0; j < DIM; ++j) fl[c][j] = -fl[c][j];
      if constexpr (VISC) {
        R gqv[NC][DIM], gt[DIM];
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < DIM; ++j) gqv[c][j] = value(V::ROW_G + c * DIM + j, n, gnd);
#pragma unroll
        for (int j = 0; j < DIM; ++j) gt[j] = value(V::ROW_G + NC * DIM + j, n, gnd);
        R fv[NC][DIM];
        viscous_flux<R, DIM, NS, MIX>(st, gqv, gt, fv);
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < DIM; ++j) fl[c][j] = fv[c][j] + fl[c][j];
      }
      bad |= !(st.p == st.p) || !(st.c == st.c);
      const R* rxe = gb + e * GEO;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          R acc = R(0);
#pragma unroll
          for (int j = 0; j < DIM; ++j) acc += rxe[r * DIM + j] * fl[c][j];
          gfl[n * FST + c * DIM + r] = acc;
        }
      if constexpr (MIX && NS > 0) {
        if (sources) {
          R om[NS];
          const R ts = STAGED ? row_s[(own_src ? V::ROW_T + 1 : V::ROW_T) * RST + n] : a.t_src[gnd];
          production_rates<R, NS>(st.rho, ts, st.y, (R)g.zero_level, om);
#pragma unroll
          for (int sp = 0; sp < NS; ++sp) src_s[sp * ENP + n] = mech<R>().mw[sp] * om[sp];
        }
      }
      R v2 = R(0);
#pragma unroll
      for (int j = 0; j < DIM; ++j) v2 += st.v[j] * st.v[j];
      const R lam = sqrt(v2) + st.c;
      if constexpr (folds<R>()) a.lam[gnd] = lam;
#pragma unroll 1
      for (int sl = 0; sl < NF; ++sl) {
        const int fm = slot_s[k * NF + sl];
        if (fm < 0) break;
        const R* nf = gb + e * GEO + DD + (fm / NFP) * DIM;
        R rec[TW];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          R acc = R(0);
#pragma unroll
          for (int j = 0; j < DIM; ++j) acc += fl[c][j] * nf[j];
          rec[c] = acc;
        }
        rec[NC] = lam;
        rec[NC + 1] = st.p;
        rec[NC + 2] = st.c;
        rec[NC + 3] = st.gamma;
#pragma unroll
        for (int i = NC + 4; i < TW; ++i) rec[i] = R(0);
        store_rec<R, TW>(a.trace + ((int64_t)(e0 + e) * NFN + fm) * TW, fm, rec);
      }
      if (k == 0) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < DIM; ++j) f0_s[e * NC * DIM + c * DIM + j] = fl[c][j];
      }
    }
    // exterior records of the tile's boundary face nodes (own loop: see k_volume)
    if (a.nbf > 0) {
      for (int fnode = threadIdx.x; fnode < ne * NFN && ok; fnode += blockDim.x) {
        const int e = fnode / NFN, fm = fnode % NFN, f = fm / NFP, m = fm % NFP;
        const int cn = conn_s[(b * EPB + e) * NF + f];
        if (cn >= 0) continue;
        const int bf = -(cn + 1);
        const int kind = (bf < a.nbf) ? a.bkind[bf] : -1;
        if ((bk_needs_bext(kind) && !a.bext) || (kind != BK_PRESCRIBED && !bk_mengaldo(kind)))
          continue;
        const int64_t gnd = (int64_t)(e0 + e) * NP + fn_s[fm];
        const R* nf = gb + e * GEO + DD + f * DIM;
        R* dst = a.btrace + ((int64_t)bf * NFP + m) * TW;
        if (kind == BK_PRESCRIBED)
          boundary_record<R, DIM, NS, MIX, VISC>(a, g, bf, m, NFP, VISC ? a.grad + gnd : nullptr,
                                                 EN, nf[0], nf[1], DIM > 2 ? nf[DIM - 1] : R(0),
                                                 dst);
        else
          mengaldo_record<R, DIM, NS, MIX, VISC>(a, g, kind, bf, m, NFP, EN, gnd,
                                                 VISC ? a.grad + gnd : nullptr, EN, nf[0], nf[1],
                                                 DIM > 2 ? nf[DIM - 1] : R(0), dst);
      }
    }
    // gfl and the sources are complete, the staged rows have been read
    if constexpr (STAGED) {
      if (__syncthreads_or(!ok)) {
        timeout = true;
        break;
      }
    } else {
      __syncthreads();
    }
    if (tile + (int)gridDim.x < ntiles) {
      if constexpr (STAGED) stage_rows(tile + gridDim.x);
      // by the last warps, which have the least divergence work
      geometry(tile + gridDim.x, b ^ 1, blockDim.x - 64, 64);
    }
    // element-constant shift of the face terms, F0 . n of every face, by the
    // same warps (by the node-0 threads it took each warp ~350 instructions
    // for one or two lanes)
    for (int i = (int)threadIdx.x - (int)blockDim.x + 64; i >= 0 && i < ne * NF * NC; i += 64) {
      const int c = i % NC, f = (i / NC) % NF, e = i / (NC * NF);
      const R* f0 = f0_s + (e * NC + c) * DIM;
      const R* nf = gb + e * GEO + DD + f * DIM;
      R acc = R(0);
#pragma unroll
      for (int j = 0; j < DIM; ++j) acc += f0[j] * nf[j];
      a.s0[(int64_t)e0 * NF * NC + i] = acc;
    }

    // volume divergence.  float32: one item per group of NTG column tiles
    // and every m-tile, so each shifted flux value is read and split into
    // its tf32 hi/lo words once
    constexpr int NNT = NCOLD / 8;
    constexpr int NTG = (NNT % 3 == 0) ? 3 : ((NNT % 2 == 0) ? 2 : 1);
    if constexpr (V::TF32) {
      for (int w = warp; w < NNT / NTG; w += nwarps) {
        const int ngp = w;
        float d[MT][NTG][NACC];
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
          for (int u = 0; u < NTG; ++u)
#pragma unroll
            for (int v = 0; v < NACC; ++v) d[t][u][v] = 0.f;
        int cbase[NTG];
#pragma unroll
        for (int u = 0; u < NTG; ++u) {
          const int col = (ngp * NTG + u) * 8 + gq;
          const int c = col / EPB, e = col % EPB;
          cbase[u] = (c < NC) ? (e * NP) * FST + c * DIM : -1;
        }
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          float g0[NTG];
#pragma unroll
          for (int u = 0; u < NTG; ++u) g0[u] = cbase[u] >= 0 ? gfl[cbase[u] + r] : 0.f;
#pragma unroll
          for (int ks = 0; ks < KUR / 8; ++ks) {
            const int k0 = ks * 8 + tq;
            SplitB bs[NTG] = {};
#pragma unroll
            for (int u = 0; u < NTG; ++u) {
              float b0 = 0.f, b1 = 0.f;
              if (cbase[u] >= 0) {
                b0 = gfl[cbase[u] + k0 * FST + r] - g0[u];
                b1 = gfl[cbase[u] + (k0 + 4) * FST + r] - g0[u];
              }
              bs[u] = SplitB(b0, b1);
            }
#pragma unroll
            for (int t = 0; t < MT; ++t) {
              uint32_t ah[4], alo[4];
              load_a_tf32_ldsm(ah, aw + r * NP * KU, KU, t * 16, ks * 8, lane);
              load_a_tf32_ldsm(alo, aw + AWN + r * NP * KU, KU, t * 16, ks * 8, lane);
#pragma unroll
              for (int u = 0; u < NTG; ++u) mma_tf32x3(d[t][u], ah, alo, bs[u]);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < NTG; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int col = (ngp * NTG + u) * 8 + 2 * tq + h;
            const int c = col / EPB, e = col % EPB;
            if (c >= NC || e >= ne) continue;
            R* outp = a.out + (int64_t)c * EN + (int64_t)(e0 + e) * NP;
#pragma unroll
            for (int t = 0; t < MT; ++t)
#pragma unroll
              for (int half = 0; half < NACC / 2; ++half) {
                const int i = t * MROW + gq + 8 * half;
                if (i >= NP) continue;
                R v = -d[t][u][2 * half + h];
                if (sources && c >= 2 + DIM) v += src_s[(c - 2 - DIM) * ENP + e * NP + i];
                outp[i] = v;
              }
          }
      }
    } else
    for (int w = warp; w < (NNT / NTG) * MT; w += nwarps) {
      const int ngp = w / MT, t = w % MT;
      R d[NTG][NACC];
#pragma unroll
      for (int u = 0; u < NTG; ++u)
#pragma unroll
        for (int v = 0; v < NACC; ++v) d[u][v] = R(0);
      int cbase[NTG];
#pragma unroll
      for (int u = 0; u < NTG; ++u) {
        const int col = (ngp * NTG + u) * 8 + gq;
        const int c = col / EPB, e = col % EPB;
        cbase[u] = (c < NC) ? (e * NP) * FST + c * DIM : -1;
      }
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
        R g0[NTG];
#pragma unroll
        for (int u = 0; u < NTG; ++u) g0[u] = cbase[u] >= 0 ? gfl[cbase[u] + r] : R(0);
        if constexpr (!V::TF32) {
#pragma unroll
          for (int ks = 0; ks < KUR / 4; ++ks) {
            const double av = aw[(r * NP + t * 8 + gq) * KU + ks * 4 + tq];
            const int kk = ks * 4 + tq;
#pragma unroll
            for (int u = 0; u < NTG; ++u) {
              const double b = cbase[u] >= 0 ? gfl[cbase[u] + kk * FST + r] - g0[u] : 0.0;
              dmma884(d[u], av, b);
            }
          }
        } else {
#pragma unroll
          for (int ks = 0; ks < KUR / 8; ++ks) {
            uint32_t ah[4], alo[4];
            load_a_tf32_ldsm(ah, aw + r * NP * KU, KU, t * 16, ks * 8, lane);
            load_a_tf32_ldsm(alo, aw + AWN + r * NP * KU, KU, t * 16, ks * 8, lane);
            const int k0 = ks * 8 + tq;
#pragma unroll
            for (int u = 0; u < NTG; ++u) {
              float b0 = 0.f, b1 = 0.f;
              if (cbase[u] >= 0) {
                b0 = gfl[cbase[u] + k0 * FST + r] - g0[u];
                b1 = gfl[cbase[u] + (k0 + 4) * FST + r] - g0[u];
              }
              mma_tf32x3(d[u], ah, alo, b0, b1);
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < NTG; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = (ngp * NTG + u) * 8 + 2 * tq + h;
          const int c = col / EPB, e = col % EPB;
          if (c >= NC || e >= ne) continue;
          R* outp = a.out + (int64_t)c * EN + (int64_t)(e0 + e) * NP;
#pragma unroll
          for (int half = 0; half < NACC / 2; ++half) {
            const int i = t * MROW + gq + 8 * half;
            if (i >= NP) continue;
            R v = -d[u][2 * half + h];
            if (sources && c >= 2 + DIM) v += src_s[(c - 2 - DIM) * ENP + e * NP + i];
            outp[i] = v;
          }
        }
    }
  }
  if (timeout && threadIdx.x == 0) {
    atomicOr(a.status, ST_WAIT_TIMEOUT);
    // the copies in flight end before the block does
    if (!mbar_wait(&staged, it & 1, nullptr)) atomicOr(a.status, ST_WAIT_TIMEOUT);
  }
  if (bad) atomicOr(a.status, ST_NAN);
}

// Face pass on interior faces with HLL, and wherever a face needs more than
// the records' Rusanov / central combination: the HLL inviscid flux from the
// two states (q, p, c, gamma), the viscous parts central
// (inviscid.py:202-287, viscous.py:296-349).  recm / recp: own and
// neighbour-convention records; qp_g: the exterior q (stride qstride).
template <class R, int DIM, int NS, bool VISC>
__device__ __noinline__ void face_flux_general(const DGArgs<R> a, int64_t EN, int64_t gm,
                                               const R* recm, int slm, const R* recp, int slp,
                                               const R* qp_g,
                                               int64_t qstride, R n0, R n1, R n2, R fsc,
                                               const R* s0, R* bcol, int cstride) {
  constexpr int NC = DIM + 2 + NS, TW = trace_width(NC);
  const R n[3] = {n0, n1, n2};
  R qm[NC], qp[NC], rm[TW], rp[TW];
  load_rec<R, TW>(recm, slm, rm);
  load_rec<R, TW>(recp, slp, rp);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    qm[c] = a.q[c * EN + gm];
    qp[c] = qp_g[c * qstride];
  }
  NodeState<R, DIM, NS> sm, sp;
  make_state_light<R, DIM, NS>(qm, rm[NC + 1], rm[NC + 2], rm[NC + 3], sm);
  make_state_light<R, DIM, NS>(qp, rp[NC + 1], rp[NC + 2], rp[NC + 3], sp);
  R fi[NC], fim[NC], fip[NC];
  inviscid_num_flux<R, DIM, NS>(sm, sp, qm, qp, n, FLUX_HLL, fi);
  inviscid_flux_n<R, DIM, NS>(sm, n, fim);
  inviscid_flux_n<R, DIM, NS>(sp, n, fip);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    R out = -fi[c];
    // F_V . n = F . n + F_I . n on each side; the neighbour record holds -F . n
    if (VISC) out += ((rm[c] + fim[c]) + (-rp[c] + fip[c])) * R(0.5);
    // less the shift and the own half that WH carries
    bcol[c * cstride] = fsc * (folds<R>() ? out - (rm[c] + s0[c]) * R(0.5) : out - s0[c]);
  }
}

// Face kernel: numerical fluxes from the face-node records, lift, added to
// the volume kernel's result.
template <class R, int DIM, int ORDER, int NS, bool MIX, bool VISC>
__global__ void __launch_bounds__((VCfg<R, DIM, ORDER, NS, MIX>::NT2),
                                  (VCfg<R, DIM, ORDER, NS, MIX>::MINB2))
    k_face(DGArgs<R> a, GasParams g) {
  using V = VCfg<R, DIM, ORDER, NS, MIX>;
  using S = Simplex<DIM, ORDER>;
  constexpr int NP = V::NP, NF = V::NF, NFP = V::NFP, NFN = V::NFN, NC = V::NC, TW = V::TW;
  constexpr int EPB = V::EPB2, MP = V::MP, MT = V::MT, KF = V::KF, KFR = V::KFR;
  constexpr int NCOL = V::NCOL2, MROW = V::MROW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* am = reinterpret_cast<R*>(smem_raw);                  // [NAC][MP][KF] LIFT
  R* bm = am + V::A_FACE;                                  // [NCOL][KF]
  R* rx_s = bm + NCOL * KF;
  R* nrm_s = rx_s + EPB * DIM * DIM;
  R* fs_s = nrm_s + EPB * NF * DIM;
  int* fn_s = reinterpret_cast<int*>(fs_s + EPB * NF);
  int32_t* conn_s = fn_s + NFN;
  uint8_t* perm_s = reinterpret_cast<uint8_t*>(conn_s + EPB * NF);
  uint8_t* fslot_s = perm_s + a.nperm * NFP;

  const int E = a.nelem;
  const int64_t EN = (int64_t)E * NP;
  for (int i = threadIdx.x; i < MP * KF; i += blockDim.x) {
    const int row = i / KF, k = i % KF;
    put_a<R>(am, MP * KF, i, (row < NP && k < NFN) ? refop(S::OFF_LIFT + row * NFN + k) : 0.0);
  }
  for (int i = threadIdx.x; i < NCOL * KF; i += blockDim.x) bm[i] = R(0);
  for (int i = threadIdx.x; i < NFN; i += blockDim.x) fn_s[i] = c_face_nodes<DIM, ORDER>(i);
  for (int i = threadIdx.x; i < a.nperm * NFP; i += blockDim.x) {
    perm_s[i] = a.perm[i];
    fslot_s[i] = a.fslot[i];
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int nwarps = blockDim.x >> 5;
  constexpr int NACC = V::TF32 ? 4 : 2;
  const int ntiles = (a.nowned + EPB - 1) / EPB;
  const int64_t bstride = (int64_t)a.nbf * NFP;
  bool bad = false;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int e0 = tile * EPB;
    const int ne = imin(EPB, a.nowned - e0);
    // (the previous tile's contraction reads am / bm only; load_geometry's
    // first barrier orders it before this tile's writes of bm)
    stage_conn<NF>(a.conn, e0, ne, conn_s);
    load_geometry<R, DIM, ORDER>(a.rx, e0, ne, rx_s, nrm_s, fs_s);
    __syncthreads();

    for (int fnode = threadIdx.x; fnode < ne * NFN; fnode += blockDim.x) {
      const int e = fnode / NFN, fm = fnode % NFN, f = fm / NFP, m = fm % NFP;
      const int k = fn_s[fm];
      const int cn = conn_s[e * NF + f];
      const R fsc = fs_s[e * NF + f];
      const int64_t gm = (int64_t)(e0 + e) * NP + k;
      const R* recm = a.trace + ((int64_t)(e0 + e) * NFN + fm) * TW;
      const R* s0 = a.s0 + ((int64_t)(e0 + e) * NF + f) * NC;
      R* bcol = bm + e * KF + fm;
      // neighbour record and exterior q; mode 0 interior, 1 prescribed,
      // 2 interior flux only (dummy boundary, or a pairing that fails its
      // index checks)
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
        int kind = (bf < a.nbf) ? a.bkind[bf] : -1;
        if ((bk_needs_bext(kind) && !a.bext) || kind > BK_OUTFLOW) kind = -1;
        if (kind >= BK_PRESCRIBED) {
          // the volume kernel filed the exterior record and state_plus
          recp = a.btrace + ((int64_t)bf * NFP + m) * TW;
          slp = m;
          qp_g = a.bplus + (int64_t)bf * NFP + m;
          qstride = bstride;
          mode = 1;
        } else if (kind < 0) {
          atomicOr(a.status, ST_BAD_INDEX);
        }
      }
      if (mode == 2) {
        // DummyBoundary: F* = F(q-) . n (boundary.py:1027-1049)
        R rm[TW];
        load_rec<R, TW>(recm, fm, rm);
#pragma unroll
        for (int c = 0; c < NC; ++c)
          bcol[c * EPB * KF] = (folds<R>() ? fsc * R(0.5) : fsc) * (rm[c] - s0[c]);
        continue;
      }
      if (a.flux_kind == FLUX_HLL) {
        const R* nf = nrm_s + (e * NF + f) * DIM;
        face_flux_general<R, DIM, NS, VISC>(a, EN, gm, recm, fm, recp, slp, qp_g, qstride, nf[0], nf[1],
                                            DIM > 2 ? nf[DIM - 1] : R(0), fsc, s0, bcol,
                                            EPB * KF);
        continue;
      }
      R rm[TW], rp[TW];
      if constexpr (!folds<R>()) load_rec<R, TW>(recm, fm, rm);
      load_rec<R, TW>(recp, slp, rp);
      const R lamm = folds<R>() ? a.lam[gm] : rm[NC];
      R qm[NC], qp[NC], sh[NC];
      constexpr int VEC = RecLayout<R, TW>::VEC;
      if constexpr (NC % VEC == 0) {
#pragma unroll
        for (int c = 0; c < NC; c += VEC) {
          R v[VEC];
          load_record<R, VEC>(s0 + c, v);
#pragma unroll
          for (int i = 0; i < VEC; ++i) sh[c + i] = v[i];
        }
      } else {
#pragma unroll
        for (int c = 0; c < NC; ++c) sh[c] = s0[c];
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        qm[c] = a.q[c * EN + gm];
        qp[c] = qp_g[c * qstride];
      }
      const R lam = (a.flux_kind == FLUX_RUSANOV) ? fmax(lamm, rp[NC]) : R(0);
      if constexpr (folds<R>()) {
        // F* . n - F0 . n less the own half (F- - F0) . n / 2 that WH carries
        const R hf = fsc * R(-0.5);
#pragma unroll
        for (int c = 0; c < NC; ++c)
          bcol[c * EPB * KF] = hf * ((rp[c] + sh[c]) + lam * (qm[c] - qp[c]));
      } else {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const R out = (rm[c] - rp[c]) * R(0.5) - lam * (qm[c] - qp[c]) * R(0.5);
          bcol[c * EPB * KF] = fsc * (out - sh[c]);
        }
      }
    }
    __syncthreads();

    // rhs += LIFT S on the tensor cores.  float32: one item per group of NTG
    // column tiles and every m-tile, each face value split into its tf32
    // hi/lo words once; float64: one m-tile and NTG column tiles per item
    constexpr int NNT = NCOL / 8;
    constexpr int NTG = (NNT % 3 == 0) ? 3 : ((NNT % 2 == 0) ? 2 : 1);
    if constexpr (V::TF32) {
      for (int ngp = warp; ngp < NNT / NTG; ngp += nwarps) {
        float d[MT][NTG][NACC];
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
          for (int u = 0; u < NTG; ++u)
#pragma unroll
            for (int v = 0; v < NACC; ++v) d[t][u][v] = 0.f;
        const R* bcol = bm + (ngp * NTG * 8 + gq) * KF + tq;
#pragma unroll
        for (int ks = 0; ks < KFR / 8; ++ks) {
          SplitB bs[NTG];
#pragma unroll
          for (int u = 0; u < NTG; ++u)
            bs[u] = SplitB(bcol[u * 8 * KF + ks * 8], bcol[u * 8 * KF + ks * 8 + 4]);
#pragma unroll
          for (int t = 0; t < MT; ++t) {
            uint32_t ah[4], alo[4];
            load_a_tf32_ldsm(ah, am, KF, t * 16, ks * 8, lane);
            load_a_tf32_ldsm(alo, am + MP * KF, KF, t * 16, ks * 8, lane);
#pragma unroll
            for (int u = 0; u < NTG; ++u) mma_tf32x3(d[t][u], ah, alo, bs[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < NTG; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int col = (ngp * NTG + u) * 8 + 2 * tq + h;
            const int c = col / EPB, e = col % EPB;
            if (c >= NC || e >= ne) continue;
            R* outp = a.out + (int64_t)c * EN + (int64_t)(e0 + e) * NP;
#pragma unroll
            for (int t = 0; t < MT; ++t)
#pragma unroll
              for (int half = 0; half < NACC / 2; ++half) {
                const int i = t * MROW + gq + 8 * half;
                if (i >= NP) continue;
                const R v = outp[i] + d[t][u][2 * half + h];
                outp[i] = v;
                bad |= !(v == v);
              }
          }
      }
    } else
    for (int w = warp; w < (NNT / NTG) * MT; w += nwarps) {
      const int ngp = w / MT, t = w % MT;
      R d[NTG][NACC];
#pragma unroll
      for (int u = 0; u < NTG; ++u)
#pragma unroll
        for (int v = 0; v < NACC; ++v) d[u][v] = R(0);
      const R* bcol = bm + (ngp * NTG * 8 + gq) * KF + tq;
      if constexpr (!V::TF32) {
#pragma unroll
        for (int ks = 0; ks < KFR / 4; ++ks) {
          const double av = am[(t * 8 + gq) * KF + ks * 4 + tq];
#pragma unroll
          for (int u = 0; u < NTG; ++u) dmma884(d[u], av, bcol[u * 8 * KF + ks * 4]);
        }
      } else {
#pragma unroll
        for (int ks = 0; ks < KFR / 8; ++ks) {
          uint32_t ah[4], alo[4];
          load_a_tf32_ldsm(ah, am, KF, t * 16, ks * 8, lane);
          load_a_tf32_ldsm(alo, am + MP * KF, KF, t * 16, ks * 8, lane);
#pragma unroll
          for (int u = 0; u < NTG; ++u)
            mma_tf32x3(d[u], ah, alo, bcol[u * 8 * KF + ks * 8], bcol[u * 8 * KF + ks * 8 + 4]);
        }
      }
#pragma unroll
      for (int u = 0; u < NTG; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = (ngp * NTG + u) * 8 + 2 * tq + h;
          const int c = col / EPB, e = col % EPB;
          if (c >= NC || e >= ne) continue;
          R* outp = a.out + (int64_t)c * EN + (int64_t)(e0 + e) * NP;
#pragma unroll
          for (int half = 0; half < NACC / 2; ++half) {
            const int i = t * MROW + gq + 8 * half;
            if (i >= NP) continue;
            const R v = outp[i] + d[u][2 * half + h];
            outp[i] = v;
            bad |= !(v == v);
          }
        }
    }
  }
  if (bad) atomicOr(a.status, ST_NAN);
}

}  // namespace

}  // namespace mgc
