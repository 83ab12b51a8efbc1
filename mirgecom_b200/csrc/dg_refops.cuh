// Reference-element operators of the nodal DG discretization.
//
// For every supported (dim, order) the host packs, in order:
//   W     [dim][Np][Np]   W_r = M^-1 D_r^T M          (weak derivative)
//   LIFT  [Np][Nf*Nfp]    M^-1 E                      (face lift)
//   NREF  [Nf][dim]       unit outward reference normals
//   FSR   [Nf]            reference face measure / face-parametrisation measure
// (refelem.py; mgc_upload_reference_operators()).  The upload adds
//   WH    [dim][Np][Np]   W_r - 1/2 sum_f NREF[f][r] FSR[f] LIFT_f E_f
// (E_f the face's nodes): the weak derivative with the element's own half of
// every central face value folded in.  On an affine element n_fj fscale_f =
// sum_r (dr_r/dx_j) NREF[f][r] FSR[f], so for a face value (u- + u+) / 2
//   sum_f n_fj LIFT_f fscale_f u* - sum_r rx_rj W_r u
//     = sum_f n_fj LIFT_f fscale_f u+ / 2 - sum_r rx_rj WH_r u,
// and the face passes read the neighbour's half only.  The gradient passes use
// it in both types, the divergence passes in float64 (folds<R>()).
//
// The matrices W and LIFT live in a global-memory table: every kernel reads
// them once per CTA, one entry per thread, to build its tensor-core operands
// in shared memory: from constant memory those per-lane addresses replay one by
// one.  (The whole call shows it little: 24^3 p3 Taylor-Green, float64, 830 us
// from constant memory, 824 us from the table; 1260 reacting tetrahedra inside
// the noise of the host path.)  NREF and FSR, a few values each thread reads for
// its face, stay in constant memory.
#pragma once
#include <cstdint>

namespace mgc {

__host__ __device__ constexpr int simplex_npts(int dim, int order) {
  return dim == 0 ? 1
       : dim == 1 ? order + 1
       : dim == 2 ? (order + 1) * (order + 2) / 2
                  : (order + 1) * (order + 2) * (order + 3) / 6;
}

// matrices of one (dim, order) as the host packs them (W, LIFT) and as the
// table holds them (W, LIFT, WH)
__host__ __device__ constexpr int refmat_size(int dim, int order) {
  return dim * simplex_npts(dim, order) * simplex_npts(dim, order) +
         simplex_npts(dim, order) * (dim + 1) * simplex_npts(dim - 1, order);
}
__host__ __device__ constexpr int refops_size(int dim, int order) {
  return refmat_size(dim, order) + dim * simplex_npts(dim, order) * simplex_npts(dim, order);
}
// NREF, FSR
__host__ __device__ constexpr int refgeo_size(int dim) { return (dim + 1) * dim + (dim + 1); }

// supported simplex discretizations, in packing order
__host__ __device__ constexpr int refops_slot(int dim, int order) {
  return (dim == 2 && order >= 1 && order <= 4) ? order - 1
       : (dim == 3 && order >= 1 && order <= 3) ? 4 + order - 1
                                                : -1;
}

__host__ __device__ constexpr int refops_offset(int dim, int order) {
  int off = 0;
  for (int o = 1; o <= 4; ++o) {
    if (dim == 2 && o == order) return off;
    off += refops_size(2, o);
  }
  for (int o = 1; o <= 3; ++o) {
    if (dim == 3 && o == order) return off;
    off += refops_size(3, o);
  }
  return -1;
}

constexpr int kRefOpsTotal = refops_offset(3, 3) + refops_size(3, 3);

constexpr int kRefGeoStride = refgeo_size(3);
constexpr int kRefGeoTotal = (refops_slot(3, 3) + 1) * kRefGeoStride;
__host__ __device__ constexpr int refgeo_offset(int dim, int order) {
  return refops_slot(dim, order) * kRefGeoStride;
}

// Every translation unit that launches kernels holds its own copy (internal
// linkage, no relocatable device code); mgc_upload_reference_operators()
// fills the copy of each unit.
static __device__ double g_refops[kRefOpsTotal];
static __constant__ double c_refgeo64[kRefGeoTotal];
static __constant__ float c_refgeo32[kRefGeoTotal];

// Whether the divergence passes of type R use WH.  float64: the face pass then
// reads one flux record per face node instead of two (32^3 p3 reacting
// right-hand side 5.67 -> 5.46 ms, 24^3 p3 Taylor-Green 0.833 -> 0.768 ms).
// float32 keeps W and both records: there the sum of the two fluxes rounds at
// the size of the flux, and dropping that rounding moves the result by up to
// 2e-3 of its rms on fine meshes (towards the float64 one), for 2 %.
template <class R>
__host__ __device__ constexpr bool folds() { return sizeof(R) == 8; }

__device__ __forceinline__ double refop(int i) { return __ldg(g_refops + i); }

__host__ __device__ constexpr int fnodes_size(int dim, int order) {
  return (dim + 1) * simplex_npts(dim - 1, order);
}

__host__ __device__ constexpr int fnodes_offset(int dim, int order) {
  int off = 0;
  for (int o = 1; o <= 4; ++o) {
    if (dim == 2 && o == order) return off;
    off += fnodes_size(2, o);
  }
  for (int o = 1; o <= 3; ++o) {
    if (dim == 3 && o == order) return off;
    off += fnodes_size(3, o);
  }
  return -1;
}

constexpr int kFaceNodesTotal = fnodes_offset(3, 3) + fnodes_size(3, 3);

// volume node index of face node m of face f, at [f * Nfp + m]
static __constant__ int c_fnodes[kFaceNodesTotal];

template <int DIM, int ORDER>
__device__ __forceinline__ int c_face_nodes(int i) {
  return c_fnodes[fnodes_offset(DIM, ORDER) + i];
}

template <int DIM, int ORDER>
struct Simplex {
  static constexpr int NP = simplex_npts(DIM, ORDER);
  static constexpr int NF = DIM + 1;
  static constexpr int NFP = simplex_npts(DIM - 1, ORDER);
  static constexpr int OFF = refops_offset(DIM, ORDER);
  static constexpr int OFF_W = OFF;
  static constexpr int OFF_LIFT = OFF_W + DIM * NP * NP;
  static constexpr int OFF_WH = OFF_LIFT + NP * NF * NFP;
  // the operator of the volume divergence in type R
  template <class R>
  static constexpr int OFF_WDIV = folds<R>() ? OFF_WH : OFF_W;
  static constexpr int OFF_NREF = refgeo_offset(DIM, ORDER);
  static constexpr int OFF_FSR = OFF_NREF + NF * DIM;
  static_assert(OFF >= 0, "unsupported simplex discretization");
};

template <class R> struct RefBank;
template <> struct RefBank<double> {
  static __device__ __forceinline__ double get(int i) { return c_refgeo64[i]; }
};
template <> struct RefBank<float> {
  static __device__ __forceinline__ float get(int i) { return c_refgeo32[i]; }
};

}  // namespace mgc
