// BR1 gradient pass on the 5th-generation tensor cores (tcgen05, TMEM).
//
// The same gradient as k_grad (dg_kernels.cuh), of every conserved field and
// the temperature, with the element-constant shift u - u_0 and the TF32
// three-term split A_hi B_hi + A_hi B_lo + A_lo B_hi (grad_operator,
// mirgecom/navierstokes.py:443-446, and grad_facial_flux,
// mirgecom/gradient.py).  On an affine element n_fj fscale_f is
// sum_r (dr_r/dx_j) c_fr with c_fr = NREF[f][r] FSR[f] (dg_refops.cuh), so the
// lift needs no per-face products: with reference matrices alone
//   D_r    = -WH_r (u - u_0) + sum_f (c_fr LIFT_f) P_f
//   grad_j = sum_r (dr_r/dx_j) D_r,       P_f = u*_f - u_0 - (u-_f - u_0) / 2
// (P = (u+ - u_0) / 2 on interior faces).  That is DIM accumulator columns per
// node instead of DIM + NF, 9 multiply-adds per node and field in the epilogue
// instead of 21, no normals, no face scale and no own face values on interior
// faces.  The work is a warp-specialised pipeline over tiles of EPB elements:
//
//   producer warps 0-11  shift and split the tile's rows of q and T and the
//                        face values P into the hi/lo copies of the A operand
//                        [row = (field, element)][k = node | face node] in one
//                        of two shared-memory stages and arrive on full[s].
//                        Each value's registers are loaded again for the NEXT
//                        tile as soon as they are stored (its face pairing is
//                        staged two tiles ahead), so the gathers' latency runs
//                        under the rest of this tile's work.  After the next
//                        tile's barrier the last thread issues the products
//                        D[row][(r, i)] = sum_k A[row][k] B[(r, i)][k] into
//                        TMEM buffer s and commits to done[s]
//   epilogue warps 12-15 wait on done[s], read their TMEM lanes (one row per
//                        thread), combine with the metric terms, store the
//                        gradients and arrive on empty[s]
//
// Tiles: NMT row blocks of 128 (MMA M) with EPM elements each, chosen so that
// the producers have one face node each: 9 order-3, 16 order-2, 32 order-1
// tetrahedra of the 7-species mixture.  With the smaller orders in single
// blocks of 9 elements the barriers and waits of a tile cost as much as the
// work in it.
//
// Bound: the producers' gathers, latency and L1 wavefronts (the products are
// 0.4 us of a 3.4 us tile).  Against the version with per-face lift columns
// and no reload in place (CUDA events): order 3, 64^3 cells 4.38 -> 4.06 ms
// (of it 0.27 by working out each thread's item indices once instead of per
// tile), 1260 tetrahedra 17.2 -> 12.2 us; order 2, 40^3 cells 687 us (799 us
// by k_grad, which it replaces there).
//
// Operands use the K-major, non-swizzled canonical layout of the UMMA
// descriptors: 8-row x 16-byte core matrices, row groups SBO = 128 bytes
// apart, k chunks LBO bytes apart; LBO is padded by 16 bytes so that a warp
// storing 32 consecutive k of one row hits distinct banks.  Every mbarrier
// wait is bounded: after kWaitNs the waiting role sets ST_WAIT_TIMEOUT in the
// status word and an abort flag that ends the other roles' loops; the kernel
// then releases its TMEM and returns.
#pragma once
#include <cstdint>

#include "async_copy.cuh"
#include "dg_kernels.cuh"

namespace mgc {

// {{{ tcgen05 primitives

__device__ __forceinline__ void fence_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// TMEM allocation by one whole warp; the base address lands in *dst
__device__ __forceinline__ void tc_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_addr(dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// Shared-memory matrix descriptor: K-major, no swizzle (layout type 0),
// descriptor version 1; addresses and offsets in 16-byte units.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::tf32: f32 accumulator, tf32 A and B, both
// K-major, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_tf32(int m, int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
// D[tmem] (+)= A[smem] * B[smem]^T, issued by one thread
__device__ __forceinline__ void tc_mma_tf32(uint32_t d, uint64_t adesc, uint64_t bdesc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on *b once every product issued so far by this thread has completed
__device__ __forceinline__ void tc_commit(uint64_t* b) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_addr(b))
      : "memory");
}
// sixteen consecutive 32-bit TMEM columns of this thread's lane
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
// wait for this thread's TMEM loads; the registers are tied to the wait so
// that no use is scheduled before it
template <int N>
__device__ __forceinline__ void tc_wait_ld(uint32_t (&v)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(v[i]));
}

// }}}

// {{{ configuration

template <int DIM, int ORDER, int NS>
struct TcGrad {
  using S = Simplex<DIM, ORDER>;
  static constexpr int NP = S::NP, NF = S::NF, NFP = S::NFP, NFN = NF * NFP;
  static constexpr int NC = DIM + 2 + NS, NU = NC + 1;
  static constexpr int ROWS = 128;                    // MMA M: rows (field, element)
  // twelve producer warps, four epilogue warps
  static constexpr int GT = 12 * 32, NEPI = 128, NT = GT + NEPI;
  // row blocks per tile and elements per block: one face node per producer
  static constexpr int NMT = ORDER == 1 ? 4 : ORDER == 2 ? 2 : 1;
  static constexpr int EPM = imin(ROWS / NU, GT / (NFN * NMT));
  static constexpr int EPB = NMT * EPM;
  static constexpr int KV = round_up(NP, 8);          // k extent of the volume part
  static constexpr int KA = KV + round_up(NFN, 8);    // k extent with the face values
  static constexpr int NV = round_up(DIM * NP, 16);   // N: columns (r, i)
  static constexpr int BUF_COLS = NMT * NV;           // TMEM columns per buffer
  static constexpr int TCOLS = 2 * BUF_COLS;
  // byte strides of the canonical layouts
  static constexpr int SBO = 128;
  static constexpr int LBO_A = ROWS / 8 * 128 + 16;
  static constexpr int LBO_B = NV / 8 * 128;
  static constexpr int A_BYTES = round_up(KA / 4 * LBO_A, 128);   // one copy of one row block
  static constexpr int STAGE = 2 * NMT * A_BYTES;                 // [block][hi, lo]
  static constexpr int B_BYTES = KA / 4 * LBO_B;                  // one copy
  // rows move in pieces of VW floats
  static constexpr int VW = NP % 4 == 0 ? 4 : 2;
  static constexpr int ROW_ITEMS = NP / VW * NU * EPB;
  static constexpr int ROW_ROUNDS = (ROW_ITEMS + GT - 1) / GT;
  // per-tile data (4-byte words): face pairing, row shifts u_0, metric rx
  static constexpr int S_U0 = EPB * NF, S_RX = S_U0 + NU * EPB, SMALL = S_RX + EPB * DIM * DIM;
  static constexpr int SMALL_ROUNDS = (SMALL + GT - 1) / GT;
  // shared-memory carve-up (bytes)
  static constexpr int OFF_BAR = 0;                   // full[2], done[2], empty[2]
  static constexpr int OFF_TMEM = 48;                 // TMEM base address
  static constexpr int OFF_ABORT = 52;                // any role gave up
  static constexpr int OFF_PABORT = 56;               // the producers' copy [2]
  static constexpr int OFF_A = 1024;                  // [stage][block][hi, lo]
  static constexpr int OFF_B = OFF_A + 2 * STAGE;     // [hi, lo]
  static constexpr int OFF_GEO = OFF_B + 2 * B_BYTES;              // [stage][EPB][DIM][DIM]
  static constexpr int OFF_SMALL = OFF_GEO + 2 * EPB * DIM * DIM * 4;  // [3][SMALL]
  static constexpr int OFF_FN = OFF_SMALL + 3 * SMALL * 4;         // [NFN] int
  static constexpr int OFF_PERM = OFF_FN + NFN * 4;                // [nperm][NFP] uint8
  static size_t smem_bytes(int nperm) { return (size_t)OFF_PERM + (size_t)nperm * NFP + 16; }
  // rows in whole pieces; products within the instruction shapes; TMEM
  // allocations are powers of two
  static constexpr bool OK = NP % 2 == 0 && EPM >= 1 && NFN * EPB <= GT && NV <= 256 &&
                             (TCOLS == 128 || TCOLS == 256 || TCOLS == 512) &&
                             OFF_PERM + 64 * NFP <= 227 * 1024;
};

// every order of the reacting mixture on tetrahedra fits
static_assert(TcGrad<3, 1, 7>::OK && TcGrad<3, 2, 7>::OK && TcGrad<3, 3, 7>::OK,
              "tcgen05 gradient kernel no longer fits the tetrahedra");

// byte offset of element (row, k) in a canonical K-major no-swizzle operand
__device__ __forceinline__ int canon_off(int row, int k, int lbo) {
  return (k >> 2) * lbo + row * 16 + (k & 3) * 4;    // row groups are 8 * 16 bytes
}

__device__ __forceinline__ void split_f32(float v, float& hi, float& lo) {
  const uint32_t h = to_tf32(v);
  hi = __uint_as_float(h);
  lo = __uint_as_float(to_tf32(v - hi));
}

// VW consecutive floats as one vector access
template <int VW> struct VecF;
template <> struct VecF<4> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = __ldg(reinterpret_cast<const float4*>(p)); }
  __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float4*>(p) = v; }
  __device__ __forceinline__ void shift_split(float u0, VecF& h, VecF& l) const {
    split_f32(v.x - u0, h.v.x, l.v.x);
    split_f32(v.y - u0, h.v.y, l.v.y);
    split_f32(v.z - u0, h.v.z, l.v.z);
    split_f32(v.w - u0, h.v.w, l.v.w);
  }
};
template <> struct VecF<2> {
  float2 v;
  __device__ __forceinline__ void load(const float* p) { v = __ldg(reinterpret_cast<const float2*>(p)); }
  __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float2*>(p) = v; }
  __device__ __forceinline__ void shift_split(float u0, VecF& h, VecF& l) const {
    split_f32(v.x - u0, h.v.x, l.v.x);
    split_f32(v.y - u0, h.v.y, l.v.y);
  }
};

// }}}

namespace {

template <int DIM, int ORDER, int NS>
__global__ void __launch_bounds__(TcGrad<DIM, ORDER, NS>::NT, 1)
    k_grad_tc(DGArgs<float> a, GasParams g) {
  using C = TcGrad<DIM, ORDER, NS>;
  using S = Simplex<DIM, ORDER>;
  constexpr int NP = C::NP, NF = C::NF, NFP = C::NFP, NFN = C::NFN, NC = C::NC, NU = C::NU;
  constexpr int EPB = C::EPB, EPM = C::EPM, NMT = C::NMT, KV = C::KV, KA = C::KA, NV = C::NV;
  constexpr int GT = C::GT, VW = C::VW, DD = DIM * DIM;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + C::OFF_BAR);
  uint64_t* done = full + 2;
  uint64_t* empty = full + 4;
  uint32_t* tmem_s = reinterpret_cast<uint32_t*>(smem_raw + C::OFF_TMEM);
  volatile int* abort_s = reinterpret_cast<volatile int*>(smem_raw + C::OFF_ABORT);
  volatile int* pabort_s = reinterpret_cast<volatile int*>(smem_raw + C::OFF_PABORT);
  float* geo_s = reinterpret_cast<float*>(smem_raw + C::OFF_GEO);
  uint32_t* small_s = reinterpret_cast<uint32_t*>(smem_raw + C::OFF_SMALL);
  int* fn_s = reinterpret_cast<int*>(smem_raw + C::OFF_FN);
  uint8_t* perm_s = smem_raw + C::OFF_PERM;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int E = a.nelem;
  const int64_t EN = (int64_t)E * NP;
  const int EOWN = a.nowned > 0 ? a.nowned : E;
  const int ntiles = (EOWN + EPB - 1) / EPB;

  // ---- setup: barriers, zeroed A stages, operator B copies, TMEM
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(full + s, C::GT);
      mbar_init(done + s, 1);
      mbar_init(empty + s, C::NEPI);
    }
    *abort_s = 0;
    pabort_s[0] = pabort_s[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  {
    float4* az = reinterpret_cast<float4*>(smem_raw + C::OFF_A);
    for (int i = tid; i < 2 * C::STAGE / 16; i += blockDim.x) az[i] = make_float4(0, 0, 0, 0);
    float* bh = reinterpret_cast<float*>(smem_raw + C::OFF_B);
    float* bl = reinterpret_cast<float*>(smem_raw + C::OFF_B + C::B_BYTES);
    for (int i = tid; i < NV * KA; i += blockDim.x) {
      const int n = i / KA, k = i % KA, r = n / NP, row = n % NP;
      double v = 0.0;
      if (n < DIM * NP) {
        if (k < NP) {
          v = -refop(S::OFF_WH + (r * NP + row) * NP + k);
        } else if (k >= KV && k - KV < NFN) {
          const int f = (k - KV) / NFP;
          v = RefBank<double>::get(S::OFF_NREF + f * DIM + r) *
              RefBank<double>::get(S::OFF_FSR + f) * refop(S::OFF_LIFT + row * NFN + k - KV);
        }
      }
      float hi, lo;
      split_tf32(v, hi, lo);
      const int o = canon_off(n, k, C::LBO_B) >> 2;
      bh[o] = hi;
      bl[o] = lo;
    }
    for (int i = tid; i < NFN; i += blockDim.x) fn_s[i] = c_face_nodes<DIM, ORDER>(i);
    for (int i = tid; i < a.nperm * NFP; i += blockDim.x) perm_s[i] = a.perm[i];
  }
  if (warp == 0) tc_alloc(tmem_s, C::TCOLS);
  // generic-proxy writes of the operands become visible to the tensor cores
  fence_async_shared();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_s;

  if (tid < GT) {
    // ================= producers
    constexpr int RR = C::ROW_ROUNDS, SR = C::SMALL_ROUNDS;
    // this thread's face node: element fe of the tile, face slot ffm
    const int ffm = tid % NFN, fe = tid / NFN;
    const int ff = ffm / NFP, fm_ = ffm % NFP;
    const int fk = fn_s[ffm];
    auto field = [&](int c) { return c < NC ? a.q + c * EN : a.t_op; };
    auto small_load = [&](int tl, uint32_t (&w)[SR]) {
      const int e1 = tl * EPB, n1 = imin(EPB, EOWN - e1);
#pragma unroll
      for (int j = 0; j < SR; ++j) {
        const int i = tid + j * GT;
        w[j] = 0;
        if (i < C::S_U0) {
          if (i / NF < n1) w[j] = (uint32_t)__ldg(a.conn + (int64_t)e1 * NF + i);
        } else if (i < C::S_RX) {
          const int e = (i - C::S_U0) % EPB, c = (i - C::S_U0) / EPB;
          if (e < n1) w[j] = __float_as_uint(__ldg(field(c) + (int64_t)(e1 + e) * NP));
        } else if (i < C::SMALL) {
          const int m = i - C::S_RX;
          if (m / DD < n1) w[j] = __float_as_uint(__ldg(a.rx + (int64_t)e1 * DD + m));
        }
      }
    };
    auto small_store = [&](const uint32_t (&w)[SR], int b) {
#pragma unroll
      for (int j = 0; j < SR; ++j)
        if (tid + j * GT < C::SMALL) small_s[b * C::SMALL + tid + j * GT] = w[j];
    };
    VecF<VW> rv[RR];
    float nb[NU];
    int fmode = -1;
    // this thread's row pieces (the same in every tile): source in element 0's
    // tile, and packed: operand offset in the stage | index of the row's shift
    // | element (63: none).  Worked out per tile, with 64-bit sums per load,
    // the indices were half of the producers' instructions.
    const float* rsrc[RR];
    uint32_t rpk[RR];
    static_assert(C::STAGE <= 1 << 17 && NU * EPB <= 512 && EPB < 63, "packed row items");
#pragma unroll
    for (int j = 0; j < RR; ++j) {
      const int idx = tid + j * GT;
      const int kc = idx % (NP / VW), e = (idx / (NP / VW)) % EPB, c = idx / (NP / VW * EPB);
      const bool in = idx < C::ROW_ITEMS;
      rsrc[j] = field(in ? c : 0) + e * NP + kc * VW;
      rpk[j] = in ? (uint32_t)(2 * (e / EPM) * C::A_BYTES + canon_off(c * EPM + e % EPM, kc * VW, C::LBO_A)) |
                        (uint32_t)(c * EPB + e) << 17 | (uint32_t)e << 26
                  : 63u << 26;
    }
    auto row_load = [&](int tl, int j) {
      const int e = (int)(rpk[j] >> 26);
      if (e < EOWN - tl * EPB && e != 63) rv[j].load(rsrc[j] + (int64_t)tl * (EPB * NP));
    };
    // the neighbour's fields at node *gi* (node numbers times four fit 32 bits)
    auto face_load = [&](int64_t gi, int c) {
      return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(field(c)) +
                                                  (uint32_t)gi * 4u));
    };
    const int foff = 2 * (fe / EPM) * C::A_BYTES + canon_off(fe % EPM, KV + ffm, C::LBO_A);
    // mode of this thread's face node in tile tl (pairing words *conn_b*):
    // -1 none, 0 interior (en, kn its neighbour node), 1 exterior value,
    // 2 interior value, 3 Mengaldo
    auto face_mode = [&](int tl, const uint32_t* conn_b, int64_t& gi) {
      gi = 0;
      if (tid >= NFN * EPB || tl * EPB + fe >= EOWN) return -1;
      const int cn = (int)conn_b[fe * NF + ff];
      if (cn >= 0) {
        const int en = cn >> 8, pr = cn & 255;
        const int kn = (pr < a.nperm) ? perm_s[pr * NFP + fm_] : NP;
        if (en < E && kn < NP) {
          gi = (int64_t)en * NP + kn;
          return 0;
        }
        atomicOr(a.status, ST_BAD_INDEX);
        return 2;
      }
      const int bf = -(cn + 1);
      int kind = (bf < a.nbf) ? a.bkind[bf] : -1;
      if ((bk_needs_bext(kind) && !a.bext) || kind > BK_OUTFLOW) kind = -1;
      if (kind < 0) atomicOr(a.status, ST_BAD_INDEX);
      return kind == BK_PRESCRIBED ? 1 : bk_mengaldo(kind) ? 3 : 2;
    };
    // D[s] = A[s] B^T, the two correction terms of every k step first: the
    // accumulator (which truncates) is then near its final size for KA / 8
    // additions instead of 3 KA / 8
    auto issue_products = [&](int s) {
      constexpr uint32_t ID = umma_idesc_tf32(C::ROWS, NV);
      const uint32_t bh = smem_addr(smem_raw + C::OFF_B), bl = bh + C::B_BYTES;
#pragma unroll 1
      for (int mt = 0; mt < NMT; ++mt) {
        const uint32_t ah = smem_addr(smem_raw + C::OFF_A) + s * C::STAGE + 2 * mt * C::A_BYTES;
        const uint32_t al = ah + C::A_BYTES;
        const uint32_t d = tmem + (uint32_t)(s * C::BUF_COLS + mt * NV);
#pragma unroll
        for (int ks = 0; ks < KA / 8; ++ks) {
          const uint32_t ao = 2 * ks * C::LBO_A, bo = 2 * ks * C::LBO_B;
          tc_mma_tf32(d, umma_desc(al + ao, C::LBO_A, C::SBO),
                      umma_desc(bh + bo, C::LBO_B, C::SBO), ID, ks > 0);
          tc_mma_tf32(d, umma_desc(ah + ao, C::LBO_A, C::SBO),
                      umma_desc(bl + bo, C::LBO_B, C::SBO), ID, 1);
        }
#pragma unroll
        for (int ks = 0; ks < KA / 8; ++ks) {
          const uint32_t ao = 2 * ks * C::LBO_A, bo = 2 * ks * C::LBO_B;
          tc_mma_tf32(d, umma_desc(ah + ao, C::LBO_A, C::SBO),
                      umma_desc(bh + bo, C::LBO_B, C::SBO), ID, 1);
        }
      }
    };
    int issued = 0, last_issued = -1;
    int pending = -1;          // a filled tile whose products are not issued yet
    auto issue_pending = [&]() {
      const int ps = pending & 1;
      if (!mbar_wait(full + ps, ((uint32_t)pending >> 1) & 1, abort_s)) {
        atomicOr(a.status, ST_WAIT_TIMEOUT);
        *abort_s = 1;
      } else {
        tc_fence_after();
        issue_products(ps);
        tc_commit(done + ps);
        ++issued;
        last_issued = pending;
      }
      pending = -1;
    };
    const int first = blockIdx.x, step = (int)gridDim.x;
    {
      // per-tile data of the first two tiles, then the first tile's values
      uint32_t w[SR];
      small_load(first, w);
      small_store(w, 0);
      if (first + step < ntiles) {
        small_load(first + step, w);
        small_store(w, 1);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(GT) : "memory");
#pragma unroll
      for (int j = 0; j < RR; ++j) row_load(first, j);
      int64_t gi;
      fmode = face_mode(first, small_s, gi);
      if (fmode == 0) {
#pragma unroll
        for (int c = 0; c < NU; ++c) nb[c] = face_load(gi, c);
      }
    }
    for (int it = 0, tile = first, b = 0; tile < ntiles; ++it, tile += step) {
      const int s = it & 1;
      const uint32_t use = (uint32_t)it >> 1;
      if (tid == 0) {
        bool ok = true;
        if (use >= 1) ok = mbar_wait(empty + s, (use - 1) & 1, abort_s);
        if (!ok) {
          atomicOr(a.status, ST_WAIT_TIMEOUT);
          *abort_s = 1;
        }
        pabort_s[s] = *abort_s;
      }
      // this tile's and the next one's per-tile data are complete, the
      // producers are done with the third buffer, and stage s is free
      asm volatile("bar.sync 1, %0;" ::"n"(GT) : "memory");
      // (thread 0 may be a tile ahead, never two: its next word is the other one)
      if (pabort_s[s]) break;
      // the previous tile's products: their issue overlaps the other
      // threads' work
      if (tid == GT - 1 && pending >= 0) issue_pending();
      const int ne = imin(EPB, EOWN - tile * EPB);
      const bool more = tile + step < ntiles;
      const int bn = b == 2 ? 0 : b + 1;
      const uint32_t* small_b = small_s + b * C::SMALL;
      const float* u0_b = reinterpret_cast<const float*>(small_b) + C::S_U0;
      const float* rx_b = reinterpret_cast<const float*>(small_b) + C::S_RX;
      unsigned char* stage = smem_raw + C::OFF_A + s * C::STAGE;
      uint32_t w[SR];
      const bool more2 = tile + 2 * step < ntiles;
      if (more2) small_load(tile + 2 * step, w);

      // ---- rows: shift, split, store; reload for the next tile
#pragma unroll
      for (int j = 0; j < RR; ++j) {
        if ((int)(rpk[j] >> 26) < ne) {
          VecF<VW> h, l;
          rv[j].shift_split(u0_b[rpk[j] >> 17 & 511], h, l);
          unsigned char* dst = stage + (rpk[j] & 0x1ffff);
          h.store(reinterpret_cast<float*>(dst));
          l.store(reinterpret_cast<float*>(dst + C::A_BYTES));
        }
        if (more) row_load(tile + step, j);
      }

      // ---- face value P of this thread's face node; reload for the next tile
      const int mode = fmode;
      int64_t gn = 0;
      if (more) fmode = face_mode(tile + step, small_s + bn * C::SMALL, gn);
      const bool reload = more && fmode == 0;
      if (mode >= 0) {
        unsigned char* fdst = stage + foff;
        if (mode == 0) {
#pragma unroll
          for (int c = 0; c < NU; ++c) {
            float hi, lo;
            split_f32((nb[c] - u0_b[c * EPB + fe]) * 0.5f, hi, lo);
            if (reload) nb[c] = face_load(gn, c);
            const int o = c * EPM * 16;
            *reinterpret_cast<float*>(fdst + o) = hi;
            *reinterpret_cast<float*>(fdst + o + C::A_BYTES) = lo;
          }
        } else {
          const int64_t gm = (int64_t)(tile * EPB + fe) * NP + fk;
          float up[NU];
          if (mode != 2) {
            const int bf = -((int)small_b[fe * NF + ff] + 1);
            if (mode == 3) {
              float nv[3] = {0.f, 0.f, 0.f}, mag2 = 0.f;
#pragma unroll
              for (int j = 0; j < DIM; ++j) {
#pragma unroll
                for (int r = 0; r < DIM; ++r)
                  nv[j] += rx_b[fe * DD + r * DIM + j] *
                           RefBank<float>::get(S::OFF_NREF + ff * DIM + r);
                mag2 += nv[j] * nv[j];
              }
              const float mag = sqrtf(mag2);
              mengaldo_grad_value<float, DIM, NS, true>(a, g, a.bkind[bf], bf, fm_, NFP, EN, gm,
                                                        nv[0] / mag, nv[1] / mag, nv[2] / mag, up);
            } else {
              const int64_t bstride = (int64_t)a.nbf * NFP, bo = (int64_t)bf * NFP + fm_;
#pragma unroll
              for (int c = 0; c < NU; ++c) up[c] = a.bext[c * bstride + bo];
            }
          }
#pragma unroll 1
          for (int c = 0; c < NU; ++c) {
            const float u0 = u0_b[c * EPB + fe];
            const float um = __ldg(field(c) + gm) - u0;
            float hi, lo;
            split_f32(mode == 2 ? um * 0.5f : (up[c] - u0) - um * 0.5f, hi, lo);
            const int o = c * EPM * 16;
            *reinterpret_cast<float*>(fdst + o) = hi;
            *reinterpret_cast<float*>(fdst + o + C::A_BYTES) = lo;
          }
        }
      }
      if (mode != 0 && reload) {
#pragma unroll
        for (int c = 0; c < NU; ++c) nb[c] = face_load(gn, c);
      }
      // ---- the epilogue's copy of the metric; per-tile data two tiles ahead
      // (into the buffer of the tile before this one)
      for (int i = tid; i < ne * DD; i += GT) geo_s[s * EPB * DD + i] = rx_b[i];
      if (more2) small_store(w, bn == 2 ? 0 : bn + 1);
      fence_async_shared();
      mbar_arrive(full + s);
      if (tid == GT - 1) pending = it;
      b = bn;
    }
    // the last tile's products (after a normal end of the loop)
    if (tid == GT - 1 && pending >= 0 && !*abort_s) issue_pending();
    // on an early exit, let the products already issued finish before the
    // TMEM is released
    if (tid == GT - 1 && *abort_s && issued > 0) {
      if (!mbar_wait(done + (last_issued & 1), ((uint32_t)last_issued >> 1) & 1, nullptr))
        atomicOr(a.status, ST_WAIT_TIMEOUT);
    }
  } else {
    // ================= epilogue: one TMEM lane (row) per thread
    const int q4 = warp & 3;
    const int row = 32 * q4 + lane;
    const int c = row / EPM, el = row % EPM;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * q4) << 16);
    for (int it = 0, tile = blockIdx.x; tile < ntiles; ++it, tile += gridDim.x) {
      const int s = it & 1;
      const uint32_t use = (uint32_t)it >> 1;
      // the products of this tile, then (already complete) the producers'
      // arrival, whose release covers the metric they wrote
      bool ok = mbar_wait(done + s, use & 1, abort_s);
      ok = ok && mbar_wait(full + s, use & 1, abort_s);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) {
          atomicOr(a.status, ST_WAIT_TIMEOUT);
          *abort_s = 1;
        }
        break;
      }
      tc_fence_after();
      const int e0 = tile * EPB;
      const int ne = imin(EPB, EOWN - e0);
#pragma unroll 1
      for (int mt = 0; mt < NMT; ++mt) {
        const int e = mt * EPM + el;
        uint32_t v[NV];
#pragma unroll
        for (int i = 0; i < NV; i += 16)
          tc_ld16(lane_base + (uint32_t)(s * C::BUF_COLS + mt * NV + i), v + i);
        tc_wait_ld<NV>(v);
        if (c < NU && e < ne) {
          const float* ge = geo_s + (s * EPB + e) * DD;
          float rxe[DIM][DIM];
#pragma unroll
          for (int r = 0; r < DIM; ++r)
#pragma unroll
            for (int j = 0; j < DIM; ++j) rxe[r][j] = ge[r * DIM + j];
          float* outp = a.out + ((int64_t)c * DIM) * EN + (int64_t)(e0 + e) * NP;
#pragma unroll
          for (int j = 0; j < DIM; ++j)
#pragma unroll
            for (int i0 = 0; i0 < NP; i0 += VW) {
              float o[VW];
#pragma unroll
              for (int i = 0; i < VW; ++i) {
                float gsum = 0.f;
#pragma unroll
                for (int r = 0; r < DIM; ++r)
                  gsum += rxe[r][j] * __uint_as_float(v[r * NP + i0 + i]);
                o[i] = gsum;
              }
              float* dst = outp + (int64_t)j * EN + i0;
              if constexpr (VW == 4)
                *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
              else
                *reinterpret_cast<float2*>(dst) = make_float2(o[0], o[1]);
            }
        }
      }
      tc_fence_before();
      mbar_arrive(empty + s);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) {
    __syncwarp();
    tc_dealloc(tmem, C::TCOLS);
  }
}

}  // namespace

}  // namespace mgc
