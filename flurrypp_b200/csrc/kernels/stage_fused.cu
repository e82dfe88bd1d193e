// One RK stage of an inviscid static case in one launch: common face flux,
// transformed flux, divergence, correction, RK update and the extrapolation
// of the new state to the flux points (reference: solver.cpp:366-445,
// 470-572), FP64 plain form and FP32 precision form.
//
// The two-kernel form of a stage writes the common flux of every face point
// to both of its sides and reads it back: at 3-D P3 the face table and Fn are
// 1776 of the stage's 4496 words per element.  Here every element forms the
// flux of its own face points from its own trace and the neighbour's, so a
// face is evaluated twice (from either side, with the same operands up to the
// sign of the normal, so both sides get the same bits) and only the
// neighbour's trace and this side's normal and area are read (912 words).
// The traces alternate between two buffers, since neighbours still read the
// old ones while this stage writes the new ones.
//
// Work split: a CTA takes EB elements and has one thread per line (of every
// dimension) and element.  A thread forms the common flux at both ends of its
// line, from neighbour records that it copied itself (cp.async, so no barrier
// between the copy and its use), and the divergence and correction along it;
// the points' fluxes and updates are spread over all threads.  Each dimension's
// flux has a slab of shared memory; one slab takes the state tile's place.
//
// Metrics, normals, neighbour slots and the step's base state are read from
// copies laid out in thread order (launch_fused_pack): one coalesced access
// per value and no shared memory.
//
// What bounds it: 3-D P3 FP64 at 32^3, an intermediate stage 0.187 ms for
// 940 MB of DRAM traffic (5.03 TB/s, 0.77 of the measured copy rate; faces
// and elements as two launches 0.063 + 0.170 ms), the rest the latency of its
// barrier-separated phases at 18 warps per SM (96 registers); FP32 0.117 ms
// (0.035 + 0.101 ms), 450 MB.  Four steps, two launches a stage -> one:
// 3-D P3 32^3 3.71 -> 2.98 ms, FP32 2.16 -> 1.85; 3-D P2 27^3 (rows without
// TMA) 1.89 -> 1.02; 2-D P3 256^2 1.05 -> 0.91, FP32 0.58 -> 0.43; 2-D P2
// 384^2 FP32 0.81 -> 0.66; 20 steps of 2-D P3 32^2 206 -> 160 us.
// Tried and slower: one thread per line of one dimension only, working on all
// three (half the threads: 3.33 ms at 32^3, 236 us at 32^2); element counts
// of half or twice the ones below; starting the next wave's tiles for L2 ahead
// (DRAM reads +44 %, 3.66 ms).
#include <type_traits>

#include "launch.cuh"
#include "stage.hpp"
#include "tma.cuh"

namespace frk {

namespace {

constexpr int ipw(int b, int e) { return e == 0 ? 1 : b * ipw(b, e - 1); }
constexpr int kLeftBit = 1 << 30;
constexpr size_t kSmemPerSm = 228 * 1024;

// Elements per CTA: enough for a few warps, few enough for several CTAs per
// SM, whose load phases then fall behind the others' arithmetic.
template <int ND, int P, typename R>
constexpr int fused_eb() {
  constexpr bool f32 = sizeof(R) == 4;
  if (ND == 2) return P == 0 ? 32 : 16;
  return P == 0 ? 32 : P == 1 ? 16 : P == 2 ? 8 : P == 3 ? 4 : (f32 || P == 4) ? 4 : 2;
}

// Worst number of lanes of a warp (FP64: half warp) on one bank for the
// x-line pattern of a slab whose rows of N points are PAD words apart beyond
// dense.
constexpr int xline_conflict(int n, int eb, int nf, int pad, bool f32) {
  const int lanes = f32 ? 32 : 16, banks = f32 ? 32 : 16;
  int worst = 0;
  for (int b = 0; b < banks; b++) {
    int hits = 0;
    for (int l = 0; l < lanes; l++) {
      const int c = l / eb, el = l % eb;
      if ((c * (n * eb * nf + pad) + el * nf) % banks == b) hits++;
    }
    worst = hits > worst ? hits : worst;
  }
  return worst;
}
constexpr int best_pad(int n, int eb, int nf, bool f32) {
  int best = 0;
  for (int p = 1; p <= 8; p++)
    if (xline_conflict(n, eb, nf, p, f32) < xline_conflict(n, eb, nf, best, f32)) best = p;
  return best;
}

template <int ND, int P, typename R>
struct Fz {
  static constexpr bool F32 = sizeof(R) == 4;
  static constexpr int N = P + 1, NF = ND + 2, NS = ipw(N, ND), NC = ipw(N, ND - 1), NFP = 2 * ND * NC;
  static constexpr int EB = fused_eb<ND, P, R>();
  static constexpr int NT = ND * NC * EB, NPT = NS * EB, ROW = EB * NF;  // threads, points, point row
  static constexpr int AL = 128 / (int)sizeof(R);
  static constexpr int al(int n) { return (n + AL - 1) / AL * AL; }
  // 3-D slabs are padded after each row of N points so that x-lines of one
  // warp fall on distinct banks (P3: 4 values; unpadded they are 4 deep);
  // 2-D records are contiguous over the warp already
  static constexpr int PAD = ND == 3 ? best_pad(N, EB, NF, F32) : 0;
  static constexpr int XROW = N * ROW + PAD;
  static constexpr int SLAB = NS / N * XROW;
  // x flux (padded in 3-D), 3-D: y flux; the last dimension's flux takes the
  // place of the state tile, which is dead once the traces are formed (every
  // thread writes the points it read)
  static constexpr int O_U = 0;
  static constexpr int O_X = al(NS * ROW);
  static constexpr int O_Y = O_X + al(SLAB);
  static constexpr int O_Q = O_Y + (ND == 3 ? al(NS * ROW) : 0);
  static constexpr int O_E = O_Q + al(NFP * ROW);
  static constexpr int O_BAR = O_E + al(4 * N);
  static constexpr size_t SMEM = sizeof(R) * (size_t)O_BAR + 16 + 128;
  static constexpr int WT = (NT + 31) / 32 * 32;
  // registers a thread needs before another CTA per SM pays (measured, ms of
  // four steps: FP64 3-D P3 96 2.99, 128 3.09; P4 96 1.59, 112 1.86; 2-D P5
  // 96 0.62, 128 0.48; FP32 3-D P3 64 1.95, 80 1.88, 96 2.09; 2-D P3 64 0.42,
  // 80 0.45)
  static constexpr int minRegs() {
    return F32 ? (ND == 3 && P == 3 ? 80 : 64) : ND == 2 ? (P == 5 ? 128 : 112) : P == 3 || P == 4 ? 96 : 112;
  }
  static constexpr int ctas(int c) { return c <= 1 || 65536 / (WT * c) >= minRegs() ? c : ctas(c - 1); }
  static constexpr int MINB0 = ctas((int)(kSmemPerSm / (SMEM + 1024)) < 24 ? (int)(kSmemPerSm / (SMEM + 1024)) : 24);
  static constexpr int MINB = MINB0 < 1 ? 1 : MINB0;
  static_assert(NT * (int)sizeof(R) % 16 == 0 && NPT * (int)sizeof(R) % 16 == 0 && NT % 2 == 0, "prefetch regions");
  static_assert(SMEM <= 227 * 1024, "fused stage tiles do not fit in shared memory");
  static_assert(NT <= 1024 && ROW <= 256, "fused stage block shape");
};

// A point's NF values in shared memory: 2-D records move as 128-bit accesses
// (FP64: two, in the order that keeps eight lanes on distinct banks, see
// stage_tma.cu), 3-D ones per value.
template <int NF, typename R>
__device__ __forceinline__ void lds(const R *p, R (&v)[NF]) {
  if constexpr (NF == 4 && sizeof(R) == 4) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else if constexpr (NF == 4) {
    const int h = (int)((smem_u32(p) >> 7) & 1);
    const double2 a = reinterpret_cast<const double2 *>(p)[h], b = reinterpret_cast<const double2 *>(p)[h ^ 1];
    v[0] = h ? b.x : a.x, v[1] = h ? b.y : a.y, v[2] = h ? a.x : b.x, v[3] = h ? a.y : b.y;
  } else {
#pragma unroll
    for (int k = 0; k < NF; k++) v[k] = p[k];
  }
}
template <int NF, typename R>
__device__ __forceinline__ void sts(R *p, const R (&v)[NF]) {
  if constexpr (NF == 4 && sizeof(R) == 4) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else if constexpr (NF == 4) {
    const int h = (int)((smem_u32(p) >> 7) & 1);
    reinterpret_cast<double2 *>(p)[h] = h ? make_double2(v[2], v[3]) : make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(p)[h ^ 1] = h ? make_double2(v[0], v[1]) : make_double2(v[2], v[3]);
  } else {
#pragma unroll
    for (int k = 0; k < NF; k++) p[k] = v[k];
  }
}
template <int NF, typename R>
__device__ __forceinline__ void ldg_rec(const R *p, R (&v)[NF]) {
  if constexpr (NF == 4 && sizeof(R) == 4) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else if constexpr (NF == 4) {
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  } else {
#pragma unroll
    for (int k = 0; k < NF; k++) v[k] = p[k];
  }
}

template <int NF, typename R>
__device__ __forceinline__ void stg_rec(R *p, const R (&v)[NF]) {
  if constexpr (NF == 4 && sizeof(R) == 4) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else if constexpr (NF == 4) {
    reinterpret_cast<double2 *>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(v[2], v[3]);
  } else {
#pragma unroll
    for (int k = 0; k < NF; k++) p[k] = v[k];
  }
}
// Start a contiguous region (16-byte aligned, a multiple of 16 bytes) on its way to L2.
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Neighbour record global -> shared, asynchronously: 16-byte words in 2-D
// (records are 16-byte aligned), single values in 3-D.
template <int NF, typename R>
__device__ __forceinline__ void copy_rec_async(R *dst, const R *src) {
  if constexpr (NF == 4) {
#pragma unroll
    for (int i = 0; i < NF * (int)sizeof(R) / 16; i++)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst) + 16 * i),
                   "l"(reinterpret_cast<const char *>(src) + 16 * i)
                   : "memory");
  } else {
#pragma unroll
    for (int k = 0; k < NF; k++) cp_async_word(dst + k, src + k);
  }
}

// s + e = a + b exactly (Knuth's TwoSum)
__device__ __forceinline__ void two_sum_f(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}



template <int ND, typename R>
__device__ __forceinline__ void ghost_state(int bc, const R *UL, const R *n, const Phys &ph, R *UR) {
  boundary_state<ND, R>(bc, UL, n, ph, UR);
}

// Common flux times dA at one face point of this element, on its outward
// normal; nb is the neighbour's slot (with kLeftBit where this side is the
// face's left side) or -(bc + 2).  Rusanov's flux is antisymmetric bit for
// bit under exchanging the sides and the normal's sign; Roe's is evaluated
// from the left side always.
template <int ND, bool ROE, typename R>
__device__ __forceinline__ void end_flux(const R (&own)[ND + 2], const R *sNb, int nb, const R (&n)[ND], R dA,
                                         const Phys &ph, double *ws, R (&Fn)[ND + 2]) {
  constexpr int NF = ND + 2;
  R other[NF];
  if (nb < 0) {
    R o[NF], u[NF], m[ND];
#pragma unroll
    for (int k = 0; k < NF; k++) u[k] = own[k];
#pragma unroll
    for (int d = 0; d < ND; d++) m[d] = n[d];
    ghost_state<ND, R>(-nb - 2, u, m, ph, o);
#pragma unroll
    for (int k = 0; k < NF; k++) other[k] = o[k];
  } else {
    lds<NF, R>(sNb, other);
  }
  const bool left = nb < 0 || (nb & kLeftBit);
  if constexpr (ROE) {
    if (nb >= 0) {
      R a[NF], b[NF], m[ND];
#pragma unroll
      for (int k = 0; k < NF; k++) {
        a[k] = left ? own[k] : other[k];
        b[k] = left ? other[k] : own[k];
      }
#pragma unroll
      for (int d = 0; d < ND; d++) m[d] = left ? n[d] : -n[d];
      roe2d<R>(a, b, m, R(ph.gamma), Fn);
      const R s = left ? dA : -dA;
#pragma unroll
      for (int k = 0; k < NF; k++) Fn[k] = Fn[k] * s;
      return;
    }
  }
  const R w = rusanov<ND, R>(own, other, n, R(ph.gamma), Fn);
  if (ws && left) *ws = w;
#pragma unroll
  for (int k = 0; k < NF; k++) Fn[k] = Fn[k] * dA;
}

// Traces at both ends of a line of a dense tile (the state), N records apart
// by `step`, summed in ascending order as everywhere.  ROT (3-D P3): the
// x-lines' records start a multiple of 128 bytes apart, four deep on the same
// banks, so a lane reads them from its own point on (rot), which spreads the
// warp over the banks, and turns them back in registers.
template <int N, int NF, bool ROT, typename R>
__device__ __forceinline__ void line_ends(const R *base, int step, int rot, const R *sE, R (&t)[2][NF]) {
  R x[N][NF];
  if constexpr (ROT) {
    static_assert(N == 4, "two conditional turns");
    int m = rot;
#pragma unroll
    for (int i = 0; i < N; i++) {
      lds<NF, R>(base + m * step, x[i]);
      m = (m + 1) & 3;
    }
    if (rot != 0) {  // x[i] holds point (i + rot) % 4
#pragma unroll
      for (int k = 0; k < NF; k++) {
        const R a = x[0][k], b = x[1][k], c = x[2][k], d = x[3][k];
        const bool r1 = rot & 1, r2 = rot & 2;
        const R e = r1 ? d : a, f = r1 ? a : b, g = r1 ? b : c, h = r1 ? c : d;
        x[0][k] = r2 ? g : e;
        x[1][k] = r2 ? h : f;
        x[2][k] = r2 ? e : g;
        x[3][k] = r2 ? f : h;
      }
    }
  } else {
#pragma unroll
    for (int m = 0; m < N; m++) lds<NF, R>(base + m * step, x[m]);
  }
#pragma unroll
  for (int k = 0; k < NF; k++) t[0][k] = t[1][k] = R(0);
#pragma unroll
  for (int m = 0; m < N; m++) {
    const R e0 = sE[m], e1 = sE[N + m];
#pragma unroll
    for (int k = 0; k < NF; k++) {
      t[0][k] += e0 * x[m][k];
      t[1][k] += e1 * x[m][k];
    }
  }
}

// Along a line with flux values x: q comes in as the end fluxes and leaves as
// the end jumps (flux minus extrapolated flux); y is the divergence, with
// CORR plus the correction from both ends.  Every sum starts from zero, as in
// the other element kernels, for the same contractions; the FP32 correction's
// contraction is written out, as the compiler forms it in k_elem_tma's line
// pass (started from zero it rounds the other product: 1 to 17 % of the FP32
// residuals moved by a last bit, and their FP64 norm by up to 4e-9).
template <int N, int NF, bool CORR, typename R>
__device__ __forceinline__ void line_div(const FusedArgsT<R> &a, const R (&x)[N][NF], R (&q)[2][NF], R (&y)[N][NF]) {
#pragma unroll
  for (int s = 0; s < 2; s++)
#pragma unroll
    for (int k = 0; k < NF; k++) {
      R t = R(0);
#pragma unroll
      for (int m = 0; m < N; m++) t += a.EFn1[s * N + m] * x[m][k];
      q[s][k] = q[s][k] - t;
    }
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int k = 0; k < NF; k++) {
      R acc = R(0), c = R(0);
#pragma unroll
      for (int m = 0; m < N; m++) acc += a.D[i * N + m] * x[m][k];
      if constexpr (CORR) {
        if constexpr (sizeof(R) == 4) {
          c = fmaf(a.C[i], q[0][k], __fmul_rn(a.C[N + i], q[1][k]));
        } else {
          c += a.C[i] * q[0][k];
          c += a.C[N + i] * q[1][k];
        }
        y[i][k] = c + acc;
      } else {
        y[i][k] = acc;
      }
    }
}

template <int ND, int P, typename R, bool TMA, bool ROE>
__global__ void __launch_bounds__(Fz<ND, P, R>::NT, Fz<ND, P, R>::MINB)
    k_fused_stage(const __grid_constant__ FusedArgsT<R> a, const __grid_constant__ FusedMaps mp) {
  using T = Fz<ND, P, R>;
  constexpr bool F32 = T::F32;
  constexpr int N = T::N, NF = T::NF, NS = T::NS, NC = T::NC, NFP = T::NFP, EB = T::EB, NT = T::NT, ROW = T::ROW;
  constexpr int NPT = T::NPT, XROW = T::XROW;
  constexpr int PT = (NPT + NT - 1) / NT;  // points per thread
  // where the correction is added: line by line, per direction, in 3-D FP64
  // and in 3-D FP32 with TMA rows, as k_elem_tma does; at the points, after the
  // directions' sum and in the reference's face order, in 2-D and in 3-D FP32
  // without TMA rows, as k_elem_tp does.  This makes 2-D and FP32 steps
  // bit-identical to the two-kernel form's (20 steps of 32^2 P3 FP64 145 -> 160
  // us; FP32 384^2 P2 653 -> 663 us, 256^2 P3 414 -> 431; a run beyond its
  // stability limit amplifies a last bit to 1e-11 in 20 steps); FP64 3-D differs
  // in last bits (both its two-kernel forms add at the points)
  constexpr bool CORR = ND == 3 && (!F32 || TMA);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R *smem = reinterpret_cast<R *>(smem_align128(smem_raw));
  R *sU = smem + T::O_U, *sX = smem + T::O_X, *sY = smem + T::O_Y, *sQ = smem + T::O_Q, *sE = smem + T::O_E;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + T::O_BAR);

  const int tid = threadIdx.x;
  const int E = a.E, e0 = blockIdx.x * EB;
  const int nValid = min(EB, E - e0);
  // this thread's line: dimension, transverse index, element
  const int dim = tid / (NC * EB), col = tid / EB - dim * NC, el = tid % EB;
  const bool valid = el < nValid;
  const long long blk = blockIdx.x;
  const R *jgp = a.jg + blk * ND * ND * NPT, *rdp = a.rdet + blk * NPT;
  R *X0p = a.X0 + blk * NF * NPT, *Sp = a.S + blk * NF * NPT;
  const bool final = a.mode == FUSED_FINAL, residual = a.mode == FUSED_RESIDUAL;

  // setup data (not written by the preceding kernel) before the wait; the
  // block's metrics, used phases later, start for L2 now
  const int fp = __ldg(&a.lineF[dim * NC + col]);
  int nb[2];
  R nv[2][ND], dA[2];
#pragma unroll
  for (int s = 0; s < 2; s++) nb[s] = __ldg(a.nb + (blk * 2 + s) * NT + tid);
  if (tid == 0) {
    if (TMA) {
      mbar_init(bar, 1);
      fence_mbar_init();
    }
    prefetch_l2(jgp, ND * ND * NPT * sizeof(R));
    if (!residual) prefetch_l2(rdp, NPT * sizeof(R));
  }
#pragma unroll
  for (int s = 0; s < 2; s++) {
    const R *g = a.nrm + (blk * 2 + s) * (ND + 1) * NT + tid;
#pragma unroll
    for (int q = 0; q < ND; q++) nv[s][q] = __ldg(g + q * NT);
    dA[s] = __ldg(g + ND * NT);
  }
  for (int i = tid; i < 2 * N; i += NT) {
    sE[i] = a.E1[i];
    sE[2 * N + i] = a.C[i];
  }
  pdl_wait();
  pdl_trigger();

  if constexpr (TMA) {
    if (tid == 0) {
      mbar_arrive_expect_tx(bar, sizeof(R) * NS * ROW);
      tma_load_2d(sU, &mp.in, e0 * NF, 0, bar);
    }
  } else {
    for (int i = tid; i < NS * ROW; i += NT) {
      const int p = i / ROW, r = i - p * ROW;
      if (r < nValid * NF) cp_async_word(&sU[i], &a.Uin[((long long)p * E + e0) * NF + r]);
    }
    cp_async_commit();
  }
  // the neighbours' traces at both ends of this thread's line
  R *q0 = &sQ[(fp & 0xffff) * ROW + el * NF], *q1 = &sQ[(fp >> 16) * ROW + el * NF];
  if (valid && nb[0] >= 0) copy_rec_async<NF, R>(q0, &a.Ufin[(long long)(nb[0] & (kLeftBit - 1)) * NF]);
  if (valid && nb[1] >= 0) copy_rec_async<NF, R>(q1, &a.Ufin[(long long)(nb[1] & (kLeftBit - 1)) * NF]);
  cp_async_commit();
  if (tid == 0 && !a.first && !residual) {
    prefetch_l2(X0p, NF * NPT * sizeof(R));
    if (a.loadS) prefetch_l2(Sp, NF * NPT * sizeof(R));
  }

  if constexpr (TMA) {
    __syncthreads();  // barrier object, sE
    if (!mbar_wait_bounded(bar, 0, 1u << 22)) {
      // give up: flag it, so that the host discards what this stage gives, and
      // let the copy in flight land (bounded).  The thread goes on, since the
      // block's barriers and tile stores need all of them; no index depends on
      // the tile.  (Leaving as a block, by a voting barrier here or after the
      // traces, took 3 % more in a batch of 24 FP32 vortex cases: 2937 -> 3030 us.)
      if (a.err) atomicOr(a.err, 1);
      mbar_wait_bounded(bar, 0, 1u << 22);
    }
  } else {
    cp_async_wait<1>();
    __syncthreads();
  }

  // A: common flux times area at both ends of the line, in place of the
  // neighbours' records
  const int base = dim == ND - 1 ? col : dim == 0 ? col * N : col % N + col / N * (N * N);
  const int stride = dim == ND - 1 ? NC : dim == 0 ? 1 : N;
  constexpr bool ROT = ND == 3 && P == 3;
  const int rot = (ROT && dim == 0) ? col % N : 0;
  {
    R t[2][NF], f0[NF], f1[NF];
    line_ends<N, NF, ROT, R>(&sU[base * ROW + el * NF], stride * ROW, rot, sE, t);
    cp_async_wait<0>();  // this thread's neighbour records
    double *w0 = nullptr, *w1 = nullptr;
    if (a.waveSp && valid) {
      w0 = &a.waveSp[(long long)(fp & 0xffff) * E + e0 + el];
      w1 = &a.waveSp[(long long)(fp >> 16) * E + e0 + el];
    }
    end_flux<ND, ROE, R>(t[0], q0, valid ? nb[0] : 0, nv[0], dA[0], a.ph, w0, f0);
    end_flux<ND, ROE, R>(t[1], q1, valid ? nb[1] : 0, nv[1], dA[1], a.ph, w1, f1);
    sts<NF, R>(q0, f0);
    sts<NF, R>(q1, f1);
  }
  if constexpr (TMA) {  // the step's base state for the caller's U0 array
    if (a.keepU0 && tid == 0) {
      tma_store_2d(&mp.keep, e0 * NF, 0, sU);
      tma_commit();
      tma_wait_read_all();
    }
  } else {
    if (a.keepU0)
      for (int i = tid; i < NS * ROW; i += NT) {
        const int p = i / ROW, r = i - p * ROW;
        if (r < nValid * NF) a.U0keep[((long long)p * E + e0) * NF + r] = sU[i];
      }
  }
  // the points' metrics (one point ahead) and what their update reads
  R J[ND * ND], x0[PT][NF], ss[F32 ? PT : 1][NF], rd[PT];
#pragma unroll
  for (int q = 0; q < ND * ND; q++) J[q] = tid < NPT ? __ldg(jgp + q * NPT + tid) : R(0);
#pragma unroll
  for (int i = 0; i < PT; i++) {
    const int it = min(tid + i * NT, NPT - 1);
    rd[i] = residual ? R(0) : __ldg(rdp + it);
#pragma unroll
    for (int k = 0; k < NF; k++) {
      // FP64: the last stage starts from the running sum, the others from
      // the base state; FP32 adds its sum of increments to the base state
      x0[i][k] = a.first ? R(0) : (!F32 && final && a.loadS) ? Sp[k * NPT + it] : X0p[k * NPT + it];
      if constexpr (F32) ss[i][k] = a.loadS ? Sp[k * NPT + it] : R(0);
    }
  }
  __syncthreads();  // every line of the state tile has been read

  // B: reference-space flux at the points
#pragma unroll
  for (int i = 0; i < PT; i++) {
    const int it = tid + i * NT;
    if (NPT % NT != 0 && it >= NPT) break;
    const int p = it / EB, o = (it % EB) * NF;
    R u[NF], Fp[ND][NF], Jm[ND * ND];
    lds<NF, R>(&sU[p * ROW + o], u);
#pragma unroll
    for (int q = 0; q < ND * ND; q++) Jm[q] = J[q];
    if (i + 1 < PT)
#pragma unroll
      for (int q = 0; q < ND * ND; q++) J[q] = it + NT < NPT ? __ldg(jgp + q * NPT + it + NT) : R(0);
    if (a.first)  // the base state in thread order
#pragma unroll
      for (int k = 0; k < NF; k++) {
        x0[i][k] = u[k];
        if (!residual) X0p[k * NPT + it] = u[k];
      }
    inviscid_flux<ND, R>(u, Fp, R(a.ph.gamma));
#pragma unroll
    for (int d1 = 0; d1 < ND; d1++) {
      R f[NF];
#pragma unroll
      for (int k = 0; k < NF; k++) {
        f[k] = R(0);
#pragma unroll
        for (int d2 = 0; d2 < ND; d2++) f[k] += Jm[d1 * ND + d2] * Fp[d2][k];
      }
      sts<NF, R>(d1 == 0 ? &sX[p / N * XROW + p % N * ROW + o] : d1 == ND - 1 ? &sU[p * ROW + o] : &sY[p * ROW + o], f);
    }
  }
  const double dtIn0 = residual ? 0.0 : *a.dt;
  __syncthreads();  // fluxes written

  // C: divergence and correction along the line, in place
  {
    R x[N][NF], y[N][NF], q[2][NF];
    R *g = (dim == 0 ? sX + col * XROW : dim == ND - 1 ? sU + base * ROW : sY + base * ROW) + el * NF;
    const int gs = stride * ROW;
#pragma unroll
    for (int m = 0; m < N; m++) lds<NF, R>(g + m * gs, x[m]);
    lds<NF, R>(q0, q[0]);
    lds<NF, R>(q1, q[1]);
    line_div<N, NF, CORR, R>(a, x, q, y);
    if constexpr (!CORR) {
      sts<NF, R>(q0, q[0]);
      sts<NF, R>(q1, q[1]);
    }
#pragma unroll
    for (int m = 0; m < N; m++) sts<NF, R>(g + m * gs, y[m]);
  }
  __syncthreads();  // divergences complete

  // D: sum over dimensions and RK update at the points
  R cmp[F32 ? PT : 1][NF];  // FP32 final stage: the state's rounding remainder
  R div[PT][NF];
#pragma unroll
  for (int i = 0; i < PT; i++) {
    const int it = tid + i * NT;
    if (NPT % NT != 0 && it >= NPT) break;
    const int p = it / EB, pe = it % EB, o = pe * NF;
    R s1[NF];
    lds<NF, R>(&sX[p / N * XROW + p % N * ROW + o], div[i]);
    if constexpr (ND == 3) {
      lds<NF, R>(&sY[p * ROW + o], s1);
#pragma unroll
      for (int k = 0; k < NF; k++) div[i][k] += s1[k];
    }
    lds<NF, R>(&sU[p * ROW + o], s1);
#pragma unroll
    for (int k = 0; k < NF; k++) div[i][k] += s1[k];
    if constexpr (!CORR) {
      const int x = p % N, y = ND == 2 ? p / N : p / N % N;
      int f[2 * ND];
      R c[2 * ND];
      const R *c0 = sE + 2 * N, *c1 = sE + 3 * N;  // the correction of the two sides along a line
      if constexpr (ND == 2) {
        const int fx = __ldg(&a.lineF[y]), fy = __ldg(&a.lineF[NC + x]);
        f[0] = fy & 0xffff, f[1] = fx >> 16, f[2] = fy >> 16, f[3] = fx & 0xffff;  // bottom, right, top, left
        c[0] = c0[y], c[1] = c1[x], c[2] = c1[y], c[3] = c0[x];
      } else {  // bottom, top, left, right, front, back
        const int z = p / (N * N);
        const int fz = __ldg(&a.lineF[2 * NC + x + N * y]), fx = __ldg(&a.lineF[y + N * z]),
                  fy = __ldg(&a.lineF[NC + x + N * z]);
        f[0] = fz & 0xffff, f[1] = fz >> 16, f[2] = fx & 0xffff, f[3] = fx >> 16;
        f[2 * ND - 2] = fy & 0xffff, f[2 * ND - 1] = fy >> 16;
        c[0] = c0[z], c[1] = c1[z], c[2] = c0[x], c[3] = c1[x], c[2 * ND - 2] = c0[y], c[2 * ND - 1] = c1[y];
      }
      R cq[NF];
#pragma unroll
      for (int k = 0; k < NF; k++) cq[k] = R(0);
#pragma unroll
      for (int j = 0; j < 2 * ND; j++) {
        R q[NF];
        lds<NF, R>(&sQ[f[j] * ROW + o], q);
#pragma unroll
        for (int k = 0; k < NF; k++) cq[k] += c[j] * q[k];
      }
#pragma unroll
      for (int k = 0; k < NF; k++) div[i][k] = cq[k] + div[i][k];
    }
    if (residual) continue;
    const bool ok = pe < nValid;
    const long long gi = ((long long)p * E + e0 + pe) * NF;
    R un[NF], cm[NF], sv[NF];
    if constexpr (!F32)
#pragma unroll
      for (int k = 0; k < NF; k++) sv[k] = a.loadS && a.saveS ? Sp[k * NPT + it] : x0[i][k];
#pragma unroll
    for (int k = 0; k < NF; k++) cm[k] = R(0);
    if constexpr (F32)
      if (final && ok) ldg_rec<NF, R>(&a.comp[gi], cm);
    const R dt = R(a.eleDt ? (ok ? a.eleDt[e0 + pe] : 0.0) : dtIn0);
#pragma unroll
    for (int k = 0; k < NF; k++) {
      R dv = div[i][k];
      if (a.src && ok) dv = dv + a.src[gi + k];
      const R inc = dv * rd[i] * dt;
      if constexpr (!F32) {
        // the reference's order of operations (timeStepA, timeStepB)
        un[k] = x0[i][k] - (final ? a.rkb : a.rka) * dv * rd[i] * dt;
        sv[k] = sv[k] - a.rkb * dv * rd[i] * dt;
      } else if (!final) {
        un[k] = x0[i][k] - R(a.rka) * inc;
        if (a.saveS) Sp[k * NPT + it] = ss[i][k] - R(a.rkb) * inc;
      } else {
        R c;
        two_sum_f(x0[i][k], cm[k] + (ss[i][k] - R(a.rkb) * inc), un[k], c);
        cmp[i][k] = c;
      }
    }
    sts<NF, R>(&sU[p * ROW + o], un);
    if constexpr (!F32)
      if (a.saveS)
#pragma unroll
        for (int k = 0; k < NF; k++) Sp[k * NPT + it] = sv[k];
  }
  // optional outputs, staged densely through the x slab: the residual; FP32
  // final stage: the remainder
  const auto store_tile = [&](const R *tile, R *out, int rows) {
    for (int i = tid; i < rows * ROW; i += NT) {
      const int p = i / ROW, r = i - p * ROW;
      if (r < nValid * NF) out[((long long)p * E + e0) * NF + r] = tile[i];
    }
  };
  const auto stage_out = [&](const R (&v)[PT][NF], R *out) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PT; i++)
      if (NPT % NT == 0 || tid + i * NT < NPT) sts<NF, R>(&sX[(tid + i * NT) * NF], v[i]);
    __syncthreads();
    store_tile(sX, out, NS);
  };
  if (a.divF) stage_out(div, a.divF);
  if constexpr (F32)
    if (final) stage_out(cmp, a.comp);
  if (residual) return;

  // E: traces of the new state
  if (TMA) fence_async_smem();
  __syncthreads();  // the new state is complete
  if constexpr (TMA) {
    if (tid == 0) {
      tma_store_2d(&mp.out, e0 * NF, 0, sU);
      tma_commit();
    }
  }
  {
    R t[2][NF];
    line_ends<N, NF, ROT, R>(&sU[base * ROW + el * NF], stride * ROW, rot, sE, t);
    sts<NF, R>(q0, t[0]);
    sts<NF, R>(q1, t[1]);
  }
  if (TMA) fence_async_smem();
  __syncthreads();
  if constexpr (TMA) {
    if (tid == 0) {
      tma_store_2d(&mp.tr, e0 * NF, 0, sQ);
      tma_commit();
      tma_wait_read_all();
    }
  } else {
    store_tile(sU, a.Uout, NS);
    store_tile(sQ, a.Ufout, NFP);
  }
  if (final && a.timeAcc && blockIdx.x == 0 && tid == 0) *a.timeAcc += *a.dt;
}

// Thread-order copies of the metrics and the face table (set up once):
// points [block][value][point, element], line ends [block][side][value][line, element].
template <typename R>
__global__ void k_pack_points(int nd, int nS, int EB, int E, const R *__restrict__ JG, const R *__restrict__ det,
                              R *__restrict__ jg, R *__restrict__ rdet, long long total) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // (block, point, element)
  if (i >= total) return;
  const int npt = nS * EB;
  const long long blk = i / npt;
  const int it = (int)(i - blk * npt), p = it / EB;
  const long long e = blk * EB + it % EB;
  for (int d1 = 0; d1 < nd; d1++)
    for (int d2 = 0; d2 < nd; d2++)
      jg[(blk * nd * nd + d1 * nd + d2) * npt + it] = e < E ? JG[(((long long)d1 * nS + p) * E + e) * nd + d2] : R(0);
  rdet[i] = e < E ? R(1) / det[(long long)p * E + e] : R(0);
}
template <typename R>
__global__ void k_pack_faces(int nd, int NC, int EB, int E, int n, const int *__restrict__ lineOf,
                             const int *__restrict__ slotL, const int *__restrict__ slotR, const R *__restrict__ nrm,
                             const R *__restrict__ dAL, const R *__restrict__ dAR, int *__restrict__ nb,
                             R *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int NT = nd * NC * EB;
  const int sL = slotL[i], sR = slotR[i];
  // slot -> (block, side, thread); lineOf[f] = 2 * (line over all dimensions) + side
  const auto put = [&](int slot, int other, R sign, R area) {
    const int f = slot / E, e = slot - f * E;
    const long long g = (long long)(e / EB) * 2 + (lineOf[f] & 1);
    const int t = (lineOf[f] >> 1) * EB + e % EB;
    nb[g * NT + t] = other;
    for (int d = 0; d < nd; d++) out[(g * (nd + 1) + d) * NT + t] = sign * nrm[(long long)i * nd + d];
    out[(g * (nd + 1) + nd) * NT + t] = area;
  };
  put(sL, sR < 0 ? sR : (sR | kLeftBit), R(1), dAL[i]);
  if (sR >= 0) put(sR, sL, R(-1), dAR[i]);
}

#define FR_FZ_ORDERS(X) X(2, 0) X(2, 1) X(2, 2) X(2, 3) X(2, 4) X(2, 5) X(3, 0) X(3, 1) X(3, 2) X(3, 3) X(3, 4) X(3, 5)

template <int ND, int P, typename R, bool TMA, bool ROE>
void launch_one(const FusedArgsT<R> &a, const FusedMaps &m, cudaStream_t st) {
  using T = Fz<ND, P, R>;
  static std::atomic<unsigned long long> attrDev{0};
  smem_attr(k_fused_stage<ND, P, R, TMA, ROE>, (int)T::SMEM, attrDev);
  launch_k(k_fused_stage<ND, P, R, TMA, ROE>, (a.E + T::EB - 1) / T::EB, T::NT, T::SMEM, st, a, m);
}

}  // namespace

template <typename R>
int fused_elems_per_block(int nDims, int order) {
#define FR_FZ_EB(ND, P) \
  if (nDims == ND && order == P) return Fz<ND, P, R>::EB;
  FR_FZ_ORDERS(FR_FZ_EB)
#undef FR_FZ_EB
  return 0;
}
template int fused_elems_per_block<double>(int, int);
template int fused_elems_per_block<float>(int, int);

template <typename R>
void launch_fused_stage(int nDims, int order, bool tma, const FusedArgsT<R> &a, const FusedMaps &m, cudaStream_t st) {
  if (a.E <= 0) return;
#define FR_FZ_CASE(ND, P)                                              \
  if (nDims == ND && order == P) {                                     \
    if constexpr (ND == 3) {                                           \
      if (!tma) return launch_one<ND, P, R, false, false>(a, m, st);   \
    } else {                                                           \
      if (a.ph.riemannType == 1) return launch_one<ND, P, R, true, true>(a, m, st); \
    }                                                                  \
    return launch_one<ND, P, R, true, false>(a, m, st);                \
  }
  FR_FZ_ORDERS(FR_FZ_CASE)
#undef FR_FZ_CASE
}
template void launch_fused_stage<double>(int, int, bool, const FusedArgsT<double> &, const FusedMaps &, cudaStream_t);
template void launch_fused_stage<float>(int, int, bool, const FusedArgsT<float> &, const FusedMaps &, cudaStream_t);

template <typename R>
void launch_fused_pack(int nDims, int order, int E, const R *JG, const R *det, const FaceTableT<R> &ft,
                       const int *lineOf, R *jg, R *rdet, int *nb, R *nrm, cudaStream_t st) {
  const int N = order + 1, NC = nDims == 2 ? N : N * N, EB = fused_elems_per_block<R>(nDims, order);
  const long long total = (long long)((E + EB - 1) / EB) * N * NC * EB;
  k_pack_points<R><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(nDims, N * NC, EB, E, JG, det, jg, rdet, total);
  if (ft.n > 0)
    k_pack_faces<R><<<(ft.n + 255) / 256, 256, 0, st>>>(nDims, NC, EB, E, ft.n, lineOf, ft.slotL, ft.slotR, ft.nrm,
                                                        ft.dAL, ft.dAR, nb, nrm);
}
template void launch_fused_pack<double>(int, int, int, const double *, const double *, const FaceTableT<double> &,
                                        const int *, double *, double *, int *, double *, cudaStream_t);
template void launch_fused_pack<float>(int, int, int, const float *, const float *, const FaceTableT<float> &,
                                       const int *, float *, float *, int *, float *, cudaStream_t);

}  // namespace frk
