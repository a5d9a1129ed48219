// Device kernels of the periodic KIFMM evaluation pass for sm_100a.
//
// Stage map (reference function -> kernel here):
//   p2p_1toN_256          (3dpp/src/kernel.cpp:258-311)   k_p2p32 / k_p2p64
//   p2m_precompute        (kernel.cpp:332-371)            k_p2m_check + k_apply_f64_tc
//   m2m_precompute / img  (kernel.cpp:395-404, 434-442)   k_apply_f64_tc per level
//   m2l_fft_precompute_t  (kernel.cpp:1140-1397)          k_m2l_up, k_m2l_hadamard8,
//     hadamard_8x8 / 1x27 (kernel.cpp:1012-1138)          k_m2l_hadamard27, k_m2l_down
//   l2l_precompute / img  (kernel.cpp:1419-1435)          k_apply_f64_tc per level
//   l2p_precompute        (kernel.cpp:1458-1511)          k_apply_f64_tc + k_l2p_eval
// (k_apply_f64_small is the operator GEMM in small tiles.)
// The adjoint adds k_swap_charges, k_restore_charges, k_adj_combine; the
// device-buffer forward k_set_charges.
//   dipole_correction, scale_bodies, sort_bodies_by_idx
//                         (kernel.cpp:1580-1596, body.cpp:88-96,177-190)  k_dipole_*, k_post
//
// Row, cell, body and slot indices come from the plan's tables, which the
// set-up fills with values below the extents of the buffers it sizes by them;
// thread indices are checked against the counts.  No kernel waits on another
// block.
#include "rtfmm_kernels.cuh"
#include "rtfmm_rsqrt.cuh"

#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <type_traits>

#include <cub/cub.cuh>

namespace rtfmm_b200 {

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------
// two complex values in one vector load
template <typename T> struct Cplx2;
template <> struct Cplx2<float> { using type = float4; };
template <> struct Cplx2<double> { using type = double4; };

// Layout of the 8x8 source spectra Q (complex, [frequency][source][slot]).
// A frequency's rows are stored in 32-byte chunks (4 slots in FP32, 2 in
// FP64): chunk 0 of every source, then chunk 1, ..., so that the Hadamard's
// lanes, which take consecutive targets and so mostly consecutive sources,
// read a chunk of their rows from consecutive sectors, and an up-pass block
// (slot pairs of one source) still writes whole sectors.
template <typename T>
__host__ __device__ __forceinline__ size_t q8_index(size_t f, int src, int slot, int nsrc) {
  constexpr int per = 32 / (2 * sizeof(T)), nch = 8 / per;  // slots per chunk, chunks per row
  return ((f * nch + slot / per) * nsrc + src) * per + slot % per;
}

// 32-byte (one sector) vector loads, sm_100: one lane reads a whole sector.
__device__ __forceinline__ void ld_sector(const float* p, float (&v)[8]) {
  asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---------------------------------------------------------------------------
// body preparation
// ---------------------------------------------------------------------------
__global__ void k_gather_bodies(const double* __restrict__ x_in, const double* __restrict__ q_in,
                                const int64_t* __restrict__ perm, int n, double4* __restrict__ body64) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t k = perm[i];
  body64[i] = make_double4(x_in[3 * k], x_in[3 * k + 1], x_in[3 * k + 2], q_in[k]);
}

// FP32 leaf-relative positions: (x - c_leaf, q) so that P2P differences stay
// accurate in single precision.
__global__ void k_prep32(const double4* __restrict__ body64, const int* __restrict__ body_leaf,
                         const LeafInfo* __restrict__ leaves, float4* __restrict__ body32, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 b = body64[i];
  const LeafInfo L = leaves[body_leaf[i]];
  body32[i] = make_float4((float)(b.x - L.cx), (float)(b.y - L.cy), (float)(b.z - L.cz), (float)b.w);
}

// body_leaf[b] = the leaf holding tree-order body b (block per leaf)
__global__ void k_body_leaf(const LeafInfo* __restrict__ leaves, int nleaf, int n, int* __restrict__ body_leaf) {
  const int l = blockIdx.x;
  if (l >= nleaf) return;
  const LeafInfo L = leaves[l];
  for (int b = threadIdx.x; b < L.bnum; b += blockDim.x)
    if (L.boff + b >= 0 && L.boff + b < n) body_leaf[L.boff + b] = l;
}

// ---------------------------------------------------------------------------
// P2P: one warp per work item, up to 32 targets of one leaf against a part of
// the leaf's source list (entries e0..e1), staged 32 bodies at a time in a
// per-warp shared-memory slot; the next tile's bodies load while the current
// tile is computed.
//
// Long entries (p2p_long_entries, FP32): a tile is up to 32 bodies of one
// entry.  Short entries and FP64: the bodies of the entries are taken as one
// sequence, so that a tile is full whatever the sizes of the source leaves,
// and 32 entries load at once.
//
// Error of the FP32 form.  Each source leaf has its own frame: the target is
// moved into it (x_t - offset, one rounding that all sources of the leaf
// share, so that it cancels where their charges do; the offset added to each
// source instead gave the potential of a lattice up to 1.4 times the error).
// FP32 sums run over at most 64 bodies of one long entry, or over 8 pairs of
// short ones (the potential over 4) divided by the number of lane groups, and
// their two halves go into FP64 each by itself.  Over 27 sets (uniform, blobs,
// lattices; mean entries of 4-256 bodies) the error against FP64 is at most
// 1.01 times that of sums over one entry each, 0.4-0.8 times for entries of
// 128 bodies and more; sums over 16 pairs across entries gave up to 1.9 times
// for the potential and 1.2 times for the gradient.  Long entries summed
// whole: 3.51 ms instead of 3.65 on leaves of 256 bodies (2^20); over 32
// bodies 3.69.
//
// A clustered tree has leaves whose lists hold forty times the mean number of
// bodies (a large leaf beside many small ones): such a list is cut into parts
// (p2p_part_bodies), each part leaves its sums in a slot of its own, and the
// last part to finish adds the slots up in order, so that the result does not
// depend on which one that is.  A plan without cut lists runs an instance
// without that code, whose two registers fewer are 0.9% (3.57 against 3.60 ms,
// 2^20 bodies in leaves of 256).
//
// Measured, with one entry a tile and uncut lists -> here: 150001 bodies in
// blobs (longest list 60593 bodies, mean 1435), FP64, 3.98 -> 0.47 ms; 30011 in
// blobs, FP32, 0.36 -> 0.052; 10^6 in blobs, FP32, 11.4 -> 2.45; uniform 2^20,
// FP32, ncrit = 32 1.36 -> 0.87, 64 0.68 and 0.70, 256 3.13 and 3.17, 512 3.58
// and 3.65 (the whole pass 5.00 -> 4.96, P = 8); FP64, ncrit = 256, 9.28 -> 7.68
// (24 -> 18 FP64 operations a pair).
// FP32: bound by the register reads of the packed FMAs (3 cycles each measured,
// 31 a pair of sources with the 2-cycle additions and products).  FP64: bound
// by dependent operations (pipe 71% busy); 28 resident warps 7.68 ms, 20 7.94,
// 24 8.04, 32 7.76.
// ---------------------------------------------------------------------------
// A block is one warp: work items differ in cost several-fold, and a block of
// four held the slots of its finished warps until its slowest one was done
// (FP32 3.33 against 3.12 ms at N = 2^20, P = 8).
constexpr int kP2PWarps = 1;
constexpr int kP2PUnroll = 4, kP2PUnroll64 = 4;  // pairs (FP32), sources (FP64)
constexpr int kP2PRun = 8, kP2PRunPhi = 4;       // pairs of short entries summed in FP32
constexpr int kP2PMinBlocks = 20, kP2PMinBlocksShort = 24, kP2PMinBlocks64 = 28;  // resident blocks per SM

// A chunk of up to 32 list entries, one per lane: `start` is the lane's
// entry's first body in the chunk's sequence, `src` + position the body in
// tree order.
struct P2PChunk {
  int start, src, total, nent;
};
__device__ __forceinline__ P2PChunk p2p_chunk(int boff, int bnum, int nent, int lane) {
  P2PChunk c;
  int s = bnum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += v;
  }
  c.start = s - bnum;
  c.src = boff - c.start;
  c.total = __shfl_sync(0xffffffffu, s, 31);
  c.nent = nent;
  return c;
}
// The entry (lane number) that holds the sequence's body base + lane: leaves
// hold at least one body, so the starts are distinct and their bits count the
// entries begun.
__device__ __forceinline__ int p2p_entry(const P2PChunk& c, int base, int lane) {
  const int rel = c.start - base;
  const bool valid = lane < c.nent;
  const unsigned before = __ballot_sync(0xffffffffu, valid && rel < 0);
  const unsigned bit = valid && rel >= 0 && rel < 32 ? 1u << rel : 0u;
  const unsigned begun = __reduce_or_sync(0xffffffffu, bit);
  return __popc(before) + __popc(begun & (0xffffffffu >> (31 - lane))) - 1;
}

// The sums of a work item: written, or left in the item's slot when its list
// is cut into parts (only where CUT).
template <bool CUT>
__device__ __forceinline__ void p2p_store(const P2PItem& it, bool writer, int ti, double P, double Gx, double Gy,
                                          double Gz, double4* __restrict__ part, int* __restrict__ done,
                                          double* __restrict__ phi, double* __restrict__ grad) {
  if (CUT && it.nparts > 1) {
    if (writer) part[(size_t)(it.slot + it.part) * 32 + ti] = make_double4(P, Gx, Gy, Gz);
    __threadfence();
    __syncwarp();
    int last = 0;
    if ((threadIdx.x & 31) == 0) last = atomicInc((unsigned*)done + it.slot, it.nparts - 1) == it.nparts - 1;
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    __threadfence();
    if (writer) {
      P = Gx = Gy = Gz = 0.0;
      for (int k = 0; k < it.nparts; ++k) {
        const double2* v = reinterpret_cast<const double2*>(part + (size_t)(it.slot + k) * 32 + ti);
        const double2 a = __ldcg(v), b = __ldcg(v + 1);
        P += a.x;
        Gx += a.y;
        Gy += b.x;
        Gz += b.y;
      }
    }
  }
  if (writer) {
    const int b = it.boff + ti;
    phi[b] = P;
    grad[3 * b + 0] = -Gx;
    grad[3 * b + 1] = -Gy;
    grad[3 * b + 2] = -Gz;
  }
}

// One source pair k of a tile against this lane's target, in packed FP32x2
// arithmetic (sm_100 FADD2/FMUL2/FFMA2): the tile is held as 16 pairs, pair k
// at s[2k] = (-x, -x', -y, -y') and s[2k+1] = (-z, -z', q, q'); the sums run
// in two interleaved halves.  All 16 pairs of a tile are written (padding
// carries no charge and sits far away).
template <bool MASK>
__device__ __forceinline__ void p2p32_pair2(const float4* __restrict__ s, int k, float2 px, float2 py, float2 pz,
                                            float2& p, float2& fx, float2& fy, float2& fz) {
  const float4 u = s[2 * k], v = s[2 * k + 1];
  const float2 dx = __fadd2_rn(px, make_float2(u.x, u.y));
  const float2 dy = __fadd2_rn(py, make_float2(u.z, u.w));
  const float2 dz = __fadd2_rn(pz, make_float2(v.x, v.y));
  float2 r2 = __fmul2_rn(dz, dz);
  r2 = __ffma2_rn(dy, dy, r2);
  r2 = __ffma2_rn(dx, dx, r2);
  float2 ir = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
  if (MASK) {
    ir.x = r2.x > 0.f ? ir.x : 0.f;
    ir.y = r2.y > 0.f ? ir.y : 0.f;
  }
  const float2 qir = __fmul2_rn(make_float2(v.z, v.w), ir);
  p = __fadd2_rn(p, qir);
  const float2 q3 = __fmul2_rn(__fmul2_rn(qir, ir), ir);
  fx = __ffma2_rn(q3, dx, fx);
  fy = __ffma2_rn(q3, dy, fy);
  fz = __ffma2_rn(q3, dz, fz);
}

// The two interleaved halves of an FP32 sum into FP64, each by itself.
__device__ __forceinline__ void widen(double& d, float2 v) { d += (double)v.x + (double)v.y; }

// Lanes of group k0 (of G groups) take the tile's source pairs k0, k0+G, ...,
// all of one entry.
template <int G, bool MASK>
__device__ __forceinline__ void p2p32_run(const float4* __restrict__ s, int k0, int npair, float2 px, float2 py,
                                          float2 pz, float2& p, float2& fx, float2& fy, float2& fz) {
#pragma unroll kP2PUnroll
  for (int k = k0; k < npair; k += G) p2p32_pair2<MASK>(s, k, px, py, pz, p, fx, fy, fz);
}
// The same for a full tile of one entry that is not the target leaf: a constant
// bound (3.65 against 3.71 ms on leaves of 256 bodies).
template <int G>
__device__ __forceinline__ void p2p32_full(const float4* __restrict__ s, int k0, float2 px, float2 py, float2 pz,
                                           float2& p, float2& fx, float2& fy, float2& fz) {
#pragma unroll kP2PUnroll
  for (int u = 0; u < 16 / G; ++u) p2p32_pair2<false>(s, k0 + u * G, px, py, pz, p, fx, fy, fz);
}
// The same for a whole tile across entries, pair k of the entry with the
// offset so[k]; FP32 sums over R pairs (the potential over RP), a lane group
// over as many fewer as there are groups.
template <int G, bool MASK>
__device__ __forceinline__ void p2p32_pairs(const float4* __restrict__ s, const float4* __restrict__ so, int k0,
                                            float4 xt, double& P, double& Gx, double& Gy, double& Gz) {
  constexpr int N = 16 / G, R = kP2PRun >= G ? kP2PRun / G : 1, RP = kP2PRunPhi >= G ? kP2PRunPhi / G : 1;
#pragma unroll 1
  for (int u = 0; u < N; u += R) {
    float2 p = make_float2(0.f, 0.f), fx = p, fy = p, fz = p;
#pragma unroll
    for (int v = 0; v < R; ++v) {
      const int k = k0 + (u + v) * G;
      const float4 o = so[k];
      const float px = xt.x - o.x, py = xt.y - o.y, pz = xt.z - o.z;
      p2p32_pair2<MASK>(s, k, make_float2(px, px), make_float2(py, py), make_float2(pz, pz), p, fx, fy, fz);
      if (v % RP == RP - 1) {
        widen(P, p);
        p = make_float2(0.f, 0.f);
      }
    }
    widen(Gx, fx);
    widen(Gy, fy);
    widen(Gz, fz);
  }
}

// One work item: W = 32/G lanes per target group, G groups per warp.
template <bool LONG, bool CUT, int G>
__device__ __forceinline__ void p2p32_item(const float4* __restrict__ body32, const P2PItem& it,
                                           const P2PSrc32* __restrict__ list, float4* __restrict__ sw, int lane,
                                           double4* __restrict__ part, int* __restrict__ done,
                                           double* __restrict__ phi, double* __restrict__ grad) {
  constexpr int W = 32 / G;
  const int grp = lane / W, ti = lane % W;
  const bool active = ti < it.nt;
  // tile padding: no charge, far from every target (finite 1/r)
  const float4 pad = make_float4(1e18f, 1e18f, 1e18f, 0.f);
  const float4 xt = active ? body32[it.boff + ti] : make_float4(0.f, 0.f, 0.f, 0.f);
  double P = 0.0, Gx = 0.0, Gy = 0.0, Gz = 0.0;
  float* sf = reinterpret_cast<float*>(sw) + 8 * (lane >> 1) + (lane & 1);
  if constexpr (LONG) {
    int e = it.e0;
    const int e1 = it.e1;
    P2PSrc32 cur{}, nxt{};
    float4 b = pad;
    if (e < e1) {
      cur = list[e];
      if (lane < cur.bnum) b = body32[cur.boff + lane];
    }
    if (e + 1 < e1) nxt = list[e + 1];
    int c0 = 0;
    float2 p = make_float2(0.f, 0.f), fx = p, fy = p, fz = p;
    while (e < e1) {
      const int cnt = min(32, cur.bnum - c0);
      __syncwarp();
      sf[0] = -b.x;
      sf[2] = -b.y;
      sf[4] = -b.z;
      sf[6] = b.w;
      __syncwarp();
      // next tile: the rest of this entry, else the first of the next one
      const bool last = c0 + 32 >= cur.bnum;
      b = pad;
      if (!last) {
        if (lane < cur.bnum - c0 - 32) b = body32[cur.boff + c0 + 32 + lane];
      } else if (e + 1 < e1) {
        if (lane < nxt.bnum) b = body32[nxt.boff + lane];
      }
      const float px = xt.x - cur.dx, py = xt.y - cur.dy, pz = xt.z - cur.dz;
      const int npair = (cnt + 1) >> 1;
      if (cur.self)
        p2p32_run<G, true>(sw, grp, npair, make_float2(px, px), make_float2(py, py), make_float2(pz, pz), p, fx, fy,
                           fz);
      else if (cnt == 32)
        p2p32_full<G>(sw, grp, make_float2(px, px), make_float2(py, py), make_float2(pz, pz), p, fx, fy, fz);
      else
        p2p32_run<G, false>(sw, grp, npair, make_float2(px, px), make_float2(py, py), make_float2(pz, pz), p, fx, fy,
                            fz);
      if (last || (c0 & 32)) {  // every 64 bodies, and at the entry's end
        P += (double)p.x + (double)p.y;
        Gx += (double)fx.x + (double)fx.y;
        Gy += (double)fy.x + (double)fy.y;
        Gz += (double)fz.x + (double)fz.y;
        p = fx = fy = fz = make_float2(0.f, 0.f);
      }
      if (last) {
        ++e;
        c0 = 0;
        cur = nxt;
        if (e + 1 < e1) nxt = list[e + 1];
      } else {
        c0 += 32;
      }
    }
  } else {
    float4* so = sw + 32;  // offsets of the tile's pairs
    auto entry = [&](int e) { return e < it.e1 ? list[e] : P2PSrc32{}; };
    P2PSrc32 cur{}, nxt{};  // this lane's entry of the chunk and of the next one
    P2PChunk c{};
    int self0 = 0, self1 = 0;  // the target leaf's own bodies in the chunk's sequence
    auto chunk = [&](int e0) {
      // entries of an odd number of bodies take a padding slot: no pair of two
      c = p2p_chunk(cur.boff, (cur.bnum + 1) & ~1, min(32, it.e1 - e0), lane);
      const unsigned own = __ballot_sync(0xffffffffu, cur.self);
      const int o = own ? __ffs(own) - 1 : 0;
      self0 = own ? __shfl_sync(0xffffffffu, c.start, o) : 0;
      self1 = own ? self0 + __shfl_sync(0xffffffffu, cur.bnum, o) : 0;
    };
    float4 b = pad, o = pad;  // the next tile's body of this lane and its entry's offset
    auto stage = [&](int base) {
      const int s = p2p_entry(c, base, lane), pos = base + lane;
      const int i = __shfl_sync(0xffffffffu, c.src, s) + pos;
      const int end = __shfl_sync(0xffffffffu, c.start + cur.bnum, s);
      o.x = __shfl_sync(0xffffffffu, cur.dx, s);
      o.y = __shfl_sync(0xffffffffu, cur.dy, s);
      o.z = __shfl_sync(0xffffffffu, cur.dz, s);
      b = pos < end ? body32[i] : pad;
    };
    int e = it.e0, base = 0;
    bool more = e < it.e1;
    if (more) {
      cur = entry(e + lane);
      nxt = entry(e + 32 + lane);
      chunk(e);
      stage(0);
    }
    while (more) {
      const bool mask = self0 < base + 32 && self1 > base;
      __syncwarp();
      sf[0] = -b.x;
      sf[2] = -b.y;
      sf[4] = -b.z;
      sf[6] = b.w;
      if (!(lane & 1)) so[lane >> 1] = o;
      __syncwarp();
      base += 32;
      if (base >= c.total) {
        e += 32;
        base = 0;
        more = e < it.e1;
        if (more) {
          cur = nxt;
          nxt = entry(e + 32 + lane);
          chunk(e);
        }
      }
      if (more) stage(base);
      if (mask)
        p2p32_pairs<G, true>(sw, so, grp, xt, P, Gx, Gy, Gz);
      else
        p2p32_pairs<G, false>(sw, so, grp, xt, P, Gx, Gy, Gz);
    }
  }
  // sum the source groups (lanes ti, ti + W, ...)
#pragma unroll
  for (int o = W; o < 32; o <<= 1) {
    P += __shfl_xor_sync(0xffffffffu, P, o);
    Gx += __shfl_xor_sync(0xffffffffu, Gx, o);
    Gy += __shfl_xor_sync(0xffffffffu, Gy, o);
    Gz += __shfl_xor_sync(0xffffffffu, Gz, o);
  }
  p2p_store<CUT>(it, active && grp == 0, ti, P, Gx, Gy, Gz, part, done, phi, grad);
}

template <bool LONG, bool CUT>
__global__ void __launch_bounds__(32 * kP2PWarps, LONG ? kP2PMinBlocks : kP2PMinBlocksShort)
    k_p2p32(const float4* __restrict__ body32, const P2PItem* __restrict__ items, int nitems,
            const P2PSrc32* __restrict__ list, double4* __restrict__ part, int* __restrict__ done,
            double* __restrict__ phi, double* __restrict__ grad) {
  __shared__ float4 sbuf[kP2PWarps][LONG ? 32 : 48];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = blockIdx.x * kP2PWarps + warp;
  if (item >= nitems) return;  // warp-uniform
  const P2PItem it = items[item];
  switch (it.lw) {
    case 5: p2p32_item<LONG, CUT, 1>(body32, it, list, sbuf[warp], lane, part, done, phi, grad); break;
    case 4: p2p32_item<LONG, CUT, 2>(body32, it, list, sbuf[warp], lane, part, done, phi, grad); break;
    case 3: p2p32_item<LONG, CUT, 4>(body32, it, list, sbuf[warp], lane, part, done, phi, grad); break;
    default: p2p32_item<LONG, CUT, 8>(body32, it, list, sbuf[warp], lane, part, done, phi, grad); break;
  }
}

// FP64 P2P, the same work items; per pair the reference's arithmetic
// (dx = x_t - (x_s + offset), kernel.cpp:283-290) in FP64, 18 operations.
template <int G>
__device__ __forceinline__ void p2p64_item(const double4* __restrict__ body64, const P2PItem& it,
                                           const P2PSrc64* __restrict__ list, double4* __restrict__ sw, int lane,
                                           double4* __restrict__ part, int* __restrict__ done,
                                           double* __restrict__ phi, double* __restrict__ grad) {
  constexpr int W = 32 / G;
  const int grp = lane / W, ti = lane % W;
  const bool active = ti < it.nt;
  const double4 zero = make_double4(0.0, 0.0, 0.0, 0.0);
  const double4 xt = active ? body64[it.boff + ti] : zero;
  double P = 0.0, Gx = 0.0, Gy = 0.0, Gz = 0.0;
  auto entry = [&](int e) { return e < it.e1 ? list[e] : P2PSrc64{}; };
  P2PSrc64 cur{}, nxt{};
  P2PChunk c{};
  double4 b = zero;
  double ox = 0.0, oy = 0.0, oz = 0.0;
  auto stage = [&](int base) {
    const int s = p2p_entry(c, base, lane), pos = base + lane;
    const int i = __shfl_sync(0xffffffffu, c.src, s) + pos;
    ox = __shfl_sync(0xffffffffu, cur.ox, s);
    oy = __shfl_sync(0xffffffffu, cur.oy, s);
    oz = __shfl_sync(0xffffffffu, cur.oz, s);
    b = pos < c.total ? body64[i] : zero;
  };
  int e = it.e0, base = 0;
  bool more = e < it.e1;
  if (more) {
    cur = entry(e + lane);
    nxt = entry(e + 32 + lane);
    c = p2p_chunk(cur.boff, cur.bnum, min(32, it.e1 - e), lane);
    stage(0);
  }
  while (more) {
    const int cnt = min(32, c.total - base);
    __syncwarp();
    sw[lane] = make_double4(b.x + ox, b.y + oy, b.z + oz, b.w);
    __syncwarp();
    base += 32;
    if (base >= c.total) {
      e += 32;
      base = 0;
      more = e < it.e1;
      if (more) {
        cur = nxt;
        nxt = entry(e + 32 + lane);
        c = p2p_chunk(cur.boff, cur.bnum, min(32, it.e1 - e), lane);
      }
    }
    if (more) stage(base);
#pragma unroll kP2PUnroll64
    for (int k = grp; k < cnt; k += G) {
      const double4 s = sw[k];
      const double dx = xt.x - s.x, dy = xt.y - s.y, dz = xt.z - s.z;
      const double ir = rsqrt_or_zero(dx * dx + dy * dy + dz * dz);
      const double qir = s.w * ir;
      P += qir;
      const double q3 = qir * ir * ir;
      Gx += q3 * dx;
      Gy += q3 * dy;
      Gz += q3 * dz;
    }
  }
#pragma unroll
  for (int o = W; o < 32; o <<= 1) {
    P += __shfl_xor_sync(0xffffffffu, P, o);
    Gx += __shfl_xor_sync(0xffffffffu, Gx, o);
    Gy += __shfl_xor_sync(0xffffffffu, Gy, o);
    Gz += __shfl_xor_sync(0xffffffffu, Gz, o);
  }
  p2p_store<true>(it, active && grp == 0, ti, P, Gx, Gy, Gz, part, done, phi, grad);
}

__global__ void __launch_bounds__(32 * kP2PWarps, kP2PMinBlocks64)
    k_p2p64(const double4* __restrict__ body64, const P2PItem* __restrict__ items, int nitems,
            const P2PSrc64* __restrict__ list, double4* __restrict__ part, int* __restrict__ done,
            double* __restrict__ phi, double* __restrict__ grad) {
  __shared__ double4 sbuf[kP2PWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = blockIdx.x * kP2PWarps + warp;
  if (item >= nitems) return;  // warp-uniform
  const P2PItem it = items[item];
  switch (it.lw) {
    case 5: p2p64_item<1>(body64, it, list, sbuf[warp], lane, part, done, phi, grad); break;
    case 4: p2p64_item<2>(body64, it, list, sbuf[warp], lane, part, done, phi, grad); break;
    case 3: p2p64_item<4>(body64, it, list, sbuf[warp], lane, part, done, phi, grad); break;
    default: p2p64_item<8>(body64, it, list, sbuf[warp], lane, part, done, phi, grad); break;
  }
}

// ---------------------------------------------------------------------------
// Close-pair refinement of the FP32 P2P (mixed form).
//
// The FP32 positions are leaf-relative, so each coordinate carries an
// absolute rounding of about 2^-24 of the leaf size, and a pair at distance
// d gets a relative error of about (leaf size / d) 2^-24 in its terms.  The
// relative L2 error of the whole gradient is dominated by the few closest
// pairs of the input (at N = 2^20 uniform bodies they sit ~1e-4 apart, a
// leaf is ~0.05 wide).  So the pairs closer than kCloseFrac times the larger
// of their two leaves' half edges are listed once per set-up (k_close_scan,
// a count pass and an emit pass in list order), and every pass replaces
// their FP32 terms by FP64 ones (k_close_fix): it recomputes the FP32 term
// of each listed pair with the P2P kernel's exact operation sequence (same
// FP32 inputs, same roundings, same rsqrt.approx) and adds the FP64 term
// minus it.  What remains of the FP32 term is its rounding inside the FP32
// partial sum, ~2^-24 of the term.
// ---------------------------------------------------------------------------
constexpr float kCloseFrac = 0.125f;

// One warp per P2P work item, one lane per target (lanes >= nt idle); the
// lanes of an item share its list, so source loads are warp broadcasts.
// EMIT = false: cnt[t] = close sources of target t.  EMIT = true: the pairs
// (source body, list entry) of target t at pairs[off[t] ...], in list order.
template <bool EMIT>
__global__ void __launch_bounds__(256)
    k_close_scan(const float4* __restrict__ body32, const P2PItem* __restrict__ items, int nitems,
                 const int* __restrict__ list_off, const P2PSrc32* __restrict__ list,
                 const LeafInfo* __restrict__ leaves, int* __restrict__ cnt, const int* __restrict__ off,
                 int2* __restrict__ pairs) {
  const int item = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (item >= nitems) return;
  const P2PItem it = items[item];
  if (it.part > 0 || lane >= it.nt) return;  // a cut list's first item scans all of it
  const int t = it.boff + lane;
  const float4 xt = body32[t];
  const float rt = (float)leaves[it.leaf].r;
  int c = 0;
  int pos = EMIT ? off[t] : 0;
  const int pend = EMIT ? off[t + 1] : 0;  // the count pass's total for t bounds the writes
  const int e1 = list_off[it.leaf + 1];
  const unsigned mask = __activemask();
  for (int e = list_off[it.leaf]; e < e1; ++e) {
    const P2PSrc32 s = list[e];
    const float rs = (float)leaves[s.leaf].r;
    const float rc = kCloseFrac * fmaxf(rt, rs);
    const float rc2 = rc * rc;
    const float px = xt.x - s.dx, py = xt.y - s.dy, pz = xt.z - s.dz;
    // the source leaf's box (half edge rs, a little margin for the FP32
    // rounding of the positions) is farther than rc from every target of
    // this warp: no close pair in it
    const float bx = fmaxf(fabsf(px) - 1.001f * rs, 0.f), by = fmaxf(fabsf(py) - 1.001f * rs, 0.f),
                bz = fmaxf(fabsf(pz) - 1.001f * rs, 0.f);
    if (!__any_sync(mask, bx * bx + by * by + bz * bz < rc2)) continue;
    for (int k = 0; k < s.bnum; ++k) {
      const float4 b = body32[s.boff + k];
      const float dx = px - b.x, dy = py - b.y, dz = pz - b.z;
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      if (r2 < rc2 && !(s.self && s.boff + k == t)) {
        if (EMIT) {
          if (pos < pend) pairs[pos++] = make_int2(s.boff + k, e);
        } else
          ++c;
      }
    }
  }
  if (!EMIT) cnt[t] = c;
}

// One thread per target body (tree order).  cycle > 0: periodic, the pair's
// FP64 difference taken at its nearest image (a close pair is far closer
// than half a period, so that is the image its list entry carries).
__global__ void k_close_fix(const double4* __restrict__ body64, const float4* __restrict__ body32,
                            const P2PSrc32* __restrict__ list, const int* __restrict__ off,
                            const int2* __restrict__ pairs, int n, double cycle, double* __restrict__ phi,
                            double* __restrict__ grad) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int b0 = off[t], b1 = off[t + 1];
  if (b0 == b1) return;
  const float4 xt = body32[t];
  const double4 yt = body64[t];
  double P = 0.0, Gx = 0.0, Gy = 0.0, Gz = 0.0;
  for (int k = b0; k < b1; ++k) {
    const int2 pr = pairs[k];
    const P2PSrc32 s = list[pr.y];
    // the FP32 terms exactly as k_p2p32 formed them
    const float4 b = body32[pr.x];
    const float px = xt.x - s.dx, py = xt.y - s.dy, pz = xt.z - s.dz;
    const float dx = __fadd_rn(px, -b.x), dy = __fadd_rn(py, -b.y), dz = __fadd_rn(pz, -b.z);
    float r2 = __fmul_rn(dz, dz);
    r2 = __fmaf_rn(dy, dy, r2);
    r2 = __fmaf_rn(dx, dx, r2);
    float ir = rsqrt_approx(r2);
    if (!(r2 > 0.f)) ir = 0.f;
    const float qir = __fmul_rn(b.w, ir);
    const float q3 = __fmul_rn(__fmul_rn(qir, ir), ir);
    // the FP64 terms of the pair
    const double4 y = body64[pr.x];
    double ex = yt.x - y.x, ey = yt.y - y.y, ez = yt.z - y.z;
    if (cycle > 0.0) {
      ex -= cycle * rint(ex / cycle);
      ey -= cycle * rint(ey / cycle);
      ez -= cycle * rint(ez / cycle);
    }
    const double rr = ex * ex + ey * ey + ez * ez;
    const double jr = rsqrt_or_zero(rr);
    const double qjr = y.w * jr;
    const double q3d = qjr * jr * jr;
    P += qjr - (double)qir;
    Gx += q3d * ex - (double)q3 * (double)dx;
    Gy += q3d * ey - (double)q3 * (double)dy;
    Gz += q3d * ez - (double)q3 * (double)dz;
  }
  phi[t] += P;
  grad[3 * t + 0] -= Gx;
  grad[3 * t + 1] -= Gy;
  grad[3 * t + 2] -= Gz;
}

// ---------------------------------------------------------------------------
// P2M: check-surface potential of each leaf's bodies (FP64).  Surface points
// are unit * (2.95 r) + centre (kernel.cpp:336).  One block per leaf, two
// surface points per thread, the block sized to the surface (160 threads for
// the 296 points of P = 8) so that few lanes idle.
// ---------------------------------------------------------------------------
constexpr int kSurfThreads = 128;
constexpr int kCheckMaxThreads = 256;
constexpr int kCheckPer = 2;

template <bool FULL>
__global__ void __launch_bounds__(kCheckMaxThreads)
    k_p2m_check(const double4* __restrict__ body64, const LeafInfo* __restrict__ leaves,
                const double* __restrict__ surf_unit, int ns, double* __restrict__ out) {
  __shared__ double4 sb[kCheckMaxThreads];
  const LeafInfo L = leaves[blockIdx.x];
  const double R = L.r * 2.95;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i0 = 0; i0 < ns; i0 += nt * kCheckPer) {
    double yx[kCheckPer], yy[kCheckPer], yz[kCheckPer], acc[kCheckPer];
#pragma unroll
    for (int k = 0; k < kCheckPer; ++k) {
      const int i = i0 + tid + k * nt;
      const int ii = i < ns ? i : 0;
      yx[k] = surf_unit[3 * ii + 0] * R + L.cx;
      yy[k] = surf_unit[3 * ii + 1] * R + L.cy;
      yz[k] = surf_unit[3 * ii + 2] * R + L.cz;
      acc[k] = 0.0;
    }
    for (int b0 = 0; b0 < L.bnum; b0 += nt) {
      const int cnt = min(nt, L.bnum - b0);
      __syncthreads();
      if (tid < cnt) {
        double4 b = body64[L.boff + b0 + tid];
        if (!FULL) b.w *= 0.5;
        sb[tid] = b;
      }
      __syncthreads();
#pragma unroll 2
      for (int j = 0; j < cnt; ++j) {
        const double4 b = sb[j];
#pragma unroll
        for (int k = 0; k < kCheckPer; ++k) {
          const double dx = yx[k] - b.x, dy = yy[k] - b.y, dz = yz[k] - b.z;
          acc[k] += b.w * rsqrt_surf<FULL>(dx * dx + dy * dy + dz * dz);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kCheckPer; ++k) {
      const int i = i0 + tid + k * nt;
      if (i < ns) out[(size_t)blockIdx.x * ns + i] = acc[k];
    }
  }
}

// ---------------------------------------------------------------------------
// L2P: potential and gradient at each leaf's bodies from the downward
// equivalent density on the 2.95 r surface (kernel.cpp:1461, 1469-1510), FP64.
// One block per leaf.  A leaf with fewer bodies than threads splits the
// surface points among G = threads / bnum groups of bnum threads (group g
// takes points g, g+G, ...) and sums the groups in shared memory, so that a
// 34-body leaf keeps 102 of 128 threads busy instead of 34.
// ---------------------------------------------------------------------------
template <bool FULL>
__global__ void __launch_bounds__(kSurfThreads)
    k_l2p_eval(const double4* __restrict__ body64, const LeafInfo* __restrict__ leaves,
               const double* __restrict__ surf_unit, int ns, const double* __restrict__ q_down,
               double* __restrict__ phi, double* __restrict__ grad) {
  extern __shared__ double4 sy[];  // ns entries
  __shared__ double red[4][kSurfThreads];
  const LeafInfo L = leaves[blockIdx.x];
  const double R = L.r * 2.95;
  for (int i = threadIdx.x; i < ns; i += blockDim.x)
    sy[i] = make_double4(surf_unit[3 * i] * R + L.cx, surf_unit[3 * i + 1] * R + L.cy,
                         surf_unit[3 * i + 2] * R + L.cz, (FULL ? 1.0 : 0.5) * q_down[(size_t)blockIdx.x * ns + i]);
  __syncthreads();
  const int bnum = L.bnum;
  if (bnum <= 0) return;  // block-uniform
  const int B = bnum < kSurfThreads ? bnum : kSurfThreads;
  const int G = kSurfThreads / B;
  const int grp = threadIdx.x / B, tl = threadIdx.x - grp * B;
  for (int t0 = 0; t0 < bnum; t0 += B) {
    double p = 0, gx = 0, gy = 0, gz = 0;
    const int t = t0 + tl;
    if (grp < G && t < bnum) {
      const double4 x = body64[L.boff + t];
      for (int i = grp; i < ns; i += G) {
        const double4 y = sy[i];
        const double dx = x.x - y.x, dy = x.y - y.y, dz = x.z - y.z;
        const double ir = rsqrt_surf<FULL>(dx * dx + dy * dy + dz * dz);
        const double qir = y.w * ir;
        p += qir;
        const double q3 = qir * ir * ir;
        gx += q3 * dx;
        gy += q3 * dy;
        gz += q3 * dz;
      }
    }
    if (G > 1) {
      red[0][threadIdx.x] = p;
      red[1][threadIdx.x] = gx;
      red[2][threadIdx.x] = gy;
      red[3][threadIdx.x] = gz;
      __syncthreads();
      if (grp == 0) {
        for (int g2 = 1; g2 < G; ++g2) {
          const int o = g2 * B + tl;
          p += red[0][o];
          gx += red[1][o];
          gy += red[2][o];
          gz += red[3][o];
        }
      }
      __syncthreads();
    }
    if (grp == 0 && t < bnum) {
      const int b = L.boff + t;
      const double sg = FULL ? -1.0 : -0.25;  // (2/r)^3 against halved charges
      phi[b] = p;
      grad[3 * b + 0] = sg * gx;
      grad[3 * b + 1] = sg * gy;
      grad[3 * b + 2] = sg * gz;
    }
  }
}

// ---------------------------------------------------------------------------
// Batched FP64 operator application:
//   C[outrow[r]][n] = beta*C + scale[r] * sum_j A[inrow[r]][j] B[g][j][n]
// on the FP64 tensor path: 64x64 output tiles per 128-thread block (2 x 2 warps of 32x32, each 4 x 4 mma.sync m8n8k4
// f64 tiles), A rows (gathered through inrow) and the B panel moved into
// shared memory by cp.async through a three-stage ring, so that the loads of
// K step t+2 are in flight while step t is multiplied.  Products and sums
// are IEEE FP64 as in the SIMT kernel; only the summation order differs.
// Every 16-byte copy is in bounds or zero-filled (ns is even: 6(P-1)^2+2).
// ---------------------------------------------------------------------------
constexpr int kGM = 64, kGN = 64, kGK = 16, kGStages = 3, kGThreads = 128;
constexpr int kAPitch = kGK + 4;  // doubles per A row in shared memory (conflict-free fragments)
constexpr int kBPitch = kGN + 4;  // doubles per B row
constexpr int kAStage = kGM * kAPitch, kBStage = kGK * kBPitch;
[[maybe_unused]] constexpr size_t kGSmem = sizeof(double) * kGStages * (kAStage + kBStage);

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int nbytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa), "l"(gmem), "r"(nbytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma8x8x4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(kGThreads) k_apply_f64_tc(ApplyBatch b) {
  extern __shared__ __align__(16) double gsm[];
  double* As = gsm;
  double* Bs = gsm + kGStages * kAStage;
  const int g = blockIdx.z;
  const int rbeg = b.group_off[g], rend = b.group_off[g + 1];
  const int r0 = rbeg + blockIdx.y * kGM;
  const int c0 = blockIdx.x * kGN;
  if (r0 >= rend) return;  // block-uniform
  const int ns = b.ns;
  const double* Bg = b.B + (size_t)g * ns * ns;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 1, wn = warp >> 1;
  const int total = (ns + kGK - 1) / kGK;
  // copies of this thread: A chunk e = tid + 128u -> row e/8, doubles 2(e%8)..+1;
  // B chunk e -> K row e/32, columns 2(e%32)..+1
  int srow[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int row = r0 + ((tid + kGThreads * u) >> 3);
    srow[u] = row < rend ? b.inrow[row] : -1;
  }
  auto issue = [&](int kt) {
    const int j0 = kt * kGK;
    double* as = As + (kt % kGStages) * kAStage;
    double* bs = Bs + (kt % kGStages) * kBStage;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = tid + kGThreads * u;
      const int r = e >> 3, ch = e & 7, j = j0 + 2 * ch;
      const bool ok = srow[u] >= 0 && j < ns;
      cp_async16(as + r * kAPitch + 2 * ch, ok ? b.A + (size_t)srow[u] * ns + j : b.A, ok);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = tid + kGThreads * u;
      const int kr = e >> 5, ch = e & 31, jj = j0 + kr, n = c0 + 2 * ch;
      const bool ok = jj < ns && n < ns;
      cp_async16(bs + kr * kBPitch + 2 * ch, ok ? Bg + (size_t)jj * ns + n : Bg, ok);
    }
  };
  double acc[4][4][2];
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = 0.0;
  // the warp's column tiles are every other 8 of the block's 64, so that a
  // block at the end of ns (24 of 64 columns at ns = 152, 40 at 296) splits
  // its tiles over both column warps; the ones past ns are not multiplied
  const int nv = min(4, max(0, (ns - c0 - 8 * wn + 15) / 16));
#pragma unroll
  for (int st = 0; st < kGStages - 1; ++st) {
    if (st < total) issue(st);
    cp_async_commit();
  }
  auto step = [&](int kt, auto nvc) {
    constexpr int NV = decltype(nvc)::value;
    const double* as = As + (kt % kGStages) * kAStage + (wm * 32 + (lane >> 2)) * kAPitch + (lane & 3);
    const double* bs = Bs + (kt % kGStages) * kBStage + (lane & 3) * kBPitch + wn * 8 + (lane >> 2);
#pragma unroll
    for (int k4 = 0; k4 < kGK; k4 += 4) {
      double fa[4], fb[NV];
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) fa[mt] = as[mt * 8 * kAPitch + k4];
#pragma unroll
      for (int nt = 0; nt < NV; ++nt) fb[nt] = bs[k4 * kBPitch + nt * 16];
#pragma unroll
      for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int nt = 0; nt < NV; ++nt) dmma8x8x4(acc[mt][nt], fa[mt], fb[nt]);
    }
  };
  for (int kt = 0; kt < total; ++kt) {
    cp_async_wait<kGStages - 2>();
    __syncthreads();  // step kt is in shared memory; step kt-1's buffer is free
    if (kt + kGStages - 1 < total) issue(kt + kGStages - 1);
    cp_async_commit();
    switch (nv) {  // warp-uniform
      case 4: step(kt, std::integral_constant<int, 4>()); break;
      case 3: step(kt, std::integral_constant<int, 3>()); break;
      case 2: step(kt, std::integral_constant<int, 2>()); break;
      case 1: step(kt, std::integral_constant<int, 1>()); break;
      default: break;
    }
  }
  cp_async_wait<0>();
  // D fragment: row lane/4, columns 2 (lane%4) + {0, 1} of each 8x8 tile
#pragma unroll
  for (int mt = 0; mt < 4; ++mt) {
    const int row = r0 + wm * 32 + mt * 8 + (lane >> 2);
    if (row >= rend) continue;
    const int o = b.outrow[row];
    const double sc = b.scale ? b.scale[row] : 1.0;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int n = c0 + (2 * nt + wn) * 8 + 2 * (lane & 3);
      if (n >= ns) continue;  // n even, ns even: n + 1 < ns as well
      double2* cp = reinterpret_cast<double2*>(b.C + (size_t)o * ns + n);
      double2 v = make_double2(sc * acc[mt][nt][0], sc * acc[mt][nt][1]);
      if (b.beta) {
        const double2 c = *cp;
        v.x += c.x;
        v.y += c.y;
      }
      *cp = v;
    }
  }
}

// The same product in 16 x 32 tiles, for batches that leave the 64 x 64 tiles
// on a few SMs (the upper tree levels, the image levels with one row, small
// body sets): a 64 x 64 tile alone takes ns/16 steps of 1024 tensor cycles on
// one SM whatever its rows hold (5 us at ns = 152, 17 us at ns = 488), a
// 16 x 32 tile an eighth of the cycles and a chain of ns/4 dependent mma.
// Each output sums its products in the same order as above, so the choice of
// the tile does not change a result.
constexpr int kSM = 16, kSN = 32, kSK = 32, kSStages = 4;
constexpr int kSAPitch = kSK + 4, kSBPitch = kSN + 4;
constexpr int kSAStage = kSM * kSAPitch, kSBStage = kSK * kSBPitch;
constexpr int kApplySmallBelow = 296;
constexpr size_t kSSmem = sizeof(double) * kSStages * (kSAStage + kSBStage);

__global__ void __launch_bounds__(128) k_apply_f64_small(ApplyBatch b) {
  extern __shared__ __align__(16) double gsm[];
  double* As = gsm;
  double* Bs = gsm + kSStages * kSAStage;
  const int g = blockIdx.z;
  const int rbeg = b.group_off[g], rend = b.group_off[g + 1];
  const int r0 = rbeg + blockIdx.y * kSM;
  const int c0 = blockIdx.x * kSN;
  if (r0 >= rend) return;  // block-uniform
  const int ns = b.ns;
  const double* Bg = b.B + (size_t)g * ns * ns;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 1, wn = warp >> 1;
  const int total = (ns + kSK - 1) / kSK;
  // copies of this thread: A chunks tid, tid + 128 -> row e/16, doubles
  // 2(e%16)..+1; B chunks tid + 128u -> K row e/16, columns 2(e%16)..+1
  int srow[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int row = r0 + ((tid + 128 * u) >> 4);
    srow[u] = row < rend ? b.inrow[row] : -1;
  }
  const int ch = 2 * (tid & 15);
  auto issue = [&](int kt) {
    const int j0 = kt * kSK;
    double* as = As + (kt % kSStages) * kSAStage;
    double* bs = Bs + (kt % kSStages) * kSBStage;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int kr = (tid + 128 * u) >> 4, jj = j0 + kr, n = c0 + ch;
      const bool ok = jj < ns && n < ns;
      cp_async16(bs + kr * kSBPitch + ch, ok ? Bg + (size_t)jj * ns + n : Bg, ok);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j = j0 + ch;
      const bool ok = srow[u] >= 0 && j < ns;
      cp_async16(as + ((tid + 128 * u) >> 4) * kSAPitch + ch, ok ? b.A + (size_t)srow[u] * ns + j : b.A, ok);
    }
  };
  double acc[2][2] = {};
#pragma unroll
  for (int st = 0; st < kSStages - 1; ++st) {
    if (st < total) issue(st);
    cp_async_commit();
  }
  for (int kt = 0; kt < total; ++kt) {
    cp_async_wait<kSStages - 2>();
    __syncthreads();  // step kt is in shared memory; step kt-1's buffer is free
    if (kt + kSStages - 1 < total) issue(kt + kSStages - 1);
    cp_async_commit();
    const double* as = As + (kt % kSStages) * kSAStage + (wm * 8 + (lane >> 2)) * kSAPitch + (lane & 3);
    const double* bs = Bs + (kt % kSStages) * kSBStage + (lane & 3) * kSBPitch + wn * 16 + (lane >> 2);
#pragma unroll
    for (int k4 = 0; k4 < kSK; k4 += 4)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) dmma8x8x4(acc[nt], as[k4], bs[k4 * kSBPitch + nt * 8]);
  }
  cp_async_wait<0>();
  const int row = r0 + wm * 8 + (lane >> 2);
  if (row >= rend) return;
  const int o = b.outrow[row];
  const double sc = b.scale ? b.scale[row] : 1.0;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    const int n = c0 + wn * 16 + nt * 8 + 2 * (lane & 3);
    if (n >= ns) continue;
    double2* cp = reinterpret_cast<double2*>(b.C + (size_t)o * ns + n);
    double2 v = make_double2(sc * acc[nt][0], sc * acc[nt][1]);
    if (b.beta) {
      const double2 c = *cp;
      v.x += c.x;
      v.y += c.y;
    }
    *cp = v;
  }
}

// Sibling sum of the per-child M2M products, in crange order
// (m2m_precompute accumulates child by child, kernel.cpp:398-403).
__global__ void k_sum_children(const int* __restrict__ list, int nparents, const double* __restrict__ Y, int ns,
                               double* __restrict__ q) {
  const int pidx = blockIdx.x;
  if (pidx >= nparents) return;
  const int par = list[3 * pidx], coff = list[3 * pidx + 1], cnum = list[3 * pidx + 2];
  for (int n = threadIdx.x; n < ns; n += blockDim.x) {
    double acc = 0.0;
    for (int c = 0; c < cnum; ++c) acc += Y[(size_t)(coff + c) * ns + n];
    q[(size_t)par * ns + n] = acc;
  }
}

// ---------------------------------------------------------------------------
// FFT-M2L.  Grids are N = 2P-1 points per edge, stored [z][y][x]; spectra are
// the r2c half-spectrum [kz][ky][kx], kx < P.  The twiddle table holds
// w^m = exp(-2 pi i m / N) for m < N.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void cmad(T& re, T& im, T ar, T ai, T br, T bi) {
  re = fma(ar, br, re);
  re = fma(-ai, bi, re);
  im = fma(ar, bi, im);
  im = fma(ai, br, im);
}

// up: one block per (source parent, group of sp child slots): scatter each
// child's equivalent density onto the [0,P)^3 corner of the grid
// (surf_conv_idx_map_up, kernel.cpp:1246-1252, 1304-1315) and take its
// forward DFT separably (x, then y, then z).  The z pass of all sp slots runs
// together so that each frequency's sp values are written contiguously into
// the frequency-major spectrum Q[f][src][slot].
// items: 10 ints per block = src, first slot, child cell per slot (-1 = none).
template <typename T>
__global__ void __launch_bounds__(256)
    k_m2l_up(const double* __restrict__ q_equiv, const int* __restrict__ items,
             const int* __restrict__ surf_ijk, const double* __restrict__ twiddle, int P, int ns, int nsrc,
             int sp, T* __restrict__ Q) {
  extern __shared__ unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);
  const int N = 2 * P - 1;
  const int P3 = P * P * P, Nf = N * N * P, PNP = P * N * P;
  T* W = sm;                       // N*N complex: W[k][n] = w^(k n mod N)
  T* cube = W + 2 * N * N;         // P^3
  T* A = cube + P3;                // P^3 complex: [z][y][kx]
  T* Bm = A + 2 * P3;              // sp * P*N*P complex: [slot][z][ky][kx]
  const int* it = items + 10 * blockIdx.x;
  const int src = it[0], slot0 = it[1];
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < N * N; e += nt) {
    const int m = ((e / N) * (e % N)) % N;
    W[2 * e] = (T)twiddle[2 * m];
    W[2 * e + 1] = (T)twiddle[2 * m + 1];
  }
  for (int j = 0; j < sp; ++j) {
    const int child = it[2 + j];
    T* Bj = Bm + 2 * (size_t)j * PNP;
    if (child < 0) {
      for (int e = tid; e < 2 * PNP; e += nt) Bj[e] = T(0);
      continue;
    }
    for (int e = tid; e < P3; e += nt) cube[e] = T(0);
    __syncthreads();
    for (int i = tid; i < ns; i += nt) {
      const int x = surf_ijk[3 * i], y = surf_ijk[3 * i + 1], z = surf_ijk[3 * i + 2];
      cube[(z * P + y) * P + x] = (T)q_equiv[(size_t)child * ns + i];
    }
    __syncthreads();
    for (int e = tid; e < P3; e += nt) {
      const int z = e / (P * P), y = (e / P) % P, kx = e % P;
      T re = 0, im = 0;
      const T* row = cube + (z * P + y) * P;
      const T* wk = W + 2 * kx * N;
      for (int x = 0; x < P; ++x) {
        re = fma(row[x], wk[2 * x], re);
        im = fma(row[x], wk[2 * x + 1], im);
      }
      A[2 * e] = re;
      A[2 * e + 1] = im;
    }
    __syncthreads();
    for (int e = tid; e < PNP; e += nt) {
      const int z = e / (N * P), ky = (e / P) % N, kx = e % P;
      T re = 0, im = 0;
      const T* wk = W + 2 * ky * N;
      for (int y = 0; y < P; ++y) {
        const int a = (z * P + y) * P + kx;
        cmad(re, im, A[2 * a], A[2 * a + 1], wk[2 * y], wk[2 * y + 1]);
      }
      Bj[2 * e] = re;
      Bj[2 * e + 1] = im;
    }
    __syncthreads();
  }
  __syncthreads();
  using V2 = typename Cplx2<T>::type;  // two complex values
  for (int f = tid; f < Nf; f += nt) {
    const int kz = f / (N * P), ky = (f / P) % N, kx = f % P;
    const T* wk = W + 2 * kz * N;
    for (int j = 0; j < sp; j += 2) {
      T* out = Q + 2 * q8_index<T>(f, src, slot0 + j, nsrc);
      T re0 = 0, im0 = 0, re1 = 0, im1 = 0;
      const T* B0 = Bm + 2 * (size_t)j * PNP;
      const T* B1 = B0 + 2 * (size_t)PNP;
      for (int z = 0; z < P; ++z) {
        const int b = (z * N + ky) * P + kx;
        cmad(re0, im0, B0[2 * b], B0[2 * b + 1], wk[2 * z], wk[2 * z + 1]);
        if (j + 1 < sp) cmad(re1, im1, B1[2 * b], B1[2 * b + 1], wk[2 * z], wk[2 * z + 1]);
      }
      if (j + 1 < sp) {
        V2 v;
        v.x = re0;
        v.y = im0;
        v.z = re1;
        v.w = im1;
        *reinterpret_cast<V2*>(out) = v;
      } else {
        out[0] = re0;
        out[1] = im0;
      }
    }
  }
}

// The up and down kernels above with register blocking, for the orders P
// fixed at compile time.  A thread takes one line of a pass (the values along
// the transformed axis) for 16 bytes of child slots (two in FP32, one in
// FP64) and forms every output of the line in registers.  The twiddles,
// indexed by constants after unrolling, are operands in the kernel's
// parameter bank (the form before read each as a shared-memory broadcast, one
// for two multiply-adds, which bounded it).  Shared memory holds one array
// [z][ky][kx][slot]; every pass works in place on it, which leaves room for
// two to seven blocks per SM.  In FP64 frequencies k and N - k share their
// cosines and sines,
//   X_k e^(it) + X_(N-k) e^(-it) = (X_k + X_(N-k)) cos t + i (X_k - X_(N-k)) sin t,
// which halves the multiply-adds; in FP32 each output sums its terms in the
// order of k_m2l_up / k_m2l_down, bit for bit: the mixed form's error is the
// rounding of these spectra, and another order would move results by as much.
// Up and down at N = 2^20, P = 8 (FP32): 0.20 and 0.34 -> 0.14 and 0.14 ms (paired
// 0.12 and 0.14);
// at P = 10 (FP64, 10^6 bodies in blobs): 1.47 and 2.38 -> 0.84 and 0.78 ms, the
// latter 40% of the measured HBM rate for the spectra alone.
template <typename T, int N>
struct Twiddles {
  T c[N], s[N];  // cos, sin (2 pi m / N)
};
template <typename T>
constexpr bool kPairFrequencies = sizeof(T) == 8;
template <typename T>
struct DftSlots {
  static constexpr int kPer = 16 / (2 * sizeof(T));  // child slots of a thread
  static constexpr int kBlock = 2 * kPer;            // child slots of a block: one sector of spectrum
};
constexpr int dft_threads(int P) { return (2 * (2 * P - 1) * P + 31) / 32 * 32; }
constexpr int dft_blocks(int P, int bytes) {  // resident blocks per SM the registers are sized for
  const int t = dft_threads(P), regs = bytes == 4 ? 64 : P <= 7 ? 80 : 84;
  return 65536 / (t * regs) < 1 ? 1 : 65536 / (t * regs) > 8 ? 8 : 65536 / (t * regs);
}

__device__ __forceinline__ void ld_slots(const float* p, float (&re)[2], float (&im)[2]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  re[0] = v.x;
  im[0] = v.y;
  re[1] = v.z;
  im[1] = v.w;
}
__device__ __forceinline__ void ld_slots(const double* p, double (&re)[1], double (&im)[1]) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  re[0] = v.x;
  im[0] = v.y;
}
__device__ __forceinline__ void st_slots(float* p, const float (&re)[2], const float (&im)[2]) {
  *reinterpret_cast<float4*>(p) = make_float4(re[0], im[0], re[1], im[1]);
}
__device__ __forceinline__ void st_slots(double* p, const double (&re)[1], const double (&im)[1]) {
  *reinterpret_cast<double2*>(p) = make_double2(re[0], im[0]);
}

// N outputs X_k = sum_y x_y exp(-2 pi i k y / N) of P inputs `in[y * si]`,
// given to put(k, re, im).
template <typename T, int P, typename Put>
__device__ __forceinline__ void dft_forward(const T* in, int si, const Twiddles<T, 2 * P - 1>& tw, Put put) {
  constexpr int N = 2 * P - 1, U = DftSlots<T>::kPer;
  T xr[P][U], xi[P][U];
#pragma unroll
  for (int y = 0; y < P; ++y) ld_slots(in + y * si, xr[y], xi[y]);
  if constexpr (!kPairFrequencies<T>) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      T re[U], im[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        re[u] = xr[0][u];
        im[u] = xi[0][u];
#pragma unroll
        for (int y = 1; y < P; ++y) {
          const T c = tw.c[(k * y) % N], s = tw.s[(k * y) % N];
          re[u] = fma(xr[y][u], c, re[u]);
          re[u] = fma(xi[y][u], s, re[u]);
          im[u] = fma(-xr[y][u], s, im[u]);
          im[u] = fma(xi[y][u], c, im[u]);
        }
      }
      put(k, re, im);
    }
  } else {
#pragma unroll
    for (int k = 0; k < P; ++k) {
      T ar[U], ai[U], br[U], bi[U];  // sums of x cos and x sin
#pragma unroll
      for (int u = 0; u < U; ++u) {
        ar[u] = xr[0][u];
        ai[u] = xi[0][u];
        br[u] = bi[u] = T(0);
      }
#pragma unroll
      for (int y = 1; y < P; ++y) {
        const T c = tw.c[(k * y) % N], s = tw.s[(k * y) % N];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          ar[u] = fma(xr[y][u], c, ar[u]);
          ai[u] = fma(xi[y][u], c, ai[u]);
          if (k > 0) {
            br[u] = fma(xr[y][u], s, br[u]);
            bi[u] = fma(xi[y][u], s, bi[u]);
          }
        }
      }
      T re[U], im[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        re[u] = ar[u] + bi[u];
        im[u] = ai[u] - br[u];
      }
      put(k, re, im);
      if (k > 0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          re[u] = ar[u] - bi[u];
          im[u] = ai[u] + br[u];
        }
        put(N - k, re, im);
      }
    }
  }
}

// P outputs x_o = sum_k X_k exp(2 pi i k (P - 1 + o) / N) of N inputs
// `in[k * si]`.
template <typename T, int P>
__device__ __forceinline__ void dft_inverse(const T* in, size_t si, const Twiddles<T, 2 * P - 1>& tw,
                                            T (&re)[P][DftSlots<T>::kPer], T (&im)[P][DftSlots<T>::kPer]) {
  constexpr int N = 2 * P - 1, U = DftSlots<T>::kPer;
  {
    T xr[U], xi[U];
    ld_slots(in, xr, xi);
#pragma unroll
    for (int o = 0; o < P; ++o)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        re[o][u] = xr[u];
        im[o][u] = xi[u];
      }
  }
  if constexpr (!kPairFrequencies<T>) {
#pragma unroll
    for (int k = 1; k < N; ++k) {
      T xr[U], xi[U];
      ld_slots(in + k * si, xr, xi);
#pragma unroll
      for (int o = 0; o < P; ++o) {
        const T c = tw.c[(k * (P - 1 + o)) % N], s = tw.s[(k * (P - 1 + o)) % N];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          re[o][u] = fma(xr[u], c, re[o][u]);
          re[o][u] = fma(-xi[u], s, re[o][u]);
          im[o][u] = fma(xr[u], s, im[o][u]);
          im[o][u] = fma(xi[u], c, im[o][u]);
        }
      }
    }
  } else {
#pragma unroll
    for (int k = 1; k < P; ++k) {
      T xr[U], xi[U], yr[U], yi[U];
      ld_slots(in + k * si, xr, xi);
      ld_slots(in + (N - k) * si, yr, yi);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const T sr = xr[u] + yr[u], sim = xi[u] + yi[u], dr = xr[u] - yr[u], di = xi[u] - yi[u];
#pragma unroll
        for (int o = 0; o < P; ++o) {
          const T c = tw.c[(k * (P - 1 + o)) % N], s = tw.s[(k * (P - 1 + o)) % N];
          re[o][u] = fma(sr, c, re[o][u]);
          re[o][u] = fma(-di, s, re[o][u]);
          im[o][u] = fma(sim, c, im[o][u]);
          im[o][u] = fma(dr, s, im[o][u]);
        }
      }
    }
  }
}

template <typename T, int P>
__global__ void __launch_bounds__(dft_threads(P), dft_blocks(P, sizeof(T)))
    k_m2l_up_rb(const double* __restrict__ q_equiv, const int* __restrict__ items, const int* __restrict__ surf_ijk,
                const __grid_constant__ Twiddles<T, 2 * P - 1> tw, int nsrc, T* __restrict__ Q) {
  constexpr int N = 2 * P - 1, U = DftSlots<T>::kPer, SP = DftSlots<T>::kBlock, ns = 6 * (P - 1) * (P - 1) + 2;
  constexpr int NT = dft_threads(P);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* B = reinterpret_cast<T*>(smem_raw);  // complex [z][ky][kx][slot]
  auto cell = [&](int z, int ky, int kx) { return B + 2 * SP * ((z * N + ky) * P + kx); };
  // the [0,P)^3 corner of the grid, [z][y][x][slot], in the rows ky >= P of
  // each z, which the first pass leaves alone and the second overwrites
  auto corner = [&](int z, int y) { return cell(z, P, 0) + SP * (y * P); };
  const int* it = items + 10 * blockIdx.x;
  const int src = it[0], slot0 = it[1], tid = threadIdx.x;
  bool any = false;
#pragma unroll
  for (int j = 0; j < SP; ++j) any |= it[2 + j] >= 0;
  if (!any) {  // no child here: zero spectra
    const T zero[U] = {};
    for (int e = tid; e < 2 * N * N * P; e += NT)
      st_slots(Q + 2 * q8_index<T>(e >> 1, src, slot0 + (e & 1) * U, nsrc), zero, zero);
    return;
  }
  for (int e = tid; e < P * P * P * SP; e += NT) corner(e / (P * P * SP), 0)[e % (P * P * SP)] = T(0);
  __syncthreads();
  for (int e = tid; e < SP * ns; e += NT) {
    const int j = e / ns, i = e - j * ns;
    const int child = it[2 + j];
    if (child < 0) continue;
    const int x = surf_ijk[3 * i], y = surf_ijk[3 * i + 1], z = surf_ijk[3 * i + 2];
    corner(z, y)[x * SP + j] = (T)q_equiv[(size_t)child * ns + i];
  }
  __syncthreads();
  // x -> kx of the rows (z, y), real input
  for (int e = tid; e < 2 * P * P; e += NT) {
    const int g = e & 1, y = (e >> 1) % P, z = (e >> 1) / P;
    const T* row = corner(z, y) + g * U;
    T r[P][U];
#pragma unroll
    for (int x = 0; x < P; ++x)
#pragma unroll
      for (int u = 0; u < U; ++u) r[x][u] = row[x * SP + u];
#pragma unroll
    for (int kx = 0; kx < P; ++kx) {
      T re[U], im[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        re[u] = r[0][u];
        im[u] = T(0);
#pragma unroll
        for (int x = 1; x < P; ++x) {
          re[u] = fma(r[x][u], tw.c[(x * kx) % N], re[u]);
          im[u] = fma(-r[x][u], tw.s[(x * kx) % N], im[u]);
        }
      }
      st_slots(cell(z, y, kx) + 2 * U * g, re, im);
    }
  }
  __syncthreads();
  // y -> ky of the columns (z, kx)
  for (int e = tid; e < 2 * P * P; e += NT) {
    const int g = e & 1, kx = (e >> 1) % P, z = (e >> 1) / P;
    T* col = cell(z, 0, kx) + 2 * U * g;
    dft_forward<T, P>(col, 2 * SP * P, tw,
                      [&](int ky, const T(&re)[U], const T(&im)[U]) { st_slots(col + ky * 2 * SP * P, re, im); });
  }
  __syncthreads();
  // z -> kz, into the spectra
  for (int e = tid; e < 2 * N * P; e += NT) {
    const int g = e & 1, l = e >> 1;  // l = ky * P + kx
    T* out = Q + 2 * q8_index<T>(l, src, slot0 + g * U, nsrc);
    const size_t so = 2 * (q8_index<T>(N * P, 0, 0, nsrc) - q8_index<T>(0, 0, 0, nsrc));
    dft_forward<T, P>(B + 2 * SP * l + 2 * U * g, 2 * SP * N * P, tw,
                      [&](int kz, const T(&re)[U], const T(&im)[U]) { st_slots(out + kz * so, re, im); });
  }
}

template <typename T, int P>
__global__ void __launch_bounds__(dft_threads(P), dft_blocks(P, sizeof(T)))
    k_m2l_down_rb(const T* __restrict__ Pk, const int* __restrict__ items, const double* __restrict__ tscale,
                  const int* __restrict__ surf_ijk, const __grid_constant__ Twiddles<T, 2 * P - 1> tw, int ntar,
                  double* __restrict__ p_check) {
  constexpr int N = 2 * P - 1, U = DftSlots<T>::kPer, SP = DftSlots<T>::kBlock, ns = 6 * (P - 1) * (P - 1) + 2;
  constexpr int NT = dft_threads(P);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Y = reinterpret_cast<T*>(smem_raw);  // complex [zo][ky][kx][slot]
  auto cell = [&](int z, int ky, int kx) { return Y + 2 * SP * ((z * N + ky) * P + kx); };
  const int* it = items + 10 * blockIdx.x;
  const int tar = it[0], slot0 = it[1], tid = threadIdx.x;
  T re[P][U], im[P][U];
  // kz -> zo, from the spectra
  for (int e = tid; e < 2 * N * P; e += NT) {
    const int g = e & 1, l = e >> 1;  // l = ky * P + kx
    dft_inverse<T, P>(Pk + (((size_t)l * ntar + tar) * 8 + slot0 + g * U) * 2, (size_t)N * P * ntar * 16, tw, re, im);
#pragma unroll
    for (int zo = 0; zo < P; ++zo) st_slots(Y + 2 * SP * (zo * N * P + l) + 2 * U * g, re[zo], im[zo]);
  }
  __syncthreads();
  // ky -> yo of the columns (zo, kx)
  for (int e = tid; e < 2 * P * P; e += NT) {
    const int g = e & 1, kx = (e >> 1) % P, zo = (e >> 1) / P;
    T* col = cell(zo, 0, kx) + 2 * U * g;
    dft_inverse<T, P>(col, 2 * SP * P, tw, re, im);
#pragma unroll
    for (int yo = 0; yo < P; ++yo) st_slots(col + yo * 2 * SP * P, re[yo], im[yo]);
  }
  __syncthreads();
  // kx -> xo of the rows (zo, yo): real output, the half kx >= 1 doubled; an
  // inner row meets the check surface at its ends only
  for (int e = tid; e < 2 * P * P; e += NT) {
    const int g = e & 1, yo = (e >> 1) % P, zo = (e >> 1) / P;
    const bool face = yo == 0 || yo == P - 1 || zo == 0 || zo == P - 1;
    T* row = cell(zo, yo, 0) + 2 * U * g;
#pragma unroll
    for (int kx = 0; kx < P; ++kx) ld_slots(row + kx * 2 * SP, re[kx], im[kx]);
#pragma unroll
    for (int xo = 0; xo < P; ++xo) {
      if (xo > 0 && xo < P - 1 && !face) continue;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        T acc = T(0);
#pragma unroll
        for (int kx = 1; kx < P; ++kx) {
          acc = fma(re[kx][u], tw.c[(kx * (P - 1 + xo)) % N], acc);
          acc = fma(-im[kx][u], tw.s[(kx * (P - 1 + xo)) % N], acc);
        }
        row[xo * 2 * SP + u] = re[0][u] + T(2) * acc;
      }
    }
  }
  __syncthreads();
  const double sc = tscale[tar];
  for (int e = tid; e < SP * ns; e += NT) {
    const int j = e / ns, i = e - j * ns;
    const int child = it[2 + j];
    if (child < 0) continue;
    const int xo = surf_ijk[3 * i], yo = surf_ijk[3 * i + 1], zo = surf_ijk[3 * i + 2];
    p_check[(size_t)child * ns + i] += (double)cell(zo, yo, xo)[(j / U) * 2 * U + j % U] * sc;
  }
}

// Hadamard 8x8 (hadamard_8x8 + c2c_8x8x2_avx, kernel.cpp:1012-1082, c2c.h:201-296):
//   Pk[f][t][itar] = sum_d sum_isrc G[f][d][isrc][itar] * Q[f][src(t,d)][isrc]
// A block holds one frequency's 26x64 kernel coefficients in shared memory
// (every coefficient read is a broadcast) and each thread owns TT targets of
// that frequency: one coefficient read feeds TT targets, and each (target,
// direction) reads one 64-byte source row with sector loads.  L1 wavefronts
// per FMA fall as 1/(4 TT) + 1/16, which is what bounds this kernel.
// FP32 partial sums over DF directions are accumulated into FP64.
constexpr int kHadTT = 2, kHadDF = 8;
constexpr int kHadThreads = 128, kHadBlocks = 4;  // resident blocks per SM

// The source rows of this thread's targets, zero where there is none: chunk c
// holds slots 4c .. 4c+3, one sector.
__device__ __forceinline__ void had_rows(const float2* __restrict__ Qf, int nsrc, const int (&sd)[kHadTT],
                                         float2 (&q)[kHadTT][8]) {
#pragma unroll
  for (int u = 0; u < kHadTT; ++u) {
    if (sd[u] >= 0) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float v[8];
        ld_sector(reinterpret_cast<const float*>(Qf) + ((size_t)c * nsrc + sd[u]) * 8, v);
#pragma unroll
        for (int k = 0; k < 4; ++k) q[u][4 * c + k] = make_float2(v[2 * k], v[2 * k + 1]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) q[u][i] = make_float2(0.f, 0.f);
    }
  }
}

__device__ __forceinline__ void had_index(const int* __restrict__ tsrcT, int d, int t0, int ntar, int (&sd)[kHadTT]) {
#pragma unroll
  for (int u = 0; u < kHadTT; ++u) {
    const int t = t0 + u * kHadThreads;
    sd[u] = t < ntar ? tsrcT[d * ntar + t] : -1;
  }
}

// A direction's product in packed FP32x2 FMAs, the coefficients of an itar pair
// laid (gr0, gr1, gi0, gi1) in shared memory; each output sums its FMAs in the
// order of the sources.
__device__ __forceinline__ void had_mac(const float4* __restrict__ g, const int (&sd)[kHadTT],
                                        const float2 (&q)[kHadTT][8], float (&pr)[kHadTT][8], float (&pi)[kHadTT][8]) {
  bool any = false;
#pragma unroll
  for (int u = 0; u < kHadTT; ++u) any |= sd[u] >= 0;
  if (!any) return;
#pragma unroll
  for (int isrc = 0; isrc < 8; ++isrc) {
    float2 qr[kHadTT], qi[kHadTT], nqi[kHadTT];
#pragma unroll
    for (int u = 0; u < kHadTT; ++u) {
      qr[u] = make_float2(q[u][isrc].x, q[u][isrc].x);
      qi[u] = make_float2(q[u][isrc].y, q[u][isrc].y);
      nqi[u] = make_float2(-q[u][isrc].y, -q[u][isrc].y);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float4 gv = g[isrc * 4 + p];
      const float2 gr = make_float2(gv.x, gv.y), gi = make_float2(gv.z, gv.w);
#pragma unroll
      for (int u = 0; u < kHadTT; ++u) {
        float2 re = make_float2(pr[u][2 * p], pr[u][2 * p + 1]);
        float2 im = make_float2(pi[u][2 * p], pi[u][2 * p + 1]);
        re = __ffma2_rn(gr, qr[u], re);
        re = __ffma2_rn(gi, nqi[u], re);
        im = __ffma2_rn(gr, qi[u], im);
        im = __ffma2_rn(gi, qr[u], im);
        pr[u][2 * p] = re.x;
        pr[u][2 * p + 1] = re.y;
        pi[u][2 * p] = im.x;
        pi[u][2 * p + 1] = im.y;
      }
    }
  }
}

__global__ void __launch_bounds__(kHadThreads, kHadBlocks)
    k_m2l_hadamard8(const float* __restrict__ Q, const float* __restrict__ G, const int* __restrict__ tsrcT, int ntar,
                    int nsrc, float* __restrict__ Pk) {
  constexpr int TT = kHadTT, NT = kHadThreads;
  __shared__ __align__(32) float2 Gs[26 * 64];
  const int f = blockIdx.y;
  const float2* Gf = reinterpret_cast<const float2*>(G) + (size_t)f * 26 * 64;
  // (gr, gi) of itar 2p, 2p+1 -> (gr0, gr1, gi0, gi1)
  float* gs = reinterpret_cast<float*>(Gs);
  for (int e = threadIdx.x; e < 26 * 64; e += NT) {
    const int h = e & 1, b = (e & ~1) * 2;
    const float2 v = Gf[e];
    gs[b + h] = v.x;
    gs[b + 2 + h] = v.y;
  }
  // targets of this thread: t0 + u * NT, u < TT (coalesced tsrcT reads)
  const int t0 = blockIdx.x * NT * TT + threadIdx.x;
  const float2* Qf = reinterpret_cast<const float2*>(Q) + (size_t)f * nsrc * 8;
  // two-stage pipeline over directions: the source rows of direction d+1
  // are in flight while direction d is multiplied, and the row indices run
  // one direction further ahead
  int ia[TT], ib[TT];
  float2 qa[TT][8], qb[TT][8];
  if (t0 < ntar) {
    had_index(tsrcT, 0, t0, ntar, ia);
    had_rows(Qf, nsrc, ia, qa);
    had_index(tsrcT, 1, t0, ntar, ib);
  }
  __syncthreads();
  if (t0 >= ntar) return;
  float pr[TT][8], pi[TT][8];
#pragma unroll
  for (int u = 0; u < TT; ++u)
#pragma unroll
    for (int i = 0; i < 8; ++i) pr[u][i] = pi[u][i] = 0.f;
  // FP64 accumulators: one shared-memory column per thread
  __shared__ double accs[TT * 16][NT];
#pragma unroll
  for (int u = 0; u < TT; ++u)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      accs[u * 16 + 2 * i][threadIdx.x] = 0.0;
      accs[u * 16 + 2 * i + 1][threadIdx.x] = 0.0;
    }
  auto flush = [&]() {
#pragma unroll
    for (int u = 0; u < TT; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        accs[u * 16 + 2 * i][threadIdx.x] += (double)pr[u][i];
        accs[u * 16 + 2 * i + 1][threadIdx.x] += (double)pi[u][i];
        pr[u][i] = pi[u][i] = 0.f;
      }
  };
  auto mac = [&](int d, const int (&sd)[TT], const float2 (&q)[TT][8]) {
    had_mac(reinterpret_cast<const float4*>(Gs + d * 64), sd, q, pr, pi);
  };
  for (int d = 0; d < 26; d += 2) {
    int ja[TT];
    had_rows(Qf, nsrc, ib, qb);
    if (d + 2 < 26) had_index(tsrcT, d + 2, t0, ntar, ja);
    mac(d, ia, qa);
    if (d + 2 < 26) {
#pragma unroll
      for (int u = 0; u < TT; ++u) ia[u] = ja[u];
      had_rows(Qf, nsrc, ia, qa);
    }
    int jb[TT];
    if (d + 3 < 26) had_index(tsrcT, d + 3, t0, ntar, jb);
    mac(d + 1, ib, qb);
    if ((d + 2) % kHadDF == 0 || d + 2 == 26) flush();
    if (d + 3 < 26) {
#pragma unroll
      for (int u = 0; u < TT; ++u) ib[u] = jb[u];
    }
  }
#pragma unroll
  for (int u = 0; u < TT; ++u) {
    const int t = t0 + u * NT;
    if (t >= ntar) break;
    float2* out = reinterpret_cast<float2*>(Pk) + ((size_t)f * ntar + t) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      out[i] = make_float2((float)accs[u * 16 + 2 * i][threadIdx.x], (float)accs[u * 16 + 2 * i + 1][threadIdx.x]);
  }
}

// ---------------------------------------------------------------------------
// Hadamard 8x8 in FP64, on the FP64 tensor path.
//
// The 8x8 block of a direction depends on a child pair only through its
// offset, so along x it is a 2x2 Toeplitz matrix of three 4x4 blocks (a on the
// diagonal, b for source x = 1 and target x = 0, c for the converse):
//   y0 = a x0 + b x1,   y1 = c x0 + a x1.
// Each product is a real 8x8 matrix (4 complex slots) applied to 8 targets by
// two mma.sync.m8n8k4 (real parts, then imaginary parts of the four source
// slots), and a coefficient read feeds 24 targets, which on the FMA pipe
// bounded this product (every multiply-add waited for its share of a
// shared-memory broadcast).  A direction's products are summed by themselves
// and then added to the sum over the directions: 0.99-1.0 times the error of
// the same order of sums in plain FP64 (tests/kernel_errors.cu).  Three
// products instead of four, a (x0 + x1), (b - a) x1 and (c - a) x0, accumulated
// over all directions take 1.92 ms instead of 2.51 (below) but have 1.4 to 4.7
// times that error.
//
// A block takes one frequency and 96 targets, a warp 24 of them as three
// tiles of 8; lane 4 r + q holds source slot q (and q + 4) of target row r.
// A tile none of whose targets has a source in a direction skips it.
// Three tiles a warp and four blocks an SM (122 registers): 2.51 ms at
// N = 2^20, P = 8, ncrit = 256 and 2.43 ms at N = 2^18, ncrit = 64, against
// 2.68 and 2.61 with four tiles and three blocks, 2.80 and 2.68 with two and
// five; 3.60 and 3.34 ms for the product on the FMA pipe.
// ---------------------------------------------------------------------------
constexpr int kHad64Tiles = 3, kHad64Threads = 128, kHad64Blocks = 4;

// Coefficients of a frequency: [direction][block][source slot][target slot]
constexpr int kG64PerDir = 3 * 16;

__device__ __forceinline__ double2 ld_nc_f64x2(const double* p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

__global__ void __launch_bounds__(kHad64Threads, kHad64Blocks)
    k_m2l_hadamard8_f64(const double* __restrict__ Q, const double2* __restrict__ G, const int* __restrict__ tsrcT,
                        int ntar, int nsrc, double* __restrict__ Pk) {
  constexpr int MT = kHad64Tiles;
  // B fragments of both mma of a block, per lane
  __shared__ __align__(16) double2 Bs[26 * 3 * 32];
  const int f = blockIdx.y;
  const double2* Gf = G + (size_t)f * 26 * kG64PerDir;
  for (int e = threadIdx.x; e < 26 * 3 * 32; e += kHad64Threads) {
    // lane 8 t + 4 c + s: source slot s, column 2 t + c (part c of target slot t)
    const double2 g = Gf[(e >> 5) * 16 + (e & 3) * 4 + ((e >> 3) & 3)];
    Bs[e] = e & 4 ? make_double2(g.y, g.x) : make_double2(g.x, -g.y);
  }
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  const int t0 = blockIdx.x * (8 * MT * (kHad64Threads / 32)) + (threadIdx.x >> 5) * (8 * MT) + r;
  // slot q of the x = 0 children; the x = 1 children are two chunks on
  const double* q0 = Q + ((size_t)f * 4 + (q >> 1)) * nsrc * 4 + (q & 1) * 2;
  const double* q1 = q0 + (size_t)nsrc * 8;
  auto index = [&](int d, int (&sd)[MT]) {
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int t = t0 + 8 * m;
      sd[m] = t < ntar ? tsrcT[d * ntar + t] : -1;
    }
  };
  auto rows = [&](const int (&sd)[MT], double2 (&x0)[MT], double2 (&x1)[MT]) {
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      x0[m] = x1[m] = make_double2(0.0, 0.0);
      if (sd[m] >= 0) {
        x0[m] = ld_nc_f64x2(q0 + (size_t)sd[m] * 4);
        x1[m] = ld_nc_f64x2(q1 + (size_t)sd[m] * 4);
      }
    }
  };
  double acc[2][MT][2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[k][m][0] = acc[k][m][1] = 0.0;
  auto mac = [&](int d, const int (&sd)[MT], const double2 (&x0)[MT], const double2 (&x1)[MT]) {
    const double2 a = Bs[(3 * d + 0) * 32 + lane], b = Bs[(3 * d + 1) * 32 + lane], c = Bs[(3 * d + 2) * 32 + lane];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      if (!__any_sync(0xffffffffu, sd[m] >= 0)) continue;
      double y0[2] = {0.0, 0.0}, y1[2] = {0.0, 0.0};
      dmma8x8x4(y0, x0[m].x, a.x);
      dmma8x8x4(y1, x0[m].x, c.x);
      dmma8x8x4(y0, x0[m].y, a.y);
      dmma8x8x4(y1, x0[m].y, c.y);
      dmma8x8x4(y0, x1[m].x, b.x);
      dmma8x8x4(y1, x1[m].x, a.x);
      dmma8x8x4(y0, x1[m].y, b.y);
      dmma8x8x4(y1, x1[m].y, a.y);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        acc[0][m][e] += y0[e];
        acc[1][m][e] += y1[e];
      }
    }
  };
  // two-stage pipeline over the directions: the source rows of direction d+1
  // are in flight while direction d is multiplied, the row indices run one
  // direction further ahead
  int ia[MT], ib[MT];
  double2 xa0[MT], xa1[MT], xb0[MT], xb1[MT];
  index(0, ia);
  rows(ia, xa0, xa1);
  index(1, ib);
  __syncthreads();
  if (t0 - r >= ntar) return;  // warp-uniform
#pragma unroll 1
  for (int d = 0; d < 26; d += 2) {
    int ja[MT], jb[MT];
    rows(ib, xb0, xb1);
    if (d + 2 < 26) index(d + 2, ja);
    mac(d, ia, xa0, xa1);
    if (d + 2 < 26) {
      rows(ja, xa0, xa1);
      index(d + 3, jb);
    }
    mac(d + 1, ib, xb0, xb1);
    if (d + 2 < 26) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        ia[m] = ja[m];
        ib[m] = jb[m];
      }
    }
  }
  // accumulator columns 2 q, 2 q + 1: target slot q, real and imaginary part
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    const int t = t0 + 8 * m;
    if (t >= ntar) break;
    double2* out = reinterpret_cast<double2*>(Pk) + ((size_t)f * ntar + t) * 8 + q;
    out[0] = make_double2(acc[0][m][0], acc[0][m][1]);
    out[4] = make_double2(acc[1][m][0], acc[1][m][1]);
  }
}

// The 8x8 kernel spectra re-laid frequency-major for the Hadamard:
// G[(f * 26 + d) * 64 + pair] = cc8[(d * 64 + pair) * Nf + f] (complex), in
// FP32 by round to nearest.
__global__ void k_g8_layout(const double2* __restrict__ cc8, int Nf, float2* __restrict__ G) {
  const size_t total = (size_t)26 * 64 * Nf;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int pr = (int)(e % 64), d = (int)((e / 64) % 26);
    const size_t f = e / (64 * 26);
    const double2 v = cc8[((size_t)d * 64 + pr) * Nf + f];
    G[e] = make_float2((float)v.x, (float)v.y);
  }
}

// The same for the FP64 form: the coefficients of its three blocks,
// G[((f * 26 + d) * 3 + k) * 16 + 4 s + t] = a, b, c (k = 0, 1, 2) of source
// slot s and target slot t (y and z octant bits).
__global__ void k_g8_layout64(const double2* __restrict__ cc8, int Nf, double2* __restrict__ G) {
  const size_t total = (size_t)26 * kG64PerDir * Nf;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(e % 4), s = (int)(e / 4 % 4), k = (int)(e / 16 % 3), d = (int)(e / 48 % 26);
    const size_t f = e / (48 * 26);
    auto at = [&](int isrc, int itar) { return cc8[((size_t)d * 64 + isrc * 8 + itar) * Nf + f]; };
    G[e] = k == 0 ? at(s, t) : k == 1 ? at(s + 4, t) : at(s, t + 4);
  }
}

// Hadamard 1x27 (hadamard_1x27 + c2c_1x27x1_AVX, kernel.cpp:1084-1138) for the
// image levels, FP64; the 27 image spectra of a direction are pre-summed.
__global__ void k_m2l_hadamard27(const double* __restrict__ Q, const double* __restrict__ G27,
                                 const int* __restrict__ tsrc, int ntar, int nsrc, int Nf,
                                 double* __restrict__ Pk) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  const int t = blockIdx.y;
  if (f >= Nf || t >= ntar) return;
  double re = 0, im = 0;
  for (int d = 0; d < 26; ++d) {
    const int s = tsrc[t * 26 + d];
    if (s < 0) continue;
    const double gr = G27[((size_t)d * Nf + f) * 2], gi = G27[((size_t)d * Nf + f) * 2 + 1];
    const size_t qo = 2 * q8_index<double>(f, s, 0, nsrc);  // the up pass's layout, slot 0
    cmad(re, im, gr, gi, Q[qo], Q[qo + 1]);
  }
  const size_t po = (((size_t)f * ntar + t) * 8 + 0) * 2;
  Pk[po] = re;
  Pk[po + 1] = im;
}

// down: one block per (target parent, group of sp child slots): read the sp
// spectra of each frequency as one contiguous run of the frequency-major
// Pk[f][tar][slot], then for each child the inverse DFT evaluated only at its
// check-surface points, which sit at [P-1, 2P-2]^3 of the grid
// (surf_conv_idx_map_down, kernel.cpp:1253-1259), and
// p_check[child] += value * scale / N^3 (kernel.cpp:1369-1382).
// items: 10 ints per block = tar, first slot, child cell per slot (-1 = none).
template <typename T>
__global__ void __launch_bounds__(256)
    k_m2l_down(const T* __restrict__ Pk, const int* __restrict__ items, const double* __restrict__ tscale,
               const int* __restrict__ surf_ijk, const double* __restrict__ twiddle, int P, int ns, int ntar,
               int sp, double* __restrict__ p_check) {
  extern __shared__ unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);
  const int N = 2 * P - 1;
  const int P3 = P * P * P, Nf = N * N * P;
  T* W = sm;                        // P*N complex: W[o][k] = conj(w)^(k (P-1+o) mod N)
  T* Y1 = W + 2 * P * N;            // P*N*P complex: [zo][ky][kx]
  T* Y2 = Y1 + 2 * P * N * P;       // P^3 complex: [zo][yo][kx]
  T* X = Y2 + 2 * P3;               // sp * Nf complex: [slot][f]
  const int* it = items + 10 * blockIdx.x;
  const int tar = it[0], slot0 = it[1];
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < P * N; e += nt) {
    const int o = e / N, k = e % N;
    const int m = (k * (P - 1 + o)) % N;
    W[2 * e] = (T)twiddle[2 * m];
    W[2 * e + 1] = -(T)twiddle[2 * m + 1];
  }
  if (sp >= 2) {
    using V2 = typename Cplx2<T>::type;
    const int hp = sp / 2;
    for (int e = tid; e < Nf * hp; e += nt) {
      const int f = e / hp, j = 2 * (e % hp);
      const V2 v = *reinterpret_cast<const V2*>(Pk + (((size_t)f * ntar + tar) * 8 + slot0 + j) * 2);
      X[2 * ((size_t)j * Nf + f)] = v.x;
      X[2 * ((size_t)j * Nf + f) + 1] = v.y;
      X[2 * ((size_t)(j + 1) * Nf + f)] = v.z;
      X[2 * ((size_t)(j + 1) * Nf + f) + 1] = v.w;
    }
  } else {
    for (int f = tid; f < Nf; f += nt) {
      const T* in = Pk + (((size_t)f * ntar + tar) * 8 + slot0) * 2;
      X[2 * f] = in[0];
      X[2 * f + 1] = in[1];
    }
  }
  __syncthreads();
  const double sc = tscale[tar];
  for (int j = 0; j < sp; ++j) {
    const int child = it[2 + j];
    if (child < 0) continue;  // block-uniform
    for (int e = tid; e < P * N * P; e += nt) {
      const int zo = e / (N * P), ky = (e / P) % N, kx = e % P;
      const T* wo = W + 2 * zo * N;
      T re = 0, im = 0;
      const T* Xj = X + 2 * (size_t)j * Nf;
      for (int kz = 0; kz < N; ++kz) {
        const int a = (kz * N + ky) * P + kx;
        cmad(re, im, Xj[2 * a], Xj[2 * a + 1], wo[2 * kz], wo[2 * kz + 1]);
      }
      Y1[2 * e] = re;
      Y1[2 * e + 1] = im;
    }
    __syncthreads();
    for (int e = tid; e < P3; e += nt) {
      const int zo = e / (P * P), yo = (e / P) % P, kx = e % P;
      const T* wo = W + 2 * yo * N;
      T re = 0, im = 0;
      for (int ky = 0; ky < N; ++ky) {
        const int a = (zo * N + ky) * P + kx;
        cmad(re, im, Y1[2 * a], Y1[2 * a + 1], wo[2 * ky], wo[2 * ky + 1]);
      }
      Y2[2 * e] = re;
      Y2[2 * e + 1] = im;
    }
    __syncthreads();
    for (int i = tid; i < ns; i += nt) {
      const int xo = surf_ijk[3 * i], yo = surf_ijk[3 * i + 1], zo = surf_ijk[3 * i + 2];
      const T* row = Y2 + 2 * ((zo * P + yo) * P);
      const T* wo = W + 2 * xo * N;
      T acc = 0;
      // Re(Y * conj(w)^m) summed over kx >= 1, doubled for the missing half
      for (int kx = 1; kx < P; ++kx) {
        acc = fma(row[2 * kx], wo[2 * kx], acc);
        acc = fma(-row[2 * kx + 1], wo[2 * kx + 1], acc);
      }
      const T v = row[0] + T(2) * acc;
      p_check[(size_t)child * ns + i] += (double)v * sc;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// post: far + near, dipole correction (kernel.cpp:1580-1596), 1/(4 pi)
// (body.cpp:88-96), and the scatter back to input order (body.cpp:177-190).
// ---------------------------------------------------------------------------
constexpr int kDipBlocks = kDipoleBlocks;

__global__ void k_dipole_partial(const double4* __restrict__ body64, int n, double* __restrict__ partial) {
  // per block: sum of q x, q y, q z and q
  __shared__ double s[4][256];
  double ax = 0, ay = 0, az = 0, aq = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double4 b = body64[i];
    ax += b.x * b.w;
    ay += b.y * b.w;
    az += b.z * b.w;
    aq += b.w;
  }
  s[0][threadIdx.x] = ax;
  s[1][threadIdx.x] = ay;
  s[2][threadIdx.x] = az;
  s[3][threadIdx.x] = aq;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h)
      for (int k = 0; k < 4; ++k) s[k][threadIdx.x] += s[k][threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 4; ++k) partial[blockIdx.x * 4 + k] = s[k][0];
}

__global__ void k_dipole_final(double* __restrict__ partial) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double d[4] = {0, 0, 0, 0};
  for (int b = 0; b < kDipBlocks; ++b)
    for (int k = 0; k < 4; ++k) d[k] += partial[b * 4 + k];
  for (int k = 0; k < 4; ++k) partial[4 * kDipBlocks + k] = d[k];
}

// Adjoint support.  k_swap_charges puts the weights w (input order) into the
// tree-order bodies and keeps their charges; k_restore_charges puts them
// back; k_adj_combine forms dL/dx_k = w_k grad(phi_q)_k + q_k grad(psi_w)_k
// in input order (k = perm[i]).
__global__ void k_swap_charges(double4* __restrict__ body64, const double* __restrict__ w,
                               const int64_t* __restrict__ perm, int n, double* __restrict__ qsave) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  qsave[i] = body64[i].w;
  body64[i].w = w[perm[i]];
}

// New charges (input order) for bodies whose positions are already on the
// device in tree order.
__global__ void k_set_charges(double4* __restrict__ body64, const double* __restrict__ q,
                              const int64_t* __restrict__ perm, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  body64[i].w = q[perm[i]];
}

__global__ void k_restore_charges(double4* __restrict__ body64, const double* __restrict__ qsave, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  body64[i].w = qsave[i];
}

__global__ void k_adj_combine(const int64_t* __restrict__ perm, const double* __restrict__ w,
                              const double* __restrict__ qsave, const double* __restrict__ grad_q,
                              const double* __restrict__ grad_w, int n, double* __restrict__ dLdx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t k = perm[i];
  const double wk = w[k], qk = qsave[i];
#pragma unroll
  for (int c = 0; c < 3; ++c) dLdx[3 * k + c] = wk * grad_q[3 * k + c] + qk * grad_w[3 * k + c];
}

__global__ void k_post(const double* __restrict__ phi_far, const double* __restrict__ grad_far,
                       const double* __restrict__ phi_near, const double* __restrict__ grad_near,
                       const double4* __restrict__ body64, const int64_t* __restrict__ perm, int n,
                       const double* __restrict__ dip, double coef, int dipole, double cx, double cy, double cz,
                       double out_scale, double* __restrict__ out_phi, double* __restrict__ out_grad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double p = 0, g0 = 0, g1 = 0, g2 = 0;
  if (phi_far) {
    p += phi_far[i];
    g0 += grad_far[3 * i];
    g1 += grad_far[3 * i + 1];
    g2 += grad_far[3 * i + 2];
  }
  if (phi_near) {
    p += phi_near[i];
    g0 += grad_near[3 * i];
    g1 += grad_near[3 * i + 1];
    g2 += grad_near[3 * i + 2];
  }
  if (dipole) {
    // mu = sum q (x - centre): the reference's dipole, whose box is centred
    // at the origin (argument.cpp:61-62)
    const double Q = dip[3];
    const double dx = dip[0] - Q * cx, dy = dip[1] - Q * cy, dz = dip[2] - Q * cz;
    if (dipole == 1) {
      // the reference's per-body form coef |mu|^2 / (N q_i) (kernel.cpp:1593)
      const double dnorm = dx * dx + dy * dy + dz * dz;
      p -= coef * dnorm / n / body64[i].w;
    } else {
      // the potential of the surface term: coef mu . (x_i - centre)
      const double4 b = body64[i];
      p -= coef * (dx * (b.x - cx) + dy * (b.y - cy) + dz * (b.z - cz));
    }
    g0 -= coef * dx;
    g1 -= coef * dy;
    g2 -= coef * dz;
  }
  const int64_t o = perm[i];
  out_phi[o] = p * out_scale;
  out_grad[3 * o + 0] = g0 * out_scale;
  out_grad[3 * o + 1] = g1 * out_scale;
  out_grad[3 * o + 2] = g2 * out_scale;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline int cdiv(int64_t a, int b) { return (int)((a + b - 1) / b); }

cudaError_t launch_gather_bodies(const double* x_in, const double* q_in, const int64_t* perm, int n,
                                 double4* body64, cudaStream_t st) {
  if (n > 0) k_gather_bodies<<<cdiv(n, 256), 256, 0, st>>>(x_in, q_in, perm, n, body64);
  return cudaGetLastError();
}

cudaError_t launch_prep32(const double4* body64, const int* body_leaf, const LeafInfo* leaves,
                          float4* body32, int n, cudaStream_t st) {
  if (n > 0) k_prep32<<<cdiv(n, 256), 256, 0, st>>>(body64, body_leaf, leaves, body32, n);
  return cudaGetLastError();
}

cudaError_t launch_p2p32(const float4* body32, const P2PItem* items, int nitems, bool long_entries, bool cut,
                         const P2PSrc32* list, double4* part, int* done, double* phi, double* grad, cudaStream_t st) {
  if (nitems > 0) {
    auto kernel = long_entries ? cut ? k_p2p32<true, true> : k_p2p32<true, false>
                               : cut ? k_p2p32<false, true> : k_p2p32<false, false>;
    kernel<<<cdiv(nitems, kP2PWarps), 32 * kP2PWarps, 0, st>>>(body32, items, nitems, list, part, done, phi, grad);
  }
  return cudaGetLastError();
}

cudaError_t launch_p2p64(const double4* body64, const P2PItem* items, int nitems, const P2PSrc64* list, double4* part,
                         int* done, double* phi, double* grad, cudaStream_t st) {
  if (nitems > 0)
    k_p2p64<<<cdiv(nitems, kP2PWarps), 32 * kP2PWarps, 0, st>>>(body64, items, nitems, list, part, done, phi, grad);
  return cudaGetLastError();
}

cudaError_t launch_close_count(const float4* body32, const P2PItem* items, int nitems, const int* list_off,
                               const P2PSrc32* list, const LeafInfo* leaves, int* cnt, cudaStream_t st) {
  if (nitems > 0)
    k_close_scan<false><<<cdiv(nitems, 8), 256, 0, st>>>(body32, items, nitems, list_off, list, leaves, cnt,
                                                         nullptr, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_close_emit(const float4* body32, const P2PItem* items, int nitems, const int* list_off,
                              const P2PSrc32* list, const LeafInfo* leaves, const int* off, int2* pairs,
                              cudaStream_t st) {
  if (nitems > 0)
    k_close_scan<true><<<cdiv(nitems, 8), 256, 0, st>>>(body32, items, nitems, list_off, list, leaves, nullptr,
                                                        off, pairs);
  return cudaGetLastError();
}

cudaError_t launch_close_fix(const double4* body64, const float4* body32, const P2PSrc32* list, const int* off,
                             const int2* pairs, int n, double cycle, double* phi, double* grad, cudaStream_t st) {
  if (n > 0) k_close_fix<<<cdiv(n, 256), 256, 0, st>>>(body64, body32, list, off, pairs, n, cycle, phi, grad);
  return cudaGetLastError();
}

cudaError_t launch_count_scan(const int* cnt, int* off, int n, void* tmp, size_t* tmp_bytes, cudaStream_t st) {
  return cub::DeviceScan::ExclusiveSum(tmp, *tmp_bytes, cnt, off, n, st);
}

cudaError_t launch_p2m_check(const double4* body64, const LeafInfo* leaves, int nleaf,
                             const double* surf_unit, int ns, double* out, cudaStream_t st, bool full) {
  if (nleaf > 0) {
    const int per = cdiv(ns, kCheckPer);
    const int nt = per >= kCheckMaxThreads ? kCheckMaxThreads : cdiv(per, 32) * 32;
    if (full)
      k_p2m_check<true><<<nleaf, nt, 0, st>>>(body64, leaves, surf_unit, ns, out);
    else
      k_p2m_check<false><<<nleaf, nt, 0, st>>>(body64, leaves, surf_unit, ns, out);
  }
  return cudaGetLastError();
}

template <bool FULL>
static cudaError_t l2p_eval(const double4* body64, const LeafInfo* leaves, int nleaf, const double* surf_unit, int ns,
                          const double* q_down, double* phi, double* grad, cudaStream_t st) {
  const size_t sm = sizeof(double4) * ns;
  if (sm > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_l2p_eval<FULL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
  }
  k_l2p_eval<FULL><<<nleaf, kSurfThreads, sm, st>>>(body64, leaves, surf_unit, ns, q_down, phi, grad);
  return cudaGetLastError();
}

cudaError_t launch_l2p_eval(const double4* body64, const LeafInfo* leaves, int nleaf,
                            const double* surf_unit, int ns, const double* q_down, double* phi,
                            double* grad, cudaStream_t st, bool full) {
  if (nleaf <= 0) return cudaGetLastError();
  return full ? l2p_eval<true>(body64, leaves, nleaf, surf_unit, ns, q_down, phi, grad, st)
              : l2p_eval<false>(body64, leaves, nleaf, surf_unit, ns, q_down, phi, grad, st);
}

cudaError_t launch_apply(const ApplyBatch& b, cudaStream_t st) {
  if (b.max_rows > 0 && b.groups > 0) {
    if (b.ns % 2 != 0) return cudaErrorInvalidValue;  // 16-byte copies need an even ns
    // the shared-memory opt-in is per function and device; set once per
    // device, safely when several host threads make their first call at once
    static std::atomic<bool> attr_set[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
      e = cudaFuncSetAttribute(k_apply_f64_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGSmem);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_apply_f64_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSSmem);
      if (e != cudaSuccess) return e;
      if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    // small tiles while there are fewer large ones than two an SM: the chip is
    // then part idle, and a large tile's ns/16 steps are the kernel's length.
    // M2M + L2L of 8192 bodies at P = 6: 0.174 ms in large tiles, 0.084 here;
    // of 2^20 at P = 8: 0.639 and 0.455; with the line at one large tile an SM
    // 0.127 against 0.119 (200003 bodies, P = 6), at four the same as at two.
    const int64_t large = (int64_t)cdiv(b.ns, kGN) * cdiv(b.max_rows, kGM) * b.groups;
    if (large < kApplySmallBelow) {
      dim3 grid(cdiv(b.ns, kSN), cdiv(b.max_rows, kSM), b.groups);
      k_apply_f64_small<<<grid, 128, kSSmem, st>>>(b);
    } else {
      dim3 grid(cdiv(b.ns, kGN), cdiv(b.max_rows, kGM), b.groups);
      k_apply_f64_tc<<<grid, kGThreads, kGSmem, st>>>(b);
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_sum_children(const int* list, int nparents, const double* Y, int ns, double* q,
                                cudaStream_t st) {
  if (nparents > 0) k_sum_children<<<nparents, 128, 0, st>>>(list, nparents, Y, ns, q);
  return cudaGetLastError();
}

// orders with a compile-time instance (the register-blocked kernels): FP32
// runs at P <= 8 only
template <typename T>
static bool fixed_p(int P) {
  return P >= 4 && P <= (sizeof(T) == 4 ? 8 : 10);
}
template <typename T>
static size_t up_smem(int P, int sp) {
  const size_t N = 2 * P - 1, P3 = (size_t)P * P * P;
  if (fixed_p<T>(P)) return sizeof(T) * 2 * DftSlots<T>::kBlock * P * N * P;
  return sizeof(T) * (2 * N * N + 3 * P3 + 2 * (size_t)sp * P * N * P);
}
template <typename T>
static size_t down_smem(int P, int sp) {
  const size_t N = 2 * P - 1, P3 = (size_t)P * P * P;
  if (fixed_p<T>(P)) return sizeof(T) * 2 * DftSlots<T>::kBlock * P * N * P;
  return sizeof(T) * (2 * (size_t)P * N + 2 * (size_t)P * N * P + 2 * P3 + 2 * (size_t)sp * N * N * P);
}
template <typename T, int N>
static Twiddles<T, N> twiddles() {
  Twiddles<T, N> t;
  for (int m = 0; m < N; ++m) {
    t.c[m] = (T)std::cos(2.0 * M_PI * m / N);
    t.s[m] = (T)std::sin(2.0 * M_PI * m / N);
  }
  return t;
}

// Largest slot group (8, 4, 2, 1) whose working set fits in shared memory.
static const size_t kSmemMax = 220 * 1024;
// Capped at one 32-byte sector of spectrum per frequency (4 FP32 or 2 FP64
// complex values), which keeps enough blocks in flight.
template <typename T>
int m2l_up_slots(int P) {
  for (int sp = (int)(32 / (2 * sizeof(T))); sp > 1; sp /= 2)
    if (up_smem<T>(P, sp) <= kSmemMax) return sp;
  return 1;
}
template <typename T>
int m2l_down_slots(int P) {
  for (int sp = (int)(32 / (2 * sizeof(T))); sp > 1; sp /= 2)
    if (down_smem<T>(P, sp) <= kSmemMax) return sp;
  return 1;
}
template int m2l_up_slots<float>(int);
template int m2l_up_slots<double>(int);
template int m2l_down_slots<float>(int);
template int m2l_down_slots<double>(int);

template <typename T, int PP>
static cudaError_t up_p(const double* q_equiv, const int* items, int nitems, const int* surf_ijk,
                        const double* twiddle, int P, int ns, int nsrc, int sp, T* Q, cudaStream_t st) {
  const size_t sm = up_smem<T>(P, sp);
  if constexpr (PP > 0) {
    cudaError_t e = cudaFuncSetAttribute(k_m2l_up_rb<T, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k_m2l_up_rb<T, PP><<<nitems, dft_threads(PP), sm, st>>>(q_equiv, items, surf_ijk, twiddles<T, 2 * PP - 1>(), nsrc,
                                                            Q);
  } else {
    cudaError_t e = cudaFuncSetAttribute(k_m2l_up<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k_m2l_up<T><<<nitems, 256, sm, st>>>(q_equiv, items, surf_ijk, twiddle, P, ns, nsrc, sp, Q);
  }
  return cudaGetLastError();
}

// calls f(integral_constant<P>) for an order with a compile-time instance, else f(0)
template <typename T, typename F>
static cudaError_t with_order(int P, F f) {
  switch (P) {
    case 4: return f(std::integral_constant<int, 4>());
    case 5: return f(std::integral_constant<int, 5>());
    case 6: return f(std::integral_constant<int, 6>());
    case 7: return f(std::integral_constant<int, 7>());
    case 8: return f(std::integral_constant<int, 8>());
    default: break;
  }
  if constexpr (sizeof(T) == 8) {
    if (P == 9) return f(std::integral_constant<int, 9>());
    if (P == 10) return f(std::integral_constant<int, 10>());
  }
  return f(std::integral_constant<int, 0>());
}

template <typename T>
cudaError_t launch_m2l_up(const double* q_equiv, const int* items, int nitems, const int* surf_ijk,
                          const double* twiddle, int P, int ns, int nsrc, int sp, T* Q, cudaStream_t st) {
  if (nitems <= 0) return cudaGetLastError();
  return with_order<T>(P, [&](auto pp) {
    return up_p<T, pp.value>(q_equiv, items, nitems, surf_ijk, twiddle, P, ns, nsrc, sp, Q, st);
  });
}

cudaError_t launch_m2l_hadamard8(const float* Q, const float* G, const int* tsrcT, int ntar, int nsrc, int Nf,
                                 float* Pk, cudaStream_t st) {
  if (ntar > 0) {
    dim3 grid(cdiv(ntar, kHadThreads * kHadTT), Nf);
    k_m2l_hadamard8<<<grid, kHadThreads, 0, st>>>(Q, G, tsrcT, ntar, nsrc, Pk);
  }
  return cudaGetLastError();
}

cudaError_t launch_m2l_hadamard8(const double* Q, const double* G, const int* tsrcT, int ntar, int nsrc, int Nf,
                                 double* Pk, cudaStream_t st) {
  if (ntar > 0) {
    dim3 grid(cdiv(ntar, 8 * kHad64Tiles * (kHad64Threads / 32)), Nf);
    k_m2l_hadamard8_f64<<<grid, kHad64Threads, 0, st>>>(Q, reinterpret_cast<const double2*>(G), tsrcT, ntar, nsrc,
                                                        Pk);
  }
  return cudaGetLastError();
}

size_t g8_layout_size(int Nf, bool fp32) { return (size_t)26 * (fp32 ? 64 : kG64PerDir) * Nf * 2; }

cudaError_t launch_g8_layout(const double* cc8, int Nf, float* G, cudaStream_t st) {
  const size_t total = (size_t)26 * 64 * Nf;
  if (total > 0)
    k_g8_layout<<<(int)std::min<size_t>((total + 255) / 256, 148 * 16), 256, 0, st>>>(
        reinterpret_cast<const double2*>(cc8), Nf, reinterpret_cast<float2*>(G));
  return cudaGetLastError();
}

cudaError_t launch_g8_layout(const double* cc8, int Nf, double* G, cudaStream_t st) {
  const size_t total = (size_t)26 * kG64PerDir * Nf;
  if (total > 0)
    k_g8_layout64<<<(int)std::min<size_t>((total + 255) / 256, 148 * 16), 256, 0, st>>>(
        reinterpret_cast<const double2*>(cc8), Nf, reinterpret_cast<double2*>(G));
  return cudaGetLastError();
}

cudaError_t launch_body_leaf(const LeafInfo* leaves, int nleaf, int n, int* body_leaf, cudaStream_t st) {
  if (nleaf > 0) k_body_leaf<<<nleaf, 128, 0, st>>>(leaves, nleaf, n, body_leaf);
  return cudaGetLastError();
}

cudaError_t launch_m2l_hadamard27(const double* Q, const double* G27, const int* tsrc, int ntar, int nsrc,
                                  int Nf, double* Pk, cudaStream_t st) {
  if (ntar > 0) {
    dim3 grid(cdiv(Nf, 128), ntar);
    k_m2l_hadamard27<<<grid, 128, 0, st>>>(Q, G27, tsrc, ntar, nsrc, Nf, Pk);
  }
  return cudaGetLastError();
}

template <typename T, int PP>
static cudaError_t down_p(const T* Pk, const int* items, const double* tscale, int nitems, const int* surf_ijk,
                          const double* twiddle, int P, int ns, int ntar, int sp, double* p_check,
                          cudaStream_t st) {
  const size_t sm = down_smem<T>(P, sp);
  if constexpr (PP > 0) {
    cudaError_t e =
        cudaFuncSetAttribute(k_m2l_down_rb<T, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k_m2l_down_rb<T, PP><<<nitems, dft_threads(PP), sm, st>>>(Pk, items, tscale, surf_ijk,
                                                              twiddles<T, 2 * PP - 1>(), ntar, p_check);
  } else {
    cudaError_t e = cudaFuncSetAttribute(k_m2l_down<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k_m2l_down<T><<<nitems, 256, sm, st>>>(Pk, items, tscale, surf_ijk, twiddle, P, ns, ntar, sp, p_check);
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_m2l_down(const T* Pk, const int* items, const double* tscale, int nitems,
                            const int* surf_ijk, const double* twiddle, int P, int ns, int ntar, int sp,
                            double* p_check, cudaStream_t st) {
  if (nitems <= 0) return cudaGetLastError();
  return with_order<T>(P, [&](auto pp) {
    return down_p<T, pp.value>(Pk, items, tscale, nitems, surf_ijk, twiddle, P, ns, ntar, sp, p_check, st);
  });
}

cudaError_t launch_dipole(const double4* body64, int n, double* partial, cudaStream_t st) {
  k_dipole_partial<<<kDipBlocks, 256, 0, st>>>(body64, n, partial);
  k_dipole_final<<<1, 32, 0, st>>>(partial);
  return cudaGetLastError();
}

cudaError_t launch_swap_charges(double4* body64, const double* w, const int64_t* perm, int n, double* qsave,
                                cudaStream_t st) {
  if (n > 0) k_swap_charges<<<cdiv(n, 256), 256, 0, st>>>(body64, w, perm, n, qsave);
  return cudaGetLastError();
}

cudaError_t launch_set_charges(double4* body64, const double* q, const int64_t* perm, int n, cudaStream_t st) {
  if (n > 0) k_set_charges<<<cdiv(n, 256), 256, 0, st>>>(body64, q, perm, n);
  return cudaGetLastError();
}

cudaError_t launch_restore_charges(double4* body64, const double* qsave, int n, cudaStream_t st) {
  if (n > 0) k_restore_charges<<<cdiv(n, 256), 256, 0, st>>>(body64, qsave, n);
  return cudaGetLastError();
}

cudaError_t launch_adj_combine(const int64_t* perm, const double* w, const double* qsave, const double* grad_q,
                               const double* grad_w, int n, double* dLdx, cudaStream_t st) {
  if (n > 0) k_adj_combine<<<cdiv(n, 256), 256, 0, st>>>(perm, w, qsave, grad_q, grad_w, n, dLdx);
  return cudaGetLastError();
}

// Leaf rows of the cell vectors <-> a leaf-ordered buffer (the exchange of
// a sharded pass): gather writes buf[l] = own[l] ? v[cell[l]] : 0 (own null:
// every row), scatter writes v[cell[l]] = buf[l].
__global__ void k_leaf_rows(double* __restrict__ v, int nrow, const int* __restrict__ cells,
                            const char* __restrict__ own, int nleaf, int ns, double* __restrict__ buf, int scatter) {
  const int l = blockIdx.x;
  if (l >= nleaf) return;
  const int c = cells[l];
  if (c < 0 || c >= nrow) return;  // not a row of v
  double* row = v + (size_t)c * ns;
  double* b = buf + (size_t)l * ns;
  if (scatter) {
    for (int i = threadIdx.x; i < ns; i += blockDim.x) row[i] = b[i];
  } else {
    const bool keep = own == nullptr || own[l];
    for (int i = threadIdx.x; i < ns; i += blockDim.x) b[i] = keep ? row[i] : 0.0;
  }
}

cudaError_t launch_leaf_rows(double* v, int nrow, const int* cells, const char* own, int nleaf, int ns,
                             double* buf, bool scatter, cudaStream_t st) {
  if (nleaf > 0 && (!v || !cells || !buf)) return cudaErrorInvalidValue;
  if (nleaf > 0) k_leaf_rows<<<nleaf, 128, 0, st>>>(v, nrow, cells, own, nleaf, ns, buf, scatter ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t launch_post(const double* phi_far, const double* grad_far, const double* phi_near,
                        const double* grad_near, const double4* body64, const int64_t* perm, int n,
                        const double* dipole_partial, double coef, int dipole, const double* centre,
                        double out_scale, double* out_phi, double* out_grad, cudaStream_t st) {
  if (n > 0)
    k_post<<<cdiv(n, 256), 256, 0, st>>>(phi_far, grad_far, phi_near, grad_near, body64, perm, n,
                                          dipole_partial + 4 * kDipBlocks, coef, dipole, centre[0], centre[1],
                                          centre[2], out_scale, out_phi, out_grad);
  return cudaGetLastError();
}

template cudaError_t launch_m2l_up<float>(const double*, const int*, int, const int*, const double*, int, int,
                                          int, int, float*, cudaStream_t);
template cudaError_t launch_m2l_up<double>(const double*, const int*, int, const int*, const double*, int, int,
                                           int, int, double*, cudaStream_t);
template cudaError_t launch_m2l_down<float>(const float*, const int*, const double*, int, const int*,
                                            const double*, int, int, int, int, double*, cudaStream_t);
template cudaError_t launch_m2l_down<double>(const double*, const int*, const double*, int, const int*,
                                             const double*, int, int, int, int, double*, cudaStream_t);

}  // namespace rtfmm_b200
