// Device kernels of the evaluation pass (sm_100a).  Declarations shared by
// rtfmm_kernels.cu and the orchestration in rtfmm_capi.cu.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace rtfmm_b200 {

// Leaf table: one entry per leaf cell.
struct LeafInfo {
  double cx, cy, cz;   // centre
  double r;            // half edge
  double scale;        // 0.5^depth (P2M / L2P operator rescaling)
  int cell;            // cell index
  int boff, bnum;      // bodies in tree order
};

// P2P work item: nt <= W targets of one leaf, W = 1 << lw
// lanes per target group; the 32/W groups of a warp split every source tile
// between them, so a leaf's last few targets do not leave most lanes idle.
// `e0`..`e1` is the item's part of the leaf's source list: a list of more than
// p2p_part_bodies bodies is cut into `nparts` items of the same targets, whose
// sums meet in slots `slot`..`slot + nparts - 1`.
struct P2PItem {
  int leaf;      // leaf-table index of the target leaf
  int boff;      // first target body (tree order)
  short nt, lw;  // targets in this item (1..W); log2 W, W in {4, 8, 16, 32}
  int e0, e1;    // source-list entries
  int part, nparts, slot;
};
// Bodies of a source list from which it is cut, for a plan with `work` =
// sum over leaves of list bodies x target groups of 32.  A part is at most
// about an eighth of what each of 20 warps an SM (148 SMs) has to do, so that
// no warp is left running alone for long, and at least 256 bodies, below which
// a part's fixed cost shows.  Stage times: 150,001 bodies in blobs, FP64, 0.59
// ms with halves, 0.51 with quarters, 0.47 with eighths, 0.45 with sixteenths,
// whose slots take 53 instead of 28 MB; 4 M bodies in blobs, mixed (across
// entries), 8.46, 8.37, 8.29, 8.24 ms.  At least 64, 256, 1024 bodies: 30,011 bodies in blobs, mixed, 75,
// 52.5, 52 us; 8192 bodies uniform, FP64, 23, 29, 47 us, where the far field's
// chain of small kernels runs beside it and takes 150.
#ifdef __CUDACC__
__host__ __device__
#endif
inline int p2p_part_bodies(unsigned long long work) {
  const unsigned long long s = work / (148 * 20 * 8);
  return s < 256 ? 256 : s > (1 << 20) ? 1 << 20 : (int)s;
}

// Whether a plan's FP32 P2P takes its sources entry by entry or fills its tiles
// across entries, by the mean bodies of an entry: `work` as above, `entries` =
// sum over leaves of list entries x target groups of 32.  Entry by entry leaves
// tiles part empty, across entries costs a frame offset a pair and more sums
// into FP64.  Stage times, entry by entry and across: mean 12.8 bodies (2^20
// uniform) 1.48 and 0.87 ms, 15.6 (64,000 on a lattice) 0.049 and 0.046, 17.9
// (100,003 uniform) 0.093 and 0.085, 24.4 0.073 and 0.081, 27.6 (150,001 in
// blobs) 0.245 and 0.251, 32 (2^20) 0.70 and 0.76, 256 3.65 and 4.6.
#ifdef __CUDACC__
__host__ __device__
#endif
inline bool p2p_long_entries(unsigned long long work, unsigned long long entries) { return work >= 20 * entries; }

// One P2P list entry (source leaf) of a target leaf, FP32 form.  Both forms
// carry the source's body range so that the kernels read bodies with one
// dependent load.
struct alignas(16) P2PSrc32 {
  float dx, dy, dz;   // c_src + offset - c_tar, for leaf-relative FP32 positions
  int leaf;           // leaf-table index of the source leaf
  int self;           // source == target with zero offset (mask r == 0)
  int boff, bnum;     // source bodies (tree order)
  int pad;
};
struct P2PSrc64 {
  double ox, oy, oz;  // periodic offset added to the source positions
  int leaf;
  int self;
  int boff, bnum;     // source bodies (tree order)
};

// Batched FP64 operator application (see k_apply_f64_tc).
struct ApplyBatch {
  const double* A;      // input vectors, row stride ns
  const int* inrow;     // input row indices (-1 = zero vector)
  const double* B;      // groups x ns x ns operator stack, row-major [j][n]
  const int* outrow;    // output row indices
  const double* scale;  // per-row scale (nullptr = 1)
  const int* group_off; // groups+1 row offsets
  double* C;            // output vectors, row stride ns
  int groups, ns, beta;
  int max_rows;         // rows of the largest group (grid sizing)
};

// Launch helpers (all asynchronous on `st`; return cudaGetLastError()).
// body_leaf[b] = leaf of tree-order body b (the leaves partition [0, n))
cudaError_t launch_body_leaf(const LeafInfo* leaves, int nleaf, int n, int* body_leaf, cudaStream_t st);
cudaError_t launch_prep32(const double4* body64, const int* body_leaf, const LeafInfo* leaves,
                          float4* body32, int n, cudaStream_t st);
// part: 32 double4 per slot of the items, done: one counter per slot, zero
// before the first pass (every pass leaves them zero)
cudaError_t launch_p2p32(const float4* body32, const P2PItem* items, int nitems, bool long_entries, bool cut,
                         const P2PSrc32* list, double4* part, int* done, double* phi, double* grad,
                         cudaStream_t st);
cudaError_t launch_p2p64(const double4* body64, const P2PItem* items, int nitems,
                         const P2PSrc64* list, double4* part, int* done, double* phi, double* grad,
                         cudaStream_t st);
// Close-pair refinement of the FP32 P2P: per-target counts of the pairs
// closer than a fraction of their leaves (cnt[t], tree order), their list
// (source body, list entry) at pairs[off[t]...], and the per-pass fix that
// replaces their FP32 terms in phi / grad (P2P outputs) by FP64 ones.
cudaError_t launch_close_count(const float4* body32, const P2PItem* items, int nitems, const int* list_off,
                               const P2PSrc32* list, const LeafInfo* leaves, int* cnt, cudaStream_t st);
cudaError_t launch_close_emit(const float4* body32, const P2PItem* items, int nitems, const int* list_off,
                              const P2PSrc32* list, const LeafInfo* leaves, const int* off, int2* pairs,
                              cudaStream_t st);
// cycle > 0: periodic (nearest image); 0: free space
cudaError_t launch_close_fix(const double4* body64, const float4* body32, const P2PSrc32* list, const int* off,
                             const int2* pairs, int n, double cycle, double* phi, double* grad, cudaStream_t st);
// off = exclusive prefix sum of cnt (n values); tmp == nullptr: *tmp_bytes
// = the scratch it needs
cudaError_t launch_count_scan(const int* cnt, int* off, int n, void* tmp, size_t* tmp_bytes, cudaStream_t st);
// full: reciprocal square roots to full precision, else to 1.3e-12 (mixed form)
cudaError_t launch_p2m_check(const double4* body64, const LeafInfo* leaves, int nleaf,
                             const double* surf_unit, int ns, double* out, cudaStream_t st, bool full = true);
cudaError_t launch_apply(const ApplyBatch& b, cudaStream_t st);
// q[parent] = sum of Y[child] over the parent's children; `list` holds
// (parent, coff, cnum) triplets
cudaError_t launch_sum_children(const int* list, int nparents, const double* Y, int ns, double* q,
                                cudaStream_t st);
// FFT-M2L spectra are frequency-major: Q[f][src][slot], Pk[f][tar][slot]
// (complex, interleaved re/im).
// items hold 10 ints per block: parent, first slot, child cell of each of the
// sp slots of the group (-1 = absent); sp from m2l_up_slots / m2l_down_slots.
template <typename T>
int m2l_up_slots(int P);
template <typename T>
int m2l_down_slots(int P);
template <typename T>
cudaError_t launch_m2l_up(const double* q_equiv, const int* items, int nitems, const int* surf_ijk,
                          const double* twiddle, int P, int ns, int nsrc, int sp, T* Q, cudaStream_t st);
cudaError_t launch_m2l_hadamard8(const float* Q, const float* G, const int* tsrcT /*[26][ntar]*/, int ntar, int nsrc,
                                 int Nf, float* Pk, cudaStream_t st);
cudaError_t launch_m2l_hadamard8(const double* Q, const double* G, const int* tsrcT, int ntar, int nsrc, int Nf,
                                 double* Pk, cudaStream_t st);
// G (frequency-major, the layout of that precision's Hadamard, g8_layout_size
// values) from cc8 [d][pair][f] (device)
size_t g8_layout_size(int Nf, bool fp32);
cudaError_t launch_g8_layout(const double* cc8, int Nf, float* G, cudaStream_t st);
cudaError_t launch_g8_layout(const double* cc8, int Nf, double* G, cudaStream_t st);
cudaError_t launch_m2l_hadamard27(const double* Q, const double* G27 /*[d][f]*/, const int* tsrc /*[ntar][26]*/,
                                  int ntar, int nsrc, int Nf, double* Pk, cudaStream_t st);
template <typename T>
cudaError_t launch_m2l_down(const T* Pk, const int* items, const double* tscale, int nitems,
                            const int* surf_ijk, const double* twiddle, int P, int ns, int ntar, int sp,
                            double* p_check, cudaStream_t st);
cudaError_t launch_l2p_eval(const double4* body64, const LeafInfo* leaves, int nleaf,
                            const double* surf_unit, int ns, const double* q_down, double* phi,
                            double* grad, cudaStream_t st, bool full = true);
// sums of q x, q y, q z and q into partial[4 * kDipoleBlocks + 0..3]; partial
// holds kDipoleScratch doubles (per-block sums, then the totals)
constexpr int kDipoleBlocks = 256;
constexpr int kDipoleScratch = 4 * kDipoleBlocks + 4;
cudaError_t launch_dipole(const double4* body64, int n, double* partial, cudaStream_t st);
// adjoint: weights into the tree-order bodies (charges kept in qsave), the
// charges back, and dL/dx = w grad(phi_q) + q grad(psi_w) in input order
cudaError_t launch_swap_charges(double4* body64, const double* w, const int64_t* perm, int n, double* qsave,
                                cudaStream_t st);
cudaError_t launch_restore_charges(double4* body64, const double* qsave, int n, cudaStream_t st);
// new charges (input order) into bodies whose positions are on the device
cudaError_t launch_set_charges(double4* body64, const double* q, const int64_t* perm, int n, cudaStream_t st);
cudaError_t launch_adj_combine(const int64_t* perm, const double* w, const double* qsave, const double* grad_q,
                               const double* grad_w, int n, double* dLdx, cudaStream_t st);
// a sharded pass's exchange: leaf rows of v (nrow rows, stride ns) into a
// leaf-ordered buffer (scatter = false; rows of leaves with own[l] == 0 are
// zero, own null keeps all) or back (scatter = true)
cudaError_t launch_leaf_rows(double* v, int nrow, const int* cells, const char* own, int nleaf, int ns,
                             double* buf, bool scatter, cudaStream_t st);
// dipole: 0 none, 1 the reference's per-body form, 2 the surface term's
// potential; centre: the box centre (3), the dipole's origin
cudaError_t launch_post(const double* phi_far, const double* grad_far, const double* phi_near,
                        const double* grad_near, const double4* body64, const int64_t* perm, int n,
                        const double* dipole_partial, double coef, int dipole, const double* centre,
                        double out_scale, double* out_phi, double* out_grad, cudaStream_t st);
cudaError_t launch_gather_bodies(const double* x_in, const double* q_in, const int64_t* perm, int n,
                                 double4* body64, cudaStream_t st);

}  // namespace rtfmm_b200
