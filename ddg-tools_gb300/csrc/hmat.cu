// Hierarchical (block cluster tree) products on the GPU: the Hs metric B~ + B~0 over face
// pairs (FaceMetricTree, RS/src/metric/hierarchical.rs:279-812) and the vertex-pair fractional
// operator L^V_{2-s} of the preconditioner (VertexFractionalTree, hierarchical.rs:998-1346),
// behind rs_metric_* / rs_vfrac_* of include/rsgpu.h.
//
// Both are kernel-matrix forms L u = 2 M^T diag(a) (diag(H~a) M u - H~(a M u)) with a block
// cluster tree H~: rank-one far blocks (cluster data) and exact near blocks, whose FP32 weights are
// evaluated once per set-up and streamed by every product.
//
// Per product (C channels per element: 9 gradient + 3 average per input vector for faces, 3
// per vector for vertices):
//   prologue    m = M x per element (float pairs and FP64), element-major [n][C], a plane per vector
//   upward      up[node] = sum_{q in node} a_q m_q, bottom-up over groups of nodes
//   far         fpart[item] = sum_b h(node, b) up[b] over slices of a node's far blocks
//   chain       per leaf the far sums of its root-to-leaf chain
//   rows        near sums of every work item (beside the three far passes, on another stream)
//   epilogue    z = near + (m_p H~a_far - H~(a m)_far) per element; y = 2 M^T diag(a) W z (faces:
//               per-vertex gather; vertices: y = 2 a z)
// H~a is formed with the same operations as H~(a m) for m = 1, so L 1 = 0 exactly (the
// reference's null-space property, hierarchical.rs:13-16).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "block_tree.hpp"
#include "common.hpp"
#include "f32x2.cuh"
#include "fp64_bits.cuh"
#include "host_tree.hpp"
#include "hmat.hpp"
#include "profile.hpp"

namespace rsg {

constexpr int FACE = 0, VERTEX = 1;
// Which of the two kernels a channel uses: FACE_CH (12 channels per vector, the last three of
// them the averages, kernel 1), VERTEX_CH (4 per vector, the last one padding; kernel 0
// throughout), ONES (channel c uses kernel c: the two-channel pass that forms the far part of
// H~a from m = 1).
constexpr int FACE_CH = 0, VERTEX_CH = 1, ONES = 2;
template <int SEL>
constexpr int kChannels = SEL == FACE_CH ? 12 : (SEL == VERTEX_CH ? 4 : 2);
template <int SEL>
__device__ __forceinline__ bool uses_k1(int c) {
  return SEL == FACE_CH ? c >= 9 : (SEL == ONES ? c == 1 : false);
}

struct HDev {
  const uint32_t *start, *end, *right, *parent, *leaves, *chain_off, *chain;
  const uint32_t *far_ptr, *far_col;
  const uint4 *far_items;       // per far work item: node, block range [y, z) (at most kFarChunk), -
  const uint32_t *far_item_off; // per node: its far items [far_item_off[a], far_item_off[a + 1])
  float2 *fpart;                // per far item: C channel partial sums (float pairs)
  const float4 *far_coef;    // per far block: (k_0, k_1) as float pairs (k_0 hi, k_0 lo, k_1 hi, k_1 lo)
  const float4 *xh;          // per BVH position: position hi (xyz), weight a (w)
  const float4 *xl;          // per BVH position: position lo (xyz): X = hi + lo to ~48 bits
  const float4 *nrm;         // per BVH position: normal (faces only)
  const uint32_t *leaf_of;   // per BVH position: its leaf ordinal
  const uint4 *grp;          // bottom groups of nodes: root, number of nodes, first leaf ordinal, leaves
  const uint32_t *grp_depth; // and the number of the root's ancestors
  const double2 *leaf_farA;  // per leaf: far sums of psi = a (k_0, k_1) along its chain, the far part of H~a
  double *leafsum;           // per leaf: C channel far sums along its chain
  const uint32_t *colidx;    // near columns of every leaf's chain, flattened, leaf by leaf
  const uint4 *items;        // per work item: leaf ordinal, column-range begin / end, weight base (in 8 float2)
  const float2 *wts;         // near weights per item: [kernel][row pair][column], see hm_weights_kernel
  const uint32_t *item_off;  // per leaf: its work items [item_off[k], item_off[k + 1])
  const uint32_t *sched;     // work items by the leaf's rows, then most columns first
  uint32_t sched_off[9];     // those of leaves of i rows: [sched_off[i - 1], sched_off[i])
  double *up;                // per node: C channel sums of a m (FP64; of group roots only)
  float2 *up2;               // per node: the same sums as float pairs (hi, lo), read by the far sums
  float2 *part;              // per work item: 8 rows x C near sums as float pairs
  const float *m;            // channel values as float pairs: [n] records of C hi, then C lo parts
  double *z;                 // [n][C]: the channel values in FP64 (hi + lo), then the results in place
  // (the buffers with C channels hold one such plane per vector, vector by vector)
  int n_nodes, n_leaves, n_el, n_items, n_far_items, n_grp;
  float neg_s;               // kernel exponent e applied to r^2: r2^e
  int pw_mode, pw_k;         // e = pw_k / pw_mode for pw_mode 2 or 3 (exact roots), else powf
};

// Error-free sum (Knuth): a + b = s + t exactly.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &t) {
  s = a + b;
  const float bv = s - a;
  t = (a - (s - bv)) + (b - bv);
}


// v as a float pair: hi = v rounded to FP32, lo = the rest rounded
__device__ __forceinline__ float2 to_pair(double v) {
  const float h = (float)v;
  return make_float2(h, (float)(v - f2d(h)));
}

// (h, l) += (oh, ol) for float pairs.
__device__ __forceinline__ void pair_add(float &h, float &l, float oh, float ol) {
  float s, t;
  two_sum(h, oh, s, t);
  h = s;
  l = (l + ol) + t;
}

__device__ __forceinline__ float ipow(float x, int n) {
  float r = 1.f;
  for (; n > 0; --n) r *= x;
  return r;
}

// r2^e. For e = k/3 or k/2 (the exponents of integer alpha, beta) the power is an integer
// power times a correctly rounded root: a few roundings, independent of the size of
// log r2 (exp2(e log2 r2) loses accuracy in proportion to it).
__device__ __forceinline__ float r2pow(const HDev &d, float r2, float ir2) {
  if (d.pw_mode == 3 || d.pw_mode == 2) {
    const int q = d.pw_mode, k = d.pw_k;
    const int a = (k >= 0) ? k / q : -((-k + q - 1) / q);  // floor(k / q)
    const int b = k - q * a;                                // 0 .. q-1
    float base = a >= 0 ? ipow(r2, a) : ipow(ir2, -a);
    if (b) {
      const float root = q == 3 ? cbrtf(r2) : sqrtf(r2);
      base *= b == 1 ? root : root * root;
    }
    return base;
  }
  return powf(r2, d.neg_s);
}

// The near kernel values of an element pair (hierarchical.rs:185-189, 224-231 and 987-991):
// faces: [r2^-s, (nu_p^2 + nu_q^2)/2 r2^-2 r2^-s]; vertices: [r2^e].
template <int KIND>
__device__ __forceinline__ void near_kernel(const HDev &d, float d0, float d1, float d2,
                                            const float4 &np, const float4 &nq, float &k0, float &k1) {
  const float r2 = d0 * d0 + d1 * d1 + d2 * d2;
  const float ir2 = __frcp_rn(r2);
  const float h = r2pow(d, r2, ir2);
  k0 = h;
  if (KIND == FACE) {
    const float a = np.x * d0 + np.y * d1 + np.z * d2;
    const float b = nq.x * d0 + nq.y * d1 + nq.z * d2;
    k1 = 0.5f * (a * a + b * b) * ir2 * ir2 * h;
  } else {
    k1 = h;
  }
}

// Bottom-up channel sums in FP64: up[node] = left + right, and for a leaf its elements added in
// order. (The far field's sums cancel against m_p H~a for a smooth input just as the near sums do.)
// The nodes are cut into bottom groups (a subtree of at most 16 leaves, a block each) and above
// them, level by level, groups of at most 128 roots of the level below, each again a block: the
// leaves of a group are summed side by side and its inner nodes in decreasing index (children
// before parents, the tree's indices being in preorder) from shared memory. Climbing from every leaf with an
// arrival counter per node took 0.125 ms at 204,800 faces: 26 levels of fence, atomic and load, and
// twelve of 32 lanes at FP64 work.
constexpr int kGrpLeaves = 16, kGrpNodes = 2 * kGrpLeaves - 1, kGrpExt = 128;

template <int SEL>
__global__ void __launch_bounds__(192) hm_upward_kernel(HDev d) {
  constexpr int CC = kChannels<SEL>;
  __shared__ double sh[kGrpNodes * CC];
  __shared__ uint32_t rt[kGrpNodes];
  const uint4 gr = d.grp[blockIdx.x];
  const size_t pn = blockIdx.y * (size_t)d.n_nodes;
  if (threadIdx.x < gr.y) rt[threadIdx.x] = d.right[gr.x + threadIdx.x];
  for (uint32_t t = threadIdx.x; t < gr.w * CC; t += blockDim.x) {
    const uint32_t l = t / CC, c = t - l * CC, leaf = d.leaves[gr.z + l], p0 = d.start[leaf], n = d.end[leaf] - p0;
    const double *z = d.z + (blockIdx.y * (size_t)d.n_el + p0) * CC + c;
    double v[8], a[8], u = 0.0;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
      v[i] = i < n ? (SEL == ONES ? 1.0 : z[i * CC]) : 0.0;
      a[i] = i < n ? f2d(d.xh[p0 + i].w) : 0.0;
    }
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
      if (i < n) u = fma(a[i], v[i], u);
    sh[(leaf - gr.x) * CC + c] = u;
  }
  __syncthreads();
  if (threadIdx.x < CC) {
    const uint32_t c = threadIdx.x;
    for (int i = (int)gr.y - 1; i >= 0; --i)
      if (rt[i]) sh[i * CC + c] = sh[(i + 1) * CC + c] + sh[(rt[i] - gr.x) * CC + c];
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < gr.y * CC; t += blockDim.x) d.up2[(pn + gr.x) * CC + t] = to_pair(sh[t]);
  if (threadIdx.x < CC) d.up[(pn + gr.x) * CC + threadIdx.x] = sh[threadIdx.x];
}

// One level above: group = (first of its roots of the level below in ext, their number, first of
// its inner nodes in inner, their number); inner nodes in decreasing index with the slots of
// their children (roots first, then the inner nodes in order).
template <int CC>
__global__ void __launch_bounds__(128) hm_upward_level_kernel(HDev d, const uint4 *__restrict__ groups,
                                                              const uint32_t *__restrict__ ext,
                                                              const uint32_t *__restrict__ inner,
                                                              const uint2 *__restrict__ child) {
  __shared__ double sh[(2 * kGrpExt - 1) * CC];
  __shared__ uint2 ch[kGrpExt];
  const uint4 gr = groups[blockIdx.x];
  const size_t pn = blockIdx.y * (size_t)d.n_nodes;
  for (uint32_t i = threadIdx.x; i < gr.w; i += blockDim.x) ch[i] = child[gr.z + i];
  for (uint32_t t = threadIdx.x; t < gr.y * CC; t += blockDim.x)
    sh[t] = d.up[(pn + ext[gr.x + t / CC]) * CC + t % CC];
  __syncthreads();
  if (threadIdx.x < CC)
    for (uint32_t i = 0; i < gr.w; ++i)
      sh[(gr.y + i) * CC + threadIdx.x] = sh[ch[i].x * CC + threadIdx.x] + sh[ch[i].y * CC + threadIdx.x];
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < gr.w * CC; t += blockDim.x) {
    const size_t o = (pn + inner[gr.z + t / CC]) * CC + t % CC;
    const double v = sh[gr.y * CC + t];
    d.up2[o] = to_pair(v);
    if (t / CC + 1 == gr.w) d.up[o] = v;  // the group's root
  }
}

constexpr uint32_t kFarChunk = 64;  // far blocks per far work item

// fpart[item][c] = sum over the item's far blocks (a, b) of h(a, b)[kernel(c)] up[b][c]
// (block_tree.rs:564-578) in double-float arithmetic: the coefficients and the node sums are float
// pairs (about 48 bits), each product is formed exactly to that width (FMA) and added by error-free
// transformations. GB300 issues FP32 at many times its FP64 rate. One warp per item, all vectors:
// lane = sub C + c holds channel c and takes the item's far blocks sub, sub + 2, ... (sub = 0, 1);
// the two partial sums are then added. The item's columns and coefficients come in first, coalesced,
// so that the gathers of the node sums are independent of one another. The operations do not
// depend on the channel count, so the pass over psi = a (two channels) and a product pass add the
// same terms in the same order.
__device__ __forceinline__ void df_fma(float &ah, float &al, float kh, float kl, float uh, float ul) {
  const float ph = kh * uh;
  float pe = fmaf(kh, uh, -ph);
  pe = fmaf(kh, ul, pe);
  pe = fmaf(kl, uh, pe);
  float sh, se;
  two_sum(ah, ph, sh, se);
  se += al + pe;
  ah = sh + se;
  al = se - (ah - sh);
}

template <int SEL>
__global__ void __launch_bounds__(256) hm_far_kernel(HDev d, int nb) {
  constexpr int CC = kChannels<SEL>;
  static_assert(2 * CC <= 32, "two blocks at a time");
  __shared__ float4 coef[8][kFarChunk];
  __shared__ uint32_t col[8][kFarChunk];
  const int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), wib = threadIdx.x >> 5;
  if (w >= d.n_far_items) return;
  const uint4 it = d.far_items[w];
  const int lane = threadIdx.x & 31, sub = lane / CC, ch = lane - sub * CC;
  const uint32_t n = it.z - it.y;
#pragma unroll
  for (uint32_t i = lane; i < kFarChunk; i += 32)
    if (i < n) coef[wib][i] = __ldg(d.far_coef + it.y + i), col[wib][i] = __ldg(d.far_col + it.y + i) * CC;
  __syncwarp();
  const float2 *kp = reinterpret_cast<const float2 *>(&coef[wib][0]) + (uses_k1<SEL>(ch) ? 1 : 0);
  for (int q = 0; q < nb; ++q) {
    const float2 *__restrict__ up2 = d.up2 + q * (size_t)d.n_nodes * CC + ch;
    float ah = 0.f, al = 0.f;
    if (sub < 2) {
      uint32_t b = sub;
      for (; b + 14 < n; b += 16) {
        float2 u[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) u[i] = __ldg(up2 + col[wib][b + 2 * i]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 k = kp[2 * (b + 2 * i)];
          df_fma(ah, al, k.x, k.y, u[i].x, u[i].y);
        }
      }
      float2 u[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) u[i] = b + 2 * i < n ? __ldg(up2 + col[wib][b + 2 * i]) : make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (b + 2 * i < n) {
          const float2 k = kp[2 * (b + 2 * i)];
          df_fma(ah, al, k.x, k.y, u[i].x, u[i].y);
        }
    }
    const float oh = __shfl_down_sync(0xffffffffu, ah, CC), ol = __shfl_down_sync(0xffffffffu, al, CC);
    pair_add(ah, al, oh, ol);
    if (sub == 0) d.fpart[(q * (size_t)d.n_far_items + w) * CC + ch] = make_float2(ah, al);
  }
}

// The far sums of a node: its item partials added in item order as float pairs, in FP64 (zero for
// a node without far blocks).
template <int CC>
__device__ __forceinline__ double far_of_node(const HDev &d, const float2 *__restrict__ fp, uint32_t a, int c) {
  float h = 0.f, l = 0.f;
  for (uint32_t i = d.far_item_off[a]; i < d.far_item_off[a + 1]; ++i) {
    const float2 v = fp[(size_t)i * CC + c];
    pair_add(h, l, v.x, v.y);
  }
  return f2d(h) + f2d(l);
}

// Per (leaf, channel): the far sums along the leaf's chain, from the root down in FP64, shared by the
// leaf's rows. A block per bottom group: the sums of the root's ancestors, then down the group's
// nodes in preorder, a node's sum being its parent's plus its own: each node is added once and
// not once per leaf below it. With psi = a (ONES) the same sums give the far part of H~a.
template <int SEL>
__global__ void __launch_bounds__(192) hm_chain_sum_kernel(HDev d, double *__restrict__ dst) {
  constexpr int CC = kChannels<SEL>, kAnc = 32;
  __shared__ double sh[kGrpNodes * CC], anc[kAnc * CC];
  __shared__ uint32_t par[kGrpNodes];
  const uint4 gr = d.grp[blockIdx.x];
  const uint32_t depth = d.grp_depth[blockIdx.x];
  const uint32_t *chain = d.chain + d.chain_off[gr.z];
  const float2 *fp = d.fpart + blockIdx.y * (size_t)d.n_far_items * CC;
  if (threadIdx.x < gr.y) par[threadIdx.x] = d.parent[gr.x + threadIdx.x] - gr.x;
  for (uint32_t t = threadIdx.x; t < gr.y * CC; t += blockDim.x) sh[t] = far_of_node<CC>(d, fp, gr.x + t / CC, t % CC);
  double s = 0.0;
  for (uint32_t a0 = 0; a0 < depth; a0 += kAnc) {
    const uint32_t na = min((uint32_t)kAnc, depth - a0);
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < na * CC; t += blockDim.x) anc[t] = far_of_node<CC>(d, fp, chain[a0 + t / CC], t % CC);
    __syncthreads();
    if (threadIdx.x < CC)
      for (uint32_t i = 0; i < na; ++i) s += anc[i * CC + threadIdx.x];
  }
  __syncthreads();
  if (threadIdx.x < CC) {
    sh[threadIdx.x] = s + sh[threadIdx.x];
    for (uint32_t i = 1; i < gr.y; ++i) sh[i * CC + threadIdx.x] = sh[par[i] * CC + threadIdx.x] + sh[i * CC + threadIdx.x];
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < gr.w * CC; t += blockDim.x) {
    const uint32_t k = gr.z + t / CC;
    dst[(blockIdx.y * (size_t)d.n_leaves + k) * CC + t % CC] = sh[(d.leaves[k] - gr.x) * CC + t % CC];
  }
}

// Far coefficients (k_0, k_1) of every far block, FP64, as float pairs (hi, lo): d the centroid
// difference of the pair (lower node index first), h = r2^e, and for faces
// k_1 = (q_lo(d) + q_hi(d)) / 2 / r2^2 h with q the node's area-weighted projector form
// (proj = null: vertices, k_1 = k_0). One warp per far work item, lanes over its blocks.
__global__ void hm_far_coef_kernel(const uint4 *__restrict__ items, int n_items, const uint32_t *__restrict__ far_col,
                                   const double *__restrict__ cen, const double *__restrict__ proj, double e,
                                   float4 *__restrict__ coef) {
  const int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= n_items) return;
  const uint4 it = items[w];
  const uint32_t a = it.x;
  auto qf = [&](uint32_t n, const double *d) {
    const double *p = proj + 6 * (size_t)n;
    return p[0] * d[0] * d[0] + p[3] * d[1] * d[1] + p[5] * d[2] * d[2] +
           2.0 * (p[1] * d[0] * d[1] + p[2] * d[0] * d[2] + p[4] * d[1] * d[2]);
  };
  for (uint32_t q = it.y + lane; q < it.z; q += 32) {
    const uint32_t b = far_col[q], lo = min(a, b), hi = max(a, b);
    const double d[3] = {cen[3 * (size_t)lo] - cen[3 * (size_t)hi], cen[3 * (size_t)lo + 1] - cen[3 * (size_t)hi + 1],
                         cen[3 * (size_t)lo + 2] - cen[3 * (size_t)hi + 2]};
    const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    const double h = pow(r2, e);
    const double h1 = proj ? 0.5 * (qf(lo, d) + qf(hi, d)) / (r2 * r2) * h : h;
    const float2 k0 = to_pair(h), k1 = to_pair(h1);
    coef[q] = make_float4(k0.x, k0.y, k1.x, k1.y);
  }
}

// How a warp takes work items of the near field (slices of a leaf's near columns): an item has
// LPI lanes (column residue j, row group rg, channel group cg), so that a warp takes 32 / LPI
// items side by side. For a leaf of NS rows the columns fall into G = 32 / NS residue classes,
// whose sums are kept apart and added in order at the end; lane (j, rg, cg) takes the columns
// j, j + G, ... for NPL of the leaf's NP = ceil(NS / 2) row pairs and CPL channels. The columns
// pass through shared memory in tiles of T (a multiple of G).
// The error-free sums are bound by the FP32 pipe: they take small tiles of registers (more warps);
// the plain sums by shared-memory reads: larger tiles, fewer bytes per product. Faces take one
// vector (NV = 1) per warp; vertices, whose vectors have three channels only, all of them.
template <int KIND, int NS, bool PLAIN, int NV>
struct NearLanes {
  static constexpr bool F = KIND == FACE;
  static constexpr int G = 32 / NS, NP = (NS + 1) / 2;
  static constexpr int CPL = !F ? 3 * NV : (NS == 1 ? 12 : NS == 2 ? 6 : NS == 3 ? 4 : NS == 6 ? (PLAIN ? 4 : 2) : 3);
  static constexpr int NCG = F ? 12 / CPL : 1;
  static constexpr int RG = !F ? NP : (NS >= 7 && !PLAIN ? 2 : 1), NPL = NP / RG;
  static constexpr int LPI = F && NS >= 6 && PLAIN ? 16 : 32;
  static constexpr int IPW = 32 / LPI;                 // items per warp
  static constexpr int T = NS == 1 ? 32 : NS == 3 ? 20 : NS == 5 ? 18
                         : NS == 6 ? (F && PLAIN ? 10 : 20) : F && NS >= 7 && PLAIN ? 8 : 16;  // columns of a tile
  static constexpr int K = F ? 2 : 1;                  // kernels
  // a tile in shared memory: the hi parts of the columns (C floats each), the lo parts, the weight
  // planes; the offsets keep the lanes of a load (and of a copy) on different banks
  static constexpr int C = F ? 12 : 4 * NV;
  static constexpr int LO = T * C + (20 - T * C % 32 + 32) % 32;
  static constexpr int W = LO + T * C;
  static constexpr int PLANE = NP * T * 2 + (K == 2 ? (16 - NP * T * 2 % 32 + 32) % 32 : 0);
  static constexpr int FLOATS = W + K * PLANE;
  static_assert(T % G == 0 && T % 2 == 0 && T <= 32 && G * RG * NCG <= LPI && NPL * RG == NP, "lane mapping");
};
constexpr int kNearStages = 3;  // tiles of a warp in shared memory: one in use, two in flight
template <int KIND, int NV>
constexpr int kStageFloats = KIND == FACE ? 960 : 256 * NV + 96;  // of all the items of a warp

// float2 weights of an item of ns rows and ncol columns, a multiple of 8
template <int KIND>
__host__ __device__ __forceinline__ uint32_t near_weights(uint32_t ns, uint32_t ncol) {
  return ((KIND == FACE ? 2u : 1u) * ((ns + 1) / 2) * ((ncol + 1) & ~1u) + 7u) & ~7u;
}

// Near weights of an element pair as the rows kernel applies them: faces (w_0, w_1) =
// a_q (k_0, k_1), vertices w_0 = a_q k_0; zero on the diagonal (q = p) and in the padding.
// Stored per work item as planes [kernel][row pair][column] of float2 (the weights of rows 2i
// and 2i + 1: a packed operand), columns padded to an even number.
template <int KIND>
__global__ void hm_weights_kernel(HDev d) {
  // one warp per (item, row); lanes strided over the item's columns
  const size_t wr = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wr >= (size_t)d.n_items * 8) return;
  const uint32_t w = (uint32_t)(wr >> 3), r = (uint32_t)(wr & 7);
  const uint4 it = d.items[w];
  const uint32_t leaf = d.leaves[it.x];
  const uint32_t s0 = d.start[leaf], ns = d.end[leaf] - s0, np2 = (ns + 1) / 2;
  if (r >= 2 * np2) return;  // the second row of the last pair may be padding
  const uint32_t p = s0 + min(r, ns - 1), ncol = it.z - it.y, npad = (ncol + 1) & ~1u;
  const float4 ph = d.xh[p], pl = d.xl[p];
  const float4 np = KIND == FACE ? d.nrm[p] : make_float4(0.f, 0.f, 0.f, 0.f);
  float *out = reinterpret_cast<float *>(const_cast<float2 *>(d.wts) + 8 * (size_t)it.w + (size_t)(r >> 1) * npad) + (r & 1);
  for (uint32_t k = lane; k < npad; k += 32) {
    float w0 = 0.f, w1 = 0.f;
    if (k < ncol) {
      const uint32_t q = d.colidx[it.y + k];
      if (q != p && r < ns) {
        const float4 qh = d.xh[q], ql = d.xl[q];
        const float d0 = (ph.x - qh.x) + (pl.x - ql.x);
        const float d1 = (ph.y - qh.y) + (pl.y - ql.y);
        const float d2 = (ph.z - qh.z) + (pl.z - ql.z);
        float k0, k1;
        near_kernel<KIND>(d, d0, d1, d2, np, KIND == FACE ? d.nrm[q] : np, k0, k1);
        w0 = k0 * qh.w, w1 = k1 * qh.w;
      }
    }
    out[2 * k] = w0;
    if (KIND == FACE) out[2 * ((size_t)np2 * npad + k)] = w1;
  }
}

// 16 bytes global -> shared, asynchronous, `bytes` (16 or 0) of them read and the rest zero
__device__ __forceinline__ void cp_async16(unsigned smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16_l2(unsigned smem, const void *gmem, unsigned bytes) {  // not kept in L1
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// N consecutive floats from shared memory (8- or 16-byte aligned when N is even or a multiple of 4)
template <int N>
__device__ __forceinline__ void lds_floats(const float *p, float (&v)[N]) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const float4 t = *reinterpret_cast<const float4 *>(p + i);
      v[i] = t.x, v[i + 1] = t.y, v[i + 2] = t.z, v[i + 3] = t.w;
    }
  } else if constexpr (N % 2 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const float2 t = *reinterpret_cast<const float2 *>(p + i);
      v[i] = t.x, v[i + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = p[i];
  }
}

// Near sums of one work item in difference form: sum_q w_pq (m_p - m_q) for the rows p of the
// leaf. m_p - m_q is formed exactly from the float pairs (their hi parts share a grid), each
// product w (m_p - m_q) is split exactly too, and the terms are summed as float pairs: the high
// parts by error-free additions (two_sum), whose errors gather with the low parts in a second
// float. (Kahan summation would leave an error of eps times each lane's partial sum, a
// first-order quantity.) The G residue classes of the columns are then added in order as float
// pairs. For a smooth input the terms are first-order quantities that cancel to a second-order
// result, and the output stage (M^T, a discrete divergence) cancels once more, so plain FP32
// sums of H~a m and H~(a m) would lose about four digits.
//
// A lane keeps its rows' values and sums in registers, so that a column's values are read from
// shared memory once for all the rows it is applied to (with a lane per row the reads of the
// column values, four wavefronts per 16 bytes of a warp, bounded the kernel). Packed operands
// run over row pairs, as the stored weights do. The tiles (column records gathered by index,
// contiguous weights) are copied by cp.async two tiles ahead.
template <int KIND, int NS, bool PLAIN, int NV>
__device__ __forceinline__ void rows_items(const HDev &d, float *st, uint32_t w, uint32_t nb) {
  using L = NearLanes<KIND, NS, PLAIN, NV>;
  constexpr int CC = KIND == FACE ? 12 : 4, CV = L::C, NP = L::NP, NPL = L::NPL, CPL = L::CPL, T = L::T, LPI = L::LPI, IPW = L::IPW;
  constexpr int F4 = CV / 2;  // 16-byte parts of a column record (of all its vectors)
  constexpr int CHM = (T * F4 + LPI - 1) / LPI, CHW = (L::K * NP * T / 2 + LPI - 1) / LPI;
  constexpr int SF = IPW == 1 ? kStageFloats<KIND, NV> : kStageFloats<KIND, NV> / IPW / 32 * 32 - 16;  // floats of an item's tile
  static_assert(L::FLOATS <= SF, "the tile fits");
  // warp w of the leaves of NS rows: items [IPW p, IPW p + IPW) of them in d.sched, vector q (of nb
  // passes); the vectors of an item in consecutive warps, so that its weights come from DRAM once
  const uint32_t p = w / nb, q = w - p * nb;
  const int wl = threadIdx.x & 31, sub = wl / LPI, lane = wl - sub * LPI;
  const uint32_t pos = d.sched_off[NS - 1] + p * IPW + sub;
  const bool have = pos < d.sched_off[NS];
  const uint32_t item = d.sched[have ? pos : d.sched_off[NS] - 1];
  const uint4 it = d.items[item];  // leaf ordinal, flat column range [y, z), weight base
  const uint32_t s0 = d.start[d.leaves[it.x]];
  const uint32_t ncol = it.z - it.y, npad = (ncol + 1) & ~1u;
  const uint32_t *ci = d.colidx + it.y;
  const float2 *wg = d.wts + 8 * (size_t)it.w;
  if (q == 0 && lane == 0 && have && ncol > 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(wg),
                 "r"(near_weights<KIND>(NS, ncol) * (uint32_t)sizeof(float2))
                 : "memory");
  const float *m = d.m + (size_t)q * d.n_el * (2 * CC);
  st += sub * SF;
  const bool act = lane < L::G * L::RG * L::NCG;
  const int la = act ? lane : 0, cg = la % L::NCG, rg = (la / L::NCG) % L::RG, j = la / (L::NCG * L::RG);
  f32x2 mh[NPL][CPL], ml[NPL][CPL], ks[NPL][CPL], kc[NPL][CPL];
  const size_t plane = (size_t)d.n_el * (2 * CC);  // from vector to vector (vertices)
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int r0 = 2 * (rg * NPL + i), r1 = min(r0 + 1, NS - 1);
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const float *u = m + (size_t)(s0 + r0) * (2 * CC) + (KIND == FACE ? cg * CPL + c : c / 3 * plane + c % 3);
      const float *v = m + (size_t)(s0 + r1) * (2 * CC) + (KIND == FACE ? cg * CPL + c : c / 3 * plane + c % 3);
      mh[i][c] = f2_pack(u[0], v[0]), ml[i][c] = f2_pack(u[CC], v[CC]);
      ks[i][c] = kc[i][c] = 0ull;
    }
  }
  // tiles of the item, and of the longest item of the warp (the others add zero-weight columns)
  const uint32_t nt = (ncol + T - 1) / T;
  uint32_t ntw = nt;
#pragma unroll
  for (int o = LPI; o < 32; o <<= 1) ntw = max(ntw, __shfl_xor_sync(0xffffffffu, ntw, o));
  // the columns of tile t by lane (past the end the last column, with zero weights)
  auto index = [&](uint32_t t) { return ncol > 0 ? __ldg(ci + min(t * T + lane, ncol - 1)) : s0; };
  auto stage = [&](uint32_t t, uint32_t x) {
    if (t < ntw) {
      float *sg = st + (t % kNearStages) * kStageFloats<KIND, NV>;
      const unsigned sm = (unsigned)__cvta_generic_to_shared(sg), sw = sm + 4 * L::W;
#pragma unroll
      for (int i = 0; i < CHM; ++i) {
        const int c = lane + LPI * i, col = c / F4, part4 = c - col * F4;
        const uint32_t qc = __shfl_sync(0xffffffffu, x, col, LPI);
        if (T * F4 % LPI == 0 || c < T * F4)
          // faces: three parts of hi, three of lo; vertices: (hi, lo) of every vector
          if constexpr (KIND == FACE)
            cp_async16(sm + 4 * (col * CV + 4 * part4 + (part4 >= 3 ? L::LO - CV : 0)), m + (size_t)qc * 24 + 4 * part4);
          else
            cp_async16(sm + 4 * (col * CV + 4 * (part4 >> 1) + (part4 & 1 ? L::LO : 0)),
                       m + (part4 >> 1) * plane + (size_t)qc * 8 + 4 * (part4 & 1));
      }
#pragma unroll
      for (int i = 0; i < CHW; ++i) {
        const int c = lane + LPI * i, row = c / (T / 2);
        const uint32_t k = t * T + 2 * (c - row * (T / 2));
        if (L::K * NP * T / 2 % LPI == 0 || c < L::K * NP * T / 2)
          cp_async16_l2(sw + 16 * c + (L::K == 2 && row >= NP ? 4 * (L::PLANE - NP * T * 2) : 0), wg + (k < npad ? (size_t)row * npad + k : 0), k < npad ? 16u : 0u);
      }
    }
    cp_async_commit();  // one group per tile, empty past the end
  };
#pragma unroll
  for (int t = 0; t < kNearStages - 1; ++t) stage(t, index(t));
  uint32_t qn = index(kNearStages - 1);
  // the planes of the first and of the last channel of the lane: channels below kTh use the first
  constexpr int kTh = KIND == VERTEX ? CPL : CPL == 12 ? 9 : CPL == 6 ? 3 : CPL == 3 ? 3 : 1;
  const int wa = rg * NPL * T + (KIND == FACE && cg * CPL >= 9 ? L::PLANE / 2 : 0);
  const int wb = rg * NPL * T + (KIND == FACE && cg * CPL + CPL > 9 ? L::PLANE / 2 : 0);
  for (uint32_t t = 0; t < ntw; ++t) {
    cp_async_wait<kNearStages - 2>();
    __syncwarp();  // tile t is there for every lane, tile t - 1 done with by every lane
    stage(t + kNearStages - 1, qn);
    qn = index(t + kNearStages);
    const float *sg = st + (t % kNearStages) * kStageFloats<KIND, NV>;
    const f32x2 *sw = reinterpret_cast<const f32x2 *>(sg + L::W);
#pragma unroll 2
    for (int k0 = 0; k0 < T; k0 += L::G) {
      const int k = k0 + j;
      constexpr int CR = KIND == FACE ? CPL : CV;
      float vh[CR], vl[CR];
      lds_floats<CR>(sg + k * CV + cg * CPL, vh);
      lds_floats<CR>(sg + L::LO + k * CV + cg * CPL, vl);
      f32x2 qh[CPL], ql[CPL];
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        const int x = KIND == FACE ? c : c / 3 * 4 + c % 3;
        qh[c] = f2_pack(vh[x], vh[x]), ql[c] = f2_pack(vl[x], vl[x]);
      }
#pragma unroll
      for (int i = 0; i < NPL; ++i) {
        const f32x2 w0 = sw[wa + i * T + k], w1 = kTh >= CPL ? w0 : sw[wb + i * T + k];
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          const f32x2 w = c < kTh ? w0 : w1;
          // dh = mh_p - mh_q is exact (the hi parts share a grid)
          const f32x2 dh = f2_sub(mh[i][c], qh[c]), dl = f2_sub(ml[i][c], ql[c]);
          if constexpr (PLAIN) {
            // the inner operator: w (m_p - m_q) from the same exact differences, summed in plain
            // FP32 (no error-free transformations)
            ks[i][c] = f2_fma(w, f2_add(dh, dl), ks[i][c]);
            continue;
          }
          // w (m_p - m_q) = pr + pe + w dl up to eps^2 terms: w dh = pr + pe (FMA), so no
          // rounding that depends on the input reaches the sum above eps^2. npr = -pr (exact);
          // the error-free sum ks + pr = s + err: bb = s - ks, err = (ks - (s - bb)) + (pr - bb).
          const f32x2 npr = f2_mul(w ^ kF2Sign, dh);
          const f32x2 lo = f2_fma(w, dl, f2_fma(w, dh, npr));
          const f32x2 sn = f2_sub(ks[i][c], npr);
          const f32x2 bb = f2_sub(sn, ks[i][c]);
          const f32x2 err = f2_sub(f2_sub(ks[i][c], f2_sub(sn, bb)), f2_add(npr, bb));
          ks[i][c] = sn;
          kc[i][c] = f2_add(kc[i][c], f2_add(err, lo));
        }
      }
    }
  }
  // the G residue classes of a row added in order as float pairs, through shared memory
  constexpr int CO = KIND == FACE ? 12 : 3 * NV;  // channels written
  static_assert(L::G * NS * CO * 2 * IPW <= kNearStages * kStageFloats<KIND, NV>, "the sums fit the warp's tiles");
  cp_async_wait<0>();
  __syncwarp();
  float2 *red = reinterpret_cast<float2 *>(st - sub * SF) + sub * (L::G * NS * CO);
  if (act)
#pragma unroll
    for (int i = 0; i < NPL; ++i)
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        const int r = 2 * (rg * NPL + i), o = (j * NS + r) * CO + cg * CPL + c;
        const float2 s2 = f2_unpack(ks[i][c]), k2 = f2_unpack(kc[i][c]);
        red[o] = make_float2(s2.x, k2.x);
        if (r + 1 < NS) red[o + CO] = make_float2(s2.y, k2.y);
      }
  __syncwarp();
  float2 *part = d.part + ((size_t)q * d.n_items + item) * 8 * CC;
  if (have)
#pragma unroll 2
    for (int o = lane; o < NS * CO; o += LPI) {
      float2 v = red[o];
#pragma unroll
      for (int g = 1; g < L::G; ++g) {
        const float2 u = red[g * NS * CO + o];
        pair_add(v.x, v.y, u.x, u.y);
      }
      if constexpr (KIND == FACE) {
        part[o] = v;
      } else {
        const int r = o / CO, c = o - r * CO;
        part[(size_t)(c / 3) * d.n_items * 8 * CC + r * CC + c % 3] = v;
      }
    }
}

// Warps [warps[i + 1], warps[i]) take the items of the leaves of i rows (warps[9] = 0).
struct RowsGrid {
  uint32_t warps[10];
};
template <int KIND, bool PLAIN, int NV>
__global__ void __launch_bounds__(128, 4) hm_rows_kernel(HDev d, RowsGrid gr, uint32_t nb) {
  __shared__ __align__(16) float stages[4][kNearStages * kStageFloats<KIND, NV>];
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  float *st = stages[threadIdx.x >> 5];
  // longest first: the leaves of 8 rows have the lowest blocks
  if (w < gr.warps[8]) rows_items<KIND, 8, PLAIN, NV>(d, st, w, nb);
  else if (w < gr.warps[7]) rows_items<KIND, 7, PLAIN, NV>(d, st, w - gr.warps[8], nb);
  else if (w < gr.warps[6]) rows_items<KIND, 6, PLAIN, NV>(d, st, w - gr.warps[7], nb);
  else if (w < gr.warps[5]) rows_items<KIND, 5, PLAIN, NV>(d, st, w - gr.warps[6], nb);
  else if (w < gr.warps[4]) rows_items<KIND, 4, PLAIN, NV>(d, st, w - gr.warps[5], nb);
  else if (w < gr.warps[3]) rows_items<KIND, 3, PLAIN, NV>(d, st, w - gr.warps[4], nb);
  else if (w < gr.warps[2]) rows_items<KIND, 2, PLAIN, NV>(d, st, w - gr.warps[3], nb);
  else if (w < gr.warps[1]) rows_items<KIND, 1, PLAIN, NV>(d, st, w - gr.warps[2], nb);
}

// Per (element, channel): z = near + (m_p H~a_far - H~(a m)_far), the near sums of the leaf's
// items (in item order, as float pairs) plus the leaf's chain sums of the far field (FP64,
// hm_chain_sum_kernel), rounded to a float pair's 48 bits. The far part of H~a was summed with the
// same operations from psi = a, so m = 1 gives z = 0 exactly.
template <int SEL>
__global__ void hm_epilogue_kernel(HDev d) {
  constexpr int CC = kChannels<SEL>;
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const uint32_t p = (uint32_t)(t / CC);
  const int c = (int)(t - (size_t)p * CC);
  if (p >= (uint32_t)d.n_el) return;
  if (SEL == VERTEX_CH && c == 3) return;  // padding
  const uint32_t k = d.leaf_of[p], r = p - d.start[d.leaves[k]];
  double *z = d.z + (blockIdx.y * (size_t)d.n_el + p) * CC + c;
  const float2 *part = d.part + blockIdx.y * (size_t)d.n_items * 8 * CC;
  float nh = 0.f, nl = 0.f;
  for (uint32_t i = d.item_off[k]; i < d.item_off[k + 1]; ++i) {
    const float2 v = part[((size_t)i * 8 + r) * CC + c];
    pair_add(nh, nl, v.x, v.y);
  }
  const double2 fa = d.leaf_farA[k];
  const double far = *z * (uses_k1<SEL>(c) ? fa.y : fa.x) - d.leafsum[(blockIdx.y * (size_t)d.n_leaves + k) * CC + c];
  const double zz = (f2d(nh) + f2d(nl)) + far;
  const double zh = rn24(zz);
  *z = zh + rn24(zz - zh);
}

// leaf_of[p] = k for the elements p of leaf k
__global__ void leaf_of_kernel(uint32_t nl, const uint32_t *__restrict__ leaves, const uint32_t *__restrict__ start,
                               const uint32_t *__restrict__ end, uint32_t *leaf_of) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nl) return;
  for (uint32_t p = start[leaves[k]]; p < end[leaves[k]]; ++p) leaf_of[p] = k;
}

// ------------------------------------------------------------------ face prologue / epilogue

struct FaceOps {  // the faces in BVH order
  const uint32_t *faces;   // 3 per face
  // FP64 both: the gradient rows of a face sum to zero and the area-weighted rows around a
  // vertex sum to zero, and a smooth input leaves only what survives those cancellations
  const double *g;         // 9 per face: g_c (df_coefficients, mod.rs:120-131)
  const double *area;      // per face
  const uint32_t *inc_off, *inc;  // vertex -> (BVH position << 2 | corner), faces by ascending index
  int nv, nf;
};

// Channel values as float pairs on a common grid per channel: hi = k Q with Q = 2^(e - 22) for
// the channel's largest magnitude 2^e <= max < 2^(e+1), so |k| < 2^24 and the difference of two
// hi values is exact in FP32; lo = v - hi (|lo| <= Q / 2) rounded to FP32. The near field then
// forms m_p - m_q with two plain subtractions. Only the exponent of the largest magnitude
// matters: qmax holds, per channel, the largest high word (sign, exponent, leading mantissa
// bits) of |v| among the channel's values, shifted into the high half of a 64-bit word (the
// bit pattern of a non-negative double, ordered like the integers). Q is a power of two, so
// v / Q is the exact product v 2^(22 - e).
__device__ __forceinline__ double pow2(int k) {  // 2^k, from the bits when it is a normal number
  return (k >= -1022 && k <= 1023) ? __longlong_as_double((long long)(k + 1023) << 52) : ldexp(1.0, k);
}
// The rounding to the grid is the addition of 1.5 2^52 Q and its subtraction (|v| < 2^51 Q), and
// the integer k stands in the low word of the sum.
__device__ __forceinline__ float2 split_q(double v, unsigned long long qbits) {
  const unsigned hw = (unsigned)(qbits >> 32);
  if (hw == 0u) return make_float2(0.f, 0.f);
  const int ef = (int)((hw >> 20) & 0x7ffu);
  if (ef - 923u < 200u) {  // 2^-100 <= max < 2^100: Q and k Q are normal FP32 numbers
    const int e = ef - 1023;
    const double c = __hiloint2double((int)(((unsigned)(e + 30 + 1023) << 20) | 0x80000u), 0);  // 1.5 2^52 Q
    const double t = v + c, hi = t - c;
    const float kq = (float)__double2loint(t) * __uint_as_float((unsigned)(e - 22 + 127) << 23);
    return make_float2(kq, (float)(v - hi));
  }
  const int e = ef ? ef - 1023 : ilogb(__longlong_as_double((long long)qbits));
  const double hi = rint(v * pow2(22 - e)) * pow2(e - 22);
  return make_float2((float)hi, (float)(v - hi));
}

// qmax[c] = the largest high word of |v[c]| over the threads of the block with `act`
// (every thread of the block takes part)
template <int C>
__device__ __forceinline__ void block_max(const double (&v)[C], bool act, unsigned long long *qmax) {
  __shared__ unsigned sh[C][8];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const unsigned a = __reduce_max_sync(0xffffffffu, act ? (unsigned)__double2hiint(v[c]) & 0x7fffffffu : 0u);
    if ((threadIdx.x & 31) == 0) sh[c][threadIdx.x >> 5] = a;
  }
  __syncthreads();
  if (threadIdx.x < C) {
    unsigned a = 0u;
    for (unsigned w = 0; w < blockDim.x / 32; ++w) a = max(a, sh[threadIdx.x][w]);
    if (a != 0u) atomicMax(qmax + threadIdx.x, (unsigned long long)a << 32);
  }
}

// The channel values per face in BVH order (FaceMetricTree::product, hierarchical.rs:711-746), in
// FP64, and the channels' largest magnitudes; channels 3k + r = sum_c x[3 t_c + k] g_c[r]
// (gradient) and 9 + k = (x_0 + x_1 + x_2)/3 for axis k (average; the division by 3 is a product
// with the rounded 1/3, within an FP64 unit of the quotient, far below the float pairs'
// resolution). blockIdx.y is the vector.
__global__ void __launch_bounds__(256) face_m_kernel(FaceOps o, const double *__restrict__ xs, size_t ldx,
                                                     double *__restrict__ z, unsigned long long *qmax) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  const bool act = p < o.nf;
  const uint32_t *t = o.faces + 3 * (size_t)(act ? p : 0);
  const double *g = o.g + 9 * (size_t)(act ? p : 0);
  const double *x = xs + q * ldx;
  double v[12];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double x0 = x[3 * (size_t)t[0] + k], x1 = x[3 * (size_t)t[1] + k], x2 = x[3 * (size_t)t[2] + k];
#pragma unroll
    for (int r = 0; r < 3; ++r) v[3 * k + r] = x0 * g[r] + x1 * g[3 + r] + x2 * g[6 + r];
    v[9 + k] = ((x0 + x1) + x2) * (1.0 / 3.0);
  }
  block_max<12>(v, act, qmax + 12 * q);
  if (act) {
    double2 *zp = reinterpret_cast<double2 *>(z + ((size_t)q * o.nf + p) * 12);
#pragma unroll
    for (int i = 0; i < 6; ++i) zp[i] = make_double2(v[2 * i], v[2 * i + 1]);
  }
}

// The channel values split into float pairs: m, and in z their sum hi + lo in FP64 in
// place of the values; one thread per four channels of an element, blockIdx.y the vector.
template <int CC>
__global__ void split_m_kernel(size_t n_el, double *__restrict__ z, float *__restrict__ m,
                               const unsigned long long *__restrict__ qmax) {
  constexpr int NC = CC == 4 ? 3 : CC;  // channels that have a magnitude (the fourth of vertices is zero)
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t p = t / (CC / 4);
  const int c0 = 4 * (int)(t - p * (CC / 4));
  if (p >= n_el) return;
  double2 *zp = reinterpret_cast<double2 *>(z + (blockIdx.y * n_el + p) * CC + c0);
  const double2 a = zp[0], b = zp[1];
  const double v[4] = {a.x, a.y, b.x, b.y};
  float2 w[4];
  double s[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    w[i] = c0 + i < NC ? split_q(v[i], qmax[blockIdx.y * NC + c0 + i]) : make_float2(0.f, 0.f);
    s[i] = f2d(w[i].x) + f2d(w[i].y);
  }
  zp[0] = make_double2(s[0], s[1]), zp[1] = make_double2(s[2], s[3]);
  float *f = m + (blockIdx.y * n_el + p) * (2 * CC) + c0;
  *reinterpret_cast<float4 *>(f) = make_float4(w[0].x, w[1].x, w[2].x, w[3].x);
  *reinterpret_cast<float4 *>(f + CC) = make_float4(w[0].y, w[1].y, w[2].y, w[3].y);
}

// y_v = 2 sum_{S ni v} a_S (w_hi g_c . z_hi + w_lo z_lo / 3) in FP64 (hierarchical.rs:779-811), the
// multiply-adds written out so that every build rounds alike (a flow's solves magnify a last bit).
__global__ void face_gather_kernel(FaceOps o, const double *__restrict__ z, double w_hi, double w_lo,
                                   double *__restrict__ ys, size_t ldy) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= o.nv) return;
  const int q = blockIdx.y;
  double acc[3] = {0.0, 0.0, 0.0};
  const double wl = __dmul_rn(w_lo, 1.0 / 3.0);
  for (uint32_t e = o.inc_off[v]; e < o.inc_off[v + 1]; ++e) {
    uint32_t pc = o.inc[e], p = pc >> 2, c = pc & 3;
    double a = o.area[p];
    const double *g = o.g + 9 * (size_t)p + 3 * c;
    const double *zs = z + ((size_t)q * o.nf + p) * 12;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double *zh = zs + 3 * k;
      const double hi = __fma_rn(g[2], zh[2], __fma_rn(g[0], zh[0], __dmul_rn(g[1], zh[1])));
      acc[k] = __fma_rn(a, __fma_rn(w_hi, hi, __dmul_rn(wl, zs[9 + k])), acc[k]);
    }
  }
  double *y = ys + q * ldy + 3 * (size_t)v;
  y[0] = 2.0 * acc[0], y[1] = 2.0 * acc[1], y[2] = 2.0 * acc[2];
}

// ------------------------------------------------------------------ vertex prologue / epilogue

// Channels of the vertex operator: m = x per axis (psi = a x in the upward sums); blockIdx.y is
// the vector.
__global__ void __launch_bounds__(256) vertex_m_kernel(const uint32_t *order, const double *__restrict__ xs, size_t ldx,
                                                       int nv, double *__restrict__ z, unsigned long long *qmax) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  const bool act = p < nv;
  const uint32_t v = act ? order[p] : 0;
  double x[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) x[k] = xs[q * ldx + 3 * (size_t)v + k];
  block_max<3>(x, act, qmax + 3 * q);
  if (act) {
    double2 *zp = reinterpret_cast<double2 *>(z + ((size_t)q * nv + p) * 4);
    zp[0] = make_double2(x[0], x[1]), zp[1] = make_double2(x[2], 0.0);
  }
}

// y = 2 a (H~a x - H~(a x)) = 2 a z (hierarchical.rs:1330-1343).
__global__ void vertex_out_kernel(const uint32_t *order, const float4 *el, const double *z, int nv, double scale,
                                  double *__restrict__ ys, size_t ldy) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nv) return;
  const int q = blockIdx.y;
  uint32_t v = order[p];
  double a = el[p].w;
  for (int k = 0; k < 3; ++k) ys[q * ldy + 3 * (size_t)v + k] = scale * 2.0 * a * z[((size_t)q * nv + p) * 4 + k];
}

// Element records: positions as float pairs (hi + lo), weights, normals; FP64 in.
__global__ void hm_pack_kernel(const double *pts, const double *wt, const double *nrm64,
                               const uint32_t *order, int n, float4 *xh, float4 *xl, float4 *nrm) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  uint32_t e = order[p];
  const double *x = pts + 3 * (size_t)e;
  float h0 = (float)x[0], h1 = (float)x[1], h2 = (float)x[2];
  xh[p] = make_float4(h0, h1, h2, (float)wt[e]);
  xl[p] = make_float4((float)(x[0] - (double)h0), (float)(x[1] - (double)h1), (float)(x[2] - (double)h2), 0.f);
  if (nrm) nrm[p] = make_float4((float)nrm64[3 * (size_t)e], (float)nrm64[3 * (size_t)e + 1],
                                (float)nrm64[3 * (size_t)e + 2], 0.f);
}

// ---- the near columns and work items of every leaf, built on the device from the block lists

// per leaf k: the length of its root-to-leaf chain, the near columns of the chain's blocks and
// the number of work items (at most item_cols columns each, at least one)
__global__ void near_count_kernel(uint32_t nl, const uint32_t *__restrict__ leaves, const uint32_t *__restrict__ parent,
                                  const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
                                  const uint32_t *__restrict__ near_ptr, const uint32_t *__restrict__ near_col,
                                  uint32_t item_cols, uint32_t *depth, unsigned long long *cols, uint32_t *nitems) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nl) return;
  uint32_t dep = 1;
  unsigned long long c = 0;
  for (uint32_t a = leaves[k];; a = parent[a]) {
    for (uint32_t q = near_ptr[a]; q < near_ptr[a + 1]; ++q) {
      const uint32_t b = near_col[q];
      c += end[b] - start[b];
    }
    if (a == 0) break;
    ++dep;
  }
  depth[k] = dep, cols[k] = c;
  nitems[k] = (uint32_t)max(1ull, (c + item_cols - 1) / item_cols);
}

// per leaf k at its scanned offsets: the chain (root first), the near columns in chain, block and
// element order, and the work items (leaf, column range [y, z), weight base filled later)
__global__ void near_fill_kernel(uint32_t nl, const uint32_t *__restrict__ leaves, const uint32_t *__restrict__ parent,
                                 const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
                                 const uint32_t *__restrict__ near_ptr, const uint32_t *__restrict__ near_col,
                                 uint32_t item_cols, const uint32_t *__restrict__ coff,
                                 const unsigned long long *__restrict__ ncol, const uint32_t *__restrict__ ioff,
                                 uint32_t *chain, uint32_t *cols, uint4 *items) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nl) return;
  const uint32_t depth = coff[k + 1] - coff[k];
  uint32_t *ch = chain + coff[k];
  uint32_t a = leaves[k];
  for (uint32_t i = depth; i-- > 0; a = parent[a]) ch[i] = a;
  uint32_t x = (uint32_t)ncol[k];
  for (uint32_t i = 0; i < depth; ++i) {
    const uint32_t n = ch[i];
    for (uint32_t q = near_ptr[n]; q < near_ptr[n + 1]; ++q) {
      const uint32_t b = near_col[q];
      for (uint32_t e = start[b]; e < end[b]; ++e) cols[x++] = e;
    }
  }
  const uint32_t c_end = (uint32_t)ncol[k + 1];
  uint32_t y0 = (uint32_t)ncol[k];
  for (uint32_t it = ioff[k]; it < ioff[k + 1]; ++it) {
    const uint32_t y1 = min(c_end, y0 + item_cols);
    items[it] = make_uint4(k, y0, y1, 0u);
    y0 = y1;
  }
}

// the weight count of every work item, in blocks of 8 float2 (kernels x row pairs x padded columns),
// and the total of rows x columns padded to 32 (the size the near field is limited by)
template <int KIND>
__global__ void item_weights_kernel(uint32_t n_items, const uint4 *__restrict__ items, const uint32_t *__restrict__ leaves,
                                    const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
                                    unsigned long long *w, unsigned long long *total) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long entries = 0;
  if (i < n_items) {
    const uint4 it = items[i];
    const uint32_t leaf = leaves[it.x], ns = end[leaf] - start[leaf], ncol = it.z - it.y;
    w[i] = near_weights<KIND>(ns, ncol) / 8;
    entries = (unsigned long long)ns * ((ncol + 31) & ~31u);
  }
  for (int o = 16; o > 0; o >>= 1) entries += __shfl_down_sync(0xffffffffu, entries, o);
  if ((threadIdx.x & 31) == 0 && entries) atomicAdd(total, entries);
}
// sort key of every work item: the leaf's rows, then most columns first
__global__ void item_key_kernel(uint32_t n_items, const uint4 *__restrict__ items, const uint32_t *__restrict__ leaves,
                                const uint32_t *__restrict__ start, const uint32_t *__restrict__ end, uint32_t *key,
                                uint32_t *idx) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_items) return;
  const uint4 it = items[i];
  const uint32_t leaf = leaves[it.x];
  key[i] = ((end[leaf] - start[leaf]) << 16) | (0xffffu - (it.z - it.y));
  idx[i] = i;
}
// What the host needs of the work items: off[i] = the first of the sorted keys of more than i rows, i = 0 .. 8; the
// weights' blocks and the near entries.
struct ItemTotals {
  unsigned long long weights, entries;
  uint32_t off[9];
};
__global__ void item_totals_kernel(uint32_t n, const uint32_t *__restrict__ key, const unsigned long long *weights,
                                   const unsigned long long *entries, ItemTotals *out) {
  const uint32_t i = threadIdx.x;
  if (i == 9) out->weights = *weights, out->entries = *entries;
  if (i > 8) return;
  uint32_t a = 0, b = n;
  while (a < b) {
    const uint32_t c = (a + b) / 2;
    if (key[c] >> 16 > i) b = c;
    else a = c + 1;
  }
  out->off[i] = a;
}
__global__ void item_base_kernel(uint32_t n_items, const unsigned long long *__restrict__ base, uint4 *items) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_items) items[i].w = (uint32_t)base[i];
}

// far work items: node a's far blocks cut into runs of at most kFarChunk
__global__ void far_count_kernel(uint32_t nn, const uint32_t *__restrict__ far_ptr, uint32_t *cnt) {
  const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < nn) cnt[a] = (far_ptr[a + 1] - far_ptr[a] + kFarChunk - 1) / kFarChunk;
}
__global__ void far_fill_kernel(uint32_t nn, const uint32_t *__restrict__ far_ptr, const uint32_t *__restrict__ off,
                                uint4 *items) {
  const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nn) return;
  const uint32_t q1 = far_ptr[a + 1];
  uint32_t j = off[a];
  for (uint32_t q0 = far_ptr[a]; q0 < q1; q0 += kFarChunk) items[j++] = make_uint4(a, q0, min(q0 + kFarChunk, q1), 0u);
}

}  // namespace rsg

// ====================================================================== host side

using namespace rsg;

namespace {

inline unsigned nblk(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

template <class T>
void up_vec(DevBuf<T> &b, const std::vector<T> &v, cudaStream_t s) {
  b.alloc(std::max<size_t>(v.size(), 1));
  if (!v.empty()) b.upload(v.data(), v.size(), s);
}

// The block cluster tree on the device with its per-step data (both operators).
struct HMat {
  rs_ctx *ctx = nullptr;
  int kind = FACE;
  Tree tree;
  Blocks blocks;
  size_t n_el = 0, n_items = 0;
  double neg_s = 0;
  DevBuf<uint32_t> start, end, right, parent, leaves, chain_off, chain, item_off;
  DevBuf<uint32_t> far_item_off, leaf_of;
  // the groups of the upward sums: the bottom ones, and the levels above (see hm_upward_kernel); the bottom
  // ones' depths, then every level's ext, inner and child
  DevBuf<uint4> grp;
  DevBuf<uint32_t> grp_words;
  size_t n_bottom = 0;
  struct Level {
    size_t first, count;        // its groups
    size_t ext, inner, child;  // its lists, in words
  };
  std::vector<Level> levels;
  // the far passes run on the context's second stream beside the near field
  struct Event {
    cudaEvent_t e = nullptr;
    ~Event() {
      if (e) cudaEventDestroy(e);
    }
  } ev_fork, ev_join;
  DevBuf<uint4> far_items;
  size_t n_far_items = 0;
  DevBuf<float2> fpart;
  DevBuf<uint32_t> colidx;
  DevBuf<uint4> items;
  DevBuf<float2> wts;  // near weights, see hm_weights_kernel
  DevBuf<uint32_t> sched;  // the work items in the order of the near field, and its groups
  uint32_t sched_off[9] = {};
  size_t n_wts = 0;
  DevBuf<float4> far_coef;
  DevBuf<double2> leaf_farA;
  DevBuf<double> leafsum;
  DevBuf<float4> xh, xl, nrm;
  DevBuf<double> up, z;
  DevBuf<float2> up2;
  DevBuf<float2> part, m;  // m: channel values (2 C floats per element)
  DevBuf<unsigned long long> qmax;  // per channel: largest |m| (see split_q)
  int pw_mode = 0, pw_k = 0;
  bool plain_rows = false;  // the near field of the next product in plain FP32 sums (inner operator)
  Profiler prof;
  double setup_times[3] = {0, 0, 0};  // seconds: work items, far coefficients, device part

  HDev dev() const {
    HDev d;
    d.start = start.p, d.end = end.p, d.right = right.p, d.parent = parent.p, d.leaves = leaves.p;
    d.chain_off = chain_off.p, d.chain = chain.p;
    d.far_ptr = blocks.far_ptr.p, d.far_col = blocks.far_col.p, d.far_coef = far_coef.p;
    d.far_items = far_items.p, d.far_item_off = far_item_off.p, d.fpart = fpart.p;
    d.n_far_items = (int)n_far_items;
    d.xh = xh.p, d.xl = xl.p, d.nrm = nrm.p, d.leaf_farA = leaf_farA.p;
    d.colidx = colidx.p, d.items = items.p, d.item_off = item_off.p, d.wts = wts.p;
    d.sched = sched.p;
    std::copy(sched_off, sched_off + 9, d.sched_off);
    d.up = up.p, d.up2 = up2.p, d.part = part.p, d.leafsum = leafsum.p;
    d.leaf_of = leaf_of.p, d.grp = grp.p, d.grp_depth = grp_words.p, d.n_grp = (int)n_bottom;
    d.m = reinterpret_cast<const float *>(m.p), d.z = z.p;
    d.n_nodes = (int)tree.n_nodes(), d.n_leaves = (int)tree.leaves.size(), d.n_el = (int)n_el;
    d.n_items = (int)n_items;
    d.neg_s = (float)neg_s;
    d.pw_mode = pw_mode, d.pw_k = pw_k;
    return d;
  }
  cudaStream_t st() const { return ctx->stream; }

  // Channel scratch for C channels.
  void reserve(int C_) {
    size_t nn = tree.n_nodes();
    if ((size_t)C_ * nn > up.n) up.alloc((size_t)C_ * nn), up2.alloc((size_t)C_ * nn);
    if ((size_t)C_ * n_far_items > fpart.n) fpart.alloc(std::max<size_t>((size_t)C_ * n_far_items, 1));
    if ((size_t)C_ * tree.leaves.size() > leafsum.n) leafsum.alloc((size_t)C_ * tree.leaves.size());
    if ((size_t)C_ * n_el > m.n) m.alloc((size_t)C_ * n_el), z.alloc((size_t)C_ * n_el);
    if (n_items * 8 * (size_t)C_ > part.n) part.alloc(std::max<size_t>(n_items * 8 * (size_t)C_, 1));
  }

  // The exponent r2^e as an integer power times a cube or square root when 3e or 2e is an
  // integer (integer alpha, beta), else powf.
  void set_exponent(double e) {
    neg_s = e;
    pw_mode = 0, pw_k = 0;
    for (int q : {1, 2, 3}) {
      double k = e * q;
      if (std::fabs(k - std::round(k)) < 1e-12 && std::fabs(k) <= 64) {
        pw_mode = q == 1 ? 3 : q, pw_k = (int)std::round(k) * (q == 1 ? 3 : 1);
        break;
      }
    }
  }

  // the upward sums, the far sums and the chain sums (into dst) on stream s
  template <int SEL>
  void upward_far(const HDev &d, int nb, double *dst, cudaStream_t s) {
    constexpr int CC = kChannels<SEL>;
    const unsigned gy = (unsigned)nb;
    prof.begin(s, kind == FACE ? "metric_upward" : "vfrac_upward");
    hm_upward_kernel<SEL><<<dim3((unsigned)d.n_grp, gy), 192, 0, s>>>(d);
    RSG_LAUNCHED(ctx, "hm_upward");
    for (const Level &l : levels) {
      const uint32_t *w = grp_words.p;
      hm_upward_level_kernel<CC><<<dim3((unsigned)l.count, gy), 128, 0, s>>>(d, grp.p + l.first, w + l.ext, w + l.inner,
                                                                             reinterpret_cast<const uint2 *>(w + l.child));
      RSG_LAUNCHED(ctx, "hm_upward");
    }
    prof.end(s);
    prof.begin(s, kind == FACE ? "metric_far" : "vfrac_far");
    if (n_far_items > 0) {  // chi = 0 (all near) has none
      hm_far_kernel<SEL><<<nblk(n_far_items * 32, 256), 256, 0, s>>>(d, nb);
      RSG_LAUNCHED(ctx, "hm_far");
    }
    hm_chain_sum_kernel<SEL><<<dim3((unsigned)d.n_grp, gy), 192, 0, s>>>(d, dst);
    RSG_LAUNCHED(ctx, "hm_chain_sum");
    prof.end(s);
  }

  // The groups of the upward sums (see hm_upward_kernel), from the tree: g, the groups (bottom, then level by
  // level), and words, their depths and lists.
  void build_groups(std::vector<uint4> &g, std::vector<uint32_t> &words) {
    const Tree &T = tree;
    const size_t nn = T.n_nodes();
    std::vector<uint32_t> size(nn, 1);
    for (size_t i = nn; i-- > 0;)
      if (T.right[i]) size[i] = 1 + size[i + 1] + size[T.right[i]];
    // the nodes not yet inside a group in preorder, each with whether it is a root of one
    std::vector<std::pair<uint32_t, bool>> cur, next;
    std::vector<uint32_t> ends;  // ends of the subtrees of the current node's ancestors
    for (uint32_t n = 0, k = 0; n < nn;) {
      while (!ends.empty() && ends.back() <= n) ends.pop_back();
      if ((size[n] + 1) / 2 <= (uint32_t)kGrpLeaves) {
        const uint32_t nl = (size[n] + 1) / 2;
        g.push_back(make_uint4(n, size[n], k, nl));
        words.push_back((uint32_t)ends.size());
        cur.push_back({n, true});
        k += nl, n += size[n];
      } else {
        cur.push_back({n, false});
        ends.push_back(n + size[n]);
        ++n;
      }
    }
    n_bottom = g.size();
    levels.clear();
    while (cur.size() > 1) {
      const size_t m = cur.size();
      std::vector<uint32_t> roots(m + 1, 0);  // roots before each entry
      for (size_t i = 0; i < m; ++i) roots[i + 1] = roots[i] + (cur[i].second ? 1u : 0u);
      Level l;
      l.first = g.size();
      std::vector<uint32_t> ext, inner, child, slot(nn);
      next.clear();
      for (size_t i = 0; i < m;) {
        const uint32_t n = cur[i].first;
        const size_t j = (size_t)(std::lower_bound(cur.begin() + i, cur.end(), std::make_pair(n + size[n], false)) - cur.begin());
        if (cur[i].second || roots[j] - roots[i] > (uint32_t)kGrpExt) {
          next.push_back(cur[i++]);
          continue;
        }
        uint4 gr = make_uint4((uint32_t)ext.size(), 0, (uint32_t)inner.size(), 0);
        for (size_t a = i; a < j; ++a)
          if (cur[a].second) slot[cur[a].first] = gr.y++, ext.push_back(cur[a].first);
        for (size_t a = j; a-- > i;)
          if (!cur[a].second) {
            const uint32_t v = cur[a].first;
            inner.push_back(v);
            child.push_back(slot[v + 1]), child.push_back(slot[T.right[v]]);
            slot[v] = gr.y + gr.w++;
          }
        g.push_back(gr);
        next.push_back({n, true});
        i = j;
      }
      l.count = g.size() - l.first;
      auto add = [&](const std::vector<uint32_t> &v) {
        words.resize((words.size() + 1) & ~size_t(1));  // pairs lie on 8 bytes
        words.insert(words.end(), v.begin(), v.end());
        return words.size() - v.size();
      };
      l.ext = add(ext), l.inner = add(inner), l.child = add(child);
      levels.push_back(l);
      cur.swap(next);
    }
  }

  // Uploads the tree, the near column ranges split into work items, the element records and
  // the far coefficients; computes the far part of H~a. pts/wt/nrm64 are per element
  // (original order), FP64.
  void setup(const double *pts, const double *wt, const double *nrm64, const double *proj6) {
    using clk = std::chrono::steady_clock;
    auto t_ph = clk::now();
    auto lap = [&](double &slot) {
      const auto now = clk::now();
      slot = std::chrono::duration<double>(now - t_ph).count();
      t_ph = now;
    };
    cudaStream_t s = st();
    const Tree &T = tree;
    size_t nn = T.n_nodes(), nl = T.leaves.size();
    std::vector<uint32_t> parent_h(nn, 0);
    const uint32_t kItemCols = 512;
    for (size_t i = 0; i < nn; ++i)
      if (T.right[i]) parent_h[i + 1] = (uint32_t)i, parent_h[T.right[i]] = (uint32_t)i;
    for (size_t k = 0; k < nl; ++k)
      if (T.end[T.leaves[k]] - T.start[T.leaves[k]] > 8)
        fail(RS_INVALID_OPTION, "InvalidOption", "upload", "the GPU path needs leaf_size <= 8");
    up_vec(start, T.start, s), up_vec(end, T.end, s), up_vec(right, T.right, s);
    up_vec(parent, parent_h, s), up_vec(leaves, T.leaves, s);
    // per leaf: its root-to-leaf chain and the near columns of the chain (chain order, block
    // order, element order), flattened and cut into items of at most kItemCols columns: counts,
    // exclusive scans (one extra zero entry gives the totals), then the fill at the offsets
    DevBuf<unsigned char> tmp;
    auto scan = [&](auto *in, auto *out, size_t m) {
      size_t bytes = 0;
      RSG_CUDA("upload", cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, (int)m, s));
      if (bytes > tmp.n) tmp.alloc(bytes);
      RSG_CUDA("upload", cub::DeviceScan::ExclusiveSum(tmp.p, bytes, in, out, (int)m, s));
    };
    {
      DevBuf<uint32_t> dep(nl + 1), nit(nl + 1);
      DevBuf<unsigned long long> cnt(nl + 1), ncol(nl + 1);
      RSG_CUDA("upload", cudaMemsetAsync(dep.p + nl, 0, sizeof(uint32_t), s));
      RSG_CUDA("upload", cudaMemsetAsync(nit.p + nl, 0, sizeof(uint32_t), s));
      RSG_CUDA("upload", cudaMemsetAsync(cnt.p + nl, 0, sizeof(unsigned long long), s));
      near_count_kernel<<<nblk(nl, 128), 128, 0, s>>>((uint32_t)nl, leaves.p, parent.p, start.p, end.p,
                                                      blocks.near_ptr.p, blocks.near_col.p, kItemCols, dep.p, cnt.p,
                                                      nit.p);
      RSG_LAUNCHED(ctx, "hm_near_count");
      chain_off.alloc(nl + 1), item_off.alloc(nl + 1);
      scan(dep.p, chain_off.p, nl + 1), scan(cnt.p, ncol.p, nl + 1), scan(nit.p, item_off.p, nl + 1);
      uint32_t n_chain = 0, n_it = 0;
      unsigned long long n_col = 0;
      RSG_CUDA("upload", copy_async(&n_chain, chain_off.p + nl, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
      RSG_CUDA("upload", copy_async(&n_col, ncol.p + nl, sizeof(n_col), cudaMemcpyDeviceToHost, s));
      RSG_CUDA("upload", copy_async(&n_it, item_off.p + nl, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
      RSG_CUDA("upload", cudaStreamSynchronize(s));
      if (n_col > UINT32_MAX) fail(RS_INVALID_OPTION, "InvalidOption", "upload", "near field too large");
      chain.alloc(std::max<uint32_t>(n_chain, 1)), colidx.alloc(std::max<size_t>(n_col, 1)), items.alloc(n_it);
      near_fill_kernel<<<nblk(nl, 128), 128, 0, s>>>((uint32_t)nl, leaves.p, parent.p, start.p, end.p,
                                                     blocks.near_ptr.p, blocks.near_col.p, kItemCols, chain_off.p,
                                                     ncol.p, item_off.p, chain.p, colidx.p, items.p);
      RSG_LAUNCHED(ctx, "hm_near_fill");
      n_items = n_it;
    }
    lap(setup_times[0]);
    // weight base of every item
    {
      DevBuf<unsigned long long> w(n_items + 2), base(n_items + 1);  // w: zero past the items, then the entries
      unsigned long long *entries = w.p + n_items + 1;
      RSG_CUDA("upload", cudaMemsetAsync(w.p + n_items, 0, 2 * sizeof(unsigned long long), s));
      if (kind == FACE)
        item_weights_kernel<FACE><<<nblk(n_items, 256), 256, 0, s>>>((uint32_t)n_items, items.p, leaves.p, start.p,
                                                                     end.p, w.p, entries);
      else
        item_weights_kernel<VERTEX><<<nblk(n_items, 256), 256, 0, s>>>((uint32_t)n_items, items.p, leaves.p, start.p,
                                                                       end.p, w.p, entries);
      RSG_LAUNCHED(ctx, "hm_item_weights");
      scan(w.p, base.p, n_items + 1);
      DevBuf<uint32_t> sort(3 * n_items);  // keys, sorted keys, items
      uint32_t *key = sort.p, *sorted = key + n_items, *idx = sorted + n_items;
      item_key_kernel<<<nblk(n_items, 256), 256, 0, s>>>((uint32_t)n_items, items.p, leaves.p, start.p, end.p, key, idx);
      RSG_LAUNCHED(ctx, "hm_item_key");
      sched.alloc(n_items);
      size_t bytes = 0;
      RSG_CUDA("upload", cub::DeviceRadixSort::SortPairs(nullptr, bytes, key, sorted, idx, sched.p, (int)n_items, 0, 20, s));
      if (bytes > tmp.n) tmp.alloc(bytes);
      RSG_CUDA("upload", cub::DeviceRadixSort::SortPairs(tmp.p, bytes, key, sorted, idx, sched.p, (int)n_items, 0, 20, s));
      DevBuf<ItemTotals> totals(1);
      item_totals_kernel<<<1, 32, 0, s>>>((uint32_t)n_items, sorted, base.p + n_items, entries, totals.p);
      RSG_LAUNCHED(ctx, "hm_item_totals");
      ItemTotals t;
      totals.download(&t, 1, s);
      RSG_CUDA("upload", cudaStreamSynchronize(s));
      std::copy(t.off, t.off + 9, sched_off);
      const unsigned long long tot = t.weights;
      if (t.entries > UINT32_MAX || tot > UINT32_MAX)
        fail(RS_INVALID_OPTION, "InvalidOption", "upload", "near field too large");
      n_wts = 8 * (size_t)tot;
      item_base_kernel<<<nblk(n_items, 256), 256, 0, s>>>((uint32_t)n_items, base.p, items.p);
      RSG_LAUNCHED(ctx, "hm_item_weights");
    }
    // far work items
    {
      DevBuf<uint32_t> cnt(nn + 1);
      RSG_CUDA("upload", cudaMemsetAsync(cnt.p + nn, 0, sizeof(uint32_t), s));
      far_count_kernel<<<nblk(nn, 256), 256, 0, s>>>((uint32_t)nn, blocks.far_ptr.p, cnt.p);
      RSG_LAUNCHED(ctx, "hm_far_items");
      far_item_off.alloc(nn + 1);
      scan(cnt.p, far_item_off.p, nn + 1);
      uint32_t nfi = 0;
      RSG_CUDA("upload", copy_async(&nfi, far_item_off.p + nn, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
      RSG_CUDA("upload", cudaStreamSynchronize(s));
      n_far_items = nfi;
      far_items.alloc(std::max<size_t>(n_far_items, 1));
      far_fill_kernel<<<nblk(nn, 256), 256, 0, s>>>((uint32_t)nn, blocks.far_ptr.p, far_item_off.p, far_items.p);
      RSG_LAUNCHED(ctx, "hm_far_items");
    }
    leaf_of.alloc(n_el);
    leaf_of_kernel<<<nblk(nl, 128), 128, 0, s>>>((uint32_t)nl, leaves.p, start.p, end.p, leaf_of.p);
    RSG_LAUNCHED(ctx, "hm_leaf_of");
    std::vector<uint4> groups;
    std::vector<uint32_t> group_words;  // both live until the stream is waited for below
    build_groups(groups, group_words);
    up_vec(grp, groups, s), up_vec(grp_words, group_words, s);
    RSG_CUDA("upload", cudaEventCreateWithFlags(&ev_fork.e, cudaEventDisableTiming));
    RSG_CUDA("upload", cudaEventCreateWithFlags(&ev_join.e, cudaEventDisableTiming));
    // far coefficients (kernel.far, hierarchical.rs:210-220 / 980-984) in FP64 on the device
    // from the node centroids (and, for faces, the node projectors)
    {
      DevBuf<double> cen, pj;
      cen.upload(T.centroid.data(), 3 * nn, s);
      if (kind == FACE) pj.upload(proj6, 6 * nn, s);
      far_coef.alloc(std::max<size_t>(blocks.n_far, 1));
      if (n_far_items > 0) {
        hm_far_coef_kernel<<<nblk(n_far_items * 32, 256), 256, 0, s>>>(
            far_items.p, (int)n_far_items, blocks.far_col.p, cen.p, kind == FACE ? pj.p : nullptr, neg_s, far_coef.p);
        RSG_LAUNCHED(ctx, "hm_far_coef");
      }
      RSG_CUDA("upload", cudaStreamSynchronize(s));  // before the staging buffers go
    }
    lap(setup_times[1]);
    // element records
    DevBuf<double> dp, dw, dn;
    dp.upload(pts, 3 * n_el, s);
    dw.upload(wt, n_el, s);
    if (nrm64) dn.upload(nrm64, 3 * n_el, s);
    DevBuf<uint32_t> ord;
    ord.upload(T.order.data(), T.order.size(), s);
    xh.alloc(n_el), xl.alloc(n_el);
    if (kind == FACE) nrm.alloc(n_el);
    hm_pack_kernel<<<nblk(n_el, 256), 256, 0, s>>>(dp.p, dw.p, nrm64 ? dn.p : nullptr, ord.p, (int)n_el,
                                                   xh.p, xl.p, kind == FACE ? nrm.p : nullptr);
    RSG_LAUNCHED(ctx, "hm_pack");
    // near weights of every work item, evaluated once; the product passes read them
    wts.alloc(std::max<size_t>(n_wts, 2));
    {
      const HDev dw0 = dev();
      const unsigned g = nblk(n_items * 8 * 32, 256);
      if (kind == FACE) hm_weights_kernel<FACE><<<g, 256, 0, s>>>(dw0);
      else hm_weights_kernel<VERTEX><<<g, 256, 0, s>>>(dw0);
      RSG_LAUNCHED(ctx, "hm_weights");
    }
    // far part of H~a: upward over psi = a (m = 1, 2 channels) and far sums per node
    reserve(4);
    HDev d = dev();
    leaf_farA.alloc(std::max<size_t>(nl, 1));
    upward_far<ONES>(d, 1, reinterpret_cast<double *>(leaf_farA.p), s);
    RSG_CUDA("upload", cudaStreamSynchronize(s));
    lap(setup_times[2]);
  }

  // the near field of nb <= 3 vectors; the warps of the leaves of 8 rows first
  template <int K, bool PLAIN, int NV>
  void rows(const HDev &d, int nb) {
    const int ipw[9] = {1,
                        NearLanes<K, 1, PLAIN, NV>::IPW,
                        NearLanes<K, 2, PLAIN, NV>::IPW,
                        NearLanes<K, 3, PLAIN, NV>::IPW,
                        NearLanes<K, 4, PLAIN, NV>::IPW,
                        NearLanes<K, 5, PLAIN, NV>::IPW,
                        NearLanes<K, 6, PLAIN, NV>::IPW,
                        NearLanes<K, 7, PLAIN, NV>::IPW,
                        NearLanes<K, 8, PLAIN, NV>::IPW};
    const uint32_t passes = (uint32_t)(nb / NV);
    RowsGrid gr;
    gr.warps[9] = gr.warps[0] = 0;
    for (int i = 8; i >= 1; --i)
      gr.warps[i] = gr.warps[i + 1] + (sched_off[i] - sched_off[i - 1] + ipw[i] - 1) / ipw[i] * passes;
    hm_rows_kernel<K, PLAIN, NV><<<nblk((size_t)gr.warps[1] * 32, 128), 128, 0, st()>>>(d, gr, passes);
    RSG_LAUNCHED(ctx, "hm_rows");
  }
  template <bool PLAIN>
  void rows_any(const HDev &d, int nb) {
    if (kind == FACE) rows<FACE, PLAIN, 1>(d, nb);
    else if (nb == 1) rows<VERTEX, PLAIN, 1>(d, nb);
    else if (nb == 2) rows<VERTEX, PLAIN, 2>(d, nb);
    else rows<VERTEX, PLAIN, 3>(d, nb);
  }

  // z of the nb vectors whose channel values are already in `z`: the far passes (latency, FP64 and
  // gathers) on the second stream beside the near field (FP32 and shared memory), unless the kernels
  // are being timed one by one
  template <int K>
  void product_on(const HDev &d, int nb, const unsigned long long *qmax_) {
    cudaStream_t s = st();
    constexpr int SEL = K == FACE ? FACE_CH : VERTEX_CH, CC = kChannels<SEL>;
    prof.begin(s, K == FACE ? "metric_m" : "vfrac_m");
    split_m_kernel<CC><<<dim3(nblk(n_el * (CC / 4), 256), (unsigned)nb), 256, 0, s>>>(n_el, d.z, const_cast<float *>(d.m), qmax_);
    RSG_LAUNCHED(ctx, "split_m");
    prof.end(s);
    cudaStream_t far = prof.active ? s : ctx->stream2;
    if (far != s) {
      RSG_CUDA("product", cudaEventRecord(ev_fork.e, s));
      RSG_CUDA("product", cudaStreamWaitEvent(far, ev_fork.e, 0));
    }
    upward_far<SEL>(d, nb, d.leafsum, far);
    if (far != s) RSG_CUDA("product", cudaEventRecord(ev_join.e, far));
    prof.begin(s, K == FACE ? "metric_rows" : "vfrac_rows");
    if (plain_rows) rows_any<true>(d, nb);
    else rows_any<false>(d, nb);
    prof.end(s);
    if (far != s) RSG_CUDA("product", cudaStreamWaitEvent(s, ev_join.e, 0));
    prof.begin(s, K == FACE ? "metric_epilogue" : "vfrac_epilogue");
    hm_epilogue_kernel<SEL><<<dim3(nblk(n_el * CC, 256), (unsigned)nb), 256, 0, s>>>(d);
    RSG_LAUNCHED(ctx, "hm_epilogue");
    prof.end(s);
  }

  void build_common(rs_ctx *c, Tree &&t, double chi, int leaf_pairs) {
    ctx = c;
    tree = std::move(t);
    if (!(std::isfinite(chi) && chi >= 0.0))
      fail(RS_INVALID_OPTION, "InvalidOption", "upload", "chi must be a finite number >= 0");
    if (leaf_pairs < 0) fail(RS_INVALID_OPTION, "InvalidOption", "upload", "leaf_pairs must be >= 0");
    blocks = classify_blocks_device(tree, chi, (size_t)leaf_pairs);
  }
};

void check_exponents(double alpha, double beta) {
  if (!std::isfinite(alpha) || !std::isfinite(beta) || alpha <= 1.0 || beta <= alpha + 2.0 ||
      beta >= 2.0 * alpha + 2.0)
    fail(RS_INVALID_EXPONENTS, "InvalidExponents", "metric",
         "exponents must satisfy alpha > 1 and alpha + 2 < beta < 2 alpha + 2");
}

}  // namespace

struct rs_metric {
  HMat h;
  int nv = 0, nf = 0;
  // build phases in seconds: geometry, tree, projectors, blocks, face records, work items,
  // far coefficients, device part (uploads, element records, weights, far part of H~a)
  double build_times[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  FaceGeom geom;
  DevBuf<uint32_t> faces, inc_off, inc;
  DevBuf<double> g, area;
  DevBuf<double> xbuf, ybuf;
  FaceOps ops() const {
    FaceOps o;
    o.faces = faces.p, o.g = g.p, o.area = area.p;
    o.inc_off = inc_off.p, o.inc = inc.p, o.nv = nv, o.nf = nf;
    return o;
  }
};

struct rs_vfrac {
  HMat h;
  int nv = 0;
  DevBuf<uint32_t> order;
  DevBuf<double> xbuf, ybuf;
};

namespace {

// FaceMetricTree::from_parts / build (hierarchical.rs:302-363): df coefficients, projectors,
// blocks, element records.
void metric_setup(rs_metric *M, rs_ctx *ctx, int nv, int nf, const uint32_t *faces,
                  const double *pos, double alpha, double beta, double chi, int leaf_size,
                  int leaf_pairs) {
  check_exponents(alpha, beta);
  validate_topology(nv, nf, faces);
  validate_positions(nv, nf, faces, pos);
  ctx->use();
  using clk = std::chrono::steady_clock;
  auto t_ph = clk::now();
  auto lap = [&](int slot) {
    const auto now = clk::now();
    M->build_times[slot] = std::chrono::duration<double>(now - t_ph).count();
    t_ph = now;
  };
  M->nv = nv, M->nf = nf;
  const SharedFaceTree *sh = shared_face_tree(faces, pos, nf, leaf_size);
  M->geom = sh ? sh->geom : face_geometry(nf, faces, pos);
  lap(0);
  Tree T = sh ? sh->tree : build_face_tree(nf, faces, pos, M->geom, leaf_size);
  lap(1);
  M->h.kind = FACE;
  M->h.n_el = nf;
  M->h.set_exponent(-(beta - 2.0) / alpha);
  // projectors P = sum a N N^T / A per node (RS/src/spatial/mod.rs:268-290), bottom-up
  size_t nn = T.n_nodes();
  std::vector<double> ps(7 * nn, 0.0), proj(6 * nn);
  for (size_t i = nn; i-- > 0;) {
    double *o = &ps[7 * i];
    if (T.right[i] == 0) {
      for (uint32_t p = T.start[i]; p < T.end[i]; ++p) {
        uint32_t f = T.order[p];
        double a = M->geom.area[f];
        const double *n = &M->geom.normal[3 * (size_t)f];
        o[0] += a, o[1] += a * n[0] * n[0], o[2] += a * n[0] * n[1], o[3] += a * n[0] * n[2];
        o[4] += a * n[1] * n[1], o[5] += a * n[1] * n[2], o[6] += a * n[2] * n[2];
      }
    } else {
      for (int k = 0; k < 7; ++k) o[k] = ps[7 * (i + 1) + k] + ps[7 * (size_t)T.right[i] + k];
    }
    for (int k = 0; k < 6; ++k) proj[6 * i + k] = o[k + 1] / o[0];
  }
  lap(2);
  M->h.build_common(ctx, std::move(T), chi, leaf_pairs);
  lap(3);
  cudaStream_t s = M->h.st();
  // df coefficients (RS/src/metric/mod.rs:120-131) in FP64
  std::vector<double> gh(9 * (size_t)nf), ah(nf);
  std::vector<uint32_t> fh(3 * (size_t)nf), posn(nf);
  for (int pp = 0; pp < nf; ++pp) {
    const uint32_t f = M->h.tree.order[pp];
    posn[f] = (uint32_t)pp;
    std::copy(faces + 3 * (size_t)f, faces + 3 * (size_t)f + 3, fh.begin() + 3 * (size_t)pp);
    const double *p0 = pos + 3 * (size_t)faces[3 * f], *p1 = pos + 3 * (size_t)faces[3 * f + 1],
                 *p2 = pos + 3 * (size_t)faces[3 * f + 2];
    double u[3], w[3], n[3];
    for (int k = 0; k < 3; ++k) u[k] = p1[k] - p0[k], w[k] = p2[k] - p0[k];
    n[0] = u[1] * w[2] - u[2] * w[1], n[1] = u[2] * w[0] - u[0] * w[2], n[2] = u[0] * w[1] - u[1] * w[0];
    double len = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    double sc = 1.0 / (len * len);
    double ww[3] = {n[0] * sc, n[1] * sc, n[2] * sc};
    const double *pa[3] = {p1, p2, p0}, *pb[3] = {p2, p0, p1};
    for (int c = 0; c < 3; ++c) {
      double e[3] = {pb[c][0] - pa[c][0], pb[c][1] - pa[c][1], pb[c][2] - pa[c][2]};
      gh[9 * (size_t)pp + 3 * c + 0] = ww[1] * e[2] - ww[2] * e[1];
      gh[9 * (size_t)pp + 3 * c + 1] = ww[2] * e[0] - ww[0] * e[2];
      gh[9 * (size_t)pp + 3 * c + 2] = ww[0] * e[1] - ww[1] * e[0];
    }
    ah[pp] = M->geom.area[f];
  }
  std::vector<uint32_t> ioff((size_t)nv + 1, 0), inc(3 * (size_t)nf);
  for (int f = 0; f < nf; ++f)
    for (int c = 0; c < 3; ++c) ioff[faces[3 * f + c] + 1]++;
  for (int v = 0; v < nv; ++v) ioff[v + 1] += ioff[v];
  {
    std::vector<uint32_t> fill(ioff.begin(), ioff.end() - 1);
    for (int f = 0; f < nf; ++f)
      for (int c = 0; c < 3; ++c) inc[fill[faces[3 * f + c]]++] = (posn[f] << 2) | c;
  }
  up_vec(M->faces, fh, s);
  up_vec(M->g, gh, s), up_vec(M->area, ah, s), up_vec(M->inc_off, ioff, s), up_vec(M->inc, inc, s);
  lap(4);
  M->h.setup(M->geom.bary.data(), M->geom.area.data(), M->geom.normal.data(), proj.data());
  for (int i = 0; i < 3; ++i) M->build_times[5 + i] = M->h.setup_times[i];
}

}  // namespace

// The product of k <= 3 vectors in one tree pass on the scratch of d and qmax.
static void face_product(rs_metric *M, const HDev &d, unsigned long long *qmax, int k, const double *xs, size_t ldx,
                         double w_hi, double w_lo, double *ys, size_t ldy) {
  HMat &h = M->h;
  cudaStream_t s = h.st();
  const unsigned gy = (unsigned)k;
  h.prof.begin(s, "metric_m");
  RSG_CUDA("product", cudaMemsetAsync(qmax, 0, 12 * k * sizeof(unsigned long long), s));
  face_m_kernel<<<dim3(nblk(M->nf, 256), gy), 256, 0, s>>>(M->ops(), xs, ldx, d.z, qmax);
  RSG_LAUNCHED(h.ctx, "face_m");
  h.prof.end(s);
  h.product_on<FACE>(d, k, qmax);
  h.prof.begin(s, "metric_gather");
  face_gather_kernel<<<dim3(nblk(M->nv, 128), gy), 128, 0, s>>>(M->ops(), d.z, w_hi, w_lo, ys, ldy);
  RSG_LAUNCHED(h.ctx, "face_gather");
  h.prof.end(s);
}

// FaceMetricTree::apply_batch (hierarchical.rs:540-622) on device vectors with leading
// dimensions ldx, ldy (>= 3V): groups of <= 3 vectors per tree pass.
void rsg::metric_apply_strided(rs_metric *M, double w_hi, double w_lo, int nb, const double *xs,
                               size_t ldx, double *ys, size_t ldy, bool plain) {
  if (!(std::isfinite(w_hi) && std::isfinite(w_lo)))
    fail(RS_INVALID_OPTION, "InvalidOption", "product", "finite weights");
  cudaStream_t s = M->h.st();
  M->h.plain_rows = plain;
  for (int q0 = 0; q0 < nb; q0 += 3) {
    int k = std::min(3, nb - q0);
    M->h.reserve(12 * k);
    if (M->h.qmax.n < 64) M->h.qmax.alloc(64);
    face_product(M, M->h.dev(), M->h.qmax.p, k, xs + q0 * ldx, ldx, w_hi, w_lo, ys + q0 * ldy, ldy);
  }
}

// VertexFractionalTree::apply_batch (hierarchical.rs:1274-1345) scaled by `scale`.
void rsg::vfrac_apply_strided(rs_vfrac *V, double scale, int nb, const double *xs, size_t ldx,
                              double *ys, size_t ldy, bool plain) {
  cudaStream_t s = V->h.st();
  V->h.plain_rows = plain;
  for (int q0 = 0; q0 < nb; q0 += 3) {
    int k = std::min(3, nb - q0);
    const unsigned gy = (unsigned)k;
    V->h.reserve(4 * k);
    if (V->h.qmax.n < 64) V->h.qmax.alloc(64);
    const HDev d = V->h.dev();
    RSG_CUDA("product", cudaMemsetAsync(V->h.qmax.p, 0, 3 * k * sizeof(unsigned long long), s));
    vertex_m_kernel<<<dim3(nblk(V->nv, 256), gy), 256, 0, s>>>(V->order.p, xs + q0 * ldx, ldx, V->nv, d.z,
                                                               V->h.qmax.p);
    RSG_LAUNCHED(V->h.ctx, "vertex_m");
    V->h.product_on<VERTEX>(d, k, V->h.qmax.p);
    vertex_out_kernel<<<dim3(nblk(V->nv, 256), gy), 256, 0, s>>>(V->order.p, V->h.xh.p, d.z, V->nv, scale,
                                                                 ys + q0 * ldy, ldy);
    RSG_LAUNCHED(V->h.ctx, "vertex_out");
  }
}

namespace {

template <class F>
void host_io(rs_ctx *ctx, DevBuf<double> &xb, DevBuf<double> &yb, size_t n, const double *xh,
             double *yh, F &&apply) {
  cudaStream_t s = ctx->stream;
  if (xb.n < n) xb.alloc(n), yb.alloc(n);
  double *stage = (double *)ctx->staging(n * sizeof(double));
  std::memcpy(stage, xh, n * sizeof(double));
  RSG_CUDA("upload", rsg::copy_async(xb.p, stage, n * sizeof(double), cudaMemcpyHostToDevice, s));
  apply(xb.p, yb.p);
  RSG_CUDA("product", rsg::copy_async(stage, yb.p, n * sizeof(double), cudaMemcpyDeviceToHost, s));
  RSG_CUDA("product", cudaStreamSynchronize(s));
  std::memcpy(yh, stage, n * sizeof(double));
}

}  // namespace

extern "C" {

int rs_metric_build(rs_ctx *ctx, int nv, int nf, const uint32_t *faces, const double *positions_host,
                    double alpha, double beta, double chi, int leaf_size, int leaf_pairs,
                    rs_metric **out) {
  *out = nullptr;
  return guard([&] {
    auto M = std::make_unique<rs_metric>();
    metric_setup(M.get(), ctx, nv, nf, faces, positions_host, alpha, beta, chi, leaf_size, leaf_pairs);
    ctx_retain(ctx);
    *out = M.release();
  });
}

void rs_metric_free(rs_metric *M) {
  if (!M) return;
  rs_ctx *ctx = M->h.ctx;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  delete M;
  ctx_release(ctx);
}

int rs_metric_apply(rs_metric *M, double w_hi, double w_lo, int nb, const double *xs_host,
                    double *ys_host) {
  return guard([&] {
    M->h.ctx->use();
    size_t n = (size_t)nb * 3 * M->nv;
    host_io(M->h.ctx, M->xbuf, M->ybuf, n, xs_host, ys_host,
            [&](const double *x, double *y) { metric_apply_strided(M, w_hi, w_lo, nb, x, 3 * (size_t)M->nv, y, 3 * (size_t)M->nv); });
  });
}

int rs_metric_apply_device(rs_metric *M, double w_hi, double w_lo, int nb, const double *xs_dev,
                           double *ys_dev) {
  return guard([&] {
    M->h.ctx->use();
    metric_apply_strided(M, w_hi, w_lo, nb, xs_dev, 3 * (size_t)M->nv, ys_dev, 3 * (size_t)M->nv);
  });
}

int rs_metric_build_times(rs_metric *M, double *out8) {
  return guard([&] { std::copy(M->build_times, M->build_times + 8, out8); });
}

int rs_metric_stats(rs_metric *M, int64_t *o) {
  return guard([&] {
    o[0] = (int64_t)M->h.blocks.n_far;
    o[1] = (int64_t)M->h.blocks.n_near;
    o[2] = (int64_t)M->h.blocks.near_entries;
    o[3] = (int64_t)M->h.blocks.depth;
    o[4] = (int64_t)M->h.tree.n_nodes();
  });
}

int rs_metric_blocks(rs_metric *M, uint32_t *far_ptr, uint32_t *far_col, uint32_t *near_ptr,
                     uint32_t *near_col) {
  return guard([&] {
    std::vector<uint32_t> fp, fc, np, nc;
    M->h.blocks.download(fp, fc, np, nc);
    std::copy(fp.begin(), fp.end(), far_ptr);
    std::copy(fc.begin(), fc.end(), far_col);
    std::copy(np.begin(), np.end(), near_ptr);
    std::copy(nc.begin(), nc.end(), near_col);
  });
}

int rs_metric_profile(rs_metric *M, double w_hi, double w_lo, int nb, int reps, char *names,
                      int names_len, double *ms, int max_kernels, int *n_kernels) {
  return guard([&] {
    M->h.ctx->use();
    size_t n = (size_t)nb * 3 * M->nv;
    if (M->xbuf.n < n) M->xbuf.alloc(n), M->ybuf.alloc(n);
    RSG_CUDA("product", cudaMemsetAsync(M->xbuf.p, 0, n * sizeof(double), M->h.st()));
    M->h.prof.start();
    for (int r = 0; r < reps; ++r)
      metric_apply_strided(M, w_hi, w_lo, nb, M->xbuf.p, 3 * (size_t)M->nv, M->ybuf.p, 3 * (size_t)M->nv);
    M->h.prof.stop(M->h.st());
    M->h.prof.report(names, names_len, ms, max_kernels, n_kernels, reps);
  });
}

int rs_vfrac_build(rs_ctx *ctx, int nv, const double *positions_host, const double *mass_host,
                   double tau, double chi, int leaf_size, int leaf_pairs, rs_vfrac **out) {
  *out = nullptr;
  return guard([&] {
    if (!std::isfinite(tau) || nv <= 0)
      fail(RS_INVALID_OPTION, "InvalidOption", "upload", "a finite order and at least one vertex");
    for (int v = 0; v < nv; ++v)
      if (!(std::isfinite(mass_host[v]) && mass_host[v] > 0.0))
        fail(RS_INVALID_OPTION, "InvalidOption", "upload", "positive finite vertex areas");
    ctx->use();
    auto V = std::make_unique<rs_vfrac>();
    V->nv = nv;
    // vertex elements: point f_v, box of the point, mass a_v (hierarchical.rs:1041-1058)
    std::vector<double> ebox(6 * (size_t)nv);
    for (int v = 0; v < nv; ++v)
      for (int k = 0; k < 3; ++k) ebox[6 * v + k] = ebox[6 * v + 3 + k] = positions_host[3 * v + k];
    Tree T = build_tree((size_t)nv, positions_host, ebox.data(), mass_host, leaf_size);
    V->h.kind = VERTEX;
    V->h.n_el = nv;
    V->h.set_exponent(-(tau + 1.0));
    V->h.build_common(ctx, std::move(T), chi, leaf_pairs);
    up_vec(V->order, V->h.tree.order, V->h.st());
    V->h.setup(positions_host, mass_host, nullptr, nullptr);
    ctx_retain(ctx);
    *out = V.release();
  });
}

void rs_vfrac_free(rs_vfrac *V) {
  if (!V) return;
  rs_ctx *ctx = V->h.ctx;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  delete V;
  ctx_release(ctx);
}

int rs_vfrac_apply(rs_vfrac *V, int nb, const double *xs_host, double *ys_host) {
  return guard([&] {
    V->h.ctx->use();
    size_t n = (size_t)nb * 3 * V->nv;
    host_io(V->h.ctx, V->xbuf, V->ybuf, n, xs_host, ys_host,
            [&](const double *x, double *y) { vfrac_apply_strided(V, 1.0, nb, x, 3 * (size_t)V->nv, y, 3 * (size_t)V->nv); });
  });
}

int rs_vfrac_apply_device(rs_vfrac *V, int nb, const double *xs_dev, double *ys_dev) {
  return guard([&] {
    V->h.ctx->use();
    vfrac_apply_strided(V, 1.0, nb, xs_dev, 3 * (size_t)V->nv, ys_dev, 3 * (size_t)V->nv);
  });
}

int rs_vfrac_stats(rs_vfrac *V, int64_t *o) {
  return guard([&] {
    o[0] = (int64_t)V->h.blocks.n_far;
    o[1] = (int64_t)V->h.blocks.n_near;
    o[2] = (int64_t)V->h.blocks.near_entries;
    o[3] = (int64_t)V->h.blocks.depth;
    o[4] = (int64_t)V->h.tree.n_nodes();
  });
}

}  // extern "C"

// ====================================================================== no-allocation product
//
// rs_metric_apply_device_noalloc: the metric product of rs_metric_apply_device with its
// per-call scratch (channel values, results, near partial sums, node sums) carved from one
// file-scope device array instead of buffers that the first call of a size allocates. It is
// for callers that must not allocate while the product runs: a host whose device memory is
// entirely reserved by its own pool after set-up, and a caller on a latency-critical stream,
// since cudaMalloc and cudaFree can synchronize the whole device.
//
// Limits: the scratch is kNoAllocScratchBytes per device, shared by every call in the process,
// so calls that overlap in time (two host threads, or two streams in flight) race on it and
// must be serialized by the caller; a call also uses the metric's own events and the
// context's second stream, so it must not overlap any other product on the same rs_metric either. The
// array is resident on every device where this file's kernels are loaded (from the first
// metric build or product there, with lazy module loading), whether or not this entry point
// is ever called. The first call on a device looks up the array's address
// (cudaGetSymbolAddress, with that device current); when that call is made inside a stream
// capture the lookup should have been done before it, by one earlier call.

namespace {

constexpr size_t kNoAllocScratchBytes = size_t(64) << 20;  // 64 MiB
constexpr int kNoAllocMaxDevices = 64;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

unsigned char *noalloc_scratch(int device) {
  static std::mutex mu;
  static unsigned char *addr[kNoAllocMaxDevices] = {};
  if (device < 0 || device >= kNoAllocMaxDevices)
    fail(RS_INVALID_OPTION, "InvalidOption", "product", "device ordinal out of range for the no-alloc scratch");
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[device]) {
    void *p = nullptr;
    RSG_CUDA("product", cudaGetSymbolAddress(&p, g_noalloc_scratch));
    addr[device] = static_cast<unsigned char *>(p);
  }
  return addr[device];
}

inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// Scratch bytes a call with C channels is admitted by: the layout carved below and an FP64 value
// per node and channel beside it (not used).
size_t noalloc_bytes(const HMat &h, int C) {
  size_t nn = h.tree.n_nodes();
  return 2 * align256(nn * C * sizeof(double)) + align256(nn * C * sizeof(float2)) +
         2 * align256(h.n_el * C * sizeof(float2)) +
         align256(std::max<size_t>(h.n_items, 1) * 8 * C * sizeof(float2)) +
         align256(h.tree.leaves.size() * C * sizeof(double)) +
         align256(std::max<size_t>(h.n_far_items, 1) * C * sizeof(float2)) + align256(64 * sizeof(unsigned long long));
}

HDev noalloc_dev(const HMat &h, int C, unsigned char *base) {
  HDev d = h.dev();
  size_t nn = h.tree.n_nodes(), off = 0;
  auto take = [&](size_t bytes) {
    unsigned char *p = base + off;
    off += align256(bytes);
    return p;
  };
  d.up = reinterpret_cast<double *>(take(nn * C * sizeof(double)));
  d.up2 = reinterpret_cast<float2 *>(take(nn * C * sizeof(float2)));
  d.m = reinterpret_cast<const float *>(take(h.n_el * C * sizeof(float2)));
  d.z = reinterpret_cast<double *>(take(h.n_el * C * sizeof(float2)));
  d.part = reinterpret_cast<float2 *>(take(std::max<size_t>(h.n_items, 1) * 8 * C * sizeof(float2)));
  d.leafsum = reinterpret_cast<double *>(take(h.tree.leaves.size() * C * sizeof(double)));
  d.fpart = reinterpret_cast<float2 *>(take(std::max<size_t>(h.n_far_items, 1) * C * sizeof(float2)));
  return d;
}

// the per-channel magnitudes of the no-alloc product, after the buffers of noalloc_dev
unsigned long long *noalloc_qmax(const HMat &h, int C, unsigned char *base) {
  return reinterpret_cast<unsigned long long *>(base + noalloc_bytes(h, C) - align256(64 * sizeof(unsigned long long)));
}

}  // namespace

extern "C" int rs_metric_apply_device_noalloc(rs_metric *M, double w_hi, double w_lo, int nb,
                                              const double *xs_dev, double *ys_dev) {
  return guard([&] {
    if (nb < 1) fail(RS_INVALID_OPTION, "InvalidOption", "product", "at least one vector");
    if (!(std::isfinite(w_hi) && std::isfinite(w_lo)))
      fail(RS_INVALID_OPTION, "InvalidOption", "product", "finite weights");
    const int Cmax = 12 * std::min(3, nb);
    const size_t need = noalloc_bytes(M->h, Cmax);
    if (need > kNoAllocScratchBytes)
      fail(RS_INVALID_OPTION, "InvalidOption", "product",
           "the no-alloc product of " + std::to_string(std::min(3, nb)) + " vector(s) on this mesh needs " +
               std::to_string(need >> 20) + " MiB of scratch, above its 64 MiB; use rs_metric_apply_device");
    M->h.ctx->use();
    unsigned char *base = noalloc_scratch(M->h.ctx->device);
    const size_t ld = 3 * (size_t)M->nv;
    for (int q0 = 0; q0 < nb; q0 += 3) {
      const int k = std::min(3, nb - q0);
      HDev d = noalloc_dev(M->h, 12 * k, base);
      unsigned long long *qm = noalloc_qmax(M->h, 12 * k, base);
      M->h.plain_rows = false;
      face_product(M, d, qm, k, xs_dev + q0 * ld, ld, w_hi, w_lo, ys_dev + q0 * ld, ld);
    }
  });
}
