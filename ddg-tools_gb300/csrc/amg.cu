// Conjugate gradients preconditioned by V-cycles of the smoothed-aggregation multigrid (see
// amg.hpp) as one persistent kernel.
//
// A solve is about thirty dependent passes per step (levels x smoothing sweeps, transfers, dot
// products, updates), each over a few thousand to a hundred thousand rows: far too little work to
// hide a kernel boundary. As a graph of one kernel per pass they took 3.3-4.0 us each; here they
// are separated by a barrier. A block keeps its rows of every level (the slices of A, P, R and
// the damped inverse diagonals) in shared memory for the whole solve, so that a pass waits for one
// gather of the other blocks' values and no more. Vectors hold the columns of a row side by side,
// padded to whole 16-byte loads.
//
// Two forms. Three columns whose vectors 16 blocks' shared memory holds beside the matrices (up to about
// 5,000 vertices): one cluster, gathers through distributed shared memory, the cluster's barrier.
// Else a block per SM (a cooperative launch), vectors in global memory, gathers from L2 and
// a counter as the barrier. With six or nine columns 16 SMs are too few for the FP64 of the dot
// products (4,356 rows: 18.3 against 16.8 ms, 17.8 against 18.0; 900 rows: 8.6 against 8.3, 9.6
// against 8.6; with three columns 14.2 against 15.2 and 6.6 against 7.3).
//
// What is left is latency: per pass 1,500-2,500 cycles of dependent loads and a barrier of
// 1,200-2,000 (cluster) or 3,400-4,000 (grid), the FP64 trees of the dot products, and at 102,400
// rows the gathers from L2 (12 values a row: 11,000 cycles a sweep).
// Measured, a GMRES solve's share, graph of kernels -> here, for 3 / 6 / 9 columns: 900 rows 10.7 / 12.8
// / 14.4 -> 6.6 / 8.3 / 8.6 ms; 4,356 rows 20.9 / 23.6 / 27.3 -> 14.2 / 16.8 / 18.0 ms; 25,600 rows 43.4
// / 50.1 / 56.4 -> 33.4 / 37.4 / 43.5 ms; 102,400 rows 101 / 124 / 154 -> 89 / 105 / 141 ms.
#include "amg.hpp"
#include "fp64_bits.cuh"

namespace rsg {

namespace {

constexpr int kDotBlocks = 304;  // fixed split of the column dot products (deterministic)
constexpr int kMaxLevels = 12;
constexpr int kCluster = 16;     // blocks of a solve in one cluster

// floats from row to row of a vector of C columns
template <int C>
constexpr int kStride = C == 3 ? 4 : (C == 6 ? 8 : 12);

struct DevMat {
  const int *ptr;   // rows + 1
  const int2 *cv;   // column, value (bits)
  int tpr;          // lanes per row
};
struct DevLevel {
  int n;
  DevMat a, p, r;   // A_l; P_l (rows of level l); R_l (rows of level l + 1)
  const float *dinv;
  float *x, *b, *res, *t;
};
struct CgArgs {
  int nl, iters;
  DevLevel l[kMaxLevels];
  const float *cinv;            // dense inverse of the coarsest level
  const float *rhs;             // n_0 x C
  float *sol;                   // n_0 x C
  float *p, *q;                 // n_0 x stride
  double *part;                 // kDotBlocks x C partial sums, two sets used in turn
  unsigned long long *counter;  // arrivals at the grid barrier, a multiple of the grid between solves
  int *error;                   // set when a barrier gave up
  unsigned polls;               // after this many
  int smem_bytes;
};

// The own rows of one matrix of a block: in shared memory when they fit, else in global memory
// (ptr then holds the global offsets). In a cluster the columns are the addresses of their values in
// the owner's shared memory.
struct Slice {
  const int *ptr;
  const int2 *cv;
  int n, tpr;
};
// A vector of a level: its own rows, and what a matrix's columns are gathered by (its address in
// global memory, or its offset among the level's vectors in the shared memory of every block).
struct Vec {
  float *own;
  unsigned long long g;
};
struct LevelSlices {
  Slice a, p, r;
  const float *dinv;  // of the own rows
  Vec x, b, res, t;   // level 0: z and r of the conjugate gradients for x and b
};

template <int C>
__device__ __forceinline__ void load_row(const float *v, size_t row, float (&x)[C]) {
  constexpr int S = kStride<C>;
  const float4 *q = reinterpret_cast<const float4 *>(v + row * S);
#pragma unroll
  for (int i = 0; i < S / 4; ++i) {
    const float4 t = q[i];
    const float e[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (4 * i + k < C) x[4 * i + k] = e[k];
  }
}
template <int C>
__device__ __forceinline__ void store_row(float *v, size_t row, const float (&x)[C]) {
  constexpr int S = kStride<C>;
  float4 *q = reinterpret_cast<float4 *>(v + row * S);
#pragma unroll
  for (int i = 0; i < S / 4; ++i) {
    float e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = 4 * i + k < C ? x[4 * i + k] : 0.f;
    q[i] = make_float4(e[0], e[1], e[2], e[3]);
  }
}

// the values of the column x of a matrix (see Slice)
template <int C, bool CLUSTER>
__device__ __forceinline__ void gather(const Vec &v, int x, float (&o)[C]) {
  if constexpr (CLUSTER) {
    constexpr int S = kStride<C>;
    const unsigned a = (unsigned)x + (unsigned)v.g;
#pragma unroll
    for (int i = 0; i < S / 4; ++i) {
      float e[4];
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(e[0]), "=f"(e[1]), "=f"(e[2]), "=f"(e[3])
                   : "r"(a + 16 * i)
                   : "memory");
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (4 * i + k < C) o[4 * i + k] = e[k];
    }
  } else {
    load_row<C>(reinterpret_cast<const float *>(v.g), (size_t)x, o);
  }
}

// Barrier across the blocks of a solve. In one cluster: the hardware's (0.3 us). Across the grid: a
// counter that one thread of every block adds to and then polls (1.2 us with 152 blocks; a flag per
// block that all blocks poll took 6 us). Both order the block's accesses before and after
// (L1 does not outlive them), so the gathers between two barriers may hit L1: a row's values are
// read by about seven others. The wait on the counter is bounded: a block that gives up
// sets *error, and the rest of the solve runs through without waiting.
template <bool CLUSTER>
struct SolveBarrier {
  unsigned long long *counter;
  int *error;
  unsigned polls_max;
  unsigned long long target;  // the count that ends the next barrier (thread 0)
  bool dead = false;
  __device__ __forceinline__ void sync() {
    if constexpr (CLUSTER) {
      asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      return;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(counter, 1ull);
      unsigned long long v;
      unsigned polls = 0;
      while (!dead) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(counter) : "memory");
        if (v >= target) break;
        if (++polls >= polls_max || ((polls & 4095u) == 0u && *(volatile int *)error)) {
          *(volatile int *)error = 1;
          dead = true;
        }
      }
      target += gridDim.x;
      __threadfence();
    }
    __syncthreads();
  }
};

// f(local row, pre(local row), product) over the own rows of a matrix: the lanes of a group of
// tpr take the nonzeros sub, sub + tpr, ... of a row and a butterfly adds them, so every lane of
// the group ends with the same sum. pre loads what f needs beside the product: ahead of the gathers
// where that is from global memory. Threads: as many as the registers of the columns allow without
// spilling much (nine on the grid: 141 ms with 384 threads, 155 with 512).
template <int C, bool CLUSTER>
constexpr int kMaxThreads = CLUSTER ? 1024 : (C <= 6 ? 512 : 384);
template <int C, bool CLUSTER, class Pre, class F>
__device__ __forceinline__ void for_rows(const Slice &m, const Vec &x, Pre pre, F f) {
  const int tpr = m.tpr, sh = __ffs(tpr) - 1, lane = threadIdx.x & 31, total = m.n << sh;
  for (int base = threadIdx.x & ~31; base < total; base += blockDim.x) {
    const int idx = base + lane, row = idx >> sh, sub = idx & (tpr - 1);
    const bool valid = row < m.n;
    decltype(pre(row)) own;
    if constexpr (!CLUSTER) own = pre(valid && sub == 0 ? row : -1);
    float acc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = 0.f;
    if (valid) {
      const int p0 = m.ptr[row] + sub, count = (m.ptr[row + 1] - p0 + tpr - 1) >> sh;
      const int2 *cv = m.cv + p0;
#pragma unroll 4
      for (int k = 0; k < count; ++k) {
        const int2 e = cv[k << sh];
        const float a = __int_as_float(e.y);
        float v[C];
        gather<C, CLUSTER>(x, e.x, v);
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] = fmaf(a, v[c], acc[c]);
      }
    }
    for (int o = tpr >> 1; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if (valid && sub == 0) {
      if constexpr (CLUSTER) own = pre(row);
      f(row, own, acc);
    }
  }
}
template <int C>
struct RowVals {
  float v[C];
};
template <int C>
struct SweepVals {
  float b[C], x[C], d;
};
struct NoVals {};

// The halving trees of four columns over 128 threads' values each (pairs 64 apart, then 32 apart, then
// 16 to 1), by one warp: past 32 apart the columns share the lanes, as FP64 instructions cost a warp
// sixteen cycles whatever its idle lanes. Lanes 0, 16, 8 and 24 end with the sums of columns 0 to 3. sh: the columns, 128
// values each, all zero from `count` on (whose additions are left out).
__device__ __forceinline__ double to_f64(double v) { return v; }
__device__ __forceinline__ double to_f64(float v) { return f2d(v); }
__device__ __forceinline__ double tree32x4(const double (&v)[4], int lane) {
  // 16 apart: lanes 0-15 keep columns 0 and 2, lanes 16-31 columns 1 and 3; 8 apart likewise
  const bool u16 = lane & 16, u8 = lane & 8;
  double a = u16 ? v[1] : v[0], b = u16 ? v[3] : v[2];
  a += __shfl_xor_sync(0xffffffffu, u16 ? v[0] : v[1], 16);
  b += __shfl_xor_sync(0xffffffffu, u16 ? v[2] : v[3], 16);
  double c = u8 ? b : a;
  c += __shfl_xor_sync(0xffffffffu, u8 ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  return c;  // lanes 0-7: column 0, 8-15: 2, 16-23: 1, 24-31: 3
}
template <class T>
__device__ __forceinline__ double tree128x4(const T (*sh)[128], int lane, int count) {
  double v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = to_f64(sh[k][lane]);
    if (count > 64) v[k] += to_f64(sh[k][lane + 64]);
    if (count > 32) {
      double u = to_f64(sh[k][lane + 32]);
      if (count > 64) u += to_f64(sh[k][lane + 96]);
      v[k] += u;
    }
  }
  return tree32x4(v, lane);
}

// own rows of block b of n rows split over the grid
__device__ __forceinline__ int row_begin(int n, unsigned b) { return (int)((long long)n * b / gridDim.x); }

template <int C, bool CLUSTER>
__global__ void __launch_bounds__(kMaxThreads<C, CLUSTER>, 1) pcg_kernel(const __grid_constant__ CgArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ LevelSlices S[kMaxLevels];
  constexpr int PARTS = kStride<C> / 4, S4 = 4 * PARTS;  // parts of four columns
  // the dot products: 128 values per column of a job (chunk and part); then the totals' values
  __shared__ __align__(16) float tree[8][4][128];
  static_assert(sizeof(tree) >= sizeof(double) * S4 * 128, "the totals' values fit");
  __shared__ double tot[S4], rz[C];
  __shared__ float scal[C];  // alpha or beta
  __shared__ int used;
  __shared__ const float *cinv;
  const unsigned bid = blockIdx.x;
  const int tid = threadIdx.x, nl = A.nl;
  // level 0 goes by the chunks of the dot products, so that a block owns whole chunks
  const int n0 = A.l[0].n, chunk = (n0 + kDotBlocks - 1) / kDotBlocks;
  const int vb0 = kDotBlocks * bid / gridDim.x, vb1 = kDotBlocks * (bid + 1) / gridDim.x;
  auto first_row = [&](int l, unsigned b) {
    return l == 0 ? min(n0, (int)(kDotBlocks * b / gridDim.x) * chunk) : row_begin(A.l[l].n, b);
  };
  const int f0 = first_row(0, bid), f1 = first_row(0, bid + 1);
  // the vectors of a level in shared memory (a cluster): rows for the block that owns most
  auto vec_bytes = [&](int l) {
    const int rows = l == 0 ? (int)((kDotBlocks + gridDim.x - 1) / gridDim.x) * chunk : (int)((A.l[l].n + gridDim.x - 1) / gridDim.x);
    return rows * kStride<C> * 4;
  };
  auto vec_base = [&](int l) {  // of the first vector of level l
    int at = 0;
    for (int k = 0; k < l; ++k) at += vec_bytes(k) * (k == 0 ? 6 : 4);
    return at;
  };
  // the cluster address of row j of the first vector of level l, whose offset is base (a cluster has
  // kCluster blocks, a divisor of the dot products' chunks)
  static_assert(kDotBlocks % kCluster == 0, "whole chunks");
  auto row_addr = [&](int l, int base, int j) -> unsigned {
    const unsigned n = (unsigned)A.l[l].n;
    unsigned o, r0;
    if (l == 0) {
      o = (unsigned)j / (unsigned)(kDotBlocks / kCluster * chunk), r0 = o * (kDotBlocks / kCluster * chunk);
    } else {
      // the last block that begins at row j or before (below 16 rows some blocks own none)
      o = (kCluster * ((unsigned)j + 1) - 1) / n;
      r0 = (unsigned)((unsigned long long)n * o / kCluster);
    }
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(smem) + base), "r"(o));
    return a + ((unsigned)j - r0) * (kStride<C> * 4);
  };
  if (tid == 0) used = CLUSTER ? vec_base(nl) : 0;
  __syncthreads();
  // the slices, level by level while they fit (in a cluster all do)
  auto take = [&](const DevMat &m, int r0, int r1, int lc, Slice &s) {  // columns: level lc; every thread
    const int p0 = m.ptr[r0], nnz = m.ptr[r1] - p0, rows = r1 - r0;
    const int at = used, need = 8 * nnz + ((4 * (rows + 1) + 15) & ~15);
    const bool fits = at + need <= A.smem_bytes;
    __syncthreads();  // everyone has read `used`
    if (fits) {
      int2 *cv = reinterpret_cast<int2 *>(smem + at);
      int *ptr = reinterpret_cast<int *>(smem + at + 8 * nnz);
      const int base = CLUSTER ? vec_base(lc) : 0;
      for (int i = tid; i < nnz; i += blockDim.x) {
        int2 e = __ldg(m.cv + p0 + i);
        if (CLUSTER) e.x = (int)row_addr(lc, base, e.x);
        cv[i] = e;
      }
      for (int i = tid; i <= rows; i += blockDim.x) ptr[i] = __ldg(m.ptr + r0 + i) - p0;
      if (tid == 0) s.ptr = ptr, s.cv = cv, used = (at + need + 15) & ~15;
    } else if (tid == 0) {
      s.ptr = m.ptr + r0, s.cv = m.cv;
    }
    if (tid == 0) s.n = rows, s.tpr = m.tpr;
    __syncthreads();
  };
  auto take_floats = [&](const float *v, int count, const float **out) {
    const int at = used, need = (4 * count + 15) & ~15;
    const bool fits = at + need <= A.smem_bytes;
    __syncthreads();
    float *d = reinterpret_cast<float *>(smem + at);
    if (fits)
      for (int i = tid; i < count; i += blockDim.x) d[i] = __ldg(v + i);
    if (tid == 0) {
      *out = fits ? d : v;
      if (fits) used = at + need;
    }
    __syncthreads();
  };
  Vec vp, vq;
  for (int l = 0; l < nl; ++l) {
    const DevLevel &v = A.l[l];
    const int r0 = first_row(l, bid), r1 = first_row(l, bid + 1);
    if (l + 1 < nl || nl == 1) take(v.a, r0, r1, l, S[l].a);
    if (l + 1 < nl) {
      take(v.p, r0, r1, l + 1, S[l].p);
      take(v.r, first_row(l + 1, bid), first_row(l + 1, bid + 1), l, S[l].r);
    } else {
      take_floats(A.cinv + (size_t)r0 * v.n, (r1 - r0) * v.n, &cinv);
    }
    take_floats(v.dinv + r0, r1 - r0, &S[l].dinv);
    const int base = CLUSTER ? vec_base(l) : 0, bytes = CLUSTER ? vec_bytes(l) : 0;
    auto vec = [&](int k, float *global) {
      Vec o;
      if constexpr (CLUSTER) o.own = reinterpret_cast<float *>(smem + base + k * bytes), o.g = (unsigned)(k * bytes);
      else o.own = global + (size_t)r0 * kStride<C>, o.g = (unsigned long long)global;
      return o;
    };
    if (tid == 0) S[l].x = vec(0, v.x), S[l].b = vec(1, v.b), S[l].res = vec(2, v.res), S[l].t = vec(3, v.t);
    if (l == 0) vp = vec(4, A.p), vq = vec(5, A.q);
  }
  // the counter stands at a multiple of the grid plus the blocks that arrived already, at most all
  // but this one
  SolveBarrier<CLUSTER> bar{A.counter, A.error, A.polls, 0ull};
  if (!CLUSTER) bar.target = (*(volatile unsigned long long *)A.counter / gridDim.x + 1) * gridDim.x;

  // out = x + dinv (b - A x)
  auto jacobi = [&](int l, const Vec &x, const Vec &out) {
    const float *dinv = S[l].dinv, *b = S[l].b.own, *xo = x.own;
    float *oo = out.own;
    for_rows<C, CLUSTER>(
        S[l].a, x,
        [&](int row) {
          SweepVals<C> o;
          if (row >= 0) {
            load_row<C>(b, (size_t)row, o.b), load_row<C>(xo, (size_t)row, o.x);
            o.d = dinv[row];
          }
          return o;
        },
        [&](int row, SweepVals<C> o, const float (&acc)[C]) {
#pragma unroll
          for (int c = 0; c < C; ++c) o.x[c] = fmaf(o.d, o.b[c] - acc[c], o.x[c]);
          store_row<C>(oo, (size_t)row, o.x);
        });
  };
  auto own_row = [](const float *v) {
    return [v](int row) {
      RowVals<C> o;
      if (row >= 0) load_row<C>(v, (size_t)row, o.v);
      return o;
    };
  };
  auto nothing = [](int) { return NoVals(); };
  // x_0 = V-cycle(b_0), the first sweep dinv b_0 of level 0 being in its t; two sweeps before and two
  // after each coarser solve
  auto vcycle = [&] {
    for (int l = 0; l + 1 < nl; ++l) {
      const LevelSlices &v = S[l], &w = S[l + 1];
      jacobi(l, v.t, v.x);
      bar.sync();
      for_rows<C, CLUSTER>(v.a, v.x, own_row(v.b.own), [&](int row, RowVals<C> o, const float (&acc)[C]) {
#pragma unroll
        for (int c = 0; c < C; ++c) o.v[c] -= acc[c];
        store_row<C>(v.res.own, (size_t)row, o.v);
      });
      bar.sync();
      // restriction, and the first sweep from zero of the next level (the coarsest is solved)
      const bool sweep = l + 2 < nl;
      for_rows<C, CLUSTER>(v.r, v.res, nothing, [&](int row, NoVals, const float (&acc)[C]) {
        store_row<C>(w.b.own, (size_t)row, acc);
        if (sweep) {
          const float d = w.dinv[row];
          float tv[C];
#pragma unroll
          for (int c = 0; c < C; ++c) tv[c] = d * acc[c];
          store_row<C>(w.t.own, (size_t)row, tv);
        }
      });
      bar.sync();
    }
    {  // coarsest: the dense inverse, one warp per row
      const int l = nl - 1, n = A.l[l].n, rows = first_row(l, bid + 1) - first_row(l, bid), lane = tid & 31;
      const Vec b = S[l].b;
      constexpr int ST = kStride<C>;
      float *all = &tree[0][0][0];
      const bool staged = CLUSTER && (size_t)n * ST * 4 <= sizeof(tree);
      if (staged) {  // the whole right-hand side, which every row reads, once across the cluster
        const int base = vec_base(l);
        for (int j = tid; j < n; j += blockDim.x) {
          float bv[C];
          gather<C, CLUSTER>(b, (int)row_addr(l, base, j), bv);
          store_row<C>(all, (size_t)j, bv);
        }
        __syncthreads();
      }
      for (int i = tid >> 5; i < rows; i += (int)(blockDim.x >> 5)) {
        float acc[C];
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] = 0.f;
        for (int j = lane; j < n; j += 32) {
          const float a = cinv[(size_t)i * n + j];
          float bv[C];
          if (staged) load_row<C>(all, (size_t)j, bv);
          else gather<C, CLUSTER>(b, CLUSTER ? (int)row_addr(l, vec_base(l), j) : j, bv);
#pragma unroll
          for (int c = 0; c < C; ++c) acc[c] = fmaf(a, bv[c], acc[c]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int c = 0; c < C; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
        if (lane == 0) store_row<C>(S[l].x.own, (size_t)i, acc);
      }
      bar.sync();
    }
    for (int l = nl - 2; l >= 0; --l) {
      const LevelSlices &v = S[l];
      // x += P x_coarse
      for_rows<C, CLUSTER>(v.p, S[l + 1].x, own_row(v.x.own), [&](int row, RowVals<C> o, const float (&acc)[C]) {
#pragma unroll
        for (int c = 0; c < C; ++c) o.v[c] += acc[c];
        store_row<C>(v.x.own, (size_t)row, o.v);
      });
      bar.sync();
      jacobi(l, v.x, v.t);
      bar.sync();
      jacobi(l, v.t, v.x);
      if (l > 0) bar.sync();  // level 0: the own rows' dot products follow first
    }
  };
  // The column dot products a.w over the own chunks into part: 128 threads a chunk, each adding
  // its rows in FP32, then a fixed tree in FP64. The sets of part alternate: a block may
  // still be adding up one when another writes the next.
  double *part = A.part, *other = A.part + (size_t)kDotBlocks * C;
  auto dots = [&](const float *a, const float *w) {
    double *const t_ = part;
    part = other, other = t_;
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5, jobs = (vb1 - vb0) * PARTS;
    auto values = [&](int job, int t) {  // the sum over the rows t, t + 128, ... of a job's chunk
      const int vb = vb0 + job / PARTS, pt = job % PARTS, i1 = min(n0, (vb + 1) * chunk) - f0;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int i = vb * chunk + t - f0; i < i1; i += 128) {
        const float4 x = reinterpret_cast<const float4 *>(a)[(size_t)i * PARTS + pt];
        const float4 y = reinterpret_cast<const float4 *>(w)[(size_t)i * PARTS + pt];
        acc.x = fmaf(x.x, y.x, acc.x), acc.y = fmaf(x.y, y.y, acc.y);
        acc.z = fmaf(x.z, y.z, acc.z), acc.w = fmaf(x.w, y.w, acc.w);
      }
      return acc;
    };
    auto put = [&](int job, double v) {
      const int c = 4 * (job % PARTS) + (lane >> 4) + ((lane >> 3) & 1) * 2;
      if ((lane & 7) == 0 && c < C) part[(size_t)(vb0 + job / PARTS) * C + c] = v;
    };
    if (chunk <= 32) {  // a row per lane: a warp per job, from registers
      for (int job = warp; job < jobs; job += (int)(blockDim.x >> 5)) {
        const float4 q = values(job, lane);
        const double v[4] = {to_f64(q.x), to_f64(q.y), to_f64(q.z), to_f64(q.w)};
        put(job, tree32x4(v, lane));
      }
      return;
    }
    const int grp = tid >> 7, t = tid & 127, ng = blockDim.x >> 7;
    for (int j0 = 0; j0 < jobs; j0 += ng) {
      if (j0 + grp < jobs) {
        const float4 q = values(j0 + grp, t);
        tree[grp][0][t] = q.x, tree[grp][1][t] = q.y, tree[grp][2][t] = q.z, tree[grp][3][t] = q.w;
      }
      __syncthreads();
      if (warp < min(ng, jobs - j0)) put(j0 + warp, tree128x4(tree[warp], lane, chunk));  // a warp per job
      __syncthreads();
    }
  };
  // The totals of part (strided over 128 threads, then the same tree), the same in every block.
  // mode 0: alpha = rz / total (a non-positive curvature stops the column); 1: beta = total / rz
  // and rz = total; 2: rz = total.
  auto scalars = [&](int mode) {
    double(*val)[128] = reinterpret_cast<double(*)[128]>(&tree[0][0][0]);
    const int lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < 128 * S4; k += blockDim.x) {
      const int c = k >> 7, t = k & 127;
      double v = 0.0;
      if (c < C) {
        v = part[(size_t)t * C + c] + part[(size_t)(t + 128) * C + c];
        if (t + 256 < kDotBlocks) v += part[(size_t)(t + 256) * C + c];
      }
      val[c][t] = v;
    }
    __syncthreads();
    if (warp < PARTS) {
      const double v = tree128x4(val + 4 * warp, lane, 128);
      if ((lane & 7) == 0) tot[4 * warp + (lane >> 4) + ((lane >> 3) & 1) * 2] = v;
    }
    __syncthreads();
    if (tid < C) {
      const double t = tot[tid], z = rz[tid];
      if (mode == 0) {
        scal[tid] = (float)((t > 0.0 && z > 0.0) ? z / t : 0.0);
      } else {
        if (mode == 1) scal[tid] = (float)(z > 0.0 ? t / z : 0.0);
        rz[tid] = t;
      }
    }
    __syncthreads();
  };

  // x = 0, r = b, z = M r, p = z, rz = r.z
  const float *dinv0 = S[0].dinv;
  float *r0 = S[0].b.own, *z0 = S[0].x.own, *t0 = S[0].t.own;
  const int own = f1 - f0;
  for (int i = tid; i < own; i += blockDim.x) {
    float bv[C], tv[C];
    const float d = dinv0[i];
#pragma unroll
    for (int c = 0; c < C; ++c) bv[c] = __ldg(A.rhs + (size_t)(f0 + i) * C + c), tv[c] = d * bv[c];
    store_row<C>(r0, (size_t)i, bv);
    if (nl > 1) store_row<C>(t0, (size_t)i, tv);
  }
  bar.sync();
  vcycle();
  dots(r0, z0);
  for (int i = tid; i < own; i += blockDim.x) {
    float zv[C];
    load_row<C>(z0, (size_t)i, zv);
    store_row<C>(vp.own, (size_t)i, zv);
  }
  bar.sync();
  scalars(2);
  for (int it = 0; it < A.iters; ++it) {
    for_rows<C, CLUSTER>(S[0].a, vp, nothing,
                         [&](int row, NoVals, const float (&acc)[C]) { store_row<C>(vq.own, (size_t)row, acc); });
    dots(vp.own, vq.own);
    bar.sync();
    scalars(0);
    // x += alpha p, r -= alpha q, and the next V-cycle's first sweep
    const bool more = it + 1 < A.iters;
    for (int i = tid; i < own; i += blockDim.x) {
      float pv[C], qv[C], rv[C], tv[C];
      load_row<C>(vp.own, (size_t)i, pv), load_row<C>(vq.own, (size_t)i, qv), load_row<C>(r0, (size_t)i, rv);
      const float d = dinv0[i];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        float *xo = A.sol + (size_t)(f0 + i) * C + c;
        *xo = fmaf(scal[c], pv[c], it == 0 ? 0.f : *xo);
        rv[c] = fmaf(-scal[c], qv[c], rv[c]);
        tv[c] = d * rv[c];
      }
      store_row<C>(r0, (size_t)i, rv);
      if (more && nl > 1) store_row<C>(t0, (size_t)i, tv);
    }
    if (!more) break;
    bar.sync();
    vcycle();
    dots(r0, z0);
    bar.sync();
    scalars(1);
    // p = z + beta p
    for (int i = tid; i < own; i += blockDim.x) {
      float zv[C], pv[C];
      load_row<C>(z0, (size_t)i, zv), load_row<C>(vp.own, (size_t)i, pv);
#pragma unroll
      for (int c = 0; c < C; ++c) pv[c] = fmaf(scal[c], pv[c], zv[c]);
      store_row<C>(vp.own, (size_t)i, pv);
    }
    bar.sync();
  }
  if (CLUSTER) bar.sync();  // no block leaves while another may read its shared memory
}

template <class T>
void up(DevBuf<T> &d, const std::vector<T> &v, cudaStream_t s) {
  d.alloc(std::max<size_t>(v.size(), 1));
  if (!v.empty()) d.upload(v.data(), v.size(), s);
}

// the FP64 setup's values rounded to the multigrid type
void up(DevBuf<mgreal> &d, const std::vector<double> &v, cudaStream_t s) {
  std::vector<mgreal> w(v.begin(), v.end());
  up(d, w, s);
}

// lanes per row: the smallest power of two (at most 32) that leaves each lane about four nonzeros
int lanes_per_row(const Csr &A) {
  const double mean = A.n > 0 ? (double)A.ptr[A.n] / A.n : 0.0;
  int t = 1;
  while (t < 32 && 4 * t < mean) t *= 2;
  return t;
}

}  // namespace

void AmgDevice::Mat::upload(const Csr &A, cudaStream_t s) {
  up(ptr, A.ptr, s);
  std::vector<int2> v(A.col.size());
  for (size_t i = 0; i < v.size(); ++i) {
    const mgreal a = (mgreal)A.val[i];
    int b;
    std::memcpy(&b, &a, sizeof(b));
    v[i] = make_int2(A.col[i], b);
  }
  up(cv, v, s);
  nnz = v.size();
  tpr = lanes_per_row(A);
}

void AmgDevice::upload(const AmgHost &h, cudaStream_t s) {
  size_t nl = h.A.size();
  if (nl > (size_t)kMaxLevels) fail(RS_INTERNAL, "Internal", "preconditioner", "too many multigrid levels");
  L.clear();
  L.resize(nl);
  for (size_t l = 0; l < nl; ++l) {
    Level &v = L[l];
    v.n = h.A[l].n;
    v.a.upload(h.A[l], s);
    up(v.dinv, h.dinv[l], s);
    if (l + 1 < nl) v.p.upload(h.P[l], s), v.r.upload(h.R[l], s);
    // the vectors, for the widest batch; level 0 lends its solution and right-hand side to the
    // conjugate gradients
    const size_t m = 12 * (size_t)v.n;
    v.b.alloc(m), v.res.alloc(m), v.t.alloc(m), v.x.alloc(m);
  }
  up(cinv, h.coarse_inv, s);
  const size_t m = 12 * (size_t)L[0].n;
  cg_p.alloc(m), cg_q.alloc(m);
  cg_part.alloc(2 * (size_t)kDotBlocks * 12);
  counter.alloc(1);
  RSG_CUDA("preconditioner", cudaMemsetAsync(counter.p, 0, sizeof(unsigned long long), s));
  if (!error) {
    RSG_CUDA("preconditioner", cudaHostAlloc((void **)&error, sizeof(int), cudaHostAllocMapped));
    *error = 0;
    RSG_CUDA("preconditioner", cudaHostGetDevicePointer((void **)&error_dev, error, 0));
  }
  // The blocks: one cluster of 16 when their shared memory holds all the matrices and vectors, else one
  // block per SM with the vectors in global memory, shared memory for the block's share of the
  // matrices with a tenth to spare for uneven rows. As many threads as the largest level gives lanes
  // per block. A preconditioner application on the grid, three vectors, with 256 threads / as many as the nine
  // columns' registers allow: 8,000 rows 0.78 / 0.78 ms, 25,600 rows 1.29 / 1.17, 102,400 rows 2.54 / 2.28; in the
  // cluster, one vector, with 256 / 512 / 1,024: 900 rows 0.43 / 0.43 / 0.43, 4,356 rows 0.73 / 0.65 / 0.62.
  int dev = 0, most = 0, sms = 0;
  RSG_CUDA("preconditioner", cudaGetDevice(&dev));
  RSG_CUDA("preconditioner", cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  RSG_CUDA("preconditioner", cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const int kOwn = 24576;  // the kernels' own (checked below)
  most -= kOwn;
  const void *cluster_fn = (const void *)pcg_kernel<3, true>;
  for (const void *fn : {(const void *)pcg_kernel<3, false>, (const void *)pcg_kernel<6, false>,
                         (const void *)pcg_kernel<9, false>, (const void *)pcg_kernel<12, false>, cluster_fn}) {
    cudaFuncAttributes fa;
    RSG_CUDA("preconditioner", cudaFuncGetAttributes(&fa, fn));
    if (fa.sharedSizeBytes > (size_t)kOwn) fail(RS_INTERNAL, "Internal", "preconditioner", "shared memory of the solve");
    RSG_CUDA("preconditioner", cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  }
  RSG_CUDA("preconditioner", cudaFuncSetAttribute(cluster_fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  size_t lanes = 0, bytes = 0;
  for (const Level &v : L) {
    lanes = std::max(lanes, (size_t)v.n * v.a.tpr);
    bytes += 8 * (v.a.nnz + v.p.nnz + v.r.nnz) + 16 * (size_t)v.n;
  }
  grid = std::min(sms, 1024);
  smem_bytes = (int)std::min<size_t>((size_t)most, bytes / grid * 11 / 10 + 8192) & ~15;
  threads = lanes > 256 * (size_t)grid ? 512 : 256;
  // the cluster: the largest share of the matrices of a block, and the vectors by their width
  const int n0 = L[0].n, chunk = (n0 + kDotBlocks - 1) / kDotBlocks;
  auto first = [&](size_t l, int b) {
    return l == 0 ? std::min(n0, kDotBlocks * b / kCluster * chunk) : (int)((long long)L[l].n * b / kCluster);
  };
  size_t mats = 0;
  for (int b = 0; b < kCluster; ++b) {
    size_t t = 0;
    for (size_t l = 0; l < nl; ++l) {
      const int r0 = first(l, b), r1 = first(l, b + 1);
      auto slice = [&](const Csr &m, int a, int e) { t += 8 * (size_t)(m.ptr[e] - m.ptr[a]) + 4 * (size_t)(e - a + 1) + 32; };
      if (l + 1 < nl || nl == 1) slice(h.A[l], r0, r1);
      if (l + 1 < nl) slice(h.P[l], r0, r1), slice(h.R[l], first(l + 1, b), first(l + 1, b + 1));
      else t += 4 * (size_t)(r1 - r0) * L[l].n + 16;
      t += 4 * (size_t)(r1 - r0) + 16;
    }
    mats = std::max(mats, t);
  }
  size_t rows = 6 * (size_t)((kDotBlocks + kCluster - 1) / kCluster) * chunk;  // rows of the vectors in a block
  for (size_t l = 1; l < nl; ++l) rows += 4 * (size_t)((L[l].n + kCluster - 1) / kCluster);
  cluster_threads = lanes > 512 * (size_t)kCluster ? 1024 : (lanes > 256 * (size_t)kCluster ? 512 : 256);
  const size_t need = (mats + rows * 4 * kStride<3> + 15) & ~size_t(15);
  cluster_smem = need <= (size_t)most ? (int)need : 0;
  if (cluster_smem > 0) {  // can a cluster of that many blocks be resident?
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config(s, at);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, cluster_fn, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      cluster_smem = 0;
    }
  }
}

cudaLaunchConfig_t AmgDevice::cluster_config(cudaStream_t s, cudaLaunchAttribute &at) const {
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kCluster, at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kCluster), cfg.blockDim = dim3((unsigned)cluster_threads);
  cfg.dynamicSmemBytes = (size_t)cluster_smem, cfg.stream = s;
  cfg.attrs = &at, cfg.numAttrs = 1;
  return cfg;
}

void AmgDevice::check() {
  if (!error || *(volatile int *)error == 0) return;
  *(volatile int *)error = 0;  // every block still arrived at every barrier: the next solve starts clean
  fail(RS_GPU, "Gpu", "preconditioner", "a multigrid solve gave up waiting for its blocks");
}

template <int C>
void AmgDevice::launch(rs_ctx *ctx, const mgreal *b, mgreal *x, int iters) {
  CgArgs A;
  A.nl = (int)L.size(), A.iters = iters;
  for (size_t l = 0; l < L.size(); ++l) {
    Level &v = L[l];
    auto mat = [](const Mat &m) { return DevMat{m.ptr.p, m.cv.p, m.tpr}; };
    A.l[l] = DevLevel{v.n, mat(v.a), mat(v.p), mat(v.r), v.dinv.p, v.x.p, v.b.p, v.res.p, v.t.p};
  }
  A.cinv = cinv.p, A.rhs = b, A.sol = x;
  A.p = cg_p.p, A.q = cg_q.p, A.part = cg_part.p, A.counter = counter.p;
  A.error = error_dev, A.polls = wait_polls, A.smem_bytes = smem_bytes;
  if (C == 3 && cluster_smem > 0) {
    A.smem_bytes = cluster_smem;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config(ctx->stream, at);
    RSG_CUDA("preconditioner", cudaLaunchKernelEx(&cfg, pcg_kernel<3, true>, A));
  } else {
    void *args[] = {&A};
    RSG_CUDA("preconditioner",
             cudaLaunchCooperativeKernel((const void *)pcg_kernel<C, false>, dim3((unsigned)grid),
                                         dim3((unsigned)std::min(threads, kMaxThreads<C, false>)), args,
                                         (size_t)smem_bytes, ctx->stream));
  }
  RSG_LAUNCHED(ctx, "pcg");
}

void AmgDevice::pcg(rs_ctx *ctx, const mgreal *b, mgreal *x, int C, int iters) {
  check();
  if (C > 12) fail(RS_INTERNAL, "Internal", "preconditioner", "at most 12 multigrid columns");
  switch (C) {
    case 3: launch<3>(ctx, b, x, iters); break;
    case 6: launch<6>(ctx, b, x, iters); break;
    case 9: launch<9>(ctx, b, x, iters); break;
    case 12: launch<12>(ctx, b, x, iters); break;
    default: fail(RS_INTERNAL, "Internal", "preconditioner", "multigrid width 3, 6, 9 or 12");
  }
}

AmgDevice::~AmgDevice() {
  if (error) cudaFreeHost(error);
}

}  // namespace rsg
