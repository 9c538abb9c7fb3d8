// Supermesh kernels for sm_100a.
//
//   K1  k_prep          element gather, FP64/FP32 boxes, measures, tolerances,
//                       B-element clip setup (lines / unit-normal planes)
//   K1b k_root_box      root box;  k_morton  Morton keys and the sort's
//                       digit counts
//   K2  radix sort      stable LSD, 8-bit digits, warp-match ranking; one
//                       kernel per pass with decoupled look-back
//                       (k_radix_onesweep)
//   K3  k_tree_build    four-wide hierarchy of outward-rounded FP32 boxes
//                       over the sorted leaves
//   K4  k_query         depth-first traversal per A element, four children a
//                       visit (k_query_warp: a warp per element, 32), exact
//                       strict box test at the leaves; the count pass caches
//                       rows, k_fill_from_cache copies
//   K5  k_clip_tris     one candidate pair per thread, polygon clipped in
//                       place in shared memory, FP64 Sutherland-Hodgman
//   K6  k_prefilter_tets two exact early-outs and the no-op plane mask;
//                       k_clip_tets_bf breadth-first clipping, a warp per
//                       batch of pairs, templated on what it does with the
//                       kept tets (measures of small and medium passes;
//                       explicit pairs' output tets; the supermesh's tets at
//                       their offsets; the P1 quadrature);
//                       k_clip_tets_ix depth-first clipping, a lane per pair,
//                       over point indices with a refill pipeline (measures
//                       of large passes; six planes: hexahedra)
//   K7  compensated reductions (per-block (sum, err), then final; per mesh
//                       pair for the batched path)
//   K8  P1-P1 mixed mass blocks + u^T M v: 2D k_p1_mass (blocks), k_p1_uv
//                       (u^T M v alone); 3D the early-out pass and
//                       k_clip_tets_bf with the quadrature sink;
//                       k_p2_inner  P2 inner product
//   K9  1D sort finder  k_prep_1d, 64-bit stable sort, max segment tree,
//                       k_rows_1d, k_sweep_1d, k_emit_1d;  k_clip_intervals
//   K10 explicit pairs  k_pairs_tris / _tets and the mixed element pairs
//                       (intervals, tri-quad, quad-quad, tet-hex, hex-hex);
//                       large tet-tet batches: k_pairs_early (setup and
//                       early-outs), tet-hex: k_setup_hex_pairs, then K6
//   K13 supermesh elements  K6's emit pass (3D), k_tris_emit (2D)
//
// Everything FP64 is compiled with -fmad=false so that each +,-,*,/ is a
// separately rounded IEEE operation, matching libsupermesh's gfortran build.
#include "lsm_geom.cuh"
#include "lsm_kernels.h"
#include "lsm_sched.h"

#include <cuda/atomic>

#include <cfloat>
#include <cstdio>
#include <cstdlib>

namespace lsm {

namespace {
unsigned long long g_launches = 0;
}  // namespace

unsigned long long launches() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }

namespace {
int g_tri_bps = 8;
int g_query_block = 128;
int g_leaf_bucket = 1;
}  // namespace

int tri_blocks_per_sm() { return g_tri_bps; }
void set_tri_blocks_per_sm(int v) { g_tri_bps = v; }
int query_block() { return g_query_block; }
void set_query_block(int v) { g_query_block = v; }
int leaf_bucket() { return g_leaf_bucket; }
void set_leaf_bucket(int v) { g_leaf_bucket = v; }

void count_launch(int n) { __atomic_fetch_add(&g_launches, (unsigned long long)n, __ATOMIC_RELAXED); }

int sm_count() {
  static int cached = -1;
  if (cached < 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached = n;
  }
  return cached;
}

int grid_for(int64_t n, int block, int per_sm) {
  int64_t need = (n + block - 1) / block;
  int64_t cap = (int64_t)sm_count() * per_sm;
  if (need < 1) need = 1;
  return (int)(need < cap ? need : cap);
}

namespace {

// Compensated (sum, err) pair helpers: TwoSum-based merge.
__device__ __forceinline__ void cs_add(double& sum, double& err, double x) {
  // Kahan step (Precision.F90:89-95)
  const double cx = err + x;
  const double s = sum + cx;
  err = (sum - s) + cx;
  sum = s;
}

__device__ __forceinline__ void two_sum_merge(double& s, double& e, double s2, double e2) {
  const double t = s + s2;
  const double bp = t - s;
  const double err = (s - (t - bp)) + (s2 - bp);
  s = t;
  e = e + e2 + err;
}

template <int BLOCK>
__device__ void block_reduce_partial(double sum, double err, unsigned long long ni, unsigned long long no,
                                     Partial* out) {
  __shared__ double ss[BLOCK / 32], se[BLOCK / 32];
  __shared__ unsigned long long si[BLOCK / 32], so[BLOCK / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double s2 = __shfl_down_sync(0xffffffffu, sum, o);
    const double e2 = __shfl_down_sync(0xffffffffu, err, o);
    two_sum_merge(sum, err, s2, e2);
    ni += __shfl_down_sync(0xffffffffu, ni, o);
    no += __shfl_down_sync(0xffffffffu, no, o);
  }
  if (lane == 0) {
    ss[wid] = sum;
    se[wid] = err;
    si[wid] = ni;
    so[wid] = no;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Partial p{ss[0], se[0], si[0], so[0]};
    for (int w = 1; w < BLOCK / 32; ++w) {
      two_sum_merge(p.sum, p.err, ss[w], se[w]);
      p.n_int += si[w];
      p.n_out += so[w];
    }
    *out = p;
  }
}

}  // namespace

// ======================================================================
// K1: element prep
// ======================================================================
// One element of the prep: gather, boxes, measure/tolerance, clip setup.
// LOC = DIM + 1 for simplices; other LOC (quads, hexes) only get boxes,
// which is all the candidate search needs.
template <int DIM, int LOC, typename IDX>
__device__ __forceinline__ void prep_element(int64_t e, const double* __restrict__ pos,
                                             const IDX* __restrict__ row, int64_t nnodes, double* coords,
                                             double* box64, float* box32, double* tolv, double* setup,
                                             int* bad, double* faces = nullptr, double* screen = nullptr) {
  constexpr bool SIMPLEX = LOC == DIM + 1;
  double v[LOC * DIM];
  bool ok = true;
#pragma unroll
  for (int k = 0; k < LOC; ++k) {
    int64_t node = (int64_t)row[k];
    if (node < 0 || node >= nnodes) {
      ok = false;
      node = 0;
    }
#pragma unroll
    for (int c = 0; c < DIM; ++c) v[k * DIM + c] = pos[node * DIM + c];
  }
  if (!ok) atomicExch(bad, 1);
  if (coords) {
    static_assert((LOC * DIM) % 2 == 0, "element rows of an even number of doubles");
#pragma unroll
    for (int j = 0; j < LOC * DIM; j += 2) st2(coords + e * LOC * DIM + j, v[j], v[j + 1]);
  }
  double lo[DIM], hi[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) lo[c] = hi[c] = v[c];
#pragma unroll
  for (int k = 1; k < LOC; ++k)
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      lo[c] = fmin(lo[c], v[k * DIM + c]);
      hi[c] = fmax(hi[c], v[k * DIM + c]);
    }
  if (box64) {
    double* o = box64 + e * 2 * DIM;
    if (DIM == 3) {
      st2(o, lo[0], lo[1]);
      st2(o + 2, lo[DIM - 1], hi[0]);
      st2(o + 4, hi[1], hi[DIM - 1]);
    } else {
      st2(o, lo[0], lo[1]);
      st2(o + 2, hi[0], hi[1]);
    }
  }
  if (box32) {
    float4 l = make_float4(0.f, 0.f, 0.f, 0.f), h = make_float4(0.f, 0.f, 0.f, 0.f);
    l.x = __double2float_rd(lo[0]);
    l.y = __double2float_rd(lo[1]);
    h.x = __double2float_ru(hi[0]);
    h.y = __double2float_ru(hi[1]);
    if (DIM == 3) {
      l.z = __double2float_rd(lo[DIM - 1]);
      h.z = __double2float_ru(hi[DIM - 1]);
    }
    reinterpret_cast<float4*>(box32)[2 * e] = l;
    reinterpret_cast<float4*>(box32)[2 * e + 1] = h;
  }
  if (!SIMPLEX) return;
  double meas;
  Tet t;
  if (DIM == 2) {
    meas = tri_area(v[0], v[1], v[2], v[3], v[4], v[5]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      t.x[k] = v[k * DIM + 0];
      t.y[k] = v[k * DIM + 1];
      t.z[k] = v[k * DIM + DIM - 1];
    }
    meas = tet_volume_v4(t);
  }
  const double tol = 10.0 * spacing(meas);
  if (tolv) tolv[e] = tol;
  if (setup) {
    if (DIM == 2) {
      double* o = setup + e * kSetup2;
#pragma unroll
      for (int i = 0; i < 3; ++i) st2(o + 2 * i, v[2 * i], v[2 * i + 1]);
      st2(o + 6, tol, tri_flipped(v) ? 1.0 : -1.0);
    } else {
      Planes P;
      tet_planes(t, P);
      double* o = setup + e * kSetup3;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        st2(o + 4 * i, P.nx[i], P.ny[i]);
        st2(o + 4 * i + 2, P.nz[i], P.c[i]);
      }
      st2(o + 16, tol, 0.0);
      st2(o + 18, 0.0, 0.0);
      if (screen) tet_screen_b(t, P, screen + e * kScreen3);
    }
  }
  if constexpr (DIM == 3) {
    if (faces) tet_faces_screen(t, faces + e * kScreen3);
  }
}

template <int DIM, int LOC, typename IDX>
__global__ void k_prep(int64_t nel, const double* __restrict__ pos, const IDX* __restrict__ en,
                       double* coords, double* box64, float* box32, double* tolv, double* setup,
                       int* bad, int64_t nnodes, double* faces, double* screen) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nel;
       e += (int64_t)gridDim.x * blockDim.x)
    prep_element<DIM, LOC, IDX>(e, pos, en + e * LOC, nnodes, coords, box64, box32, tolv, setup, bad, faces,
                                screen);
}

// Batched prep over the concatenation of many meshes.  Element e belongs to
// mesh p = the last p with elem_off[p] <= e; its nodes are read through the
// per-mesh pointer tables.  pair_of[e] receives p.
__device__ __forceinline__ int find_mesh(const int64_t* __restrict__ off, int nm, int64_t e) {
  int lo = 0, hi = nm;  // off[lo] <= e < off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= e)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

template <int DIM, typename IDX>
__global__ void k_prep_batched(int64_t nel, int nm, const int64_t* __restrict__ elem_off,
                               const unsigned long long* __restrict__ pos_ptr,
                               const unsigned long long* __restrict__ en_ptr,
                               const int64_t* __restrict__ nnodes, double* coords, double* box64,
                               float* box32, double* tolv, double* setup, int32_t* pair_of, int* bad,
                               double* faces, double* screen) {
  constexpr int LOC = DIM + 1;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nel;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int p = find_mesh(elem_off, nm, e);
    const int64_t local = e - elem_off[p];
    const double* pos = reinterpret_cast<const double*>(pos_ptr[p]);
    const IDX* en = reinterpret_cast<const IDX*>(en_ptr[p]);
    prep_element<DIM, LOC, IDX>(e, pos, en + local * LOC, nnodes[p], coords, box64, box32, tolv, setup, bad,
                                faces, screen);
    pair_of[e] = p;
  }
}

template <int DIM, int LOC>
static void prep_dispatch_idx(int g, int B, cudaStream_t s, int64_t nel, const double* pos,
                              const void* enlist, int idx_bytes, double* coords, double* box64,
                              float* box32, double* tolv, double* setup, int* bad, int64_t nnodes,
                              double* faces, double* screen) {
  count_launch();
  if (idx_bytes == 4)
    k_prep<DIM, LOC, int32_t><<<g, B, 0, s>>>(nel, pos, (const int32_t*)enlist, coords, box64, box32, tolv, setup, bad,
                                              nnodes, faces, screen);
  else
    k_prep<DIM, LOC, int64_t><<<g, B, 0, s>>>(nel, pos, (const int64_t*)enlist, coords, box64, box32, tolv, setup, bad,
                                              nnodes, faces, screen);
}

cudaError_t launch_prep(int dim, int loc, int64_t nel, const double* pos, const void* enlist, int idx_bytes,
                        double* coords, double* box64, float* box32, double* tolv, double* setup,
                        int* bad_index, int64_t nnodes, cudaStream_t s, double* faces, double* screen) {
  if (nel <= 0) return cudaSuccess;
  const int B = 256;
  const int g = grid_for(nel, B, 8);
  if (dim == 2 && loc == 3)
    prep_dispatch_idx<2, 3>(g, B, s, nel, pos, enlist, idx_bytes, coords, box64, box32, tolv, setup, bad_index, nnodes,
                            nullptr, nullptr);
  else if (dim == 2 && loc == 4)
    prep_dispatch_idx<2, 4>(g, B, s, nel, pos, enlist, idx_bytes, coords, box64, box32, tolv, setup, bad_index, nnodes,
                            nullptr, nullptr);
  else if (dim == 3 && loc == 4)
    prep_dispatch_idx<3, 4>(g, B, s, nel, pos, enlist, idx_bytes, coords, box64, box32, tolv, setup, bad_index, nnodes,
                            faces, screen);
  else if (dim == 3 && loc == 8)
    prep_dispatch_idx<3, 8>(g, B, s, nel, pos, enlist, idx_bytes, coords, box64, box32, tolv, setup, bad_index, nnodes,
                            nullptr, nullptr);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_prep_batched(int dim, int64_t nel, int nm, const int64_t* elem_off,
                                const unsigned long long* pos_ptr, const unsigned long long* en_ptr,
                                const int64_t* nnodes, int idx_bytes, double* coords, double* box64,
                                float* box32, double* tolv, double* setup, int32_t* pair_of, int* bad,
                                cudaStream_t s, double* faces, double* screen) {
  if (nel <= 0) return cudaSuccess;
  const int B = 256;
  const int g = grid_for(nel, B, 8);
  count_launch();
  if (dim == 2 && idx_bytes == 4)
    k_prep_batched<2, int32_t><<<g, B, 0, s>>>(nel, nm, elem_off, pos_ptr, en_ptr, nnodes, coords, box64, box32,
                                                 tolv, setup, pair_of, bad, nullptr, nullptr);
  else if (dim == 2)
    k_prep_batched<2, int64_t><<<g, B, 0, s>>>(nel, nm, elem_off, pos_ptr, en_ptr, nnodes, coords, box64, box32,
                                                 tolv, setup, pair_of, bad, nullptr, nullptr);
  else if (idx_bytes == 4)
    k_prep_batched<3, int32_t><<<g, B, 0, s>>>(nel, nm, elem_off, pos_ptr, en_ptr, nnodes, coords, box64, box32,
                                                 tolv, setup, pair_of, bad, faces, screen);
  else
    k_prep_batched<3, int64_t><<<g, B, 0, s>>>(nel, nm, elem_off, pos_ptr, en_ptr, nnodes, coords, box64, box32,
                                                 tolv, setup, pair_of, bad, faces, screen);
  return cudaGetLastError();
}

// ======================================================================
// K1b: root box and Morton keys
// ======================================================================
template <int DIM>
__global__ void __launch_bounds__(256) k_root_box(int64_t nel, const double* __restrict__ box64, double* partial,
                                                  double* root, unsigned* ticket) {
  double lo[DIM], hi[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    lo[c] = DBL_MAX;
    hi[c] = -DBL_MAX;
  }
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nel;
       e += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      lo[c] = fmin(lo[c], box64[e * 2 * DIM + c]);
      hi[c] = fmax(hi[c], box64[e * 2 * DIM + DIM + c]);
    }
  }
  __shared__ double sl[8][DIM], sh[8][DIM];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // the block's box, then, in the block that finishes last (*ticket, zero
  // before the launch), the box of all blocks' boxes
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        lo[c] = fmin(lo[c], __shfl_down_sync(0xffffffffu, lo[c], o));
        hi[c] = fmax(hi[c], __shfl_down_sync(0xffffffffu, hi[c], o));
      }
    if (lane == 0)
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        sl[wid][c] = lo[c];
        sh[wid][c] = hi[c];
      }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w)
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
          lo[c] = fmin(lo[c], sl[w][c]);
          hi[c] = fmax(hi[c], sh[w][c]);
        }
      double* o = pass == 0 ? partial + (int64_t)blockIdx.x * 2 * DIM : root;
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        o[c] = lo[c];
        o[DIM + c] = hi[c];
      }
      if (pass == 0) {
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        __threadfence();
      }
    }
    __syncthreads();
    if (pass == 1 || !s_last) return;
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      lo[c] = DBL_MAX;
      hi[c] = -DBL_MAX;
    }
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        lo[c] = fmin(lo[c], __ldcg(partial + b * 2 * DIM + c));
        hi[c] = fmax(hi[c], __ldcg(partial + b * 2 * DIM + DIM + c));
      }
  }
}

cudaError_t launch_root_box(int dim, int64_t nel, const double* box64, double* partial,
                            int partial_cap, double* rootbox, unsigned* ticket, cudaStream_t s) {
  const int B = 256;
  int g = grid_for(nel, B, 2);
  if (g > partial_cap) g = partial_cap;
  count_launch();
  if (dim == 2)
    k_root_box<2><<<g, B, 0, s>>>(nel, box64, partial, rootbox, ticket);
  else
    k_root_box<3><<<g, B, 0, s>>>(nel, box64, partial, rootbox, ticket);
  return cudaGetLastError();
}

__device__ __forceinline__ uint32_t spread2(uint32_t x) {  // 16 bits -> even bits
  x &= 0xffffu;
  x = (x | (x << 8)) & 0x00ff00ffu;
  x = (x | (x << 4)) & 0x0f0f0f0fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}

__device__ __forceinline__ uint32_t spread3(uint32_t x) {  // 10 bits -> every 3rd bit
  x &= 0x3ffu;
  x = (x | (x << 16)) & 0x030000ffu;
  x = (x | (x << 8)) & 0x0300f00fu;
  x = (x | (x << 4)) & 0x030c30c3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

// counts: the sort's digit counts of all four passes (k_radix_counts).
template <int DIM>
__global__ void __launch_bounds__(256) k_morton(int64_t nel, const double* __restrict__ box64,
                                                const double* __restrict__ root, uint32_t* keys, int32_t* vals,
                                                uint32_t* counts) {
  __shared__ uint32_t h[4][256];
  for (int i = threadIdx.x; i < 4 * 256; i += 256) (&h[0][0])[i] = 0;
  __syncthreads();
  constexpr double kScale = DIM == 2 ? 65536.0 : 1024.0;
  constexpr uint32_t kMax = DIM == 2 ? 65535u : 1023u;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nel;
       e += (int64_t)gridDim.x * blockDim.x) {
    uint32_t q[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      const double mid = 0.5 * (box64[e * 2 * DIM + c] + box64[e * 2 * DIM + DIM + c]);
      const double ext = root[DIM + c] - root[c];
      double u = ext > 0.0 ? (mid - root[c]) / ext : 0.0;
      u = fmin(fmax(u, 0.0), 1.0);
      const double f = u * kScale;
      q[c] = f >= (double)kMax ? kMax : (uint32_t)f;
    }
    uint32_t key;
    if (DIM == 2)
      key = (spread2(q[1]) << 1) | spread2(q[0]);
    else
      key = (spread3(q[DIM - 1]) << 2) | (spread3(q[1]) << 1) | spread3(q[0]);
    keys[e] = key;
    vals[e] = (int32_t)e;
#pragma unroll
    for (int p = 0; p < 4; ++p) atomicAdd(&h[p][(key >> (8 * p)) & 255u], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * 256; i += 256) {
    const uint32_t c = (&h[0][0])[i];
    if (c) atomicAdd(&counts[i], c);
  }
}

// ======================================================================
// K2: stable LSD radix sort (8-bit digits, one kernel per pass)
// ======================================================================
namespace {
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;                           // per thread
constexpr int kSortTile = kSortThreads * kSortItems;  // 2048 keys per block
constexpr int kWarpTile = 32 * kSortItems;             // contiguous per warp
constexpr int kLookBack = 8;                            // blocks looked back over at once
}  // namespace

// Single-pass digit binning per pass ("onesweep"): one kernel counts every
// digit of every pass over all keys; each pass is then one kernel in which
// block b (in ticket order) ranks its 2048 keys, publishes its digit counts,
// looks back over the blocks before it for their prefix (decoupled
// look-back: a block publishes its local count first and its inclusive
// prefix once known) and scatters.  Stable: ranks follow key order within a
// block and blocks follow key order.
//
// Scratch layout (uint32, radix_hist_entries(n)): counts[4][256] |
// tickets[4] | err | pad | status[4][nblocks][256].  A status word holds a
// 2-bit flag (0 not ready, 1 local count, 2 inclusive prefix) over a 30-bit
// count (n < 2^30).  Waits are bounded: a block that gives up sets err and
// treats the missing prefix as 0 (wrong order, never a hang); forward
// progress does not need the bound, since a block only waits for blocks
// that took earlier tickets and are running or done.  After that some keys
// overwrite others and a later pass reads what the gaps held, so positions
// are checked, and k_sort_repair (or k_tree_build, which reads the same word)
// turns the output back into a permutation (identity values, equal keys) so
// that the kernels after the sort never read an element number that does not
// exist.  The caller sees err and reports the failure.
//
// Test hooks (process-wide, off by default): the bound of each wait
// (set_sort_spin_limit) and one block per pass that never publishes its
// counts (set_sort_stall_block, sorts given an err word only), which makes
// the waits of the blocks after it run out.
namespace {
constexpr int kSortPassesMax = 4;
constexpr int kSortHdr = kSortPassesMax * 256 + 8;
constexpr uint32_t kFlagLocal = 1u << 30, kFlagIncl = 2u << 30, kFlagMask = 3u << 30;
}  // namespace

namespace {
int g_sort_spin_limit = 1 << 22;
int g_sort_stall = -1;
}  // namespace

void set_sort_spin_limit(int v) { g_sort_spin_limit = v > 0 ? v : 1; }
int sort_spin_limit() { return g_sort_spin_limit; }
void set_sort_stall_block(int b) { g_sort_stall = b >= 1 ? b : -1; }
int sort_stall_block() { return g_sort_stall; }

int64_t radix_hist_entries(int64_t n) {
  const int64_t nb = (n + kSortTile - 1) / kSortTile;
  return kSortHdr + (int64_t)kSortPassesMax * 256 * (nb > 0 ? nb : 1);
}

// Words of the scratch that a sort of n keys in `passes` passes needs zeroed.
static int64_t radix_zeros(int64_t n, int passes) {
  return kSortHdr + (int64_t)passes * 256 * ((n + kSortTile - 1) / kSortTile);
}

cudaError_t launch_morton(int dim, int64_t nel, const double* box64, const double* rootbox, uint32_t* keys,
                          int32_t* vals, uint32_t* hist, cudaStream_t s) {
  if (nel <= 0) return cudaSuccess;
  cudaMemsetAsync(hist, 0, sizeof(uint32_t) * radix_zeros(nel, kSortPassesMax), s);
  const int g = grid_for(nel, 256, 8);
  count_launch();
  if (dim == 2)
    k_morton<2><<<g, 256, 0, s>>>(nel, box64, rootbox, keys, vals, hist);
  else
    k_morton<3><<<g, 256, 0, s>>>(nel, box64, rootbox, keys, vals, hist);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(kSortThreads) k_radix_counts(int64_t n, int passes,
                                                               const uint32_t* __restrict__ keys, uint32_t* counts) {
  __shared__ uint32_t h[kSortPassesMax][256];
  for (int i = threadIdx.x; i < kSortPassesMax * 256; i += blockDim.x) (&h[0][0])[i] = 0;
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = keys[i];
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (8 * p)) & 255u], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) {
    const uint32_t v = (&h[0][0])[i];
    if (v) atomicAdd(&counts[i], v);
  }
}

__global__ void __launch_bounds__(kSortThreads) k_radix_onesweep(int64_t n, int shift,
                                                                 const uint32_t* __restrict__ keys_in,
                                                                 const int32_t* __restrict__ vals_in,
                                                                 uint32_t* keys_out, int32_t* vals_out,
                                                                 const uint32_t* __restrict__ counts,
                                                                 uint32_t* status, uint32_t* ticket,
                                                                 uint32_t* err, int spin_limit, int stall) {
  __shared__ uint32_t wh[kSortWarps][256];
  __shared__ uint32_t base_s[256];
  __shared__ uint32_t wt[kSortWarps];
  __shared__ int bid_s;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  if (threadIdx.x == 0) bid_s = (int)atomicAdd(ticket, 1u);
  for (int i = lane; i < 256; i += 32) wh[wid][i] = 0;
  __syncthreads();
  const int b = bid_s;
  const int64_t base = (int64_t)b * kSortTile + (int64_t)wid * kWarpTile;
  const uint32_t digit_count = counts[threadIdx.x];
  uint32_t k[kSortItems], rank[kSortItems];
  int32_t v[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int64_t i = base + r * 32 + lane;
    k[r] = i < n ? keys_in[i] : 0u;
    v[r] = i < n ? vals_in[i] : 0;
  }
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    // rank among the warp's keys of the same digit, in key order
    const int dg = base + r * 32 + lane < n ? (int)((k[r] >> shift) & 255u) : 256;
    const unsigned peers = __match_any_sync(0xffffffffu, dg);
    if (dg < 256) rank[r] = wh[wid][dg] + __popc(peers & lt);
    __syncwarp();
    if (dg < 256 && (peers & lt) == 0) wh[wid][dg] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // thread d: this block's count of digit d, published, then the prefix of
  // the blocks before it; the warps' offsets within the block
  const int d = threadIdx.x;  // blockDim.x == 256
  uint32_t local = 0;
  for (int w = 0; w < kSortWarps; ++w) local += wh[w][d];
  cuda::atomic_ref<uint32_t, cuda::thread_scope_device> mine(status[(int64_t)b * 256 + d]);
  const bool publish = b != stall;
  if (publish) mine.store((b == 0 ? kFlagIncl : kFlagLocal) | local, cuda::memory_order_relaxed);
  // (kLookBack blocks' words at once: with all blocks of a pass resident the
  // chain of single look-backs was most of its time)
  uint32_t prefix = 0;
  bool more = true;
  for (int j = b - 1; more && j >= 0; j -= kLookBack) {
    uint32_t w[kLookBack];
#pragma unroll
    for (int q = 0; q < kLookBack; ++q) {
      w[q] = kFlagIncl;
      if (j - q >= 0)
        w[q] = cuda::atomic_ref<uint32_t, cuda::thread_scope_device>(status[(int64_t)(j - q) * 256 + d])
                   .load(cuda::memory_order_relaxed);
    }
#pragma unroll
    for (int q = 0; q < kLookBack; ++q) {
      if (!more) continue;
      uint32_t x = w[q];
      if ((x & kFlagMask) == 0) {
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device> st(status[(int64_t)(j - q) * 256 + d]);
        x = st.load(cuda::memory_order_relaxed);
        for (int spin = 0; (x & kFlagMask) == 0; ++spin) {
          if (spin > spin_limit) {
            atomicExch(err, 1u);
            x = kFlagIncl;
            break;
          }
          __nanosleep(64);
          x = st.load(cuda::memory_order_relaxed);
        }
      }
      prefix += x & ~kFlagMask;
      more = (x & kFlagMask) != kFlagIncl;
    }
  }
  if (b > 0 && publish) mine.store(kFlagIncl | (prefix + local), cuda::memory_order_relaxed);
  // global start of digit d: exclusive scan of the pass's digit counts
  {
    const uint32_t c = digit_count;
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) wt[wid] = inc;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < wid; ++w) before += wt[w];
    base_s[d] = before + inc - c + prefix;
  }
  __syncthreads();
  {
    uint32_t run = base_s[d];
    for (int w = 0; w < kSortWarps; ++w) {
      const uint32_t c = wh[w][d];
      wh[w][d] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    if (base + r * 32 + lane < n) {
      const uint32_t pos = wh[wid][(k[r] >> shift) & 255u] + rank[r];
      if (pos < n) {  // (always, unless a wait gave up)
        keys_out[pos] = k[r];
        vals_out[pos] = v[r];
      }
    }
  }
}

// After a sort whose look-back gave up (*err != 0): identity values and
// equal keys, a permutation that every later kernel can read safely.
__global__ void k_sort_repair(int64_t n, const uint32_t* __restrict__ err, uint32_t* keys, int32_t* vals) {
  if (*err == 0u) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    keys[i] = 0u;
    vals[i] = (int32_t)i;
  }
}

cudaError_t radix_sort_pairs(int64_t n, int bits, uint32_t* keys, int32_t* vals, uint32_t* keys_tmp,
                             int32_t* vals_tmp, uint32_t* hist, cudaStream_t s, int* err, bool counted,
                             bool repair) {
  if (n <= 1) return cudaSuccess;
  if (n >= (int64_t)1 << 30 || bits > 32) return cudaErrorInvalidValue;
  const int nb = (int)((n + kSortTile - 1) / kSortTile);
  const int passes = (bits + 7) / 8;
  uint32_t* counts = hist;
  uint32_t* tickets = hist + kSortPassesMax * 256;
  uint32_t* errw = err ? reinterpret_cast<uint32_t*>(err) : tickets + kSortPassesMax;
  uint32_t* status = hist + kSortHdr;
  if (!counted) cudaMemsetAsync(hist, 0, sizeof(uint32_t) * radix_zeros(n, passes), s);
  uint32_t *ki = keys, *ko = keys_tmp;
  int32_t *vi = vals, *vo = vals_tmp;
  count_launch(passes + !counted);
  if (!counted) k_radix_counts<<<grid_for(n, kSortThreads, 4), kSortThreads, 0, s>>>(n, passes, ki, counts);
  for (int p = 0; p < passes; ++p) {
    k_radix_onesweep<<<nb, kSortThreads, 0, s>>>(n, 8 * p, ki, vi, ko, vo, counts + 256 * p,
                                                 status + (int64_t)p * 256 * nb, tickets + p, errw,
                                                 g_sort_spin_limit, err ? g_sort_stall : -1);
    uint32_t* tk = ki;
    ki = ko;
    ko = tk;
    int32_t* tv = vi;
    vi = vo;
    vo = tv;
  }
  if (ki != keys) {
    cudaMemcpyAsync(keys, ki, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s);
    cudaMemcpyAsync(vals, vi, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s);
  }
  if (err && repair) {
    count_launch();
    k_sort_repair<<<grid_for(n, 256, 4), 256, 0, s>>>(n, errw, keys, vals);
  }
  return cudaGetLastError();
}

// ======================================================================
// K3: four-wide box hierarchy over the sorted leaves
// ======================================================================
// Level 0 is the leaves in Morton order; node j of level l+1 holds nodes 4j ..
// 4j+3 of level l, up to the first level of at most four nodes.  A group of
// four siblings is one record of their outward-rounded FP32 boxes, component
// by component (lo.x of the four, lo.y, .., hi.z: six float4 in 3D, four in
// 2D), so that a visit is one round of independent 16-byte loads and decides
// four children at once; nodes past the end have empty boxes.  The search
// waits for its chain of dependent visits, and this takes about a third of
// those of a binary hierarchy with escape links, one node at a time; the
// hierarchy follows from the sorted order alone, where the binary one was
// built by two searches per node and a bottom-up merge over one counter per
// node.  Search of tet3d_graded_55x51 / tri2d_777x1024_rot7: 1.85 -> 1.76 / 1.20 -> 0.76 ms.
template <int DIM>
__device__ __forceinline__ void tree_put(float* __restrict__ rec, int64_t node, const float (&lo)[3],
                                         const float (&hi)[3]) {
  float* r = rec + (node >> 2) * (8 * DIM) + (node & 3);
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    r[4 * c] = lo[c];
    r[4 * (DIM + c)] = hi[c];
  }
}

template <int DIM>
__device__ __forceinline__ void tree_join(const float* __restrict__ rec, int64_t group, float (&lo)[3],
                                          float (&hi)[3]) {
  const float4* r = reinterpret_cast<const float4*>(rec + group * (8 * DIM));
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    const float4 l = __ldcg(r + c), h = __ldcg(r + DIM + c);
    lo[c] = fminf(fminf(l.x, l.y), fminf(l.z, l.w));
    hi[c] = fmaxf(fmaxf(h.x, h.y), fmaxf(h.z, h.w));
  }
}

constexpr int kTreeBlock = 256;  // threads, one group of leaves each

// Levels 0 to 5 of the block's 1024 leaves; the block that finishes last
// (*ticket, zero before the launch) builds the levels above.  *sort_err: the
// sort gave up (see k_sort_repair, whose work on vals is done here).
template <int DIM>
__global__ void __launch_bounds__(kTreeBlock) k_tree_build(const __grid_constant__ Tree T, int32_t* vals,
                                                           const float4* __restrict__ box32, float* rec,
                                                           unsigned* ticket, const int* __restrict__ sort_err) {
  __shared__ float sl[kTreeBlock][DIM], sh[kTreeBlock][DIM];
  __shared__ bool s_last;
  const float inf = __int_as_float(0x7f800000);
  const int t = threadIdx.x;
  const int64_t g = (int64_t)blockIdx.x * kTreeBlock + t;
  const int64_t groups0 = T.off[1];
  float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
  if (g < groups0) {
    float4 L[4], H[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      L[k] = make_float4(inf, inf, inf, 0.0f);
      H[k] = make_float4(-inf, -inf, -inf, 0.0f);
      if (4 * g + k < T.n) {
        // (after a sort whose look-back gave up, any permutation will do: the
        // call reports the failure)
        if (*sort_err) vals[4 * g + k] = (int32_t)(4 * g + k);
        const int64_t e = vals[4 * g + k];
        L[k] = box32[2 * e];
        H[k] = box32[2 * e + 1];
      }
    }
    float4* r = reinterpret_cast<float4*>(rec + g * (8 * DIM));
    r[0] = make_float4(L[0].x, L[1].x, L[2].x, L[3].x);
    r[1] = make_float4(L[0].y, L[1].y, L[2].y, L[3].y);
    if (DIM == 3) r[2] = make_float4(L[0].z, L[1].z, L[2].z, L[3].z);
    r[DIM] = make_float4(H[0].x, H[1].x, H[2].x, H[3].x);
    r[DIM + 1] = make_float4(H[0].y, H[1].y, H[2].y, H[3].y);
    if (DIM == 3) r[DIM + 2] = make_float4(H[0].z, H[1].z, H[2].z, H[3].z);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      lo[0] = fminf(lo[0], L[k].x);
      lo[1] = fminf(lo[1], L[k].y);
      lo[2] = fminf(lo[2], L[k].z);
      hi[0] = fmaxf(hi[0], H[k].x);
      hi[1] = fmaxf(hi[1], H[k].y);
      hi[2] = fmaxf(hi[2], H[k].z);
    }
  }
  // thread t < w of step l holds node blockIdx * w + t of level l
  int w = kTreeBlock;
  for (int l = 1; l <= T.top; ++l) {
    const int64_t node = (int64_t)blockIdx.x * w + t;
    if (t < w) {
      if ((node >> 2) < T.off[l + 1] - T.off[l]) tree_put<DIM>(rec + (int64_t)T.off[l] * (8 * DIM), node, lo, hi);
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        sl[t][c] = lo[c];
        sh[t][c] = hi[c];
      }
    }
    if (w == 1) break;
    w >>= 2;
    __syncthreads();
    if (t < w) {
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        lo[c] = fminf(fminf(sl[4 * t][c], sl[4 * t + 1][c]), fminf(sl[4 * t + 2][c], sl[4 * t + 3][c]));
        hi[c] = fmaxf(fmaxf(sh[4 * t][c], sh[4 * t + 1][c]), fmaxf(sh[4 * t + 2][c], sh[4 * t + 3][c]));
      }
    }
    __syncthreads();
  }
  if (T.top <= 4) return;  // one block
  if (t == 0) {
    // the block's level-5 node out, then the ticket; the last block's reads
    // after it
    __threadfence();
    s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  // empty nodes fill level 5's last group
  for (int l = 5; l <= T.top; ++l) {
    const int64_t groups = T.off[l + 1] - T.off[l];
    float* r = rec + (int64_t)T.off[l] * (8 * DIM);
    const int64_t nodes = l == 5 ? gridDim.x : (int64_t)T.off[l] - T.off[l - 1];
    for (int64_t j = t; j < 4 * groups; j += kTreeBlock) {
      if (j >= nodes) {
        const float el[3] = {inf, inf, inf}, eh[3] = {-inf, -inf, -inf};
        tree_put<DIM>(r, j, el, eh);
      } else if (l > 5) {
        tree_join<DIM>(rec + (int64_t)T.off[l - 1] * (8 * DIM), j, lo, hi);
        tree_put<DIM>(r, j, lo, hi);
      }
    }
    __threadfence();
    __syncthreads();
  }
}

int64_t tree_floats(int dim, int64_t n) {
  int64_t g = 0, k = n;
  do {
    k = (k + 3) / 4;
    g += k;
  } while (k > 1);
  return g * 8 * dim;
}

Tree make_tree(int dim, int n, int32_t* sorted_vals, float* rec) {
  Tree T;
  T.n = n;
  T.vals = sorted_vals;
  T.rec = rec;
  int64_t k = n;
  int l = 0;
  T.off[0] = 0;
  do {
    k = (k + 3) / 4;
    T.off[l + 1] = T.off[l] + (int)k;
    ++l;
  } while (k > 1);
  T.top = l - 1;
  return T;
}

cudaError_t launch_tree_build(int dim, const Tree& T, const float* box32, unsigned* ticket, const int* sort_err,
                              cudaStream_t s) {
  if (T.n <= 0) return cudaSuccess;
  const int g = (T.off[1] + kTreeBlock - 1) / kTreeBlock;
  count_launch();
  if (dim == 2)
    k_tree_build<2><<<g, kTreeBlock, 0, s>>>(T, T.vals, reinterpret_cast<const float4*>(box32), T.rec, ticket,
                                              sort_err);
  else
    k_tree_build<3><<<g, kTreeBlock, 0, s>>>(T, T.vals, reinterpret_cast<const float4*>(box32), T.rec, ticket,
                                              sort_err);
  return cudaGetLastError();
}

// ======================================================================
// K4: candidate search
// ======================================================================
// Row cache of the count pass: the first `cap` candidates of row a at
// cache[a * cap ..]; later ones spill into chunks of kSpillChunk entries
// taken from a pool (sp.next counts the chunks handed out), chained per row
// (sp.row_chunk[a] = first chunk, sp.chunk_next[c] = the next one) in
// traversal order.  A row that finds the pool exhausted, or runs without a
// pool, is `lost`: it is listed for a second traversal instead.  Only the
// batched search spills (its mesh pairs of unrelated resolutions give many
// long rows); the single-mesh search (k_query) keeps the tighter walk, with
// fewer registers, and lists its (rare) long rows.
__device__ __forceinline__ void cache_put(int32_t* cache, int cap, const Spill& sp, int64_t a, int cnt, int w,
                                          int& ch, bool& lost) {
  if (cnt < cap) {
    cache[a * cap + cnt] = w;
    return;
  }
  if (lost || !sp.pool) {
    lost = true;
    return;
  }
  const int q = cnt - cap, o = q & (kSpillChunk - 1);
  if (o == 0) {
    const int nc = atomicAdd(sp.next, 1);
    if (nc >= sp.chunks) {
      lost = true;
      return;
    }
    if (q == 0)
      sp.row_chunk[a] = nc;
    else
      sp.chunk_next[ch] = nc;
    ch = nc;
  }
  sp.pool[(int64_t)ch * kSpillChunk + o] = w;
}

// One thread per row, depth first: the pending children of the levels above
// are four bits each in one 64-bit word.  A leaf's box test is decided in FP32
// where the outward-rounded boxes leave no doubt, and by the element's FP64
// box otherwise: the strict test of the reference in either case.  No doubt:
// a leaf's lower bound b has the FP32 bound L, b <= L + 2^-23 |L| (plus one
// subnormal); if L < t - 2^-21 |t| - tiny for t = the query's upper bound
// rounded down, then either |L| <= 2 |t| and b < t, or L < -2 |t| and b < -|t|;
// likewise for the other sides.
// The count pass (FILL = false) also keeps the first `cap` candidates of
// every row in cache[a * cap ..] (when cache is given) and lists rows with
// more than cap candidates in over_rows; the fill then copies cached rows
// (k_fill_from_cache) and traverses again only for the listed rows
// (FILL = true with `rows`).  MESH: rows of mesh pair_of_a[a] take only the
// leaves of that B mesh, mesh_off[m] .. mesh_off[m+1]-1 in sorted order, and
// may spill (cache_put).
template <int DIM, bool FILL, bool MESH>
__global__ void __launch_bounds__(256) k_query(int64_t nel_a, const double* __restrict__ box64_a, const __grid_constant__ Tree T,
                                               const double* __restrict__ box64_b, int* counts,
                                               const int64_t* __restrict__ offsets, int32_t* pair_a,
                                               int32_t* pair_b, int32_t* cache, int cap,
                                               const int32_t* __restrict__ rows, int* over_rows, int64_t pair_cap,
                                               const int32_t* __restrict__ pair_of_a,
                                               const int64_t* __restrict__ mesh_off, Spill sp) {
  const int64_t nrows = rows ? (int64_t)*over_rows : nel_a;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = rows ? rows[r] : r;
    const double* qb = box64_a + a * 2 * DIM;
    // the query box, rounded outwards, and inwards by the margin
    float ql[DIM], qh[DIM], il[DIM], ih[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      const double lo = qb[c], hi = qb[DIM + c];
      const float l = __double2float_ru(lo), h = __double2float_rd(hi);
      ql[c] = __double2float_rd(lo);
      qh[c] = __double2float_ru(hi);
      il[c] = fmaf(fabsf(l), 0x1p-21f, l) + 0x1p-140f;
      ih[c] = fmaf(fabsf(h), -0x1p-21f, h) - 0x1p-140f;
    }
    int first = 0, last = T.n - 1;
    if (MESH) {
      const int m = pair_of_a[a];
      first = (int)mesh_off[m];
      last = (int)mesh_off[m + 1] - 1;
    }
    int cnt = 0;
    const int64_t out = FILL ? offsets[a] : 0;
    int chunk = -1;     // MESH: current spill chunk of this row
    bool lost = false;  // MESH: the row goes to the second traversal
    int lvl = T.top, grp = 0;
    unsigned long long pending = 0;  // levels lvl + 1 and up, lowest first
    while (first <= last) {
      const float4* g = reinterpret_cast<const float4*>(T.rec) + ((int64_t)T.off[lvl] + grp) * (2 * DIM);
      float4 L[DIM], H[DIM];
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        L[c] = __ldg(g + c);
        H[c] = __ldg(g + DIM + c);
      }
      bool o0 = true, o1 = true, o2 = true, o3 = true;
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        o0 = o0 && H[c].x > ql[c] && L[c].x < qh[c];
        o1 = o1 && H[c].y > ql[c] && L[c].y < qh[c];
        o2 = o2 && H[c].z > ql[c] && L[c].z < qh[c];
        o3 = o3 && H[c].w > ql[c] && L[c].w < qh[c];
      }
      unsigned mask = (o0 ? 1u : 0u) | (o1 ? 2u : 0u) | (o2 ? 4u : 0u) | (o3 ? 8u : 0u);
      if (MESH) {
        const int j0 = (first >> (2 * lvl)) - 4 * grp, j1 = (last >> (2 * lvl)) - 4 * grp;
        if (j0 > 0) mask &= 15u << min(j0, 4);
        if (j1 < 3) mask &= j1 < 0 ? 0u : 15u >> (3 - j1);
      }
      if (lvl > 0 && mask) {
        const int c = __ffs(mask) - 1;
        pending = pending << 4 | (mask & (mask - 1u));
        --lvl;
        grp = 4 * grp + c;
        continue;
      }
      if (lvl == 0 && mask) {
        // which of the hits the FP32 boxes prove
        bool s0 = true, s1 = true, s2 = true, s3 = true;
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
          s0 = s0 && H[c].x > il[c] && L[c].x < ih[c];
          s1 = s1 && H[c].y > il[c] && L[c].y < ih[c];
          s2 = s2 && H[c].z > il[c] && L[c].z < ih[c];
          s3 = s3 && H[c].w > il[c] && L[c].w < ih[c];
        }
        const unsigned sure = (s0 ? 1u : 0u) | (s1 ? 2u : 0u) | (s2 ? 4u : 0u) | (s3 ? 8u : 0u);
        do {
          const int c = __ffs(mask) - 1;
          mask &= mask - 1u;
          const int e = T.vals[4 * grp + c];
          bool ex = (sure >> c) & 1u;
          if (!ex) {
            const double* bb = box64_b + (int64_t)e * 2 * DIM;
            ex = true;
#pragma unroll
            for (int d = 0; d < DIM; ++d) ex = ex && qb[DIM + d] > bb[d] && qb[d] < bb[DIM + d];
          }
          if (ex) {
            if (FILL) {
              if (out + cnt < pair_cap) {
                pair_a[out + cnt] = (int32_t)a;
                pair_b[out + cnt] = e;
              }
            } else if (cache) {
              if (MESH)
                cache_put(cache, cap, sp, a, cnt, e, chunk, lost);
              else if (cnt < cap)
                cache[a * cap + cnt] = e;
            }
            ++cnt;
          }
        } while (mask);
      }
      // the nearest pending child
      if (!pending) break;
      const int z = (__ffsll((long long)pending) - 1) >> 2;
      const unsigned m = (unsigned)(pending >> (4 * z)) & 15u;
      lvl += z;
      grp = ((grp >> (2 * z + 2)) << 2) + __ffs(m) - 1;
      pending = (pending >> (4 * z)) & ~15ull | (m & (m - 1u));
    }
    if (!FILL) {
      counts[a] = cnt;
      if (cache && (MESH ? lost : cnt > cap)) {
        if (MESH && sp.row_chunk) sp.row_chunk[a] = -2;
        over_rows[1 + atomicAdd(over_rows, 1)] = (int32_t)a;
      }
    }
  }
}

// The count pass with a warp per row: for meshes too small for a thread per
// row to fill the chip, where the longest row's serial walk is the time, and
// (3D) up to medium ones, whose rows of 50 and more candidates keep 32 lanes
// busy.  The warp takes two levels of the hierarchy at once: the 16 + 16
// grandchildren of two nodes, one per lane; then the first two hits' in turn,
// the others pending in lane l for level 2 l.  Hits are appended in leaf
// order, as by k_query.
template <int DIM>
__global__ void __launch_bounds__(256) k_query_warp(int64_t nel_a, const double* __restrict__ box64_a,
                                                    const __grid_constant__ Tree T,
                                                    const double* __restrict__ box64_b, int* counts, int32_t* cache,
                                                    int cap, int* over_rows) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int warps = (int)(gridDim.x * (blockDim.x >> 5));
  for (int64_t a = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); a < nel_a; a += warps) {
    const double* qb = box64_a + a * 2 * DIM;
    float ql[DIM], qh[DIM], il[DIM], ih[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      const double lo = qb[c], hi = qb[DIM + c];
      const float l = __double2float_ru(lo), h = __double2float_rd(hi);
      ql[c] = __double2float_rd(lo);
      qh[c] = __double2float_ru(hi);
      il[c] = fmaf(fabsf(l), 0x1p-21f, l) + 0x1p-140f;
      ih[c] = fmaf(fabsf(h), -0x1p-21f, h) - 0x1p-140f;
    }
    int cnt = 0;
    int lvl = T.top & ~1;
    // the two parents (the first level: nodes 0-15 and no second)
    int p0 = 0, p1 = -1;
    int s0 = 0, s1 = 0;  // lane l: parents of level 2 l's tested nodes,
    unsigned sm = 0;     // and those of them still pending
    for (;;) {
      const int p = lane < 16 ? p0 : p1;
      const int64_t node = 16 * (int64_t)p + (lane & 15);
      bool hit = false, sure = false;
      const int64_t groups = T.off[lvl + 1] - T.off[lvl];
      if (p >= 0 && (node >> 2) < groups) {
        const float* r = T.rec + ((int64_t)T.off[lvl] + (node >> 2)) * (8 * DIM) + (node & 3);
        float L[DIM], H[DIM];
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
          L[c] = __ldg(r + 4 * c);
          H[c] = __ldg(r + 4 * (DIM + c));
        }
        hit = sure = true;
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
          hit = hit && H[c] > ql[c] && L[c] < qh[c];
          sure = sure && H[c] > il[c] && L[c] < ih[c];
        }
      }
      if (lvl == 0) {
        int e = 0;
        if (hit) {
          e = T.vals[node];
          if (!sure) {
            const double* bb = box64_b + (int64_t)e * 2 * DIM;
#pragma unroll
            for (int c = 0; c < DIM; ++c) hit = hit && qb[DIM + c] > bb[c] && qb[c] < bb[DIM + c];
          }
        }
        const unsigned hm = __ballot_sync(full, hit);
        const int at = cnt + __popc(hm & lt);
        if (hit && cache && at < cap) cache[a * cap + at] = e;
        cnt += __popc(hm);
      } else {
        const unsigned hm = __ballot_sync(full, hit);
        if (lane == lvl >> 1) {
          s0 = p0;
          s1 = p1;
          sm = hm;
        }
      }
      // the lowest level with pending nodes: its first two are the next parents
      const unsigned lv = __ballot_sync(full, sm != 0);
      if (!lv) break;
      const int k = __ffs(lv) - 1;
      const unsigned m = __shfl_sync(full, sm, k);
      const int q0 = __shfl_sync(full, s0, k), q1 = __shfl_sync(full, s1, k);
      const int b0 = __ffs(m) - 1;
      const unsigned m1 = m & (m - 1u);
      const int b1 = __ffs(m1) - 1;
      p0 = 16 * (b0 < 16 ? q0 : q1) + (b0 & 15);
      p1 = m1 ? 16 * (b1 < 16 ? q0 : q1) + (b1 & 15) : -1;
      if (lane == k) sm = m1 & (m1 - 1u);
      lvl = 2 * k - 2;
    }
    if (lane == 0) {
      counts[a] = cnt;
      if (cache && cnt > cap) over_rows[1 + atomicAdd(over_rows, 1)] = (int32_t)a;
    }
  }
}

// Fill of the rows whose candidates the count pass cached: each warp copies
// rpw rows, 32 / G at a time, G lanes striding over a row (coalesced reads of
// the cache and writes of the pair arrays).  2D rows hold a dozen candidates,
// which left most of 32 lanes idle and one row's reads in flight.
template <int G>
__global__ void __launch_bounds__(256) k_fill_from_cache(int64_t nel_a, const int* __restrict__ counts,
                                                         const int64_t* __restrict__ offsets,
                                                         const int32_t* __restrict__ cache, int cap,
                                                         int32_t* pair_a, int32_t* pair_b, Spill sp,
                                                         int64_t pair_cap, int rpw) {
  const int lane = threadIdx.x & 31, sub = lane / G, l = lane % G;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * rpw; base < nel_a;
       base += warps * rpw) {
    const int64_t a = base + lane;
    int cnt = 0;
    int64_t off = 0;
    if (lane < rpw && a < nel_a) {
      cnt = counts[a];
      off = offsets[a];
    }
    for (int r0 = 0; r0 < rpw; r0 += 32 / G) {
      const int r = (r0 + sub) & 31;
      // (lanes from rpw on hold empty rows)
      const int c = __shfl_sync(0xffffffffu, cnt, r);
      const int64_t o = __shfl_sync(0xffffffffu, off, r);
      const int64_t row = base + r;
      // entries of this row that fit the pair arrays (all of them unless a
      // capacity-mode call outgrew its arrays)
      const int64_t room = pair_cap - o;
      const int lim = room >= c ? c : (room > 0 ? (int)room : 0);
      if (c > cap) {
        // the cached head, then the row's chain of spill chunks; rows that
        // lost theirs (-2) are filled by the traversal over the listed rows
        const int first = sp.row_chunk ? sp.row_chunk[row] : -2;
        if (first < 0) continue;
        const int head = lim < cap ? lim : cap;
        for (int k = l; k < head; k += G) {
          pair_a[o + k] = (int32_t)row;
          pair_b[o + k] = cache[row * cap + k];
        }
        int ch = first;
        for (int k0 = cap; k0 < c; k0 += kSpillChunk) {
          for (int k = l; k < kSpillChunk && k0 + k < lim; k += G) {
            pair_a[o + k0 + k] = (int32_t)row;
            pair_b[o + k0 + k] = sp.pool[(int64_t)ch * kSpillChunk + k];
          }
          if (k0 + kSpillChunk < c) ch = sp.chunk_next[ch];
        }
        continue;
      }
      for (int k = l; k < lim; k += G) {
        pair_a[o + k] = (int32_t)row;
        pair_b[o + k] = cache[row * cap + k];
      }
    }
  }
}

// The count pass takes a warp per row below this many rows.  Whole search
// (prep to pair arrays), thread / warp per row: 2D 10,658 rows 165 / 146 us,
// 45,000 rows 168 / 186 us; 3D 6,000 rows 288 / 162 us, 48,000 rows 369 / 338
// us, 118,098 rows 401 / 465 us.
constexpr int64_t kWarpRows2 = 24 << 10, kWarpRows3 = 64 << 10;
// Lanes per row of the fill (2D 4 / 8 / 16 / 32: whole call 1513 / 1494 / 1503 /
// 1543 us, 14.9 M candidates; 3D 8 / 16 / 32: 9819 / 9740 / 9723 us, 56 M).
constexpr int kFill2 = 8, kFill3 = 32;

// Threads per block of the search: the option's, or a warp where that leaves
// SMs without a block (the row's serial walk is then the time).
static int query_threads(int64_t nel_a) {
  return nel_a < (int64_t)sm_count() * 4 * query_block() ? 32 : query_block();
}

template <bool MESH>
static cudaError_t run_query(int dim, bool fill, int64_t nel_a, const double* box64_a, const Tree& T,
                             const double* box64_b, int* counts, const int64_t* offsets, int32_t* pair_a,
                             int32_t* pair_b, cudaStream_t s, int32_t* cache, int cap, int* over_rows,
                             int64_t pair_cap, const int32_t* pair_of_a, const int64_t* mesh_off, const Spill& sp) {
  if (nel_a <= 0 || T.n <= 0) return cudaSuccess;
  const int B = query_threads(nel_a);
  const int g = grid_for(nel_a, B, 2048 / B);
  if (fill && cache) {
    count_launch(2);
    // 32 rows per warp, fewer while that leaves warps to spare
    int rpw = 32;
    while (rpw > 1 && nel_a < (int64_t)sm_count() * 32 * rpw) rpw >>= 1;
    (dim == 2 ? k_fill_from_cache<kFill2> : k_fill_from_cache<kFill3>)
        <<<grid_for((nel_a + rpw - 1) / rpw * 32, 256, 8), 256, 0, s>>>(nel_a, counts, offsets, cache, cap, pair_a,
                                                                       pair_b, sp, pair_cap, rpw);
  } else {
    count_launch();
  }
  if (!MESH && !fill && cache && nel_a < (dim == 2 ? kWarpRows2 : kWarpRows3)) {
    const int gw = grid_for(nel_a * 32, 256, 8);
    (dim == 2 ? k_query_warp<2> : k_query_warp<3>)<<<gw, 256, 0, s>>>(nel_a, box64_a, T, box64_b, counts, cache, cap,
                                                                      over_rows);
    return cudaGetLastError();
  }
  const int32_t* rows = (fill && cache) ? over_rows + 1 : nullptr;
  int32_t* cc = fill ? nullptr : cache;
  const auto k = dim == 2 ? (fill ? k_query<2, true, MESH> : k_query<2, false, MESH>)
                          : (fill ? k_query<3, true, MESH> : k_query<3, false, MESH>);
  k<<<g, B, 0, s>>>(nel_a, box64_a, T, box64_b, counts, offsets, pair_a, pair_b, cc, cap, rows, over_rows, pair_cap,
                    pair_of_a, mesh_off, sp);
  return cudaGetLastError();
}

cudaError_t launch_query(int dim, bool fill, int64_t nel_a, const double* box64_a, const Tree& T,
                         const double* box64_b, int* counts, const int64_t* offsets, int32_t* pair_a,
                         int32_t* pair_b, cudaStream_t s, int32_t* cache, int cap, int* over_rows, Spill sp,
                         int64_t pair_cap) {
  return run_query<false>(dim, fill, nel_a, box64_a, T, box64_b, counts, offsets, pair_a, pair_b, s, cache, cap,
                          over_rows, pair_cap, nullptr, nullptr, sp);
}

cudaError_t launch_query_batched(int dim, bool fill, int64_t nel_a, const double* box64_a,
                                 const int32_t* pair_of_a, const int64_t* mesh_off_b, const Tree& T,
                                 const double* box64_b, int* counts, const int64_t* offsets, int32_t* pair_a,
                                 int32_t* pair_b, cudaStream_t s, int32_t* cache, int cap, int* over_rows,
                                 Spill sp, int64_t pair_cap) {
  return run_query<true>(dim, fill, nel_a, box64_a, T, box64_b, counts, offsets, pair_a, pair_b, s, cache, cap,
                         over_rows, pair_cap, pair_of_a, mesh_off_b, sp);
}

// ======================================================================
// Scan of int32 counts -> int64 offsets
// ======================================================================
namespace {
constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;
}  // namespace

int64_t scan_tmp_entries(int64_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

template <int BLOCK>
__device__ int64_t block_excl_scan(int64_t v, int64_t* total) {
  __shared__ int64_t wt[BLOCK / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) wt[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    int64_t w = lane < BLOCK / 32 ? wt[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    if (lane < BLOCK / 32) wt[lane] = w;
  }
  __syncthreads();
  const int64_t r = inc - v + (wid > 0 ? wt[wid - 1] : 0);
  if (total) *total = wt[BLOCK / 32 - 1];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(int64_t n, const int* __restrict__ counts, int64_t* tmp) {
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i)
    if (base + i < n) s += counts[base + i];
  int64_t tot;
  block_excl_scan<kScanThreads>(s, &tot);
  if (threadIdx.x == 0) tmp[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(1024) k_scan_top(int nb, int64_t* tmp) {
  // exclusive scan of tmp[0..nb) in place; tmp[nb] = total
  __shared__ int64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nb; base += 1024) {
    const int i = base + threadIdx.x;
    const int64_t v = i < nb ? tmp[i] : 0;
    int64_t tot;
    const int64_t ex = block_excl_scan<1024>(v, &tot);
    if (i < nb) tmp[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) tmp[nb] = carry;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_down(int64_t n, const int* __restrict__ counts,
                                                            const int64_t* __restrict__ tmp, int64_t* out,
                                                            int nb) {
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int v[kScanItems];
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = base + i < n ? counts[base + i] : 0;
    s += v[i];
  }
  int64_t run = block_excl_scan<kScanThreads>(s, nullptr) + tmp[blockIdx.x];
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n) out[base + i] = run;
    run += v[i];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = tmp[nb];
}

// The whole scan in one block, for counts that three launches would only
// spread thin (10,658 rows: 11 -> 10 us).  A warp takes 256 counts in
// four rows of 64, two neighbours a lane, so that its loads and stores are
// nearly whole lines: with eight neighbours a lane the stores alone, each to
// 32 lines, took most of 11 us.
__global__ void __launch_bounds__(1024) k_scan_one(int64_t n, const int* __restrict__ counts, int64_t* out) {
  constexpr int kRows = 4;
  __shared__ int64_t wsum[2][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t carry = 0;
  for (int64_t b0 = 0, it = 0; b0 < n; b0 += 1024 * 2 * kRows, ++it) {
    const int64_t base = b0 + wid * 64 * kRows + 2 * lane;
    int v[kRows][2];
    int64_t ex[kRows];  // before the lane's pair, from the warp's first count
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int64_t i = base + 64 * r;
      v[r][0] = i < n ? counts[i] : 0;
      v[r][1] = i + 1 < n ? counts[i + 1] : 0;
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) ex[r] = (int64_t)v[r][0] + v[r][1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        const int64_t t = __shfl_up_sync(0xffffffffu, ex[r], o);
        if (lane >= o) ex[r] += t;
      }
    int64_t run = 0;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int64_t tot = __shfl_sync(0xffffffffu, ex[r], 31);
      ex[r] += run - v[r][0] - v[r][1];
      run += tot;
    }
    // (two rows of sums, so that one barrier a tile is enough)
    if (lane == 0) wsum[it & 1][wid] = run;
    __syncthreads();
    int64_t w = wsum[it & 1][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    const int64_t first = carry + __shfl_sync(0xffffffffu, w, wid) - run;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int64_t i = base + 64 * r;
      if (i < n) out[i] = first + ex[r];
      if (i + 1 < n) out[i + 1] = first + ex[r] + v[r][0];
    }
    carry += __shfl_sync(0xffffffffu, w, 31);
  }
  if (threadIdx.x == 0) out[n] = carry;
}

cudaError_t launch_scan(int64_t n, const int* counts, int64_t* offsets, int64_t* tmp, cudaStream_t s) {
  if (n <= 0) {
    cudaMemsetAsync(offsets, 0, sizeof(int64_t), s);
    return cudaGetLastError();
  }
  if (n <= 32 << 10) {
    count_launch();
    k_scan_one<<<1, 1024, 0, s>>>(n, counts, offsets);
    return cudaGetLastError();
  }
  const int nb = (int)((n + kScanTile - 1) / kScanTile);
  count_launch(3);
  k_scan_reduce<<<nb, kScanThreads, 0, s>>>(n, counts, tmp);
  k_scan_top<<<1, 1024, 0, s>>>(nb, tmp);
  k_scan_down<<<nb, kScanThreads, 0, s>>>(n, counts, tmp, offsets, nb);
  return cudaGetLastError();
}

// ======================================================================
// K5: triangle clipping
// ======================================================================
namespace {
constexpr int kTriBlock = 96;
constexpr int kTriCap = 6;  // fast-path polygon slots (the geometric maximum)
constexpr int kTriWideCap = 24;
constexpr int kTetStack = 6;      // max pending tets: 2 per level for planes 0-2
}  // namespace

template <int CAP>
struct LocalPoly {
  double px[CAP], py[CAP];
  __device__ __forceinline__ double x(int i) const { return px[i]; }
  __device__ __forceinline__ double y(int i) const { return py[i]; }
  __device__ __forceinline__ void set(int i, double a, double b) {
    px[i] = a;
    py[i] = b;
  }
};

struct NoEmit {
  __device__ __forceinline__ void operator()(int, double, double, double, double, double, double) const {}
};

// A 2D setup row in four 16-byte loads: the vertices, the tolerance and, as
// a sign, the orientation.  The lines' normals are differences of the vertices
// (tri_lines); rows with the lines written out were 112 bytes of gathered
// loads a pair.
__device__ __forceinline__ void load_lines(const double* __restrict__ o, Lines& L, double& tol) {
  const double2* q = reinterpret_cast<const double2*>(o);
  const double2 v[3] = {__ldg(q), __ldg(q + 1), __ldg(q + 2)}, t = __ldg(q + 3);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    L.nx[i] = (v[(i + 1) % 3].y - v[i].y) * t.y;
    L.ny[i] = (v[i].x - v[(i + 1) % 3].x) * t.y;
    L.px[i] = v[i].x;
    L.py[i] = v[i].y;
  }
  tol = t.x;
}

// The supermesh triangles of one pair, as clip_tri gives them, by way of
// clip_tri_c (whole calls: triangles of 180,000 x 320,000 elements 722 -> 596
// us; blocks of 80,000 x 135,000, k_p1_mass 132 -> 99 us).  p: the thread's column of kTriCap vertices in shared memory.
template <int B, class Emit>
__device__ __forceinline__ void clip_tri_fan(const double2 (&a)[3], const Lines& L, double tol, double2* p, bool on,
                                             const Emit& emit) {
  const int n = clip_tri_c<B>(a, L, p, on);
  int kept = 0;
#pragma unroll 1
  for (int k = 2; k < n; ++k) {
    const double2 o = p[0], s = p[(k - 1) * B], t = p[k * B];
    if (!(tri_area(o.x, o.y, s.x, s.y, t.x, t.y) < tol)) emit(kept++, o.x, o.y, s.x, s.y, t.x, t.y);
  }
  if (n < 0) {
    LocalPoly<kTriWideCap> f, g;
    double m;
    clip_tri(a[0].x, a[0].y, a[1].x, a[1].y, a[2].x, a[2].y, L, tol, f, g, kTriWideCap, m, emit);
  }
}

// One pair a lane.  Bound by instructions (issue 64 %) and L1 and shared
// wavefronts (69 %), both of which divergence multiplies: with the walking
// clip on 112-byte rows of lines 12 of 32 lanes were active on average and
// 14.9 M pairs took 1190 us; clip_tri_c alone would have given 1108 (in two
// buffers), in place and with 64-byte rows 630.  Eight blocks an SM, all
// resident: 96 threads at 80 registers 629 us, 128 at 64 646, 64 at 104 642.
__global__ void __launch_bounds__(kTriBlock, 8) k_clip_tris(int64_t npairs, const int32_t* __restrict__ pa,
                                                         const int32_t* __restrict__ pb,
                                                         const double* __restrict__ coords_a,
                                                         const double* __restrict__ tol_a,
                                                         const double* __restrict__ setup_b,
                                                         double* pair_measure, int32_t* pair_nout,
                                                         int32_t* ovf_list, int* ovf_count,
                                                         const int32_t* __restrict__ order,
                                                         const int64_t* __restrict__ n_dev) {
  // n_dev (optional): the pair count on the device, npairs its upper bound
  if (n_dev && *n_dev < npairs) npairs = *n_dev;
  __shared__ double2 poly[kTriCap * kTriBlock];
  double2* p = poly + threadIdx.x;
  // each iteration loads the next one's pair indices (which stream from
  // DRAM) before it clips its own pair; a warp's lanes go on together
  const int64_t stride = (int64_t)gridDim.x * kTriBlock;
  int64_t j = (int64_t)blockIdx.x * kTriBlock + threadIdx.x;
  int64_t ni = j;
  int na = 0, nb = 0;
  if (j < npairs) {
    if (order) ni = order[ni];
    na = pa[ni];
    nb = pb[ni];
  }
  for (; j - (threadIdx.x & 31) < npairs; j += stride) {
    const int64_t i = ni;
    const int a = na, b = nb;
    const bool on = j < npairs;
    if (j + stride < npairs) {
      ni = order ? (int64_t)order[j + stride] : j + stride;
      na = pa[ni];
      nb = pb[ni];
    }
    const double2* va = reinterpret_cast<const double2*>(coords_a + (int64_t)a * 6);
    const double2 v[3] = {__ldg(va), __ldg(va + 1), __ldg(va + 2)};
    Lines L;
    double tolb;
    load_lines(setup_b + (int64_t)b * kSetup2, L, tolb);
    const double tol = fmin(tol_a[a], tolb);
    const int n = clip_tri_c<kTriBlock>(v, L, p, on);
    double m = 0.0;
    int kept = 0;
    if (n > 0) {
      const double2 o = p[0];
      double2 s = p[kTriBlock];
#pragma unroll
      for (int k = 2; k < kTriCap; ++k) {
        if (k < n) {
          const double2 t = p[k * kTriBlock];
          const double ar = tri_area(o.x, o.y, s.x, s.y, t.x, t.y);
          const bool in = !(ar < tol);
          m = in ? m + ar : m;
          kept += in;
          s = t;
        }
      }
    }
    if (n < 0) {
      ovf_list[atomicAdd(ovf_count, 1)] = (int32_t)i;
    } else if (on) {
      pair_measure[i] = m;
      pair_nout[i] = kept;
    }
  }
}

// The pairs that k_clip_tris lists, with room for polygons that are not convex
// any more.  Almost always none; slivers as wide as rounding give 0.3 % of
// their candidates.  Over the whole chip: 250,000 such pairs took one warp 19
// ms and take 0.11 ms so, the narrow phase of 75.9 M candidates of such
// slivers 5.6 -> 3.3 ms, an empty list as long as before.
constexpr int kTriWideBlock = 64;
__global__ void __launch_bounds__(kTriWideBlock) k_clip_tris_wide(const int32_t* __restrict__ list, const int* __restrict__ count,
                                                       int64_t cap, const int32_t* __restrict__ pa,
                                                       const int32_t* __restrict__ pb,
                                                       const double* __restrict__ coords_a,
                                                       const double* __restrict__ tol_a,
                                                       const double* __restrict__ setup_b,
                                                       double* pair_measure, int32_t* pair_nout) {
  int64_t nl = *count;
  if (nl > cap) nl = cap;
  for (int64_t j = (int64_t)blockIdx.x * kTriWideBlock + threadIdx.x; j < nl;
       j += (int64_t)gridDim.x * kTriWideBlock) {
    const int64_t i = list[j];
    const int a = pa[i], b = pb[i];
    const double* va = coords_a + (int64_t)a * 6;
    Lines L;
    double tolb;
    load_lines(setup_b + (int64_t)b * kSetup2, L, tolb);
    const double tol = fmin(tol_a[a], tolb);
    LocalPoly<kTriWideCap> p, q;
    double m;
    int n = clip_tri(va[0], va[1], va[2], va[3], va[4], va[5], L, tol, p, q, kTriWideCap, m, NoEmit{});
    if (n < 0) {  // cannot happen: 3 -> 6 -> 12 -> 24 vertices at most
      n = 0;
      m = 0.0;
    }
    pair_measure[i] = m;
    pair_nout[i] = n;
  }
}

// ======================================================================
// K6: tetrahedron clipping, depth-first
// ======================================================================
struct TetStackLocal {
  Tet slot[kTetStack];
  __device__ __forceinline__ void store(int s, const Tet& t) { slot[s] = t; }
  __device__ __forceinline__ void load(int s, Tet& t) const { t = slot[s]; }
};

// Sink for clip_tet_plane inside the depth-first walk: at the last plane it
// evaluates final tets (vol_v4 >= tol, then the vertex-1 volume) in order;
// before that it parks children 1..k-1 on the stack so that child 1 is on
// top (pre-order = the reference's breadth-first output order).
template <class Stack, class Leaf>
struct DfsSink {
  Stack& stk;
  Leaf& leaf;
  int sp;
  bool last;
  double tol;
  int k;
  int kept;
  __device__ __forceinline__ void begin(int kk) { k = kk; }
  __device__ __forceinline__ void child(int j, const Tet& c) {
    if (last) {
      if (tet_volume_v4(c) >= tol) {
        leaf(c);
        ++kept;
      }
    } else if (j > 0) {
      stk.store(sp + (k - 1) - j, c);
    }
  }
};

__device__ __forceinline__ void load_plane(const double* __restrict__ planes, int L, double& nx, double& ny,
                                           double& nz, double& c) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(planes + 4 * L));
  const double2 b = __ldg(reinterpret_cast<const double2*>(planes + 4 * L + 2));
  nx = a.x;
  ny = a.y;
  nz = b.x;
  c = b.y;
}

// Plane source for the depth-first walk: planes computed in registers.
struct RegPlanes {
  const Planes& P;
  __device__ __forceinline__ void get(int L, double& nx, double& ny, double& nz, double& c) const {
    nx = sel4(L, P.nx[0], P.nx[1], P.nx[2], P.nx[3]);
    ny = sel4(L, P.ny[0], P.ny[1], P.ny[2], P.ny[3]);
    nz = sel4(L, P.nz[0], P.nz[1], P.nz[2], P.nz[3]);
    c = sel4(L, P.c[0], P.c[1], P.c[2], P.c[3]);
  }
};

// Depth-first clip of tet `t` by NP planes; calls leaf(tet) for each final
// tet with vol_v4 >= tol, in the reference's output order.  Returns the
// number of kept tets.  The stack needs 2*(NP-1) slots.
template <int NP = 4, class Src, class Stack, class Leaf>
__device__ __forceinline__ int clip_tet_dfs(Tet t, const Src& planes, double tol, Stack& stk, Leaf leaf) {
  int sp = 0;
  unsigned long long levels = 0;  // 3 bits per stack slot
  int L = 0;
  int kept = 0;
  for (int guard = 0; guard < 1200; ++guard) {  // at most (3^NP - 1)/2 tets are clipped
    double nx, ny, nz, c;
    planes.get(L, nx, ny, nz, c);
    DfsSink<Stack, Leaf> sink{stk, leaf, sp, L == NP - 1, tol, 0, 0};
    const int k = clip_tet_plane(t, nx, ny, nz, c, sink);
    kept += sink.kept;
    if (L < NP - 1 && k > 0) {
      if (k > 1) levels |= (unsigned long long)(L + 1) << (3 * sp);
      if (k > 2) levels |= (unsigned long long)(L + 1) << (3 * (sp + 1));
      sp += k - 1;
      ++L;
      continue;
    }
    if (sp == 0) break;
    --sp;
    stk.load(sp, t);
    L = (int)((levels >> (3 * sp)) & 7ull);
    levels &= ~(7ull << (3 * sp));
  }
  return kept;
}

// Planes in a per-thread array (explicit pairs: hex faces).
template <int NP>
struct ArrPlanes {
  double nx[NP], ny[NP], nz[NP], c[NP];
  __device__ __forceinline__ void get(int L, double& a, double& b, double& d, double& e) const {
    a = nx[L];
    b = ny[L];
    d = nz[L];
    e = c[L];
  }
};

template <int N>
struct TetStackN {
  Tet slot[N];
  __device__ __forceinline__ void store(int s, const Tet& t) { slot[s] = t; }
  __device__ __forceinline__ void load(int s, Tet& t) const { t = slot[s]; }
};

__device__ __forceinline__ void load_tet(const double* __restrict__ v, Tet& t) {
  const double2* q = reinterpret_cast<const double2*>(v);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double2 a = __ldg(q + 3 * k), b = __ldg(q + 3 * k + 1), c = __ldg(q + 3 * k + 2);
    // vertices 2k and 2k+1: (a.x a.y b.x) (b.y c.x c.y)
    t.x[2 * k] = a.x;
    t.y[2 * k] = a.y;
    t.z[2 * k] = b.x;
    t.x[2 * k + 1] = b.y;
    t.y[2 * k + 1] = c.x;
    t.z[2 * k + 1] = c.y;
  }
}

// Exact early-out for the tet clipper.  If every vertex of A lies at
// distance >= eps + margin on the outer side of one of B's face planes, then
// so does every tet the reference's clipping derives from A: derived
// vertices are convex combinations of A's vertices, and the rounding of at
// most three nested interpolations plus the distance evaluation moves them by
// far less than margin = 64*eps*(1 + 2M) (M bounds the coordinates and plane
// offsets involved).  Such a tet is classified entirely positive at that
// plane and discarded, so the reference returns no tets: the pair's result is
// written here (0 tets, measure 0) and only the remaining pairs are listed
// for the clipper.
// With faces_a / screen_b (optional) a pair that passes this test gets the
// second one: B beyond a face plane of A by the margin derived next to
// tet_screen_b, which again proves that the reference returns no tets.
// `order` (optional) lists the pairs in the order the clipper should take
// them (a schedule); survivors are appended in that order, warp by warp.
// A plane of B with every vertex of A at distance <= -(eps + margin) keeps
// every tet derived from A whole (all its vertices classify negative), so it
// changes nothing in the reference's result; such planes form the pair's
// no-op mask.  With all four planes no-op the reference returns A itself,
// which is settled here (volume test and measure as in the clipper).
// Survivors are written as {pair, a, b, no-op mask} so that the clipper
// gets the element numbers and the planes to skip in one load.
// kSettle false (the P1 mass pass, explicit pairs with output tets): pairs
// with all four planes no-op are listed too, for the clipper to emit A
// itself; rejected pairs get measure 0 and count 0 where pair_measure is
// given (the P1 pass passes none and zero-fills its blocks).
#ifndef LSM_PREFILTER_BPS
#define LSM_PREFILTER_BPS 2
#endif
// NP planes per B element in setup rows of clip_row(NP) doubles (4: tets,
// 6: hexahedra; the second early-out is for tets only).  The margin covers
// the up to NP-1 nested interpolations of a derived vertex (each within
// ~7 eps M of an exact convex combination) with room to spare.
__host__ __device__ constexpr int clip_row(int np) { return 4 * np + 4; }

// Pairs per block of the early-out pass (256 threads): one contiguous range
// each, a multiple of the block size.
constexpr int kSegChunk = 64;
__host__ __device__ inline int64_t seg_per(int64_t npairs, int grid) {
  return ((npairs + grid - 1) / grid + 255) / 256 * 256;
}

// Last word of a survivor record for k_clip_tets_bf (kCode; otherwise just the
// no-op mask): the no-op mask in bits 0-3, then
// the signs of A's vertices at B's planes (plane l, vertex v at bit 4 +
// 4 (3-l) + 3-v, as the pass shifts them in), and in bit 30 whether some
// distance is neither clearly positive nor clearly negative to the clipper
// (|d| < eps, infinite or NaN; the clipper then classifies A itself).  irr is
// the largest 2 * (high word of |d|) - 2 * kEpsHi, modulo 2^32: it reaches
// 2 * (0x7ff00000 - kEpsHi) exactly for such distances.
constexpr unsigned kEpsHi = 0x3cb00000u;  // high word of eps = 2^-52
__device__ __forceinline__ int surv_code(int noop, unsigned neg, unsigned irr) {
  return noop | (int)(neg << 4) | (irr >= 2u * (0x7ff00000u - kEpsHi) ? 1 << 30 : 0);
}

// max(m, |x|) for m >= 0; a NaN x leaves m.
__device__ __forceinline__ double max_abs(double m, double x) { return fabs(x) > m ? fabs(x) : m; }

template <bool kSettle, int NP, bool kSeg, bool kCode>
__global__ void __launch_bounds__(256, LSM_PREFILTER_BPS) k_prefilter_tets(int64_t npairs, const int32_t* __restrict__ order,
                                                        const int32_t* __restrict__ pa,
                                                        const int32_t* __restrict__ pb,
                                                        const double* __restrict__ coords_a,
                                                        const double* __restrict__ tol_a,
                                                        const double* __restrict__ setup_b,
                                                        double* pair_measure, int32_t* pair_nout,
                                                        int32_t* survivors, unsigned long long* nsurv,
                                                        const double* __restrict__ faces_a,
                                                        const double* __restrict__ screen_b,
                                                        const int64_t* __restrict__ n_dev, int* seg_count = nullptr) {
  // n_dev (optional): the pair count on the device, npairs its upper bound
  if (n_dev && *n_dev < npairs) npairs = *n_dev;
  __shared__ unsigned s_cnt;
  if (kSeg) {
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
  }
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  // each block takes one contiguous range of pairs (consecutive iterations
  // then share A rows and most B elements in L1)
  const int64_t per = seg_per(npairs, gridDim.x);  // a multiple of the block size (256)
  const int64_t beg = (int64_t)blockIdx.x * per;
  const int64_t end = beg + per < npairs ? beg + per : npairs;
  // the pair indices stream from DRAM: each iteration loads the next one's
  // (ni, na, nb) while it tests its own pair
  int64_t ni = beg + threadIdx.x;
  int na = 0, nb = 0;
  if (ni < end) {
    if (order) ni = order[ni];
    na = pa[ni];
    nb = pb[ni];
  }
  for (int64_t base = beg; base < end; base += blockDim.x) {
    const int64_t j = base + threadIdx.x;
    bool live = false;
    const int64_t i = ni;
    const int a = na, b = nb;
    int noop = 0, code = 0;
    {
      const int64_t jn = j + blockDim.x;
      if (jn < end) {
        ni = order ? (int64_t)order[jn] : jn;
        na = pa[ni];
        nb = pb[ni];
      }
    }
    if (j < end) {
      Tet t;
      load_tet(coords_a + (int64_t)a * 12, t);
      const double* pl = setup_b + (int64_t)b * clip_row(NP);
      double M = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) M = max_abs(max_abs(max_abs(M, t.x[k]), t.y[k]), t.z[k]);
      bool reject = false;
      unsigned neg = 0, irr = 0;  // sign bits of the distances, and the clipper's class test (surv_code)
#pragma unroll
      for (int L = 0; L < NP; ++L) {
        double nx, ny, nz, c;
        load_plane(pl, L, nx, ny, nz, c);
        const double thr = kEps + 64.0 * kEps * (1.0 + 2.0 * max_abs(M, c));
        // One predicate per distance: the smallest and largest of them, as
        // doubles, were a third of the pass's instructions.  Without
        // short-circuits, whose branches cost more (1,000,000 x 800,000 graded tets, 2444 -> 2264 us;
        // with them 2830).  With an infinite bound nothing is proven; a
        // distance that is NaN does not count against the others.
        bool out = thr <= DBL_MAX, in = out;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const double d = ((nx * t.x[k] + ny * t.y[k]) + nz * t.z[k]) - c;
          if (kCode) {
            const unsigned hi = (unsigned)__double2hiint(d);
            neg = __funnelshift_l(hi, neg, 1);
            irr = max(irr, 2u * hi - 2u * kEpsHi);
          }
          out = out & !(d < thr);
          in = in & !(d > -thr);
        }
        reject = reject || out;
        noop |= in ? 1 << L : 0;
      }
      code = kCode ? surv_code(noop, neg, irr) : noop;
      if (NP == 4 && !reject && faces_a) {
        const double2* sb = reinterpret_cast<const double2*>(screen_b + (int64_t)b * kScreen3);
        const double2 gt = __ldg(sb + 6), mz = __ldg(sb + 7);
        if (gt.x < DBL_MAX) {  // B's planes bound a proper tet
          Tet u;
          load_tet(screen_b + (int64_t)b * kScreen3, u);
          const double Mp = fmax(M, mz.x);
          const double e = kEps + 128.0 * kEps * (1.0 + 2.0 * Mp);
          const double slack = 1.01 * gt.x * (gt.y + e) + 16.0 * kEps * (1.0 + Mp);
          const double2* fa = reinterpret_cast<const double2*>(faces_a + (int64_t)a * kScreen3);
#pragma unroll
          for (int P = 0; P < 4; ++P) {
            const double2 n01 = __ldg(fa + 2 * P), n2h = __ldg(fa + 2 * P + 1);
            const double h = n2h.y + slack;
            bool out = h <= DBL_MAX;
#pragma unroll
            for (int k = 0; k < 4; ++k) out = out & !((n01.x * u.x[k] + n01.y * u.y[k]) + n2h.x * u.z[k] < h);
            reject = reject || out;
          }
        }
      }
      if (!kSettle) {
        live = !reject;
        if (reject && pair_measure) {
          pair_measure[i] = 0.0;
          pair_nout[i] = 0;
        }
      } else if (reject) {
        pair_measure[i] = 0.0;
        pair_nout[i] = 0;
      } else if (noop == (1 << NP) - 1) {
        // A inside all planes: the reference keeps A as its one tet
        double v1;
        const bool keep = final_tet_keep(t, fmin(tol_a[a], pl[4 * NP]), v1);
        pair_measure[i] = keep ? v1 : 0.0;
        pair_nout[i] = keep ? 1 : 0;
      } else {
        live = true;
      }
    }
    const unsigned mask = __ballot_sync(0xffffffffu, live);
    if (mask) {
      const int leader = __ffs(mask) - 1;
      unsigned long long off = 0;
      if (lane == leader)
        off = kSeg ? (unsigned long long)beg + atomicAdd(&s_cnt, (unsigned)__popc(mask))
                   : atomicAdd(nsurv, (unsigned long long)__popc(mask));
      off = __shfl_sync(0xffffffffu, off, leader);
      if (live) {
        const int64_t o = (int64_t)off + __popc(mask & lt);
        reinterpret_cast<int4*>(survivors)[o] = make_int4((int)i, a, b, code);
      }
    }
  }
  if (kSeg) {
    __syncthreads();
    if (threadIdx.x == 0) seg_count[blockIdx.x] = (int)s_cnt;
  }
}

// Segmented survivor lists.  With kSeg the early-out pass takes no global
// atomic per warp: block k appends its survivors at k * per (per = the pairs
// a block takes, so a segment never outgrows its range) through a counter
// in shared memory and writes the segment's length to seg_count[k].  The
// clipper then claims whole chunks of at most kIxChunk records that lie in
// one segment from a table, in segment order: {first, end, position in the
// compacted list, 0}.  The table kernel runs one block per segment (the
// early-out pass's grid) and writes the survivor count (work[0]) and the
// chunk count (work[2]).
int64_t seg_table_entries(int64_t npairs) { return npairs / kSegChunk + (int64_t)sm_count() * 8 + 1; }
int seg_blocks(int64_t npairs) { return grid_for(npairs, 256, 8); }

__global__ void __launch_bounds__(256) k_seg_chunks(int64_t npairs, const int64_t* __restrict__ n_dev,
                                                    const int* __restrict__ seg_count, int4* table,
                                                    unsigned long long* work) {
  if (n_dev && *n_dev < npairs) npairs = *n_dev;
  const int64_t per = seg_per(npairs, gridDim.x);
  __shared__ long long part[2][8];
  long long sn = 0, sc = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += blockDim.x) {
    const int c = seg_count[k];
    sn += c;
    sc += (c + kSegChunk - 1) / kSegChunk;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sn += __shfl_xor_sync(0xffffffffu, sn, o);
    sc += __shfl_xor_sync(0xffffffffu, sc, o);
  }
  if ((threadIdx.x & 31) == 0) {
    part[0][threadIdx.x >> 5] = sn;
    part[1][threadIdx.x >> 5] = sc;
  }
  __syncthreads();
  long long pn = 0, pc = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    pn += part[0][w];
    pc += part[1][w];
  }
  const int cnt = seg_count[blockIdx.x];
  const int nch = (cnt + kSegChunk - 1) / kSegChunk;
  const int64_t first = (int64_t)blockIdx.x * per;
  for (int j = threadIdx.x; j < nch; j += blockDim.x) {
    const int lo = j * kSegChunk, hi = lo + kSegChunk < cnt ? lo + kSegChunk : cnt;
    table[pc + j] = make_int4((int)(first + lo), (int)(first + hi), (int)(pn + lo), 0);
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    work[0] = (unsigned long long)(pn + cnt);
    work[2] = (unsigned long long)(pc + nch);
  }
}

// The segmented list gathered into one compacted list (in table order): for
// consumers that index survivors directly.  One warp per chunk.
__global__ void __launch_bounds__(256) k_seg_compact(int64_t max_chunks, const unsigned long long* __restrict__ nchunks,
                                                     const int4* __restrict__ table, const int4* __restrict__ seg,
                                                     int4* out) {
  const int64_t nc = (int64_t)*nchunks < max_chunks ? (int64_t)*nchunks : max_chunks;
  const int lane = threadIdx.x & 31;
  for (int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nc;
       c += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int4 t = table[c];
    for (int k = lane; k < t.y - t.x; k += 32) out[(int64_t)t.z + k] = seg[(int64_t)t.x + k];
  }
}

cudaError_t launch_seg_compact(int64_t npairs, const unsigned long long* nchunks, const int4* table,
                               const int4* seg, int4* out, cudaStream_t s) {
  const int64_t maxc = seg_table_entries(npairs);
  count_launch();
  k_seg_compact<<<grid_for(maxc * 32, 256, 8), 256, 0, s>>>(maxc, nchunks, table, seg, out);
  return cudaGetLastError();
}

// The early-out pass over n pairs into `survivors`: one list counted in
// work[0], or, with seg, per-block segments and their chunk table (work[0]
// survivors, work[2] chunks).  The clipper then takes seg_nlist(seg, work)
// and seg_table(seg).
namespace {
inline bool seg_on(const SegList* seg) { return seg && seg->count && seg->table; }
inline const unsigned long long* seg_nlist(const SegList* seg, const unsigned long long* work) {
  return seg_on(seg) ? work + 2 : work;
}
inline const int4* seg_table(const SegList* seg) { return seg_on(seg) ? seg->table : nullptr; }
template <bool kSettle, int NP, bool kCode>
void run_prefilter(int64_t n, const int32_t* order, const int32_t* pa, const int32_t* pb, const double* coords_a,
                   const double* tol_a, const double* setup, double* measure, int32_t* nout, int32_t* survivors,
                   unsigned long long* work, const double* faces_a, const double* screen_b, const int64_t* n_dev,
                   const SegList* seg, cudaStream_t s) {
  const int gp = grid_for(n, 256, 8);
  if (seg_on(seg)) {
    count_launch(2);
    k_prefilter_tets<kSettle, NP, true, kCode><<<gp, 256, 0, s>>>(n, order, pa, pb, coords_a, tol_a, setup, measure, nout,
                                                           survivors, work, faces_a, screen_b, n_dev, seg->count);
    k_seg_chunks<<<gp, 256, 0, s>>>(n, n_dev, seg->count, seg->table, work);
  } else {
    count_launch();
    k_prefilter_tets<kSettle, NP, false, kCode><<<gp, 256, 0, s>>>(n, order, pa, pb, coords_a, tol_a, setup, measure, nout,
                                                     survivors, work, faces_a, screen_b, n_dev);
  }
}
}  // namespace

// ----------------------------------------------------------------------
// K6: depth-first tet clipper over point indices
// ----------------------------------------------------------------------
// One pair per lane, depth-first, lanes refilled from the survivor list; a
// tet is four byte indices into the lane's point pool in shared memory
// instead of twelve doubles in registers.  Pool slots 0-3 hold A's vertices; the split at
// plane L writes its (at most four) new points to slots 4+4L .. 7+4L.  In
// depth-first order that is safe: a tet at plane L references only points of
// planes < L, and when a sibling is taken from the stack every point written
// by the previous sibling's subtree belongs to planes >= its own.
// What a visit costs is mostly integer work around 24 FP64 operations: lists of
// vertices by class, indices picked from them, children put together case by
// case.  All of that comes from the split table (below) instead: a table word
// for the classes gives the order in which to fetch the vertices, so that the
// interpolated edges are the same registers in every case, and the children
// as byte permutes of the old tet and the new points.  Early-out pass and
// clipper, tet3d_graded_55x51 8.61 -> 7.66 ms, tet3d_27x32 1.83 -> 1.61 ms
// (952 -> 709 million warp instructions in the clipper); 524,288 tet-hexahedron pairs, whole
// call, 1.06 -> 0.92 ms.
constexpr int kIxPoints = 20;  // 4 + 4 per plane
#ifndef LSM_IX_BLOCK
#define LSM_IX_BLOCK 480
#endif
#ifndef LSM_IX_BPS
#define LSM_IX_BPS 1
#endif
// 480 B of shared memory per lane (the point pool; pending tets are kept in
// registers): one block of 480 threads (15 warps) fills the 228 KB of an SM.
constexpr int kIxBlock = LSM_IX_BLOCK;
constexpr int kIxBlocksPerSm = LSM_IX_BPS;

__device__ __forceinline__ unsigned ix_pack(unsigned a, unsigned b, unsigned c, unsigned d) {
  return a | b << 5 | c << 10 | d << 15;
}

__device__ __forceinline__ unsigned ix_vert(unsigned tet, int v) { return (tet >> (5 * v)) & 31u; }

__device__ __forceinline__ unsigned ix_set(unsigned tet, int v, unsigned j) {
  return (tet & ~(31u << (5 * v))) | j << (5 * v);
}

// A lane's point pool: point j, coordinate c at pool[(3j + c) * BLOCK]
// (consecutive lanes hit consecutive banks).
template <int BLOCK>
struct IxPool {
  double* pool;
  __device__ __forceinline__ V3 get(unsigned j) const {
    const double* q = pool + 3 * j * BLOCK;
    return V3{q[0], q[BLOCK], q[2 * BLOCK]};
  }
  __device__ __forceinline__ void put(unsigned j, const V3& v) const {
    double* q = pool + 3 * j * BLOCK;
    q[0] = v.x;
    q[BLOCK] = v.y;
    q[2 * BLOCK] = v.z;
  }
};

template <class Pool>
__device__ __forceinline__ void ix_gather(const Pool& pool, unsigned tet, Tet& t) {
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const V3 q = pool.get(ix_vert(tet, v));
    t.x[v] = q.x;
    t.y[v] = q.y;
    t.z[v] = q.z;
  }
}

// Coordinates of a tet of four byte indices.
template <class Pool>
__device__ __forceinline__ void ix_bytes(const Pool& pool, unsigned tet, Tet& t) {
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const V3 q = pool.get((tet >> (8 * v)) & 255u);
    t.x[v] = q.x;
    t.y[v] = q.y;
    t.z[v] = q.z;
  }
}

// Split of tet `cur` (coordinates t, classification k) at the plane whose new
// points go to pool slots base .. base+3 (Tetrahedron_Intersection.F90:290-434,
// same cases, interpolations and child order as split_tet).  Returns the
// number of children; c0..c2 receive their index tuples.
template <class Pool>
__device__ __forceinline__ int ix_split(unsigned cur, const TetClass& k, const Pool& pool, unsigned base,
                                        unsigned& c0, unsigned& c1, unsigned& c2) {
  const int nn = k.nn, np = k.np;
  const int n0 = k.negl & 3, n1 = (k.negl >> 2) & 3, n2 = (k.negl >> 4) & 3;
  const int p0 = k.posl & 3, p1 = (k.posl >> 2) & 3, p2 = (k.posl >> 4) & 3;
  int ni;
  unsigned pairs;
  if (nn == 1) {
    ni = np;
    pairs = (unsigned)(p0 | n0 << 2) | (unsigned)(p1 | n0 << 2) << 4 | (unsigned)(p2 | n0 << 2) << 8;
  } else if (np == 2) {
    ni = 4;
    pairs = (unsigned)(p0 | n0 << 2) | (unsigned)(p1 | n0 << 2) << 4 | (unsigned)(p0 | n1 << 2) << 8 |
            (unsigned)(p1 | n1 << 2) << 12;
  } else {
    ni = nn;
    pairs = (unsigned)(p0 | n0 << 2) | (unsigned)(p0 | n1 << 2) << 4 | (unsigned)(p0 | n2 << 2) << 8;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (i < ni) {
      const int P = (pairs >> (4 * i)) & 3, N = (pairs >> (4 * i + 2)) & 3;
      const V3 T = interp(pool.get(ix_vert(cur, P)), pool.get(ix_vert(cur, N)),
                          sel4(P, k.d[0], k.d[1], k.d[2], k.d[3]), sel4(N, k.d[0], k.d[1], k.d[2], k.d[3]));
      pool.put(base + i, T);
    }
  }
  if (nn == 1) {  // +++-, ++-0, +-00: the r-th positive vertex becomes new point r
    unsigned c = cur;
#pragma unroll
    for (int r = 0; r < 3; ++r)
      if (r < np) c = ix_set(c, (k.posl >> (2 * r)) & 3, base + r);
    c0 = c;
    return 1;
  }
  if (np == 2) {  // ++--
    c0 = ix_set(ix_set(cur, p0, base + 2), p1, base + 1);
    c1 = ix_pack(ix_vert(cur, n1), base + 3, base + 2, base + 1);
    c2 = ix_pack(ix_vert(cur, n0), base + 0, base + 1, base + 2);
    return 3;
  }
  c0 = ix_set(cur, p0, base);
  if (nn == 3) {  // +---
    c1 = ix_pack(base + 0, ix_vert(cur, n1), ix_vert(cur, n2), base + 1);
    c2 = ix_pack(ix_vert(cur, n2), base + 1, base + 2, base + 0);
    return 3;
  }
  // +--0
  c1 = ix_pack(base + 1, ix_vert(cur, k.zerl & 3), ix_vert(cur, n1), base + 0);
  return 2;
}

// Pairs reach the lanes through a software pipeline so that the dependent
// loads of a new pair (survivor record {pair, a, b} -> A coordinates and
// tolerances) never stall the warp: every lane prefetches its next pair one
// stage per loop iteration while it clips the current one.  Records are
// taken from a warp-private cursor over chunks of kIxChunk list entries (one
// atomic per chunk).
constexpr int kIxChunk = 64;

// What the clipper does with a pair's kept output tets (each passed with
// its vertex-1 volume, in the reference's output order).  kInside: the list
// may hold pairs whose every plane is a no-op (A inside B: its one output
// tet is A itself), which the supermesh's early-out pass settles itself.
struct IxMeasureSink {
  static constexpr bool kInside = false;
  double* pair_measure;
  int32_t* pair_nout;
  double m;
  int kept;
  __device__ __forceinline__ void begin(const int4&) {
    m = 0.0;
    kept = 0;
  }
  __device__ __forceinline__ void tet(const Tet&, double v1) {
    m = m + v1;
    ++kept;
  }
  __device__ __forceinline__ void end(int64_t p) {
    pair_measure[p] = m;
    pair_nout[p] = kept;
  }
};

// Measure and count per pair and, for explicit pairs, the output tets:
// elems (optional) [n][kCap][4][3] in the reference's order (tets beyond
// kCap are counted, not stored: 729 for tet-hex).  The list includes pairs
// with every plane a no-op.
template <int kCap>
struct IxElemSinkT {
  static constexpr bool kInside = true;
  double* pair_measure;
  int32_t* pair_nout;
  double* elems;
  double m;
  int kept;
  int pid;
  __device__ __forceinline__ void begin(const int4& r) {
    m = 0.0;
    kept = 0;
    pid = r.x;
  }
  __device__ __forceinline__ void tet(const Tet& o, double v1) {
    if (elems && kept < kCap) {
      double2* e = reinterpret_cast<double2*>(elems + ((int64_t)pid * kCap + kept) * 12);
      e[0] = make_double2(o.x[0], o.y[0]);
      e[1] = make_double2(o.z[0], o.x[1]);
      e[2] = make_double2(o.y[1], o.z[1]);
      e[3] = make_double2(o.x[2], o.y[2]);
      e[4] = make_double2(o.z[2], o.x[3]);
      e[5] = make_double2(o.y[3], o.z[3]);
    }
    m = m + v1;
    ++kept;
  }
  __device__ __forceinline__ void end(int64_t p) {
    pair_measure[p] = m;
    pair_nout[p] = kept;
  }
};

// As IxMeasureSink, for a list that also holds the pairs with every plane a
// no-op.
struct IxInsideSink : IxMeasureSink {
  static constexpr bool kInside = true;
};

// As IxElemSinkT, but a pair's sum, count and output tets continue from
// what an earlier launch left in pair_measure / pair_nout / elems: the
// hexahedron-hexahedron pairs clip A's five tets in five launches, and the
// reference sums and lists all their output tets in one running order.
template <int kCap>
struct IxCarrySinkT {
  static constexpr bool kInside = true;
  double* pair_measure;
  int32_t* pair_nout;
  double* elems;
  double m;
  int kept;
  int pid;
  __device__ __forceinline__ void begin(const int4& r) {
    pid = r.x;
    m = pair_measure[pid];
    kept = pair_nout[pid];
  }
  __device__ __forceinline__ void tet(const Tet& o, double v1) {
    if (elems && kept < kCap) {
      double2* e = reinterpret_cast<double2*>(elems + ((int64_t)pid * kCap + kept) * 12);
      e[0] = make_double2(o.x[0], o.y[0]);
      e[1] = make_double2(o.z[0], o.x[1]);
      e[2] = make_double2(o.y[1], o.z[1]);
      e[3] = make_double2(o.x[2], o.y[2]);
      e[4] = make_double2(o.z[2], o.x[3]);
      e[5] = make_double2(o.y[3], o.z[3]);
    }
    m = m + v1;
    ++kept;
  }
  __device__ __forceinline__ void end(int64_t p) {
    pair_measure[p] = m;
    pair_nout[p] = kept;
  }
};
constexpr int kHexHexCap = 5 * 729;  // output tets per hexahedron pair

// Split table: for the 2-bit classes of a tet's vertices (0 zero, 1 negative,
// 2 positive) the order in which to gather them (their roles), and each child
// as a byte permute of (old tet, new points).  In role order the interpolated
// edges are the same for all cases: (0,3), (1,3), (2,3), except that ++-- takes
// (0,2) third and (1,2) fourth; interp_edge is symmetric in its ends, so a
// role's sign does not matter, and the edges that a case does not have give
// points nothing refers to.
// Byte permute: byte i of the result is byte s_i of (b : a), s_i the i-th
// nibble of s; with s_i's top bit set, that byte's sign instead (0 or 0xff).
__device__ __forceinline__ unsigned prmt(unsigned a, unsigned b, unsigned s) {
  unsigned r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(s));
  return r;
}

struct ClipTable {
  uint2 e[256];
};

// Entry for classes c: x = child 0 | child 1 << 16, y = child 2 | roles << 16,
// each four nibbles (vertex i of the child: 0-3 old vertex, 4-7 new point;
// roles: old vertex).  Bit 2 of the roles' nibbles 0-3: ++--, two or more
// children, three, a split (Tetrahedron_Intersection.F90:290-434: the same
// cases, interpolation and child order as split_tet).  Without a negative
// vertex the roles are 0: no child.
constexpr ClipTable make_clip_table() {
  ClipTable T{};
  for (unsigned c = 0; c < 256; ++c) {
    unsigned neg[4] = {}, pos[4] = {}, zer[4] = {};
    unsigned nn = 0, np = 0, nz = 0;
    bool ok = true;
    for (unsigned v = 0; v < 4; ++v) {
      const unsigned k = (c >> (2 * v)) & 3u;
      if (k == 0) zer[nz++] = v;
      if (k == 1) neg[nn++] = v;
      if (k == 2) pos[np++] = v;
      if (k == 3) ok = false;
    }
    unsigned role[4] = {0, 1, 2, 3}, ch[3][4] = {{0, 1, 2, 3}, {0, 1, 2, 3}, {0, 1, 2, 3}};
    unsigned kids = 1;
    bool two = false;
    if (ok && nn > 0 && np > 0) {
      if (nn == 1) {  // +++-, ++-0, +-00: the r-th positive vertex becomes new point r
        for (unsigned r = 0; r < 3; ++r) role[r] = r < np ? pos[r] : zer[r - np];
        role[3] = neg[0];
        for (unsigned r = 0; r < np; ++r) ch[0][pos[r]] = 4 + r;
      } else if (np == 2) {  // ++--
        two = true;
        kids = 3;
        role[0] = pos[0];
        role[1] = pos[1];
        role[2] = neg[1];
        role[3] = neg[0];
        ch[0][pos[0]] = 6;
        ch[0][pos[1]] = 5;
        const unsigned a[4] = {neg[1], 7, 6, 5}, b[4] = {neg[0], 4, 5, 6};
        for (unsigned i = 0; i < 4; ++i) {
          ch[1][i] = a[i];
          ch[2][i] = b[i];
        }
      } else {  // +---, +--0
        role[0] = neg[0];
        role[1] = neg[1];
        role[2] = nn == 3 ? neg[2] : zer[0];
        role[3] = pos[0];
        ch[0][pos[0]] = 4;
        kids = nn;
        const unsigned a3[4] = {4, neg[1], neg[2], 5}, b3[4] = {neg[2], 5, 6, 4}, a2[4] = {5, zer[0], neg[1], 4};
        for (unsigned i = 0; i < 4; ++i) {
          ch[1][i] = nn == 3 ? a3[i] : a2[i];
          if (nn == 3) ch[2][i] = b3[i];
        }
      }
    }
    unsigned w[4] = {};
    for (unsigned i = 0; i < 4; ++i) {
      for (unsigned j = 0; j < 3; ++j) w[j] |= ch[j][i] << (4 * i);
      w[3] |= role[i] << (4 * i);
    }
    if (ok && nn > 0 && np > 0) w[3] |= 1u << 14;
    if (!ok || nn == 0) w[3] = 0;
    if (two) w[3] |= 1u << 2;
    if (kids >= 2) w[3] |= 1u << 6;
    if (kids == 3) w[3] |= 1u << 10;
    T.e[c].x = w[0] | w[1] << 16;
    T.e[c].y = w[2] | w[3] << 16;
  }
  return T;
}
__device__ const ClipTable g_clip_table = make_clip_table();
constexpr int kClipTableBytes = sizeof(ClipTable);

// The point where edge (X, Y) meets the plane, dx and dy the ends' distances
// (of opposite sign).  With i = 1/(dx - dy) it is (-dy i) X + (dx i) Y: for
// X positive exactly the reference's w0, w1; for X negative both the
// difference and the reciprocal change sign, which negates nothing in the
// products, and the sum's two terms change places.
__device__ __forceinline__ V3 interp_edge(const V3& X, const V3& Y, double dx, double dy) {
  const double i = __drcp_rn(dx - dy);
  const double wx = -dy * i, wy = dx * i;
  return V3{wx * X.x + wy * Y.x, wx * X.y + wy * Y.y, wx * X.z + wy * Y.z};
}

// Class bits of a distance at plane q (zero if |d| < eps; NaN is neither):
// bit q negative, bit 4 + q positive.
__device__ __forceinline__ unsigned class_bits(double d, unsigned neg_bit) {
  const unsigned hi = (unsigned)__double2hiint(d);
  const unsigned lim = 0x7ff00000u - kEpsHi;
  unsigned w = 0;
  if (hi - kEpsHi <= lim) w = neg_bit << 4;
  if ((hi ^ 0x80000000u) - kEpsHi <= lim) w = neg_bit;
  return w;
}

// Points in a lane's pool for NP planes: A's 4 vertices + 4 per plane.
__host__ __device__ constexpr int ix_points(int np) { return 4 + 4 * np; }

template <class Sink, int BLOCK, int BPS, int NP = 4>
__global__ void __launch_bounds__(BLOCK, BPS) k_clip_tets_ix(
    const int4* __restrict__ list, const unsigned long long* __restrict__ nlist, const double* __restrict__ coords_a,
    const double* __restrict__ tol_a, const double* __restrict__ setup_b, Sink sk, unsigned long long* work,
    const int4* __restrict__ chunks = nullptr) {
  // chunks (optional): the list is segmented; nlist then counts the table's
  // chunks and work counts the chunks taken
  static_assert(ix_points(NP) <= 32, "the last point byte leaves three bits for the plane");
  extern __shared__ double ix_mem[];
  uint2* table = reinterpret_cast<uint2*>(ix_mem);
  for (int i = threadIdx.x; i < 256; i += BLOCK) table[i] = g_clip_table.e[i];
  __syncthreads();
  IxPool<BLOCK> pool{ix_mem + kClipTableBytes / 8 + threadIdx.x};
  // pending tets (at most 2 per plane but the last), newest first: four point
  // bytes each, the plane to clip at next in the top bits
  constexpr int kW = 2 * (NP - 1);
  unsigned stk[kW];
#pragma unroll
  for (int w = 0; w < kW; ++w) stk[w] = 0;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t npairs = (int64_t)*nlist;
  // warp cursor over the list (warp-uniform)
  int64_t cbeg = 0, cend = 0;
  bool exhausted = false;
  // prefetch pipeline of the next pair: stage 0 idle, 1 record loading,
  // 2 element data loading (ready for the next refill)
  int nstage = 0;
  int4 nrec = make_int4(0, 0, 0, 0);
  Tet nt;
  double ntol = 0.0;
  // current pair
  int64_t p = -1;
  const double* planes = setup_b;
  unsigned cur = 0;
  double tol = 0.0;
  int L = 0, sp = 0;
  // planes this pair clips at (bit L; the prefilter's no-op planes are
  // skipped) and the last of them
  constexpr unsigned kAll = (1u << NP) - 1u;
  unsigned act = kAll;
  int lastL = NP - 1;
  for (;;) {
    // ---- prefetch pipeline
    if (nstage == 1) {
      load_tet(coords_a + (int64_t)nrec.y * 12, nt);
      ntol = fmin(tol_a[nrec.y], setup_b[(int64_t)nrec.z * clip_row(NP) + 4 * NP]);
      nstage = 2;
    }
    if (p < 0 && nstage == 2) {
      p = nrec.x;
#pragma unroll
      for (int v = 0; v < 4; ++v) pool.put(v, V3{nt.x[v], nt.y[v], nt.z[v]});
      planes = setup_b + (int64_t)nrec.z * clip_row(NP);
      tol = ntol;
      cur = 0x03020100u;
      sk.begin(nrec);
      act = ~(unsigned)nrec.w & kAll;  // never 0 unless Sink::kInside
      L = __ffs(act) - 1;
      lastL = 31 - __clz(act);
      sp = 0;
      nstage = 0;
      if (Sink::kInside && act == 0u) {
        // A inside all four planes: the reference keeps A as its one tet
        Tet o;
        ix_bytes(pool, cur, o);
        double v1;
        if (final_tet_keep(o, tol, v1)) sk.tet(o, v1);
        sk.end(p);
        p = -1;
      }
    }
    {
      const bool want = nstage == 0 && !exhausted;
      unsigned wm = __ballot_sync(full, want);
      while (wm) {
        if (cbeg >= cend) {
          unsigned long long base = 0;
          if (lane == 0) base = atomicAdd(work, chunks ? 1ull : (unsigned long long)kIxChunk);
          base = __shfl_sync(full, base, 0);
          if ((int64_t)base >= npairs) {
            exhausted = true;
            break;
          }
          if (chunks) {
            const int4 ch = chunks[base];
            cbeg = ch.x;
            cend = ch.y;
          } else {
            cbeg = (int64_t)base;
            cend = cbeg + kIxChunk < npairs ? cbeg + kIxChunk : npairs;
          }
        }
        const int navail = (int)(cend - cbeg);
        const int rank = __popc(wm & lt);
        const bool take = want && ((wm >> lane) & 1u) && rank < navail;
        if (take) {
          nrec = list[cbeg + rank];
          nstage = 1;
        }
        const unsigned tm = __ballot_sync(full, take);
        cbeg += __popc(tm);
        wm &= ~tm;
      }
    }
    if (__all_sync(full, p < 0 && nstage == 0 && exhausted)) break;
    if (p < 0) continue;
    double nx, ny, nz, c;
    load_plane(planes, L, nx, ny, nz, c);
    // classes from the signs, one bit each, unless a distance is neither
    // clearly positive nor clearly negative (as in surv_code)
    uint2 e;
    {
      unsigned neg = 0, irr = 0;
      double d[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const V3 v = pool.get((cur >> (8 * i)) & 255u);
        d[i] = ((nx * v.x + ny * v.y) + nz * v.z) - c;
        const unsigned hi = (unsigned)__double2hiint(d[i]);
        neg |= (hi >> 31) << (2 * i);
        irr = max(irr, 2u * hi - 2u * kEpsHi);
      }
      unsigned code = neg | (neg ^ 0x55u) << 1;
      if (irr >= 2u * (0x7ff00000u - kEpsHi)) {
        code = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned b = class_bits(d[i], 1u);
          code |= ((b & 1u) | (b >> 4) << 1) << (2 * i);
        }
      }
      e = table[code];
    }
    int k = (int)(e.y >> 20 & 1u);
    unsigned c0 = cur, c1 = 0, c2 = 0;
    if (e.y >> 30 & 1u) {
      const unsigned r = prmt(cur, cur, e.y >> 16);
      V3 v[4];
      double d[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i] = pool.get((r >> (8 * i)) & 255u);
        d[i] = ((nx * v[i].x + ny * v[i].y) + nz * v[i].z) - c;
      }
      const bool two = (e.y >> 18) & 1u;
      const unsigned base = 4u + 4u * (unsigned)L;
      pool.put(base, interp_edge(v[0], v[3], d[0], d[3]));
      pool.put(base + 1, interp_edge(v[1], v[3], d[1], d[3]));
      pool.put(base + 2, interp_edge(v[2], two ? v[0] : v[3], d[2], two ? d[0] : d[3]));
      if (two) pool.put(base + 3, interp_edge(v[1], v[2], d[1], d[2]));
      const unsigned fresh = base * 0x01010101u + 0x03020100u;
      c0 = prmt(cur, fresh, e.x);
      c1 = prmt(cur, fresh, e.x >> 16);
      c2 = prmt(cur, fresh, e.y);
      k = 1 + (int)(e.y >> 22 & 1u) + (int)(e.y >> 26 & 1u);
      // (the zero vertex of +--0 is the first of the reference's list, which a
      // NaN distance does not enter: then vertex 0)
      if (k == 2 && isnan(d[2])) c1 = prmt(c1, cur, 0x3240);
    }
    if (L == lastL) {
      // final tets, in the reference's order
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (j < k) {
          Tet o;
          ix_bytes(pool, j == 0 ? c0 : (j == 1 ? c1 : c2), o);
          double v1;
          if (final_tet_keep(o, tol, v1)) sk.tet(o, v1);
        }
      }
      k = 0;
    }
    if (k > 0) {
      const unsigned lv = (unsigned)(__ffs(act & (~0u << (L + 1))) - 1);  // next plane clipped at
      if (k == 3) {
#pragma unroll
        for (int w = kW - 1; w > 1; --w) stk[w] = stk[w - 2];
        stk[0] = c1 | lv << 29;
        stk[1] = c2 | lv << 29;
        sp += 2;
      } else if (k == 2) {
#pragma unroll
        for (int w = kW - 1; w > 0; --w) stk[w] = stk[w - 1];
        stk[0] = c1 | lv << 29;
        ++sp;
      }
      cur = c0;
      L = (int)lv;
      continue;
    }
    if (sp > 0) {
      cur = stk[0] & 0x1fffffffu;
      L = (int)(stk[0] >> 29);
#pragma unroll
      for (int w = 0; w < kW - 1; ++w) stk[w] = stk[w + 1];
      --sp;
      continue;
    }
    sk.end(p);
    p = -1;
  }
}

// ----------------------------------------------------------------------
// K6: breadth-first tet clipper, a warp per batch of pairs
// ----------------------------------------------------------------------
// A pair whose distances are not all finite, by visits as in k_clip_tets_ix
// (A's vertices in the pool): a vertex with a NaN distance belongs to none of
// the reference's three lists, which class bits cannot say.
template <class Pool, class Sink>
__device__ __forceinline__ void clip_nonfinite(const Pool& pool, const double* planes, unsigned act, double tol,
                                               unsigned (&st)[8], Sink& sk) {
  const int last = 31 - __clz(act);
  unsigned cur = ix_pack(0, 1, 2, 3), lv = 0;  // lv: 2 bits per pending tet
  int L = __ffs(act) - 1, sp = 0;
  for (;;) {
    Tet t;
    ix_gather(pool, cur, t);
    double nx, ny, nz, c;
    load_plane(planes, L, nx, ny, nz, c);
    TetClass cls;
    classify_tet(t, nx, ny, nz, c, cls);
    int k = 0;
    unsigned ch[3] = {cur, 0, 0};
    if (cls.nn > 0) k = cls.np == 0 ? 1 : ix_split(cur, cls, pool, 4 + 4 * L, ch[0], ch[1], ch[2]);
    if (L == last) {
#pragma unroll 1
      for (int j = 0; j < k; ++j) {
        ix_gather(pool, j == 0 ? ch[0] : (j == 1 ? ch[1] : ch[2]), t);
        double v1;
        if (final_tet_keep(t, tol, v1)) sk(t, v1);
      }
      k = 0;
    }
    const int next = __ffs(act & (~0u << (L + 1))) - 1;
#pragma unroll
    for (int j = 2; j > 0; --j)
      if (j < k) {
#pragma unroll
        for (int i = 7; i > 0; --i) st[i] = st[i - 1];
        st[0] = ch[j];
        lv = lv << 2 | (unsigned)next;
        ++sp;
      }
    if (k > 0) {
      cur = ch[0];
      L = next;
      continue;
    }
    if (sp == 0) break;
    cur = st[0];
    L = (int)(lv & 3u);
#pragma unroll
    for (int i = 0; i < 7; ++i) st[i] = st[i + 1];
    lv >>= 2;
    --sp;
  }
}

// Depth-first clipping by one lane per pair (k_clip_tets_ix) leaves half the
// lanes idle: they keep, drop or split at different moments, and at the last
// plane up to three volumes run in a row while the others wait.  Where a final
// tet costs more than its volume (the P1 quadrature, the stores of the
// supermesh's tets), or where there are too few pairs for a lane each to fill
// the chip and the longest pair's serial walk is the time (a hundred visits of
// about 1000 instructions), the whole warp works on the tets of a batch of
// pairs instead, breadth first: one list of tets per generation (the number of
// the pair's active planes left), one round at a time over up to 32 tets of
// one generation, children appended in order.  Every list keeps a pair's tets
// together and in the reference's breadth-first order, so the last
// generation's children come out in output order; a lane per pair then adds
// its volumes up.
// A point carries one byte with its class at the pair's planes (bits 0-3
// negative, 4-7 positive, in the order of the generations), evaluated once,
// when the point is created; a list entry carries its four vertices' bytes,
// and the same byte permute that makes a child's vertex indices out of the old
// tet's and the new points' makes its classes.
// Measured (tet3d_27x32 unless said): P1 mass 12.8 -> 5.9 ms; the emitting pass of the
// supermesh's elements 1.86 -> 1.53 ms; measures of 330 thousand candidates (10^3 x 6 against 12^3 x 6
// tets), early-out pass included, 0.212 -> 0.136 ms.  On the large measure
// passes k_clip_tets_ix is ahead (1.18 against 1.34 ms; as many instructions go
// into the lists and rounds as into the idle lanes of the other).
//
// Shared memory of a warp: the point pool (groups of four points: point i of
// group q at index 4 q + (i ^ (q >> 2 & 3)), so that the i-th points of
// sixteen consecutive groups fall into different banks; a split's new points
// are a group, and so are A's vertices), the planes of each slot's pair in the order
// of the generations, the lists, and the final tets of one round.
constexpr int kBfRow = 18;     // doubles per slot: four planes, tolerance, pad
constexpr int kBfRing = 128;   // entries in the list of generations 1-3
constexpr int kBfFinals = 96;  // final tets of one round, at most
template <int Q>
struct BfPool {
  static_assert(Q <= 128, "nine index bits");
  double* x;
  __device__ __forceinline__ V3 get(unsigned j) const { return V3{x[j], x[4 * Q + j], x[8 * Q + j]}; }
  __device__ __forceinline__ void put(unsigned j, const V3& v) const {
    x[j] = v.x;
    x[4 * Q + j] = v.y;
    x[8 * Q + j] = v.z;
  }
  static __device__ __forceinline__ unsigned at(unsigned q, unsigned i) { return 4 * q + (i ^ (q >> 2 & 3u)); }
  // A tet's point indices: their low bytes in one word, their high bits in
  // the bytes of another.  Those of group q:
  static __device__ __forceinline__ unsigned lo(unsigned q) {
    return (4 * q & 255u) * 0x01010101u + (0x03020100u ^ (q >> 2 & 3u) * 0x01010101u);
  }
  static __device__ __forceinline__ unsigned hi(unsigned q) { return (q >> 6) * 0x01010101u; }
};
template <int V>
__device__ __forceinline__ unsigned bf_vert(unsigned lo, unsigned hi) {
  return prmt(lo, hi, V | (4 + V) << 4 | (12 + V) << 8 | (12 + V) << 12);
}
template <class Pool>
__device__ __forceinline__ void bf_gather(const Pool& pool, unsigned lo, unsigned hi, V3 (&v)[4]) {
  v[0] = pool.get(bf_vert<0>(lo, hi));
  v[1] = pool.get(bf_vert<1>(lo, hi));
  v[2] = pool.get(bf_vert<2>(lo, hi));
  v[3] = pool.get(bf_vert<3>(lo, hi));
}
template <class Pool>
__device__ __forceinline__ void bf_tet(const Pool& pool, unsigned lo, unsigned hi, Tet& t) {
  V3 v[4];
  bf_gather(pool, lo, hi, v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    t.x[i] = v[i].x;
    t.y[i] = v[i].y;
    t.z[i] = v[i].z;
  }
}
template <int P, int Q>
__host__ __device__ constexpr int bf_warp_bytes() {
  return 8 * (12 * Q + P * kBfRow + kBfFinals) + 12 * (3 * kBfRing + 32) + 4 * 32;
}
__device__ __forceinline__ void store_tet(double* at, const Tet& o) {
  double2* e = reinterpret_cast<double2*>(at);
  e[0] = make_double2(o.x[0], o.y[0]);
  e[1] = make_double2(o.z[0], o.x[1]);
  e[2] = make_double2(o.y[1], o.z[1]);
  e[3] = make_double2(o.x[2], o.y[2]);
  e[4] = make_double2(o.z[2], o.x[3]);
  e[5] = make_double2(o.y[3], o.z[3]);
}

// What is done with a pair's kept output tets.  kSum: their vertex-1 volumes
// are added up in the reference's order, stored with their count; kStore: the
// tets are written, the k-th of the pair in slot s at place(s) + k; kP1: the
// P1 quadrature.  kSlots: pairs per batch; kWarps: warps per SM; kQuads:
// groups of points; kKeep: groups left to every deeper generation; kRoom:
// groups a generation must be able to take for its next round to come before
// a deeper partial one; kExtra: bytes of shared memory per warp beyond the
// clipper's own.
struct BfMeasureSink {
  static constexpr bool kSum = true, kStore = false, kP1 = false;
  static constexpr int kSlots = 32, kWarps = 10, kQuads = 128, kRoom = 24, kKeep = 8, kExtra = 0;
  double* pair_measure;
  int32_t* pair_nout;
};

// Explicit pairs' output tets: elems [n][81][4][3] (tets beyond 81 are
// counted, not stored).
struct BfElemSink {
  static constexpr bool kSum = true, kStore = true, kP1 = false;
  static constexpr int kSlots = 32, kWarps = 9, kQuads = 128, kRoom = 24, kKeep = 8, kExtra = 32 * 20;
  double* pair_measure;
  int32_t* pair_nout;
  double* elems;
  __device__ __forceinline__ int64_t place(const int4& rec) const { return (int64_t)rec.x * 81; }
  __device__ __forceinline__ void store(const Tet& o, int64_t base, int k, int2) const {
    if (k < 81) store_tet(elems + (base + k) * 12, o);
  }
};

// The supermesh's tets, written where the scan of the per-pair counts puts
// them, with their parents.
struct BfEmitSink {
  static constexpr bool kSum = false, kStore = true, kP1 = false;
  static constexpr int kSlots = 32, kWarps = 9, kQuads = 128, kRoom = 24, kKeep = 8, kExtra = 32 * 20;
  const int64_t* pair_off;
  double* elems;
  int64_t* parent_a;
  int64_t* parent_b;
  __device__ __forceinline__ int64_t place(const int4& rec) const { return pair_off[rec.x]; }
  __device__ __forceinline__ void store(const Tet& o, int64_t base, int k, int2 ab) const {
    store_tet(elems + (base + k) * 12, o);
    if (parent_a) parent_a[base + k] = ab.x;
    if (parent_b) parent_b[base + k] = ab.y;
  }
};

template <class Sink>
__host__ __device__ constexpr int bf_bytes() {
  return bf_warp_bytes<Sink::kSlots, Sink::kQuads>() + Sink::kExtra;
}

template <class Sink>
__global__ void __launch_bounds__(Sink::kWarps * 32, 1) k_clip_tets_bf(
    const int4* __restrict__ list, const unsigned long long* __restrict__ nlist, const double* __restrict__ coords_a,
    const double* __restrict__ tol_a, const double* __restrict__ setup_b, Sink sk, unsigned long long* work,
    const int4* __restrict__ chunks) {
  constexpr int P = Sink::kSlots, Q = Sink::kQuads;
  extern __shared__ double ix_mem[];
  uint2* table = reinterpret_cast<uint2*>(ix_mem);
  for (int i = threadIdx.x; i < 256; i += Sink::kWarps * 32) table[i] = g_clip_table.e[i];
  __syncthreads();
  char* wm = reinterpret_cast<char*>(ix_mem) + kClipTableBytes + (threadIdx.x >> 5) * bf_bytes<Sink>();
  BfPool<Q> pool{reinterpret_cast<double*>(wm)};
  double* rows = pool.x + 12 * Q;
  uint2* fin = reinterpret_cast<uint2*>(rows + P * kBfRow);  // {low bytes, high bits | slot << 27}
  // lists of generations 1-3 (kBfRing entries each), then 0 (32)
  unsigned* llo = reinterpret_cast<unsigned*>(fin + kBfFinals);
  unsigned* lhi = llo + 3 * kBfRing + 32;
  unsigned* lcl = lhi + 3 * kBfRing + 32;
  unsigned short* seg = reinterpret_cast<unsigned short*>(lcl + 3 * kBfRing + 32);  // [2][32]
  char* extra = wm + bf_warp_bytes<P, Q>();
  // a final tet's volume takes the place of its indices, except where those
  // are needed again
  double* vol = Sink::kP1 ? reinterpret_cast<double*>(extra) : reinterpret_cast<double*>(fin);
  int64_t* s_base = reinterpret_cast<int64_t*>(extra);         // kStore: [32]
  int2* s_ab = reinterpret_cast<int2*>(extra + 32 * 8);        // kStore: [32]
  int* s_run = reinterpret_cast<int*>(extra + 32 * 16);        // kStore: [32] tets stored so far
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t npairs = (int64_t)*nlist;
  int64_t cbeg = 0, cend = 0;
  // the next batch's records, fetched while the current one is clipped
  int nnext = 0;
  int4 nrec = make_int4(0, -1, 0, 0);
  bool done = false;
  auto fetch = [&] {
    nnext = 0;
    if (cbeg >= cend && !done) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(work, chunks ? 1ull : (unsigned long long)kIxChunk);
      base = __shfl_sync(full, base, 0);
      if ((int64_t)base >= npairs) {
        done = true;
      } else if (chunks) {
        const int4 ch = chunks[base];
        cbeg = ch.x;
        cend = ch.y;
      } else {
        cbeg = (int64_t)base;
        cend = cbeg + kIxChunk < npairs ? cbeg + kIxChunk : npairs;
      }
    }
    if (cbeg < cend) {
      nnext = cend - cbeg < P ? (int)(cend - cbeg) : P;
      if (lane < nnext) nrec = list[cbeg + lane];
      cbeg += nnext;
    }
  };
  fetch();
  while (nnext) {
    // ---- a batch of up to P pairs, slot = lane; neighbours with the same A
    // share its points
    const int n = nnext;
    const bool mine = lane < n;
    const int4 rec = nrec;
    const int prev = __shfl_up_sync(full, rec.y, 1);
    const bool fresh = mine && (lane == 0 || prev != rec.y);
    const unsigned fm = __ballot_sync(full, fresh);
    const unsigned aq = __popc(fm & (lt | 1u << lane)) - 1u;
    const unsigned act = ~(unsigned)rec.w & 15u;
    const int gen = mine ? 4 - __popc(act) : -1;  // generation the pair enters at
    unsigned x = 0;
    bool odd = false;
    if (mine) {
      const double* row = setup_b + (int64_t)rec.z * clip_row(4);
      const unsigned w = (unsigned)rec.w;
      Tet t;
      if (fresh || (w >> 30)) load_tet(coords_a + (int64_t)rec.y * 12, t);
      double* o = rows + lane * kBfRow;
      st2(o + 16, fmin(tol_a[rec.y], row[16]), 0.0);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (act >> q & 1u) {
          const int h = 4 - __popc(act >> q);
          double nx, ny, nz, c;
          load_plane(row, q, nx, ny, nz, c);
          st2(o + 4 * h, nx, ny);
          st2(o + 4 * h + 2, nz, c);
          if (w >> 30) {
            int bad = 0, nan = 0;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const double d = ((nx * t.x[v] + ny * t.y[v]) + nz * t.z[v]) - c;
              x |= class_bits(d, 1u << h) << (8 * v);
              bad += !isfinite(d);
              nan += isnan(d);
            }
            // (a plane of a degenerate B is NaN at every vertex and drops every tet)
            odd = odd || (bad > 0 && nan < 4);
          } else {
            x |= (((w >> (4 + 4 * (3 - q))) & 15u) * 0x00204081u & 0x01010101u) << h;
          }
        }
      }
      if (!(w >> 30)) {
        x = prmt(x, 0, 0x0123);
        x |= (~x & 0x0f0f0f0fu) << 4;
      }
      if (fresh) {
#pragma unroll
        for (int v = 0; v < 4; ++v) pool.put(pool.at(aq, v), V3{t.x[v], t.y[v], t.z[v]});
      }
      if constexpr (Sink::kStore) {
        s_base[lane] = sk.place(rec);
        s_ab[lane] = make_int2(rec.y, rec.z);
        s_run[lane] = 0;
      }
      if constexpr (Sink::kP1) sk.begin(extra, lane, rec);
    }
    fetch();
    if (lane < nnext) {  // the next batch's rows into L2
      const double* ca = coords_a + (int64_t)nrec.y * 12;
      const double* row = setup_b + (int64_t)nrec.z * clip_row(4);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(ca));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(row));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(row + 16));
    }
    double m = 0.0;
    int kept = 0;
    // lists: counts and heads, 8 bits per generation; groups in use below
    // each generation's own
    unsigned cnt = 0, head = 0, mark = (unsigned)__popc(fm) * 0x01010101u;
    int nf = 0;  // final tets to take
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const bool in = gen == g && !odd && (x & (0x01010101u << g));
      const unsigned b = __ballot_sync(full, in);
      if (in) {
        const int at = (g == 0 ? 3 : g - 1) * kBfRing + __popc(b & lt);
        llo[at] = pool.lo(aq);
        lhi[at] = pool.hi(aq) | (unsigned)lane << 27;
        lcl[at] = x;
      }
      cnt |= (unsigned)__popc(b) << (8 * g);
    }
    {  // pairs whose every plane is a no-op: A itself is the final tet
      const unsigned b = __ballot_sync(full, gen == 4);
      nf = __popc(b);
      if (nf) {
        const int at = __popc(b & lt);
        if (gen == 4) fin[at] = make_uint2(pool.lo(aq), pool.hi(aq) | (unsigned)lane << 27);
        seg[lane] = (unsigned short)at;
        seg[32 + lane] = (unsigned short)(at + (gen == 4));
      }
    }
    __syncwarp();
    for (;;) {
      if (nf) {
        // ---- final tets, in the pairs' order
        for (int f0 = 0; f0 < nf; f0 += 32) {
          const int f = f0 + lane;
          const bool on = f < nf;
          uint2 t = make_uint2(0, 0xffffffffu);
          Tet o;
          double v1 = 0.0;
          bool keep = false;
          if (on) {
            t = fin[f];
            bf_tet(pool, t.x, t.y & 0x03030303u, o);
            keep = final_tet_keep(o, rows[(t.y >> 27) * kBfRow + 16], v1);
          }
          if constexpr (Sink::kStore) {
            // rank among the pair's kept tets: those stored so far, and those
            // of this step's lanes from the pair's first one on
            const unsigned slot = t.y >> 27;
            const unsigned before = __shfl_up_sync(full, slot, 1), after = __shfl_down_sync(full, slot, 1);
            const unsigned km = __ballot_sync(full, keep);
            const unsigned hm = __ballot_sync(full, lane == 0 || before != slot);
            const unsigned first = 31 - __clz(hm & (lt | 1u << lane));
            const int k = on ? s_run[slot] + __popc(km & lt & ~((1u << first) - 1u)) : 0;
            if (keep) sk.store(o, s_base[slot], k, s_ab[slot]);
            __syncwarp();
            if (on && (lane == 31 || f + 1 == nf || after != slot)) s_run[slot] = k + keep;
            __syncwarp();
          }
          // (-1: dropped; a kept tet's volume may be NaN, where its products overflow)
          if (on && (Sink::kSum || Sink::kP1)) vol[f] = keep ? v1 : -1.0;
        }
        __syncwarp();
        if constexpr (Sink::kSum) {
          int f = seg[lane];
          const int fe = seg[32 + lane];
#pragma unroll 1
          for (; f < fe; f += 4) {
            double v1[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v1[i] = f + i < fe ? vol[f + i] : -1.0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (!(v1[i] < 0.0)) {
                m = m + v1[i];
                ++kept;
              }
          }
        }
        if constexpr (Sink::kP1) sk.integrate(extra, pool, fin, vol, nf, lane);
        nf = 0;
        __syncwarp();
      }
      if (!cnt) break;
      // ---- a round: the deepest generation with tets; with fewer than a warp
      // of them, the one before it first, if its new points still fit
      int g = (31 - __clz(cnt)) >> 3;
      {
        const unsigned here = (cnt >> (8 * g)) & 255u;
        if (g > 0 && here < 32 && ((cnt >> (8 * (g - 1))) & 255u) &&
            ((mark >> (8 * g)) & 255u) + Sink::kRoom <= Q - Sink::kKeep * (4 - g))
          --g;
      }
      // new points go behind those that tets in the lists still refer to
      const unsigned deeper = cnt >> (8 * g) >> 8;
      unsigned top = (mark >> (8 * (g + (deeper != 0)))) & 255u;
      const unsigned room = Q - Sink::kKeep * (3 - g) - top;
      unsigned r = min((cnt >> (8 * g)) & 255u, 32u);
      const int src =
          (g == 0 ? 3 : g - 1) * kBfRing + ((((head >> (8 * g)) & 255u) + lane) & (g == 0 ? 31 : kBfRing - 1));
      const unsigned lo = llo[src], hs = lhi[src];
      x = lcl[src];
      const unsigned slot = hs >> 27, hi = hs & 0x03030303u;
      const unsigned cls = ((x >> g) & 0x01010101u) | ((x >> (g + 3)) & 0x02020202u);
      const uint2 e = table[(cls * 0x01041040u) >> 24];
      bool split = lane < (int)r && (e.y >> 30 & 1u);
      unsigned sm = __ballot_sync(full, split);
      if (__popc(sm) > (int)room) {  // the round ends before the first split that finds no room
        const unsigned over = __ballot_sync(full, split && __popc(sm & lt) >= (int)room);
        r = __ffs(over) - 1;
        sm &= (1u << r) - 1u;
        split = split && lane < (int)r;
      }
      const bool on = lane < (int)r;
      const unsigned quad = top + __popc(sm & lt);
      unsigned nm = 0;
      if (split) {
        const double* pr = rows + slot * kBfRow;
        V3 v[4];
        bf_gather(pool, prmt(lo, lo, e.y >> 16), prmt(hi, hi, e.y >> 16), v);
        double d[4];
        {
          const double2 n01 = *reinterpret_cast<const double2*>(pr + 4 * g);
          const double2 n2c = *reinterpret_cast<const double2*>(pr + 4 * g + 2);
#pragma unroll
          for (int i = 0; i < 4; ++i) d[i] = ((n01.x * v[i].x + n01.y * v[i].y) + n2c.x * v[i].z) - n2c.y;
        }
        const bool two = (e.y >> 18) & 1u;
        V3 T[4];
        T[0] = interp_edge(v[0], v[3], d[0], d[3]);
        T[1] = interp_edge(v[1], v[3], d[1], d[3]);
        T[2] = interp_edge(v[2], two ? v[0] : v[3], d[2], two ? d[0] : d[3]);
        T[3] = V3{0.0, 0.0, 0.0};
        if (two) T[3] = interp_edge(v[1], v[2], d[1], d[2]);
#pragma unroll
        for (int i = 0; i < 4; ++i) pool.put(pool.at(quad, i), T[i]);
        // classes of the new points: negative up to this plane (it keeps what
        // is left of the tet), evaluated at those after it
        nm = ((2u << g) - 1u) * 0x01010101u;
#pragma unroll 1
        for (int h = g + 1; h < 4; ++h) {
          const double2 n01 = *reinterpret_cast<const double2*>(pr + 4 * h);
          const double2 n2c = *reinterpret_cast<const double2*>(pr + 4 * h + 2);
          double q[4];
          unsigned neg = 0, irr = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            q[i] = ((n01.x * T[i].x + n01.y * T[i].y) + n2c.x * T[i].z) - n2c.y;
            const unsigned qh = (unsigned)__double2hiint(q[i]);
            neg = __funnelshift_l(qh, neg, 1);
            irr = max(irr, 2u * qh - 2u * kEpsHi);
          }
          if (irr < 2u * (0x7ff00000u - kEpsHi)) {
            const unsigned nb = prmt(neg * 0x00204081u & 0x01010101u, 0, 0x0123);
            nm |= (nb | (nb ^ 0x01010101u) << 4) << h;
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) nm |= class_bits(q[i], 1u << h) << (8 * i);
          }
        }
      }
      const unsigned nlo = pool.lo(quad), nhi = pool.hi(quad), sl = slot << 27;
      const bool k2 = on && (e.y >> 22 & 1u), k3 = on && (e.y >> 26 & 1u);
      const unsigned sel1 = e.x >> 16;
      // this round's tets leave the list
      top += __popc(sm);
      cnt -= r << (8 * g);
      head = (head & ~(255u << (8 * g))) | (((((head >> (8 * g)) & 255u) + r) & (kBfRing - 1)) << (8 * g));
      if (g < 3) {
        // children without a negative vertex at the next plane are dropped
        const unsigned nb = 0x01010101u << (g + 1);
        const unsigned x0 = prmt(x, nm, e.x), x1 = prmt(x, nm, sel1), x2 = prmt(x, nm, e.y);
        const bool f0 = on && (x0 & nb), f1 = k2 && (x1 & nb), f2 = k3 && (x2 & nb);
        const unsigned b0 = __ballot_sync(full, f0), b1 = __ballot_sync(full, f1), b2 = __ballot_sync(full, f2);
        unsigned at = ((head >> (8 * g + 8)) & 255u) + ((cnt >> (8 * g + 8)) & 255u) + __popc(b0 & lt) +
                      __popc(b1 & lt) + __popc(b2 & lt);
        auto put = [&](unsigned sel, unsigned xc) {
          const int l = g * kBfRing + (at++ & (kBfRing - 1));
          llo[l] = prmt(lo, nlo, sel);
          lhi[l] = prmt(hi, nhi, sel) | sl;
          lcl[l] = xc;
        };
        if (f0) put(e.x, x0);
        if (f1) put(sel1, x1);
        if (f2) put(e.y, x2);
        cnt += (unsigned)(__popc(b0) + __popc(b1) + __popc(b2)) << (8 * g + 8);
        mark = (mark & ~(255u << (8 * g + 8))) | top << (8 * g + 8);
      } else {
        // the children are final tets
        const unsigned b0 = __ballot_sync(full, on), b1 = __ballot_sync(full, k2), b2 = __ballot_sync(full, k3);
        unsigned at = __popc(b0 & lt) + __popc(b1 & lt) + __popc(b2 & lt);
        nf = __popc(b0) + __popc(b1) + __popc(b2);
        if (Sink::kSum) {
          seg[lane] = 0;
          seg[32 + lane] = 0;
        }
        const unsigned before = __shfl_up_sync(full, slot, 1), after = __shfl_down_sync(full, slot, 1);
        __syncwarp();
        if (on) {
          if (Sink::kSum && (lane == 0 || before != slot)) seg[slot] = (unsigned short)at;
          fin[at++] = make_uint2(prmt(lo, nlo, e.x), prmt(hi, nhi, e.x) | sl);
          if (k2) fin[at++] = make_uint2(prmt(lo, nlo, sel1), prmt(hi, nhi, sel1) | sl);
          if (k3) fin[at++] = make_uint2(prmt(lo, nlo, e.y), prmt(hi, nhi, e.y) | sl);
          if (Sink::kSum && (lane == (int)r - 1 || after != slot)) seg[32 + slot] = (unsigned short)at;
        }
      }
      __syncwarp();
    }
    // ---- pairs with distances that are not finite, one at a time
    for (unsigned om = __ballot_sync(full, odd); om; om &= om - 1u) {
      if (lane == __ffs(om) - 1) {
        Tet t;
        load_tet(coords_a + (int64_t)rec.y * 12, t);
#pragma unroll
        for (int v = 0; v < 4; ++v) pool.put(v, V3{t.x[v], t.y[v], t.z[v]});
        unsigned st[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) st[i] = 0;
        auto each = [&](const Tet& o, double v1) {
          if constexpr (Sink::kStore) sk.store(o, s_base[lane], kept, s_ab[lane]);
          if constexpr (Sink::kP1) sk.tet(extra, lane, o, v1);
          m = m + v1;
          ++kept;
        };
        clip_nonfinite(pool, setup_b + (int64_t)rec.z * clip_row(4), act, rows[lane * kBfRow + 16], st, each);
      }
      __syncwarp();
    }
    if constexpr (Sink::kSum) {
      if (mine) {
        sk.pair_measure[rec.x] = m;
        sk.pair_nout[rec.x] = kept;
      }
    }
    if constexpr (Sink::kP1) sk.end(extra, n, rec, lane);
    __syncwarp();
  }
}

// Measure passes of fewer candidate pairs than this go through
// k_clip_tets_bf.  Narrow phase of two meshes, k_clip_tets_ix / k_clip_tets_bf:
// 44 thousand candidates 148 / 93 us, 452 thousand 205 / 157, 1.37 million
// 300 / 277, 1.81 million 388 / 385, 4.2 million 661 / 698, 10 million 1655 /
// 1837 us.
constexpr int64_t kBfMeasureMax = 3 << 19;

template <class Sink>
size_t bf_smem_bytes() {
  return kClipTableBytes + (size_t)Sink::kWarps * bf_bytes<Sink>();
}
template <class Sink>
cudaError_t bf_attributes() {
  return cudaFuncSetAttribute(k_clip_tets_bf<Sink>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)bf_smem_bytes<Sink>());
}
template <class Sink>
void run_bf(const int4* list, const unsigned long long* nlist, const double* coords_a, const double* tol_a,
            const double* setup_b, const Sink& sk, unsigned long long* work, const int4* chunks, cudaStream_t s) {
  k_clip_tets_bf<Sink><<<sm_count(), Sink::kWarps * 32, bf_smem_bytes<Sink>(), s>>>(list, nlist, coords_a, tol_a,
                                                                                    setup_b, sk, work, chunks);
}

size_t ix_smem_bytes() { return (size_t)kIxBlock * 3 * kIxPoints * sizeof(double) + kClipTableBytes; }

// Per-pair setup of explicit tetrahedron pairs (the prep kernel's work for
// one-element meshes): B's planes and tolerance (setup row), A's tolerance,
// identity pair indices.
__global__ void k_setup_pairs3(int64_t n, const double* __restrict__ tet_a, const double* __restrict__ tet_b,
                               double* setup, double* tol_a, int32_t* iota) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    // both pair arrays are 16-byte aligned (checked by the entry points)
    Tet a, b;
    load_tet(tet_a + 12 * i, a);
    load_tet(tet_b + 12 * i, b);
    Planes P;
    tet_planes(b, P);
    double* o = setup + i * kSetup3;
#pragma unroll
    for (int L = 0; L < 4; ++L) {
      st2(o + 4 * L, P.nx[L], P.ny[L]);
      st2(o + 4 * L + 2, P.nz[L], P.c[L]);
    }
    st2(o + 16, 10.0 * spacing(tet_volume_v4(b)), 0.0);
    st2(o + 18, 0.0, 0.0);
    tol_a[i] = 10.0 * spacing(tet_volume_v4(a));
    iota[i] = (int32_t)i;
  }
}

// Setup and early-outs of explicit tetrahedron pairs in one pass, a thread per
// pair: B's planes stay in registers for k_prefilter_tets' tests, and only the
// pairs they leave write a setup row, A's tolerance and a survivor record (as
// kSeg and kCode there; pairs inside all planes are listed).  The separate
// passes wrote 428 bytes of setup per pair and read them back: 1,048,576
// pairs, of which a third survive, 0.32 -> 0.15 ms.  A's faces enter the second
// test as they come from the cross product: a direction need not be of unit
// length there, only the margins scaled (kept clear of underflow and, as the
// cross product is of the coordinates' square, of overflow).
__global__ void __launch_bounds__(256, 2) k_pairs_early(int64_t n, const double* __restrict__ tet_a,
                                                        const double* __restrict__ tet_b, double* setup,
                                                        double* tol_a, double* measure, int32_t* nout, int4* survivors,
                                                        int* seg_count, bool second) {
  __shared__ unsigned s_cnt;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t per = seg_per(n, gridDim.x);
  const int64_t beg = (int64_t)blockIdx.x * per;
  const int64_t end = beg + per < n ? beg + per : n;
  for (int64_t base = beg; base < end; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    bool live = false;
    int code = 0;
    if (i < end) {
      Tet t, u;
      load_tet(tet_a + 12 * i, t);
      load_tet(tet_b + 12 * i, u);
      Planes P;
      tet_planes(u, P);
      const double M = max_abs_tet(t);
      bool reject = false;
      unsigned neg = 0, irr = 0;
      int noop = 0;
#pragma unroll
      for (int L = 0; L < 4; ++L) {
        const double thr = kEps + 64.0 * kEps * (1.0 + 2.0 * fmax(M, fabs(P.c[L])));
        double dmin = DBL_MAX, dmax = -DBL_MAX;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const double d = ((P.nx[L] * t.x[k] + P.ny[L] * t.y[k]) + P.nz[L] * t.z[k]) - P.c[L];
          const unsigned hi = (unsigned)__double2hiint(d);
          neg = __funnelshift_l(hi, neg, 1);
          irr = max(irr, 2u * hi - 2u * kEpsHi);
          dmin = fmin(dmin, d);
          dmax = fmax(dmax, d);
        }
        reject = reject || dmin >= thr;
        noop |= dmax <= -thr ? 1 << L : 0;
      }
      code = surv_code(noop, neg, irr);
      if (!reject && second) {
        double g, tau, MB;
        tet_screen_factors(u, P, g, tau, MB);
        // B's planes bound a proper tet, and no partial sum of a projection (at
        // most 24 Mp^3) leaves the range
        const double Mp = fmax(M, MB);
        if (g < DBL_MAX && Mp < 0x1p330) {
          const double e = kEps + 128.0 * kEps * (1.0 + 2.0 * Mp);
          const double margin =
              1.01 * g * (tau + e) + 16.0 * kEps * (1.0 + Mp) + 128.0 * kEps * (1.0 + M);
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            // the face opposite vertex f, outwards
            const int p = f == 0 ? 1 : 0, q = f <= 1 ? 2 : 1, r = f <= 2 ? 3 : 2;
            const double ax = t.x[q] - t.x[p], ay = t.y[q] - t.y[p], az = t.z[q] - t.z[p];
            const double bx = t.x[r] - t.x[p], by = t.y[r] - t.y[p], bz = t.z[r] - t.z[p];
            double nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
            const double side = (nx * (t.x[f] - t.x[p]) + ny * (t.y[f] - t.y[p])) + nz * (t.z[f] - t.z[p]);
            if (side > 0.0) {
              nx = -nx;
              ny = -ny;
              nz = -nz;
            }
            const double size = (fabs(nx) + fabs(ny)) + fabs(nz);
            double h = -DBL_MAX, m = DBL_MAX;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              h = fmax(h, (nx * t.x[k] + ny * t.y[k]) + nz * t.z[k]);
              m = fmin(m, (nx * u.x[k] + ny * u.y[k]) + nz * u.z[k]);
            }
            reject = reject || (size > 0x1p-800 && m - h >= size * margin);
          }
        }
      }
      live = !reject;
      if (reject) {
        measure[i] = 0.0;
        nout[i] = 0;
      } else {
        double* o = setup + i * kSetup3;
#pragma unroll
        for (int L = 0; L < 4; ++L) {
          st2(o + 4 * L, P.nx[L], P.ny[L]);
          st2(o + 4 * L + 2, P.nz[L], P.c[L]);
        }
        st2(o + 16, 10.0 * spacing(tet_volume_v4(u)), 0.0);
        tol_a[i] = 10.0 * spacing(tet_volume_v4(t));
      }
    }
    const unsigned mask = __ballot_sync(0xffffffffu, live);
    if (mask) {
      const int leader = __ffs(mask) - 1;
      unsigned off = 0;
      if (lane == leader) off = atomicAdd(&s_cnt, (unsigned)__popc(mask));
      off = __shfl_sync(0xffffffffu, off, leader);
      if (live) survivors[beg + off + __popc(mask & ((1u << lane) - 1u))] = make_int4((int)i, (int)i, (int)i, code);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) seg_count[blockIdx.x] = (int)s_cnt;
}

cudaError_t launch_setup_pairs3(int64_t n, const double* tet_a, const double* tet_b, double* setup, double* tol_a,
                                int32_t* iota, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  k_setup_pairs3<<<grid_for(n, 256, 8), 256, 0, s>>>(n, tet_a, tet_b, setup, tol_a, iota);
  return cudaGetLastError();
}

// Explicit tet-hexahedron pairs through the same pipeline with six planes
// (Supermesh.F90:262-280 planes, tolerance from the tet alone): per-pair
// setup rows of clip_row(6) doubles (planes, +inf in the tolerance slot so
// that fmin keeps A's), the first early-out and the no-op planes, then the
// index clipper with a pool of 28 points.  320 threads per SM: 672 B of pool
// per lane.
constexpr int kIxHexBlock = 320;

size_t ix_hex_smem_bytes() { return (size_t)kIxHexBlock * 3 * ix_points(6) * sizeof(double) + kClipTableBytes; }

// kVec: hex_b is 16-byte aligned, each hexahedron is read in 12 16-byte loads
template <bool kVec>
__global__ void k_setup_hex_pairs(int64_t n, const double* __restrict__ tet_a, const double* __restrict__ hex_b,
                                  double* setup, double* tol_a, int32_t* iota) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double nx[6], ny[6], nz[6], c[6];
    if (kVec) {
      double h[24];
      const double2* q = reinterpret_cast<const double2*>(hex_b + 24 * i);
#pragma unroll
      for (int k = 0; k < 12; ++k) {
        const double2 v = __ldg(q + k);
        h[2 * k] = v.x;
        h[2 * k + 1] = v.y;
      }
      hex_planes(h, nx, ny, nz, c);
    } else {
      hex_planes(hex_b + 24 * i, nx, ny, nz, c);
    }
    double* o = setup + i * clip_row(6);
#pragma unroll
    for (int L = 0; L < 6; ++L) {
      st2(o + 4 * L, nx[L], ny[L]);
      st2(o + 4 * L + 2, nz[L], c[L]);
    }
    st2(o + 24, pos_inf(), 0.0);
    st2(o + 26, 0.0, 0.0);
    Tet a;
    load_tet(tet_a + 12 * i, a);
    tol_a[i] = 10.0 * spacing(tet_volume_v4(a));
    iota[i] = (int32_t)i;
  }
}

cudaError_t launch_tet_hex_pairs(int64_t n, const double* tet_a, const double* hex_b, double* measure, int32_t* nout,
                                 double* elems, double* setup, double* tol_a, int32_t* iota, int32_t* survivors,
                                 unsigned long long* work, cudaStream_t s, const SegList* seg) {
  cudaMemsetAsync(work, 0, 2 * sizeof(unsigned long long), s);
  if (n <= 0) return cudaGetLastError();
  count_launch(2);
  if ((reinterpret_cast<uintptr_t>(hex_b) & 15u) == 0)
    k_setup_hex_pairs<true><<<grid_for(n, 256, 8), 256, 0, s>>>(n, tet_a, hex_b, setup, tol_a, iota);
  else
    k_setup_hex_pairs<false><<<grid_for(n, 256, 8), 256, 0, s>>>(n, tet_a, hex_b, setup, tol_a, iota);
  const int4* list = reinterpret_cast<const int4*>(survivors);
  const int g = sm_count();
  if (elems) {
    run_prefilter<false, 6, false>(n, nullptr, iota, iota, tet_a, tol_a, setup, measure, nout, survivors, work, nullptr,
                            nullptr, nullptr, seg, s);
    k_clip_tets_ix<IxElemSinkT<729>, kIxHexBlock, 1, 6><<<g, kIxHexBlock, ix_hex_smem_bytes(), s>>>(
        list, seg_nlist(seg, work), tet_a, tol_a, setup, IxElemSinkT<729>{measure, nout, elems}, work + 1,
        seg_table(seg));
  } else {
    run_prefilter<true, 6, false>(n, nullptr, iota, iota, tet_a, tol_a, setup, measure, nout, survivors, work, nullptr,
                           nullptr, nullptr, seg, s);
    k_clip_tets_ix<IxMeasureSink, kIxHexBlock, 1, 6><<<g, kIxHexBlock, ix_hex_smem_bytes(), s>>>(
        list, seg_nlist(seg, work), tet_a, tol_a, setup, IxMeasureSink{measure, nout, 0.0, 0}, work + 1,
        seg_table(seg));
  }
  return cudaGetLastError();
}

// A hexahedron (Gmsh node order) as five tets, in the order and with the
// vertex order of the reference's slicing (Supermesh.F90:303-334).
__device__ constexpr int kHexTets[5][4] = {{2, 5, 6, 7}, {0, 2, 3, 7}, {0, 4, 5, 7}, {0, 1, 2, 5}, {0, 2, 5, 7}};

// Hexahedron-hexahedron pairs: B's six face planes (setup rows of
// clip_row(6) doubles with +inf in the tolerance slot), and A's five tets
// in the reference's slicing order (Supermesh.F90:303-334), tet k
// of pair i at sub[(k * n + i) * 12] with its tolerance at tol[k * n + i].
__global__ void k_setup_hex_hex(int64_t n, const double* __restrict__ hex_a, const double* __restrict__ hex_b,
                                double* setup, double* sub, double* tol, int32_t* iota) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double nx[6], ny[6], nz[6], c[6];
    hex_planes(hex_b + 24 * i, nx, ny, nz, c);
    double* o = setup + i * clip_row(6);
#pragma unroll
    for (int L = 0; L < 6; ++L) {
      st2(o + 4 * L, nx[L], ny[L]);
      st2(o + 4 * L + 2, nz[L], c[L]);
    }
    st2(o + 24, pos_inf(), 0.0);
    st2(o + 26, 0.0, 0.0);
    const double* h = hex_a + 24 * i;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      Tet t;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        t.x[v] = h[3 * kHexTets[k][v]];
        t.y[v] = h[3 * kHexTets[k][v] + 1];
        t.z[v] = h[3 * kHexTets[k][v] + 2];
      }
      double* q = sub + ((int64_t)k * n + i) * 12;
      st2(q + 0, t.x[0], t.y[0]);
      st2(q + 2, t.z[0], t.x[1]);
      st2(q + 4, t.y[1], t.z[1]);
      st2(q + 6, t.x[2], t.y[2]);
      st2(q + 8, t.z[2], t.x[3]);
      st2(q + 10, t.y[3], t.z[3]);
      tol[(int64_t)k * n + i] = 10.0 * spacing(tet_volume_v4(t));
    }
    iota[i] = (int32_t)i;
  }
}

cudaError_t launch_hex_hex_pairs(int64_t n, const double* hex_a, const double* hex_b, double* measure, int32_t* nout,
                                 double* elems, double* setup, double* sub, double* tol, int32_t* iota,
                                 int32_t* survivors, unsigned long long* work, cudaStream_t s, const SegList* seg) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  k_setup_hex_hex<<<grid_for(n, 256, 8), 256, 0, s>>>(n, hex_a, hex_b, setup, sub, tol, iota);
  cudaMemsetAsync(measure, 0, sizeof(double) * n, s);
  cudaMemsetAsync(nout, 0, sizeof(int32_t) * n, s);
  const int4* list = reinterpret_cast<const int4*>(survivors);
  for (int k = 0; k < 5; ++k) {
    // tet k of every pair: rejected pairs keep their carried results, the
    // others (A's tet inside all six planes included) add to them
    const double* tk = sub + (int64_t)k * n * 12;
    const double* lk = tol + (int64_t)k * n;
    cudaMemsetAsync(work, 0, 2 * sizeof(unsigned long long), s);
    run_prefilter<false, 6, false>(n, nullptr, iota, iota, tk, lk, setup, nullptr, nullptr, survivors, work, nullptr,
                            nullptr, nullptr, seg, s);
    count_launch();
    k_clip_tets_ix<IxCarrySinkT<kHexHexCap>, kIxHexBlock, 1, 6><<<sm_count(), kIxHexBlock, ix_hex_smem_bytes(), s>>>(
        list, seg_nlist(seg, work), tk, lk, setup, IxCarrySinkT<kHexHexCap>{measure, nout, elems}, work + 1,
        seg_table(seg));
  }
  return cudaGetLastError();
}

// The clipper over a survivor list that holds the pairs with every plane a
// no-op, with kCode words: measures and counts, and the output tets (elems).
static cudaError_t clip_listed(int64_t n, const double* tet_a, const double* tol_a, const double* setup,
                               double* measure, int32_t* nout, double* elems, int32_t* survivors,
                               unsigned long long* work, const SegList* seg, cudaStream_t s) {
  count_launch();
  const int4* list = reinterpret_cast<const int4*>(survivors);
  if (elems)
    run_bf(list, seg_nlist(seg, work), tet_a, tol_a, setup, BfElemSink{measure, nout, elems}, work + 1, seg_table(seg),
           s);
  else if (n < kBfMeasureMax)
    run_bf(list, seg_nlist(seg, work), tet_a, tol_a, setup, BfMeasureSink{measure, nout}, work + 1, seg_table(seg), s);
  else
    k_clip_tets_ix<IxInsideSink, kIxBlock, kIxBlocksPerSm>
        <<<sm_count() * kIxBlocksPerSm, kIxBlock, ix_smem_bytes(), s>>>(list, seg_nlist(seg, work), tet_a, tol_a, setup,
                                                                        IxInsideSink{{measure, nout, 0.0, 0}}, work + 1,
                                                                        seg_table(seg));
  return cudaGetLastError();
}

cudaError_t launch_clip_elems(int64_t n, const int32_t* pair_a, const int32_t* pair_b, const double* tet_a,
                              const double* tol_a, const double* setup, double* measure, int32_t* nout,
                              double* elems, int32_t* survivors, unsigned long long* work, const double* faces_a,
                              const double* screen_b, cudaStream_t s, const SegList* seg) {
  cudaMemsetAsync(work, 0, 2 * sizeof(unsigned long long), s);
  if (n <= 0) return cudaGetLastError();
  run_prefilter<false, 4, true>(n, nullptr, pair_a, pair_b, tet_a, tol_a, setup, measure, nout, survivors, work,
                                faces_a, screen_b, nullptr, seg, s);
  return clip_listed(n, tet_a, tol_a, setup, measure, nout, elems, survivors, work, seg, s);
}

cudaError_t launch_tet_pairs(int64_t n, const double* tet_a, const double* tet_b, double* measure, int32_t* nout,
                             double* elems, double* setup, double* tol_a, int32_t* survivors,
                             unsigned long long* work, bool second, const SegList& seg, cudaStream_t s) {
  cudaMemsetAsync(work, 0, 2 * sizeof(unsigned long long), s);
  if (n <= 0) return cudaGetLastError();
  const int gp = seg_blocks(n);
  count_launch(2);
  k_pairs_early<<<gp, 256, 0, s>>>(n, tet_a, tet_b, setup, tol_a, measure, nout, reinterpret_cast<int4*>(survivors),
                                   seg.count, second);
  k_seg_chunks<<<gp, 256, 0, s>>>(n, nullptr, seg.count, seg.table, work);
  return clip_listed(n, tet_a, tol_a, setup, measure, nout, elems, survivors, work, &seg, s);
}




// Deterministic per-block partials of the pair measures: block b reduces the
// contiguous range [b*chunk, (b+1)*chunk) in a fixed thread order.
__global__ void __launch_bounds__(256) k_reduce_pairs(int64_t npairs, const double* __restrict__ pm,
                                                      const int32_t* __restrict__ pn, Partial* partials,
                                                      const int64_t* __restrict__ n_dev) {
  if (n_dev && *n_dev < npairs) npairs = *n_dev;
  const int64_t chunk = (npairs + gridDim.x - 1) / gridDim.x;
  const int64_t beg = (int64_t)blockIdx.x * chunk;
  const int64_t end = beg + chunk < npairs ? beg + chunk : npairs;
  double sum = 0.0, err = 0.0;
  unsigned long long ni = 0, no = 0;
  for (int64_t i = beg + threadIdx.x; i < end; i += blockDim.x) {
    cs_add(sum, err, pm[i]);
    const int k = pn ? pn[i] : 0;
    ni += k > 0;
    no += k;
  }
  block_reduce_partial<256>(sum, err, ni, no, &partials[blockIdx.x]);
}

int clip_grid_blocks(int dim) { return sm_count() * (dim == 2 ? tri_blocks_per_sm() : kIxBlocksPerSm); }

cudaError_t launch_clip(int dim, int64_t npairs, const int32_t* pair_a, const int32_t* pair_b,
                        const double* coords_a, const double* tol_a, const double* setup_b,
                        double* pair_measure, int32_t* pair_nout, int32_t* overflow_list,
                        int* overflow_count, unsigned long long* work, cudaStream_t s,
                        const int32_t* order, cudaEvent_t ev_begin, cudaEvent_t ev_end, const double* faces_a,
                        const double* screen_b, const SchedBin* bin, const int64_t* n_dev, const SegList* seg) {
  const int g = clip_grid_blocks(dim);
  count_launch();
  if (dim == 2) {
    if (ev_begin) cudaEventRecord(ev_begin, s);
    k_clip_tris<<<g, kTriBlock, 0, s>>>(npairs, pair_a, pair_b, coords_a, tol_a, setup_b, pair_measure,
                                        pair_nout, overflow_list, overflow_count, order, n_dev);
  } else {
    // work[0]: survivor count, work[1]: clipper pair counter
    // the timed span covers the early-out pass and the clipper: together
    // they settle every candidate
    if (ev_begin) cudaEventRecord(ev_begin, s);
    cudaMemsetAsync(work, 0, 2 * sizeof(unsigned long long), s);
    // the binned orders read one list: with bin->flat the segments are
    // gathered into it first
    const SegList sg = (bin && !bin->flat) ? SegList{} : (seg ? *seg : SegList{});
    const bool bf = !bin && npairs < kBfMeasureMax;
    const auto early = bf ? run_prefilter<true, 4, true> : run_prefilter<true, 4, false>;
    early(npairs, order, pair_a, pair_b, coords_a, tol_a, setup_b, pair_measure, pair_nout,
                           overflow_list, work, faces_a, screen_b, n_dev, &sg, s);
    const int4* list = reinterpret_cast<const int4*>(overflow_list);
    if (bin) {
      if (seg_on(&sg)) {
        cudaError_t e = launch_seg_compact(npairs, work + 2, sg.table, list, bin->flat, s);
        if (e != cudaSuccess) return e;
        list = bin->flat;
      }
      // the survivors reordered into class-uniform runs within windows
      cudaError_t e = launch_sched_bin(*bin, list, work, bin->out, coords_a, s);
      if (e != cudaSuccess) return e;
      list = bin->out;
    }
    if (bf)
      run_bf(list, seg_nlist(&sg, work), coords_a, tol_a, setup_b, BfMeasureSink{pair_measure, pair_nout}, work + 1,
             seg_table(&sg), s);
    else
      k_clip_tets_ix<IxMeasureSink, kIxBlock, kIxBlocksPerSm>
          <<<sm_count() * kIxBlocksPerSm, kIxBlock, ix_smem_bytes(), s>>>(
              list, bin ? work : seg_nlist(&sg, work), coords_a, tol_a, setup_b,
              IxMeasureSink{pair_measure, pair_nout, 0.0, 0}, work + 1, bin ? nullptr : seg_table(&sg));
  }
  if (ev_end) cudaEventRecord(ev_end, s);
  return cudaGetLastError();
}

int reduce_pairs_blocks() { return kReduceBlocks; }

cudaError_t launch_reduce_pairs(int64_t npairs, const double* pair_measure, const int32_t* pair_nout,
                                Partial* partials, cudaStream_t s, const int64_t* n_dev) {
  count_launch();
  k_reduce_pairs<<<kReduceBlocks, 256, 0, s>>>(npairs, pair_measure, pair_nout, partials, n_dev);
  return cudaGetLastError();
}

// 2D supermesh triangles: one candidate pair per thread, clipped again with
// the narrow phase's arithmetic; pairs without output triangles are skipped
// (their offsets are equal).
__global__ void __launch_bounds__(128) k_tris_emit(int64_t npairs, const int32_t* __restrict__ pa,
                                                   const int32_t* __restrict__ pb, const double* __restrict__ coords_a,
                                                   const double* __restrict__ tol_a, const double* __restrict__ setup_b,
                                                   const int64_t* __restrict__ pair_off, double* elems,
                                                   int64_t* parent_a, int64_t* parent_b) {
  __shared__ double2 poly[kTriCap * 128];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < npairs;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t at = pair_off[i];
    if (pair_off[i + 1] == at) continue;
    const int a = pa[i], b = pb[i];
    const double2* va = reinterpret_cast<const double2*>(coords_a + (int64_t)a * 6);
    const double2 v[3] = {__ldg(va), __ldg(va + 1), __ldg(va + 2)};
    Lines L;
    double tolb;
    load_lines(setup_b + (int64_t)b * kSetup2, L, tolb);
    const double tol = fmin(tol_a[a], tolb);
    clip_tri_fan<128>(v, L, tol, poly + threadIdx.x, true,
             [&](int k, double x0, double y0, double x1, double y1, double x2, double y2) {
               double2* e = reinterpret_cast<double2*>(elems + (at + k) * 6);
               e[0] = make_double2(x0, y0);
               e[1] = make_double2(x1, y1);
               e[2] = make_double2(x2, y2);
               if (parent_a) parent_a[at + k] = a;
               if (parent_b) parent_b[at + k] = b;
             });
  }
}

cudaError_t launch_emit_elements(int dim, int64_t npairs, const int32_t* pair_a, const int32_t* pair_b,
                                 const double* coords_a, const double* tol_a, const double* setup_b,
                                 const int32_t* survivors, unsigned long long* work, const int64_t* pair_off,
                                 double* elems, int64_t* parent_a, int64_t* parent_b, cudaStream_t s,
                                 const SegList* seg) {
  if (npairs <= 0) return cudaSuccess;
  count_launch();
  if (dim == 2) {
    k_tris_emit<<<grid_for(npairs, 128, 8), 128, 0, s>>>(npairs, pair_a, pair_b, coords_a, tol_a, setup_b, pair_off,
                                                         elems, parent_a, parent_b);
    return cudaGetLastError();
  }
  // the survivors of the counting pass again (work[0] holds their number);
  // only the clipper's pair counter starts over
  cudaMemsetAsync(work + 1, 0, sizeof(unsigned long long), s);
  run_bf(reinterpret_cast<const int4*>(survivors), seg_nlist(seg, work), coords_a, tol_a, setup_b,
         BfEmitSink{pair_off, elems, parent_a, parent_b}, work + 1, seg_table(seg), s);
  return cudaGetLastError();
}

cudaError_t init_p1_attributes();

cudaError_t init_device_attributes() {
  cudaError_t e = cudaFuncSetAttribute(k_clip_tets_ix<IxMeasureSink, kIxBlock, kIxBlocksPerSm>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ix_smem_bytes());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_clip_tets_ix<IxInsideSink, kIxBlock, kIxBlocksPerSm>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ix_smem_bytes());
  if (e == cudaSuccess) e = bf_attributes<BfMeasureSink>();
  if (e == cudaSuccess) e = bf_attributes<BfElemSink>();
  if (e == cudaSuccess) e = bf_attributes<BfEmitSink>();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_clip_tets_ix<IxMeasureSink, kIxHexBlock, 1, 6>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ix_hex_smem_bytes());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_clip_tets_ix<IxCarrySinkT<kHexHexCap>, kIxHexBlock, 1, 6>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ix_hex_smem_bytes());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_clip_tets_ix<IxElemSinkT<729>, kIxHexBlock, 1, 6>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ix_hex_smem_bytes());
  if (e == cudaSuccess) e = init_p1_attributes();
  if (e != cudaSuccess) return e;
  return init_sched_attributes(kSchedMaxWindow);
}



cudaError_t launch_clip_tris_wide(const int32_t* overflow_list, const int* overflow_count, int64_t cap,
                                  const int32_t* pair_a, const int32_t* pair_b,
                                  const double* coords_a, const double* tol_a,
                                  const double* setup_b, double* pair_measure, int32_t* pair_nout,
                                  cudaStream_t s) {
  count_launch();
  k_clip_tris_wide<<<sm_count(), kTriWideBlock, 0, s>>>(overflow_list, overflow_count, cap, pair_a, pair_b, coords_a,
                                                        tol_a, setup_b, pair_measure, pair_nout);
  return cudaGetLastError();
}

// ======================================================================
// K7: finalize totals and per-row sums
// ======================================================================
// Merges the per-block partials in a fixed tree order (deterministic).
__global__ void __launch_bounds__(1024) k_finalize(const Partial* __restrict__ partials, int np, Partial* out) {
  double sum = 0.0, err = 0.0;
  unsigned long long ni = 0, no = 0;
  for (int b = threadIdx.x; b < np; b += blockDim.x) {
    two_sum_merge(sum, err, partials[b].sum, partials[b].err);
    ni += partials[b].n_int;
    no += partials[b].n_out;
  }
  __shared__ Partial r;
  block_reduce_partial<1024>(sum, err, ni, no, &r);
  __syncthreads();
  if (threadIdx.x == 0) {
    Partial p = r;
    p.sum = p.sum + p.err;
    *out = p;
  }
}

cudaError_t launch_finalize(const Partial* partials, int npartials, Partial* out, cudaStream_t s) {
  count_launch();
  k_finalize<<<1, 1024, 0, s>>>(partials, npartials, out);
  return cudaGetLastError();
}

// One thread per row, eight loads ahead of the adds (in row order).
__global__ void k_row_sums(int64_t nel_a, const int64_t* __restrict__ off, const double* __restrict__ pm,
                           double* out) {
  for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < nel_a;
       a += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    const int64_t end = off[a + 1];
    for (int64_t p = off[a]; p < end; p += 8) {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = p + k < end ? pm[p + k] : 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (p + k < end) s = s + v[k];
    }
    out[a] = s;
  }
}

cudaError_t launch_row_sums(int64_t nel_a, const int64_t* offsets, const double* pair_measure,
                            double* elem_measure, cudaStream_t s) {
  if (nel_a <= 0) return cudaSuccess;
  count_launch();
  const int B = nel_a < (int64_t)sm_count() * 512 ? 32 : 256;
  k_row_sums<<<grid_for(nel_a, B, 2048 / B), B, 0, s>>>(nel_a, offsets, pair_measure, elem_measure);
  return cudaGetLastError();
}

__global__ void k_i32_to_i64(int64_t n, const int32_t* __restrict__ in, int64_t* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[i];
}

cudaError_t launch_i32_to_i64(int64_t n, const int32_t* in, int64_t* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  k_i32_to_i64<<<grid_for(n, 256, 8), 256, 0, s>>>(n, in, out);
  return cudaGetLastError();
}

// ======================================================================
// Batched search: one hierarchy over many meshes
// ======================================================================
// The B elements of all meshes are sorted by (mesh, Morton), so a mesh's
// leaves are one range of the sorted order, its element range; a row visits
// only nodes that reach into the range of its own B mesh.
__global__ void k_pair_keys(int64_t n, const int32_t* __restrict__ vals, const int32_t* __restrict__ pair_of,
                            uint32_t* keys) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    keys[i] = (uint32_t)pair_of[vals[i]];
}

cudaError_t launch_pair_keys(int64_t n, const int32_t* vals, const int32_t* pair_of, uint32_t* keys,
                             cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  k_pair_keys<<<grid_for(n, 256, 8), 256, 0, s>>>(n, vals, pair_of, keys);
  return cudaGetLastError();
}

// Per-mesh-pair totals of the batched path (mesh pair p owns the CSR rows
// elem_off_a[p] .. elem_off_a[p+1]-1).  Mesh pairs differ in size by
// 100x, so each pair's candidate range is split into kMeshSplit contiguous
// pieces reduced by separate blocks (grid nm x kMeshSplit), and the pieces
// are merged in piece order by k_mesh_combine: deterministic, and no block
// walks a whole large mesh alone.
constexpr int kMeshSplit = 32;

__global__ void __launch_bounds__(256) k_mesh_totals(int nm, const int64_t* __restrict__ elem_off_a,
                                                     const int64_t* __restrict__ offsets,
                                                     const double* __restrict__ pm, const int32_t* __restrict__ pn,
                                                     Partial* pieces, int64_t cap) {
  const int p = blockIdx.x, g = blockIdx.y;
  if (p >= nm) return;
  // cap: entries the pair arrays hold (a count beyond it is reported by the
  // host, which then runs the batch again with larger arrays)
  const int64_t beg = min(offsets[elem_off_a[p]], cap), end = min(offsets[elem_off_a[p + 1]], cap);
  const int64_t len = end - beg;
  const int64_t b0 = beg + len * g / kMeshSplit, b1 = beg + len * (g + 1) / kMeshSplit;
  double sum = 0.0, err = 0.0;
  unsigned long long ni = 0, no = 0;
  for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
    cs_add(sum, err, pm[i]);
    const int k = pn[i];
    ni += k > 0;
    no += k;
  }
  block_reduce_partial<256>(sum, err, ni, no, &pieces[(int64_t)p * kMeshSplit + g]);
}

__global__ void k_mesh_combine(int nm, const int64_t* __restrict__ elem_off_a, const int64_t* __restrict__ offsets,
                               const Partial* __restrict__ pieces, Partial* out, int64_t* ncand) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nm) return;
  Partial q = pieces[(int64_t)p * kMeshSplit];
  for (int g = 1; g < kMeshSplit; ++g) {
    const Partial r = pieces[(int64_t)p * kMeshSplit + g];
    two_sum_merge(q.sum, q.err, r.sum, r.err);
    q.n_int += r.n_int;
    q.n_out += r.n_out;
  }
  q.sum = q.sum + q.err;
  out[p] = q;
  ncand[p] = offsets[elem_off_a[p + 1]] - offsets[elem_off_a[p]];
}

int64_t mesh_totals_pieces(int nm) { return (int64_t)nm * kMeshSplit; }

// Per-pair CSR of a batch group in the get_output layout of the C API
// (C_bindings.F90:377-391): mesh pair k owns rows eoa[k] .. eoa[k+1]-1 and
// writes out[rowbase[k] + r] = offsets[eoa[k] + r] - offsets[eoa[k]] for
// r = 0 .. nel_a(k) (the last entry is the pair's candidate count).
__global__ void k_batch_indptr(int64_t na, int nm, const int32_t* __restrict__ pair_of_a,
                               const int64_t* __restrict__ eoa, const int64_t* __restrict__ offsets,
                               const int64_t* __restrict__ rowbase, int64_t* out) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < na + nm; e += (int64_t)gridDim.x * blockDim.x) {
    if (e < na) {
      const int k = pair_of_a[e];
      out[rowbase[k] + (e - eoa[k])] = offsets[e] - offsets[eoa[k]];
    } else {
      const int k = (int)(e - na);
      out[rowbase[k] + (eoa[k + 1] - eoa[k])] = offsets[eoa[k + 1]] - offsets[eoa[k]];
    }
  }
}

// Candidate B elements as numbers local to their mesh pair, int64.
__global__ void k_batch_indices(int64_t n, const int32_t* __restrict__ pair_b, const int32_t* __restrict__ pair_of_b,
                                const int64_t* __restrict__ eob, int64_t* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t b = pair_b[i];
    out[i] = (int64_t)b - eob[pair_of_b[b]];
  }
}

cudaError_t launch_batch_csr(int64_t na, int nm, const int32_t* pair_of_a, const int64_t* eoa, const int64_t* offsets,
                             const int64_t* rowbase, int64_t* ind_ptr, int64_t ncand, const int32_t* pair_b,
                             const int32_t* pair_of_b, const int64_t* eob, int64_t* indices, cudaStream_t s) {
  if (ind_ptr && na + nm > 0) {
    count_launch();
    k_batch_indptr<<<grid_for(na + nm, 256, 8), 256, 0, s>>>(na, nm, pair_of_a, eoa, offsets, rowbase, ind_ptr);
  }
  if (indices && ncand > 0) {
    count_launch();
    k_batch_indices<<<grid_for(ncand, 256, 8), 256, 0, s>>>(ncand, pair_b, pair_of_b, eob, indices);
  }
  return cudaGetLastError();
}

cudaError_t launch_mesh_totals(int nm, const int64_t* elem_off_a, const int64_t* offsets, const double* pm,
                               const int32_t* pn, Partial* pieces, Partial* out, int64_t* ncand, cudaStream_t s,
                               int64_t cap) {
  if (nm <= 0) return cudaSuccess;
  count_launch(2);
  k_mesh_totals<<<dim3(nm, kMeshSplit), 256, 0, s>>>(nm, elem_off_a, offsets, pm, pn, pieces, cap);
  k_mesh_combine<<<(nm + 127) / 128, 128, 0, s>>>(nm, elem_off_a, offsets, pieces, out, ncand);
  return cudaGetLastError();
}

// ======================================================================
// Explicit element pairs (the single-pair C API and its batched form)
// ======================================================================
struct TriEmit {
  double* out;  // [22][3][2] for this pair, or nullptr
  __device__ __forceinline__ void operator()(int k, double x0, double y0, double x1, double y1, double x2,
                                             double y2) const {
    if (!out || k >= 22) return;
    double* o = out + 6 * k;
    o[0] = x0;
    o[1] = y0;
    o[2] = x1;
    o[3] = y1;
    o[4] = x2;
    o[5] = y2;
  }
};

__global__ void k_pairs_tris(int64_t n, const double* __restrict__ A, const double* __restrict__ B,
                             double* measure, int32_t* nout, double* out_elems) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* va = A + 6 * i;
    const double* vb = B + 6 * i;
    Lines L;
    tri_lines(vb, L);
    const double tol = 10.0 * fmin(spacing(tri_area(va[0], va[1], va[2], va[3], va[4], va[5])),
                                   spacing(tri_area(vb[0], vb[1], vb[2], vb[3], vb[4], vb[5])));
    LocalPoly<kTriWideCap> p, q;
    double m;
    int k = clip_tri(va[0], va[1], va[2], va[3], va[4], va[5], L, tol, p, q, kTriWideCap, m,
                     TriEmit{out_elems ? out_elems + 22 * 6 * i : nullptr});
    if (k < 0) {
      k = 0;
      m = 0.0;
    }
    if (measure) measure[i] = m;
    if (nout) nout[i] = k;
  }
}

__global__ void k_pairs_tets(int64_t n, const double* __restrict__ A, const double* __restrict__ B,
                             double* measure, int32_t* nout, double* out_elems) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    Tet ta, tb;
    load_tet(A + 12 * i, ta);
    load_tet(B + 12 * i, tb);
    Planes P;
    tet_planes(tb, P);
    const double tol = 10.0 * fmin(spacing(tet_volume_v4(ta)), spacing(tet_volume_v4(tb)));
    TetStackLocal stk;
    double m = 0.0;
    int idx = 0;
    double* o = out_elems ? out_elems + (int64_t)81 * 12 * i : nullptr;
    const int k = clip_tet_dfs(ta, RegPlanes{P}, tol, stk, [&](const Tet& t) {
      m = m + tet_volume_v1(t);
      if (o && idx < 81) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          o[12 * idx + 3 * v + 0] = t.x[v];
          o[12 * idx + 3 * v + 1] = t.y[v];
          o[12 * idx + 3 * v + 2] = t.z[v];
        }
      }
      ++idx;
    });
    if (measure) measure[i] = m;
    if (nout) nout[i] = k;
  }
}

// Triangle vs quadrilateral (Supermesh.F90:211-228): clip by the quad's 4
// edge lines, tolerance from the triangle's area only.
struct TriQuadEmit {
  double* out;  // [46][3][2] for this pair, or nullptr
  __device__ __forceinline__ void operator()(int k, double x0, double y0, double x1, double y1, double x2,
                                             double y2) const {
    if (!out || k >= 46) return;
    double* o = out + 6 * k;
    o[0] = x0;
    o[1] = y0;
    o[2] = x1;
    o[3] = y1;
    o[4] = x2;
    o[5] = y2;
  }
};

__global__ void k_pairs_tri_quad(int64_t n, const double* __restrict__ A, const double* __restrict__ B,
                                 double* measure, int32_t* nout, double* out_elems) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* va = A + 6 * i;
    double nx[4], ny[4], px[4], py[4];
    poly_lines<4>(B + 8 * i, nx, ny, px, py);
    const double tol = 10.0 * spacing(tri_area(va[0], va[1], va[2], va[3], va[4], va[5]));
    LocalPoly<48> p, q;
    p.set(0, va[0], va[1]);
    p.set(1, va[2], va[3]);
    p.set(2, va[4], va[5]);
    int m = 3;
    bool empty = false;
    for (int l = 0; l < 4 && !empty; ++l) {
      m = (l & 1) ? clip_stage(q, p, m, 48, nx[l], ny[l], px[l], py[l])
                  : clip_stage(p, q, m, 48, nx[l], ny[l], px[l], py[l]);
      empty = m < 3;
    }
    double meas = 0.0;
    int kept = 0;
    if (!empty) {  // after 4 stages the polygon is back in p
      TriQuadEmit emit{out_elems ? out_elems + 46 * 6 * i : nullptr};
      const double x0 = p.x(0), y0 = p.y(0);
      for (int j = 1; j < m - 1; ++j) {
        const double xi = p.x(j), yi = p.y(j), xj = p.x(j + 1), yj = p.y(j + 1);
        const double ar = tri_area(x0, y0, xi, yi, xj, yj);
        if (!(ar < tol)) {
          meas = meas + ar;
          emit(kept, x0, y0, xi, yi, xj, yj);
          ++kept;
        }
      }
    }
    if (measure) measure[i] = meas;
    if (nout) nout[i] = kept;
  }
}

// Tetrahedron vs hexahedron (Supermesh.F90:248-295): clip by the hex's 6
// face planes, tolerance from the tet's volume only.
__global__ void __launch_bounds__(64) k_pairs_tet_hex(int64_t n, const double* __restrict__ A,
                                                      const double* __restrict__ B, double* measure,
                                                      int32_t* nout, double* out_elems) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    Tet ta;
    load_tet(A + 12 * i, ta);
    ArrPlanes<6> P;
    hex_planes(B + 24 * i, P.nx, P.ny, P.nz, P.c);
    const double tol = 10.0 * spacing(tet_volume_v4(ta));
    TetStackN<10> stk;
    double m = 0.0;
    int idx = 0;
    double* o = out_elems ? out_elems + (int64_t)729 * 12 * i : nullptr;
    const int k = clip_tet_dfs<6>(ta, P, tol, stk, [&](const Tet& t) {
      m = m + tet_volume_v1(t);
      if (o && idx < 729) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          o[12 * idx + 3 * v + 0] = t.x[v];
          o[12 * idx + 3 * v + 1] = t.y[v];
          o[12 * idx + 3 * v + 2] = t.z[v];
        }
      }
      ++idx;
    });
    if (measure) measure[i] = m;
    if (nout) nout[i] = k;
  }
}

// Quadrilateral vs quadrilateral (Supermesh.F90:230-246): clip quad A by
// quad B's 4 edge lines; no element area is given, so the fan keeps
// triangles with area >= 10*tiny (Triangle_Intersection.F90:255-264).
__global__ void k_pairs_quad_quad(int64_t n, const double* __restrict__ A, const double* __restrict__ B,
                                  double* measure, int32_t* nout, double* out_elems) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* va = A + 8 * i;
    double nx[4], ny[4], px[4], py[4];
    poly_lines<4>(B + 8 * i, nx, ny, px, py);
    LocalPoly<16> p, q;
#pragma unroll
    for (int v = 0; v < 4; ++v) p.set(v, va[2 * v], va[2 * v + 1]);
    int m = 4;
    bool empty = false;
    for (int l = 0; l < 4 && !empty; ++l) {
      m = (l & 1) ? clip_stage(q, p, m, 16, nx[l], ny[l], px[l], py[l])
                  : clip_stage(p, q, m, 16, nx[l], ny[l], px[l], py[l]);
      empty = m < 3;
    }
    double meas = 0.0;
    int kept = 0;
    if (!empty) {
      const double tol = 10.0 * DBL_MIN;
      double* o = out_elems ? out_elems + 62 * 6 * i : nullptr;
      const double x0 = p.x(0), y0 = p.y(0);
      for (int j = 1; j < m - 1; ++j) {
        const double xi = p.x(j), yi = p.y(j), xj = p.x(j + 1), yj = p.y(j + 1);
        const double ar = tri_area(x0, y0, xi, yi, xj, yj);
        if (!(ar < tol)) {
          meas = meas + ar;
          if (o && kept < 62) {
            double* t = o + 6 * kept;
            t[0] = x0;
            t[1] = y0;
            t[2] = xi;
            t[3] = yi;
            t[4] = xj;
            t[5] = yj;
          }
          ++kept;
        }
      }
    }
    if (measure) measure[i] = meas;
    if (nout) nout[i] = kept;
  }
}

// Hexahedron vs hexahedron (Supermesh.F90:303-334): hex A sliced into five
// tets (Gmsh corners 3,6,7,8 / 1,3,4,8 / 1,5,6,8 / 1,2,3,6 / 1,3,6,8), each
// clipped by hex B as in intersect_tet_hex; outputs concatenated.
__global__ void __launch_bounds__(64) k_pairs_hex_hex(int64_t n, const double* __restrict__ A,
                                                      const double* __restrict__ B, double* measure,
                                                      int32_t* nout, double* out_elems) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* h = A + 24 * i;
    ArrPlanes<6> P;
    hex_planes(B + 24 * i, P.nx, P.ny, P.nz, P.c);
    double m = 0.0;
    int total = 0;
    double* o = out_elems ? out_elems + (int64_t)5 * 729 * 12 * i : nullptr;
    for (int s = 0; s < 5; ++s) {
      Tet ta;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        ta.x[v] = h[3 * kHexTets[s][v]];
        ta.y[v] = h[3 * kHexTets[s][v] + 1];
        ta.z[v] = h[3 * kHexTets[s][v] + 2];
      }
      const double tol = 10.0 * spacing(tet_volume_v4(ta));
      TetStackN<10> stk;
      const int k = clip_tet_dfs<6>(ta, P, tol, stk, [&](const Tet& t) {
        m = m + tet_volume_v1(t);
        if (o && total < 5 * 729) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            o[12 * total + 3 * v + 0] = t.x[v];
            o[12 * total + 3 * v + 1] = t.y[v];
            o[12 * total + 3 * v + 2] = t.z[v];
          }
        }
        ++total;
      });
      (void)k;
    }
    if (measure) measure[i] = m;
    if (nout) nout[i] = total;
  }
}

__global__ void k_pairs_intervals(int64_t n, const double* __restrict__ A, const double* __restrict__ B,
                                  double* measure, int32_t* nout, double* out_elems) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double c0 = 0.0, c1 = 0.0;
    const int k = intersect_intervals(A[2 * i], A[2 * i + 1], B[2 * i], B[2 * i + 1], c0, c1);
    if (out_elems && k) {
      out_elems[2 * i] = c0;
      out_elems[2 * i + 1] = c1;
    }
    if (measure) measure[i] = k ? interval_size(c0, c1) : 0.0;
    if (nout) nout[i] = k;
  }
}

cudaError_t launch_pairs_mixed(int kind, int64_t n, const double* a, const double* b, double* measure,
                               int32_t* nout, double* out_elems, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  if (kind == 0)
    k_pairs_intervals<<<grid_for(n, 256, 8), 256, 0, s>>>(n, a, b, measure, nout, out_elems);
  else if (kind == 1)
    k_pairs_tri_quad<<<grid_for(n, 128, 8), 128, 0, s>>>(n, a, b, measure, nout, out_elems);
  else if (kind == 2)
    k_pairs_tet_hex<<<grid_for(n, 64, 8), 64, 0, s>>>(n, a, b, measure, nout, out_elems);
  else if (kind == 3)
    k_pairs_quad_quad<<<grid_for(n, 128, 8), 128, 0, s>>>(n, a, b, measure, nout, out_elems);
  else
    k_pairs_hex_hex<<<grid_for(n, 64, 8), 64, 0, s>>>(n, a, b, measure, nout, out_elems);
  return cudaGetLastError();
}

// ======================================================================
// 1D sort finder (Intersection_Finder.F90:811-921): elements sorted by left
// end, then one sweep pointer over the sorted B elements.  Restated as
//   E_i  = first sorted B element whose left end >= right end of sorted A_i
//   L_i  = last sorted B element before E_i whose right end > left end of A_i
//   row_i records {j in [js_i, E_i) : right_B(j) > left_A(i)}
//   js_{i+1} = y_i - [js_i <= L_i],  y_i = max(js_i, E_i) advanced past B
//              points equal to a point A_i
// E_i and L_i (binary search, max segment tree) and the rows are computed in
// parallel; only the integer recurrence for js runs on one warp.
// ======================================================================
__device__ __forceinline__ uint64_t ordered_key(double x) {
  if (x == 0.0) x = 0.0;  // -0 and +0 compare equal: give them one key
  const uint64_t u = (uint64_t)__double_as_longlong(x);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

__global__ void k_prep_1d(int64_t nel, const double* __restrict__ pos, int stride, const void* __restrict__ en,
                          int idx_bytes, int64_t nnodes, double* coords, uint32_t* key_lo, uint32_t* key_hi,
                          int32_t* vals, int* bad) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nel; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t n0, n1;
    if (idx_bytes == 8) {
      n0 = static_cast<const int64_t*>(en)[2 * e];
      n1 = static_cast<const int64_t*>(en)[2 * e + 1];
    } else {
      n0 = static_cast<const int32_t*>(en)[2 * e];
      n1 = static_cast<const int32_t*>(en)[2 * e + 1];
    }
    if (n0 < 0 || n0 >= nnodes || n1 < 0 || n1 >= nnodes) {
      atomicExch(bad, 1);
      n0 = n1 = 0;
    }
    const double x0 = pos[n0 * stride], x1 = pos[n1 * stride];
    coords[2 * e] = x0;
    coords[2 * e + 1] = x1;
    const uint64_t k = ordered_key(x1 < x0 ? x1 : x0);
    key_lo[e] = (uint32_t)k;
    key_hi[e] = (uint32_t)(k >> 32);
    vals[e] = (int32_t)e;
  }
}

__global__ void k_permute_u32(int64_t n, const int32_t* __restrict__ perm, const uint32_t* __restrict__ in,
                              uint32_t* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[perm[i]];
}

__global__ void k_sorted_ends_1d(int64_t n, const int32_t* __restrict__ perm, const double* __restrict__ coords,
                                 double* lo, double* hi) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t e = perm[i];
    const double x0 = coords[2 * e], x1 = coords[2 * e + 1];
    lo[i] = x1 < x0 ? x1 : x0;
    hi[i] = x1 > x0 ? x1 : x0;
  }
}

__global__ void k_tree_leaves(int64_t n, int64_t P, const double* __restrict__ v, double* tree) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P; i += (int64_t)gridDim.x * blockDim.x)
    tree[P + i] = i < n ? v[i] : -INFINITY;
}

__global__ void k_tree_level(int64_t w, double* tree) {
  for (int64_t k = w + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < 2 * w; k += (int64_t)gridDim.x * blockDim.x)
    tree[k] = fmax(tree[2 * k], tree[2 * k + 1]);
}

// Last leaf index < E whose value is > t, or -1 (tree over P leaves).
__device__ __forceinline__ int rightmost_greater(const double* __restrict__ tree, int64_t P, int64_t E, double t) {
  if (E <= 0) return -1;
  int64_t node = P + E - 1;
  for (int guard = 0; guard < 256; ++guard) {
    if (tree[node] > t) {
      while (node < P) node = tree[2 * node + 1] > t ? 2 * node + 1 : 2 * node;
      return (int)(node - P);
    }
    // move to the subtree just left of `node`
    while ((node & (node - 1)) != 0 && (node & 1) == 0) node >>= 1;
    if ((node & (node - 1)) == 0) return -1;  // leftmost at its level
    node -= 1;
  }
  return -1;
}

__global__ void k_rows_1d(int64_t na, const double* __restrict__ lo_a, const double* __restrict__ hi_a, int64_t nb,
                          const double* __restrict__ lo_b, const double* __restrict__ tree, int64_t P, int32_t* E,
                          int32_t* L) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < na; i += (int64_t)gridDim.x * blockDim.x) {
    const double h = hi_a[i];
    int64_t lo = 0, hi = nb;  // first j with lo_b[j] >= h
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (lo_b[mid] < h)
        lo = mid + 1;
      else
        hi = mid;
    }
    E[i] = (int32_t)lo;
    L[i] = nb > 0 ? rightmost_greater(tree, P, lo, lo_a[i]) : -1;
  }
}

__global__ void __launch_bounds__(32) k_sweep_1d(int64_t na, int64_t nb, const int32_t* __restrict__ E,
                                                 const int32_t* __restrict__ L, const double* __restrict__ lo_a,
                                                 const double* __restrict__ hi_a, const double* __restrict__ hi_b,
                                                 int32_t* JS) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x;
  int64_t js = 0;
  for (int64_t base = 0; base < na; base += 32) {
    const int64_t i = base + lane;
    int e = 0, l = -1;
    double lo = 0.0, hi = 1.0;
    if (i < na) {
      e = E[i];
      l = L[i];
      lo = lo_a[i];
      hi = hi_a[i];
    }
    const unsigned point = __ballot_sync(full, i < na && !(lo < hi));
    const int cnt = (int)(na - base < 32 ? na - base : 32);
    int64_t mine = 0;
    for (int k = 0; k < cnt; ++k) {
      const int ek = __shfl_sync(full, e, k);
      const int lk = __shfl_sync(full, l, k);
      if (lane == k) mine = js;
      int64_t y = js > ek ? js : ek;
      if ((point >> k) & 1u) {
        const double t = __shfl_sync(full, lo, k);
        while (y < nb && hi_b[y] <= t) ++y;
      }
      js = js <= lk ? y - 1 : y;
    }
    if (i < na) JS[i] = (int32_t)mine;
  }
}

template <bool FILL>
__global__ void k_emit_1d(int64_t na, const int32_t* __restrict__ JS, const int32_t* __restrict__ E,
                          const double* __restrict__ lo_a, const double* __restrict__ hi_b,
                          const int32_t* __restrict__ perm_a, const int32_t* __restrict__ perm_b, int* counts,
                          const int64_t* __restrict__ offsets, int32_t* pair_a, int32_t* pair_b) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < na; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t a = perm_a[i];
    const double t = lo_a[i];
    const int32_t end = E[i];
    int64_t out = FILL ? offsets[a] : 0;
    int cnt = 0;
    for (int32_t j = JS[i]; j < end; ++j) {
      if (hi_b[j] > t) {
        if (FILL) {
          pair_a[out + cnt] = a;
          pair_b[out + cnt] = perm_b[j];
        }
        ++cnt;
      }
    }
    if (!FILL) counts[a] = cnt;
  }
}

cudaError_t launch_prep_1d(int64_t nel, const double* pos, int stride, const void* en, int idx_bytes,
                           int64_t nnodes, double* coords, uint32_t* key_lo, uint32_t* key_hi, int32_t* vals,
                           int* bad, cudaStream_t s) {
  if (nel <= 0) return cudaSuccess;
  count_launch();
  k_prep_1d<<<grid_for(nel, 256, 8), 256, 0, s>>>(nel, pos, stride, en, idx_bytes, nnodes, coords, key_lo, key_hi,
                                                  vals, bad);
  return cudaGetLastError();
}

cudaError_t sort_by_key64(int64_t n, uint32_t* key_lo, const uint32_t* key_hi, int32_t* vals, uint32_t* keys_tmp,
                          int32_t* vals_tmp, uint32_t* hist, cudaStream_t s) {
  if (n <= 1) return cudaSuccess;
  cudaError_t e = radix_sort_pairs(n, 32, key_lo, vals, keys_tmp, vals_tmp, hist, s);
  if (e != cudaSuccess) return e;
  count_launch();
  k_permute_u32<<<grid_for(n, 256, 8), 256, 0, s>>>(n, vals, key_hi, key_lo);
  return radix_sort_pairs(n, 32, key_lo, vals, keys_tmp, vals_tmp, hist, s);
}

cudaError_t launch_sorted_ends_1d(int64_t n, const int32_t* perm, const double* coords, double* lo, double* hi,
                                  cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  k_sorted_ends_1d<<<grid_for(n, 256, 8), 256, 0, s>>>(n, perm, coords, lo, hi);
  return cudaGetLastError();
}

int64_t tree_leaves_1d(int64_t n) {
  int64_t P = 1;
  while (P < n) P <<= 1;
  return P;
}

cudaError_t launch_max_tree(int64_t n, const double* v, double* tree, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int64_t P = tree_leaves_1d(n);
  count_launch();
  k_tree_leaves<<<grid_for(P, 256, 8), 256, 0, s>>>(n, P, v, tree);
  for (int64_t w = P / 2; w >= 1; w /= 2) {
    count_launch();
    k_tree_level<<<grid_for(w, 256, 8), 256, 0, s>>>(w, tree);
  }
  return cudaGetLastError();
}

cudaError_t launch_rows_1d(int64_t na, const double* lo_a, const double* hi_a, int64_t nb, const double* lo_b,
                           const double* tree, int32_t* E, int32_t* L, cudaStream_t s) {
  if (na <= 0) return cudaSuccess;
  count_launch();
  k_rows_1d<<<grid_for(na, 256, 8), 256, 0, s>>>(na, lo_a, hi_a, nb, lo_b, tree, tree_leaves_1d(nb), E, L);
  return cudaGetLastError();
}

cudaError_t launch_sweep_1d(int64_t na, int64_t nb, const int32_t* E, const int32_t* L, const double* lo_a,
                            const double* hi_a, const double* hi_b, int32_t* JS, cudaStream_t s) {
  if (na <= 0) return cudaSuccess;
  count_launch();
  k_sweep_1d<<<1, 32, 0, s>>>(na, nb, E, L, lo_a, hi_a, hi_b, JS);
  return cudaGetLastError();
}

cudaError_t launch_emit_1d(bool fill, int64_t na, const int32_t* JS, const int32_t* E, const double* lo_a,
                           const double* hi_b, const int32_t* perm_a, const int32_t* perm_b, int* counts,
                           const int64_t* offsets, int32_t* pair_a, int32_t* pair_b, cudaStream_t s) {
  if (na <= 0) return cudaSuccess;
  count_launch();
  if (fill)
    k_emit_1d<true><<<grid_for(na, 256, 8), 256, 0, s>>>(na, JS, E, lo_a, hi_b, perm_a, perm_b, counts, offsets,
                                                         pair_a, pair_b);
  else
    k_emit_1d<false><<<grid_for(na, 256, 8), 256, 0, s>>>(na, JS, E, lo_a, hi_b, perm_a, perm_b, counts, offsets,
                                                          pair_a, pair_b);
  return cudaGetLastError();
}

// Narrow phase of 1D candidates: intersect_intervals per pair.
__global__ void k_clip_intervals(int64_t n, const int32_t* __restrict__ pa, const int32_t* __restrict__ pb,
                                 const double* __restrict__ ca, const double* __restrict__ cb, double* measure,
                                 int32_t* nout) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t a = pa[i], b = pb[i];
    double c0 = 0.0, c1 = 0.0;
    const int k = intersect_intervals(ca[2 * a], ca[2 * a + 1], cb[2 * b], cb[2 * b + 1], c0, c1);
    measure[i] = k ? interval_size(c0, c1) : 0.0;
    nout[i] = k;
  }
}

cudaError_t launch_clip_intervals(int64_t n, const int32_t* pa, const int32_t* pb, const double* ca,
                                  const double* cb, double* measure, int32_t* nout, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  k_clip_intervals<<<grid_for(n, 256, 8), 256, 0, s>>>(n, pa, pb, ca, cb, measure, nout);
  return cudaGetLastError();
}

cudaError_t launch_pairs_explicit(int dim, int64_t n, const double* a, const double* b,
                                  double* measure, int32_t* nout, double* out_elems,
                                  cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int B = 128;
  const int g = grid_for(n, B, 8);
  count_launch();
  if (dim == 2)
    k_pairs_tris<<<g, B, 0, s>>>(n, a, b, measure, nout, out_elems);
  else
    k_pairs_tets<<<g, B, 0, s>>>(n, a, b, measure, nout, out_elems);
  return cudaGetLastError();
}

__global__ void k_measure_explicit(int dim, int64_t n, const double* __restrict__ e, double* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if (dim == 1) {
      out[i] = interval_size(e[2 * i], e[2 * i + 1]);
    } else if (dim == 2) {
      const double* v = e + 6 * i;
      out[i] = tri_area(v[0], v[1], v[2], v[3], v[4], v[5]);
    } else {
      Tet t;
      load_tet(e + 12 * i, t);
      out[i] = tet_volume_v1(t);
    }
  }
}

cudaError_t launch_measure_explicit(int dim, int64_t n, const double* elems, double* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  k_measure_explicit<<<grid_for(n, 256, 8), 256, 0, s>>>(dim, n, elems, out);
  return cudaGetLastError();
}

// ======================================================================
// K8: P1-P1 mixed mass matrix
// ======================================================================
// P1 basis on a triangle (test_parallel_p1_inner_product_2d.F90:206-229):
// the inverse Jacobian (divided by the determinant entry by entry) depends
// only on the element and is formed once per pair; each point then takes
// the same products and sums as the reference.
struct P1Fac2 {
  double ox, oy, j11, j12, j21, j22;
};

__device__ __forceinline__ P1Fac2 p1_factor_2d(const double* cc) {
  const double e1x = cc[2] - cc[0], e1y = cc[3] - cc[1];
  const double e2x = cc[4] - cc[0], e2y = cc[5] - cc[1];
  double j11 = e2y, j12 = -e2x, j21 = -e1y, j22 = e1x;
  const double det = j11 * j22 - j12 * j21;
  return P1Fac2{cc[0], cc[1], j11 / det, j12 / det, j21 / det, j22 / det};
}

__device__ __forceinline__ void p1_apply_2d(const P1Fac2& F, double x, double y, double f[3]) {
  const double dx = x - F.ox, dy = y - F.oy;
  f[1] = F.j11 * dx + F.j12 * dy;
  f[2] = F.j21 * dx + F.j22 * dy;
  f[0] = 1.0 - f[1] - f[2];
}

template <typename IDX>
__device__ __forceinline__ int64_t node_of(const void* en, int64_t e, int loc, int k) {
  return (int64_t)((const IDX*)en)[e * loc + k];
}

// P1 basis on a tetrahedron (test_parallel_p1_inner_product_3d.F90:215-250):
// the local coordinates of point x solve [v1-v0 | v2-v0 | v3-v0] l = x - v0
// by Gaussian elimination with partial pivoting on the augmented 3x4 matrix
// (pivot search, row swap, pivot row divided by the pivot, rows below
// reduced; then back substitution from the last row), f = (1 - l1 - l2 - l3,
// l1, l2, l3).  The pivot choices, pivots and multipliers depend only on the
// element's edge matrix, so p1_factor_3d runs that elimination on the three
// matrix columns once per element and stores, at stride S: the origin v0
// (3), the pivots (3), the forward multipliers of rows (1,0) (2,0) (2,1) and
// the back-substitution multipliers of rows (1,2) (0,2) (0,1); it returns the
// row swaps (row exchanged with row 0 in bits 0-1, with row 1 in bits 2-3).
// p1_apply_3d applies to the point's right-hand side exactly the operations
// the elimination applies to the augmented column, in the same order.
// Entries 12-14 hold the pivots' reciprocals, for div_by.
constexpr int kP1Fac3 = 15;

template <int S>
__device__ __forceinline__ int p1_factor_3d(const double* cc, double* F) {
  double m[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
#pragma unroll
    for (int c = 0; c < 3; ++c) m[r][c] = cc[3 * (c + 1) + r] - cc[r];
    F[r * S] = cc[r];
  }
  int sw = 0, nl = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    int j = i;
    double best = fabs(m[i][i]);
#pragma unroll
    for (int k = i + 1; k < 3; ++k)
      if (fabs(m[k][i]) > best) {
        best = fabs(m[k][i]);
        j = k;
      }
#pragma unroll
    for (int k = i + 1; k < 3; ++k) {
      if (j == k) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double t = m[i][c];
          m[i][c] = m[k][c];
          m[k][c] = t;
        }
      }
    }
    sw |= j << (2 * i);
    const double piv = m[i][i];
    F[(3 + i) * S] = piv;
    F[(12 + i) * S] = __drcp_rn(piv);
#pragma unroll
    for (int c = 0; c < 3; ++c) m[i][c] = m[i][c] / piv;
#pragma unroll
    for (int k = i + 1; k < 3; ++k) {
      const double fk = m[k][i];
      F[(6 + nl++) * S] = fk;
#pragma unroll
      for (int c = 0; c < 3; ++c) m[k][c] = m[k][c] - fk * m[i][c];
    }
  }
  int nu = 0;
#pragma unroll
  for (int i = 2; i >= 0; --i)
#pragma unroll
    for (int k = i - 1; k >= 0; --k) {
      const double fk = m[k][i];
      F[(9 + nu++) * S] = fk;
#pragma unroll
      for (int c = 0; c < 3; ++c) m[k][c] = m[k][c] - fk * m[i][c];
    }
  return sw;
}

// FAST: the three divisions through the stored reciprocals; range gathers
// their numerators.
template <int S, bool FAST>
__device__ __forceinline__ void p1_apply_3d(const double* F, int sw, double x, double y, double z, double f[4],
                                            unsigned& range) {
  double r0 = x - F[0], r1 = y - F[S], r2 = z - F[2 * S];
  const int j0 = sw & 3, j1 = (sw >> 2) & 3;
  {
    const double t0 = r0;
    r0 = j0 == 1 ? r1 : (j0 == 2 ? r2 : r0);
    r1 = j0 == 1 ? t0 : r1;
    r2 = j0 == 2 ? t0 : r2;
  }
  if (FAST) range = div_range(range, r0);
  r0 = FAST ? div_by(r0, F[3 * S], F[12 * S]) : r0 / F[3 * S];
  r1 = r1 - F[6 * S] * r0;
  r2 = r2 - F[7 * S] * r0;
  {
    const double t1 = r1;
    r1 = j1 == 2 ? r2 : r1;
    r2 = j1 == 2 ? t1 : r2;
  }
  if (FAST) range = div_range(range, r1);
  r1 = FAST ? div_by(r1, F[4 * S], F[13 * S]) : r1 / F[4 * S];
  r2 = r2 - F[8 * S] * r1;
  if (FAST) range = div_range(range, r2);
  r2 = FAST ? div_by(r2, F[5 * S], F[14 * S]) : r2 / F[5 * S];
  r1 = r1 - F[9 * S] * r2;
  r0 = r0 - F[10 * S] * r2;
  r0 = r0 - F[11 * S] * r1;
  f[1] = r0;
  f[2] = r1;
  f[3] = r2;
  f[0] = 1.0 - f[1] - f[2] - f[3];
}

// P1-P1 mixed mass block of a pair (test_parallel_p1_inner_product_3d.F90:
// four-point rule, P1 bases of A and B by elimination at each point), per
// kept output tet in the reference's order; at the end of the pair the block
// is stored and u^T M v written per pair (the caller sums them in pair order).
// The per-element part of both eliminations is done once per pair
// (p1_factor_3d).  Sixteen final tets at a time: two lanes evaluate a tet's
// bases, two points each, into shared memory; then sixteen lanes, one per
// entry of the block, add the products up, tet by tet (the other sixteen take
// the tets from the first pair boundary after the eighth on).
template <typename IDX>
struct BfP1Sink {
  static constexpr bool kSum = false, kStore = false, kP1 = true;
  static constexpr int kSlots = 16, kWarps = 8, kQuads = 64, kRoom = 12, kKeep = 4;
  static constexpr int kLane = 18;  // doubles per lane: w phi_A, then phi_B, of two points interleaved; pad
  static constexpr int kVol = 0, kFac = kVol + 8 * kBfFinals, kBlk = kFac + 8 * 2 * kP1Fac3 * kSlots,
                       kBuf = kBlk + 8 * 16 * kSlots, kMeta = kBuf + 8 * 32 * kLane,
                       kExtra = kMeta + 8 * kSlots;
  const double* coords_a;
  const double* coords_b;
  const void* en_a;
  const void* en_b;
  const double* u_a;
  const double* v_b;
  double* blocks;
  double* pair_uv;  // u^T M v per pair (when u_a and v_b are given), summed in pair order afterwards
  __device__ __forceinline__ void begin(char* mem, int slot, const int4& r) const {
    double* fa = reinterpret_cast<double*>(mem + kFac) + slot;
    double* fb = fa + kP1Fac3 * kSlots;
    double* blk = reinterpret_cast<double*>(mem + kBlk) + 16 * slot;
    const int swa = p1_factor_3d<kSlots>(coords_a + (int64_t)r.y * 12, fa);
    const int swb = p1_factor_3d<kSlots>(coords_b + (int64_t)r.z * 12, fb);
    unsigned range = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      range = div_range(range, fa[(3 + i) * kSlots]);
      range = div_range(range, fb[(3 + i) * kSlots]);
    }
    reinterpret_cast<uint2*>(mem + kMeta)[slot] = make_uint2((unsigned)((swa & 15) | swb << 4), range);
#pragma unroll
    for (int j = 0; j < 16; ++j) blk[j] = 0.0;
  }
  // Quadrature point qq of tet o, in the reference's order of operations.
  static __device__ __forceinline__ V3 point(const Tet& o, int qq) {
    const double qa = 5.8541019662496852e-1, qb = 1.3819660112501050e-1;
    V3 p{0.0, 0.0, 0.0};
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double wv = v == qq ? qa : qb;
      p.x = p.x + wv * o.x[v];
      p.y = p.y + wv * o.y[v];
      p.z = p.z + wv * o.z[v];
    }
    return p;
  }
  // One tet of one lane's pair (pairs with distances that are not finite).
  __device__ __forceinline__ void tet(char* mem, int slot, const Tet& o, double v1) const {
    const double* fac = reinterpret_cast<const double*>(mem + kFac) + slot;
    double* blk = reinterpret_cast<double*>(mem + kBlk) + 16 * slot;
    const unsigned sw = reinterpret_cast<const uint2*>(mem + kMeta)[slot].x;
    const double w = 0.25 * v1;
    unsigned range = 0;
#pragma unroll 1
    for (int qq = 0; qq < 4; ++qq) {
      const V3 p = point(o, qq);
      double fa[4], fb[4];
      p1_apply_3d<kSlots, false>(fac, sw & 15, p.x, p.y, p.z, fa, range);
      p1_apply_3d<kSlots, false>(fac + kP1Fac3 * kSlots, sw >> 4, p.x, p.y, p.z, fb, range);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) blk[r * 4 + c] += w * fa[r] * fb[c];
    }
  }
  template <class Pool>
  __device__ __forceinline__ void integrate(char* mem, const Pool& pool, const uint2* fin, const double* vol, int nf,
                                            int lane) const {
    const unsigned full = 0xffffffffu;
    double* buf = reinterpret_cast<double*>(mem + kBuf);
    double* blk = reinterpret_cast<double*>(mem + kBlk);
#pragma unroll 1
    for (int f0 = 0; f0 < nf; f0 += 16) {
      const int nt = nf - f0 < 16 ? nf - f0 : 16;
      const int t = lane >> 1;
      uint2 id = make_uint2(0, 0xffffffffu);
      double v1 = -1.0;
      if (t < nt) {
        id = fin[f0 + t];
        v1 = vol[f0 + t];
      }
      const unsigned slot = id.y >> 27;
      if (!(v1 < 0.0)) {
        Tet o;
        bf_tet(pool, id.x, id.y & 0x03030303u, o);
        const double* fac = reinterpret_cast<const double*>(mem + kFac) + slot;
        const uint2 meta = reinterpret_cast<const uint2*>(mem + kMeta)[slot];
        const double w = 0.25 * v1;
        double fa[2][4], fb[2][4];
        unsigned range = meta.y;
        // this lane's points 0 and 1, or 2 and 3: the vertices' weights
        const bool second = lane & 1;
        V3 p[2];
        {
          const double qa = 5.8541019662496852e-1, qb = 1.3819660112501050e-1;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            p[j] = V3{0.0, 0.0, 0.0};
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const double wv = (v & 1) == j && (v >> 1) == (int)second ? qa : qb;
              p[j].x = p[j].x + wv * o.x[v];
              p[j].y = p[j].y + wv * o.y[v];
              p[j].z = p[j].z + wv * o.z[v];
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          p1_apply_3d<kSlots, true>(fac, meta.x & 15, p[j].x, p[j].y, p[j].z, fa[j], range);
          p1_apply_3d<kSlots, true>(fac + kP1Fac3 * kSlots, meta.x >> 4, p[j].x, p[j].y, p[j].z, fb[j], range);
        }
        if (!div_ok(range)) {
#pragma unroll 1
          for (int j = 0; j < 2; ++j) {
            const V3 pj = point(o, 2 * (int)second + j);
            double ga[4], gb[4];
            p1_apply_3d<kSlots, false>(fac, meta.x & 15, pj.x, pj.y, pj.z, ga, range);
            p1_apply_3d<kSlots, false>(fac + kP1Fac3 * kSlots, meta.x >> 4, pj.x, pj.y, pj.z, gb, range);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (j == 0) {
                fa[0][i] = ga[i];
                fb[0][i] = gb[i];
              } else {
                fa[1][i] = ga[i];
                fb[1][i] = gb[i];
              }
            }
          }
        }
        double* out = buf + lane * kLane;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          st2(out + 2 * i, w * fa[0][i], w * fa[1][i]);
          st2(out + 8 + 2 * i, fb[0][i], fb[1][i]);
        }
      } else {  // (a sum is not changed by adding +0)
        double* out = buf + lane * kLane;
#pragma unroll
        for (int i = 0; i < 8; ++i) st2(out + 2 * i, 0.0, 0.0);
      }
      // pair boundaries among the sixteen tets
      const unsigned before = __shfl_up_sync(full, slot, 2);
      const unsigned heads = __ballot_sync(full, t < nt && (t == 0 || before != slot));
      __syncwarp();
      const int h = lane >> 4;
      const unsigned late = heads >> 16;  // boundaries from the eighth tet on
      const int mid = late ? 8 + ((__ffs(late) - 1) >> 1) : nt;
      int i = h ? mid : 0;
      const int ie = h ? nt : mid;
      const double* q = buf + 2 * i * kLane + 2 * ((lane >> 2) & 3);
      const int cb = 8 + 2 * ((lane & 3) - ((lane >> 2) & 3));
      while (i < ie) {  // one pair's tets (the first of the sixteen go on from the ones before)
        double* at = blk + 16 * (fin[f0 + i].y >> 27) + (lane & 15);
        const unsigned next = heads & ~((4u << (2 * i)) - 1u);
        const int end = next ? min(ie, (__ffs(next) - 1) >> 1) : ie;
        double acc = *at;
#pragma unroll 2
        for (; i < end; ++i) {
          const double2 a0 = *reinterpret_cast<const double2*>(q), b0 = *reinterpret_cast<const double2*>(q + cb);
          const double2 a1 = *reinterpret_cast<const double2*>(q + kLane);
          const double2 b1 = *reinterpret_cast<const double2*>(q + kLane + cb);
          acc = acc + a0.x * b0.x;
          acc = acc + a0.y * b0.y;
          acc = acc + a1.x * b1.x;
          acc = acc + a1.y * b1.y;
          q += 2 * kLane;
        }
        *at = acc;
      }
      __syncwarp();
    }
  }
  __device__ __forceinline__ void end(char* mem, int n, const int4& rec, int lane) const {
    const double* blk = reinterpret_cast<const double*>(mem + kBlk);
    __syncwarp();
    if (blocks) {
      for (int s = lane >> 4; s < ((n + 1) & ~1); s += 2) {
        const int64_t p = __shfl_sync(0xffffffffu, rec.x, s);
        if (s < n) blocks[p * 16 + (lane & 15)] = blk[16 * s + (lane & 15)];
      }
    }
    if (u_a && v_b && lane < n) {
      blk += 16 * lane;
      double sv = 0.0;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const double ur = u_a[node_of<IDX>(en_a, rec.y, 4, r)];
#pragma unroll
        for (int c = 0; c < 4; ++c) sv += ur * blk[r * 4 + c] * v_b[node_of<IDX>(en_b, rec.z, 4, c)];
      }
      pair_uv[rec.x] = sv;
    }
  }
};

// 2D: one pair per thread, clipped with the triangle clipper; per supermesh
// triangle the degree-2 rule (three points), P1 bases of A and B, 3x3 block.
template <typename IDX>
__global__ void __launch_bounds__(128, 4) k_p1_mass(int64_t npairs, const int32_t* __restrict__ pa,
                                                 const int32_t* __restrict__ pb,
                                                 const double* __restrict__ coords_a,
                                                 const double* __restrict__ tol_a,
                                                 const double* __restrict__ coords_b,
                                                 const double* __restrict__ setup_b, const void* en_a,
                                                 const void* en_b, const double* __restrict__ u_a,
                                                 const double* __restrict__ v_b, double* blocks,
                                                 Partial* partials) {
  __shared__ double2 poly[kTriCap * 128];
  double sum = 0.0, err = 0.0;
  unsigned long long ni = 0;
  // each iteration loads the next one's pair indices (which stream from
  // DRAM) before it works on its own pair
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int na = 0, nb = 0;
  {
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 < npairs) {
      na = pa[i0];
      nb = pb[i0];
    }
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < npairs; i += stride) {
    const int a = na, b = nb;
    if (i + stride < npairs) {
      na = pa[i + stride];
      nb = pb[i + stride];
    }
    const double* ca = coords_a + (int64_t)a * 6;
    double blk[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) blk[j] = 0.0;
    Lines L;
    double tolb;
    load_lines(setup_b + (int64_t)b * kSetup2, L, tolb);
    const double tol = fmin(tol_a[a], tolb);
    const P1Fac2 fa_ = p1_factor_2d(ca), fb_ = p1_factor_2d(coords_b + (int64_t)b * 6);
    const double2 v[3] = {{ca[0], ca[1]}, {ca[2], ca[3]}, {ca[4], ca[5]}};
    const double qp0 = 4.0 / 6.0, qp1 = 1.0 / 6.0;
    clip_tri_fan<128>(v, L, tol, poly + threadIdx.x, true,
             [&](int, double x0, double y0, double x1, double y1, double x2, double y2) {
               const double meas = tri_area(x0, y0, x1, y1, x2, y2);
               const double w = (1.0 / 3.0) * meas;
#pragma unroll
               for (int qq = 0; qq < 3; ++qq) {
                 const double w0 = qq == 0 ? qp0 : qp1;
                 const double w1 = qq == 1 ? qp0 : qp1;
                 const double w2 = qq == 2 ? qp0 : qp1;
                 const double x = (w0 * x0 + w1 * x1) + w2 * x2;
                 const double y = (w0 * y0 + w1 * y1) + w2 * y2;
                 double fa[3], fb[3];
                 p1_apply_2d(fa_, x, y, fa);
                 p1_apply_2d(fb_, x, y, fb);
#pragma unroll
                 for (int r = 0; r < 3; ++r)
#pragma unroll
                   for (int c = 0; c < 3; ++c) blk[r * 3 + c] += w * fa[r] * fb[c];
               }
             });
    if (blocks) {
#pragma unroll
      for (int j = 0; j < 9; ++j) blocks[i * 9 + j] = blk[j];
    }
    if (u_a && v_b) {
      double sv = 0.0;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const double ur = u_a[node_of<IDX>(en_a, a, 3, r)];
#pragma unroll
        for (int c = 0; c < 3; ++c) sv += ur * blk[r * 3 + c] * v_b[node_of<IDX>(en_b, b, 3, c)];
      }
      cs_add(sum, err, sv);
    }
    ++ni;
  }
  block_reduce_partial<128>(sum, err, ni, 0ull, &partials[blockIdx.x]);
}

// 2D, u^T M v alone: the same sum by triangles, w (u_h v_h) at each point, with
// full warps.  A pair of candidates has one supermesh triangle on average, 41 %
// have none and some four, so a lane that integrates its own pair's triangles
// waits three quarters of the time; here a warp clips 32 pairs (clip_tri_c),
// queues their triangles and takes 32 at a time from the queue's end.  9.5 M
// candidate pairs: 1206 us by k_p1_mass with the walking clip, 617 here
// (threads and registers, without a profiler: 160 at 96 610 us, 192 at 80 638,
// 128 at 120 640), bound by
// L1 and shared wavefronts (72 %) and instructions.  Error of the integral
// against 80-bit arithmetic as before or smaller (at most 2e-16 of the sum of
// the terms' sizes).
constexpr int kUvThreads = 160;
constexpr int kUvQueue = 64;  // fewer than 32 left over, 32 more
template <typename IDX>
__device__ __forceinline__ double p1_uv_2d(const double2 (&t)[3], double w, int a, int b,
                                           const double* __restrict__ coords_a, const double* __restrict__ coords_b,
                                           const void* en_a, const void* en_b, const double* __restrict__ u_a,
                                           const double* __restrict__ v_b) {
  double ca[6], cb[6], u[3], v[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    u[k] = u_a[node_of<IDX>(en_a, a, 3, k)];
    v[k] = v_b[node_of<IDX>(en_b, b, 3, k)];
    const double2 x = __ldg(reinterpret_cast<const double2*>(coords_a + (int64_t)a * 6) + k);
    const double2 y = __ldg(reinterpret_cast<const double2*>(coords_b + (int64_t)b * 6) + k);
    ca[2 * k] = x.x;
    ca[2 * k + 1] = x.y;
    cb[2 * k] = y.x;
    cb[2 * k + 1] = y.y;
  }
  const P1Fac2 fa = p1_factor_2d(ca), fb = p1_factor_2d(cb);
  const double qp0 = 4.0 / 6.0, qp1 = 1.0 / 6.0;
  double sv = 0.0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double w0 = q == 0 ? qp0 : qp1, w1 = q == 1 ? qp0 : qp1, w2 = q == 2 ? qp0 : qp1;
    const double x = (w0 * t[0].x + w1 * t[1].x) + w2 * t[2].x;
    const double y = (w0 * t[0].y + w1 * t[1].y) + w2 * t[2].y;
    double ga[3], gb[3];
    p1_apply_2d(fa, x, y, ga);
    p1_apply_2d(fb, x, y, gb);
    sv += w * ((u[0] * ga[0] + u[1] * ga[1]) + u[2] * ga[2]) * ((v[0] * gb[0] + v[1] * gb[1]) + v[2] * gb[2]);
  }
  return sv;
}

template <typename IDX>
__global__ void __launch_bounds__(kUvThreads, 4)
    k_p1_uv(int64_t npairs, const int32_t* __restrict__ pa, const int32_t* __restrict__ pb,
            const double* __restrict__ coords_a, const double* __restrict__ tol_a,
            const double* __restrict__ coords_b, const double* __restrict__ setup_b, const void* en_a,
            const void* en_b, const double* __restrict__ u_a, const double* __restrict__ v_b, Partial* partials) {
  __shared__ double2 poly[kTriCap * kUvThreads];
  __shared__ double2 queue[kUvThreads / 32][4][kUvQueue];  // the vertices; the weight and the pair
  double2* p = poly + threadIdx.x;
  const int lane = threadIdx.x & 31;
  auto& qu = queue[threadIdx.x >> 5];
  int qn = 0;  // the warp's
  double sum = 0.0, err = 0.0;
  unsigned long long ni = 0;
  bool any_wide = false;
  const auto take = [&](int c) {
    if (lane < c) {
      const int e = qn - c + lane;
      const double2 t[3] = {qu[0][e], qu[1][e], qu[2][e]}, w = qu[3][e];
      cs_add(sum, err,
             p1_uv_2d<IDX>(t, w.x, __double2hiint(w.y), __double2loint(w.y), coords_a, coords_b, en_a, en_b, u_a, v_b));
    }
    qn -= c;
    __syncwarp();
  };
  // each iteration loads the next one's pair indices (which stream from
  // DRAM) before it works on its own pair
  const int64_t stride = (int64_t)gridDim.x * kUvThreads;
  int64_t i = (int64_t)blockIdx.x * kUvThreads + threadIdx.x;
  int na = 0, nb = 0;
  if (i < npairs) {
    na = pa[i];
    nb = pb[i];
  }
  for (; i - lane < npairs; i += stride) {
    const int a = na, b = nb;
    const bool on = i < npairs;
    if (i + stride < npairs) {
      na = pa[i + stride];
      nb = pb[i + stride];
    }
    const double2* va = reinterpret_cast<const double2*>(coords_a + (int64_t)a * 6);
    const double2 v[3] = {__ldg(va), __ldg(va + 1), __ldg(va + 2)};
    Lines L;
    double tolb;
    load_lines(setup_b + (int64_t)b * kSetup2, L, tolb);
    const double tol = fmin(tol_a[a], tolb);
    const int n = clip_tri_c<kUvThreads>(v, L, p, on);
    any_wide |= n < 0;
    ni += on;
    __syncwarp();
#pragma unroll 1
    for (int k = 2; __any_sync(0xffffffffu, k < n); ++k) {
      double2 t[3] = {};
      double ar = 0.0;
      bool in = k < n;
      if (in) {
        t[0] = p[0];
        t[1] = p[(k - 1) * kUvThreads];
        t[2] = p[k * kUvThreads];
        ar = tri_area(t[0].x, t[0].y, t[1].x, t[1].y, t[2].x, t[2].y);
        in = !(ar < tol);
      }
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int e = qn + __popc(m & ((1u << lane) - 1u));
#pragma unroll
        for (int r = 0; r < 3; ++r) qu[r][e] = t[r];
        qu[3][e] = make_double2((1.0 / 3.0) * ar, __hiloint2double(a, b));
      }
      qn += __popc(m);
      __syncwarp();
      if (qn >= 32) take(32);
    }
  }
  take(qn);
  // pairs that clip_tri_c leaves to clip_tri.  (A thread with one goes over all
  // of its pairs again.  Clipping it in the loop above takes registers that
  // every call pays for: whole calls, 9.5 M ordinary candidates 1283 -> 1313
  // us, 75.9 M of slivers as wide as rounding 11.1 -> 8.3 ms, 30.9 ms by
  // k_p1_mass.)
  if (any_wide) {
    for (i = (int64_t)blockIdx.x * kUvThreads + threadIdx.x; i < npairs; i += stride) {
      const int a = pa[i], b = pb[i];
      const double2* va = reinterpret_cast<const double2*>(coords_a + (int64_t)a * 6);
      const double2 v[3] = {__ldg(va), __ldg(va + 1), __ldg(va + 2)};
      Lines L;
      double tolb, m;
      load_lines(setup_b + (int64_t)b * kSetup2, L, tolb);
      const double tol = fmin(tol_a[a], tolb);
      if (clip_tri_c<kUvThreads>(v, L, p, true) >= 0) continue;
      LocalPoly<kTriWideCap> f, g;
      clip_tri(v[0].x, v[0].y, v[1].x, v[1].y, v[2].x, v[2].y, L, tol, f, g, kTriWideCap, m,
               [&](int, double x0, double y0, double x1, double y1, double x2, double y2) {
                 const double2 t[3] = {{x0, y0}, {x1, y1}, {x2, y2}};
                 cs_add(sum, err, p1_uv_2d<IDX>(t, (1.0 / 3.0) * tri_area(x0, y0, x1, y1, x2, y2), a, b, coords_a,
                                                coords_b, en_a, en_b, u_a, v_b));
               });
    }
  }
  block_reduce_partial<kUvThreads>(sum, err, ni, 0ull, &partials[blockIdx.x]);
}

// ----------------------------------------------------------------------
// P2 inner product (test_parallel_p2_inner_product_2d.F90:398-522)
// ----------------------------------------------------------------------
// P2 basis of triangle cc ([3][2]) at point (x, y), basis_functions_p2
// (:399-433): local coordinates through the inverse Jacobian, then the six
// quadratic Lagrange functions (vertices 1-3, edge midpoints 1-2, 2-3, 1-3).
__device__ __forceinline__ void p2_basis_2d(const double* cc, double x, double y, double f[6]) {
  const double e10 = cc[2] - cc[0], e11 = cc[3] - cc[1];
  const double e20 = cc[4] - cc[0], e21 = cc[5] - cc[1];
  double j11 = e21, j12 = -e20, j21 = -e11, j22 = e10;
  const double det = j11 * j22 - j12 * j21;
  j11 = j11 / det;
  j12 = j12 / det;
  j21 = j21 / det;
  j22 = j22 / det;
  const double d1 = x - cc[0], d2 = y - cc[1];
  const double lx = j11 * d1 + j12 * d2, ly = j21 * d1 + j22 * d2;
  f[0] = ((1.0 - lx) - ly) * ((1.0 - 2.0 * lx) - 2.0 * ly);
  f[1] = lx * (2.0 * lx - 1.0);
  f[2] = ly * (2.0 * ly - 1.0);
  f[3] = (4.0 * lx) * ((1.0 - lx) - ly);
  f[4] = (4.0 * lx) * ly;
  f[5] = (4.0 * ly) * ((1.0 - lx) - ly);
}

__device__ __forceinline__ double p2_interp_2d(const double* cc, const double v[6], double x, double y) {
  double f[6];
  p2_basis_2d(cc, x, y, f);
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) s = s + f[k] * v[k];
  return s;
}

// Per candidate pair: clip, then for every supermesh triangle c the P2
// fields of A and B at c's vertices and edge midpoints and the contribution
// 2 |c| f_b . (M f_a), summed over c in output order.
template <class IDX>
__global__ void __launch_bounds__(128) k_p2_inner(int64_t npairs, const int32_t* __restrict__ pa,
                                                  const int32_t* __restrict__ pb,
                                                  const double* __restrict__ coords_a,
                                                  const double* __restrict__ tol_a,
                                                  const double* __restrict__ coords_b,
                                                  const double* __restrict__ setup_b, const void* en_p2_a,
                                                  const double* __restrict__ field_a, const void* en_p2_b,
                                                  const double* __restrict__ field_b, double* pair_value,
                                                  double* pair_area, int32_t* pair_n) {
  constexpr double M[6][6] = {
      {6.0 / 360.0, -1.0 / 360.0, -1.0 / 360.0, 0.0 / 360.0, -4.0 / 360.0, 0.0 / 360.0},
      {-1.0 / 360.0, 6.0 / 360.0, -1.0 / 360.0, 0.0 / 360.0, 0.0 / 360.0, -4.0 / 360.0},
      {-1.0 / 360.0, -1.0 / 360.0, 6.0 / 360.0, -4.0 / 360.0, 0.0 / 360.0, 0.0 / 360.0},
      {0.0 / 360.0, 0.0 / 360.0, -4.0 / 360.0, 32.0 / 360.0, 16.0 / 360.0, 16.0 / 360.0},
      {-4.0 / 360.0, 0.0 / 360.0, 0.0 / 360.0, 16.0 / 360.0, 32.0 / 360.0, 16.0 / 360.0},
      {0.0 / 360.0, -4.0 / 360.0, 0.0 / 360.0, 16.0 / 360.0, 16.0 / 360.0, 32.0 / 360.0}};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < npairs;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int a = pa[i], b = pb[i];
    const double* ca = coords_a + (int64_t)a * 6;
    const double* cb = coords_b + (int64_t)b * 6;
    double va[6], vb[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      va[k] = field_a[node_of<IDX>(en_p2_a, a, 6, k)];
      vb[k] = field_b[node_of<IDX>(en_p2_b, b, 6, k)];
    }
    Lines L;
    double tolb;
    load_lines(setup_b + (int64_t)b * kSetup2, L, tolb);
    const double tol = fmin(tol_a[a], tolb);
    LocalPoly<kTriWideCap> p, q;
    double m;
    double sp = 0.0, sa = 0.0;
    int nt = 0;
    clip_tri(ca[0], ca[1], ca[2], ca[3], ca[4], ca[5], L, tol, p, q, kTriWideCap, m,
             [&](int, double x0, double y0, double x1, double y1, double x2, double y2) {
               const double ar = tri_area(x0, y0, x1, y1, x2, y2);
               sa = sa + ar;
               ++nt;
               const double px[6] = {x0, x1, x2, 0.5 * (x0 + x1), 0.5 * (x1 + x2), 0.5 * (x0 + x2)};
               const double py[6] = {y0, y1, y2, 0.5 * (y0 + y1), 0.5 * (y1 + y2), 0.5 * (y0 + y2)};
               double fa[6], fb[6];
#pragma unroll
               for (int l = 0; l < 6; ++l) {
                 fb[l] = p2_interp_2d(cb, vb, px[l], py[l]);
                 fa[l] = p2_interp_2d(ca, va, px[l], py[l]);
               }
               double dot = 0.0;
#pragma unroll
               for (int r = 0; r < 6; ++r) {
                 double mi = 0.0;
#pragma unroll
                 for (int k = 0; k < 6; ++k) mi = mi + M[r][k] * fa[k];
                 dot = dot + fb[r] * mi;
               }
               sp = sp + (2.0 * ar) * dot;
             });
    pair_value[i] = sp;
    pair_area[i] = sa;
    pair_n[i] = nt;
  }
}

__global__ void k_check_index(int64_t n, const void* en, int idx_bytes, int64_t limit, int* bad) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = idx_bytes == 8 ? static_cast<const int64_t*>(en)[i] : static_cast<const int32_t*>(en)[i];
    if (v < 0 || v >= limit) atomicExch(bad, 1);
  }
}

cudaError_t launch_check_index(int64_t n, const void* en, int idx_bytes, int64_t limit, int* bad, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  count_launch();
  k_check_index<<<grid_for(n, 256, 8), 256, 0, s>>>(n, en, idx_bytes, limit, bad);
  return cudaGetLastError();
}

cudaError_t launch_p2_inner(int64_t npairs, const int32_t* pair_a, const int32_t* pair_b, const double* coords_a,
                            const double* tol_a, const double* coords_b, const double* setup_b,
                            const void* en_p2_a, const double* field_a, const void* en_p2_b,
                            const double* field_b, int idx_bytes, double* pair_value, double* pair_area,
                            int32_t* pair_n, cudaStream_t s) {
  if (npairs <= 0) return cudaSuccess;
  count_launch();
  const int g = sm_count() * 4;
  if (idx_bytes == 4)
    k_p2_inner<int32_t><<<g, 128, 0, s>>>(npairs, pair_a, pair_b, coords_a, tol_a, coords_b, setup_b, en_p2_a,
                                          field_a, en_p2_b, field_b, pair_value, pair_area, pair_n);
  else
    k_p2_inner<int64_t><<<g, 128, 0, s>>>(npairs, pair_a, pair_b, coords_a, tol_a, coords_b, setup_b, en_p2_a,
                                          field_a, en_p2_b, field_b, pair_value, pair_area, pair_n);
  return cudaGetLastError();
}

// partials written by launch_p1_mass: one per 2D block, or the fixed-order
// reduction's blocks in 3D
int p1_grid_blocks(int dim) { return dim == 2 ? sm_count() * 4 : kReduceBlocks; }

cudaError_t launch_p1_mass(int dim, int64_t npairs, const int32_t* pair_a, const int32_t* pair_b,
                           const double* coords_a, const double* tol_a, const double* coords_b,
                           const double* setup_b, const void* enlist_a, const void* enlist_b,
                           int idx_bytes, const double* u_a, const double* v_b, double* blocks,
                           Partial* partials, cudaStream_t s, int32_t* survivors, unsigned long long* work,
                           const double* faces_a, const double* screen_b, double* pair_uv, const SegList* seg) {
  if (dim == 2) {
    const int g = p1_grid_blocks(2);
    count_launch();
    if (!blocks && u_a && v_b) {
      if (idx_bytes == 4)
        k_p1_uv<int32_t><<<g, kUvThreads, 0, s>>>(npairs, pair_a, pair_b, coords_a, tol_a, coords_b, setup_b, enlist_a,
                                                  enlist_b, u_a, v_b, partials);
      else
        k_p1_uv<int64_t><<<g, kUvThreads, 0, s>>>(npairs, pair_a, pair_b, coords_a, tol_a, coords_b, setup_b, enlist_a,
                                                  enlist_b, u_a, v_b, partials);
    } else if (idx_bytes == 4)
      k_p1_mass<int32_t><<<g, 128, 0, s>>>(npairs, pair_a, pair_b, coords_a, tol_a, coords_b, setup_b, enlist_a, enlist_b, u_a, v_b, blocks, partials);
    else
      k_p1_mass<int64_t><<<g, 128, 0, s>>>(npairs, pair_a, pair_b, coords_a, tol_a, coords_b, setup_b, enlist_a, enlist_b, u_a, v_b, blocks, partials);
    return cudaGetLastError();
  }
  // the early-out pass lists the pairs with output tets (blocks and u^T M v
  // of the others stay zero), then the breadth-first clipper integrates their tets;
  // u^T M v per pair is summed in pair order (a fixed-order reduction into
  // reduce_pairs_blocks() partials), so the integral does not depend on the
  // order in which the lanes took the pairs
  const bool uv = u_a && v_b;
  cudaMemsetAsync(work, 0, 2 * sizeof(unsigned long long), s);
  if (blocks && npairs > 0) cudaMemsetAsync(blocks, 0, sizeof(double) * 16 * npairs, s);
  if (uv && npairs > 0) cudaMemsetAsync(pair_uv, 0, sizeof(double) * npairs, s);
  if (npairs > 0)
    run_prefilter<false, 4, true>(npairs, nullptr, pair_a, pair_b, coords_a, tol_a, setup_b, nullptr, nullptr, survivors,
                            work, faces_a, screen_b, nullptr, seg, s);
  const bool sg = seg_on(seg) && npairs > 0;
  const int4* list = reinterpret_cast<const int4*>(survivors);
  const int4* table = sg ? seg->table : nullptr;
  if (idx_bytes == 4)
    run_bf(list, sg ? work + 2 : work, coords_a, tol_a, setup_b,
           BfP1Sink<int32_t>{coords_a, coords_b, enlist_a, enlist_b, u_a, v_b, blocks, pair_uv}, work + 1, table, s);
  else
    run_bf(list, sg ? work + 2 : work, coords_a, tol_a, setup_b,
           BfP1Sink<int64_t>{coords_a, coords_b, enlist_a, enlist_b, u_a, v_b, blocks, pair_uv}, work + 1, table, s);
  if (uv) {
    count_launch();
    k_reduce_pairs<<<kReduceBlocks, 256, 0, s>>>(npairs, pair_uv, nullptr, partials, nullptr);
  } else {
    cudaMemsetAsync(partials, 0, sizeof(Partial) * kReduceBlocks, s);
  }
  return cudaGetLastError();
}

cudaError_t init_p1_attributes() {
  cudaError_t e = bf_attributes<BfP1Sink<int32_t>>();
  if (e == cudaSuccess) e = bf_attributes<BfP1Sink<int64_t>>();
  return e;
}

}  // namespace lsm
