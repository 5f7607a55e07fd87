// k_collider.cu -- GPU collider for the DEM engine: the GB300 replacement of Woo's
// InsertionSortCollider (src/dem/InsertionSortCollider.cpp:386-613) and AabbCollider's verlet
// boxes (src/dem/Collision.cpp:80-184).
//
// A rebuild runs whenever a particle left its verlet box (aabbIsDirty).  It produces the same
// candidate set as the reference collider on the same boxes: every pair whose closed boxes overlap
// on all three axes (spatialOverlap, InsertionSortCollider.cpp:67-73) and that mayCollide
// (Collision.cpp:21-43), plus every real contact carried over from before (the reference never
// removes real contacts in the collider).  Instead of an incremental insertion sort, the rebuild
//   1. sorts small particles by (grid column in the two long axes, quantised box minimum along the
//      shortest axis): counted into buckets of the key's upper bits, ranked within their buckets,
//   2. sweeps each particle forward along the sweep axis in its own and the 8 neighbouring columns,
//      testing the exact FP64 closed-interval overlap (grid cell >= widest box, so no pair is missed),
//   3. tests walls, facets and other large boxes against every particle of their scene,
//   4. writes the pairs in a deterministic order (count pass with each particle's first pairs buffered,
//      exclusive scan, write pass),
//   5. carries contact history over, finding each pair's old contact by a binary search in the old
//      CSR's row of the lower id, whose partners are sorted,
//   6. builds the per-particle contact CSR with rows ordered by the partner id.
#include "wdem_internal.h"
#include "wdem_math.cuh"
#include "wdem_peri.cuh"
#include "../../include/wdem.h"
#include <algorithm>
#include <cstdio>

namespace wdem {

// columns of the sweep grid at most (32-bit keys: 20 column bits and 12 quantisation bits)
static const int SWEEP_MAX_COLS = (1 << 20) - 2;

// ------------------------------------------------------------------------------------------ boxes
// Bo1_Sphere_Aabb::go / Bo1_Wall_Aabb::go + AabbCollider::updateAabb: pos +- bboxFactor*r,
// walls unbounded except along their axis; both enlarged by verletDist; nodeLastPos = pos.
__global__ void k_bboxes(StepParams P, Particles p, int n) {
  chainWait(false);
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4_32a pr = p.posr[i];
  int sh = p.meta[i].x & 15;
  double4_32a mn, mx;
  if (sh == WDEM_SHAPE_SPHERE) {
    double h = P.bboxFactor * pr.w;
    if (!P.periodic) {
      mn = make_double4_32a(pr.x - h, pr.y - h, pr.z - h, 0);
      mx = make_double4_32a(pr.x + h, pr.y + h, pr.z + h, 0);
    } else {
      // periodic (Sphere.cpp:66-81): unsheared centre, extents enlarged by Cell::shearAlignedExtents
      double hx = h, hy = h, hz = h;
      if (P.hasShear) {
        double e[3] = {h, h, h};
        for (int ax = 0; ax < 3; ax++) {
          int ax1 = (ax + 1) % 3, ax2 = (ax + 2) % 3;
          e[ax1] = e[ax1] + .5 * h * P.sae[ax];
          e[ax2] = e[ax2] + .5 * h * P.sae[ax];
        }
        hx = e[0]; hy = e[1]; hz = e[2];
      }
      const d3 c = mvec(P.unsh, mk(pr.x, pr.y, pr.z));
      mn = make_double4_32a(c.x - hx, c.y - hy, c.z - hz, 0);
      mx = make_double4_32a(c.x + hx, c.y + hy, c.z + hz, 0);
    }
  } else if (sh == WDEM_SHAPE_ELLIPSOID) {
    // Bo1_Ellipsoid_Aabb::go (Ellipsoid.cpp:97-107): half-extents = row norms of trsfFromUnitSphere
    const double4_32a sa = p.semi[i], o4 = p.ori[i];
    qd q;
    q.w = o4.x; q.x = o4.y; q.y = o4.z; q.z = o4.w;
    const d3 c0 = qrot(q, mk(sa.x, 0, 0)), c1 = qrot(q, mk(0, sa.y, 0)), c2 = qrot(q, mk(0, 0, sa.z));
    const double hx = sqrt(c0.x * c0.x + c1.x * c1.x + c2.x * c2.x);
    const double hy = sqrt(c0.y * c0.y + c1.y * c1.y + c2.y * c2.y);
    const double hz = sqrt(c0.z * c0.z + c1.z * c1.z + c2.z * c2.z);
    mn = make_double4_32a(pr.x - hx, pr.y - hy, pr.z - hz, 0);
    mx = make_double4_32a(pr.x + hx, pr.y + hy, pr.z + hz, 0);
  } else if (sh == WDEM_SHAPE_CAPSULE) {
    // Bo1_Capsule_Aabb::go (Capsule.cpp:97-114) with Capsule::alignedBox (:67-73): the box of the four points
    // pos +- dShaft +- radius (1,1,1), dShaft = ori (shaft/2, 0, 0), min/max as Eigen's AlignedBox::extend
    const double4_32a cs = p.semi[i], o4 = p.ori[i];
    qd q;
    q.w = o4.x; q.x = o4.y; q.y = o4.z; q.z = o4.w;
    const d3 ds = qrot(q, mk(.5 * cs.y, 0, 0));
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    mn = make_double4_32a(inf, inf, inf, 0);
    mx = make_double4_32a(-inf, -inf, -inf, 0);
    for (int sa = -1; sa <= 1; sa += 2)
      for (int sb = -1; sb <= 1; sb += 2) {
        const double br = (double)sb * cs.x;
        const d3 e = mk(pr.x, pr.y, pr.z) + (double)sa * ds;
        const double x = e.x + br, y = e.y + br, z = e.z + br;
        mn.x = (x < mn.x) ? x : mn.x; mn.y = (y < mn.y) ? y : mn.y; mn.z = (z < mn.z) ? z : mn.z;
        mx.x = (mx.x < x) ? x : mx.x; mx.y = (mx.y < y) ? y : mx.y; mx.z = (mx.z < z) ? z : mx.z;
      }
  } else if (sh == WDEM_SHAPE_FACET) {
    // Bo1_Facet_Aabb::go (Facet.cpp:275-298), aperiodic: the three nodes +- halfThick (posr.w), coefficient-wise
    // min/max in the order of Eigen's array().min()/max() (std::min/std::max semantics)
    const double ht = pr.w;
    mn = make_double4_32a(pr.x - ht, pr.y - ht, pr.z - ht, 0);
    mx = make_double4_32a(pr.x + ht, pr.y + ht, pr.z + ht, 0);
    const double4_32a v[2] = {p.fv1[i], p.fv2[i]};
    for (int k = 0; k < 2; k++) {
      const double lx = v[k].x - ht, ly = v[k].y - ht, lz = v[k].z - ht;
      const double ux = v[k].x + ht, uy = v[k].y + ht, uz = v[k].z + ht;
      mn.x = (lx < mn.x) ? lx : mn.x; mn.y = (ly < mn.y) ? ly : mn.y; mn.z = (lz < mn.z) ? lz : mn.z;
      mx.x = (mx.x < ux) ? ux : mx.x; mx.y = (mx.y < uy) ? uy : mx.y; mx.z = (mx.z < uz) ? uz : mx.z;
    }
  } else {
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    int ax = (p.meta[i].x >> 4) & 3;
    mn = make_double4_32a(-inf, -inf, -inf, 0);
    mx = make_double4_32a(inf, inf, inf, 0);
    double c = ax == 0 ? pr.x : (ax == 1 ? pr.y : pr.z);
    if (ax == 0) { mn.x = c; mx.x = c; } else if (ax == 1) { mn.y = c; mx.y = c; } else { mn.z = c; mx.z = c; }
  }
  if (p.maxRot) {
    // Aabb.maxRot: -1 (ignored) for spheres and walls; ellipsoids start at 0 and get
    // atan(verletDist / largest half-extent) when verletDist > 0 (Collision.cpp:152-158)
    double mr = -1.;
    if (sh == WDEM_SHAPE_ELLIPSOID || sh == WDEM_SHAPE_CAPSULE) {
      mr = 0.;
      if (P.verletDist > 0) {
        const double arm = .5 * dmax3(mk(mx.x - mn.x, mx.y - mn.y, mx.z - mn.z));
        mr = (arm > 0.) ? atan(P.verletDist / arm) : 0.;
      }
    }
    p.maxRot[i] = mr;
    p.lastOri[i] = p.ori[i];
  }
  if (P.verletDist > 0) {
    double vd = P.verletDist;
    mx.x = mx.x + vd; mx.y = mx.y + vd; mx.z = mx.z + vd;
    mn.x = mn.x - vd; mn.y = mn.y - vd; mn.z = mn.z - vd;
  }
  p.bbmin[i] = mn;
  p.bbmax[i] = mx;
  p.lastPos[i] = make_double4_32a(pr.x, pr.y, pr.z, 0);
  if (p.lastPosf) p.lastPosf[i] = make_float4(truncF(pr.x), truncF(pr.y), truncF(pr.z), 0.f);
}

void launch_bboxes(cudaStream_t s, const StepParams& P, Particles p, int n) {
  if (n <= 0) return;
  launchChained(k_bboxes, (n + 255) / 256, 256, s, P, p, n);
}

// ------------------------------------------------------------------------------------ grid setup
// Order-preserving map double -> unsigned 64 for atomic min/max.
__device__ __forceinline__ unsigned long long ordKey(double d) {
  unsigned long long u = (unsigned long long)__double_as_longlong(d);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double ordVal(unsigned long long k) {
  unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)u);
}

// ext layout (ordered keys): [0..2] min centre, [3..5] max centre (stored as ~key for max via min),
// [6..8] min box lower bound, [9..11] max box upper bound, [12..14] max box width; [15] the blocks done
enum { EXT_WORDS = 16, EXT_VALUES = 15 };

__device__ void gridSetup(const unsigned long long* ext, int nSmall, int maxCols, int maxBuckets, int qbits, GridParams* g) {
  GridParams G;
  G.nSmall = nSmall;
  G.qbits = qbits;
  G.qmax = (1u << qbits) - 1;
  if (nSmall == 0) {
    G.ok = 0; G.sweepAxis = 0; G.ax1 = 1; G.ax2 = 2; G.ncx = G.ncy = 1; G.lo1 = G.lo2 = 0; G.cell = 1; G.invCell = 1;
    G.loS = 0; G.invQ = 0; G.kbits = 0;
    *g = G;
    return;
  }
  double cmin[3], cmax[3], bmin[3], bmax[3], w[3];
  for (int a = 0; a < 3; a++) {
    cmin[a] = ordVal(ext[a]);
    cmax[a] = ordVal(~ext[3 + a]);
    bmin[a] = ordVal(ext[6 + a]);
    bmax[a] = ordVal(~ext[9 + a]);
    w[a] = ordVal(~ext[12 + a]);
  }
  // the sweep runs along the shortest extent of the box centres and the columns tile the two longest: the
  // most columns for the cap, so the fewest boxes per column and the shortest walks into them
  // (a row of batched scenes along one axis would otherwise put all scenes into the same few long columns)
  int ax = 0;
  for (int a = 1; a < 3; a++) if (cmax[a] - cmin[a] < cmax[ax] - cmin[ax]) ax = a;
  int a1 = (ax + 1) % 3, a2 = (ax + 2) % 3;
  double W = fmax(w[a1], w[a2]);
  double cell = W * (1.0 + 1e-6) + 1e-300;
  double e1 = cmax[a1] - cmin[a1], e2 = cmax[a2] - cmin[a2];
  // cap the column count; a larger cell stays correct (only the cell >= W bound matters)
  for (int it = 0; it < 64; it++) {
    double n1 = floor(e1 / cell) + 1, n2 = floor(e2 / cell) + 1;
    if (n1 * n2 <= (double)maxCols) break;
    cell *= 1.25;
  }
  // non-finite extents (NaN or infinite positions) or a grid still too fine: one column
  if (!(e1 >= 0 && e2 >= 0 && e1 < 1e300 && e2 < 1e300 && cell > 0 && cell < 1e300) ||
      (floor(e1 / cell) + 1) * (floor(e2 / cell) + 1) > (double)maxCols) {
    e1 = 0; e2 = 0; cell = 1e300;
    cmin[a1] = 0; cmin[a2] = 0;
  }
  G.sweepAxis = ax; G.ax1 = a1; G.ax2 = a2;
  G.cell = cell;
  G.invCell = 1.0 / cell;
  G.lo1 = cmin[a1]; G.lo2 = cmin[a2];
  G.ncx = (int)(floor(e1 / cell) + 1);
  G.ncy = (int)(floor(e2 / cell) + 1);
  // the buckets: each column divided by the upper kbits bits of the quantised lower bound, as many as fit
  int kb = 0;
  while (kb < qbits && ((long long)G.ncx * G.ncy) << (kb + 1) <= (long long)maxBuckets) kb++;
  G.kbits = kb;
  G.loS = bmin[ax];
  double span = bmax[ax] - bmin[ax];
  G.invQ = (span > 0 && span < 1e300) ? (double)(G.qmax - 1) / span : 0.0;
  if (!(G.invQ == G.invQ)) G.invQ = 0.0;
  if (!(G.loS == G.loS)) G.loS = 0.0;
  G.ok = 1;
  *g = G;
}

// Cells of the periodic box (unsheared coordinates), at least as wide as the widest box per axis, so
// overlapping periodic images of two boxes lie in neighbouring cells (with wrap-around).  Axes with
// fewer than 3 cells get one cell.  Candidates are then decided by the exact spatialOverlapPeri.
struct PeriGrid {
  int nc[3];
  double cw[3], invCw[3], invL[3];
  int ok;
};

__device__ void gridSetupPeri(const unsigned long long* ext, const StepParams& P, int maxCells, PeriGrid* g) {
  PeriGrid G;
  long long tot = 1;
  for (int k = 0; k < 3; k++) {
    double W = ordVal(~ext[12 + k]);
    int n = (W > 0 && W < 1e300) ? (int)floor(P.csize[k] / (W * (1 + 1e-6))) : 1;
    if (n < 3) n = 1;
    if (n > 1024) n = 1024;
    G.nc[k] = n;
    tot *= n;
  }
  while (tot > maxCells) {
    int kmax = 0;
    for (int k = 1; k < 3; k++) if (G.nc[k] > G.nc[kmax]) kmax = k;
    G.nc[kmax] = G.nc[kmax] * 3 / 4;
    if (G.nc[kmax] < 3) G.nc[kmax] = 1;
    tot = (long long)G.nc[0] * G.nc[1] * G.nc[2];
  }
  for (int k = 0; k < 3; k++) {
    G.cw[k] = P.csize[k] / G.nc[k];
    G.invCw[k] = 1.0 / G.cw[k];
    G.invL[k] = 1.0 / P.csize[k];
  }
  G.ok = 1;
  *g = G;
}

// Extents of the small bodies, and the grid from them: every thread keeps the minima of its bodies, a warp's are
// combined by shuffles, the block's in shared memory; the last block to finish sets up the grid (the grid's single
// thread was a launch of its own, 6 us, and the extents took 15 shared atomics a body).
struct GridArgs {
  int maxCols, maxBuckets, qbits;
  GridParams* grid;  // null: periodic
  PeriGrid* peri;
  DeviceStatus* st;
};
static const int EXT_T = 256;
__global__ void __launch_bounds__(EXT_T) k_extents(StepParams P, Particles p, const int* small, int nSmall,
                                                   unsigned long long* ext, GridArgs A) {
  chainWait(false);
  __shared__ unsigned long long sh[EXT_VALUES];
  __shared__ bool last;
  if (threadIdx.x < EXT_VALUES) sh[threadIdx.x] = ~0ull;
  __syncthreads();
  unsigned long long v[EXT_VALUES];
#pragma unroll
  for (int q = 0; q < EXT_VALUES; q++) v[q] = ~0ull;
  auto lower = [](unsigned long long& a, unsigned long long b) { if (b < a) a = b; };
  for (int k = blockIdx.x * EXT_T + threadIdx.x; k < nSmall; k += gridDim.x * EXT_T) {
    const int i = small[k];
    const double4_32a pr = p.posr[i], mn = p.bbmin[i], mx = p.bbmax[i];
    lower(v[0], ordKey(pr.x)); lower(v[1], ordKey(pr.y)); lower(v[2], ordKey(pr.z));
    lower(v[3], ~ordKey(pr.x)); lower(v[4], ~ordKey(pr.y)); lower(v[5], ~ordKey(pr.z));
    lower(v[6], ordKey(mn.x)); lower(v[7], ordKey(mn.y)); lower(v[8], ordKey(mn.z));
    lower(v[9], ~ordKey(mx.x)); lower(v[10], ~ordKey(mx.y)); lower(v[11], ~ordKey(mx.z));
    lower(v[12], ~ordKey(mx.x - mn.x)); lower(v[13], ~ordKey(mx.y - mn.y)); lower(v[14], ~ordKey(mx.z - mn.z));
  }
#pragma unroll
  for (int q = 0; q < EXT_VALUES; q++) {
    for (int off = 16; off > 0; off >>= 1) lower(v[q], __shfl_xor_sync(0xffffffffu, v[q], off));
    if ((threadIdx.x & 31) == 0) atomicMin(&sh[q], v[q]);
  }
  __syncthreads();
  if (threadIdx.x < EXT_VALUES) atomicMin(&ext[threadIdx.x], sh[threadIdx.x]);
  __threadfence();
  __syncthreads();
  // the counter starts at all ones, like the minima
  if (threadIdx.x == 0) last = (unsigned)(atomicAdd(&ext[EXT_VALUES], 1ull) + 1ull) == gridDim.x - 1;
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  A.st->longBucket = 0;
  unsigned long long e[EXT_VALUES];
  for (int q = 0; q < EXT_VALUES; q++) e[q] = *(volatile unsigned long long*)(ext + q);
  if (A.peri) gridSetupPeri(e, P, A.maxBuckets, A.peri);
  else gridSetup(e, nSmall, A.maxCols, A.maxBuckets, A.qbits, A.grid);
}

__device__ __forceinline__ double cmp3(const double4_32a& v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// monotone non-decreasing quantisation along the sweep axis (any such map gives the same pair set: ties
// are ordered by particle id; coarser steps only lengthen the walks a little)
__device__ __forceinline__ unsigned quant(double x, const GridParams& G) {
  double t = (x - G.loS) * G.invQ;
  if (!(t > 0)) return 0;                 // also NaN
  if (t >= (double)G.qmax) return G.qmax;
  return (unsigned)t;                      // truncation == floor for t >= 0
}

__device__ __forceinline__ void columnOf(const double4_32a& pr, const GridParams& G, int& cx, int& cy) {
  // multiplying by the rounded reciprocal moves a centre at most a few ulp across a column edge: two centres
  // closer than the widest box (cell = widest box x (1 + 1e-6)) still fall into the same or adjacent columns
  double t1 = floor((cmp3(pr, G.ax1) - G.lo1) * G.invCell);
  double t2 = floor((cmp3(pr, G.ax2) - G.lo2) * G.invCell);
  cx = (int)fmin(fmax(t1, 0.0), (double)(G.ncx - 1));
  cy = (int)fmin(fmax(t2, 0.0), (double)(G.ncy - 1));
}

// sweep key of each small body (column, quantised lower bound) and its place in its bucket
__global__ void k_make_keys(Particles p, const int* small, int nSmall, const GridParams* g, unsigned* keys, unsigned* place,
                            unsigned* count) {
  chainWait(false);
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nSmall) return;
  GridParams G = *g;
  int i = small[k];
  int cx, cy;
  columnOf(p.posr[i], G, cx, cy);
  const unsigned col = (unsigned)(cx + G.ncx * cy);
  const unsigned key = (col << G.qbits) | quant(cmp3(p.bbmin[i], G.sweepAxis), G);
  keys[k] = key;
  place[k] = atomicAdd(&count[key >> (G.qbits - G.kbits)], 1u);
}

// ------------------------------------------------------------------------------------ scan
// Exclusive scan of a[0..n) in place, a[n] <- total, in one kernel (decoupled look-back, Merrill & Garland 2016).
// A block takes its tile in the order of a ticket, so every earlier tile is running or done; it publishes the
// tile's sum, its first warp looks back over 32 earlier tiles at a time up to the nearest published prefix, and it
// publishes its own prefix.  A published word carries the number of the scan, so nothing is cleared between scans,
// and the ticket counts on from where the last scan left it.  A rebuild's scans were 3 to 5 launches each before
// (tile scans, the scan of their sums, the sums added back), of 3 us for 15k bodies.
static const int SCAN_T = 256, SCAN_I = 16, SCAN_TILE = SCAN_T * SCAN_I;
//
// A look-back whose wait runs out says so in scanFailed and takes 0 for what it waited for; so does a block whose ticket
// is not one of this launch's (a launch that never ran after its tickets were counted).  The scanned values are then
// not offsets of anything, and every kernel that uses them, or what was made from them, returns at once.
static const unsigned SCAN_AGG = 1u, SCAN_PRE = 2u, SCAN_EPOCHS = 1u << 30;
__device__ __forceinline__ void scanGaveUp(DeviceStatus* st) {
  st->scanFailed = 1;
  st->haltAt = -1;
  if (atomicCAS(&st->code, 0, WDEM_ERR_TIMEOUT) == 0) st->detail = DETAIL_SCAN;
}

__global__ void __launch_bounds__(SCAN_T) k_scan(unsigned* a, long long n, unsigned long long* status, unsigned* ticket,
                                                 unsigned ticket0, unsigned epoch, int looks, int total, DeviceStatus* st) {
  chainWait(false);
  __shared__ unsigned tileS, prefixS;
  __shared__ unsigned warpSum[SCAN_T / 32];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t == 0) tileS = atomicAdd(ticket, 1u) - ticket0;
  __syncthreads();
  if (tileS >= gridDim.x) {
    if (t == 0) scanGaveUp(st);
    return;
  }
  const long long tile = tileS;
  const long long first = tile * SCAN_TILE + (long long)t * SCAN_I;
  unsigned v[SCAN_I];
  unsigned sum = 0;
#pragma unroll
  for (int k = 0; k < SCAN_I; k += 4) {
    uint4 q = make_uint4(0, 0, 0, 0);
    if (first + k + 4 <= n) q = *reinterpret_cast<const uint4*>(a + first + k);
    else {
      if (first + k < n) q.x = a[first + k];
      if (first + k + 1 < n) q.y = a[first + k + 1];
      if (first + k + 2 < n) q.z = a[first + k + 2];
    }
    v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
    sum += q.x + q.y + q.z + q.w;
  }
  unsigned inc = sum;  // inclusive scan of the threads' sums within the warp
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += u;
  }
  if (lane == 31) warpSum[warp] = inc;
  __syncthreads();
  unsigned before = 0, tileSum = 0;
#pragma unroll
  for (int w = 0; w < SCAN_T / 32; w++) {
    if (w < warp) before += warpSum[w];
    tileSum += warpSum[w];
  }
  if (warp == 0) {
    const unsigned long long tag = (unsigned long long)epoch << 34;
    unsigned prefix = 0;
    if (tile > 0) {
      if (lane == 0) *(volatile unsigned long long*)(status + tile) = tag | ((unsigned long long)SCAN_AGG << 32) | tileSum;
      for (long long j = tile - 1; j >= 0; j -= 32) {
        const long long q = j - lane;
        unsigned long long w = tag | ((unsigned long long)SCAN_PRE << 32);  // before the first tile: prefix 0
        if (q >= 0) {
          for (int left = looks;; left--) {
            if (left <= 0) {
              scanGaveUp(st);
              break;  // w: prefix 0
            }
            const unsigned long long seen = *(volatile unsigned long long*)(status + q);
            if ((seen >> 34) == epoch && ((seen >> 32) & 3u) != 0) {
              w = seen;
              break;
            }
            __nanosleep(20);
          }
        }
        const unsigned pre = __ballot_sync(0xffffffffu, ((w >> 32) & 3u) == SCAN_PRE);
        const int stop = pre ? __ffs(pre) - 1 : 31;  // the nearest tile whose prefix is known
        prefix += __reduce_add_sync(0xffffffffu, lane <= stop ? (unsigned)w : 0u);
        if (pre) break;
      }
    }
    if (lane == 0) {
      *(volatile unsigned long long*)(status + tile) = tag | ((unsigned long long)SCAN_PRE << 32) | (prefix + tileSum);
      prefixS = prefix;
    }
  }
  __syncthreads();
  unsigned run = prefixS + before + (inc - sum);
#pragma unroll
  for (int k = 0; k < SCAN_I; k += 4) {
    uint4 q;
    q.x = run; run += v[k];
    q.y = run; run += v[k + 1];
    q.z = run; run += v[k + 2];
    q.w = run; run += v[k + 3];
    if (first + k + 4 <= n) *reinterpret_cast<uint4*>(a + first + k) = q;
    else {
      if (first + k < n) a[first + k] = q.x;
      if (first + k + 1 < n) a[first + k + 1] = q.y;
      if (first + k + 2 < n) a[first + k + 2] = q.z;
    }
  }
  // the thread after the last value (of the last tile, also when n fills it) holds the total
  if ((tile + 1) * SCAN_TILE >= n && t == SCAN_T - 1) {
    a[n] = prefixS + tileSum;
    if (total >= 0) st->totals[total] = prefixS + tileSum;
  }
}

// 32-bit words of scan scratch (ticket, then one 64-bit status word per tile) for scans of n values
long long scan_scratch_words(long long n) { return 64 + 2 * ((n + SCAN_TILE - 1) / SCAN_TILE + 1); }

void exclusive_scan_u32(cudaStream_t s, unsigned* a, long long n, ColliderScratch& cs, int total) {
  if (n <= 0) {
    cudaMemsetAsync(a, 0, sizeof(unsigned), s);  // empty: total 0
    if (total >= 0) cudaMemsetAsync(&cs.st->totals[total], 0, sizeof(unsigned), s);
    return;
  }
  if (++cs.scanEpoch >= SCAN_EPOCHS) {  // the numbers start again: no word of the old ones may be left
    cudaMemsetAsync(cs.scanScratch, 0, cs.scanCap * sizeof(unsigned), s);
    cs.scanEpoch = 1;
    cs.scanTickets = 0;
  }
  const unsigned nt = (unsigned)((n + SCAN_TILE - 1) / SCAN_TILE);
  launchChained(k_scan, nt, SCAN_T, s, a, n, reinterpret_cast<unsigned long long*>(cs.scanScratch + 64), cs.scanScratch,
                cs.scanTickets, cs.scanEpoch, cs.scanLooks, total, cs.st);
  cs.scanTickets += nt;
}

// ------------------------------------------------------------------------------------ bucket sort
// Small bodies in the order of (key, id): each takes a place in the bucket of its key's upper bits (k_make_keys,
// k_keys_peri), a scan of the buckets' counts gives their starts, the bodies go to their places and are ranked
// within their buckets, which hold a body or two (sweep keys) or a cell's handful (periodic).  The start of any key
// is then a table lookup for the sweep.  An LSD radix sort of the keys took 4 passes of 8 bits, each a
// dependent launch of 10 us at 15k bodies and 25 us at 500k.
//
// Ranking costs a bucket the square of its length.  A body far from all others stretches the grid (its columns are
// widened until they are no more than the buckets) and the others share few buckets: 100k spheres with one 100 edge
// lengths away along each axis have 9,212 in a bucket, 1M with one 10,000 away along two axes 503,892.  The sweep
// kernel's start in a neighbouring column is bisected for the same reason.  Above BUCKET_RANKED the bodies are sorted
// by merges instead (col_sort_merge; k_bucket_place tells, the count behind it is void and made again).  Rebuild in
// ms, ranked and merged, by the longest bucket: 423 0.178 and 0.237, 1175 0.258 and 0.292 (100k bodies); 2500 1.48
// and 1.31, 12,100 8.9 and 6.9, 503,892 149 and 19.0 (1M; a radix sort with bisection 20.4).  A cell of the periodic
// grid is no smaller than the widest box, and the walk over its candidates is quadratic too and 14 times as long:
// always ranked.
static const unsigned BUCKET_RANKED = 2048;
__global__ void k_bucket_place(const int* small, int nSmall, const unsigned* keys, const unsigned* place,
                               const unsigned* start, const GridParams* g, unsigned long long* tmp, DeviceStatus* st) {
  chainWait(false);
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nSmall || st->scanFailed) return;
  const unsigned key = keys[k];
  const unsigned b = g ? key >> (g->qbits - g->kbits) : key;
  const unsigned first = start[b];
  tmp[first + place[k]] = ((unsigned long long)key << 32) | (unsigned)small[k];
  if (g && start[b + 1] - first > BUCKET_RANKED) st->longBucket = 1;
}
__device__ __forceinline__ unsigned rankInBucket(const unsigned long long* tmp, unsigned long long v, unsigned beg, unsigned end) {
  unsigned pos = beg;
  for (unsigned q = beg; q < end; q++) pos += tmp[q] < v ? 1u : 0u;
  return pos;
}
// Sweep order, with the sweep records, two float4 per body: the box in FP32 with the minimum rounded down and
// the maximum rounded up (every pair of FP64 boxes that overlap overlaps in FP32 too, so a pair the FP32
// test rejects needs no FP64 test), the mask (lo.w) and meta.x with shape and scene (hi.w).  The sweep
// walks these contiguous records instead of gathering meta, bbmin and bbmax by particle id.
template <bool SORTED>
__global__ void k_bucket_rank(Particles p, int nSmall, const unsigned long long* tmp, const unsigned* start,
                              const GridParams* g, unsigned* keys, unsigned* vals, float4* rec, const DeviceStatus* st) {
  chainWait(false);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nSmall || st->scanFailed || (!SORTED && st->longBucket)) return;
  const unsigned long long v = tmp[e];
  const unsigned key = (unsigned)(v >> 32);
  const int i = (int)(unsigned)v;
  const double4_32a mn = p.bbmin[i], mx = p.bbmax[i];
  const int4 m = p.meta[i];
  unsigned s = (unsigned)e;
  if (!SORTED) {
    const unsigned b = key >> (g->qbits - g->kbits);
    s = rankInBucket(tmp, v, start[b], start[b + 1]);
  }
  keys[s] = key;
  vals[s] = (unsigned)i;
  rec[2 * s] = make_float4(__double2float_rd(mn.x), __double2float_rd(mn.y), __double2float_rd(mn.z), __uint_as_float((unsigned)m.z));
  rec[2 * s + 1] = make_float4(__double2float_ru(mx.x), __double2float_ru(mx.y), __double2float_ru(mx.z), __int_as_float(m.x));
}

// The bodies sorted by merges: tiles of SORT_TILE by a bitonic network in shared memory, then runs of twice the length
// a pass, every entry finding its place in the neighbouring run by bisection (entries are all different).
static const int SORT_T = 256, SORT_TILE = 2048;
__global__ void __launch_bounds__(SORT_T) k_tile_sort(const unsigned long long* in, unsigned long long* out, int n) {
  chainWait(false);
  __shared__ unsigned long long v[SORT_TILE];
  const int base = blockIdx.x * SORT_TILE;
  for (int k = threadIdx.x; k < SORT_TILE; k += SORT_T) v[k] = base + k < n ? in[base + k] : ~0ull;
  for (int size = 2; size <= SORT_TILE; size *= 2)
    for (int step = size / 2; step > 0; step /= 2) {
      __syncthreads();
      for (int q = threadIdx.x; q < SORT_TILE / 2; q += SORT_T) {
        const int a = 2 * q - (q & (step - 1)), b = a + step;
        const unsigned long long x = v[a], y = v[b];
        if ((x > y) == ((a & size) == 0)) { v[a] = y; v[b] = x; }
      }
    }
  __syncthreads();
  for (int k = threadIdx.x; k < SORT_TILE; k += SORT_T)
    if (base + k < n) out[base + k] = v[k];
}
__global__ void k_merge_runs(const unsigned long long* in, unsigned long long* out, int n, int run) {
  chainWait(false);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const unsigned long long v = in[e];
  const int first = e / run * run;                          // of this entry's run
  const bool left = (e / run) % 2 == 0;
  int lo = left ? min(first + run, n) : first - run;        // the other run
  int hi = left ? min(first + 2 * (long long)run, (long long)n) : first;
  const int other = lo;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (in[mid] < v) lo = mid + 1; else hi = mid;
  }
  out[(left ? e : e - run) + (lo - other)] = v;
}

// ------------------------------------------------------------------------------------ sweep
__device__ __forceinline__ bool overlap3(const double4_32a& mn1, const double4_32a& mx1, const double4_32a& mn2, const double4_32a& mx2) {
  return (mn1.x <= mx2.x) && (mx1.x >= mn2.x) && (mn1.y <= mx2.y) && (mx1.y >= mn2.y) && (mn1.z <= mx2.z) && (mx1.z >= mn2.z);
}
__device__ __forceinline__ bool mayCollide(unsigned m1, unsigned m2, unsigned lone) {
  return (m1 & m2) != 0 && (m1 & m2 & lone) == 0;
}
// contact orientation: same shape -> (lower id, higher id); otherwise the order of the Cg2 functor
// (Wall+Sphere, Facet+Sphere, Sphere+Ellipsoid, Wall+Ellipsoid)
__device__ __forceinline__ int2 orient(int i, int j, int shi, int shj) {
  int a = min(i, j), b = max(i, j);
  int sa = (a == i) ? shi : shj, sb = (a == i) ? shj : shi;
  if (pairSwaps(sa, sb)) {
    int t = a; a = b; b = t;
  }
  return make_int2(a, b);
}

__device__ __forceinline__ bool overlapF(const float4& mn1, const float4& mx1, const float4& mn2, const float4& mx2) {
  return (mn1.x <= mx2.x) && (mx1.x >= mn2.x) && (mn1.y <= mx2.y) && (mx1.y >= mn2.y) && (mn1.z <= mx2.z) && (mx1.z >= mn2.z);
}

// The boxes overlap beyond the rounding of their FP32 copies: each bound was rounded outward by at most 2^-23 of
// itself and the difference of two rounds by 2^-24, so a closed FP64 interval test holds when every difference of a
// maximum and a minimum exceeds 4e-7 of their magnitudes.  An FP64 compare holds a scheduler for 64 cycles whichever
// lanes need it, and the six of a box pair ran in nearly every round of a warp's walk: 175 of the 217 us of the
// sweep over 508k bodies.  NaN fails.  The added 1e-37 is for magnitudes near FP32's subnormals, which round to
// multiples of 2^-149.
__device__ __forceinline__ bool clearlyAbove(float mx, float mn) { return mx - mn > __fmaf_rn(4e-7f, fabsf(mx) + fabsf(mn), 1e-37f); }
__device__ __forceinline__ bool overlapSure(const float4& mn1, const float4& mx1, const float4& mn2, const float4& mx2) {
  return clearlyAbove(mx2.x, mn1.x) && clearlyAbove(mx1.x, mn2.x) && clearlyAbove(mx2.y, mn1.y) && clearlyAbove(mx1.y, mn2.y) &&
         clearlyAbove(mx2.z, mn1.z) && clearlyAbove(mx1.z, mn2.z);
}
// a bound of a large body in FP32, within 2^-23 of itself, on the integer pipe: infinities kept; NaN for NaN and for
// what only FP64 can hold, so that every test on it fails and the FP64 test decides
__device__ __forceinline__ float boundF(double x) {
  const Halves h = halvesOf(x);
  const unsigned a = h.hi & 0x7fffffffu;
  if (a >= 0x47f00000u)  // 2^128
    return __uint_as_float(a == 0x7ff00000u && h.lo == 0 ? (h.hi & 0x80000000u) | 0x7f800000u : 0x7fc00000u);
  return truncF(x);
}
// clearlyAbove where the large body's bound, the first argument, is infinite: beyond any bound of a small body, whose
// copy may be infinite too but stands for a finite number (NaN fails)
__device__ __forceinline__ bool infAbove(float mx, float fmn) { return mx == __int_as_float(0x7f800000) && fmn < mx; }
__device__ __forceinline__ bool infBelow(float mn, float fmx) { return mn == -__int_as_float(0x7f800000) && fmx > mn; }
__device__ __forceinline__ bool overlapSureLarge(const float4& fmn, const float4& fmx, const float4& gn, const float4& gx) {
  return (infAbove(gx.x, fmn.x) || clearlyAbove(gx.x, fmn.x)) && (infBelow(gn.x, fmx.x) || clearlyAbove(fmx.x, gn.x)) &&
         (infAbove(gx.y, fmn.y) || clearlyAbove(gx.y, fmn.y)) && (infBelow(gn.y, fmx.y) || clearlyAbove(fmx.y, gn.y)) &&
         (infAbove(gx.z, fmn.z) || clearlyAbove(gx.z, fmn.z)) && (infBelow(gn.z, fmx.z) || clearlyAbove(fmx.z, gn.z));
}

struct SweepArgs {
  const float4* rec;
  const unsigned* keys;
  const unsigned* vals;
  const unsigned* start;  // first sorted position of each bucket
  const int* large;
  int nLarge;
  int nSmall;
  unsigned loneMask;
  const int* sceneWall;  // per-scene ranges of the large list (null: one scene)
  unsigned* buf;         // SWEEP_BUF partners per thread (thread minor), written by the counting pass: the other
                         //   body's id, bit 31 when it comes first in the pair (null: none kept)
};

// The sweep runs twice: counting (WRITE false) and writing at the scanned offsets (WRITE true).  With a
// buffer, the counting pass keeps each thread's first SWEEP_BUF pairs in walk order and the writing pass
// copies them, walking again only for threads that found more: the output is the same, in the same order.
template <bool WRITE>
__global__ void k_sweep(Particles p, SweepArgs A, const GridParams* g, unsigned* counts, int2* out, long long cap,
                        const DeviceStatus* st) {
  chainWait(false);
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= sweepThreads(A.nSmall, A.nLarge) || st->scanFailed || st->longBucket) return;
  unsigned cnt = 0;
  unsigned long long base = WRITE ? counts[s] : 0;
  if (WRITE && A.buf) {
    const unsigned found = counts[s + 1] - counts[s];
    if (found <= (unsigned)SWEEP_BUF) {
      const long long T = sweepThreads(A.nSmall, A.nLarge);
      const int i = s < A.nSmall ? (int)A.vals[s] : A.nLarge > 0 ? A.large[s - A.nSmall] : 0;
      for (unsigned k = 0; k < found; k++) {
        const unsigned v = A.buf[k * T + s];
        const int j = (int)(v & 0x7fffffffu);
        if (base + k < (unsigned long long)cap) out[base + k] = (v >> 31) ? make_int2(j, i) : make_int2(i, j);
      }
      return;
    }
  }
  // the pair of the thread's body i with j, as orient() gives it
  auto emit = [&](int i, int2 pr) {
    if (WRITE) {
      const unsigned long long o = base + cnt;
      if (o < (unsigned long long)cap) out[o] = pr;
    } else if (A.buf && cnt < (unsigned)SWEEP_BUF) {
      const long long T = sweepThreads(A.nSmall, A.nLarge);
      A.buf[(long long)cnt * T + s] = pr.x == i ? (unsigned)pr.y : (unsigned)pr.x | 0x80000000u;
    }
    cnt++;
  };
  if (s >= A.nSmall) {
    // large-large pairs, one thread per large body a: the bodies after it in the large list up to the
    // first one of another scene (the list is grouped by scene)
    const int a = s - A.nSmall;
    if (a < A.nLarge) {
      const int i = A.large[a];
      const int4 mi = p.meta[i];
      const double4_32a mn = p.bbmin[i], mx = p.bbmax[i];
      for (int b = a + 1; b < A.nLarge; b++) {
        const int j = A.large[b];
        const int4 mj = p.meta[j];
        if (sceneOf(mi.x) != sceneOf(mj.x)) break;
        if (!mayCollide((unsigned)mi.z, (unsigned)mj.z, A.loneMask)) continue;
        if (!overlap3(mn, mx, p.bbmin[j], p.bbmax[j])) continue;
        emit(i, orient(i, j, mi.x & 15, mj.x & 15));
      }
    }
    if (!WRITE) counts[s] = cnt;
    return;
  }
  GridParams G = *g;
  const unsigned key = A.keys[s];
  int i = (int)A.vals[s];
  int4 mi = p.meta[i];
  double4_32a mn = p.bbmin[i], mx = p.bbmax[i];
  const float4 fmn = A.rec[2 * s], fmx = A.rec[2 * s + 1];
  unsigned qi = key & G.qmax;
  unsigned qmax = quant(cmp3(mx, G.sweepAxis), G);
  const int col = (int)(key >> G.qbits);
  const int cx = col % G.ncx, cy = col / G.ncx;
  const int kshift = G.qbits - G.kbits;
  for (int dy = -1; dy <= 1; dy++) {
    int y = cy + dy;
    if (y < 0 || y >= G.ncy) continue;
    for (int dx = -1; dx <= 1; dx++) {
      int x = cx + dx;
      if (x < 0 || x >= G.ncx) continue;
      const int c2 = x + G.ncx * y;
      const int end = (int)A.start[(unsigned)(c2 + 1) << G.kbits];
      int q;
      if (c2 == col) q = s + 1;
      else {
        // the first box of the column after (key, id): bisected within its bucket
        const unsigned target = ((unsigned)c2 << G.qbits) | qi, b = target >> kshift;
        q = (int)A.start[b];
        int to = (int)A.start[b + 1];
        while (q < to) {
          const int mid = (q + to) >> 1;
          const unsigned km = A.keys[mid];
          if (km < target || (km == target && (int)A.vals[mid] < i)) q = mid + 1; else to = mid;
        }
      }
      for (; q < end; q++) {
        if ((A.keys[q] & G.qmax) > qmax) break;
        const float4 gmn = A.rec[2 * q], gmx = A.rec[2 * q + 1];
        const unsigned maskj = __float_as_uint(gmn.w);
        const int metaxj = __float_as_int(gmx.w);
        if (!mayCollide((unsigned)mi.z, maskj, A.loneMask)) continue;
        if (sceneOf(mi.x) != sceneOf(metaxj)) continue;
        if (!overlapF(fmn, fmx, gmn, gmx)) continue;
        int j = (int)A.vals[q];
        if (!overlapSure(fmn, fmx, gmn, gmx)) {
          WDEM_REAL_BRANCH();
          if (!overlap3(mn, mx, p.bbmin[j], p.bbmax[j])) continue;
        }
        emit(i, orient(i, j, mi.x & 15, metaxj & 15));
      }
    }
  }
  const int sc = sceneOf(mi.x);
  const int a0 = A.sceneWall ? A.sceneWall[sc] : 0, a1 = A.sceneWall ? A.sceneWall[sc + 1] : A.nLarge;
  for (int a = a0; a < a1; a++) {
    int j = A.large[a];
    int4 mj = p.meta[j];
    if (!mayCollide((unsigned)mi.z, (unsigned)mj.z, A.loneMask)) continue;
    const double4_32a ln = p.bbmin[j], lx = p.bbmax[j];
    const float4 gn = make_float4(boundF(ln.x), boundF(ln.y), boundF(ln.z), 0.f);
    const float4 gx = make_float4(boundF(lx.x), boundF(lx.y), boundF(lx.z), 0.f);
    // apart beyond the rounding on some axis, or overlapping beyond it on all: decided; else the FP64 test
    if (clearlyAbove(gn.x, fmx.x) || clearlyAbove(fmn.x, gx.x) || clearlyAbove(gn.y, fmx.y) || clearlyAbove(fmn.y, gx.y) ||
        clearlyAbove(gn.z, fmx.z) || clearlyAbove(fmn.z, gx.z))
      continue;
    if (!overlapSureLarge(fmn, fmx, gn, gx)) {
      WDEM_REAL_BRANCH();
      if (!overlap3(mn, mx, ln, lx)) continue;
    }
    emit(i, orient(i, j, mi.x & 15, mj.x & 15));
  }
  if (!WRITE) counts[s] = cnt;
}

// ------------------------------------------------------------------------------------ retain
// Real contacts whose new boxes no longer overlap stay in the container (the reference collider
// removes only non-real contacts on separation, InsertionSortCollider.cpp:107-110).
__global__ void k_retain_flag(StepParams P, Particles p, Contacts old, long long nOld, unsigned* flag,
                              const float4* pci, const float4* phi) {
  chainWait(false);
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nOld) return;
  unsigned f = 0;
  if ((old.state[c] & CS_MASK) == CS_REAL) {
    int2 id = old.ids[c];
    bool ov;
    if (P.periodic) {
      // boxes that overlap on every axis by more than the FP32 margin (both narrow: no ambiguity) overlap
      // in the exact test too (the FP32 copies of this rebuild, k_keys_peri)
      const float4 c1 = pci[id.x], h1 = phi[id.x], c2 = pci[id.y], h2 = phi[id.y];
      const float L0 = (float)P.csize[0], L1 = (float)P.csize[1], L2 = (float)P.csize[2];
      if (h1.w == 0.f && h2.w == 0.f && periNear(c1.x, h1.x, c2.x, h2.x, L0, 1.f / L0) &&
          periNear(c1.y, h1.y, c2.y, h2.y, L1, 1.f / L1) && periNear(c1.z, h1.z, c2.z, h2.z, L2, 1.f / L2))
        ov = true;
      else {
        int4 per; bool amb = false;
        ov = overlapPeri(p.bbmin[id.x], p.bbmax[id.x], p.bbmin[id.y], p.bbmax[id.y], P.csize, per, amb);
      }
    } else ov = overlap3(p.bbmin[id.x], p.bbmax[id.x], p.bbmin[id.y], p.bbmax[id.y]);
    if (!ov) f = 1;
  }
  flag[c] = f;
}
__global__ void k_retain_write_dist(Contacts old, long long nOld, const unsigned* flagScan, int4* out, long long base, long long cap) {
  chainWait(false);
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nOld) return;
  if (flagScan[c + 1] != flagScan[c]) {
    long long o = base + flagScan[c];
    if (o < cap) out[o] = old.cdist[c];
  }
}
__global__ void k_retain_write(Contacts old, long long nOld, const unsigned* flagScan, int2* out, long long base, long long cap) {
  chainWait(false);
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nOld) return;
  if (flagScan[c + 1] != flagScan[c]) {
    long long o = base + flagScan[c];
    if (o < cap) out[o] = old.ids[c];
  }
}

// ------------------------------------------------------------------------------------ old-contact lookup
// The contact of the pair (a, b) in the container whose CSR is `csr` (built at the last rebuild or upload):
// binary search of the partner in the row of the lower id, which is sorted by partner; -1 if none.
__device__ __forceinline__ long long csrFind(const Csr& csr, int a, int b) {
  const int lo = min(a, b), hi = max(a, b);
  if (lo < 0 || hi >= csr.n) return -1;  // ids the rows do not cover (appended since) had no contact
  int l = csr.rowptr[lo], r = csr.rowptr[lo + 1];
  const int end = r;
  while (l < r) {
    const int m = (l + r) >> 1;
    if (csr.partner[m] < (unsigned)hi) l = m + 1; else r = m;
  }
  if (l < end && csr.partner[l] == (unsigned)hi) return (long long)(csr.ent[l] & 0x7fffffffu);
  return -1;
}

// ------------------------------------------------------------------------------------ CSR rows
// The CSR is built by counting: every entry takes a place in its row (one atomic per entry), a scan of the rows'
// counts gives their starts, the entries go to their places, and each entry's rank among its row's partners is its
// final position.  Rows of bodies of like size hold ten or twenty entries, so the ranks are a few loads from L1; the
// order does not depend on the atomics.  The radix sort of 2 C keys of up to 46 bits this replaces took 6 passes over 12 bytes an entry
// (9 launches of 41 us a rebuild with 500k bodies and 2 M pairs; k_csr_fill and k_csr_rank now take 28 + 55 us).
// A wall's or facet's row can hold every body: it is divided into V ranges of S partner ids, counted apart (so the
// atomics spread as well), and an entry is ranked within its range.  A large sphere among small ones has a long row
// too, ranked in the square of its length; but its box also widens the sweep's columns and its thread walks every
// partner, which takes far longer: of the 67 ms of a rebuild with a sphere that 38,000 others meet, k_sweep's two
// passes take 33 and 40 at one launch each, k_csr_rank 0.97 (107 ms with the radix sorts; 3,500 partners among 1M
// spheres 19.1 and 24.4 ms).
struct RowCount {
  unsigned* cnt;        // rowptr as counts, then starts
  unsigned* sub;        // nLarge x V counts of the large bodies' ranges, then starts within their rows
  const int* largeIdx;  // index of a body in the large list, -1 for the others
  int V, S;
};
// V ranges for each of nLarge bodies of n: about n ranges in all, none of fewer than 1024 ids
static void largeRanges(int n, int nLarge, int& V, int& S) {
  V = 1;
  if (nLarge > 0) V = std::max(1, std::min(n / 1024 + 1, n / nLarge));
  S = (n + V - 1) / V;
  if (S < 1) S = 1;
}
// index of the range that partner's entry in a large body's row falls into, -1 for the other rows
__device__ __forceinline__ int rangeOf(const RowCount& R, int row, int partner, bool maybeLarge) {
  if (!maybeLarge) return -1;
  const int l = R.largeIdx[row];
  return l < 0 ? -1 : l * R.V + partner / R.S;
}
__device__ __forceinline__ int takePlace(const RowCount& R, int row, int partner, bool maybeLarge) {
  const int k = rangeOf(R, row, partner, maybeLarge);
  return (int)atomicAdd(k < 0 ? &R.cnt[row] : &R.sub[k], 1u);
}
// pairs with a wall or a facet carry one of these bits (and so do pairs without a functor)
__device__ __forceinline__ bool maybeLarge(uint8_t state) { return (state & (CS_WALL_A | CS_WALL_B | CS_FACET)) != 0; }

// ------------------------------------------------------------------------------------ carry-over
// History of pairs already in the container is copied; new pairs start as potential contacts
// created in this step (InsertionSortCollider.hpp:106-113 stepCreated=scene->step).  A contact that
// the law broke in the previous step (pending) becomes potential: removePending in a full run keeps
// it only when its new boxes overlap, which holds for every pair the sweep emitted.
// Compaction: the pairs that were real contacts before the rebuild go to the front of the new container,
// in emission order (the role of ContactLoop's reorderContacts, ContactLoop.cpp:75-91), so that the real
// contacts the contact pass and the force gather touch every step are dense in every per-contact array.
// Pass 1 finds each new pair's old index (or none) and flags the real ones; after a scan of the flags,
// pass 2 writes each contact at its place: real ones at their rank, the others after them in order.
__global__ void k_part_flag(Contacts neu, long long nNew, Contacts old, Csr oldCsr, unsigned long long* tmpIds,
                            unsigned* tmpJ, unsigned* flag, int4* tmpDist) {
  chainWait(false);
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nNew) return;
  const int2 id = neu.ids[c];
  tmpIds[c] = ((unsigned long long)(unsigned)id.y << 32) | (unsigned)id.x;
  if (tmpDist) tmpDist[c] = neu.cdist[c];
  const long long j = csrFind(oldCsr, id.x, id.y);
  unsigned jj = 0xffffffffu, f = 0;
  if (j >= 0) {
    const uint8_t os = old.state[j] & CS_MASK;
    if (os != CS_DEAD) { jj = (unsigned)j; f = (os == CS_REAL) ? 1u : 0u; }
  }
  tmpJ[c] = jj;
  flag[c] = f;
}
__global__ void k_carry_compact(Particles p, Contacts neu, long long nNew, Contacts old, const unsigned long long* tmpIds,
                                const unsigned* tmpJ, const unsigned* scan, const int4* tmpDist, long long step, int nHist,
                                RowCount R, const DeviceStatus* st) {
  chainWait(false);
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nNew || st->scanFailed) return;
  const unsigned before = scan[c];
  const bool wasReal = scan[c + 1] != before;
  const long long d = wasReal ? (long long)before : (long long)scan[nNew] + (c - (long long)before);
  const unsigned long long t = tmpIds[c];
  const int2 id = make_int2((int)(unsigned)(t & 0xffffffffu), (int)(unsigned)(t >> 32));
  const unsigned jj = tmpJ[c];
  if (jj == 0xffffffffu) {
    const uint8_t sb = pairShapeBits(p.meta[id.x].x & 15, p.meta[id.y].x & 15);
    neu.ids[d] = id;
    if (neu.cdist) neu.cdist[d] = tmpDist[c];
    neu.state[d] = CS_POTENTIAL | sb;
    neu.step0[d] = (int)step;
    if (neu.lam) neu.lam[d] = __longlong_as_double(0x7ff8000000000000ll);
    neu.slot[d] = make_int2(takePlace(R, id.x, id.y, maybeLarge(sb)), takePlace(R, id.y, id.x, maybeLarge(sb)));
    return;
  }
  const long long j = jj;
  if (neu.lam && old.lam) neu.lam[d] = old.lam[j];
  else if (neu.lam) neu.lam[d] = __longlong_as_double(0x7ff8000000000000ll);
  const uint8_t sh = old.state[j] & CS_SHAPES;
  const int2 oid = old.ids[j];
  neu.ids[d] = oid;  // keep the stored orientation (and, periodic, the stored cellDist)
  neu.slot[d] = make_int2(takePlace(R, oid.x, oid.y, maybeLarge(sh)), takePlace(R, oid.y, oid.x, maybeLarge(sh)));
  if (neu.cdist) neu.cdist[d] = old.cdist ? old.cdist[j] : tmpDist[c];
  neu.state[d] = (wasReal ? CS_REAL : CS_POTENTIAL) | sh;
  neu.step0[d] = old.step0[j];
  if (wasReal) {
    for (int h = 0; h < nHist; h++) neu.hist[h][d] = old.hist[h][j];
    neu.tanPhi[d] = old.tanPhi[j];
  }
}

// ------------------------------------------------------------------------------------ CSR
// places in the rows of an uploaded container's contacts (a rebuild takes them in k_carry_compact)
__global__ void k_csr_places(Contacts c, long long nc, RowCount R) {
  chainWait(false);
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nc) return;
  const int2 id = c.ids[e];
  const bool big = maybeLarge(c.state[e]);
  c.slot[e] = make_int2(takePlace(R, id.x, id.y, big), takePlace(R, id.y, id.x, big));
}
// the ranges of one large body: counts to starts within its row (one block a body); the row's length to cnt
__global__ void __launch_bounds__(256) k_csr_large(const int* large, RowCount R) {
  chainWait(false);
  __shared__ unsigned warpSum[8];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  unsigned* sub = R.sub + (long long)blockIdx.x * R.V;
  unsigned carry = 0;
  for (int base = 0; base < R.V; base += 256) {
    const unsigned v = base + t < R.V ? sub[base + t] : 0;
    unsigned inc = v;
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += u;
    }
    if (lane == 31) warpSum[warp] = inc;
    __syncthreads();
    unsigned before = 0, total = 0;
    for (int w = 0; w < 8; w++) {
      if (w < warp) before += warpSum[w];
      total += warpSum[w];
    }
    if (base + t < R.V) sub[base + t] = carry + before + inc - v;
    carry += total;
    __syncthreads();
  }
  if (t == 0) R.cnt[large[blockIdx.x]] = carry;
}
// the entries at their places: (partner, contact | isB << 31)
__global__ void k_csr_fill(Contacts c, long long nc, RowCount R, unsigned long long* tmp, const DeviceStatus* st) {
  chainWait(false);
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nc || st->scanFailed) return;
  const int2 id = c.ids[e], place = c.slot[e];
  const bool big = maybeLarge(c.state[e]);
  const int kA = rangeOf(R, id.x, id.y, big), kB = rangeOf(R, id.y, id.x, big);
  tmp[R.cnt[id.x] + (kA < 0 ? 0u : R.sub[kA]) + place.x] = ((unsigned long long)(unsigned)id.y << 32) | (unsigned)e;
  tmp[R.cnt[id.y] + (kB < 0 ? 0u : R.sub[kB]) + place.y] = ((unsigned long long)(unsigned)id.x << 32) | ((unsigned)e | 0x80000000u);
}
// Each entry's final position: the start of its row (or range) plus the number of smaller entries in it.  Writes
// the row's contacts and partners in order, the contact's two entry positions (where the contact pass writes its
// shares) and their positions in the rows (which bit of the row's mask it sets).  Threads follow the entries of tmp,
// so the threads of a warp read the same few rows from L1.
__global__ void k_csr_rank(Contacts c, long long ne, RowCount R, const unsigned long long* tmp, unsigned* ent,
                           unsigned* partner, const DeviceStatus* st) {
  chainWait(false);
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne || st->scanFailed) return;
  const unsigned long long v = tmp[e];
  const unsigned val = (unsigned)v, ci = val & 0x7fffffffu;
  const bool isB = (val >> 31) != 0;
  const int2 id = c.ids[ci];
  const int row = isB ? id.y : id.x, other = isB ? id.x : id.y;
  const unsigned row0 = R.cnt[row], row1 = R.cnt[row + 1];
  unsigned beg = row0, end = row1;
  const int k = rangeOf(R, row, other, maybeLarge(c.state[ci]));
  if (k >= 0) {
    beg = row0 + R.sub[k];
    if ((k + 1) % R.V != 0) end = row0 + R.sub[k + 1];
  }
  unsigned pos = beg;
  for (unsigned q = beg; q < end; q++) pos += tmp[q] < v ? 1u : 0u;
  ent[pos] = val;
  partner[pos] = (unsigned)other;
  const unsigned in = pos - row0;
  const unsigned char bit = (unsigned char)(in < 31 ? in : 31);
  if (isB) { c.slot[ci].y = (int)pos; c.rowBit[ci].y = bit; }
  else { c.slot[ci].x = (int)pos; c.rowBit[ci].x = bit; }
}

// ------------------------------------------------------------------------------------ periodic grid
// Each box's centre wrapped into the cell, in FP32 with its half-widths (pci, phi, by particle id), the number of
// periods taken off per axis with the mask (wrap), its grid cell and its place in the cell's bucket.  The candidate
// loop rejects with the FP32 copies the pairs whose minimum-image centre distance exceeds the sum of the
// half-widths by more than the rounding of these copies on some axis: such boxes are disjoint on that axis for
// every period shift, so spatialOverlapPeri rejects them too.  Boxes wider than a quarter of the cell skip
// the filter (there the exact test may find an ambiguous contact, which is an error to report).
__global__ void k_keys_peri(StepParams P, Particles p, const int* small, int nSmall, const PeriGrid* g, unsigned* keys,
                            unsigned* place, unsigned* count, float4* pci, float4* phi, int4* wrap) {
  chainWait(false);
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nSmall) return;
  const PeriGrid G = *g;
  const int i = small[k];
  const double4_32a mn = p.bbmin[i], mx = p.bbmax[i];
  const double lo[3] = {mn.x, mn.y, mn.z}, hi[3] = {mx.x, mx.y, mx.z};
  float c[3], h[3];
  int f[3], cell[3];
  bool wide = false;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double L = P.csize[a];
    const double ctr = .5 * (lo[a] + hi[a]), half = .5 * (hi[a] - lo[a]);
    // a product with the rounded 1 / L may put a centre at a period's edge into the next period: w and the count
    // of periods agree with each other, which is all that is used
    const double per = floor(ctr * G.invL[a]);
    const double w = ctr - per * L;
    c[a] = (float)w;
    h[a] = (float)half;
    // far out (also infinite and NaN): the exact test decides
    wide |= !(half < .25 * L) || !(fabs(per) < WDEM_PERI_PERIODS);
    f[a] = wide ? 0 : (int)per;
    cell[a] = (int)fmin(fmax(floor(w * G.invCw[a]), 0.0), (double)(G.nc[a] - 1));
  }
  pci[i] = make_float4(c[0], c[1], c[2], 0.f);
  phi[i] = make_float4(h[0], h[1], h[2], wide ? 1.f : 0.f);
  wrap[i] = make_int4(f[0], f[1], f[2], p.meta[i].z);
  const unsigned key = ((unsigned)cell[2] * G.nc[1] + cell[1]) * G.nc[0] + cell[0];
  keys[k] = key;
  place[k] = atomicAdd(&count[key], 1u);
}

// the bodies in cell order: key, and the FP32 copies with the id in the centre's fourth word
__global__ void k_bucket_rank_peri(int nSmall, const unsigned long long* tmp, const unsigned* start, unsigned* keys,
                                   const float4* pci, const float4* phi, float4* pc, float4* ph, const DeviceStatus* st) {
  chainWait(false);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nSmall || st->scanFailed) return;
  const unsigned long long v = tmp[e];
  const unsigned key = (unsigned)(v >> 32);
  const int i = (int)(unsigned)v;
  float4 c = pci[i];
  const float4 h = phi[i];
  const unsigned s = rankInBucket(tmp, v, start[key], start[key + 1]);
  keys[s] = key;
  c.w = __int_as_float(i);
  pc[s] = c;
  ph[s] = h;
}

// Candidate pass: thread q takes the q-th box in cell order and runs the FP32 filter against the boxes after it in
// its cell and those of the 13 cells ahead of it (wrapped), so that every pair of cells is seen once; a cell with
// fewer than 3 cells along some axis meets the same neighbour on both sides, and there the boxes of all (different)
// neighbouring cells with a larger particle id are tested.  It counts (WRITE false) or writes (WRITE true, at its
// scanned offset) the survivors; the counting pass keeps each thread's first SWEEP_BUF and the writing pass copies
// them, walking again only for threads with more (two full walks of all 27 cells took 2 x 280 us at 400k bodies).
// The exact test runs in a separate dense pass (k_peri_exact): inside this loop the survivors of
// one warp's 32 boxes differ per lane, and the FP64 test would run with a few lanes at a time.
struct CandArgs {
  const unsigned* keys;
  const float4 *pc, *ph;
  const unsigned* start;
  unsigned* buf;  // SWEEP_BUF partners per thread (thread minor), or null
  int nSmall;
};
template <bool WRITE>
__global__ void __launch_bounds__(128) k_peri_cand(StepParams P, CandArgs A, const PeriGrid* g, unsigned* counts, int2* cand,
                                                   long long cap, const DeviceStatus* st) {
  chainWait(false);
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q > A.nSmall || st->scanFailed) return;
  if (q == A.nSmall) { if (!WRITE) counts[q] = 0; return; }
  const float4 c1 = A.pc[q];
  const int i = __float_as_int(c1.w);
  unsigned cnt = 0;
  const unsigned long long base = WRITE ? counts[q] : 0;
  if (WRITE && A.buf) {
    const unsigned found = counts[q + 1] - counts[q];
    if (found <= (unsigned)SWEEP_BUF) {
      for (unsigned k = 0; k < found; k++) {
        const int j = (int)A.buf[(long long)k * A.nSmall + q];
        if (base + k < (unsigned long long)cap) cand[base + k] = make_int2(min(i, j), max(i, j));
      }
      return;
    }
  }
  const float4 h1 = A.ph[q];
  const PeriGrid G = *g;
  const float L0 = (float)P.csize[0], L1 = (float)P.csize[1], L2 = (float)P.csize[2];
  const float iL0 = 1.f / L0, iL1 = 1.f / L1, iL2 = 1.f / L2;
  const int key0 = (int)A.keys[q];
  int c[3];
  c[0] = key0 % G.nc[0];
  c[1] = (key0 / G.nc[0]) % G.nc[1];
  c[2] = key0 / (G.nc[0] * G.nc[1]);
  auto walk = [&](int beg, int end, bool byId) {
    for (int q2 = beg; q2 < end; q2++) {
      const float4 c2 = A.pc[q2];
      const int j = __float_as_int(c2.w);
      if (byId && j <= i) continue;
      const float4 h2 = A.ph[q2];
      if (h1.w == 0.f && h2.w == 0.f &&
          (periFar(c1.x, h1.x, c2.x, h2.x, L0, iL0) || periFar(c1.y, h1.y, c2.y, h2.y, L1, iL1) ||
           periFar(c1.z, h1.z, c2.z, h2.z, L2, iL2)))
        continue;
      if (WRITE) {
        const unsigned long long o = base + cnt;
        if (o < (unsigned long long)cap) cand[o] = make_int2(min(i, j), max(i, j));
      } else if (A.buf && cnt < (unsigned)SWEEP_BUF) {
        A.buf[(long long)cnt * A.nSmall + q] = (unsigned)j;
      }
      cnt++;
    }
  };
  if (G.nc[0] >= 3 && G.nc[1] >= 3 && G.nc[2] >= 3) {
    const int xm = c[0] > 0 ? c[0] - 1 : G.nc[0] - 1, xp = c[0] + 1 < G.nc[0] ? c[0] + 1 : 0;
    const int ym = c[1] > 0 ? c[1] - 1 : G.nc[1] - 1, yp = c[1] + 1 < G.nc[1] ? c[1] + 1 : 0;
    const int zp = c[2] + 1 < G.nc[2] ? c[2] + 1 : 0;
    // the rest of the own cell, and the cell ahead in x: one range unless that cell wraps
    const int row0 = key0 - c[0];
    if (xp > c[0]) walk(q + 1, (int)A.start[row0 + xp + 1], false);
    else {
      walk(q + 1, (int)A.start[key0 + 1], false);
      walk((int)A.start[row0 + xp], (int)A.start[row0 + xp + 1], false);
    }
    // four whole rows of three cells: (y+1, z) and (y-1 .. y+1, z+1)
    for (int r = 0; r < 4; r++) {
      const int y = r == 0 || r == 3 ? yp : (r == 1 ? ym : c[1]), z = r == 0 ? c[2] : zp;
      const int row = (z * G.nc[1] + y) * G.nc[0];
      if (xm < c[0] && xp > c[0]) walk((int)A.start[row + xm], (int)A.start[row + xp + 1], false);
      else {
        walk((int)A.start[row + xm], (int)A.start[row + xm + 1], false);
        walk((int)A.start[row + c[0]], (int)A.start[row + c[0] + 1], false);
        walk((int)A.start[row + xp], (int)A.start[row + xp + 1], false);
      }
    }
  } else {
    // neighbouring cells per axis, each index once (axes of one cell have one)
    int nbr[3][3], nn[3];
    for (int a = 0; a < 3; a++) {
      nn[a] = 0;
      for (int d = -1; d <= 1; d++) {
        const int v = ((c[a] + d) % G.nc[a] + G.nc[a]) % G.nc[a];
        bool dup = false;
        for (int b = 0; b < nn[a]; b++) dup |= (nbr[a][b] == v);
        if (!dup) nbr[a][nn[a]++] = v;
      }
    }
    for (int az = 0; az < nn[2]; az++)
      for (int ay = 0; ay < nn[1]; ay++)
        for (int ax = 0; ax < nn[0]; ax++) {
          const int key = (nbr[2][az] * G.nc[1] + nbr[1][ay]) * G.nc[0] + nbr[0][ax];
          walk((int)A.start[key], (int)A.start[key + 1], true);
        }
  }
  if (!WRITE) counts[q] = cnt;
}

// Exact pass, one thread per candidate: spatialOverlapPeri and Collider::mayCollide.  Boxes that overlap on every
// axis by more than the FP32 margin for the nearest image (both narrow: no ambiguity) overlap in the reference's
// test too, whose period is then the one of that image, counted from the wrapped centres; nearly all candidates
// end there.  The rest (within the margin, or wide) take the reference's FP64 operations, 12 divisions a pair: with
// those for every candidate this pass took 486 us for the 1.6 M pairs of 400k bodies.
__global__ void k_peri_exact(StepParams P, Particles p, const int2* cand, long long nc, const float4* pci, const float4* phi,
                             const int4* wrap, unsigned* flag, int4* per, DeviceStatus* st) {
  chainWait(false);
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nc) return;
  const int2 ij = cand[k];
  const float4 c1 = pci[ij.x], h1 = phi[ij.x], c2 = pci[ij.y], h2 = phi[ij.y];
  const int4 w1 = wrap[ij.x], w2 = wrap[ij.y];
  const float L0 = (float)P.csize[0], L1 = (float)P.csize[1], L2 = (float)P.csize[2];
  const float iL0 = 1.f / L0, iL1 = 1.f / L1, iL2 = 1.f / L2;
  int4 pr = make_int4(0, 0, 0, 0);
  bool ok;
  if (h1.w == 0.f && h2.w == 0.f && periNear(c1.x, h1.x, c2.x, h2.x, L0, iL0) && periNear(c1.y, h1.y, c2.y, h2.y, L1, iL1) &&
      periNear(c1.z, h1.z, c2.z, h2.z, L2, iL2)) {
    ok = true;
    pr = make_int4(w1.x - w2.x - (int)rintf((c2.x - c1.x) * iL0), w1.y - w2.y - (int)rintf((c2.y - c1.y) * iL1),
                   w1.z - w2.z - (int)rintf((c2.z - c1.z) * iL2), 0);
  } else {
    bool amb = false;
    ok = overlapPeri(p.bbmin[ij.x], p.bbmax[ij.x], p.bbmin[ij.y], p.bbmax[ij.y], P.csize, pr, amb);
    if (amb) { if (atomicCAS(&st->code, 0, WDEM_ERR_TOO_BIG) == 0) st->detail = ij.x; ok = false; }
  }
  if (ok) ok = mayCollide((unsigned)w1.w, (unsigned)w2.w, P.loneMask);
  flag[k] = ok ? 1u : 0u;
  per[k] = pr;
}

// the accepted candidates, in candidate order, with their cellDist
__global__ void k_peri_emit(const int2* cand, const int4* per, const unsigned* flagScan, long long nc, int2* out,
                            int4* outDist, long long cap) {
  chainWait(false);
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nc || flagScan[k + 1] == flagScan[k]) return;
  const long long o = flagScan[k];
  if (o < cap) { out[o] = cand[k]; outDist[o] = per[k]; }
}

// ------------------------------------------------------------------------------------ stress
// ContactLoop stress (ContactLoop.cpp:218-229): F (global, on pA) x branch (pB image - pA) per real
// contact; the nine components are summed by the deterministic energy reduction.
__global__ void k_stress_terms(StepParams P, Particles p, Contacts c, long long nc, double* terms) {
  chainWait(false);
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if ((c.state[i] & CS_MASK) == CS_REAL) {
    const int2 id = c.ids[i];
    d3 branch = xyz(p.posr[id.y]) - xyz(p.posr[id.x]);
    if (P.periodic) {
      const int4 cd = c.cdist[i];
      branch = branch + mvec(P.hS, mk((double)cd.x, (double)cd.y, (double)cd.z));
    }
    const double4_32a f4 = c.out[OUT_RECORDS * (long long)c.slot[i].x + OUT_F];  // pA's entry: the force on pA
    const double F[3] = {f4.x, f4.y, f4.z};
    const double b[3] = {branch.x, branch.y, branch.z};
    for (int r = 0; r < 3; r++) for (int q = 0; q < 3; q++) v[3 * r + q] = F[r] * b[q];
  }
  for (int q = 0; q < 9; q++) terms[(long long)q * nc + i] = v[q];
}

}  // namespace wdem

// ============================================================================== host orchestration
namespace wdem {


static int bitsFor(unsigned long long v) { int b = 0; while ((1ull << b) < v) b++; return b < 1 ? 1 : b; }
// buckets of the sort: two per body (half a body each on average), at most what cellStart holds
static int maxBuckets(const ColliderScratch& cs, int nSmall) {
  return (int)std::min<long long>(cs.maxCols, std::max<long long>(1024, 2ll * nSmall));
}
// the sweep grid's column cap and the quantisation bits of its keys: column bits + qbits fit 32 bits, with at
// least 12 quantisation bits (SWEEP_MAX_COLS) and at most 24
static int sweepCols(const ColliderScratch& cs, int nSmall) { return std::min(maxBuckets(cs, nSmall), SWEEP_MAX_COLS); }
static int sweepQbits(const ColliderScratch& cs, int nSmall) {
  return std::min(24, 32 - bitsFor((unsigned long long)sweepCols(cs, nSmall) + 1));
}
// the sort's arrays in the collider's scratch: keys and places by body, (key, id) by bucket, keys and ids in order
struct SortArrays {
  unsigned *keyIn, *place, *key, *id, *start;
  unsigned long long* tmp;
};
static SortArrays sortArrays(const ColliderScratch& cs) {
  SortArrays a;
  a.keyIn = cs.vals;
  a.place = cs.valsAlt;
  a.tmp = cs.keysAlt;
  a.key = reinterpret_cast<unsigned*>(cs.keys);
  a.id = a.key + cs.sortCap;
  a.start = cs.cellStart;
  return a;
}
static void launchExtents(cudaStream_t s, const StepParams& P, Particles p, const int* small, int nSmall,
                          ColliderScratch& cs, const GridArgs& A) {
  unsigned long long* ext = (unsigned long long*)cs.temp;
  cudaMemsetAsync(ext, 0xff, EXT_WORDS * sizeof(unsigned long long), s);
  const unsigned blocks = (unsigned)std::max(1, std::min((nSmall + EXT_T - 1) / EXT_T, 2 * 152));
  launchChained(k_extents, blocks, EXT_T, s, P, p, small, nSmall, ext, A);
}

// The collider sub-steps are called from wdem_api.cu through these thin wrappers.
void col_extents_and_grid(cudaStream_t s, Particles p, const int* small, int nSmall, ColliderScratch& cs) {
  GridArgs A{sweepCols(cs, nSmall), maxBuckets(cs, nSmall), sweepQbits(cs, nSmall), cs.grid, nullptr, cs.st};
  launchExtents(s, StepParams{}, p, small, nSmall, cs, A);
}

void col_sort(cudaStream_t s, Particles p, const int* small, int nSmall, ColliderScratch& cs) {
  const SortArrays a = sortArrays(cs);
  const int nb = maxBuckets(cs, nSmall);
  cudaMemsetAsync(a.start, 0, ((size_t)nb + 1) * sizeof(unsigned), s);
  if (nSmall <= 0) return;
  const unsigned blocks = (unsigned)((nSmall + 255) / 256);
  launchChained(k_make_keys, blocks, 256, s, p, small, nSmall, cs.grid, a.keyIn, a.place, a.start);
  exclusive_scan_u32(s, a.start, nb, cs);
  launchChained(k_bucket_place, blocks, 256, s, small, nSmall, a.keyIn, a.place, a.start, cs.grid, a.tmp, cs.st);
  launchChained(k_bucket_rank<false>, blocks, 256, s, p, nSmall, a.tmp, a.start, cs.grid, a.key, a.id, cs.srec, cs.st);
}

void col_sort_merge(cudaStream_t s, Particles p, int nSmall, ColliderScratch& cs) {
  const SortArrays a = sortArrays(cs);
  const unsigned blocks = (unsigned)((nSmall + 255) / 256);
  // the runs alternate between tmp and the array that k_bucket_rank writes, and end in tmp
  unsigned long long* buf[2] = {a.tmp, cs.keys};
  int passes = 0;
  while (((long long)SORT_TILE << passes) < nSmall) passes++;
  int at = passes & 1;
  launchChained(k_tile_sort, (unsigned)((nSmall + SORT_TILE - 1) / SORT_TILE), SORT_T, s, a.tmp, buf[at], nSmall);
  for (int k = 0; k < passes; k++, at ^= 1) launchChained(k_merge_runs, blocks, 256, s, buf[at], buf[at ^ 1], nSmall, SORT_TILE << k);
  cudaMemsetAsync(&cs.st->longBucket, 0, sizeof(int), s);
  launchChained(k_bucket_rank<true>, blocks, 256, s, p, nSmall, a.tmp, a.start, cs.grid, a.key, a.id, cs.srec, cs.st);
}

void col_sweep(cudaStream_t s, Particles p, int nSmall, unsigned loneMask, ColliderScratch& cs, int2* out, long long cap,
               bool write) {
  SweepArgs A;
  A.rec = cs.srec;
  const SortArrays a = sortArrays(cs);
  A.keys = a.key; A.vals = a.id; A.start = a.start; A.large = cs.large; A.nLarge = cs.nLarge;
  A.nSmall = nSmall; A.loneMask = loneMask;
  A.sceneWall = cs.nScenes > 1 ? cs.sceneWall : nullptr;
  A.buf = cs.sweepBufCap >= sweepThreads(nSmall, cs.nLarge) ? cs.sweepBuf : nullptr;
  const int threads = sweepThreads(nSmall, cs.nLarge);
  if (write) launchChained(k_sweep<true>, (threads + 127) / 128, 128, s, p, A, cs.grid, cs.counts, out, cap, cs.st);
  else launchChained(k_sweep<false>, (threads + 127) / 128, 128, s, p, A, cs.grid, cs.counts, out, cap, cs.st);
}

void col_retain_write_dist(cudaStream_t s, Contacts old, long long nOld, ColliderScratch& cs, int4* out, long long base,
                           long long cap) {
  if (nOld > 0) launchChained(k_retain_write_dist, (unsigned)((nOld + 255) / 256), 256, s, old, nOld, cs.retainFlag, out, base, cap);
}

void col_retain_flags(cudaStream_t s, const StepParams& P, Particles p, Contacts old, long long nOld, ColliderScratch& cs) {
  if (nOld > 0) launchChained(k_retain_flag, (unsigned)((nOld + 255) / 256), 256, s, P, p, old, nOld, cs.retainFlag, cs.periCi, cs.periHi);
  exclusive_scan_u32(s, cs.retainFlag, nOld, cs, TOTAL_RETAINED);
}
void col_retain_write(cudaStream_t s, Contacts old, long long nOld, ColliderScratch& cs, int2* out, long long base, long long cap) {
  if (nOld > 0) launchChained(k_retain_write, (unsigned)((nOld + 255) / 256), 256, s, old, nOld, cs.retainFlag, out, base, cap);
}

// periodic pair search, part 1: grid, cell sort, FP32 candidates counted (write false; counts
// scanned, total at counts[nSmall + 1]) or written (write true)
void col_periodic_cand(cudaStream_t s, const StepParams& P, Particles p, const int* small, int nSmall,
                       ColliderScratch& cs, bool write) {
  PeriGrid* g = (PeriGrid*)((char*)cs.temp + 256);
  const SortArrays a = sortArrays(cs);
  const int threads = nSmall + 1;
  CandArgs A{a.key, cs.periC, cs.periH, a.start, cs.sweepBufCap >= nSmall ? cs.sweepBuf : nullptr, nSmall};
  if (!write) {
    const int nb = maxBuckets(cs, nSmall);
    GridArgs GA{0, nb, 0, nullptr, g, cs.st};
    launchExtents(s, P, p, small, nSmall, cs, GA);
    cudaMemsetAsync(a.start, 0, ((size_t)nb + 1) * sizeof(unsigned), s);
    if (nSmall > 0) {
      const unsigned blocks = (unsigned)((nSmall + 255) / 256);
      launchChained(k_keys_peri, blocks, 256, s, P, p, small, nSmall, g, a.keyIn, a.place, a.start, cs.periCi, cs.periHi, cs.periWrap);
      exclusive_scan_u32(s, a.start, nb, cs);
      launchChained(k_bucket_place, blocks, 256, s, small, nSmall, a.keyIn, a.place, a.start, nullptr, a.tmp, cs.st);
      launchChained(k_bucket_rank_peri, blocks, 256, s, nSmall, a.tmp, a.start, a.key, cs.periCi, cs.periHi, cs.periC, cs.periH, cs.st);
    }
    launchChained(k_peri_cand<false>, (threads + 127) / 128, 128, s, P, A, g, cs.counts, nullptr, 0, cs.st);
    exclusive_scan_u32(s, cs.counts, nSmall + 1, cs, TOTAL_PAIRS);
  } else {
    launchChained(k_peri_cand<true>, (threads + 127) / 128, 128, s, P, A, g, cs.counts, cs.cand, cs.candCap, cs.st);
  }
}

// part 2: the exact test of nCand candidates; flags scanned, accepted total at candFlag[nCand]
void col_periodic_exact(cudaStream_t s, const StepParams& P, Particles p, ColliderScratch& cs, long long nCand,
                        DeviceStatus* st) {
  if (nCand > 0)
    launchChained(k_peri_exact, (unsigned)((nCand + 255) / 256), 256, s, P, p, cs.cand, nCand, cs.periCi, cs.periHi,
                  cs.periWrap, cs.candFlag, cs.candPer, st);
  exclusive_scan_u32(s, cs.candFlag, nCand, cs, TOTAL_PAIRS);
}

// part 3: accepted pairs and their cellDist into the new container
void col_periodic_emit(cudaStream_t s, ColliderScratch& cs, long long nCand, int2* out, int4* outDist, long long cap) {
  if (nCand > 0)
    launchChained(k_peri_emit, (unsigned)((nCand + 255) / 256), 256, s, cs.cand, cs.candPer, cs.candFlag, nCand, out,
                  outDist, cap);
}

void launch_stress(cudaStream_t s, const StepParams& P, Particles p, Contacts c, long long nc, double* scratch9,
                   double* partials, double* out9, DeviceStatus* st) {
  if (nc > 0) launchChained(k_stress_terms, (unsigned)((nc + 255) / 256), 256, s, P, p, c, nc, scratch9);
  SumSet S{};
  for (int q = 0; q < 9; q++) {
    S.x[q] = scratch9 + (long long)q * nc;
    S.n[q] = nc;
    S.acc[q] = out9 + q;
  }
  S.reset = (1 << 9) - 1;
  launch_sums(s, P, S, 0, 9, partials, st);
}

static RowCount rowCount(int n, const Csr& csr, const ColliderScratch& cs) {
  RowCount R;
  R.cnt = reinterpret_cast<unsigned*>(csr.rowptr);
  R.sub = cs.rowSub;
  R.largeIdx = cs.largeIdx;
  largeRanges(n, cs.nLarge, R.V, R.S);
  return R;
}
static void clearRows(cudaStream_t s, int n, const RowCount& R, const ColliderScratch& cs) {
  cudaMemsetAsync(R.cnt, 0, (size_t)n * sizeof(unsigned), s);
  if (cs.nLarge > 0) cudaMemsetAsync(R.sub, 0, (size_t)cs.nLarge * R.V * sizeof(unsigned), s);
}

void col_carry_compact(cudaStream_t s, Particles p, Contacts neu, long long nNew, Contacts old, Csr csr, int nRowsOld,
                       int n, long long step, int nHist, ColliderScratch& cs) {
  Csr oldCsr = csr;
  oldCsr.n = nRowsOld;
  const RowCount R = rowCount(n, csr, cs);
  if (nNew <= 0) {
    clearRows(s, n, R, cs);
    return;
  }
  unsigned long long* tmpIds = cs.keys;
  unsigned* tmpJ = cs.vals;
  unsigned* flag = cs.valsAlt;
  int4* tmpDist = neu.cdist ? reinterpret_cast<int4*>(cs.keysAlt) : nullptr;
  const unsigned blocks = (unsigned)((nNew + 255) / 256);
  launchChained(k_part_flag, blocks, 256, s, neu, nNew, old, oldCsr, tmpIds, tmpJ, flag, tmpDist);
  exclusive_scan_u32(s, flag, nNew, cs);
  clearRows(s, n, R, cs);  // the old rows have been read
  launchChained(k_carry_compact, blocks, 256, s, p, neu, nNew, old, tmpIds, tmpJ, flag, tmpDist, step, nHist, R, cs.st);
}

// The CSR of the container.  placed: its contacts have taken their places (k_carry_compact).
void col_csr(cudaStream_t s, Contacts c, long long nc, int n, Csr& csr, ColliderScratch& cs, bool placed) {
  const RowCount R = rowCount(n, csr, cs);
  const unsigned blocks = (unsigned)((nc + 255) / 256);
  if (!placed) {
    clearRows(s, n, R, cs);
    if (nc > 0) launchChained(k_csr_places, blocks, 256, s, c, nc, R);
  }
  csr.n = n;
  if (cs.nLarge > 0) launchChained(k_csr_large, (unsigned)cs.nLarge, 256, s, cs.large, R);
  exclusive_scan_u32(s, R.cnt, n, cs);
  if (nc <= 0) return;
  unsigned long long* tmp = cs.keysAlt;
  launchChained(k_csr_fill, blocks, 256, s, c, nc, R, tmp, cs.st);
  launchChained(k_csr_rank, (unsigned)((2 * nc + 255) / 256), 256, s, c, 2 * nc, R, tmp, csr.ent, csr.partner, cs.st);
}

}  // namespace wdem
