// particles.cu -- particle <-> lattice kernels (FP64, compiled with -fmad=false).
//
// Map (replaces ExchangeParticleData::setParticlesOnLattice and
// calcSolidFraction, src/LBM_PSM_exchangeParticleData.cpp:24-169, with
// LBMPSMLattice::setParticleOnLattice / setToZero,
// src/LBM_PSM_lattice.cpp:257-324).  The reference walks the particle images
// in array order and, for each, the nodes of its bounding box, updating a
// persistent two-slot table per node; the final table depends on that order.
// Here every node applies, in its own thread, the updates of the images whose
// boxes contain it in ascending image order, which yields the same table
// without atomics on the table:
//   1. img_prep   : per image, box in device coordinates, coarse cells touched
//   2. cell_scan  : offsets of the per-cell image lists
//   3. img_fill   : scatter image ids into the cell lists
//   4. cell_sort  : sort each list ascending (restores image order)
//   5. node_apply : per node, walk its cell's list and apply the 4-way update
// The solid fraction counts the reference's 10^d sub-cell centres; each
// comparison is decided in FP32 when it is far from the threshold (proven
// margins, solid_fraction.cuh) and otherwise evaluated with the reference's
// FP64 expression, so the count is the reference's count.
//
// Reduce (replaces calculateHydrodynamicInteractions,
// src/LBM_PSM_exchangeParticleData.cpp:172-244): the node forces of an image's
// tag summed over the box clamped to interior nodes in a fixed order
// (deterministic run to run).
#include <cooperative_groups.h>

#include <algorithm>

#include "lbmpsm_internal.cuh"
#include "solid_fraction.cuh"

namespace lbmpsm {

// Whether n images are too few to fill the device with one block each.
static bool few_images(int n, int sm_count) { return n < sm_count; }

static __device__ __forceinline__ int clampi(int v, int lo, int hi) {
  return v < lo ? lo : (v > hi ? hi : v);
}

// lattice-local centre on one rank (src/LBM_PSM_exchangeParticleData.cpp:31-37)
static __device__ __forceinline__ double local_centre(double x, double origin, double dx) {
  const double g = (x - origin) / dx;
  return g - ((0 - ((double)0 * 2.0 * (double)1)) - 1);
}

// Box of one image for the force reduction, clamped to interior nodes
// (src/LBM_PSM_exchangeParticleData.cpp:188-195).
static __device__ __forceinline__ void reduce_box_of(const Geom& g, const double xl[3], double r,
                                                     int lo[3], int hi[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    int a = (int)(xl[d] - r) - 2;
    int c = (int)(xl[d] + r) + 2;
    if (d < 2 || g.dim == 3) {
      a = clampi(a, 1, g.L[d] - 1);
      c = clampi(c, 1, g.L[d] - 1);
      if (d == 2) {
        if (a < 0) a = 0;
        if (c < 1) c = 1;
      }
    } else {
      // fmax(fmin(fmax(z, 1), nz - 1), slot) with nz = 1 in 2-D
      a = a < 1 ? 1 : a;
      a = a > g.L[2] - 1 ? g.L[2] - 1 : a;
      a = a < 0 ? 0 : a;
      c = c < 1 ? 1 : c;
      c = c > g.L[2] - 1 ? g.L[2] - 1 : c;
      c = c < 1 ? 1 : c;
    }
    lo[d] = a;
    hi[d] = c;
  }
}

// One thread per image builds its record (the FP64 arithmetic of
// src/LBM_PSM_exchangeParticleData.cpp:31-55), counts the image into the
// cells its box touches, and the warp reserves its images' ranges of
// solid-fraction codes with one atomic.
// Images per block of img_prep (a partial warp): each thread's image record
// is a long FP64 chain, and FP64 runs at 1/64 of the FP32 rate on this GPU,
// so the images are spread over as many multiprocessors as possible.
constexpr int IMG_LANES = 16;
__global__ void img_prep_kernel(MapParams p) {
  constexpr unsigned M = IMG_LANES == 32 ? 0xffffffffu : (1u << IMG_LANES) - 1u;
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool mine = i < p.n;
  int cr[6] = {0, 0, 0, -1, -1, -1};  // clo[3], chi[3]
  unsigned long long vol = 0;
  Img im;
  if (mine) {
    const Geom& g = p.g;
    // every input first, all in flight at once: the arrays may lie in host
    // memory, and behind a store or a division each load waits for the one
    // before it
    im.bidx = p.img_box ? p.img_box[i] : 0;
    const int tag = p.tag[i];
    const double radius = p.radius[i];
    double x[3], v[3], om[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      x[c] = p.x[3 * (size_t)i + c];
      v[c] = p.v[3 * (size_t)i + c];
      om[c] = p.omega[3 * (size_t)i + c];
    }
    const BoxParams& bp = p.box[im.bidx];
    const double origin[3] = {bp.origin[0], bp.origin[1], bp.origin[2]};
    const double Uc = bp.Uc, u_lb = bp.u_lb, tc = bp.tc, dt_d = bp.dt_d;
    im.tag = tag;
    if (p.copy_tag) {  // the caller's arrays, kept for later steps with these images
      const size_t nn = (size_t)p.n;
      p.copy_tag[i] = tag;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        p.copy_xvw[3 * (size_t)i + c] = x[c];
        p.copy_xvw[3 * nn + 3 * (size_t)i + c] = v[c];
        p.copy_xvw[6 * nn + 3 * (size_t)i + c] = om[c];
      }
      p.copy_xvw[9 * nn + i] = radius;
    }
    im.zoff = im.bidx * g.bz;
    const double r = radius / p.dx;
    im.r = r;
    bool valid = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double xl = local_centre(x[d], origin[d], p.dx);
      im.xl[d] = xl;
      int lo = (int)(xl - r) - 2;
      int hi = (int)(xl + r) + 2;
      lo = clampi(lo, 0, g.L[d]);
      hi = clampi(hi, 0, g.L[d]);
      if (d == 2) {  // 2-D keeps its single z layer
        if (lo < 0) lo = 0;
        if (hi < 1) hi = 1;
      }
      // reference halo frame -> device storage
      int slo, shi;
      if (g.off[d] == 1) {
        slo = (lo < 1 ? 1 : lo) - 1;
        shi = (hi > g.L[d] - 1 ? g.L[d] - 1 : hi) - 1;
      } else {
        slo = lo;
        shi = hi;
      }
      const int z0 = d == 2 ? im.zoff : 0;  // boxes of an ensemble stack along z
      im.lo[d] = slo + z0;
      im.hi[d] = shi + z0;
      if (slo >= shi) valid = false;
      im.uT[d] = v[d] / Uc * u_lb;
      im.om[d] = om[d] * tc * dt_d;
      im.uTf[d] = (float)im.uT[d];
      im.omf[d] = (float)im.om[d];
    }
    im.valid = valid;
    const double rP = r + p.sqrt2half;
    const double rM = r - p.sqrt2half;
    im.rP2 = rP * rP;
    im.rM2 = rM * rM;
    im.rSq = r * r;
    im.rP2f = (float)im.rP2;
    im.rM2f = (float)im.rM2;
    im.rSqf = (float)im.rSq;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      split_centre(im.xl[d], im.xi[d], im.xf[d]);
    }
    // the node velocity reduces to uT + 0.0 bit for bit when every omega
    // component is +0.0 and no uT component is -0.0 (signed-zero arithmetic)
    bool plain = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (__double_as_longlong(im.om[d]) != 0ll) plain = false;
      if (__double_as_longlong(im.uT[d]) == (long long)0x8000000000000000ull) plain = false;
    }
    im.has_spin = plain ? 0 : 1;
    reduce_box_of(g, im.xl, r, im.rlo, im.rhi);
    // When no periodic copy of this particle can have an overlapping box
    // (box width below the period on every periodic axis), the nodes of the
    // box that hold its tag after the map all have eps > 0 from this image,
    // hence lie within the early-out radius rP: the reduction then only
    // visits the box part around the sphere (and still checks each tag).
    {
      bool solo = true;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (d >= g.dim) break;
        const int w = ((int)(im.xl[d] + r) + 2) - ((int)(im.xl[d] - r) - 2);
        if (g.per[d] && w >= (d == 2 ? g.bz : g.S[d])) solo = false;
      }
      im.solo = solo ? 1 : 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        im.qlo[d] = im.rlo[d];
        im.qhi[d] = im.rhi[d];
        if (solo && (d < 2 || g.dim == 3)) {
          const int a = (int)floor(im.xl[d] - rP), b = (int)floor(im.xl[d] + rP) + 1;
          im.qlo[d] = max(im.qlo[d], a);
          im.qhi[d] = min(im.qhi[d], b);
        }
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) im.box[d] = valid ? im.hi[d] - im.lo[d] : 0;
    if (valid) {
      vol = (unsigned long long)im.box[0] * im.box[1] * im.box[2];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        im.clo[d] = im.lo[d] / p.cb[d];
        im.chi[d] = (im.hi[d] - 1) / p.cb[d];
        cr[d] = im.clo[d];
        cr[3 + d] = im.chi[d];
      }
    } else {
#pragma unroll
      for (int d = 0; d < 3; ++d) im.clo[d] = 0, im.chi[d] = -1;
    }
  }
  // code ranges: warp prefix of the box volumes, one atomic per warp
  unsigned long long incl = vol;
#pragma unroll
  for (int o = 1; o < IMG_LANES; o <<= 1) {
    const unsigned long long x = __shfl_up_sync(M, incl, o);
    if (lane >= o) incl += x;
  }
  unsigned long long base = 0;
  if (lane == IMG_LANES - 1) base = atomicAdd(&p.pair_total[1], incl);
  base = __shfl_sync(M, base, IMG_LANES - 1);
  if (mine) {
    im.sf_off = (long long)(base + incl - vol);
    p.img[i] = im;
    int4 a = make_int4(0, 0, 0, im.tag), b;
    if (im.valid)
      a = make_int4(im.lo[0] | (im.hi[0] << 16), im.lo[1] | (im.hi[1] << 16),
                    im.lo[2] | (im.hi[2] << 16), im.tag);
    b = make_int4((int)(unsigned)(unsigned long long)im.sf_off,
                  (int)(unsigned)((unsigned long long)im.sf_off >> 32),
                  im.box[0] | (im.box[1] << 16), im.has_spin);
    p.arec[3 * i] = a;
    p.arec[3 * i + 1] = b;
    p.arec[3 * i + 2] = make_int4(__float_as_int(im.uTf[0]), __float_as_int(im.uTf[1]),
                                  __float_as_int(im.uTf[2]), 0);
  }
  // cell counts: each lane walks the cells its image's box touches (integer
  // sums, so the order of the atomics does not matter); one atomic per warp
  // for the pair total
  unsigned long long pairs = 0;
  if (cr[3] >= cr[0] && cr[4] >= cr[1] && cr[5] >= cr[2]) {
    for (int cz = cr[2]; cz <= cr[5]; ++cz)
      for (int cy = cr[1]; cy <= cr[4]; ++cy) {
        int* row = p.cell_count + (cz * p.C[1] + cy) * p.C[0];
        for (int cx = cr[0]; cx <= cr[3]; ++cx) atomicAdd(row + cx, 1);
      }
    pairs = (unsigned long long)(cr[3] - cr[0] + 1) * (unsigned long long)(cr[4] - cr[1] + 1) *
            (unsigned long long)(cr[5] - cr[2] + 1);
  }
#pragma unroll
  for (int o = IMG_LANES / 2; o > 0; o >>= 1) pairs += __shfl_xor_sync(M, pairs, o);
  if (lane == 0 && pairs) atomicAdd(&p.pair_total[0], pairs);
}

// Exclusive scan of the cell counts: one block of 1024 threads walking tiles
// of 8192 counts (8 consecutive per thread, two 16-byte loads), warp shuffles
// within a tile and a running carry between tiles; the offsets go through
// shared memory so that the stores to global memory are coalesced.
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_PER_THREAD = 8;
__global__ void __launch_bounds__(SCAN_THREADS) cell_scan_kernel(const int* __restrict__ count,
                                                                 int* __restrict__ off,
                                                                 int ncells) {
  constexpr int V = SCAN_PER_THREAD;
  constexpr int TILE = V * SCAN_THREADS;
  __shared__ int wsum[SCAN_THREADS / 32];
  __shared__ int carry_s;
  __shared__ int tile[TILE + TILE / 32];  // one pad word per 32: conflict-free strided writes
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) carry_s = 0;
  __syncthreads();
  for (int base = 0; base < ncells; base += TILE) {
    const int i0 = base + V * t;
    int v[V];
    if (i0 + V <= ncells) {  // i0 is a multiple of 8: aligned 16-byte loads
      const int4* c4 = reinterpret_cast<const int4*>(count + i0);
#pragma unroll
      for (int k = 0; k < V / 4; ++k) {
        const int4 w = c4[k];
        v[4 * k] = w.x;
        v[4 * k + 1] = w.y;
        v[4 * k + 2] = w.z;
        v[4 * k + 3] = w.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < V; ++k) v[k] = i0 + k < ncells ? count[i0 + k] : 0;
    }
    int own = 0;
#pragma unroll
    for (int k = 0; k < V; ++k) own += v[k];
    int incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = wsum[lane];
      int wi = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += x;
      }
      wsum[lane] = wi - w;  // exclusive prefix of the warps
    }
    __syncthreads();
    int run = carry_s + wsum[warp] + incl - own;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int j = V * t + k;
      tile[j + (j >> 5)] = run;
      run += v[k];
    }
    __syncthreads();
    if (t == SCAN_THREADS - 1) carry_s = run;
    const int m = min(TILE, ncells - base);
    for (int j = t; j < m; j += SCAN_THREADS) off[base + j] = tile[j + (j >> 5)];
    __syncthreads();
  }
}

// One warp per image: the lanes enter the image into its cells' lists.
__global__ void img_fill_kernel(MapParams p) {
  const int lane = threadIdx.x & 31;
  const int i = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
  if (i >= p.n) return;
  if (p.pair_total[0] > (unsigned long long)p.list_cap ||
      p.pair_total[1] > (unsigned long long)p.sf_cap) {
    if (i == 0 && lane == 0) atomicOr(p.status, STATUS_LIST_OVERFLOW);
    return;
  }
  const Img& im = p.img[i];
  if (!im.valid) return;
  const int nx = im.chi[0] - im.clo[0] + 1, ny = im.chi[1] - im.clo[1] + 1,
            nz = im.chi[2] - im.clo[2] + 1;
  const int ncell = nx * ny * nz;
  for (int t = lane; t < ncell; t += 32) {
    const int cx = im.clo[0] + t % nx, cy = im.clo[1] + (t / nx) % ny, cz = im.clo[2] + t / (nx * ny);
    const int c = (cz * p.C[1] + cy) * p.C[0] + cx;
    const int pos = atomicAdd(&p.cell_fill[c], 1);
    p.list[(long long)p.cell_off[c] + pos] = i;
  }
}

__global__ void cell_sort_kernel(MapParams p, int ncells) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  if (p.pair_total[0] > (unsigned long long)p.list_cap) return;
  const int off = p.cell_off[c];
  int* a = p.list + off;
  const int m = p.cell_count[c];
  for (int k = 1; k < m; ++k) {
    const int v = a[k];
    int j = k - 1;
    while (j >= 0 && a[j] > v) {
      a[j + 1] = a[j];
      --j;
    }
    a[j + 1] = v;
  }
  // the images' table-update records in list order
  for (int k = 0; k < m; ++k) {
    const int ii = a[k];
    int4* r = p.lrec + 3 * ((long long)off + k);
    r[0] = p.arec[3 * ii];
    r[1] = p.arec[3 * ii + 1];
    const int4 u = p.arec[3 * ii + 2];
    r[2] = make_int4(u.x, u.y, u.z, ii);
  }
}

// A shell node (between the early-out radii) whose sub-cells all lie on one
// side of the surface: the count calcSolidFraction's loop would give
// (src/LBM_PSM_exchangeParticleData.cpp:151-165), 10^dim or 0, else -1.
// Every FP64 sub-cell sum (dx_sq[i] + dy_sq[j]) + dz_sq[k] is monotone in
// each term and each term is convex in the sub-cell offset, so the largest
// sum is the far corner's (|d| + 0.45 per axis) and the smallest is at least
// the sum of max(|d| - 0.45, 0)^2.  Decided in FP32 with the margin M that
// bounds the FP32 error of every sub-cell sum of the node (the one the shell
// count uses); undecided nodes stay in the shell.
static __device__ __forceinline__ int corner_count(int dim, float dxf, float dyf, float dzf,
                                                   float rSqf) {
  const float u = 5.9604644775390625e-08f;  // 2^-24
  const float ax = fabsf(dxf), ay = fabsf(dyf), az = dim == 3 ? fabsf(dzf) : 0.0f;
  const float Ea = ax + 2.0f, Eb = ay + 2.0f, Ec = az + 2.0f;
  const float M = 16.0f * u * (Ea * Ea + Eb * Eb + (dim == 3 ? Ec * Ec : 0.0f) + rSqf);
  const float fx = ax + 0.45f, fy = ay + 0.45f, fz = az + 0.45f;
  const float far = fx * fx + fy * fy + (dim == 3 ? fz * fz : 0.0f);
  if (far < rSqf - M) return dim == 3 ? 1000 : 100;
  const float nx = fmaxf(ax - 0.45f, 0.0f), ny = fmaxf(ay - 0.45f, 0.0f),
              nz = fmaxf(az - 0.45f, 0.0f);
  const float near = nx * nx + ny * ny + (dim == 3 ? nz * nz : 0.0f);
  if (near > rSqf + M) return 0;
  return -1;
}

constexpr int SFC_THREADS = 64;   // classification: one block per image
constexpr int SFS_THREADS = 128;  // shell counting: persistent warps

// Phase 1 of the map.  An image's box is walked in groups of x-rows, one warp
// a group.  The warp first sets the group's codes to 0 with coalesced stores;
// then only the nodes of each row that may lie within rP (an FP32 bound
// widened by 0.01 node: a superset of the nodes classify_node does not put
// beyond rP for certain) are classified by the early-out radii of
// calcSolidFraction.  Inside nodes get their code here, and so do shell nodes
// whose sub-cells all lie on one side of the surface; the other shell nodes
// (whose sub-cells must be counted) are queued per warp in shared memory and
// appended to a global list with one atomic per flush.  The rows' segments go
// one per lane, and the warp walks their nodes 32 at a time (consecutive lanes
// on consecutive nodes of a row).
//
// With many images 32 rows a group: one block an image, or, for fewer than four
// images a multiprocessor, as many as keep 16 blocks of two warps on each, up to
// eight (classify_parts; 284 images: 8 us less a step.  About 900 images in three
// blocks each: one workload 5 us a step faster, another 1.3 slower, so one).
// With few images, groups of 8 rows are dealt to SFC_PARTS blocks (one image of
// diameter 16 by one block: 30 us).
constexpr int SFC_QW = 256;  // per-warp queue of shell nodes
constexpr int SFC_PARTS = 16;
static unsigned classify_parts(int n, int sm_count) {
  return n < 4 * sm_count ? (unsigned)std::min(SFC_PARTS / 2, 16 * sm_count / n) : 1u;
}
template <int ROWS>
__global__ void __launch_bounds__(SFC_THREADS) sf_classify_kernel(MapParams p) {
  const Img& im = p.img[blockIdx.x];
  if (!im.valid) return;
  if (p.pair_total[0] > (unsigned long long)p.list_cap ||
      p.pair_total[1] > (unsigned long long)p.sf_cap)
    return;
  constexpr int NW = SFC_THREADS / 32;
  __shared__ int4 q[NW][SFC_QW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Geom& g = p.g;
  const int wx = im.box[0], wy = im.box[1], wz = im.box[2];
  unsigned short* code = p.sfcode + im.sf_off;
  // reference-frame coordinates of the box's first node
  const int h0 = im.lo[0] + g.off[0], h1 = im.lo[1] + g.off[1];
  const int h2 = im.lo[2] - im.zoff + g.off[2];  // z in the box's own frame
  const float rem0 = im.rP2f * 1.0001f + 0.01f;
  const FastDiv fy = make_fastdiv((unsigned)wy);
  int qn = 0;  // entries in this warp's queue (warp-uniform)
  auto flush = [&]() {
    unsigned long long qb = 0;
    if (lane == 0) qb = atomicAdd(&p.pair_total[2], (unsigned long long)qn);
    qb = __shfl_sync(0xffffffffu, qb, 0);
    for (int k = lane; k < qn; k += 32) {
      const unsigned long long pos = qb + k;
      if (pos < (unsigned long long)p.shell_cap)
        p.shell[pos] = q[warp][k];
      else
        atomicOr(p.status, STATUS_LIST_OVERFLOW);
    }
    __syncwarp();
    qn = 0;
  };
  const int R = wy * wz;
  for (int r0 = ((int)blockIdx.y * NW + warp) * ROWS; r0 < R; r0 += (int)gridDim.y * NW * ROWS) {
    const int r = r0 + lane;
    for (int li = r0 * wx + lane; li < min(R, r0 + ROWS) * wx; li += 32) code[li] = 0;
    __syncwarp();  // the zeros land before any code of the group
    int xa = 0, len = 0, by = 0, bz = 0;
    if (lane < ROWS && r < R) {
      bz = (int)fast_div((unsigned)r, fy);
      by = r - bz * wy;
      const float dy = small_int_to_float(h1 + by - im.xi[1]) - im.xf[1];
      const float dz = small_int_to_float(h2 + bz - im.xi[2]) - im.xf[2];
      const float rem = rem0 - dy * dy - dz * dz;
      if (rem >= 0.0f) {
        const float h = sqrtf(rem) + 0.01f;
        xa = max(0, im.xi[0] + (int)ceilf(im.xf[0] - h) - h0);
        const int xb = min(wx, im.xi[0] + (int)floorf(im.xf[0] + h) + 1 - h0);
        len = max(xb - xa, 0);
      }
    }
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const int excl = incl - len;
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int base = 0; base < total; base += 32) {
      const int t = base + lane;
      // the row holding node t: the last lane whose offset is <= t
      int l = 0;
#pragma unroll
      for (int st = 16; st >= 1; st >>= 1)
        if (__shfl_sync(0xffffffffu, excl, l + st) <= t) l += st;
      const int ax = __shfl_sync(0xffffffffu, xa, l) + t - __shfl_sync(0xffffffffu, excl, l);
      const int ay = __shfl_sync(0xffffffffu, by, l), az = __shfl_sync(0xffffffffu, bz, l);
      const int hx = h0 + ax, hy = h1 + ay, hz = h2 + az;
      const int li = (az * wy + ay) * wx + ax;
      int c = 0;
      if (t < total) {
        float dxf, dyf, dzf;
        c = classify_node(hx, hy, hz, im, dxf, dyf, dzf);
        if (c < 0) c = corner_count(g.dim, dxf, dyf, dzf, im.rSqf);
        if (c > 0) code[li] = (unsigned short)c;
      }
      const unsigned sm = __ballot_sync(0xffffffffu, c < 0);
      if (sm) {
        if (qn + 32 > SFC_QW) flush();
        if (c < 0) q[warp][qn + __popc(sm & ((1u << lane) - 1u))] = make_int4((int)blockIdx.x, li,
                                                                          hx | (hy << 16), hz);
        qn += __popc(sm);
        __syncwarp();
      }
    }
  }
  if (qn) flush();
}

// Phase 2: sub-cell counts of the shell nodes (shell_count, the rule and its
// margins there), one node per lane, the list walked by a persistent grid in
// warp-sized chunks.  Every lane walks the same 100 rows without branches or
// shared memory (suspension of 2260 images in 256^3: 60 us; sorting each
// node's terms and compacting its crossing rows across the warp took 135).
__global__ void __launch_bounds__(SFS_THREADS, 8) sf_shell_kernel(MapParams p) {
  const unsigned long long tot = p.pair_total[2];
  const int total = (int)min(tot, (unsigned long long)p.shell_cap);
  const int stride = (int)(gridDim.x * SFS_THREADS);
  for (int e = (int)(blockIdx.x * SFS_THREADS + threadIdx.x); e < total; e += stride) {
    const int4 ent = p.shell[e];
    const Img& im = p.img[ent.x];
    const int hx = ent.z & 0xFFFF, hy = (int)((unsigned)ent.z >> 16), hz = ent.w;
    const float dxf = small_int_to_float(hx - im.xi[0]) - im.xf[0];
    const float dyf = small_int_to_float(hy - im.xi[1]) - im.xf[1];
    const float dzf = small_int_to_float(hz - im.xi[2]) - im.xf[2];
    p.sfcode[im.sf_off + ent.y] =
        (unsigned short)shell_count(p.g.dim, im, hx, hy, hz, dxf, dyf, dzf);
  }
}

// Phase 2 of the map, per node: the images whose boxes contain it, in image
// order (the cell list is sorted), through the update of setParticlesOnLattice
// (src/LBM_PSM_exchangeParticleData.cpp:69-106) on the two-slot table
// (setParticleOnLattice / setToZero, src/LBM_PSM_lattice.cpp:257-324).
// decFlag = (sf > 1e-5) + 2*(sf_old > 1e-5): cases 0 and 2 clear the tag's slot
// (case 0 finds none unless the tag is the empty marker 0), cases 1 and 3 set
// it (case 3's condition sf > sf_old || id_old == tag holds because
// sf_old > 1e-5 means the tag matched), so only the sf bit decides.  sf > 1e-5
// exactly when the code is non-zero.  The table is written back only where it
// changed.
//
// FP64 storage: the table is ids, eps and us, the reference's values bit for
// bit.  FP32 / FP16 storage: ids and the FP32 records the collide kernel reads
// (eps, u_s per slot), their FP32 roundings (for spinning images the node
// velocity is formed in FP32), no FP64.
//
// One node's update state: the tags of its two slots as they stand after
// the images applied so far.  Slot records are written through (the table
// ends with the same records as when only changed ones are written, without
// a read before the write), so only the ids live in registers; the ids and
// the flag are written back at the end if they changed.
template <bool F64>
struct Apply {
  int id0, id1;
  bool ids_dirty;

  __device__ __forceinline__ void init(int2 ids) {
    id0 = ids.x;
    id1 = ids.y;
    ids_dirty = false;
  }

  // the slot that an image with code cd writes at this node (-1: none); cd = 0:
  // setToZero, the slot left empty (src/LBM_PSM_lattice.cpp:302-324)
  __device__ __forceinline__ int slot_of(int tag, unsigned short cd) {
    if (cd == 0) {
      const int m = tag == id0 ? 0 : (tag == id1 ? 1 : -1);
      if (m >= 0) {
        if (m == 0) id0 = 0; else id1 = 0;
        ids_dirty = true;
      }
      return m;
    }
    // setParticleOnLattice: matching slot, else the first empty one, else drop
    int slot = -1;
    if (id0 == tag)
      slot = 0;
    else if (id1 == tag)
      slot = 1;
    else if (id0 == 0)
      slot = 0;
    else if (id1 == 0)
      slot = 1;
    if (slot >= 0 && (slot == 0 ? id0 : id1) != tag) {
      if (slot == 0) id0 = tag; else id1 = tag;
      ids_dirty = true;
    }
    return slot;
  }

  // FP32: one image with code cd at node n; nv.yzw is the node velocity it sets
  __device__ __forceinline__ void image(const MapParams& p, long long n, int tag,
                                        unsigned short cd, float4 nv) {
    const int slot = slot_of(tag, cd);
    if (slot < 0) return;
    nv.x = cd == SF_ONE ? 1.0f : p.sf_value32[cd];
    // written whether or not it changes: a store does not wait, whereas
    // reading the record first to skip an unchanged one would
    p.tab.rec32[2 * n + slot] = cd == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : nv;
  }

  // FP64: the same at the node (hi, hj, hk) of the box's own frame
  __device__ __forceinline__ void image(const MapParams& p, long long n, int tag, unsigned short cd,
                                        const Img& im, bool spin, int hi, int hj, int hk) {
    const int slot = slot_of(tag, cd);
    if (slot < 0) return;
    double sf = 0.0, u[3] = {0.0, 0.0, 0.0};
    if (cd != 0) {
      sf = cd == SF_ONE ? 1.0 : p.sf_value[cd];
      // rigid-body velocity of the node (src/LBM_PSM_exchangeParticleData.cpp:83-89)
      if (spin) {
        const double dx = small_int_to_double(hi) - im.xl[0];
        const double dy = small_int_to_double(hj) - im.xl[1];
        const double dz = small_int_to_double(hk) - im.xl[2];
        u[0] = im.uT[0] + im.om[1] * dz - im.om[2] * dy;
        u[1] = im.uT[1] + im.om[2] * dx - im.om[0] * dz;
        u[2] = im.uT[2] + im.om[0] * dy - im.om[1] * dx;
      } else {
        // every omega component +0.0 and no uT component -0.0: the reference's
        // (uT + 0*dz) - 0*dy is uT bit for bit
        for (int k = 0; k < 3; ++k) u[k] = im.uT[k];
      }
    }
    reinterpret_cast<double*>(p.tab.eps)[2 * n + slot] = sf;
    for (int k = 0; k < 3; ++k) p.tab.us[6 * n + 3 * slot + k] = u[k];
  }

  __device__ __forceinline__ void store(const MapParams& p, long long n) const {
    if (ids_dirty) {
      if (p.changed) *p.changed = 1;
      p.tab.ids[n] = make_int2(id0, id1);
      p.tab.flag[n] = (uint8_t)((id0 > 0 ? 1 : 0) | (id1 > 0 ? 2 : 0));
    }
  }
};

// rigid-body velocity of node (hi, hj, hk) of a spinning image, in FP32
// (src/LBM_PSM_exchangeParticleData.cpp:83-89)
static __device__ __forceinline__ float4 spin_velocity(const Img& im, int hi, int hj, int hk) {
  const float dx = small_int_to_float(hi - im.xi[0]) - im.xf[0];
  const float dy = small_int_to_float(hj - im.xi[1]) - im.xf[1];
  const float dz = small_int_to_float(hk - im.xi[2]) - im.xf[2];
  return make_float4(0.f, im.uTf[0] + im.omf[1] * dz - im.omf[2] * dy,
                     im.uTf[1] + im.omf[2] * dx - im.omf[0] * dz,
                     im.uTf[2] + im.omf[0] * dy - im.omf[1] * dx);
}

// NPT nodes per thread (z, z + blockDim.z, ... within the cell; one node in
// 2-D) of a cell that some image box touches.  The images of the cell's list
// are visited in image order through their compact records, which cell_sort
// copied next to the list entries (three 16-byte loads straight after the
// cell's offset, instead of list index, then record, then the scattered
// fields of Img), each record serving all the thread's nodes, whose code
// and slot record loads are independent.  The slot ids are loaded with the
// cell's count and offset, so that they add no round of dependent loads.
//
// FP64 storage takes the same kernel at four blocks per multiprocessor (the
// velocities need the registers); an image's record is read only where a node
// is set (128 x 96 x 160 nodes, 230 spheres: 12 us a step faster than one node a
// thread walking the images' full records).
template <bool F64, int NPT>
__global__ void __launch_bounds__(512 / NPT, F64 ? 4 : 8) node_apply_kernel(MapParams p) {
  const int c = (blockIdx.z * p.C[1] + blockIdx.y) * p.C[0] + blockIdx.x;
  const Geom& g = p.g;
  const int sx = blockIdx.x * p.cb[0] + threadIdx.x;
  const int sy = blockIdx.y * p.cb[1] + threadIdx.y;
  const int sz0 = blockIdx.z * p.cb[2] + threadIdx.z;
  const int dz = (int)blockDim.z;
  const long long n0 = node_index(g, sx, sy, sz0);
  const long long zstride = (long long)dz * g.P0 * g.S[1];
  const bool inside = sx < g.S[0] && sy < g.S[1] && sz0 < g.S[2];
  bool has[NPT];
#pragma unroll
  for (int k = 0; k < NPT; ++k)
    has[k] = inside && (int)threadIdx.z + k * dz < p.cb[2] && sz0 + k * dz < g.S[2];
  // the cell's count and offset, the overflow words and the slot ids of the
  // thread's nodes: independent loads, issued together
  const int cnt = __ldg(p.cell_count + c);
  const int coff = __ldg(p.cell_off + c);
  const unsigned long long tot0 = __ldg(p.pair_total), tot1 = __ldg(p.pair_total + 1);
  int2 ids0[NPT];
#pragma unroll
  for (int k = 0; k < NPT; ++k)
    ids0[k] = has[k] && cnt ? p.tab.ids[n0 + k * zstride] : make_int2(0, 0);
  if (cnt == 0 || !inside) return;
  if (tot0 > (unsigned long long)p.list_cap || tot1 > (unsigned long long)p.sf_cap) return;
  const int4* __restrict__ lrec = p.lrec + 3 * (long long)coff;
  Apply<F64> st[NPT];
#pragma unroll
  for (int k = 0; k < NPT; ++k) st[k].init(ids0[k]);
  bool touched[NPT];
#pragma unroll
  for (int k = 0; k < NPT; ++k) touched[k] = false;
  for (int t = 0; t < cnt; ++t) {
    const int4 A = __ldg(lrec + 3 * t);
    const unsigned ax = (unsigned)A.x, ay = (unsigned)A.y, az = (unsigned)A.z;
    const int lo0 = (int)(ax & 0xFFFFu), lo1 = (int)(ay & 0xFFFFu), lo2 = (int)(az & 0xFFFFu);
    const int hi2 = (int)(az >> 16);
    if (sx < lo0 || sx >= (int)(ax >> 16) || sy < lo1 || sy >= (int)(ay >> 16)) continue;
    bool in[NPT];
    bool any = false;
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
      const int z = sz0 + k * dz;
      in[k] = has[k] && z >= lo2 && z < hi2;
      any = any || in[k];
    }
    if (!any) continue;
    const int4 B = __ldg(lrec + 3 * t + 1);
    const int4 U = __ldg(lrec + 3 * t + 2);
    const unsigned bz = (unsigned)B.z;
    const int bx = (int)(bz & 0xFFFFu), by = (int)(bz >> 16);
    const long long off = (long long)(((unsigned long long)(unsigned)B.y << 32) |
                                      (unsigned long long)(unsigned)B.x) +
                          (long long)(sy - lo1) * bx + (sx - lo0);
    const long long plane = (long long)by * bx;
    unsigned short cd[NPT];
#pragma unroll
    for (int k = 0; k < NPT; ++k)
      cd[k] = in[k] ? __ldg(p.sfcode + off + (sz0 + k * dz - lo2) * plane) : (unsigned short)0;
#pragma unroll
    for (int k = 0; k < NPT; ++k) touched[k] = touched[k] || in[k];
    if (F64 || B.w) {
      const int hi = sx + g.off[0], hj = sy + g.off[1];
#pragma unroll
      for (int k = 0; k < NPT; ++k) {
        if (!in[k]) continue;
        const int z = sz0 + k * dz;
        const int hk = z - box_of_z(g, z) * g.bz + g.off[2];  // z in the box's own frame
        if constexpr (F64)
          st[k].image(p, n0 + k * zstride, A.w, cd[k], p.img[U.w], B.w != 0, hi, hj, hk);
        else
          st[k].image(p, n0 + k * zstride, A.w, cd[k], spin_velocity(p.img[U.w], hi, hj, hk));
      }
    } else if constexpr (!F64) {
      const float4 nv = make_float4(0.f, __int_as_float(U.x), __int_as_float(U.y),
                                    __int_as_float(U.z));
#pragma unroll
      for (int k = 0; k < NPT; ++k)
        if (in[k]) st[k].image(p, n0 + k * zstride, A.w, cd[k], nv);
    }
  }
#pragma unroll
  for (int k = 0; k < NPT; ++k)
    if (touched[k]) st[k].store(p, n0 + k * zstride);
}

// img_prep; then two independent chains: the cell lists (scan, fill, sort)
// and the solid fractions (classify, shell); then the table update, which
// needs both.  With an aux stream the cell-list chain runs there.
cudaError_t launch_map(const MapParams& p, cudaStream_t st, cudaStream_t aux, cudaEvent_t fork,
                       cudaEvent_t join) {
  if (p.n <= 0) return cudaSuccess;
  const int ncells = p.C[0] * p.C[1] * p.C[2];
  const int tb = 128;
  const unsigned wblocks = (unsigned)(((long long)p.n * 32 + tb - 1) / tb);
  // IMG_LANES images per block, spread over as many multiprocessors as possible
  img_prep_kernel<<<(p.n + IMG_LANES - 1) / IMG_LANES, IMG_LANES, 0, st>>>(p);
  const bool two = aux && fork && join;
  cudaStream_t cl = two ? aux : st;
  cudaError_t e;
  if (two) {
    if ((e = cudaEventRecord(fork, st)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(aux, fork, 0)) != cudaSuccess) return e;
  }
  cell_scan_kernel<<<1, SCAN_THREADS, 0, cl>>>(p.cell_count, p.cell_off, ncells);
  img_fill_kernel<<<wblocks, tb, 0, cl>>>(p);
  cell_sort_kernel<<<(ncells + 255) / 256, 256, 0, cl>>>(p, ncells);
  if (few_images(p.n, p.sm_count))
    sf_classify_kernel<8><<<dim3((unsigned)p.n, SFC_PARTS), SFC_THREADS, 0, st>>>(p);
  else
    sf_classify_kernel<32><<<dim3((unsigned)p.n, classify_parts(p.n, p.sm_count)), SFC_THREADS, 0, st>>>(p);
  sf_shell_kernel<<<p.sm_count * 8, SFS_THREADS, 0, st>>>(p);
  if (two) {
    if ((e = cudaEventRecord(join, aux)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(st, join, 0)) != cudaSuccess) return e;
  }
  constexpr int NPT = 2;  // nodes per thread along z
  const dim3 cells((unsigned)p.C[0], (unsigned)p.C[1], (unsigned)p.C[2]);
  const dim3 part(p.cb[0], p.cb[1], (p.cb[2] + NPT - 1) / NPT);
  if (p.write32)
    node_apply_kernel<false, NPT><<<cells, part, 0, st>>>(p);
  else
    node_apply_kernel<true, NPT><<<cells, part, 0, st>>>(p);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ reduce
// The step's status word into host memory for the host-pointer step (every
// kernel that sets a bit ran before the reduction in stream order).
static __device__ __forceinline__ void copy_status(const ReduceParams& p) {
  if (p.status_out && blockIdx.x == 0 && threadIdx.x == 0)
    *p.status_out = *static_cast<const volatile int*>(p.status);
}

// Error-free transformation: a + b = s + e exactly (Knuth's TwoSum; no
// contraction or reassociation under -fmad=false).
static __device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Twelve running sums of a lane (F, T, S before the unit factors).
//
// FP32 node forces (FP32 / FP16 / BF16 storage): per-node terms in FP32 (the
// node forces carry FP32 precision), summed in double-float (hi + lo pairs
// combined with TwoSum, ~48-bit significand) on the FP32 pipe.
template <bool F64>
struct Sums;
template <>
struct Sums<false> {
  typedef float2 Pair;  // a partial sum, hi and lo
  float hi[12], lo[12];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < 12; ++k) hi[k] = lo[k] = 0.0f;
  }
  __device__ __forceinline__ void node(float F0, float F1, float F2, float dx, float dy, float dz) {
    const float term[12] = {F0,
                            F1,
                            F2,
                            dy * F2 - dz * F1,
                            dz * F0 - dx * F2,
                            dx * F1 - dy * F0,
                            dx * F0,
                            dy * F1,
                            dz * F2,
                            0.5f * (dy * F0 + dx * F1),
                            0.5f * (dz * F0 + dx * F2),
                            0.5f * (dz * F1 + dy * F2)};
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      float sv, e;
      two_sum(hi[q], term[q], sv, e);
      hi[q] = sv;
      lo[q] += e;
    }
  }
  static __device__ __forceinline__ Pair get(const Sums& s, int k) { return make_float2(s.hi[k], s.lo[k]); }
  static __device__ __forceinline__ Pair zero() { return make_float2(0.0f, 0.0f); }
  static __device__ __forceinline__ Pair pick(bool b, Pair x, Pair y) {
    return make_float2(b ? x.x : y.x, b ? x.y : y.y);
  }
  static __device__ __forceinline__ Pair other(Pair x, int o) {
    return make_float2(__shfl_xor_sync(0xffffffffu, x.x, o), __shfl_xor_sync(0xffffffffu, x.y, o));
  }
  static __device__ __forceinline__ Pair plus(Pair x, Pair y) {
    float sv, e;
    two_sum(x.x, y.x, sv, e);
    return make_float2(sv, x.y + y.y + e);
  }
  // the groups' sums in order, and their total times the unit factor
  static __device__ __forceinline__ void add(Pair& s, double&, Pair x) { s = plus(s, x); }
  static __device__ __forceinline__ double scaled(Pair s, double, double factor) {
    return ((double)s.x + (double)s.y) * factor;
  }
};
// FP64 node forces: FP64 sums (the products in fused multiply-adds, the unit
// factors once at the end: half the FP64 operations of the reference's
// per-node expressions, on a pipe of 1.7 per clock and multiprocessor).  The
// groups' sums are added and scaled with the roundings kept (TwoSum, and the
// product's remainder), and a group's rows come from all over the box, so that
// opposite terms of a stresslet cancel within a group.  Error of F, T and S (rms,
// relative to the largest component, 40 spheres of diameter 8 to 14, units of
// 1e-17): 4.2, 4.8, 639; plain sums of neighbouring rows 7.4, 9.8, 3360; every term scaled
// and summed by 128 threads in strides 6.5, 6.9, 1070.
template <>
struct Sums<true> {
  typedef double Pair;
  double s[12];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < 12; ++k) s[k] = 0.0;
  }
  __device__ __forceinline__ void node(double F0, double F1, double F2, double dx, double dy, double dz) {
    s[0] += F0;
    s[1] += F1;
    s[2] += F2;
    s[3] += __fma_rn(dy, F2, -(dz * F1));
    s[4] += __fma_rn(dz, F0, -(dx * F2));
    s[5] += __fma_rn(dx, F1, -(dy * F0));
    s[6] = __fma_rn(dx, F0, s[6]);
    s[7] = __fma_rn(dy, F1, s[7]);
    s[8] = __fma_rn(dz, F2, s[8]);
    s[9] += __fma_rn(dy, F0, dx * F1);  // twice the stresslet term, halved at the end
    s[10] += __fma_rn(dz, F0, dx * F2);
    s[11] += __fma_rn(dz, F1, dy * F2);
  }
  static __device__ __forceinline__ Pair get(const Sums& s, int k) { return s.s[k]; }
  static __device__ __forceinline__ Pair zero() { return 0.0; }
  static __device__ __forceinline__ Pair pick(bool b, Pair x, Pair y) { return b ? x : y; }
  static __device__ __forceinline__ Pair other(Pair x, int o) { return __shfl_xor_sync(0xffffffffu, x, o); }
  static __device__ __forceinline__ Pair plus(Pair x, Pair y) { return x + y; }
  static __device__ __forceinline__ void add(Pair& s, double& lo, Pair x) {
    const double t = s + x, b = t - s;
    lo += (s - (t - b)) + (x - b);
    s = t;
  }
  static __device__ __forceinline__ double scaled(Pair s, double lo, double factor) {
    const double p = s * factor, c = __fma_rn(s, factor, -p) + lo * factor;
    return fabs(c) <= 1.7976931348623157e308 ? p + c : p;  // (not finite: as the plain product)
  }
};

// Per-image force, torque and stresslet (calculateHydrodynamicInteractions,
// src/LBM_PSM_exchangeParticleData.cpp:172-244): the node forces of the
// image's tag over its box.
//
// A solo image's tag can only sit on nodes within rP (eps > 0 from this
// image), so each row is cut to the x-range that may lie within rP: an FP32
// bound widened by 0.01 node, a superset (extra nodes fail the tag test).  The
// rows of the box are taken in groups (red_group), one warp a group, up to 32
// rows at a time, one per lane: the warp walks the nodes of their segments 32 at a time
// (x fastest, consecutive lanes on consecutive nodes), a lane finding its
// node's row by a binary search of the segments' offsets across the warp.  The
// lanes' sums of a group are combined in a fixed tree, the groups' sums in
// order, so the result depends on the image's box alone, however many warps
// and blocks share its groups.
//
// C blocks (a cluster) share an image.  With many images one block of two
// warps each keeps every multiprocessor busy (2260 images of diameter 12: one
// wave); with few, eight blocks spread an image's groups over eight
// multiprocessors, their sums meeting in the first block's shared memory (one
// image of diameter 16: 45 us by one block).
//
// Rows per group: a node's FP64 sums are 27 operations on a pipe that a
// multiprocessor's warps share, and a disc has few rows, so FP64 images take
// small groups that reach all eight blocks (groups of 64 and 32/8: a step with
// one disc of diameter 40 79.4 and 77.4 us, 16 tangent steps with four spheres
// of diameter 12 3.85 and 3.71 ms); FP32 sums keep 64 (a 2-D step the same with 8).
// Row r of an FP64 image is in group r mod G.
constexpr int RED_THREADS = 64;
static __device__ __forceinline__ int red_group(const Geom& g, bool f64) {
  return !f64 ? 64 : (g.dim == 2 ? 8 : 32);
}
constexpr int RED_MAX_GROUPS = 64;  // groups whose sums are held at a time
constexpr int RED_CLUSTER = 8;

template <bool F64, int C>
static __device__ __forceinline__ void reduce_image(const ReduceParams& p) {
  typedef Sums<F64> S;
  typedef typename S::Pair Pair;
  constexpr int NW = RED_THREADS / 32;
  // nodes per lane and round, loaded before any is summed (a lane sums its
  // nodes in the same order whatever U)
  constexpr int U = C == 1 ? (F64 ? 1 : 2) : (F64 ? 4 : 8);
  __shared__ Pair part[RED_MAX_GROUPS][12];
  // the first block's shared memory may be written once every block of the
  // cluster is known to run: all arrive here and wait before their groups, so
  // that the loads of the image lie between
  if (C > 1) cooperative_groups::this_cluster().barrier_arrive();
  const int ip = C == 1 ? (int)blockIdx.x : (int)blockIdx.x / C;
  const int rank = C == 1 ? 0 : (int)blockIdx.x % C;
  const Geom& g = p.g;
  const int tag = p.tag[ip];
  const Img& bx = p.img[ip];  // box and centre from the map's image record
  const int wx = bx.qhi[0] - bx.qlo[0], wy = bx.qhi[1] - bx.qlo[1], wz = bx.qhi[2] - bx.qlo[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int R = wx > 0 && wy > 0 && wz > 0 ? wy * wz : 0;  // x-rows of the box
  const int group = red_group(g, F64), Gmin = (R + group - 1) / group;
  // FP64 groups are alike (their rows come from all over the box): an even
  // number of them leaves both warps of a block the same work
  const int G = F64 ? (Gmin + 1) & ~1 : Gmin;
  const FastDiv fy = make_fastdiv((unsigned)max(wy, 1));
  const int xi[3] = {bx.xi[0], bx.xi[1], bx.xi[2]};  // xl = xi + xf exactly
  const float xf[3] = {bx.xf[0], bx.xf[1], bx.xf[2]};
  const double xl0 = F64 ? bx.xl[0] : 0.0;
  const float rem0 = bx.rP2f * 1.0001f + 0.01f;
  Pair total = S::zero();  // thread k < 12 of the first block: sum k
  double rest = 0.0;       // and (FP64) what its roundings left
  if (C > 1) cooperative_groups::this_cluster().barrier_wait();
  for (int g0 = 0; g0 < G || g0 == 0; g0 += RED_MAX_GROUPS) {
    const int gend = min(G, g0 + RED_MAX_GROUPS);
    for (int gi = g0 + warp * C + rank; gi < gend; gi += C * NW) {
      // FP32: rows gi*group + m; FP64: rows gi + m*G, from all over the box
      const int first = F64 ? gi : gi * group, stride = F64 ? G : 1;
      S acc;
      acc.clear();
#pragma unroll 1
      for (int m0 = 0; m0 < group && first + m0 * stride < R; m0 += 32) {
        const int m = m0 + lane, r = first + m * stride;
        int xa = bx.qlo[0], len = 0, j = 0, k = 0;
        float fdy = 0.0f, fdz = 0.0f;
        double ddy = 0.0, ddz = 0.0;
        if (m < group && r < R) {
          const int q = (int)fast_div((unsigned)r, fy);
          j = bx.qlo[1] + r - q * wy;
          k = bx.qlo[2] + q;
          int xb = bx.qhi[0];
          fdy = small_int_to_float(j - xi[1]) - xf[1];
          fdz = small_int_to_float(k - xi[2]) - xf[2];
          if (bx.solo) {
            const float rem = rem0 - fdy * fdy - fdz * fdz;
            if (rem < 0.0f) {
              xb = xa;
            } else {
              const float h = sqrtf(rem) + 0.01f;
              xa = max(xa, xi[0] + (int)ceilf(xf[0] - h));
              xb = min(xb, xi[0] + (int)floorf(xf[0] + h) + 1);
            }
          }
          len = max(xb - xa, 0);
          if (F64) {
            ddy = small_int_to_double(j) - bx.xl[1];
            ddz = small_int_to_double(k) - bx.xl[2];
          }
        }
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        const int excl = incl - len;
        const int count = __shfl_sync(0xffffffffu, incl, 31);
        for (int base = 0; base < count; base += U * 32) {
          int2 id[U];
          float2 f01[U], f23[U], f45[U];
          double d0[U], d1[U], d2[U], d3[U], d4[U], d5[U];
          float dx[U], dy[U], dz[U];
          double ex[U], ey[U], ez[U];
          bool ok[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int t = base + u * 32 + lane;
            // the row holding node t: the last lane whose offset is <= t (a
            // row of length 0 shares its offset with the next row)
            int l = 0;
#pragma unroll
            for (int st = 16; st >= 1; st >>= 1)
              if (__shfl_sync(0xffffffffu, excl, l + st) <= t) l += st;
            const int ra = __shfl_sync(0xffffffffu, xa, l);
            const int re = __shfl_sync(0xffffffffu, excl, l);
            const int jj = __shfl_sync(0xffffffffu, j, l);
            const int kk = __shfl_sync(0xffffffffu, k, l);
            const int i = ra + t - re;
            ok[u] = t < count;
            id[u] = make_int2(0, 0);
            if (F64) {
              ey[u] = __shfl_sync(0xffffffffu, ddy, l);
              ez[u] = __shfl_sync(0xffffffffu, ddz, l);
            } else {
              f01[u] = f23[u] = f45[u] = make_float2(0.f, 0.f);
              dx[u] = small_int_to_float(i - xi[0]) - xf[0];
              dy[u] = small_int_to_float(jj - xi[1]) - xf[1];
              dz[u] = small_int_to_float(kk - xi[2]) - xf[2];
            }
            if (ok[u]) {
              const long long n = node_index(g, i - g.off[0], jj - g.off[1], kk - g.off[2] + bx.zoff);
              // both slots' forces are loaded with the ids (no second dependent load)
              id[u] = p.tab.ids[n];
              if (F64) {
                const double2* nf2 = reinterpret_cast<const double2*>(static_cast<const double*>(p.tab.nodeF) + 6 * n);
                const double2 a = nf2[0], b = nf2[1], c = nf2[2];
                d0[u] = a.x; d1[u] = a.y; d2[u] = b.x;
                d3[u] = b.y; d4[u] = c.x; d5[u] = c.y;
                ex[u] = small_int_to_double(i) - xl0;
              } else {
                const float2* nf2 = reinterpret_cast<const float2*>(static_cast<const float*>(p.tab.nodeF) + 6 * n);
                f01[u] = nf2[0];
                f23[u] = nf2[1];
                f45[u] = nf2[2];
              }
            }
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (!ok[u]) continue;
            const bool one = tag == id[u].x, two = tag == id[u].y;
            if (!one && !two) continue;
            if constexpr (F64)
              acc.node(one ? d0[u] : d3[u], one ? d1[u] : d4[u], one ? d2[u] : d5[u], ex[u], ey[u], ez[u]);
            else
              acc.node(one ? f01[u].x : f23[u].y, one ? f01[u].y : f45[u].x, one ? f23[u].x : f45[u].y,
                       dx[u], dy[u], dz[u]);
          }
        }
      }
      // fixed-order reduction within the warp: the first two levels halve the
      // terms each lane carries (12 -> 6 -> 3, partners keeping complementary
      // halves), the last three are a butterfly on three terms
      const bool up16 = (lane & 16) != 0, up8 = (lane & 8) != 0;
      Pair h6[6], h3[3];
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const Pair x = S::get(acc, k), y = S::get(acc, k + 6);
        h6[k] = S::plus(S::pick(up16, y, x), S::other(S::pick(up16, x, y), 16));
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        h3[k] = S::plus(S::pick(up8, h6[k + 3], h6[k]), S::other(S::pick(up8, h6[k], h6[k + 3]), 8));
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) h3[k] = S::plus(h3[k], S::other(h3[k], o));
      if ((lane & 7) == 0) {  // lanes 0, 8, 16, 24 hold terms 0-2, 3-5, 6-8, 9-11
        const int q0 = (up16 ? 6 : 0) + (up8 ? 3 : 0);
        Pair* dst = &part[gi - g0][q0];
        if (C > 1) dst = cooperative_groups::this_cluster().map_shared_rank(dst, 0);
#pragma unroll
        for (int k = 0; k < 3; ++k) dst[k] = h3[k];
      }
    }
    if (C > 1)
      cooperative_groups::this_cluster().sync();
    else
      __syncthreads();
    if (rank == 0 && threadIdx.x < 12)
      for (int k = 0; k < gend - g0; ++k) S::add(total, rest, part[k][threadIdx.x]);
    if (G > RED_MAX_GROUPS) {  // the sums are read before the next groups' arrive
      if (C > 1)
        cooperative_groups::this_cluster().sync();
      else
        __syncthreads();
    }
  }
  if (rank == 0 && threadIdx.x < 12) {
    const int q = threadIdx.x;
    const BoxParams& bp = p.box[bx.bidx];
    const double sum = S::scaled(total, rest, q < 3 ? bp.forceFactor : bp.torqueFactor);
    if (q < 3) {
      const double v = sum;
      p.fh[3 * ip + q] = v;
      if (p.fh2) p.fh2[3 * ip + q] = v;
    } else if (q < 6) {
      const double v = sum;
      p.th[3 * ip + (q - 3)] = v;
      if (p.th2) p.th2[3 * ip + (q - 3)] = v;
    } else {
      const double v = -(F64 && q >= 9 ? 0.5 * sum : sum);
      p.S[6 * ip + (q - 6)] = v;
      if (p.S2) p.S2[6 * ip + (q - 6)] = v;
    }
  }
  copy_status(p);
}

__global__ void __launch_bounds__(RED_THREADS, 16) reduce_f32_kernel(ReduceParams p) {
  reduce_image<false, 1>(p);
}
__global__ void __launch_bounds__(RED_THREADS) reduce_f64_kernel(ReduceParams p) {
  reduce_image<true, 1>(p);
}
__global__ void __launch_bounds__(RED_THREADS) __cluster_dims__(RED_CLUSTER, 1, 1)
    reduce_f32_few_kernel(ReduceParams p) {
  reduce_image<false, RED_CLUSTER>(p);
}
__global__ void __launch_bounds__(RED_THREADS) __cluster_dims__(RED_CLUSTER, 1, 1)
    reduce_f64_few_kernel(ReduceParams p) {
  reduce_image<true, RED_CLUSTER>(p);
}

cudaError_t launch_reduce(const ReduceParams& p, cudaStream_t st) {
  if (p.n <= 0) return cudaSuccess;
  const bool few = few_images(p.n, p.sm_count);
  const unsigned grid = (unsigned)p.n * (few ? RED_CLUSTER : 1);
  if (p.nodeF_is_double) {
    if (few)
      reduce_f64_few_kernel<<<grid, RED_THREADS, 0, st>>>(p);
    else
      reduce_f64_kernel<<<grid, RED_THREADS, 0, st>>>(p);
  } else {
    if (few)
      reduce_f32_few_kernel<<<grid, RED_THREADS, 0, st>>>(p);
    else
      reduce_f32_kernel<<<grid, RED_THREADS, 0, st>>>(p);
  }
  return cudaGetLastError();
}

// the kernels whose parameters a replayed device-step graph updates per call
const void* img_prep_fn() { return (const void*)img_prep_kernel; }
const void* reduce_fn(int nodeF_is_double, int n, int sm_count) {
  if (few_images(n, sm_count))
    return nodeF_is_double ? (const void*)reduce_f64_few_kernel : (const void*)reduce_f32_few_kernel;
  return nodeF_is_double ? (const void*)reduce_f64_kernel : (const void*)reduce_f32_kernel;
}

// ------------------------------------------------------------------ exports
// particle table in the reference layout (halo nodes of periodic axes empty)
__global__ void table_export_kernel(Geom g, Table t, int* ids, double* eps, double* us) {
  const long long total = (long long)g.L[0] * g.L[1] * g.L[2];
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= total) return;
  const int k = (int)(r % g.L[2]);
  const int j = (int)((r / g.L[2]) % g.L[1]);
  const int i = (int)(r / ((long long)g.L[2] * g.L[1]));
  const int sx = i - g.off[0], sy = j - g.off[1], sz = k - g.off[2];
  const bool ok = sx >= 0 && sx < g.S[0] && sy >= 0 && sy < g.S[1] && sz >= 0 && sz < g.S[2];
  int2 id = make_int2(0, 0);
  double2 e = make_double2(0.0, 0.0);
  double u[6] = {0, 0, 0, 0, 0, 0};
  if (ok) {
    const long long n = node_index(g, sx, sy, sz);
    id = t.ids[n];
    if (t.eps) {
      e = t.eps[n];
      for (int c = 0; c < 6; ++c) u[c] = t.us[6 * n + c];
    } else {  // FP32 / FP16 storage keeps only the FP32 records
      const float4 r0 = t.rec32[2 * n], r1 = t.rec32[2 * n + 1];
      e = make_double2(r0.x, r1.x);
      u[0] = r0.y; u[1] = r0.z; u[2] = r0.w;
      u[3] = r1.y; u[4] = r1.z; u[5] = r1.w;
    }
  }
  if (ids) {
    ids[2 * r] = id.x;
    ids[2 * r + 1] = id.y;
  }
  if (eps) {
    eps[2 * r] = e.x;
    eps[2 * r + 1] = e.y;
  }
  if (us)
    for (int c = 0; c < 6; ++c) us[6 * r + c] = u[c];
}

cudaError_t launch_table_export(const Geom& g, const Table& t, int* ids, double* eps, double* us,
                                cudaStream_t st) {
  const long long total = (long long)g.L[0] * g.L[1] * g.L[2];
  table_export_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(g, t, ids, eps, us);
  return cudaGetLastError();
}

// execute_write_vti field read (src/fix_LBM_PSM_writeVTI.h:146-169): z
// outermost, x innermost.  One block per 256 nodes of an x-row; the velocities
// (three values a node) go through shared memory, so that every field leaves in
// full runs, to device memory or, over NVLink-C2C, to the caller's arrays.
constexpr int EXP_THREADS = 256;
template <typename T>
__global__ void __launch_bounds__(EXP_THREADS) export_fields_kernel(Geom g, Table t, const double* rho,
                                                                    const double* u, double B0, double rho0,
                                                                    double u0, T* solid_out, T* rho_out,
                                                                    T* u_out) {
  __shared__ T su[3 * EXP_THREADS];
  const int nxi = g.L[0] - 2, nyi = g.L[1] - 2;
  const int xblocks = (nxi + EXP_THREADS - 1) / EXP_THREADS;
  const unsigned row = blockIdx.x / (unsigned)xblocks;
  const int x0 = (int)(blockIdx.x - row * (unsigned)xblocks) * EXP_THREADS;
  const int k = (int)(row / (unsigned)nyi), j = (int)(row - (unsigned)k * (unsigned)nyi);
  const int cnt = min(EXP_THREADS, nxi - x0), tid = threadIdx.x;
  const long long id0 = (long long)row * nxi + x0;
  if (tid < cnt) {
    const long long n = node_index(g, 1 + x0 + tid - g.off[0], 1 + j - g.off[1],
                                   (g.dim == 3 ? 1 : 0) + k - g.off[2]);
    if (solid_out) {
      const double2 e = t.eps ? t.eps[n] : make_double2(t.rec32[2 * n].x, t.rec32[2 * n + 1].x);
      const double Bv = (e.x + e.y);
      solid_out[id0 + tid] = (T)((Bv > 1.0 ? 1.0 : Bv) * B0);
    }
    if (rho_out) rho_out[id0 + tid] = (T)((rho ? rho[n] : 1.0) * rho0);
    if (u_out) {
      su[3 * tid] = (T)((u ? u[3 * n + 0] : 0.0) * u0);
      su[3 * tid + 1] = (T)((u ? u[3 * n + 1] : 0.0) * u0);
      su[3 * tid + 2] = g.dim == 3 ? (T)((u ? u[3 * n + 2] : 0.0) * u0) : (T)0;
    }
  }
  if (!u_out) return;
  __syncthreads();
  for (int c = tid; c < 3 * cnt; c += EXP_THREADS) u_out[3 * id0 + c] = su[c];
}

cudaError_t launch_export_fields(const Geom& g, const Table& t, const double* rho, const double* u,
                                 int as_double, double B0, double rho0, double u0, void* solid_out,
                                 void* rho_out, void* u_out, cudaStream_t st) {
  const long long rows = (long long)(g.L[1] - 2) * (g.dim == 3 ? g.L[2] - 2 : 1);
  if (rows <= 0 || g.L[0] <= 2) return cudaSuccess;
  const unsigned grid = (unsigned)(rows * ((g.L[0] - 2 + EXP_THREADS - 1) / EXP_THREADS));
  if (as_double)
    export_fields_kernel<double><<<grid, EXP_THREADS, 0, st>>>(
        g, t, rho, u, B0, rho0, u0, static_cast<double*>(solid_out), static_cast<double*>(rho_out),
        static_cast<double*>(u_out));
  else
    export_fields_kernel<float><<<grid, EXP_THREADS, 0, st>>>(
        g, t, rho, u, B0, rho0, u0, static_cast<float*>(solid_out), static_cast<float*>(rho_out),
        static_cast<float*>(u_out));
  return cudaGetLastError();
}

}  // namespace lbmpsm
