// pme_direct.cu -- direct-space (real-space) PME nonbonded terms on sm_100a (include/pme_direct.h).
//
// The role of CudaPMEDirectForce<long long, float> with its topological exclusions, for the
// models of the reference's direct test: shifted Lennard-Jones (VDW_VSH,
// CudaDirectForceKernels.cu:175-195) and Ewald real-space electrostatics (EWALD, :353-391).
//
// One calc_force is a clear and five launches on the handle's stream:
//   k_direct_cell     atom -> (y, z) column and x bin, counts (columns a fraction of roff wide);
//   k_direct_columns  one warp per column: room for its atoms, first atom of every bin, clusters of 8
//                     consecutive atoms;
//   k_direct_fill     atoms into their bins (unordered);
//   k_direct_order    order every bin's atoms by x and index (so every run sums in the same order) and
//                     gather coordinates, type, global index and exclusion window;
//   k_direct_pairs    one warp per cluster: candidates are the x intervals of the columns in reach; a
//                     cheap FP32 distance pass queues them per atom, the pair terms then run on full
//                     lanes.
// Each pair is evaluated from both sides (no third-law scatter): each pair's force is rounded once
// to 2^-40 and every sum after that is exact int64, so results are run-to-run identical.  Energies
// are rounded to 2^-32 per pair and summed in int64; both sides give the same pair distance, so the
// doubled sums halve exactly (1-4 terms are added twice to match).
// Exclusions: a 128-bit window per atom over global indices g_j - g_i in [-64, 64) (bit 64: the
// atom itself), plus an explicit list for partners beyond the window.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/pme_direct.h"
#include "pme_direct_plan.h"
#include "pme_direct_math.h"
#include "pme_state.h"

namespace pme {
namespace direct {

constexpr int kTasksPerWarp = 5;      // pair tasks per resident warp to aim at (24,000 atoms: 5 per warp 275 us a step, 3 279, 1 308)
constexpr int kMaxTypes = 200;        // vdW types
constexpr float kEnergyScale = 4294967296.0f;     // 2^32
constexpr float kForceScaleF = 1099511627776.0f;  // 2^40
constexpr int kTabShift = 15;        // high word of r^2 -> table interval
static_assert(kTabOctave == 1 << (20 - kTabShift), "the interval's bits");
constexpr float kTwoSqrtPi = 1.1283791670955126f; // 2/sqrt(pi)

struct Params {
  float box[3], inv_box[3];
  float kappa, kappa2, roff2, ro6, ro12, ro18;   // roff^-6, roff^-12, roff^-18
  float e14fac;
  int vdw, elec;
  int nc[3];          // x look-up bins per column; columns along y and z
  int reach[2];       // column offsets -reach .. reach along y and z
  float cut2, marg;   // widened squared cutoff of the cheap pass; slack of the candidate intervals (A)
  int ntype;          // vdW types
  int square;         // shared memory holds the vdW table as ntype x ntype (else the packed triangle is read)
  int big_hi;         // high word of 1024 / roff: forces above it take the slow rounding
  int slices;         // tasks per cluster, each with some of the column rows along z
  double kappad, roff2d, ro6d, ro12d, ro18d;   // FP64 for the main-list pair terms
  double boxd[3];
  // Ewald real space (ewald_table): F = (r dE/dr) / r^2 of E = erfc(kappa r) / r, then E itself
  const double2* tab;
  int tab_n;          // intervals (0: no table); s outside them uses erfc() and exp()
};

enum Acc { kAccVdw = 0, kAccElec = 1, kAccExcl = 2, kAccVir = 3, kAccN = 9 };   // vir: xx xy xz yy yz zz

// r dU/dr / r^2 and the energies of one pair at squared distance r2.  a_elec is the factor of
// qq / r in U_elec: erfc(kappa r) for ordinary pairs, e14fac - erf(kappa r) for 1-4 pairs,
// -erf(kappa r) for excluded pairs (formed with erff, not as erfc + s - 1, which cancels in FP32).
// c6 / c12 carry the reference's factors 6 and 12.
__device__ __forceinline__ float pair_terms(float r2, float qq, float c6, float c12, const Params& p, int kind,
                                            bool vdw, float& u_vdw, float& u_elec) {
  const float r = sqrtf(r2);        // IEEE square root and reciprocal, as the reference computes them
  const float rinv = 1.0f / r;
  const float rinv2 = rinv * rinv;
  float fr = 0.0f;
  u_vdw = 0.0f;
  if (vdw) {
    const float rinv6 = rinv2 * rinv2 * rinv2, rinv12 = rinv6 * rinv6, r6 = r2 * r2 * r2;
    fr = c6 * (rinv6 - r6 * p.ro12) - c12 * (rinv12 + r6 * p.ro18);
    u_vdw = c12 * (1.0f / 12.0f) * (rinv12 + 2.0f * r6 * p.ro18 - 3.0f * p.ro12) -
            c6 * (1.0f / 6.0f) * (rinv6 + r6 * p.ro12 - 2.0f * p.ro6);
  }
  u_elec = 0.0f;
  if (p.elec == PME_ELEC_NONE) return fr * rinv2;
  const float kr = p.kappa * r;
  const float a = kind == 0 ? erfcf(kr) : (kind == 1 ? p.e14fac - erff(kr) : -erff(kr));
  const float e = qq * a * rinv;
  u_elec = e;
  fr += -qq * kTwoSqrtPi * p.kappa * expf(-p.kappa2 * r2) - e;
  return fr * rinv2;
}

// The same terms in FP64 from the FP32 pair geometry, for the main pair list: the atoms' net
// forces are small differences of large pair forces (close contacts of ~1e3 kcal/mol/A), where
// the few-ulp error of an FP32 evaluation shows.

static_assert(kTabTerms == 6, "quintics");
__device__ __forceinline__ double quintic(const double2* c, double t) {
  const double2 lo = c[0], mid = c[1], hi = c[2];
  return __fma_rn(__fma_rn(__fma_rn(__fma_rn(__fma_rn(hi.y, t, hi.x), t, mid.y), t, mid.x), t, lo.y), t, lo.x);
}

// Shifted Lennard-Jones: (r dU/dr) and U from s = r^2 and 1 / s.
template <bool EV>
__device__ __forceinline__ double vdw_terms_f64(double s, double sinv, float2 cc, const Params& p, double& u_vdw) {
  const double c6 = cc.x, c12 = cc.y;
  const double rinv6 = sinv * sinv * sinv, r6 = s * s * s, rinv12 = rinv6 * rinv6;
  if (EV)
    u_vdw = c12 * (1.0 / 12.0) * (rinv12 + 2.0 * r6 * p.ro18d - 3.0 * p.ro12d) -
            c6 * (1.0 / 6.0) * (rinv6 + r6 * p.ro12d - 2.0 * p.ro6d);
  return c6 * (rinv6 - r6 * p.ro12d) - c12 * (rinv12 + r6 * p.ro18d);
}

// All terms without the Ewald table: (r dU/dr) / r^2.
__device__ __forceinline__ double pair_terms_f64(double s, double qq, float2 cc, const Params& p, double& u_vdw,
                                              double& u_elec) {
  const double rinv = rsqrt(s), r = s * rinv, sinv = rinv * rinv;
  double fr = vdw_terms_f64<true>(s, sinv, cc, p, u_vdw);
  u_elec = 0.0;
  if (p.elec != PME_ELEC_NONE) {
    u_elec = qq * erfc(p.kappad * r) * rinv;
    fr += -qq * 1.1283791670955126 * p.kappad * exp(-p.kappad * p.kappad * s) - u_elec;
  }
  return fr * sinv;
}

__device__ __forceinline__ float2 vdw_c6c12(const float2* tab, int ta, int tb) {
  const int a = max(ta, tb), b = min(ta, tb);
  return tab[a * (a + 1) / 2 + b];
}

__device__ __forceinline__ long long warp_sum_ll(long long v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// ---------------------------------------------------------------------------------------------
// Binning
// ---------------------------------------------------------------------------------------------
// Coordinate wrapped into the box: x - L floor(x / L), which FP32 rounding can leave a hair below
// 0 or equal to L; non-finite inputs become 0.  The column and x bin come from this same value, so
// they and an atom's stored position always agree (the candidate intervals have that slack).
__device__ __forceinline__ float wrap_coord(float x, float box, float inv_box) {
  const float w = x - box * floorf(x * inv_box);
  return (w >= -box && w <= 2.0f * box) ? w : 0.0f;
}

__device__ __forceinline__ int cell_of_wrapped(float w, float inv_box, int n) {
  return max(0, min((int)(w * inv_box * (float)n), n - 1));
}

__global__ void k_direct_cell(const float4* __restrict__ xyzq, int n, const Params p, int2* __restrict__ cell_of,
                              int* __restrict__ count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 a = xyzq[i];
  const int cx = cell_of_wrapped(wrap_coord(a.x, p.box[0], p.inv_box[0]), p.inv_box[0], p.nc[0]);
  const int cy = cell_of_wrapped(wrap_coord(a.y, p.box[1], p.inv_box[1]), p.inv_box[1], p.nc[1]);
  const int cz = cell_of_wrapped(wrap_coord(a.z, p.box[2], p.inv_box[2]), p.inv_box[2], p.nc[2]);
  const int c = (cz * p.nc[1] + cy) * (p.nc[0] + 1) + cx;
  cell_of[i] = make_int2(c, atomicAdd(&count[c], 1));
}

// One warp per column: reserves room for the column's atoms and clusters (columns come in any order:
// no result depends on where they lie), writes xstart[cell] = first atom of every x bin (entry nbx of
// a column: its end) and the column's clusters (first atom, column).
__global__ void k_direct_columns(const Params p, const int* __restrict__ count, int ncol, int* __restrict__ totals,
                                 int* __restrict__ xstart, int2* __restrict__ clusters) {
  const int lane = threadIdx.x & 31, nbx = p.nc[0];
  const int col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (col >= ncol) return;
  const int* cnt = count + (size_t)col * (nbx + 1);
  int n = 0;
  for (int b = lane; b < nbx; b += 32) n += cnt[b];
  n = __reduce_add_sync(0xffffffffu, n);
  const int nc = (n + kCluster - 1) / kCluster;
  int first = 0, clus = 0;
  if (lane == 0 && n > 0) {
    first = atomicAdd(&totals[0], n);
    clus = atomicAdd(&totals[1], nc);
  }
  first = __shfl_sync(0xffffffffu, first, 0);
  clus = __shfl_sync(0xffffffffu, clus, 0);
  for (int k = lane; k < nc; k += 32) clusters[clus + k] = make_int2(first + k * kCluster, col);
  int run = first;
  for (int b0 = 0; b0 <= nbx; b0 += 32) {
    const int b = b0 + lane, v = b < nbx ? cnt[b] : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (b <= nbx) xstart[(size_t)col * (nbx + 1) + b] = run + incl - v;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
}

// Order of an atom in its bin: by wrapped x, then by index (as one 64-bit integer).
__device__ __forceinline__ unsigned long long order_key(float x, int atom) {
  const unsigned int b = (unsigned int)__float_as_int(x);
  return (unsigned long long)(b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u)) << 32 | (unsigned int)atom;
}

__global__ void k_direct_fill(const int2* __restrict__ cell_of, int n, const Params p, const float4* __restrict__ xyzq,
                              const int* __restrict__ xstart, unsigned long long* __restrict__ keys) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int2 c = cell_of[i];
  keys[xstart[c.x] + c.y] = order_key(wrap_coord(xyzq[i].x, p.box[0], p.inv_box[0]), i);
}

// One thread per filled slot: rank its atom among the few of its bin and gather its data there.
__global__ void k_direct_order(const Params p, int n, const unsigned long long* __restrict__ keys,
                               const int2* __restrict__ cell_of, const int* __restrict__ xstart,
                               const float4* __restrict__ xyzq, const int* __restrict__ vdwtype,
                               const int* __restrict__ glob, const ulonglong2* __restrict__ win,
                               const int* __restrict__ far_ptr, float4* __restrict__ pos, int4* __restrict__ info,
                               ulonglong2* __restrict__ mask) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const unsigned long long key = keys[k];
  const int a = (int)(unsigned int)key;
  const int cell = cell_of[a].x;
  const int s = xstart[cell], e = xstart[cell + 1];
  int d = s;
  for (int m = s; m < e; m++) d += keys[m] < key ? 1 : 0;
  float4 q = xyzq[a];
  q.x = wrap_coord(q.x, p.box[0], p.inv_box[0]);
  q.y = wrap_coord(q.y, p.box[1], p.inv_box[1]);
  q.z = wrap_coord(q.z, p.box[2], p.inv_box[2]);
  pos[d] = q;
  info[d] = make_int4(vdwtype[a], glob[a], a, far_ptr[a + 1] > far_ptr[a] ? 1 : 0);
  mask[d] = win[a];
}

// ---------------------------------------------------------------------------------------------
// Pairs
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ bool far_excluded(const int* __restrict__ far_ptr, const int* __restrict__ far_idx,
                                             int i, int gj) {
  for (int k = far_ptr[i]; k < far_ptr[i + 1]; k++)
    if (far_idx[k] == gj) return true;
  return false;
}

// d - n L for the image number n = field - 1 (field in 0..2), n made a double by placing the field in
// the low bits of 1.5 * 2^52.
__device__ __forceinline__ double shift_image(double d, int field, double box) {
  const double n = __dadd_rn(__hiloint2double(0x43380000, field), -6755399441055745.0);
  return __fma_rn(-n, box, d);
}

// Two FP32 values in one 64-bit register and packed arithmetic on them (sm_100).
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  return (unsigned long long)(unsigned int)__float_as_int(b) << 32 | (unsigned int)__float_as_int(a);
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Predicated 8-byte shared-memory store (an if around it costs three branch instructions).
__device__ __forceinline__ void store_if_less(float a, float b, unsigned int addr, int x, int y) {
  asm volatile("{\n .reg .pred p;\n setp.lt.f32 p, %0, %1;\n @p st.shared.v2.b32 [%2], {%3, %4};\n}" ::"f"(a), "f"(b),
               "r"(addr), "r"(x), "r"(y)
               : "memory");
}

// One warp per cluster of 8 atoms consecutive along x in a column (a compact block at liquid
// density) and slice of its column rows.  Each column in reach contributes the x interval that the
// cluster's bounding box can reach at that column's distance, once per periodic image.  The cheap
// pass takes the intervals' atoms in blocks of 32 (lane = candidate), tests each against the 8 atoms
// in FP32 with a slightly widened cutoff and queues the hits per atom in shared memory; when a queue
// fills (or at the end), lanes 4 i .. 4 i + 3 take atom i's hits in whole rounds and run the pair
// terms in FP64 from the exact FP32 geometry: cutoff, exclusions, forces rounded once to 2^-40 and
// summed in int64 in registers (exact: no accumulation error and no dependence on the order).  FP64
// because an atom's net force is a small difference of large pair forces, where the few-ulp error of
// FP32 pair terms reaches ~1e-5 kcal/mol/A.
// STD: vdW (square table) and Ewald (table) both on, the flags known at compile time.
template <bool EV, bool STD>
__global__ void __launch_bounds__(kWarps * 32, kPairCtas) k_direct_pairs(
    const __grid_constant__ Params p, const int* __restrict__ nclus, const int2* __restrict__ clusters,
    const int* __restrict__ xstart, const float4* __restrict__ pos, const int4* __restrict__ info,
    const ulonglong2* __restrict__ mask, const int* __restrict__ far_ptr, const int* __restrict__ far_idx,
    const float2* __restrict__ vdwp, int calc_energy, int calc_virial, int stride, long long* __restrict__ force,
    long long* __restrict__ acc, int* __restrict__ next_task) {
  extern __shared__ double2 sh_dyn[];   // Ewald quintics (with EV: F and E of an interval together), then vdW table
  constexpr int kEntry = EV ? 6 : 3;    // double2 per interval
  float2* const sh_vdw = reinterpret_cast<float2*>(sh_dyn + kEntry * p.tab_n);
  for (int k = threadIdx.x; k < kEntry * p.tab_n; k += blockDim.x)
    sh_dyn[k] = __ldg(p.tab + (EV ? k : k + k / 3 * 3));
  __shared__ int2 sh_queue[kWarps][kCluster][kQueue + 1];   // j and its image (2 bits per axis)
  __shared__ ulonglong2 sh_xy[kWarps][kCluster / 2];        // the cluster's coordinates, atoms in pairs
  __shared__ unsigned long long sh_z[kWarps][kCluster / 2];
  static_assert(sizeof(sh_queue) + sizeof(sh_xy) + sizeof(sh_z) == kPairShared, "what square_types counts");
  if (p.square)
    for (int k = threadIdx.x; k < p.ntype * p.ntype; k += blockDim.x) sh_vdw[k] = vdw_c6c12(vdwp, k / p.ntype, k % p.ntype);
  __syncthreads();
  const unsigned kFull = 0xffffffffu;
  const int kNoImage = 1 | 1 << 2 | 1 << 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & 3;
  const unsigned below = (1u << lane) - 1u;
  const unsigned int queues = (unsigned int)__cvta_generic_to_shared(&sh_queue[warp][0][0]);
  const bool vdw_on = p.vdw != PME_VDW_NONE;
  const int ncy = p.nc[1], ncz = p.nc[2], nbx = p.nc[0];
  const int spany = 2 * p.reach[0] + 1, spanz = 2 * p.reach[1] + 1;
  const float wy = p.box[1] / (float)ncy, wz = p.box[2] / (float)ncz;
  const int ntask = *nclus * p.slices;
  long long ev = 0, ee = 0;
  long long wv[6] = {0, 0, 0, 0, 0, 0};   // virial at 2^32: each task's FP64 partials folded in (exact)
  // tasks differ in cost: warps take them one at a time from a counter
  for (;;) {
    int task = 0;
    if (lane == 0) task = atomicAdd(next_task, 1);
    task = __shfl_sync(kFull, task, 0);
    if (task >= ntask) break;
    const int slice = task % p.slices;
    const int2 cl = clusters[task / p.slices];
    const int cy = cl.y % ncy, cz = cl.y / ncy;
    const int i = cl.x + (lane >> 2);
    const bool act = i < xstart[(size_t)cl.y * (nbx + 1) + nbx];
    const float nan = __int_as_float(0x7fffffff);
    const float4 pi = act ? pos[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int4 ii = act ? info[i] : make_int4(0, 0, 0, 0);
    const ulonglong2 mi = act ? mask[i] : make_ulonglong2(0ull, 0ull);
    // idle lanes: NaN coordinates, which no candidate's distance passes
    float lo[3] = {act ? pi.x : nan, act ? pi.y : nan, act ? pi.z : nan}, hi[3] = {lo[0], lo[1], lo[2]};
    __syncwarp();
    if (sub == 0) {
      const int h = (lane >> 2) & 1;
      float* xy = reinterpret_cast<float*>(&sh_xy[warp][lane >> 3]);
      xy[h] = lo[0];
      xy[2 + h] = lo[1];
      reinterpret_cast<float*>(&sh_z[warp][lane >> 3])[h] = lo[2];
    }
    // bounding box of the cluster's atoms (fminf / fmaxf pass the NaN of idle lanes over)
#pragma unroll
    for (int d = 4; d < 32; d <<= 1)
#pragma unroll
      for (int c = 0; c < 3; c++) {
        lo[c] = fminf(lo[c], __shfl_xor_sync(kFull, lo[c], d));
        hi[c] = fmaxf(hi[c], __shfl_xor_sync(kFull, hi[c], d));
      }
    __syncwarp();
    RoundedSum ax, ay, az;              // force sums at 2^40
    int terms = 0;                      // terms added by add_rounded
    int cnt[kCluster];                  // queued hits per atom (the same on every lane)
#pragma unroll
    for (int q = 0; q < kCluster; q++) cnt[q] = 0;
    double w0 = 0.0, w1 = 0.0, w2 = 0.0, w3 = 0.0, w4 = 0.0, w5 = 0.0;   // this task's, in a fixed order
    // this slice's columns, in groups of 32 (lane = column), once per x image
    const int kend = spany * (spanz * (slice + 1) / p.slices);
    int kcol = spany * (spanz * slice / p.slices) - 32, img = 1;
    int col_js = 0, col_excl = 0, col_image = 0;   // this lane's column: first atom, offset in the group
    int at = 0, total = 0;                         // candidates of the group: done, all
    for (;;) {
      while (at >= total && kcol < kend) {
        // the next group of columns or x image (images -1 and +1 only where that side of the box is near)
        if (++img > 1) {
          img = -1;
          kcol += 32;
          if (kcol >= kend) break;
        }
        const float shx = (float)img * p.box[0];
        const int k = kcol + lane;
        int len = 0;
        if (k < kend) {
          const int oy = cy + k % spany - p.reach[0], oz = cz + k / spany - p.reach[1];
          const float ylo = (float)oy * wy, zlo = (float)oz * wz;
          const float gy = fmaxf(0.0f, fmaxf(ylo - hi[1], lo[1] - (ylo + wy)) - p.marg);
          const float gz = fmaxf(0.0f, fmaxf(zlo - hi[2], lo[2] - (zlo + wz)) - p.marg);
          const float rr = p.cut2 - gy * gy - gz * gz;
          const float r = sqrtf(fmaxf(rr, 0.0f)) + p.marg;
          const float a = lo[0] - r, b = hi[0] + r;
          if (rr > 0.0f && (img == 0 || (img < 0 ? a < p.marg : b > p.box[0] - p.marg))) {
            int y = oy, z = oz, iy = 1, iz = 1;
            if (y < 0) { y += ncy; iy = 0; } else if (y >= ncy) { y -= ncy; iy = 2; }
            if (z < 0) { z += ncz; iz = 0; } else if (z >= ncz) { z -= ncz; iz = 2; }
            col_image = (img + 1) | iy << 2 | iz << 4;
            const int* xs = xstart + (size_t)(z * ncy + y) * (nbx + 1);
            col_js = xs[cell_of_wrapped(a - shx, p.inv_box[0], nbx)];
            len = xs[cell_of_wrapped(b - shx, p.inv_box[0], nbx) + 1] - col_js;
          }
        }
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += t;
        }
        col_excl = incl - len;
        total = __shfl_sync(kFull, incl, 31);
        at = 0;
      }
      const bool last = at >= total;
      if (!last) {
        // this lane's candidate: the last column whose offset is not beyond it (empty columns share
        // the next one's offset and are passed over)
        const int want = at + lane;
        int c = 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const int t = __shfl_sync(kFull, col_excl, c + o);
          if (t <= want) c += o;
        }
        const int j = __shfl_sync(kFull, col_js, c) + want - __shfl_sync(kFull, col_excl, c);
        const int jimg = __shfl_sync(kFull, col_image, c);
        float bx = nan, by = nan, bz = nan;
        if (want < total) {
          const float4 pj = __ldg(&pos[j]);
          bx = pj.x; by = pj.y; bz = pj.z;
          if (jimg != kNoImage) {
            bx += (float)((jimg & 3) - 1) * p.box[0];
            by += (float)(((jimg >> 2) & 3) - 1) * p.box[1];
            bz += (float)((jimg >> 4) - 1) * p.box[2];
          }
        }
        const unsigned long long bx2 = pack2(-bx, -bx), by2 = pack2(-by, -by), bz2 = pack2(-bz, -bz);
#pragma unroll
        for (int h = 0; h < kCluster / 2; h++) {
          const ulonglong2 xy = sh_xy[warp][h];
          const unsigned long long dx = add2(xy.x, bx2), dy = add2(xy.y, by2), dz = add2(sh_z[warp][h], bz2);
          const unsigned long long r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
#pragma unroll
          for (int g = 0; g < 2; g++) {
            const int q = 2 * h + g;
            const float d2 = __int_as_float((int)(g ? r2 >> 32 : r2));
            const unsigned m = __ballot_sync(kFull, d2 < p.cut2);
            store_if_less(d2, p.cut2, queues + 8 * (q * (kQueue + 1) + cnt[q] + __popc(m & below)), j, jimg);
            cnt[q] += __popc(m);
          }
        }
        at += 32;
      }
      int most = cnt[0];
#pragma unroll
      for (int q = 1; q < kCluster; q++) most = max(most, cnt[q]);
      if (!last && most <= kQueue - 32) continue;
      // pair terms, from the end of each atom's queue, 4 hits per atom and round: everything at the
      // end, else what every atom can fill, or what the fullest queue needs to take a block more
      __syncwarp();
      int mine = cnt[0];
#pragma unroll
      for (int q = 1; q < kCluster; q++) mine = (lane >> 2) == q ? cnt[q] : mine;
      const int least = __reduce_min_sync(kFull, act ? mine : kQueue);
      const int rounds = last ? (most + 3) >> 2 : max(least >> 2, (most - (kQueue - 32) + 3) >> 2);
      const int2* const queue = &sh_queue[warp][lane >> 2][0];
      const double qi = kCcelec * (double)pi.w;
      const float2* const vrow = sh_vdw + ii.x * p.ntype;
      for (int e = mine - 1 - sub, k = 0; k < rounds; k++, e -= 4) {
        bool ok = e >= 0;
        const int2 it = ok ? queue[e] : make_int2(0, kNoImage);
        const float4 pj = __ldg(&pos[it.x]);
        const int2 tj = __ldg(reinterpret_cast<const int2*>(&info[it.x]));   // type, global index
        double dx = (double)pi.x - (double)pj.x, dy = (double)pi.y - (double)pj.y, dz = (double)pi.z - (double)pj.z;
        const unsigned w = (unsigned)(tj.y - ii.y + 64);
        if (it.y != kNoImage || w < 128u || ii.w != 0) {
          dx = shift_image(dx, it.y & 3, p.boxd[0]);
          dy = shift_image(dy, (it.y >> 2) & 3, p.boxd[1]);
          dz = shift_image(dz, it.y >> 4, p.boxd[2]);
          if (w < 128u) {   // exclusions
            if (((w < 64u ? mi.x : mi.y) >> (w & 63u)) & 1ull) ok = false;
          } else if (ii.w != 0 && ok) {
            ok = !far_excluded(far_ptr, far_idx, ii.z, tj.y);
          }
        }
        const double r2 = dx * dx + dy * dy + dz * dz;
        ok = ok && r2 < p.roff2d;
        const double qq = qi * (double)pj.w;
        float2 cc = make_float2(0.0f, 0.0f);
        if (STD) cc = vrow[tj.x];
        else if (vdw_on) cc = p.square ? vrow[tj.x] : vdw_c6c12(vdwp, ii.x, tj.x);
        double uv = 0.0, ue = 0.0, f = 0.0;
        bool slow = false;
        // Ewald: the interval is the exponent and leading bits of r^2, t its offset from the middle
        const int hi_s = __double2hiint(r2);
        const unsigned at_s = (unsigned)(hi_s >> kTabShift) - (0x40000000u >> kTabShift);
        if (STD || p.tab_n > 0) {
          const double t = r2 - __hiloint2double((hi_s & -(1 << kTabShift)) | 1 << (kTabShift - 1), 0);
          const double2* const c = sh_dyn + kEntry * (at_s < (unsigned)p.tab_n ? at_s : 0u);
          f = qq * quintic(c, t);
          if (EV) ue = qq * quintic(c + 3, t);
        }
        if (STD || p.elec != PME_ELEC_NONE) slow = at_s >= (unsigned)p.tab_n;
        if (STD || vdw_on) {
          const double sinv = reciprocal(r2);
          f = __fma_rn(vdw_terms_f64<EV>(r2, sinv, cc, p, uv), sinv, f);
        }
        f = ok ? f : 0.0;
        if (EV) {
          uv = ok ? uv : 0.0;
          ue = ok ? ue : 0.0;
          slow = slow || !(fabs(uv) < 262144.0) || !(fabs(ue) < 262144.0);
        }
        // |f| r < 1024 unless f's high word (sign off) reaches 1024 / roff's
        slow = ok && (slow || (__double2hiint(f) & 0x7fffffff) >= p.big_hi);
        double fx = f * dx, fy = f * dy, fz = f * dz;
        // rint(v 2^40) by one addition where |v| 2^40 < 2^51: the integer is the sum's low bits
        if (!slow) {
          ax.add_rounded(__fma_rn(fx, 1099511627776.0, kRoundMagic));
          ay.add_rounded(__fma_rn(fy, 1099511627776.0, kRoundMagic));
          az.add_rounded(__fma_rn(fz, 1099511627776.0, kRoundMagic));
          terms++;
          if (EV) {
            const long long bits = __double_as_longlong(kRoundMagic);
            ev += __double_as_longlong(__fma_rn(uv, 4294967296.0, kRoundMagic)) - bits;
            ee += __double_as_longlong(__fma_rn(ue, 4294967296.0, kRoundMagic)) - bits;
          }
        } else {   // outside the table, or a large (or non-finite) term: rounded by conversion
          f = pair_terms_f64(r2, qq, cc, p, uv, ue);
          fx = f * dx;
          fy = f * dy;
          fz = f * dz;
          ax.add(__double2ll_rn(fx * 1099511627776.0));
          ay.add(__double2ll_rn(fy * 1099511627776.0));
          az.add(__double2ll_rn(fz * 1099511627776.0));
          if (EV) {
            ev += __double2ll_rn(uv * 4294967296.0);
            ee += __double2ll_rn(ue * 4294967296.0);
          }
        }
        if (EV) {
          w0 -= fx * dx; w1 -= fx * dy; w2 -= fx * dz;
          w3 -= fy * dy; w4 -= fy * dz; w5 -= fz * dz;
        }
      }
#pragma unroll
      for (int q = 0; q < kCluster; q++) cnt[q] = max(0, cnt[q] - 4 * rounds);
      __syncwarp();
      if (last) break;
    }
    // the 4 lanes of an atom join their sums; one lane per component adds it to the force array
    unsigned long long fx = ax.total(terms), fy = ay.total(terms), fz = az.total(terms);
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
      fx += __shfl_xor_sync(kFull, fx, d);
      fy += __shfl_xor_sync(kFull, fy, d);
      fz += __shfl_xor_sync(kFull, fz, d);
    }
    if (act && sub < 3)
      atomicAdd((unsigned long long*)&force[ii.z + (size_t)sub * stride], sub == 0 ? fx : (sub == 1 ? fy : fz));
    if (EV) {
      wv[0] += __double2ll_rn(w0 * 4294967296.0); wv[1] += __double2ll_rn(w1 * 4294967296.0);
      wv[2] += __double2ll_rn(w2 * 4294967296.0); wv[3] += __double2ll_rn(w3 * 4294967296.0);
      wv[4] += __double2ll_rn(w4 * 4294967296.0); wv[5] += __double2ll_rn(w5 * 4294967296.0);
    }
  }
  if (EV && calc_energy) {
    ev = warp_sum_ll(ev);
    ee = warp_sum_ll(ee);
    if (lane == 0) {
      atomicAdd((unsigned long long*)&acc[kAccVdw], (unsigned long long)ev);
      atomicAdd((unsigned long long*)&acc[kAccElec], (unsigned long long)ee);
    }
  }
  if (EV && calc_virial) {
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const long long sv = warp_sum_ll(wv[q]);
      if (lane == 0) atomicAdd((unsigned long long*)&acc[kAccVir + q], (unsigned long long)sv);
    }
  }
}

// 1-4 lists: one thread per (i, j, ishift, kind) entry, kind 1 = inclusion, 2 = exclusion.  Both
// atoms' forces by int64 atomics; energies and virial added twice (the doubled-sum convention).
__global__ void k_direct_14(const Params p, const int4* __restrict__ list, int nlist, const float4* __restrict__ xyzq,
                            const int* __restrict__ vdwtype, const float2* __restrict__ vdwp14, int calc_energy,
                            int calc_virial, int stride, long long* __restrict__ force, long long* __restrict__ acc) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  long long e[3] = {0, 0, 0};
  float w[6] = {0, 0, 0, 0, 0, 0};
  if (k < nlist) {
    const int4 L = list[k];
    const int i = L.x, j = L.y;
    const int ish = L.z;
    const float4 a = xyzq[i], b = xyzq[j];
    const float sx = (float)(ish % 3 - 1) * p.box[0];
    const float sy = (float)((ish / 3) % 3 - 1) * p.box[1];
    const float sz = (float)(ish / 9 - 1) * p.box[2];
    const float dx = a.x - b.x + sx, dy = a.y - b.y + sy, dz = a.z - b.z + sz;
    const float r2 = dx * dx + dy * dy + dz * dz;
    const bool in14 = L.w == 1;
    const bool vdw = in14 && p.vdw != PME_VDW_NONE;
    float2 cc = make_float2(0.0f, 0.0f);
    if (vdw) cc = vdw_c6c12(vdwp14, vdwtype[i], vdwtype[j]);
    float u_vdw, u_elec;
    const float g = pair_terms(r2, (float)kCcelec * a.w * b.w, cc.x, cc.y, p, in14 ? 1 : 2, vdw, u_vdw, u_elec);
    const long long fxi = __float2ll_rn(g * dx * kForceScaleF);
    const long long fyi = __float2ll_rn(g * dy * kForceScaleF);
    const long long fzi = __float2ll_rn(g * dz * kForceScaleF);
    atomicAdd((unsigned long long*)&force[i], (unsigned long long)fxi);
    atomicAdd((unsigned long long*)&force[i + stride], (unsigned long long)fyi);
    atomicAdd((unsigned long long*)&force[i + 2 * (size_t)stride], (unsigned long long)fzi);
    atomicAdd((unsigned long long*)&force[j], (unsigned long long)(-fxi));
    atomicAdd((unsigned long long*)&force[j + stride], (unsigned long long)(-fyi));
    atomicAdd((unsigned long long*)&force[j + 2 * (size_t)stride], (unsigned long long)(-fzi));
    if (calc_energy) {
      if (in14) {
        e[0] = 2 * __float2ll_rn(u_vdw * kEnergyScale);
        e[1] = 2 * __float2ll_rn(u_elec * kEnergyScale);
      } else {
        e[2] = 2 * __float2ll_rn(u_elec * kEnergyScale);
      }
    }
    if (calc_virial) {
      w[0] = -g * dx * dx; w[1] = -g * dx * dy; w[2] = -g * dx * dz;
      w[3] = -g * dy * dy; w[4] = -g * dy * dz; w[5] = -g * dz * dz;
    }
  }
  const int lane = threadIdx.x & 31;
  if (calc_energy) {
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const long long s = warp_sum_ll(e[q]);
      if (lane == 0 && s != 0) atomicAdd((unsigned long long*)&acc[kAccVdw + q], (unsigned long long)s);
    }
  }
  if (calc_virial) {
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const long long s = warp_sum_ll(2 * __float2ll_rn(w[q] * kEnergyScale));
      if (lane == 0 && s != 0) atomicAdd((unsigned long long*)&acc[kAccVir + q], (unsigned long long)s);
    }
  }
}

}  // namespace direct
}  // namespace pme

using namespace pme;
using namespace pme::direct;

struct pme_direct {
  int device = 0;
  int sm_shared = 0;         // the device's shared memory per SM, bytes
  cudaStream_t stream = nullptr;
  bool configured = false;
  double box[3] = {0, 0, 0};
  double kappa = 0, roff = 0, ron = 0, e14fac = 1.0;
  int vdw_model = PME_VDW_VSH, elec_model = PME_ELEC_EWALD;
  // tables
  int ntype = 0, ntype14 = 0;
  float2* d_vdw = nullptr;
  float2* d_vdw14 = nullptr;
  int n_types = 0;           // atoms of the vdW type table, and its largest type
  int max_type = -1;
  int n_excl = 0;            // atoms of the exclusion tables
  int* d_vdwtype = nullptr;
  int* d_glob = nullptr;     // global (original) index of every coordinate
  ulonglong2* d_win = nullptr;
  int* d_far_ptr = nullptr;
  int* d_far_idx = nullptr;
  bool excl_set = false;
  double* d_tab = nullptr;   // Ewald table for the current kappa and roff
  int tab_n = 0;
  double tab_kappa = -1.0, tab_roff = -1.0;
  int4* d_list14 = nullptr;
  int n14 = 0;
  int max14 = -1;            // largest atom index in the 1-4 lists
  // per-call work space
  int cap_atoms = 0, cap_clusters = 0;
  size_t cap_cells = 0;
  char* d_atoms = nullptr;    // the block of the next six
  float4* d_pos = nullptr;
  int4* d_info = nullptr;
  ulonglong2* d_mask = nullptr;
  unsigned long long* d_keys = nullptr;
  int2* d_cell_of = nullptr;  // bin and slot of every atom
  int2* d_clusters = nullptr; // first atom and column
  int* d_count = nullptr;     // [atoms placed, clusters, pair-task counter, 0], then [cap_cells] counts
  int* d_xstart = nullptr;    // (in d_count's block) [cap_cells]: per column, its x bins and its end
  long long* d_acc = nullptr;  // kAccN
};

namespace {

int check_handle(const pme_direct* h) { return h ? PME_OK : fail(PME_EINVAL, "direct handle is NULL"); }

template <class T>
cudaError_t upload(T** dst, const T* src, size_t n, cudaStream_t s) {
  cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  if (*dst) cudaFree(*dst);
  *dst = nullptr;
  if (n == 0) return cudaSuccess;
  e = cudaMalloc(dst, n * sizeof(T));
  if (e == cudaSuccess) e = cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice);
  return e;
}

Params make_params(const pme_direct* h) {
  Params p;
  std::memset(&p, 0, sizeof(p));
  for (int d = 0; d < 3; d++) {
    p.box[d] = (float)h->box[d];
    p.inv_box[d] = (float)(1.0 / h->box[d]);
    p.boxd[d] = h->box[d];
  }
  p.kappa = (float)h->kappa;
  p.kappa2 = (float)(h->kappa * h->kappa);
  p.roff2 = (float)(h->roff * h->roff);
  p.ro6 = (float)std::pow(h->roff, -6.0);
  p.ro12 = (float)std::pow(h->roff, -12.0);
  p.ro18 = (float)std::pow(h->roff, -18.0);
  p.e14fac = (float)h->e14fac;
  p.vdw = h->vdw_model;
  p.elec = h->elec_model;
  p.ntype = h->ntype;
  const double big = 1024.0 / h->roff;
  long long big_bits;
  std::memcpy(&big_bits, &big, sizeof(big));
  p.big_hi = (int)(big_bits >> 32);
  p.kappad = h->kappa;
  p.roff2d = h->roff * h->roff;
  p.ro6d = std::pow(h->roff, -6.0);
  p.ro12d = std::pow(h->roff, -12.0);
  p.ro18d = std::pow(h->roff, -18.0);
  const double longest = std::max(h->box[0], std::max(h->box[1], h->box[2]));
  p.cut2 = p.roff2 * 1.00001f + (float)(1e-6 * longest * h->roff);
  p.marg = (float)(1e-5 + 1e-6 * longest);
  p.tab = reinterpret_cast<const double2*>(h->d_tab);
  p.tab_n = h->elec_model == PME_ELEC_NONE ? 0 : h->tab_n;
  return p;
}

// The Ewald table in device memory (close pairs, s < 2, use the formulas).  Every CTA copies it to its
// shared memory: 8 KB of F for roff = 9 A, 16 KB with E; three 16-byte loads and five FMAs per pair.
// 192,000 atoms, forces only, 730 us, error against 64 bits 6.9e-10; cubics on twice the intervals 722 us and
// 1.9e-9; polynomials over the whole range (26 coefficients fetched and 37 FP64 operations) a fifth slower.
int ensure_ewald(pme_direct* h) {
  if (h->elec_model == PME_ELEC_NONE) return PME_OK;
  if (h->tab_kappa == h->kappa && h->tab_roff == h->roff) return PME_OK;
  h->tab_kappa = -1.0;
  const std::vector<double> t = ewald_table(h->kappa, h->roff);
  cudaError_t e = upload(&h->d_tab, t.data(), t.size(), h->stream);
  if (e != cudaSuccess) return cuda_fail(e, "direct: Ewald table");
  h->tab_n = (int)(t.size() / (2 * kTabTerms));
  h->tab_kappa = h->kappa;
  h->tab_roff = h->roff;
  return PME_OK;
}

// Work space for n atoms in `c`: one block for the atoms' arrays, one for the cells' (few allocations: a
// first call on new sizes pays for each), with room for a somewhat larger box.
int ensure_work(pme_direct* h, int n, const Columns& c) {
  if (n <= h->cap_atoms && most_clusters(n, c) <= h->cap_clusters && c.cells() <= h->cap_cells) return PME_OK;
  const Columns room = room_columns(h->box, h->roff, n);
  const int nclus = std::max(most_clusters(n, c), most_clusters(n, room));
  const size_t ncell = std::max(c.cells(), room.cells());
  if (n > h->cap_atoms || nclus > h->cap_clusters) {
    cudaFree(h->d_atoms);
    h->d_atoms = nullptr;
    h->cap_atoms = h->cap_clusters = 0;
    const size_t m = (size_t)std::max(n, 1);
    const size_t per_atom = sizeof(float4) + sizeof(int4) + sizeof(ulonglong2) + sizeof(unsigned long long) + sizeof(int2);
    if (cudaMalloc(&h->d_atoms, m * per_atom + (size_t)nclus * sizeof(int2)) != cudaSuccess) {
      cudaGetLastError();
      return fail(PME_ENOMEM, "direct: atom work space");
    }
    h->d_pos = reinterpret_cast<float4*>(h->d_atoms);
    h->d_info = reinterpret_cast<int4*>(h->d_pos + m);
    h->d_mask = reinterpret_cast<ulonglong2*>(h->d_info + m);
    h->d_keys = reinterpret_cast<unsigned long long*>(h->d_mask + m);
    h->d_cell_of = reinterpret_cast<int2*>(h->d_keys + m);
    h->d_clusters = h->d_cell_of + m;
    h->cap_atoms = n;
    h->cap_clusters = nclus;
  }
  if (ncell > h->cap_cells) {
    cudaFree(h->d_count);
    h->d_count = h->d_xstart = nullptr;
    h->cap_cells = 0;
    if (cudaMalloc(&h->d_count, (2 * ncell + 4) * sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      return fail(PME_ENOMEM, "direct: cell work space");
    }
    h->d_xstart = h->d_count + 4 + ncell;
    h->cap_cells = ncell;
  }
  return PME_OK;
}

// Every build of the pair kernel may take all of the device's shared memory per CTA.  The limit belongs
// to the process, so it is only ever set to this one value: a handle that set it to what its own tables
// need could lower it between another thread's choice and launch.
cudaError_t configure_pair_kernels(int device) {
  int most = 0;
  cudaError_t e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  for (auto kern : {k_direct_pairs<true, true>, k_direct_pairs<false, true>, k_direct_pairs<true, false>, k_direct_pairs<false, false>}) {
    cudaFuncAttributes fa;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kern);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes);
  }
  return e;
}

// Exclusion windows of n atoms with no exclusions but themselves.
int self_exclusions(pme_direct* h, int n) {
  std::vector<ulonglong2> win((size_t)n, make_ulonglong2(0ull, 1ull));   // bit 64: offset 0
  std::vector<int> glob((size_t)n), ptr((size_t)n + 1, 0);
  for (int i = 0; i < n; i++) glob[i] = i;
  cudaError_t e = upload(&h->d_win, win.data(), win.size(), h->stream);
  if (e == cudaSuccess) e = upload(&h->d_glob, glob.data(), glob.size(), h->stream);
  if (e == cudaSuccess) e = upload(&h->d_far_ptr, ptr.data(), ptr.size(), h->stream);
  if (e == cudaSuccess) e = upload(&h->d_far_idx, (const int*)nullptr, 0, h->stream);
  return e == cudaSuccess ? PME_OK : cuda_fail(e, "direct: exclusions");
}

int upload_vdw(pme_direct* h, int nvdwparam, const float* hp, bool in14) {
  if (int rc = check_handle(h)) return rc;
  if (nvdwparam < 2 || (nvdwparam & 1) || !hp) return fail(PME_EINVAL, "vdwparam: need (c6, c12) pairs");
  const int npair = nvdwparam / 2;
  int ntype = 0;
  while ((ntype + 1) * (ntype + 2) / 2 <= npair) ntype++;
  if (ntype * (ntype + 1) / 2 != npair) return fail(PME_EINVAL, "vdwparam: not a packed lower triangle of types");
  if (ntype > kMaxTypes) return fail(PME_EUNSUPPORTED, "vdwparam: more than 200 vdW types");
  std::vector<float2> t((size_t)npair);
  for (int k = 0; k < npair; k++) t[k] = make_float2(6.0f * hp[2 * k], 12.0f * hp[2 * k + 1]);
  DeviceGuard dg(h->device);
  cudaError_t e = upload(in14 ? &h->d_vdw14 : &h->d_vdw, t.data(), t.size(), h->stream);
  if (e != cudaSuccess) return cuda_fail(e, "vdwparam: upload");
  (in14 ? h->ntype14 : h->ntype) = ntype;
  return PME_OK;
}

}  // namespace

extern "C" {

int pme_direct_create(void* stream, pme_direct** out) {
  if (!out) return fail(PME_EINVAL, "out is NULL");
  *out = nullptr;
  pme_direct* h = new (std::nothrow) pme_direct();
  if (!h) return fail(PME_ENOMEM, "host allocation failed");
  cudaError_t e = cudaGetDevice(&h->device);
  h->stream = (cudaStream_t)stream;
  if (e == cudaSuccess) e = configure_pair_kernels(h->device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&h->sm_shared, cudaDevAttrMaxSharedMemoryPerMultiprocessor, h->device);
  if (e == cudaSuccess && cudaMalloc(&h->d_acc, kAccN * sizeof(long long)) != cudaSuccess) e = cudaErrorMemoryAllocation;
  if (e == cudaSuccess) e = cudaMemset(h->d_acc, 0, kAccN * sizeof(long long));
  if (e != cudaSuccess) {
    cudaGetLastError();
    cudaFree(h->d_acc);
    delete h;
    return cuda_fail(e, "direct: create");
  }
  *out = h;
  return PME_OK;
}

int pme_direct_destroy(pme_direct* h) {
  if (!h) return PME_OK;
  DeviceGuard dg(h->device);
  cudaStreamSynchronize(h->stream);
  for (void* p : {(void*)h->d_vdw, (void*)h->d_vdw14, (void*)h->d_vdwtype, (void*)h->d_glob, (void*)h->d_win,
                  (void*)h->d_far_ptr, (void*)h->d_far_idx, (void*)h->d_list14, (void*)h->d_tab, (void*)h->d_atoms,
                  (void*)h->d_count, (void*)h->d_acc})
    if (p) cudaFree(p);
  delete h;
  return PME_OK;
}

int pme_direct_set_stream(pme_direct* h, void* stream) {
  if (int rc = check_handle(h)) return rc;
  h->stream = (cudaStream_t)stream;
  return PME_OK;
}

int pme_direct_setup(pme_direct* h, double boxx, double boxy, double boxz, double kappa, double roff,
                     double ron, double e14fac, int vdw_model, int elec_model) {
  if (int rc = check_handle(h)) return rc;
  if (vdw_model != PME_VDW_VSH && vdw_model != PME_VDW_NONE)
    return fail(PME_EUNSUPPORTED, "direct: only the VDW_VSH (and NONE) vdW model is built");
  if (elec_model != PME_ELEC_EWALD && elec_model != PME_ELEC_NONE)
    return fail(PME_EUNSUPPORTED, "direct: only the EWALD (and NONE) electrostatics model is built");
  if (!(kappa >= 0.0) || !std::isfinite(kappa) || !std::isfinite(e14fac) || !std::isfinite(ron))
    return fail(PME_EINVAL, "direct: kappa, ron and e14fac must be finite (kappa >= 0)");
  h->kappa = kappa;
  h->roff = roff;
  h->ron = ron;
  h->e14fac = e14fac;
  h->vdw_model = vdw_model;
  h->elec_model = elec_model;
  h->configured = false;
  if (int rc = pme_direct_set_box_size(h, boxx, boxy, boxz)) return rc;
  h->configured = true;
  return PME_OK;
}

int pme_direct_set_box_size(pme_direct* h, double boxx, double boxy, double boxz) {
  if (int rc = check_handle(h)) return rc;
  const double b[3] = {boxx, boxy, boxz};
  for (double v : b)
    if (!(v > 0.0) || !std::isfinite(v)) return fail(PME_EINVAL, "direct: box edges must be finite and positive");
  if (!(h->roff > 0.0) || 2.0 * h->roff > std::min(boxx, std::min(boxy, boxz)))
    return fail(PME_EINVAL, "direct: roff must be positive and at most half the shortest box edge");
  for (int d = 0; d < 3; d++) h->box[d] = b[d];
  return PME_OK;
}

int pme_direct_set_vdwparam(pme_direct* h, int nvdwparam, const float* hp) { return upload_vdw(h, nvdwparam, hp, false); }
int pme_direct_set_vdwparam14(pme_direct* h, int nvdwparam, const float* hp) { return upload_vdw(h, nvdwparam, hp, true); }

int pme_direct_set_vdwtype(pme_direct* h, int ncoord, const int* hv) {
  if (int rc = check_handle(h)) return rc;
  if (ncoord < 0 || (ncoord > 0 && !hv)) return fail(PME_EINVAL, "vdwtype: bad arguments");
  int mx = -1;
  for (int i = 0; i < ncoord; i++) {
    if (hv[i] < 0) return fail(PME_EINVAL, "vdwtype: negative type");
    mx = std::max(mx, hv[i]);
  }
  DeviceGuard dg(h->device);
  cudaError_t e = upload(&h->d_vdwtype, hv, (size_t)ncoord, h->stream);
  if (e != cudaSuccess) return cuda_fail(e, "vdwtype: upload");
  h->n_types = ncoord;
  h->max_type = mx;
  return PME_OK;
}

int pme_direct_set_exclusions(pme_direct* h, int ncoord, const int* iblo14, const int* inb14, const int* loc2glo) {
  if (int rc = check_handle(h)) return rc;
  if (ncoord < 0 || (ncoord > 0 && !iblo14)) return fail(PME_EINVAL, "exclusions: bad arguments");
  const int n = ncoord;
  std::vector<int> glob((size_t)n), glo2loc((size_t)n, -1);
  for (int i = 0; i < n; i++) {
    const int g = loc2glo ? loc2glo[i] : i;
    if (g < 0 || g >= n || glo2loc[g] >= 0) return fail(PME_EINVAL, "exclusions: loc2glo is not a permutation");
    glob[i] = g;
    glo2loc[g] = i;
  }
  std::vector<ulonglong2> win((size_t)n, make_ulonglong2(0ull, 1ull));   // bit 64: the atom itself
  std::vector<std::vector<int>> far((size_t)n);
  auto add = [&](int ga, int gb) {   // exclude gb from ga's list (global indices)
    const int i = glo2loc[ga];
    const int k = gb - ga + 64;
    if (k >= 0 && k < 128) {
      if (k < 64) win[i].x |= 1ull << k;
      else win[i].y |= 1ull << (k - 64);
    } else {
      far[i].push_back(gb);
    }
  };
  int prev = 0;
  for (int ga = 0; ga < n; ga++) {
    const int end = iblo14[ga];
    if (end < prev || (end > prev && !inb14)) return fail(PME_EINVAL, "exclusions: iblo14 must be non-decreasing");
    for (int k = prev; k < end; k++) {
      const int gb = std::abs(inb14[k]) - 1;
      if (gb < 0 || gb >= n) return fail(PME_EINVAL, "exclusions: inb14 entry out of range");
      add(ga, gb);
      add(gb, ga);
    }
    prev = end;
  }
  std::vector<int> ptr((size_t)n + 1, 0), idx;
  for (int i = 0; i < n; i++) {
    std::sort(far[i].begin(), far[i].end());
    far[i].erase(std::unique(far[i].begin(), far[i].end()), far[i].end());
    ptr[i + 1] = ptr[i] + (int)far[i].size();
    idx.insert(idx.end(), far[i].begin(), far[i].end());
  }
  DeviceGuard dg(h->device);
  cudaError_t e = upload(&h->d_win, win.data(), win.size(), h->stream);
  if (e == cudaSuccess) e = upload(&h->d_glob, glob.data(), glob.size(), h->stream);
  if (e == cudaSuccess) e = upload(&h->d_far_ptr, ptr.data(), ptr.size(), h->stream);
  if (e == cudaSuccess) e = upload(&h->d_far_idx, idx.data(), idx.size(), h->stream);
  if (e != cudaSuccess) return cuda_fail(e, "exclusions: upload");
  h->excl_set = true;
  h->n_excl = n;
  return PME_OK;
}

int pme_direct_set_14_list(pme_direct* h, int nin14, int nex14, const int* in14, const int* ex14) {
  if (int rc = check_handle(h)) return rc;
  if (nin14 < 0 || nex14 < 0 || (nin14 > 0 && !in14) || (nex14 > 0 && !ex14)) return fail(PME_EINVAL, "14 list: bad arguments");
  std::vector<int4> L;
  L.reserve((size_t)nin14 + nex14);
  int mx = -1;
  for (int pass = 0; pass < 2; pass++) {
    const int* s = pass == 0 ? in14 : ex14;
    const int n = pass == 0 ? nin14 : nex14;
    for (int k = 0; k < n; k++) {
      const int i = s[3 * k], j = s[3 * k + 1], ish = s[3 * k + 2];
      if (i < 0 || j < 0 || ish < 0 || ish > 26) return fail(PME_EINVAL, "14 list: bad entry");
      L.push_back(make_int4(i, j, ish, pass + 1));
      mx = std::max(mx, std::max(i, j));
    }
  }
  DeviceGuard dg(h->device);
  cudaError_t e = upload(&h->d_list14, L.data(), L.size(), h->stream);
  if (e != cudaSuccess) return cuda_fail(e, "14 list: upload");
  h->n14 = (int)L.size();
  h->max14 = mx;
  return PME_OK;
}

int pme_direct_calc_force(pme_direct* h, const void* xyzq, int ncoord, int calc_energy, int calc_virial, int stride,
                          long long* force) {
  if (int rc = check_handle(h)) return rc;
  if (!h->configured) return fail(PME_ESTATE, "direct: setup first");
  if (ncoord < 0 || (ncoord > 0 && (!xyzq || !force)) || stride < ncoord) return fail(PME_EINVAL, "direct: bad arguments");
  if (ncoord == 0) return PME_OK;
  if (h->vdw_model != PME_VDW_NONE) {
    if (!h->d_vdw || !h->d_vdwtype) return fail(PME_ESTATE, "direct: set vdwparam and vdwtype first");
    if (h->n_types != ncoord) return fail(PME_EINVAL, "direct: ncoord differs from the vdW types' count");
    if (h->max_type >= h->ntype) return fail(PME_EINVAL, "direct: a vdW type is beyond the parameter table");
  }
  if (h->excl_set && h->n_excl != ncoord) return fail(PME_EINVAL, "direct: ncoord differs from the exclusions' count");
  DeviceGuard dg(h->device);
  if (!h->excl_set) {   // no exclusion lists: every atom excludes only itself
    if (int rc = self_exclusions(h, ncoord)) return rc;
    h->excl_set = true;
    h->n_excl = ncoord;
  }
  if (h->n_types != ncoord) {   // no vdW: every atom type 0
    std::vector<int> zeros((size_t)ncoord, 0);
    cudaError_t e = upload(&h->d_vdwtype, zeros.data(), zeros.size(), h->stream);
    if (e != cudaSuccess) return cuda_fail(e, "direct: types");
    h->n_types = ncoord;
    h->max_type = 0;
  }
  if (int rc = ensure_ewald(h)) return rc;
  Params p = make_params(h);
  if (h->vdw_model == PME_VDW_NONE) p.ntype = 0;
  const Columns cols = plan_columns(h->box, h->roff, ncoord);
  for (int d = 0; d < 3; d++) p.nc[d] = cols.nc[d];
  p.reach[0] = p.reach[1] = cols.reach;
  const int ncol = cols.count();
  const size_t ncell = cols.cells();
  if (int rc = ensure_work(h, ncoord, cols)) return rc;
  cudaStream_t s = h->stream;
  int* const count = h->d_count + 4;
  cudaError_t e = cudaMemsetAsync(h->d_count, 0, (ncell + 4) * sizeof(int), s);
  if (e != cudaSuccess) return cuda_fail(e, "direct: clear counts");
  const int nb = (ncoord + 255) / 256;
  k_direct_cell<<<nb, 256, 0, s>>>((const float4*)xyzq, ncoord, p, h->d_cell_of, count);
  k_direct_columns<<<(ncol + 3) / 4, 128, 0, s>>>(p, count, ncol, h->d_count, h->d_xstart, h->d_clusters);
  k_direct_fill<<<nb, 256, 0, s>>>(h->d_cell_of, ncoord, p, (const float4*)xyzq, h->d_xstart, h->d_keys);
  k_direct_order<<<nb, 256, 0, s>>>(p, ncoord, h->d_keys, h->d_cell_of, h->d_xstart, (const float4*)xyzq, h->d_vdwtype,
                                    h->d_glob, h->d_win, h->d_far_ptr, h->d_pos, h->d_info, h->d_mask);
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
  const bool ev = calc_energy || calc_virial;
  const size_t table = (size_t)p.tab_n * (ev ? 2 : 1) * kTabTerms * sizeof(double);
  p.square = square_types(p.ntype, table, h->sm_shared) ? 1 : 0;
  const bool std_terms = h->vdw_model != PME_VDW_NONE && p.square && p.tab_n > 0;
  auto kern = std_terms ? (ev ? k_direct_pairs<true, true> : k_direct_pairs<false, true>)
                        : (ev ? k_direct_pairs<true, false> : k_direct_pairs<false, false>);
  const size_t smem = table + (size_t)(p.square ? p.ntype * p.ntype : 0) * sizeof(float2);
  // one wave of resident CTAs; their warps draw the tasks from a counter.  Few clusters: more tasks
  // each, so that the last ones to finish are short
  int occ = 1;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kWarps * 32, smem);
  if (e != cudaSuccess) return cuda_fail(e, "direct: occupancy");
  const long long warps = (long long)sms * std::max(occ, 1) * kWarps;
  const long long nclus = ncoord / kCluster + 1;
  p.slices = (int)std::max<long long>(1, std::min<long long>((kTasksPerWarp * warps + nclus - 1) / nclus, 2 * p.reach[1] + 1));
  const long long tasks = (long long)most_clusters(ncoord, cols) * p.slices;
  const int pg = (int)std::max<long long>(1, std::min<long long>((tasks + kWarps - 1) / kWarps, warps / kWarps));
  kern<<<pg, kWarps * 32, smem, s>>>(p, h->d_count + 1, h->d_clusters, h->d_xstart, h->d_pos, h->d_info, h->d_mask,
                                     h->d_far_ptr, h->d_far_idx, h->d_vdw, calc_energy ? 1 : 0, calc_virial ? 1 : 0,
                                     stride, force, h->d_acc, h->d_count + 2);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "direct: launch");
  return PME_OK;
}

int pme_direct_calc_14_force(pme_direct* h, const void* xyzq, int calc_energy, int calc_virial, int stride,
                             long long* force) {
  if (int rc = check_handle(h)) return rc;
  if (!h->configured) return fail(PME_ESTATE, "direct: setup first");
  if (h->n14 == 0) return PME_OK;
  if (!xyzq || !force || stride < 1) return fail(PME_EINVAL, "direct 14: bad arguments");
  if (h->max14 >= stride) return fail(PME_EINVAL, "direct 14: a list entry is beyond the force stride");
  if (h->max14 >= std::max(h->n_types, h->n_excl))
    return fail(PME_EINVAL, "direct 14: a list entry is beyond the atoms (set vdwtype or exclusions first)");
  if (h->vdw_model != PME_VDW_NONE) {
    if (!h->d_vdw14 || !h->d_vdwtype) return fail(PME_ESTATE, "direct 14: set vdwparam14 and vdwtype first");
    if (h->max14 >= h->n_types) return fail(PME_EINVAL, "direct 14: a list entry is beyond the vdW types");
    if (h->max_type >= h->ntype14) return fail(PME_EINVAL, "direct 14: a vdW type is beyond the 1-4 table");
  }
  DeviceGuard dg(h->device);
  const Params p = make_params(h);
  k_direct_14<<<(h->n14 + 255) / 256, 256, 0, h->stream>>>(p, h->d_list14, h->n14, (const float4*)xyzq, h->d_vdwtype,
                                                           h->d_vdw14, calc_energy ? 1 : 0, calc_virial ? 1 : 0,
                                                           stride, force, h->d_acc);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "direct 14: launch");
  return PME_OK;
}

int pme_direct_clear_energy_virial(pme_direct* h) {
  if (int rc = check_handle(h)) return rc;
  DeviceGuard dg(h->device);
  cudaError_t e = cudaMemsetAsync(h->d_acc, 0, kAccN * sizeof(long long), h->stream);
  return e == cudaSuccess ? PME_OK : cuda_fail(e, "direct: clear");
}

int pme_direct_get_energy_virial(pme_direct* h, double* e_vdw, double* e_elec, double* e_excl, double* vir9) {
  if (int rc = check_handle(h)) return rc;
  DeviceGuard dg(h->device);
  long long a[kAccN];
  cudaError_t e = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) e = cudaMemcpy(a, h->d_acc, sizeof(a), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "direct: read energies");
  const double sc = 0.5 / 4294967296.0;   // doubled sums at 2^32
  if (e_vdw) *e_vdw = (double)a[kAccVdw] * sc;
  if (e_elec) *e_elec = (double)a[kAccElec] * sc;
  if (e_excl) *e_excl = (double)a[kAccExcl] * sc;
  if (vir9) {
    const double w[6] = {(double)a[3] * sc, (double)a[4] * sc, (double)a[5] * sc,
                         (double)a[6] * sc, (double)a[7] * sc, (double)a[8] * sc};
    const double t[9] = {w[0], w[1], w[2], w[1], w[3], w[4], w[2], w[4], w[5]};
    for (int k = 0; k < 9; k++) vir9[k] = t[k];
  }
  return PME_OK;
}

}  // extern "C"
