// Solvent-accessible surface area by sphere points, as STORMM's MM-GBSA application scores it
// (Potential/surface_area.tpp:28-161 with the Lennard-Jones radii of surface_area.tpp:163-173).
//
// FP64 throughout.  Each atom carries a sphere of points at its radius plus the probe; a point
// survives unless it lies strictly inside another atom's probe-enlarged sphere.  The reference
// bins atoms into cells of at least twice the largest probe-enlarged radius over the system's
// bounding box and tests a point of an atom in cell (i, j, k) only against atoms in cells i-1..i,
// j-1..j, k-1..k (its loop bounds stop below the upper neighbours); the kernels apply the same
// cell rule, so the surviving points are the same.  A system with no extent along an axis has no
// cells there and scores zero, as in the reference.  Point, displacement and distance arithmetic
// use round-to-nearest multiplies and adds without fused multiply-add, in the reference's order,
// so each point's verdict is the host's.
//
// Three launches: kSasaSetup (a block per system: box, cells, coordinates and reaches in double),
// kSasaAtoms (a warp per atom) and kSasaSum (a block per system, fixed order).  A warp first
// gathers the few tens of atoms that pass the cell rule and come within reach of its atom's
// sphere, 32 candidates a step, into shared memory, and then tests its points, one a lane,
// against that list alone.  Only atoms that can hide no point are left out, so no verdict
// changes.  Work is FP64 arithmetic on the lists (about 9 operations a test), where one block
// per system walked every atom of the system for every point from global memory, with an integer
// conversion per coordinate: one receptor of 500
// atoms, 31 poses of a 40-atom ligand and their complexes (18,480 atoms, 272 points each) 25,400
// us -> 140 us for the three launches.
#include <cuda_runtime.h>

#include "device_kits.h"

namespace sb {
namespace {

constexpr int kSasaThreads = 256;
constexpr int kSasaList = 96;             // spheres a warp lists before it tests them

__device__ __forceinline__ double blockReduce(double v, bool take_max, double* scratch) {
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, v, o);
    v = take_max ? fmax(v, w) : fmin(v, w);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = (lane < (kSasaThreads >> 5)) ? scratch[lane] : scratch[0];
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, v, o);
      v = take_max ? fmax(v, w) : fmin(v, w);
    }
    if (lane == 0) scratch[0] = v;
  }
  __syncthreads();
  const double out = scratch[0];
  __syncthreads();
  return out;
}

__device__ __forceinline__ int cellOf(double x, double origin, double width, int count) {
  int c = static_cast<int>(__ddiv_rn(__dsub_rn(x, origin), width));
  return c < 0 ? 0 : (c >= count ? count - 1 : c);
}

// Box and cells of one system a block: at (x, y, z, radius + probe) of every atom and its packed
// cell coordinates; shape 0: scored, 1: no extent along an axis (area 0), 2: not representable
__global__ void __launch_bounds__(kSasaThreads)
kSasaSetup(const long long* xcrd, const long long* ycrd, const long long* zcrd,
           double inv_gpos_scale, const int* atom_start, const int* atom_count,
           const double* radius, double probe, double4* at, int* cell, int* shape) {
  __shared__ double scratch[32];
  const int sys = blockIdx.x;
  const int base = atom_start[sys], n = atom_count[sys];
  double lo[3] = {1.0e300, 1.0e300, 1.0e300}, hi[3] = {-1.0e300, -1.0e300, -1.0e300};
  double rmax = 0.0;
  for (int i = threadIdx.x; i < n; i += kSasaThreads) {
    const double x[3] = {static_cast<double>(xcrd[base + i]) * inv_gpos_scale,
                         static_cast<double>(ycrd[base + i]) * inv_gpos_scale,
                         static_cast<double>(zcrd[base + i]) * inv_gpos_scale};
    const double r = radius[base + i];
    at[base + i] = make_double4(x[0], x[1], x[2], __dadd_rn(r, probe));
    for (int d = 0; d < 3; d++) {
      lo[d] = fmin(lo[d], x[d]);
      hi[d] = fmax(hi[d], x[d]);
    }
    rmax = fmax(rmax, r);
  }
  double origin[3], len[3];
  for (int d = 0; d < 3; d++) {
    origin[d] = blockReduce(lo[d], false, scratch);
    len[d] = __dsub_rn(blockReduce(hi[d], true, scratch), origin[d]);
  }
  rmax = blockReduce(rmax, true, scratch);
  const double min_width = 2.0 * __dadd_rn(rmax, probe);
  int count[3];
  double width[3];
  for (int d = 0; d < 3; d++) {
    count[d] = static_cast<int>(ceil(__ddiv_rn(len[d], min_width)));
    width[d] = __ddiv_rn(len[d], static_cast<double>(count[d]));
  }
  // more than 1,024 cells along an axis (an extent of kilometres) overflow the packed index
  const bool flat = count[0] == 0 || count[1] == 0 || count[2] == 0;
  const bool wide = count[0] > 1024 || count[1] > 1024 || count[2] > 1024;
  if (threadIdx.x == 0) shape[sys] = flat ? 1 : (wide ? 2 : 0);
  if (flat || wide) return;
  for (int i = threadIdx.x; i < n; i += kSasaThreads) {
    const double4 a = at[base + i];      // this thread's own store above
    const int cx = cellOf(a.x, origin[0], width[0], count[0]);
    const int cy = cellOf(a.y, origin[1], width[1], count[1]);
    const int cz = cellOf(a.z, origin[2], width[2], count[2]);
    cell[base + i] = (cz << 20) | (cy << 10) | cx;
  }
}

// Clear the alive bits of a lane's points (point first + 32 it + lane is bit it) that lie inside
// one of the count listed spheres (x, y, z, squared reach)
__device__ __forceinline__ unsigned testPoints(unsigned alive, int iters, int first, int lane,
                                               const double3* pts, double4 a,
                                               const double4* list, int count) {
  for (int it = 0; it < iters; it++) {
    bool live = ((alive >> it) & 1u) != 0u;
    if (!__any_sync(0xffffffffu, live)) continue;
    // dead lanes (points beyond the last among them) repeat the group's first point
    const double3 s = pts[live ? first + 32 * it + lane : first];
    const double px = __dadd_rn(a.x, __dmul_rn(s.x, a.w));
    const double py = __dadd_rn(a.y, __dmul_rn(s.y, a.w));
    const double pz = __dadd_rn(a.z, __dmul_rn(s.z, a.w));
    for (int e0 = 0; e0 < count; e0 += 4) {
      const int e1 = min(e0 + 4, count);
      for (int e = e0; e < e1; e++) {
        const double4 v = list[e];
        const double dx = __dsub_rn(px, v.x);
        const double dy = __dsub_rn(py, v.y);
        const double dz = __dsub_rn(pz, v.z);
        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)),
                                    __dmul_rn(dz, dz));
        live = live && !(d2 < v.w);
      }
      if (!__any_sync(0xffffffffu, live)) break;
    }
    if (!live) alive &= ~(1u << it);
  }
  return alive;
}

// One warp per atom; map: padded index of each atom without padding, stretch: the length of
// the longest sphere point (1 for unit vectors)
__global__ void __launch_bounds__(kSasaThreads)
kSasaAtoms(const double4* at, const int* cell, const int* shape, const int* map, int natom,
           const int* atom_start, const int* atom_count, int nsys, const double3* pts, int npts,
           double stretch, double* area) {
  __shared__ double4 lists[kSasaThreads / 32][kSasaList];
  const int lane = threadIdx.x & 31;
  double4* list = lists[threadIdx.x >> 5];
  const int q = (blockIdx.x * kSasaThreads + threadIdx.x) >> 5;
  if (q >= natom) return;
  const int gi = map[q];
  int lo = 0, hi = nsys - 1;             // the system that owns the atom
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (atom_start[mid] <= gi) lo = mid;
    else hi = mid - 1;
  }
  if (shape[lo] != 0) return;
  const int base = atom_start[lo], n = atom_count[lo];
  const double4 a = at[gi];
  const int cm = cell[gi];
  const int mx = cm & 1023, my = (cm >> 10) & 1023, mz = cm >> 20;
  int survivors = 0;
  for (int first = 0; first < npts; first += 1024) {
    const int here = min(1024, npts - first);
    const int iters = (here + 31) / 32;
    // bit it of a lane: point first + 32 it + lane, where there is one
    const int mine = (here - lane + 31) / 32;
    unsigned alive = (mine >= 32) ? 0xffffffffu : ((1u << mine) - 1u);
    int count = 0;
    for (int v0 = 0; v0 < n; v0 += 32) {
      const int v = v0 + lane;
      bool near = false;
      double4 b = make_double4(0.0, 0.0, 0.0, 0.0);
      if (v < n && base + v != gi) {
        const int cv = cell[base + v];
        const int vx = cv & 1023, vy = (cv >> 10) & 1023, vz = cv >> 20;
        if (vx <= mx && vx >= mx - 1 && vy <= my && vy >= my - 1 && vz <= mz && vz >= mz - 1) {
          b = at[base + v];
          const double dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
          const double far = fma(a.w, stretch, b.w);
          near = !(fma(dx, dx, fma(dy, dy, dz * dz)) > far * far * (1.0 + 1.0e-9));
        }
      }
      const unsigned took = __ballot_sync(0xffffffffu, near);
      if (near) {
        b.w = __dmul_rn(b.w, b.w);
        list[count + __popc(took & ((1u << lane) - 1u))] = b;
      }
      count += __popc(took);
      if (count > kSasaList - 32) {
        __syncwarp();
        alive = testPoints(alive, iters, first, lane, pts, a, list, count);
        __syncwarp();
        count = 0;
      }
    }
    __syncwarp();
    alive = testPoints(alive, iters, first, lane, pts, a, list, count);
    __syncwarp();
    survivors += __popc(alive);
  }
  for (int o = 16; o > 0; o >>= 1) survivors += __shfl_xor_sync(0xffffffffu, survivors, o);
  if (lane == 0) {
    // area per surviving point: (4 pi / npts) r^2
    const double patch = __ddiv_rn(4.0 * 3.141592653589793, static_cast<double>(npts));
    area[gi] = static_cast<double>(survivors) * __dmul_rn(__dmul_rn(patch, a.w), a.w);
  }
}

// A system's area from its atoms', in a fixed order
__global__ void __launch_bounds__(kSasaThreads)
kSasaSum(const double* area, const int* shape, const int* atom_start, const int* atom_count,
         double weight, double* out) {
  __shared__ double scratch[32];
  const int sys = blockIdx.x;
  if (shape[sys] != 0) {
    if (threadIdx.x == 0) {
      out[sys] = (shape[sys] == 1) ? 0.0 : __longlong_as_double(0x7ff8000000000000ll);
    }
    return;
  }
  const int base = atom_start[sys], n = atom_count[sys];
  double sum = 0.0;
  for (int i = threadIdx.x; i < n; i += kSasaThreads) sum += area[base + i];
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) scratch[warp] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int k = 0; k < (kSasaThreads >> 5); k++) total += scratch[k];
    out[sys] = total * weight;
  }
}

}  // namespace

// map: padded index of each of natom atoms; at, cell, area: per padded atom scratch, shape: per
// system; stretch: at least the length of the longest sphere point
cudaError_t launchSurfaceArea(const long long* xcrd, const long long* ycrd,
                              const long long* zcrd, double inv_gpos_scale,
                              const int* atom_start, const int* atom_count, int nsys,
                              const int* map, int natom, const double* radius,
                              const double3* pts, int npts, double stretch, double probe,
                              double weight, double4* at, int* cell, int* shape, double* area,
                              double* out, cudaStream_t stream) {
  if (nsys <= 0) return cudaSuccess;
  kSasaSetup<<<nsys, kSasaThreads, 0, stream>>>(xcrd, ycrd, zcrd, inv_gpos_scale, atom_start,
                                                atom_count, radius, probe, at, cell, shape);
  const int warps = kSasaThreads / 32;
  kSasaAtoms<<<(natom + warps - 1) / warps, kSasaThreads, 0, stream>>>(
      at, cell, shape, map, natom, atom_start, atom_count, nsys, pts, npts, stretch, area);
  kSasaSum<<<nsys, kSasaThreads, 0, stream>>>(area, shape, atom_start, atom_count, weight, out);
  return cudaGetLastError();
}

}  // namespace sb
