// Tiled evaluation of molecules too large for one block's shared memory (the 2,000-5,000-atom
// chains of the large-system workload), with the same pair functors, valence code and integer
// accumulation as the fused kernel: the two paths agree to FP32 rounding (the compiler may
// contract a few operations differently in the two kernels) and each is bit-identical from run
// to run.
//
// Every 32 x 32 tile of every tiled molecule is a warp task. kTiledPrepare lays the atoms out as
// pair records (coordinates as hi / lo float pairs, the passes' payloads); a warp copies the
// tile's two blocks of records into its own slice of shared memory, walks the tile with the fused
// kernel's functors, and adds its accumulators to global integer arrays. Passes that need the
// whole molecule finished first (effective radii after pass 1, the chain-rule prefactor after pass
// 2) are separate per-atom kernels. Warps take contiguous runs of tiles, so a warp's energy sums
// change molecule rarely and flush once per molecule.
#include <cuda_runtime.h>

#include "launch.cuh"
#include "unit_eval.cuh"
#include "tile_tasks.cuh"

namespace sb {

namespace {

constexpr int kStageSlots = 2 * kTile;    // block I in slots 0-31, block J in slots 32-63

// Valence terms reading atoms straight from the global fixed-point arrays and adding forces and
// energies with global integer atomics (one molecule per block row of the launch grid)
struct GlobalValence {
  const DevSynthesis &d;
  int sys;
  int first;     // the molecule's first atom
  __device__ GlobalValence(const DevSynthesis &d_in, int sys_in) :
      d(d_in), sys(sys_in), first(d_in.atom_start[sys_in]) {}
  __device__ __forceinline__ const int* starts(int kind) const {
    return (kind == kBondTerms) ? d.bond_start :
           (kind == kAnglTerms) ? d.angl_start : d.dihe_start;
  }
  __device__ __forceinline__ int chunks(int kind) const {
    return (starts(kind)[sys + 1] - starts(kind)[sys] + 31) / 32;
  }
  __device__ __forceinline__ int begin(int before) const {
    return dealFrom((threadIdx.x >> 5) + blockIdx.y * (blockDim.x >> 5), chunkStride(), before);
  }
  __device__ __forceinline__ int chunkStride() const { return (blockDim.x >> 5) * gridDim.y; }
  __device__ __forceinline__ ValenceTerm term(int kind, int c, int lane) const {
    const int index = starts(kind)[sys] + 32 * c + lane;
    return ValenceTerm{0, index, index < starts(kind)[sys + 1]};
  }
  __device__ __forceinline__ int slot0(int) const { return first; }
  __device__ __forceinline__ float3 part(int i, bool high) const {
    float3 h, l;
    splitCoordinate(static_cast<double>(d.xcrd[i]) * d.inv_gpos_scale, &h.x, &l.x);
    splitCoordinate(static_cast<double>(d.ycrd[i]) * d.inv_gpos_scale, &h.y, &l.y);
    splitCoordinate(static_cast<double>(d.zcrd[i]) * d.inv_gpos_scale, &h.z, &l.z);
    return high ? h : l;
  }
  __device__ __forceinline__ float3 hi(int i) const { return part(i, true); }
  __device__ __forceinline__ float3 lo(int i) const { return part(i, false); }
  __device__ __forceinline__ void force(int i, float fx, float fy, float fz, float scale) const {
    atomicAdd(reinterpret_cast<unsigned long long*>(&d.xfrc[i]),
              static_cast<unsigned long long>(__float2ll_rn(fx * scale)));
    atomicAdd(reinterpret_cast<unsigned long long*>(&d.yfrc[i]),
              static_cast<unsigned long long>(__float2ll_rn(fy * scale)));
    atomicAdd(reinterpret_cast<unsigned long long*>(&d.zfrc[i]),
              static_cast<unsigned long long>(__float2ll_rn(fz * scale)));
  }
  __device__ __forceinline__ void energy(int, int slot, float e, float scale) const {
    const long long v = warpSum(__float2ll_rn(e * scale));
    if ((threadIdx.x & 31) == 0 && v != 0) {
      atomicAdd(&d.energies[sys * kNrgStride + slot], static_cast<unsigned long long>(v));
    }
  }
  __device__ __forceinline__ double3 pos64(int i) const {
    return make_double3(static_cast<double>(d.xcrd[i]) * d.inv_gpos_scale,
                        static_cast<double>(d.ycrd[i]) * d.inv_gpos_scale,
                        static_cast<double>(d.zcrd[i]) * d.inv_gpos_scale);
  }
  __device__ __forceinline__ void force64(int i, double fx, double fy, double fz,
                                          float scale) const {
    const double s = static_cast<double>(scale);
    atomicAdd(reinterpret_cast<unsigned long long*>(&d.xfrc[i]),
              static_cast<unsigned long long>(__double2ll_rn(fx * s)));
    atomicAdd(reinterpret_cast<unsigned long long*>(&d.yfrc[i]),
              static_cast<unsigned long long>(__double2ll_rn(fy * s)));
    atomicAdd(reinterpret_cast<unsigned long long*>(&d.zfrc[i]),
              static_cast<unsigned long long>(__double2ll_rn(fz * s)));
  }
  __device__ __forceinline__ void energy64(int, int slot, double e, float scale) const {
    const long long v = warpSum(__double2ll_rn(e * static_cast<double>(scale)));
    if ((threadIdx.x & 31) == 0 && v != 0) {
      atomicAdd(&d.energies[sys * kNrgStride + slot], static_cast<unsigned long long>(v));
    }
  }
  __device__ __forceinline__ float2 clash(int) const {
    const int cycle = (d.clash_cycle != nullptr) ? d.clash_cycle[sys] : -1;
    return clashScaled(d.clash_distance, d.clash_ratio, d.clash_cycles, cycle);
  }
};

// Valence terms of tiled molecule blockIdx.x (plus mol_begin), chunks spread over blockIdx.y
template <bool FORCE, bool ENERGY, bool CLASH>
__global__ void __launch_bounds__(256)
kTiledValence(const DevSynthesis d, const DevTiled t, int mol_begin) {
  gridWait();
  valenceTerms<FORCE, ENERGY, GlobalValence, CLASH>(
      d, GlobalValence(d, t.systems[mol_begin + blockIdx.x]));
}

// Component c (0: first pair, 2: second pair) of padded atom gi in record array arr
__device__ __forceinline__ float &blockValue(const DevTiled &t, int gi, int arr, int c) {
  const int r = (gi / kTile) * kBlockRecords + arr * kRecords + (gi & (kRecords - 1));
  return reinterpret_cast<float*>(t.records)[4 * static_cast<size_t>(r) + c + slotHalf(gi)];
}

// One warp per 32 padded positions of the tiled atoms [atom_begin, atom_end): cleared psi and dE/dR
// sums, the atoms' records and the block's box.  The tile passes meet every block some hundred
// times; converting its fixed-point coordinates once and copying 16-byte records from then on, in
// place of the conversion per tile, and knowing which tiles are plain is what this buys:
// 32 chains of 2,000-5,000 atoms, force + energy with copies, 1,600 -> 1,318 us.
__global__ void __launch_bounds__(256)
kTiledPrepare(const DevSynthesis d, const DevTiled t, int atom_begin, int atom_end) {
  gridWait();
  const int lane = threadIdx.x & 31;
  for (int q = atom_begin + blockIdx.x * blockDim.x + threadIdx.x; q < atom_end;
       q += gridDim.x * blockDim.x) {
    int sysid, a;
    const int gi = tiledAtom(d, t, q, &sysid, &a);
    const bool real = a < d.atom_count[sysid];
    t.psi_acc[gi] = 0;
    t.de_acc[gi] = 0;
    // padding (of a molecule's last block alone) sits far from everything and from other padding
    float3 hi = make_float3(5000.0f + 16.0f * static_cast<float>(lane), 0.0f, 0.0f);
    float3 lo = make_float3(0.0f, 0.0f, 0.0f);
    float srho = 0.0f, rho = 1.0f, charge = 0.0f, code = 0.0f;
    if (real) {
      splitCoordinate(static_cast<double>(d.xcrd[gi]) * d.inv_gpos_scale, &hi.x, &lo.x);
      splitCoordinate(static_cast<double>(d.ycrd[gi]) * d.inv_gpos_scale, &hi.y, &lo.y);
      splitCoordinate(static_cast<double>(d.zcrd[gi]) * d.inv_gpos_scale, &hi.z, &lo.z);
      const int ty = d.lj_idx[gi];
      srho = d.srho[gi];
      rho = d.rho[gi];
      charge = d.charge[gi];
      code = __int_as_float((ty * d.lj_ntypes[sysid]) | (ty << 16));
    }
    blockValue(t, gi, kRecXY, 0) = hi.x;
    blockValue(t, gi, kRecXY, 2) = hi.y;
    blockValue(t, gi, kRecXYLo, 0) = lo.x;
    blockValue(t, gi, kRecXYLo, 2) = lo.y;
    blockValue(t, gi, kRecZ1, 0) = hi.z;
    blockValue(t, gi, kRecZ1, 2) = srho;
    blockValue(t, gi, kRecZ1Lo, 0) = lo.z;
    blockValue(t, gi, kRecZ1Lo, 2) = rho;
    blockValue(t, gi, kRecZ2, 0) = hi.z;
    blockValue(t, gi, kRecZ2, 2) = charge;
    blockValue(t, gi, kRecZ2Lo, 0) = lo.z;
    blockValue(t, gi, kRecZ2Lo, 2) = 1.0f;     // effective radius: kTiledAtoms
    blockValue(t, gi, kRecG2, 0) = 1.0f;
    blockValue(t, gi, kRecG2, 2) = code;
    blockValue(t, gi, kRecG3, 0) = 0.0f;
    blockValue(t, gi, kRecG3, 2) = 0.0f;       // dE/dR: kTiledChain
    // the box of the block's atoms
    float3 low = real ? hi : make_float3(1.0e30f, 1.0e30f, 1.0e30f);
    float3 top = real ? hi : make_float3(-1.0e30f, -1.0e30f, -1.0e30f);
    float smax = srho, rmax = real ? rho : 0.0f;
    for (int o = 16; o > 0; o >>= 1) {
      low.x = fminf(low.x, __shfl_xor_sync(kFullMask, low.x, o));
      low.y = fminf(low.y, __shfl_xor_sync(kFullMask, low.y, o));
      low.z = fminf(low.z, __shfl_xor_sync(kFullMask, low.z, o));
      top.x = fmaxf(top.x, __shfl_xor_sync(kFullMask, top.x, o));
      top.y = fmaxf(top.y, __shfl_xor_sync(kFullMask, top.y, o));
      top.z = fmaxf(top.z, __shfl_xor_sync(kFullMask, top.z, o));
      smax = fmaxf(smax, __shfl_xor_sync(kFullMask, smax, o));
      rmax = fmaxf(rmax, __shfl_xor_sync(kFullMask, rmax, o));
    }
    if (lane == 0) {
      t.boxes[2 * (gi / kTile)] = make_float4(0.5f * (low.x + top.x), 0.5f * (low.y + top.y),
                                              0.5f * (low.z + top.z), smax);
      t.boxes[2 * (gi / kTile) + 1] = make_float4(0.5f * (top.x - low.x), 0.5f * (top.y - low.y),
                                                  0.5f * (top.z - low.z), rmax);
    }
  }
}

// Whether every pair of two blocks is at least kPlainDistance apart and beyond the reach of the
// near forms of the descreening (4 times the screened radius, overlapping spheres, the neck)
constexpr float kPlainDistance = 10.0f;

__device__ __forceinline__ bool tilePlain(const DevSynthesis &d, const DevTiled &t, int ia,
                                          int ja) {
  const float4 ci = t.boxes[2 * (ia / kTile)], hi = t.boxes[2 * (ia / kTile) + 1];
  const float4 cj = t.boxes[2 * (ja / kTile)], hj = t.boxes[2 * (ja / kTile) + 1];
  const float gx = fmaxf(fabsf(ci.x - cj.x) - hi.x - hj.x, 0.0f);
  const float gy = fmaxf(fabsf(ci.y - cj.y) - hi.y - hj.y, 0.0f);
  const float gz = fmaxf(fabsf(ci.z - cj.z) - hi.z - hj.z, 0.0f);
  float reach = fmaxf(kPlainDistance, 4.0f * fmaxf(ci.w, cj.w));
  reach = fmaxf(reach, fmaxf(hi.w + cj.w, hj.w + ci.w));
  if (d.neck_size > 0) {
    reach = fmaxf(reach, hi.w + hj.w + 2.0f * d.gb_offset + d.neck_cut);
  }
  reach += 0.05f;     // the boxes hold the hi parts (2^-11 A) and are rounded
  return gx * gx + gy * gy + gz * gz > reach * reach;
}

// Copy one tile's records into a warp's slice: block I in slots 0-31, block J in 32-63 (a diagonal
// tile stages block I only).  ia, ja: the blocks' first padded atoms
template <int PASS>
__device__ __forceinline__ void stageTile(const DevSynthesis &d, const DevTiled &t,
                                          const UnitSmem &v, int ia, int ja, bool diag, int lane) {
  // lanes 0-15 take block I's records, lanes 16-31 block J's
  const int half = lane >> 4;
  if (half == 0 || !diag) {
    const float4* src = t.records +
                        static_cast<size_t>((half == 0 ? ia : ja) / kTile) * kBlockRecords +
                        (lane & 15);
    v.pa[lane] = src[kRecXY * kRecords];
    v.pc[lane] = src[kRecXYLo * kRecords];
    v.pb[lane] = src[(PASS == 2 ? kRecZ2 : kRecZ1) * kRecords];
    v.pd[lane] = src[(PASS == 2 ? kRecZ2Lo : kRecZ1Lo) * kRecords];
    if (PASS != 1) {
      v.pg[lane] = src[(PASS == 2 ? kRecG2 : kRecG3) * kRecords];
    }
  }
  if (PASS != 2 && d.neck_size > 0) {
    v.neck[lane] = d.neck_idx[ia + lane];
    if (!diag) {
      v.neck[kTile + lane] = d.neck_idx[ja + lane];
    }
  }
  __syncwarp();
}

// A warp's slice of a tile kernel's shared memory
struct TileStage {
  float4 rec[kTiledWarps][5][kStageSlots / 2];
  int neck[kTiledWarps][kStageSlots];
  unsigned short late[kTiledWarps][kLateEntries];
};

__device__ __forceinline__ UnitSmem warpView(TileStage &m, const float2* lj) {
  UnitSmem v{};
  const int w = threadIdx.x >> 5;
  v.pa = m.rec[w][0];
  v.pb = m.rec[w][1];
  v.pc = m.rec[w][2];
  v.pd = m.rec[w][3];
  v.pg = m.rec[w][4];
  v.neck = m.neck[w];
  v.late = m.late[w];
  v.lj = const_cast<float2*>(lj);
  return v;
}

__device__ __forceinline__ void addGlobal(long long* acc, float v) {
  atomicAdd(reinterpret_cast<unsigned long long*>(acc),
            static_cast<unsigned long long>(__float2ll_rn(v)));
}

// GB pass 1 over tiles [tile_begin, tile_end)
template <bool NECK>
__global__ void __launch_bounds__(256, 4)
kTiledRadii(const DevSynthesis d, const DevTiled t, int tile_begin, int tile_end) {
  gridWait();
  __shared__ TileStage stage;
  const int lane = threadIdx.x & 31;
  const float ps = static_cast<float>(1 << kPsiBits);
  int first, last;
  warpTileRange(t, tile_begin, tile_end, &first, &last);
  const UnitSmem v = warpView(stage, d.ljab);
  RadiiPass<false, NECK, true> p(v, d);
  for (int g = first; g < last; g++) {
    const int m = tiledOwner(t, g);
    const int sysid = t.systems[m];
    int I, J;
    const TileInfo ti = tiledTileInfo(d, sysid, g - t.tile_prefix[m], &I, &J);
    const int ia = d.atom_start[sysid] + I * kTile, ja = d.atom_start[sysid] + J * kTile;
    stageTile<1>(d, t, v, ia, ja, ti.diag, lane);
    const TileWalk w = tileWalk(ti, lane);
    p.begin(ti, w);
    if (!ti.diag && tilePlain(d, t, ia, ja)) {
      walkTile<true>(p, ti, w, lane);
    }
    else {
      walkTile(p, ti, w, lane);
    }
    const float vi = iShare(p.psi_i, w);
    const float vj = jShare(p.psi_j, w, lane);
    if (ownsAtom(ti, w, lane)) {
      addGlobal(&t.psi_acc[ia + lane], vi * ps);
    }
    const int jl = sharedAtom(w, lane);
    if (jl < ti.nj) {
      addGlobal(&t.psi_acc[ja + jl], vj * ps);
    }
    p.finish(ti, lane, v.late, nullptr, [&](int slot, float x) {
      addGlobal(&t.psi_acc[slot < kTile ? ia + slot : ja + slot - kTile], x * ps);
    });
    __syncwarp();
  }
}

// Pass 2 (Coulomb + Lennard-Jones and GB pair terms) over tiles [tile_begin, tile_end)
template <bool FORCE, bool ENERGY, bool NB, bool GB, bool CLASH>
__global__ void __launch_bounds__(256, 3)
kTiledPair(const DevSynthesis d, const DevTiled t, int tile_begin, int tile_end) {
  gridWait();
  __shared__ TileStage stage;
  const int lane = threadIdx.x & 31;
  const float fs = d.frc_scale;
  const float es = d.nrg_scale;
  const float ds = static_cast<float>(1 << kDeijdaBits);
  int first, last;
  warpTileRange(t, tile_begin, tile_end, &first, &last);
  long long acc_elec = 0, acc_vdw = 0, acc_gb = 0;
  int acc_sys = -1;
  auto flush = [&]() {
    // per-tile energies rounded to the output grid (tileEnergy), the same value in every lane
    if (lane == 0 && acc_sys >= 0) {
      if (NB) {
        atomicAdd(&d.energies[acc_sys * kNrgStride + kElec],
                  static_cast<unsigned long long>(acc_elec));
        atomicAdd(&d.energies[acc_sys * kNrgStride + kVdw],
                  static_cast<unsigned long long>(acc_vdw));
      }
      if (GB) {
        atomicAdd(&d.energies[acc_sys * kNrgStride + kGb], static_cast<unsigned long long>(acc_gb));
      }
    }
    acc_elec = acc_vdw = acc_gb = 0;
  };
  for (int g = first; g < last; g++) {
    const int m = tiledOwner(t, g);
    const int sysid = t.systems[m];
    if (ENERGY && sysid != acc_sys) {
      flush();
      acc_sys = sysid;
    }
    int I, J;
    const TileInfo ti = tiledTileInfo(d, sysid, g - t.tile_prefix[m], &I, &J);
    const UnitSmem v = warpView(stage, d.ljab + d.lj_start[sysid]);
    const int ia = d.atom_start[sysid] + I * kTile, ja = d.atom_start[sysid] + J * kTile;
    stageTile<2>(d, t, v, ia, ja, ti.diag, lane);
    const TileWalk w = tileWalk(ti, lane);
    bool plain = !ti.diag && tilePlain(d, t, ia, ja);
    unsigned mask = 0u;
    if (NB) {
      const int midx = d.tile_mask_idx[d.tile_start[sysid] + ti.local];
      if (midx != 0) {
        mask = __ldg(&d.mask_pool[static_cast<size_t>(midx) * 32 + w.il]);
        plain = false;
      }
    }
    PairPass<FORCE, ENERGY, NB, GB, CLASH> p(v, d.kappa, d.inv_dielectric);
    float2 clash = make_float2(0.0f, 0.0f);
    if (CLASH) {
      const int cycle = (d.clash_cycle != nullptr) ? d.clash_cycle[sysid] : -1;
      clash = clashScaled(d.clash_distance, d.clash_ratio, d.clash_cycles, cycle);
    }
    p.begin(ti, w, mask, clash);
    if (!CLASH && plain) {
      walkTile<true>(p, ti, w, lane);
    }
    else {
      walkTile(p, ti, w, lane);
    }
    if (FORCE) {
      const float fxi = iShare(p.fxi, w), fyi = iShare(p.fyi, w), fzi = iShare(p.fzi, w);
      const float dei = GB ? iShare(p.dei, w) : 0.0f;
      const float fxj = jShare(p.fxj, w, lane), fyj = jShare(p.fyj, w, lane);
      const float fzj = jShare(p.fzj, w, lane);
      const float dej = GB ? jShare(p.dej, w, lane) : 0.0f;
      if (ownsAtom(ti, w, lane)) {
        const int gi = ia + lane;
        addGlobal(&d.xfrc[gi], fxi * fs);
        addGlobal(&d.yfrc[gi], fyi * fs);
        addGlobal(&d.zfrc[gi], fzi * fs);
        if (GB) {
          addGlobal(&t.de_acc[gi], dei * ds);
        }
      }
      const int jl = sharedAtom(w, lane);
      if (jl < ti.nj) {
        const int gj = ja + jl;
        addGlobal(&d.xfrc[gj], -fxj * fs);
        addGlobal(&d.yfrc[gj], -fyj * fs);
        addGlobal(&d.zfrc[gj], -fzj * fs);
        if (GB) {
          addGlobal(&t.de_acc[gj], dej * ds);
        }
      }
    }
    if (ENERGY) {
      if (NB) {
        acc_elec += tileEnergy(p.t_elec, es);
        acc_vdw += tileEnergy(p.t_vdw, es);
      }
      if (GB) {
        acc_gb += tileEnergy(p.t_gb, es);
      }
    }
    __syncwarp();
  }
  if (ENERGY) {
    flush();
  }
}

// Pass 3 (radius chain-rule forces) over tiles [tile_begin, tile_end)
template <bool NECK>
__global__ void __launch_bounds__(256, 4)
kTiledDeriv(const DevSynthesis d, const DevTiled t, int tile_begin, int tile_end) {
  gridWait();
  __shared__ TileStage stage;
  const int lane = threadIdx.x & 31;
  const float fs = d.frc_scale;
  int first, last;
  warpTileRange(t, tile_begin, tile_end, &first, &last);
  const UnitSmem v = warpView(stage, d.ljab);
  DerivPass<NECK> p(v, d);
  for (int g = first; g < last; g++) {
    const int m = tiledOwner(t, g);
    const int sysid = t.systems[m];
    int I, J;
    const TileInfo ti = tiledTileInfo(d, sysid, g - t.tile_prefix[m], &I, &J);
    const int ia = d.atom_start[sysid] + I * kTile, ja = d.atom_start[sysid] + J * kTile;
    stageTile<3>(d, t, v, ia, ja, ti.diag, lane);
    const TileWalk w = tileWalk(ti, lane);
    p.begin(ti, w);
    if (!ti.diag && tilePlain(d, t, ia, ja)) {
      walkTile<true>(p, ti, w, lane);
    }
    else {
      walkTile(p, ti, w, lane);
    }
    const auto add = [&](int gi, float fx, float fy, float fz) {
      addGlobal(&d.xfrc[gi], fx * fs);
      addGlobal(&d.yfrc[gi], fy * fs);
      addGlobal(&d.zfrc[gi], fz * fs);
    };
    const float fxi = iShare(p.fxi, w), fyi = iShare(p.fyi, w), fzi = iShare(p.fzi, w);
    const float fxj = jShare(p.fxj, w, lane), fyj = jShare(p.fyj, w, lane);
    const float fzj = jShare(p.fzj, w, lane);
    if (ownsAtom(ti, w, lane)) {
      add(ia + lane, -fxi, -fyi, -fzi);
    }
    const int jl = sharedAtom(w, lane);
    if (jl < ti.nj) {
      add(ja + jl, fxj, fyj, fzj);
    }
    p.finish(ti, lane, v.late, [&](int slot, float fx, float fy, float fz) {
      add(slot < kTile ? ia + slot : ja + slot - kTile, fx, fy, fz);
    });
    __syncwarp();
  }
}

// Effective radii and GB self terms of the tiled atoms [atom_begin, atom_end) (padded
// positions; a warp's 32 positions always belong to one molecule)
template <bool FORCE, bool ENERGY, bool WS>
__global__ void __launch_bounds__(256)
kTiledAtoms(const DevSynthesis d, const DevTiled t, int atom_begin, int atom_end) {
  gridWait();
  const float inv_ps = 1.0f / static_cast<float>(1 << kPsiBits);
  const float ds = static_cast<float>(1 << kDeijdaBits);
  for (int q = atom_begin + blockIdx.x * blockDim.x + threadIdx.x; q < atom_end;
       q += gridDim.x * blockDim.x) {
    int sysid, a;
    const int gi = tiledAtom(d, t, q, &sysid, &a);
    float e_self = 0.0f;
    float egbi = 1.0f;
    if (a < d.atom_count[sysid]) {
      const double psi = static_cast<double>(t.psi_acc[gi]) * static_cast<double>(inv_ps);
      egbi = effectiveRadius(d, gi, psi);
      float self_de;
      e_self = gbSelfTerm(d, d.charge[gi], egbi, &self_de);
      if (FORCE) {
        addGlobal(&t.de_acc[gi], self_de * ds);
      }
      if (WS) {
        d.born_radii[gi] = egbi;
        d.psi[gi] = __double2ll_rn(static_cast<double>(psi) * d.psi_out_scale);
        d.psi_ovrf[gi] = 0;
      }
    }
    blockValue(t, gi, kRecZ2Lo, 2) = egbi;
    blockValue(t, gi, kRecG2, 0) = 1.0f / egbi;
    if (ENERGY) {
      const long long v = warpSum(__float2ll_rn(e_self * d.nrg_scale));
      if ((threadIdx.x & 31) == 0 && v != 0) {
        atomicAdd(&d.energies[sysid * kNrgStride + kGb], static_cast<unsigned long long>(v));
      }
    }
  }
}

// Chain-rule prefactor of the tiled atoms' dE/dR sums
template <bool WS>
__global__ void __launch_bounds__(256)
kTiledChain(const DevSynthesis d, const DevTiled t, int atom_begin, int atom_end) {
  gridWait();
  const float inv_ds = 1.0f / static_cast<float>(1 << kDeijdaBits);
  const float inv_ps = 1.0f / static_cast<float>(1 << kPsiBits);
  for (int q = atom_begin + blockIdx.x * blockDim.x + threadIdx.x; q < atom_end;
       q += gridDim.x * blockDim.x) {
    int sysid, a;
    const int gi = tiledAtom(d, t, q, &sysid, &a);
    float sde = 0.0f;
    if (a < d.atom_count[sysid]) {
      sde = static_cast<float>(t.de_acc[gi]) * inv_ds;
      if (d.igb != 1) {
        const double psi = static_cast<double>(t.psi_acc[gi]) * static_cast<double>(inv_ps);
        sde *= obcChainFactor(d, gi, psi);
      }
      if (WS) {
        d.sumdeijda[gi] = __double2ll_rn(static_cast<double>(sde) * d.psi_out_scale);
        d.sumdeijda_ovrf[gi] = 0;
      }
    }
    blockValue(t, gi, kRecG3, 2) = sde;
  }
}

}  // namespace

// All requested terms of tiled molecules [mol_begin, mol_end)
cudaError_t launchTiled(const DevSynthesis &d, const DevTiled &t, const int* h_tile_prefix,
                        const int* h_atom_prefix, int mol_begin, int mol_end, int terms,
                        bool force, bool energy, bool workspace, int sm_count,
                        cudaStream_t stream, bool clash) {
  if (mol_end <= mol_begin) {
    return cudaSuccess;
  }
  const bool vale = (terms & 1) != 0;
  const bool nb = (terms & 2) != 0;
  const bool gb = ((terms & 4) != 0) && d.igb != 0;
  const int tb = h_tile_prefix[mol_begin], te = h_tile_prefix[mol_end];
  const int ab = h_atom_prefix[mol_begin], ae = h_atom_prefix[mol_end];
  const int tgrid = tileGrid(te - tb, sm_count);
  const int agrid = atomGrid(ae - ab, sm_count);
  const int nmol = mol_end - mol_begin;
  if (vale) {
    // four blocks a molecule when there are many; a lone molecule's chunks of 32 terms spread
    // over up to 32 blocks (one 2,500-atom chain: 23 us on 4 blocks, 10 on 32)
    int vrows = 2 * sm_count / nmol;
    vrows = vrows < 4 ? 4 : (vrows > 32 ? 32 : vrows);
    const dim3 vgrid(nmol, vrows);
#define SB_VALE_GO(F, E, C)                                                                    \
    launchAfter(kTiledValence<F, E, C>, vgrid, 256, 0, stream, d, t, mol_begin);
#define SB_VALE(C)                                                                             \
    if (force && energy) SB_VALE_GO(true, true, C)                                             \
    else if (force) SB_VALE_GO(true, false, C)                                                 \
    else SB_VALE_GO(false, true, C)
    if (clash) { SB_VALE(true) }
    else { SB_VALE(false) }
#undef SB_VALE
#undef SB_VALE_GO
  }
  if (nb || gb) {
    launchAfter(kTiledPrepare, agrid, 256, 0, stream, d, t, ab, ae);
  }
  if (gb) {
    if (d.neck_size > 0) launchAfter(kTiledRadii<true>, tgrid, 256, 0, stream, d, t, tb, te);
    else launchAfter(kTiledRadii<false>, tgrid, 256, 0, stream, d, t, tb, te);
#define SB_ATOMS(F, E) \
    if (workspace) launchAfter(kTiledAtoms<F, E, true>, agrid, 256, 0, stream, d, t, ab, ae); \
    else launchAfter(kTiledAtoms<F, E, false>, agrid, 256, 0, stream, d, t, ab, ae);
    if (force && energy) { SB_ATOMS(true, true) }
    else if (force) { SB_ATOMS(true, false) }
    else { SB_ATOMS(false, true) }
#undef SB_ATOMS
  }
  if (nb || gb) {
#define SB_PAIR_GO(F, E, NB, GB, C)                                                           \
    launchAfter(kTiledPair<F, E, NB, GB, C>, tgrid, 256, 0, stream, d, t, tb, te);
#define SB_PAIR(F, E, C)                                                                      \
    if (nb && gb) SB_PAIR_GO(F, E, true, true, C)                                             \
    else if (nb) SB_PAIR_GO(F, E, true, false, C)                                             \
    else SB_PAIR_GO(F, E, false, true, false)
    if (clash) {
      if (force && energy) { SB_PAIR(true, true, true) }
      else if (force) { SB_PAIR(true, false, true) }
      else { SB_PAIR(false, true, true) }
    }
    else {
      if (force && energy) { SB_PAIR(true, true, false) }
      else if (force) { SB_PAIR(true, false, false) }
      else { SB_PAIR(false, true, false) }
    }
#undef SB_PAIR
#undef SB_PAIR_GO
  }
  if (gb && force) {
    if (workspace) launchAfter(kTiledChain<true>, agrid, 256, 0, stream, d, t, ab, ae);
    else launchAfter(kTiledChain<false>, agrid, 256, 0, stream, d, t, ab, ae);
    if (d.neck_size > 0) launchAfter(kTiledDeriv<true>, tgrid, 256, 0, stream, d, t, tb, te);
    else launchAfter(kTiledDeriv<false>, tgrid, 256, 0, stream, d, t, tb, te);
  }
  return cudaGetLastError();
}

}  // namespace sb
