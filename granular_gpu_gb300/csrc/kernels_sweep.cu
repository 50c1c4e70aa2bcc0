// kernels_sweep.cu — the Jacobi contact sweep (compute_delta_pos,
// Solver.cu:361-401, with boundary_constraint :272-307 and
// particles_constraint :309-359), race-free.
//
// Semantics.  The reference's scatters into delta_pos[j] are overwritten by
// each thread's final `delta_pos[i] = dp` when the whole grid is resident,
// while its constraint-count increments all land.  This kernel produces that
// outcome with gathers only:
//   delta_i = thread i's own corrections, accumulated in the reference's
//             loop order (27 cells; walls, then particles, by index);
//   n_i     = contacts i finds + particles that find i.
// "j finds i" is decided by i: i's binning cell lies in the stencil of
// trunc(x*_j / L) (the contact test itself is symmetric).  When it does not,
// i hands the count to j through s_extra (rare: only where predicted and
// binned cells disagree).
//
// Pruning.  Cells that cannot hold a partner (farther than r_i + r_max plus
// the largest displacement since binning) are skipped; they contribute
// nothing, so the sum and its order are unchanged.
//
// Kernels.  The default keeps per-particle contact lists across the sweeps
// of a substep: a group of lanes to a particle in small systems
// (k_sweep_group), a thread to a particle in large ones
// (k_sweep_nlist_build / k_sweep_nlist_keep, with short rebuild queues and
// overlong lists left to groups, k_sweep_rest); without lists, k_sweep_list
// scans the 27 cells; k_sweep is the pruned one-thread-per-particle scan the
// autotuner may pick where lists do not pay.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "common.cuh"

namespace gg {

// The arguments of the sweep kernels.  No pointer is __restrict__: the kernels
// with contact lists are launched chained (pdl_wait), at every size.  Against
// plain launches with __restrict__ above 400,000 particles: the 8.4 M column
// 28.5 to 28.0 ms a substep, a batch of 643,000 4.52 to 4.37 for two, 8 M
// particles falling free of each other 4.21 and 4.31.  The kernels without
// lists measured the same either way.
struct SweepArgs {
  Grid g;
  int n;
  int it;
  const float4* xs;
  const float* inv_m;
  const uint32_t* keys;
  const int32_t* cs;
  const int32_t* bcs;
  const float4* bpos;
  float4* delta;
  int32_t* s_extra;
  DevScalars* scal;
  double brad;  // boundary radius (double literal 0.01)
  double fcap;  // friction cap (double literal 0.8)
  float fcapf;  // the same as float
  float bradf;  // brad as float (conservative cuts only)
  const float2* window;  // per cell coordinate: positions whose query cell is within one of it
  float minr;  // floor of the particle radius against walls (0.01f)
  // contact candidate lists (the default sweep)
  int32_t* nl_idx;
  int4* nl_meta;
  float* nl_acc;
  int32_t* nl_queue;
  int32_t* nl_over;  // particles with long lists, left to the groups
  int32_t* nl_long;  // the long lists, kLongMax entries each
  int long_rows;
  size_t li_row, li_step;  // entry k of particle i's list: nl_idx[i * li_row + k * li_step]
  const uint32_t* cell_inc;  // the last sweep's increments
  uint32_t* cell_clear;  // the table of this sweep's, to be cleared (two take turns), or null
  ResidualSlot* res;  // residual mode: this sweep's penetrations (kernels with bit 2 of MM)
  int group_queue;  // queues up to this length are rebuilt by groups
  float skin;
  float eabs;  // bound on the rounding of one position update
  UDiv div_yz, div_z;  // division by ny * nz and by nz (binning cell of a key)
  // batched scenes: scene of a particle = its x* slab, floor(x / width);
  // each scene has its own friction cap (null: a.fcap for every particle)
  const float* scene_fcap;
  float scene_inv_w;
  int n_scenes;
  // configured mode (gg_params.contact_law): substep-start positions for
  // the friction law and its output, the summed friction corrections and
  // their count (both null with the reference's law)
  const float4* pos0;
  float4* fdelta;
};

// The kernels' template argument MM: bit 0 the math mode (0 CUDA's
// functions, 1 rounded once from double), bit 1 the contact law (0 the
// reference's, 1 Coulomb friction), bit 2 the residual mode (also sum the
// penetrations at x*, which the candidates of the sweep hold all of).

// Which of the three cell columns [c-1, c, c+1] along one axis can hold a
// partner: bit k set for offset k-1.  Cells are [cL, (c+1)L) in binning
// coordinates; a partner binned there is within R of x.
__device__ __forceinline__ unsigned axis_mask(float x, int q, float L, float R) {
  unsigned m = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float lo = (float)(q + k - 1) * L;
    const float hi = (float)(q + k) * L;
    // NaN in x or R leaves the column in (never prunes)
    if (!(x < lo - R) && !(x > hi + R)) m |= 1u << k;
  }
  return m;
}

// Everything one target particle needs for its sweep.
struct Target {
  float3 x;
  float rc, rb;
  float Bf;       // 0.01 + r_b as float arithmetic gives it (conservative cuts only)
  float Bru;      // Bd rounded up to float: (double)d < Bd  <=>  d < Bru for every float d
  float capBru;   // (r_b + 0.01) * 0.8 in double, rounded up to float (same use)
  float Bcut;     // conservative float cut for the wall test
  float inv_m;
  int3 q;         // query cell trunc(x*/L)
  float3 wlo, whi; // partners at wlo <= x*_j < whi (every axis) find this particle
  unsigned pm[3], bm[3];
  float fcapf;    // friction cap factor (0.8 in the reference; per scene in a batch), as float
  float3 x0;      // position at the substep's start (Coulomb law only)
};

// One contact's share of the corrections: dp of the position, df of the
// friction target (Coulomb law).  The caller adds them in the reference's
// order (a subtraction is an addition of the negated value, to the bit).
struct Share {
  float3 dp, df;
};

// The friction cap in double, as the reference's comparisons and ratios use
// it (rare paths only, so targets carry the float copy).
__device__ __forceinline__ double target_fcap(const SweepArgs& a, const Target& t) {
  if (!a.scene_fcap) return a.fcap;
  const int s = min(max(__float2int_rz(t.x.x * a.scene_inv_w), 0), a.n_scenes - 1);
  return (double)a.scene_fcap[s];
}
// 0.01 + r_b in double (Solver.cu:283).
__device__ __forceinline__ double target_bd(const SweepArgs& a, const Target& t) { return a.brad + (double)t.rb; }

// The thresholds of the wall contacts, in double; needed only by targets
// with walls in reach (FP64 issues at 1/64 of the FP32 rate).
__device__ __forceinline__ void target_walls(const SweepArgs& a, Target& t) {
  t.Bru = __double2float_ru(target_bd(a, t));
  t.capBru = __double2float_ru(((double)t.rb + a.brad) * target_fcap(a, t));
}

// The per-target values every sweep needs (no pruning masks, no wall
// thresholds).
__device__ __forceinline__ void make_target_lite(const SweepArgs& a, int i, float4 xi4, Target& t) {
  const Grid& g = a.g;
  t.x = f3(xi4);
  t.rc = xi4.w;
  t.rb = fmaxf(t.rc, a.minr);
  t.Bf = a.bradf + t.rb;
  t.Bcut = t.Bf * t.Bf * 1.0001f;
  t.fcapf = a.scene_fcap ? a.scene_fcap[min(max(__float2int_rz(t.x.x * a.scene_inv_w), 0), a.n_scenes - 1)] : a.fcapf;
  t.inv_m = a.inv_m[i];
  t.x0 = a.pos0 ? f3(a.pos0[i]) : t.x;
  t.q = trunc_cell(g, t.x);
  const uint32_t key = a.keys[i];
  t.wlo = make_float3(INFINITY, INFINITY, INFINITY);  // outside the grid: in nobody's stencil
  t.whi = t.wlo;
  if ((int)key < g.C) {
    const int cx = (int)udiv(key, a.div_yz);
    const int r = (int)key - cx * g.ny * g.nz;
    const int cy = (int)udiv((uint32_t)r, a.div_z);
    const float2 wx = a.window[cx], wy = a.window[cy], wz = a.window[r - cy * g.nz];
    t.wlo = make_float3(wx.x, wy.x, wz.x);
    t.whi = make_float3(wx.y, wy.y, wz.y);
  }
}

// Pruning masks: the stencil columns that can hold a partner within
// r_i + r_max plus the displacement since binning, or a wall within reach.
__device__ __forceinline__ void target_masks(const SweepArgs& a, Target& t) {
  const Grid& g = a.g;
  float disp = __uint_as_float(a.scal->disp0_bits);
  for (int k = 0; k < a.it; ++k) disp += __uint_as_float(a.scal->inc_bits[k]);
  const float rmax = __uint_as_float(a.scal->rmax_bits);
  const float ax = fmaxf(fmaxf(fabsf(t.x.x), fabsf(t.x.y)), fabsf(t.x.z));
  const float slack = 4e-6f * (ax + 1.0f) + 1e-5f * g.L;
  const float Rp = (t.rc + rmax + disp) * 1.0001f + slack;
  const float Rb = t.Bf * 1.0001f + slack;
  t.pm[0] = axis_mask(t.x.x, t.q.x, g.L, Rp);
  t.pm[1] = axis_mask(t.x.y, t.q.y, g.L, Rp);
  t.pm[2] = axis_mask(t.x.z, t.q.z, g.L, Rp);
  t.bm[0] = axis_mask(t.x.x, t.q.x, g.L, Rb);
  t.bm[1] = axis_mask(t.x.y, t.q.y, g.L, Rb);
  t.bm[2] = axis_mask(t.x.z, t.q.z, g.L, Rb);
}

__device__ __forceinline__ void make_target(const SweepArgs& a, int i, float4 xi4, Target& t) {
  make_target_lite(a, i, xi4, t);
  target_walls(a, t);
  target_masks(a, t);
}

// boundary_constraint for one wall particle within the float cut
// (Solver.cu:272-307): whether it is a contact, and its share.  A float d
// compares below a double D exactly when it compares below D rounded up to
// float (no float lies strictly between the two roundings of D), so the
// double comparisons are decided in float.
template <int MM>
__device__ __forceinline__ bool wall_contact(const SweepArgs& a, const Target& t, float4 pb, Share& s) {
  const float bx = t.x.x - pb.x, by = t.x.y - pb.y, bz = t.x.z - pb.z;
  const float dis = m_norm3<(MM & 1)>(bx, by, bz);
  if (!(dis < t.Bru)) return false;  // mag < 0
  const float mag = (float)((double)dis - target_bd(a, t));
  const float3 p12 = make_float3(bx, by, bz);
  const float3 dpi = smul3(mag / dis, p12);
  if (MM & 2) {
    // Coulomb law: the normal push, and the friction target: cancel the
    // tangential displacement since the substep began (the apply kernel
    // limits the averaged friction by the particle's normal corrections)
    const float3 drel = sub3(t.x, t.x0);
    const float dn = dot3(drel, p12) / (dis * dis);
    const float3 dtan = sub3(drel, smul3(dn, p12));
    s.dp = neg3(dpi);
    s.df = neg3(dtan);
    return true;
  }
  const float3 perp = sub3(dpi, div3s(smul3(dot3(dpi, p12), p12), dis * dis));
  const float pn = m_norm3<(MM & 1)>(perp.x, perp.y, perp.z);
  if (pn < t.capBru) {
    s.dp = neg3(dpi);
  } else {
    const float minf = (float)fmin((a.brad + (double)t.rb) * target_fcap(a, t) / (double)pn, 1.0);
    s.dp = neg3(mul3s(dpi, minf));
  }
  return true;
}

__device__ __forceinline__ bool wall_near(const Target& t, float4 pb) {
  const float bx = t.x.x - pb.x, by = t.x.y - pb.y, bz = t.x.z - pb.z;
  const float d2 = __fmaf_rn(bx, bx, __fmaf_rn(by, by, __fmul_rn(bz, bz)));
  return !(d2 > t.Bcut);
}

// particles_constraint for one candidate j (Solver.cu:314-357): whether it
// is a contact, its share, and whether j finds the target too (else the
// count is handed to j here).
template <int MM>
__device__ __forceinline__ bool pair_contact(const SweepArgs& a, const Target& t, int j, float4 xj4, float inv_mj,
                                             Share& s, bool& back) {
  back = false;
  const float dx = t.x.x - xj4.x, dy = t.x.y - xj4.y, dz = t.x.z - xj4.z;
  const float rr = t.rc + xj4.w;
  const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
  if (d2 > rr * rr * 1.0001f) return false;
  const float dis = m_norm3<(MM & 1)>(dx, dy, dz);
  const float mag = rr - dis;
  if (!(mag >= 0.0f)) return false;
  // (float)(1.0 / (double)s) equals the IEEE float reciprocal of s (no
  // double-rounding case exists for 24-bit significands).
  const float inv_sum = __frcp_rn(t.inv_m + inv_mj);
  const float tt = mag / dis;
  const float3 p12 = make_float3(dx, dy, dz);
  const float w = inv_sum * t.inv_m;
  if (MM & 2) {
    // Coulomb law: i's share of the normal push, and its share of cancelling
    // the relative tangential displacement since the substep began (limited
    // by the apply kernel)
    const float4 xj0 = a.pos0[j];
    const float3 drel = sub3(sub3(t.x, t.x0), make_float3(xj4.x - xj0.x, xj4.y - xj0.y, xj4.z - xj0.z));
    const float dn = dot3(drel, p12) / (dis * dis);
    const float3 dtan = sub3(drel, smul3(dn, p12));
    s.dp = smul3(w * tt, p12);
    s.df = neg3(smul3(w, dtan));
  } else {
    const float si = (-inv_sum * t.inv_m) * tt, sj = (inv_sum * inv_mj) * tt;
    const float3 dpij = sub3(smul3(si, p12), smul3(sj, p12));
    const float capf = rr * t.fcapf;
    // The tangential part `perp` of dpij (which is parallel to p12) is
    // rounding noise: |perp| <= 2 (|a| + |b|) dis (1 + 8 eps) with a, b the
    // two scalar factors above.  When that bound is below the cap the
    // reference's branch is decided and perp need not be formed.
    const float bound = 2.0001f * (fabsf(si) + fabsf(sj)) * dis;
    bool within = true;
    float pn = 0.0f;
    if (!(bound < capf * 0.999f)) {
      const float3 perp = sub3(dpij, div3s(smul3(dot3(dpij, p12), p12), dis * dis));
      pn = m_norm3<(MM & 1)>(perp.x, perp.y, perp.z);
      // (double)pn < (double)rr * 0.8, decided in float when clear-cut
      if (pn < capf * 0.999999f) within = true;
      else if (pn > capf * 1.000001f) within = false;
      else within = (double)pn < (double)rr * target_fcap(a, t);
    }
    s.dp = smul3(-w, dpij);
    if (!within) s.dp = mul3s(s.dp, (float)fmin((double)rr * target_fcap(a, t) / (double)pn, 1.0));
  }
  // j's query cell trunc(x*_j / L) is within one cell of i's binning cell on
  // every axis exactly when x*_j lies in i's window (window_table)
  back = xj4.x >= t.wlo.x && xj4.x < t.whi.x && xj4.y >= t.wlo.y && xj4.y < t.whi.y && xj4.z >= t.wlo.z &&
         xj4.z < t.whi.z;
  if (!back) atomicAdd(&a.s_extra[j], 1);
  return true;
}

// Residual mode: a thread's penetrations r_i + r_j - |x_i - x_j| over the
// pairs in the sweep's stencil and (0.01 + max(r_i, 0.01)) - |x - b| over
// wall particles, as k_residual takes them (a pair counts once from each
// side; the mean is unchanged by that).  Every positive one is a listed
// candidate, since lists reach past contact.
struct Penetration {
  float sum = 0.0f, most = 0.0f;
  unsigned int count = 0;
};
__device__ __forceinline__ void add_penetration(const Target& t, int e, float4 p, Penetration& u) {
  const float dx = t.x.x - p.x, dy = t.x.y - p.y, dz = t.x.z - p.z;
  const float R = e >= 0 ? t.rc + p.w : t.Bf;
  const float d2 = dx * dx + dy * dy + dz * dz;
  if (d2 < R * R) {
    const float pen = R - sqrtf(d2);
    u.most = fmaxf(u.most, pen);
    u.sum += pen;
    ++u.count;
  }
}
// A block's penetrations into its sweep's slot (every thread calls it).
__device__ __forceinline__ void store_penetration(const SweepArgs& a, const Penetration& u) {
  __shared__ float s_sum[8];
  __shared__ unsigned int s_count[8], s_most[8];
  float ws = u.sum;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ws += __shfl_xor_sync(0xffffffffu, ws, o);
  const unsigned int wc = __reduce_add_sync(0xffffffffu, u.count);
  const unsigned int wm = __reduce_max_sync(0xffffffffu, __float_as_uint(u.most));
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_sum[w] = ws;
    s_count[w] = wc;
    s_most[w] = wm;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double bs = 0.0;
    unsigned int bc = 0, bm = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      bs += (double)s_sum[k];
      bc += s_count[k];
      bm = max(bm, s_most[k]);
    }
    if (bc) {
      atomicAdd(&a.res->sum, bs);
      atomicAdd(&a.res->count, bc);
      atomicMax(&a.res->most_bits, bm);
    }
  }
}

// The running sums of one thread's target.
struct Sums {
  float3 dp = {0.f, 0.f, 0.f}, df = {0.f, 0.f, 0.f};
  int c = 0, s_loc = 0;
};
template <int MM>
__device__ __forceinline__ void add_wall(const SweepArgs& a, const Target& t, float4 pb, Sums& u) {
  Share s;
  if (!wall_contact<MM>(a, t, pb, s)) return;
  u.dp = add3(u.dp, s.dp);
  if (MM & 2) u.df = add3(u.df, s.df);
  ++u.c;
}
template <int MM>
__device__ __forceinline__ void add_pair(const SweepArgs& a, const Target& t, int j, float4 xj4, float inv_mj, Sums& u) {
  Share s;
  bool back;
  if (!pair_contact<MM>(a, t, j, xj4, inv_mj, s, back)) return;
  u.dp = add3(u.dp, s.dp);
  if (MM & 2) u.df = add3(u.df, s.df);
  ++u.c;
  if (back) ++u.s_loc;
}
template <int MM>
__device__ __forceinline__ void store_sums(const SweepArgs& a, int i, const Sums& u) {
  a.delta[i] = make_float4(u.dp.x, u.dp.y, u.dp.z, __int_as_float((u.c & 0xffff) | (u.s_loc << 16)));
  // (every contact emits one friction target, so their count is c)
  if (MM & 2) a.fdelta[i] = make_float4(u.df.x, u.df.y, u.df.z, __int_as_float(u.c));
}

__device__ __forceinline__ bool use_cell(const unsigned* m, int ox, int oy, int oz) {
  return ((m[0] >> ox) & (m[1] >> oy) & (m[2] >> oz) & 1u) != 0;
}

// The reference loop for one target over global memory.
template <int MM>
__device__ void sweep_global(const SweepArgs& a, int i, const Target& t) {
  const Grid& g = a.g;
  Sums u;
  for (int ox = 0; ox < 3; ++ox) {
    for (int oy = 0; oy < 3; ++oy) {
      for (int oz = 0; oz < 3; ++oz) {
        const bool usep = use_cell(t.pm, ox, oy, oz);
        const bool useb = use_cell(t.bm, ox, oy, oz);
        if (!usep && !useb) continue;
        const int cell = cell_key(g, t.q.x + ox - 1, t.q.y + oy - 1, t.q.z + oz - 1);
        if (cell == g.C) continue;
        if (useb) {
          const int b1 = a.bcs[cell + 1];
          for (int b = a.bcs[cell]; b < b1; ++b) {
            const float4 pb = a.bpos[b];
            if (wall_near(t, pb)) add_wall<MM>(a, t, pb, u);
          }
        }
        if (usep) {
          const int j1 = a.cs[cell + 1];
          for (int j = a.cs[cell]; j < j1; ++j) {
            if (j != i) add_pair<MM>(a, t, j, a.xs[j], a.inv_m[j], u);
          }
        }
      }
    }
  }
  store_sums<MM>(a, i, u);
}

template <int MM>
__global__ void __launch_bounds__(256) k_sweep(SweepArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  Target t;
  make_target(a, i, a.xs[i], t);
  sweep_global<MM>(a, i, t);
}

// ------------------------------------------------------------ listed scan
//
// The reference sums a particle's corrections over its 27 cells in the
// order m = (dx+1)*9 + (dy+1)*3 + (dz+1) and, inside a cell, walls then
// particles by index.  Without contact lists (nlist_skin = 0) each lane
// walks its 27 cells in that order and keeps the candidates that pass a
// cheap distance test in a short list in shared memory (in order); the
// lanes then run the exact test on their k-th listed candidate together,
// which keeps the expensive contact body convergent across the warp.

constexpr int kWarpList = 32;      // listed candidates per lane before a flush
constexpr int kWarpThreads = 256;

template <int MM>
__device__ __forceinline__ void process_entry(const SweepArgs& a, const Target& t, int e, Sums& u) {
  if (e < 0) add_wall<MM>(a, t, a.bpos[-e - 1], u);
  else add_pair<MM>(a, t, e, a.xs[e], a.inv_m[e], u);
}

// One thread per particle over all 27 cells (no per-lane pruning, so the
// lanes of a warp walk the same cell sequence), with the candidates that
// pass the cheap distance test listed in order and processed by all lanes
// together afterwards.
// 4 resident blocks of 256: it hides its loads with warps.  With the 78
// registers that it takes unbounded (3 blocks) 2 M particles 1.9 r apart took
// 7.34 ms of sweeps a substep, 6.08 with 64 and a few bytes spilled; 300,000
// 1.24 and 1.02 ms, 50,000 0.438 and 0.443.
template <int MM>
__global__ void __launch_bounds__(kWarpThreads, 4) k_sweep_list(SweepArgs a) {
  __shared__ int s_list[kWarpThreads / 32][kWarpList][32];
  const Grid& g = a.g;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * kWarpThreads + threadIdx.x;
  if (i >= a.n) return;
  Target t;
  make_target(a, i, a.xs[i], t);
  Sums u;
  int cnt = 0;
  auto flush = [&]() {
    for (int k = 0; k < cnt; ++k) process_entry<MM>(a, t, s_list[w][k][lane], u);
    cnt = 0;
  };
  auto push = [&](int e) {
    if (cnt == kWarpList) flush();
    s_list[w][cnt++][lane] = e;
  };
  for (int m = 0; m < 27; ++m) {
    const int ox = m / 9, oy = (m % 9) / 3, oz = m % 3;
    const int cell = cell_key(g, t.q.x + ox - 1, t.q.y + oy - 1, t.q.z + oz - 1);
    if (cell == g.C) continue;
    if (use_cell(t.bm, ox, oy, oz)) {
      const int b1 = a.bcs[cell + 1];
      for (int b = a.bcs[cell]; b < b1; ++b) {
        const float4 pb = a.bpos[b];
        const float bx = t.x.x - pb.x, by = t.x.y - pb.y, bz = t.x.z - pb.z;
        const float d2 = __fmaf_rn(bx, bx, __fmaf_rn(by, by, __fmul_rn(bz, bz)));
        if (!(d2 > t.Bcut)) push(-b - 1);
      }
    }
    const int j1 = a.cs[cell + 1];
    for (int j = a.cs[cell]; j < j1; ++j) {
      const float4 xj = a.xs[j];
      const float dx = t.x.x - xj.x, dy = t.x.y - xj.y, dz = t.x.z - xj.z;
      const float rr = t.rc + xj.w;
      const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
      if (!(d2 > rr * rr * 1.0001f) && j != i) push(j);
    }
  }
  flush();
  store_sums<MM>(a, i, u);
}

// ------------------------------------------------------------ listed sweep
//
// The grid is fixed for all sweeps of a substep and particles move little
// between sweeps, so each particle keeps the candidates of its stencil that
// lie within r_i + r_j + skin (walls within 0.01 + r_b + skin), in the
// reference's order, and runs the contact test on that list only.
//
// A list built at sweep t stays exact at sweep s while the particle's query
// cell (hence its stencil) is unchanged and
//   A * 1.0001 + 4 e < skin,   A = sum over sweeps u in [t, s) of 2 (N_u + sqrt(3) e),
// where N_u bounds the length of the x* increment of sweep u of the particle
// and of every particle binned in its stencil, and e bounds the rounding of
// one coordinate's position update.  A candidate left out was farther than
// r_i + r_j + skin and has since closed in by less than the skin, so it is
// still no contact: the corrections, their order and the counts are those
// of the full scan.  N_u is the sweep's global maximum increment length when
// that is small enough, else the largest per-cell maximum (recorded by the
// apply kernel) over the 27 stencil cells and the particle's own cell.
// Lists whose bound runs out are rebuilt; the others are kept.

// nl_meta[i].w: the list's length, with flags when it holds walls and when it
// is a long one; or why there is none.  From kNlistLong up it is the groups'.
constexpr int kNlistWalls = 1 << 16, kNlistLong = 1 << 17, kNlistCount = kNlistWalls - 1;
constexpr int kNlistNone = 1 << 18;  // too many for its long one (or all are taken): the groups scan every sweep
constexpr int kNlistNew = -1;        // too many candidates for a list of kNlistMax: the groups make a long one
constexpr int kNlistAgain = -2;      // the same, found in a short queue: queued again at the next sweep

// The listed candidates in order, with the next entry's gathers issued
// before the current one is processed.  entry(k) gives the k-th entry: a
// particle index, or -(wall index) - 1.
__device__ __forceinline__ void fetch_entry(const SweepArgs& a, int e, float4& p, float& im) {
  if (e >= 0) {
    p = a.xs[e];
    im = a.inv_m[e];
  } else if (e != INT_MIN) {
    p = a.bpos[-e - 1];
  }
}

template <int MM, class EntryF>
__device__ __forceinline__ void apply_entries(const SweepArgs& a, const Target& t, int cnt, EntryF&& entry,
                                              Sums& u, Penetration& pen) {
  if (cnt <= 0) return;
  int e_next = entry(0);
  int e_after = cnt > 1 ? entry(1) : INT_MIN;
  float4 p_next = make_float4(0.f, 0.f, 0.f, 0.f);
  float im_next = 0.0f;
  fetch_entry(a, e_next, p_next, im_next);
  for (int k = 0; k < cnt; ++k) {
    const int e = e_next;
    const float4 p = p_next;
    const float im = im_next;
    e_next = e_after;
    fetch_entry(a, e_next, p_next, im_next);
    e_after = (k + 2 < cnt) ? entry(k + 2) : INT_MIN;
    if (MM & 4) add_penetration(t, e, p, pen);
    if (e >= 0) add_pair<MM>(a, t, e, p, im, u);
    else if (wall_near(t, p)) add_wall<MM>(a, t, p, u);
  }
}

// Clears the table that the apply kernel of this sweep adds to (null where a
// memset does: kClearPer).
__device__ __forceinline__ void clear_increments(const SweepArgs& a, int tid) {
  if (!a.cell_clear) return;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + tid; c <= a.g.C; c += (int64_t)gridDim.x * blockDim.x)
    a.cell_clear[c] = 0u;
}

__device__ __forceinline__ bool nlist_bound_ok(const SweepArgs& a, float A) {
  return A * 1.0001f + 4.0f * a.eabs < a.skin;
}

// One sweep's share of the bound A for an increment-length bound N.
__device__ __forceinline__ float nlist_step(const SweepArgs& a, float N) { return 2.0f * (N + 1.7320509f * a.eabs); }

// Largest per-cell increment of the last sweep over the stencil of q and the
// particle's own binning cell.  Every cell_inc entry holds the largest
// increment over its cell and the cell's two z neighbours (k_apply), so the
// stencil's 27 cells are covered by the nine entries of its columns at q.z;
// the own cell adds its entry when it is not one of the 27 (the entry bounds
// its increment from above).  A query cell outside the grid in z reads the
// stencil's cells one by one (entries that may bound from above as well).
__device__ __forceinline__ float nlist_cell_bound(const SweepArgs& a, int3 q, uint32_t own_key) {
  const Grid& g = a.g;
  uint32_t m = 0u;
  if (q.z >= 0 && q.z < g.nz) {
    bool own_in = false;
    for (int ox = -1; ox <= 1; ++ox)
      for (int oy = -1; oy <= 1; ++oy) {
        const int c = cell_key(g, q.x + ox, q.y + oy, q.z);
        if (c == g.C) continue;
        m = max(m, a.cell_inc[c]);
        own_in |= own_key == (uint32_t)c || (own_key == (uint32_t)(c - 1) && q.z > 0) ||
                  (own_key == (uint32_t)(c + 1) && q.z < g.nz - 1);
      }
    if (!own_in) m = max(m, a.cell_inc[own_key]);
    return __uint_as_float(m);
  }
  m = a.cell_inc[own_key];
  for (int ox = -1; ox <= 1; ++ox)
    for (int oy = -1; oy <= 1; ++oy) {
      const int c0 = cell_key(g, q.x + ox, q.y + oy, q.z - 1);
      const int c1 = cell_key(g, q.x + ox, q.y + oy, q.z);
      const int c2 = cell_key(g, q.x + ox, q.y + oy, q.z + 1);
      if (c0 != g.C) m = max(m, a.cell_inc[c0]);
      if (c1 != g.C) m = max(m, a.cell_inc[c1]);
      if (c2 != g.C) m = max(m, a.cell_inc[c2]);
    }
  return __uint_as_float(m);
}

// Sweeps after the first: particles whose list is still exact run it; the
// others are queued for k_sweep_nlist_build.
// 4 resident blocks of 256 (64 registers) against 5 (48, and some spills): the
// 8.4 M column 28.3 ms a substep and 28.7, warm-started 144,000 4.33 and 4.66,
// a batch of 643,000 4.40 and 4.57.  5 in large systems under the Coulomb law
// (kKeepWide).  8 M particles under the reference's law that fall free of each
// other, whose lists are empty, take 4.44 ms with 4 and 4.26 with 5.
template <int MM, int kBlocks>
__global__ void __launch_bounds__(256, kBlocks) k_sweep_nlist_keep(SweepArgs a) {
  const Grid& g = a.g;
  const int tid = (int)pdl_wait(threadIdx.x);
  if ((MM & 4) && a.scal->res_done) return;
  clear_increments(a, tid);
  const int i = blockIdx.x * blockDim.x + tid;
  bool rebuild = false;
  Penetration pen;
  if (i < a.n) {
    const float4 xi4 = a.xs[i];
    const int3 q = trunc_cell(g, f3(xi4));
    const int4 m = a.nl_meta[i];
    bool keep = false;
    rebuild = m.w < kNlistLong;
    if ((unsigned)m.w < (unsigned)kNlistLong && m.x == q.x && m.y == q.y && m.z == q.z) {
      const float A0 = a.nl_acc[i];
      float A = A0 + nlist_step(a, __uint_as_float(a.scal->inc_norm_bits[a.it - 1]));
      if (!nlist_bound_ok(a, A)) A = A0 + nlist_step(a, nlist_cell_bound(a, q, a.keys[i]));
      if (nlist_bound_ok(a, A)) {
        keep = true;
        rebuild = false;
        a.nl_acc[i] = A;
      }
    }
    if (keep) {
      Target t;
      make_target_lite(a, i, xi4, t);
      if (m.w & kNlistWalls) target_walls(a, t);
      Sums u;
      const int32_t* li = a.nl_idx + i;
      apply_entries<MM>(a, t, m.w & kNlistCount, [&](int k) { return __ldcs(li + k * a.li_step); }, u, pen);
      store_sums<MM>(a, i, u);
    }
  }
  // The block's rebuilds go to the queue together, in index order: the
  // rebuild kernel then takes neighbouring particles into one warp (warps
  // appending on their own interleave the regions all SMs work on).
  __shared__ int s_cnt[8], s_base;
  const unsigned bal = __ballot_sync(0xffffffffu, rebuild);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) s_cnt[w] = __popc(bal);
  __syncthreads();
  if (threadIdx.x == 0) {
    int tot = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      const int c = s_cnt[k];
      s_cnt[k] = tot;
      tot += c;
    }
    s_base = tot ? atomicAdd(&a.scal->nl_queued[a.it], tot) : 0;
  }
  __syncthreads();
  if (rebuild) a.nl_queue[s_base + s_cnt[w] + __popc(bal & lanemask_lt())] = i;
  if (MM & 4) store_penetration(a, pen);
}

// List build: scan the 27 cells in the reference order, write the
// candidates within reach of the skin to the particle's list as they are
// found, then run the list.  Every particle at the first sweep of a substep;
// the queued ones later.
constexpr int kBuildThreads = 128;

// 8 resident blocks of 128 (64 registers): the rebuilds are latency-bound
// (72 registers and 7 blocks measured 3 % slower over the sweeps).
template <int MM>
__global__ void __launch_bounds__(kBuildThreads, 8) k_sweep_nlist_build(SweepArgs a, int queued) {
  const Grid& g = a.g;
  const int tid = (int)pdl_wait(threadIdx.x), lane = tid & 31;
  const int total = queued ? a.scal->nl_queued[a.it] : a.n;
  if (queued && total <= a.group_queue) return;  // the groups take a short queue
  if ((MM & 4) && a.scal->res_done) return;
  if (!queued) clear_increments(a, tid);
  Penetration pen;
  for (int base = blockIdx.x * kBuildThreads; base < total; base += gridDim.x * kBuildThreads) {
    const int slot = base + tid;
    const bool act = slot < total;
    {
      // (the vote also brings the warp back together: 8.4 M column 28.2 ms a
      // substep, 28.5 with the vote inside the condition and a __syncwarp)
      const unsigned bal = __ballot_sync(0xffffffffu, act);
      if (a.scal->count_builds && lane == 0 && bal)
        atomicAdd(&a.scal->nlist_rebuilds, (unsigned long long)__popc(bal));
    }
    if (!act) continue;
    const int i = queued ? a.nl_queue[slot] : slot;
    Target t;
    make_target_lite(a, i, a.xs[i], t);
    const float Bs = t.Bf + a.skin;
    const float Bs2 = Bs * Bs * 1.0001f;
    const float rcs = t.rc + a.skin;
    int cnt = 0;
    bool walls = false;
    int32_t* li = a.nl_idx + i;
    auto push = [&](int e) {
      if (cnt < kNlistMax) li[cnt * a.li_step] = e;
      ++cnt;
    };
    // candidates in chunks of 32: a mask of those within their own reach
    // (1.00005 squared covers the roundings), then the pushes in index order.
    // Against a mask for the largest radius by comparisons and an exact test
    // of each hit, sweeps per substep: 8.4 M particles 9.65 to 9.18 ms,
    // 655,000 4.13 to 3.74 (unrolled by 8 9.27 and 3.77)
    const float rcm = rcs * 1.00005f;
    auto scan_particles = [&](int j0, int j1) {
      for (int c0 = j0; c0 < j1; c0 += 32) {
        const int cn = min(32, j1 - c0);
        unsigned far = 0u;
#pragma unroll 4
        for (int b = 0; b < cn; ++b) {
          const float4 xj = a.xs[c0 + b];
          const float rs = __fmaf_rn(xj.w, 1.00005f, rcm);
          far = push_far(far, reach_left(__fmul_rn(rs, rs), sub3(t.x, f3(xj))));
        }
        unsigned mask = near_mask(far, cn);
        const unsigned self = (unsigned)(i - c0);
        if (self < 32u) mask &= ~(1u << self);
        while (mask) {
          push(c0 + __ffs(mask) - 1);
          mask &= mask - 1u;
        }
      }
    };
    for_each_stencil_column(g, t.q, [&](int k0, int nc) {
      if (a.bcs[k0] == a.bcs[k0 + nc]) {
        // no walls in this column: its particles in index order
        scan_particles(a.cs[k0], a.cs[k0 + nc]);
        return;
      }
      for (int z = 0; z < nc; ++z) {
        const int b1 = a.bcs[k0 + z + 1];
        for (int b = a.bcs[k0 + z]; b < b1; ++b) {
          const float4 pb = a.bpos[b];
          const float bx = t.x.x - pb.x, by = t.x.y - pb.y, bz = t.x.z - pb.z;
          const float d2 = __fmaf_rn(bx, bx, __fmaf_rn(by, by, __fmul_rn(bz, bz)));
          if (!(d2 > Bs2)) {
            push(-b - 1);
            walls = true;
          }
        }
        scan_particles(a.cs[k0 + z], a.cs[k0 + z + 1]);
      }
    });
    if (cnt > kNlistMax) {
      // too many candidates to list here: the groups take over
      a.nl_meta[i] = make_int4(0, 0, 0, kNlistNew);
      a.nl_over[atomicAdd(&a.scal->nl_over, 1)] = i;
      continue;
    }
    a.nl_meta[i] = make_int4(t.q.x, t.q.y, t.q.z, cnt | (walls ? kNlistWalls : 0));
    a.nl_acc[i] = 0.0f;
    if (walls) target_walls(a, t);
    Sums u;
    // the list this thread just wrote (its own stores: read back in order)
    apply_entries<MM>(a, t, cnt, [&](int k) { return li[k * a.li_step]; }, u, pen);
    store_sums<MM>(a, i, u);
  }
  if (MM & 4) store_penetration(a, pen);
}

// ------------------------------------------------------------ group sweep
//
// The listed sweep with G lanes to a particle, for systems too small to fill
// the chip with one thread each: a thread alone walks some hundred stencil
// candidates and a dozen contacts one after the other, and the launch lasts
// as long as its longest walk, however few particles it rebuilds.  Here the
// lanes of a group test G candidates at a time, append the hits in order
// (ballots), run G listed contacts at a time, and add their shares in the
// reference's order, one lane to a component.  A list that runs out is
// rebuilt by its own group in the same launch.  Lists are then stored
// particle by particle.  A particle with more candidates than a list holds
// runs each full list as the scan goes on, and gets a long list, of kLongMax
// entries, as long as there are any.
//
// Measured on a GB300 against one thread to a particle (same bits): a frame
// of 4 substeps of 1,000 particles 1.90 to 0.92 ms, of 32,768 particles 2.2
// to 0.91 ms; a substep of the box scene (51,000 particles, 2.5 M render
// points) 2.19 to 1.66 ms.  With the queues of the thread kernels: two
// substeps of 16 settled scenes (643,000 particles) 9.6 to 5.6 ms, a queued
// rebuild launch 800 to about 60 us there.  8 lanes are bound by issue (the
// target's values are computed by every lane of a group), 32 by latency.
//
// The work is all particles, or (k_sweep_rest) what the thread kernels leave:
// the particles with long lists, nl_over, in the order of their lists, checked
// and run in the same way, and the rebuilds of a short queue.
constexpr int kGroupThreads = 256;
constexpr int kLongMax = 160;

enum GroupWork { kWorkAll, kWorkLong, kWorkQueue };

// The shared memory of a block's groups (a kernel's kinds of work take turns
// in it).
template <int MM, int G>
struct GroupSmem {
  static constexpr int kGroups = kGroupThreads / G;
  static constexpr int kStep = 2 * G;              // candidates of a scan step, two a lane
  static constexpr int NC = (MM & 2) ? 6 : 3;      // components of a share
  // a group's rows of shares, padded so that the groups of a warp use
  // different banks
  static constexpr int kRow = G == 8 ? (NC == 6 ? 56 : 24) : G == 16 ? (NC == 6 ? 112 : 48) : NC * G;
  int4 col[kGroups][9];
  int32_t list[kGroups][kNlistMax + kStep];
  float share[kGroups][kRow];
};

template <int MM, int G, GroupWork kWork>
__device__ __forceinline__ void sweep_groups(const SweepArgs& a, int tid, void* smem, Penetration& pen) {
  using Smem = GroupSmem<MM, G>;
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kGroups = Smem::kGroups, NC = Smem::NC, kStep = Smem::kStep, kAhead = kStep / G;
  auto& s_list = static_cast<Smem*>(smem)->list;
  auto& s_col = static_cast<Smem*>(smem)->col;
  auto& s_share = static_cast<Smem*>(smem)->share;
  const Grid& g = a.g;
  const int lane = tid & 31, gl = lane & (G - 1), grp = tid / G;
  const unsigned glt = (1u << gl) - 1u;
  const bool count = a.scal->count_builds != 0;
  auto gballot = [&](bool p) {
    const unsigned b = __ballot_sync(kAll, p);
    return G == 32 ? b : (b >> (lane & ~(G - 1))) & ((1u << (G & 31)) - 1u);
  };
  int total = a.n;
  if (kWork == kWorkLong) total = a.scal->nl_over;
  if (kWork == kWorkQueue) {
    total = a.scal->nl_queued[a.it];
    if (total > a.group_queue) return;  // the threads took it
  }
  // a warp's groups at a time, the warps of a block on their own (the work of
  // one differs much from that of the next)
  constexpr int kWarpGroups = 32 / G;
  for (int base = (blockIdx.x * (kGroupThreads / 32) + (tid >> 5)) * kWarpGroups; base < total;
       base = kWork == kWorkAll ? total : base + (int)gridDim.x * kGroups) {
  const int own = base + (lane / G);
  const bool act = own < total;
  // (groups past the end follow along and write nothing)
  const int slot = act ? own : total - 1;
  const int is = kWork == kWorkAll ? slot : kWork == kWorkLong ? a.nl_over[slot] : a.nl_queue[slot];
  const int i = act ? is : -1;
  Target t;
  make_target_lite(a, is, a.xs[is], t);
  int cnt = 0;
  bool walls = false, rebuild = act, counted = true;
  // the particle's long list: -1 none yet, -2 none to be had.  Once it has one
  // it keeps it, through sweeps whose candidates it does not hold as well
  // (row[0] remembers which).
  int long_row = kWork == kWorkAll ? -1 : kWork == kWorkLong && slot < a.long_rows ? slot : -2;
  int32_t* row = a.nl_idx + is * a.li_row;
  if (kWork == kWorkLong || (kWork == kWorkAll && a.it > 0)) {
    const int4 m = a.nl_meta[is];
    if (kWork == kWorkAll && m.w >= 0 && (m.w & (kNlistLong | kNlistNone))) long_row = row[0];
    counted = m.w != kNlistNew;  // (the threads that left it counted it)
    const bool same = act && m.w >= 0 && m.w != kNlistNone && m.x == t.q.x && m.y == t.q.y && m.z == t.q.z;
    const float A0 = a.nl_acc[is];
    float A = A0 + nlist_step(a, __uint_as_float(a.scal->inc_norm_bits[max(a.it, 1) - 1]));
    bool ok = same && nlist_bound_ok(a, A);
    const bool need = same && !ok;
    if (__any_sync(kAll, need)) {
      const float A2 = A0 + nlist_step(a, nlist_cell_bound(a, t.q, a.keys[is]));
      if (need && nlist_bound_ok(a, A2)) {
        ok = true;
        A = A2;
      }
    }
    if (ok) {  // the list is still exact
      rebuild = false;
      cnt = m.w & kNlistCount;
      walls = (m.w & kNlistWalls) != 0;
      if (m.w & kNlistLong) row = a.nl_long + (size_t)long_row * kLongMax;
      if (gl == 0) a.nl_acc[i] = A;
    }
  }
  if (rebuild) {
    // the stencil columns, as for_each_stencil_column gives them: their
    // particles, and the first cell of a column that holds walls
    const long long zl = max((long long)t.q.z - 1, 0LL), zh = min((long long)t.q.z + 1, (long long)g.nz - 1);
    for (int k = gl; k < 9; k += G) {
      int4 col = make_int4(0, 0, -1, 0);
      const long long x = (long long)t.q.x + k / 3 - 1, y = (long long)t.q.y + k % 3 - 1;
      if (zl <= zh && x >= 0 && x < g.nx && y >= 0 && y < g.ny) {
        const int k0 = (int)((x * g.ny + y) * g.nz + zl), nc = (int)(zh - zl + 1);
        col = make_int4(a.cs[k0], a.cs[k0 + nc], a.bcs[k0] < a.bcs[k0 + nc] ? k0 : -1, nc);
      }
      s_col[grp][k] = col;
    }
  }
  __syncwarp();
  const float Bs = t.Bf + a.skin, Bs2 = Bs * Bs * 1.0001f;
  const float rcs = t.rc + a.skin;
  bool over = false, fits = true;
  int stored = 0;  // entries for the long list, which it holds if it fits
  float sum = 0.0f;  // component gl of the corrections
  int c = 0, s_loc = 0;
  // the scan's place (the same for all groups of a warp): column and cell,
  // and this lane's candidate there
  int seg = __any_sync(kAll, rebuild) ? 0 : 27, v = gl;
  for (;;) {
    while (seg < 27) {
      const int k = seg / 3, z = seg - 3 * k;
      const int4 col = rebuild ? s_col[grp][k] : make_int4(0, 0, -1, 0);
      const bool cells = __any_sync(kAll, col.z >= 0);  // some group goes cell by cell, walls first
      int j0 = col.x, np = z == 0 ? col.y - col.x : 0, b0 = 0, nb = 0;
      if (col.z >= 0) {
        const bool in = z < col.w;
        j0 = in ? a.cs[col.z + z] : 0;
        np = in ? a.cs[col.z + z + 1] - j0 : 0;
        b0 = in ? a.bcs[col.z + z] : 0;
        nb = in ? a.bcs[col.z + z + 1] - b0 : 0;
      }
      bool full = false;
      if (G < 32 && !__any_sync(kAll, nb > 0)) {
        // particles alone: a step's loads in flight together (small groups
        // take many steps; to a whole warp the shorter code is worth more)
        for (; __any_sync(kAll, v - gl < np); v += kStep) {
          if ((full = __any_sync(kAll, cnt > kNlistMax && rebuild))) break;
          float4 xj[kAhead];
#pragma unroll
          for (int u = 0; u < kAhead; ++u) xj[u] = a.xs[v + u * G < np ? j0 + v + u * G : is];
#pragma unroll
          for (int u = 0; u < kAhead; ++u) {
            const float dx = t.x.x - xj[u].x, dy = t.x.y - xj[u].y, dz = t.x.z - xj[u].z;
            const float rs = rcs + xj[u].w;
            const int e = j0 + v + u * G;
            const bool hit = v + u * G < np && e != i &&
                             !(__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz))) > rs * rs * 1.0001f);
            const unsigned hb = gballot(hit);
            if (hit) s_list[grp][cnt + __popc(hb & glt)] = e;
            cnt += __popc(hb);
          }
        }
      } else for (; __any_sync(kAll, v - gl < nb + np); v += kStep) {
        if ((full = __any_sync(kAll, cnt > kNlistMax && rebuild))) break;
#pragma unroll 1
        for (int u = 0; u < kStep; u += G) {
          const int w = v + u;
          bool hit = false;
          int e = 0;
          if (w < nb) {
            e = -(b0 + w) - 1;
            const float4 pb = a.bpos[b0 + w];
            const float bx = t.x.x - pb.x, by = t.x.y - pb.y, bz = t.x.z - pb.z;
            hit = !(__fmaf_rn(bx, bx, __fmaf_rn(by, by, __fmul_rn(bz, bz))) > Bs2);
            walls |= hit;
          } else if (w < nb + np) {
            e = j0 + w - nb;
            const float4 xj = a.xs[e];
            const float dx = t.x.x - xj.x, dy = t.x.y - xj.y, dz = t.x.z - xj.z;
            const float rs = rcs + xj.w;
            hit = !(__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz))) > rs * rs * 1.0001f) && e != i;
          }
          const unsigned hb = gballot(hit);
          if (hit) s_list[grp][cnt + __popc(hb & glt)] = e;
          cnt += __popc(hb);
        }
      }
      if (full) break;
      v = gl;
      seg += cells ? 1 : 3;
    }
    const bool done = seg >= 27;
    const unsigned wb = gballot(walls);  // (every lane votes; kept lists carry the flag in all of theirs)
    walls = wb != 0;
    // a list that overflowed runs as far as it goes; once the scan is done,
    // every list runs (and, if it holds every candidate, is kept)
    const bool filled = rebuild && cnt > kNlistMax;
    over |= filled;
    __syncwarp();
    if (kWork == kWorkAll && __any_sync(kAll, filled && long_row == -1)) {
      int r = 0;
      if (filled && long_row == -1 && gl == 0) r = atomicAdd(&a.scal->nl_over, 1);
      r = __shfl_sync(kAll, r, 0, G);
      if (filled && long_row == -1) long_row = r < a.long_rows ? r : -2;
    }
    if (rebuild && (filled || done)) {
      // (a particle that has a long list keeps to it)
      if (over || long_row >= 0) {
        fits &= stored + cnt <= kLongMax;
        if (long_row >= 0 && fits)
          for (int k = gl; k < cnt; k += G) a.nl_long[(size_t)long_row * kLongMax + stored + k] = s_list[grp][k];
        stored += cnt;
      } else {
        for (int k = gl; k < cnt; k += G) row[k * a.li_step] = s_list[grp][k];
      }
      if (done && gl == 0) {
        int w = cnt;
        if (long_row >= 0 && fits) w = stored | kNlistLong;
        else if (over || kWork == kWorkLong) w = kWork == kWorkQueue ? kNlistAgain : kNlistNone;
        if (kWork == kWorkAll && w >= kNlistLong) row[0] = long_row;
        if (walls && w >= 0 && w != kNlistNone) w |= kNlistWalls;
        a.nl_meta[i] = make_int4(t.q.x, t.q.y, t.q.z, w);
        a.nl_acc[i] = 0.0f;
      }
    }
    const int n = done || filled ? cnt : 0;
    if (walls && n > 0) target_walls(a, t);
    for (int k0 = 0; __any_sync(kAll, k0 < n); k0 += G) {
      Share s;
      bool con = false, back = false;
      if (k0 + gl < n) {
        const int e = rebuild ? s_list[grp][k0 + gl] : row[k0 + gl];
        const float4 p = e >= 0 ? a.xs[e] : a.bpos[-e - 1];
        if (MM & 4) add_penetration(t, e, p, pen);
        if (e >= 0) con = pair_contact<MM>(a, t, e, p, a.inv_m[e], s, back);
        else con = wall_near(t, p) && wall_contact<MM>(a, t, p, s);
      }
      const unsigned cb = gballot(con);
      const int num = __popc(cb);
      s_loc += __popc(gballot(back));
      c += num;
      if (con) {
        float* sh = &s_share[grp][__popc(cb & glt)];
        sh[0] = s.dp.x;
        sh[G] = s.dp.y;
        sh[2 * G] = s.dp.z;
        if (MM & 2) {
          sh[3 * G] = s.df.x;
          sh[4 * G] = s.df.y;
          sh[5 * G] = s.df.z;
        }
      }
      __syncwarp();
      if (gl < NC) {
        const float* sh = &s_share[grp][gl * G];
        for (int k = 0; k < num; ++k) sum += sh[k];
      }
      __syncwarp();
    }
    if (done) break;
    if (filled) cnt = 0;
  }
  if (act) {
    float* out = reinterpret_cast<float*>(a.delta + i);
    if (gl < 3) out[gl] = sum;
    if (gl == 3) out[3] = __int_as_float((c & 0xffff) | (s_loc << 16));
    if (MM & 2) {
      out = reinterpret_cast<float*>(a.fdelta + i);
      if (gl >= 3 && gl < 6) out[gl - 3] = sum;
      if (gl == 6) out[3] = __int_as_float(c);
    }
  }
  if (count) {
    const unsigned b = __ballot_sync(kAll, rebuild && counted && gl == 0);
    if (lane == 0 && b) atomicAdd(&a.scal->nlist_rebuilds, (unsigned long long)__popc(b));
  }
  __syncwarp();
  }
}

template <int MM, int G>
__global__ void __launch_bounds__(kGroupThreads, 3) k_sweep_group(SweepArgs a) {
  const int tid = (int)pdl_wait(threadIdx.x);
  if ((MM & 4) && a.scal->res_done) return;
  clear_increments(a, tid);
  __shared__ GroupSmem<MM, G> smem;
  Penetration pen;
  sweep_groups<MM, G, kWorkAll>(a, tid, &smem, pen);
  if (MM & 4) store_penetration(a, pen);
}

// What the thread kernels leave: the long lists, by whole warps (their scans
// and lists are long), and short queues, by whole warps as well where
// particles lie so close that one in 256 has a long list, else by groups of
// 8: 16 settled scenes 4.90 ms with 8 and 4.63 with 32, a settled pile 2.44
// and 2.28, but a loosely packed warm-started solve 4.6 and 5.6.
template <int MM>
__global__ void __launch_bounds__(kGroupThreads, 3) k_sweep_rest(SweepArgs a) {
  const int tid = (int)pdl_wait(threadIdx.x);
  if ((MM & 4) && a.scal->res_done) return;
  __shared__ union {
    GroupSmem<MM, 32> wide;
    GroupSmem<MM, 8> narrow;
  } smem;
  Penetration pen;
  sweep_groups<MM, 32, kWorkLong>(a, tid, &smem, pen);
  if (a.it > 0) {
    const bool wide = a.scal->nl_over > (a.n >> 8);
    __syncthreads();  // the warps lay their shared memory out differently
    if (wide) sweep_groups<MM, 32, kWorkQueue>(a, tid, &smem, pen);
    else sweep_groups<MM, 8, kWorkQueue>(a, tid, &smem, pen);
  }
  if (MM & 4) store_penetration(a, pen);
}

// The window of a cell coordinate c: [lo, hi) holds exactly the positions x
// with c - 1 <= trunc(x / L) <= c + 1 (IEEE division, then truncation; x / L
// rounds monotonically, so they are an interval).  With T(k) the smallest x
// whose quotient reaches k >= 1: hi = T(c + 2); lo = T(c - 1) for c >= 2,
// and for c = 1 and 0, where truncation takes quotients above -1 and -2, the
// negative of the largest x below T(1) and T(2).  A contact then costs six
// comparisons in place of three divisions; with the wall thresholds in double
// only for targets that have walls in reach, the settled pile of 262,144
// particles went from 6.33 to 5.84 ms per substep and two substeps of 16
// settled scenes (643,000 particles, 15 contacts each) from 10.58 to 9.70 ms.
__device__ float quotient_reaches(float L, int k) {
  float x = (float)k * L;
  while (x > 0.0f && (double)(x / L) >= (double)k) x = nextafterf(x, 0.0f);
  while ((double)(x / L) < (double)k) x = nextafterf(x, INFINITY);
  return x;
}
__global__ void k_window_table(int n, float L, float2* __restrict__ window) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const float lo = c >= 2 ? quotient_reaches(L, c - 1) : -nextafterf(quotient_reaches(L, 2 - c), 0.0f);
  window[c] = make_float2(lo, quotient_reaches(L, c + 2));
}
gg_status window_table(gg_system* S, cudaStream_t st) {
  const int n = std::max(S->grid.nx, std::max(S->grid.ny, S->grid.nz));
  k_window_table<<<blocks_for(n, 128), 128, 0, st>>>(n, S->grid.L, S->window);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

// Systems up to this size give every particle a group of lanes.  Where threads
// take over depends on the packing, which the host does not know; sweeps of a
// substep by threads and by groups in us: 2.6 r apart (no neighbours) 20,000
// 105 and 94, 60,000 108 and 163, 100,000 113 and 229; 1.9 r apart 60,000 274
// and 246, 100,000 364 and 434; 1.5 r apart 60,000 444 and 387, 100,000 482 and
// 540; settled piles 64,000 937 and 552, 111,000 1,338 and 898, 176,000 1,581
// and 1,543, 262,000 2,668 and 2,786; collapsed columns 96,000 1,576 and 1,104,
// 178,000 2,169 and 1,689, 448,000 3,140 and 3,608.
constexpr int64_t kGroupMax = 100000;

// Above this size the keep kernel has 5 resident blocks under the Coulomb law,
// with 4 and 5 in ms a substep: a batch of 7.9 M in 64 scenes 6.67 and 6.54,
// 4.5 M particles 2.0 r apart 2.76 and 2.73, 2.6 r apart 2.00 and 1.94, 1.75 r
// apart 3.55 and 3.55; 1.5 M 1.04 and 1.04, 0.74 and 0.73, 1.35 and 1.36.
constexpr int64_t kKeepWide = 1500000;

// The sweep's threads clear the increment table for its apply kernel where
// that leaves each at most this many entries; a few particles in a large grid
// leave it to a memset, which has the whole chip (and costs a launch, about
// 3 us a sweep).  Substeps of 7 sweeps, by the threads and by memset: 300
// particles in 1 M cells 122 and 134 us, 10 M 268 and 210, 100 M 1,654 and
// 896; 4,000 in 100 M 948 and 957, 512 M 4,203 and 3,972; 120,000 (a thread
// each) in 33 M 746 and 768, 100 M 1,310 and 1,265.
constexpr int64_t kClearPer = 512;
static gg_status clear_by_memset(gg_system* S, SweepArgs& a, int64_t threads, cudaStream_t st) {
  if ((int64_t)S->grid.C + 1 <= kClearPer * threads) return GG_OK;
  GG_CUDA(cudaMemsetAsync(a.cell_clear, 0, sizeof(uint32_t) * ((size_t)S->grid.C + 1), st));
  a.cell_clear = nullptr;
  return GG_OK;
}

// Queues up to this length are rebuilt by groups (30,000 to 240,000 measured
// the same; 15,000 lost 30 % on 643,000 settled particles).
constexpr int kGroupQueue = 65536;

// Lanes to a particle: 1,000 particles ran a frame in 925 us with 32, 950
// with 16 and 1,000 with 8; 32,768 particles in 1,136, 958 and 914 us.
constexpr int64_t kGroup32Max = 4096, kGroup16Max = 16384;

// A sweep kernel by its template argument (math mode 1 sums no penetrations:
// sweep_sums_residual).
#define GG_SWEEP_KERNEL(MMVAL, ...)                                                                       \
  [&]() {                                                                                                 \
    auto pick = [](auto m) { constexpr int MM = decltype(m)::value; return &__VA_ARGS__; };               \
    using std::integral_constant;                                                                         \
    switch (MMVAL) {                                                                                      \
      case 0: return pick(integral_constant<int, 0>());                                                   \
      case 1: return pick(integral_constant<int, 1>());                                                   \
      case 2: return pick(integral_constant<int, 2>());                                                   \
      case 3: return pick(integral_constant<int, 3>());                                                   \
      case 4: return pick(integral_constant<int, 4>());                                                   \
      default: return pick(integral_constant<int, 6>());                                                  \
    }                                                                                                     \
  }()

template <int G>
static gg_status launch_group(gg_system* S, SweepArgs& a, int mm, cudaStream_t st) {
  const int blocks = blocks_for(a.n, kGroupThreads / G);
  gg_status rc = clear_by_memset(S, a, (int64_t)blocks * kGroupThreads, st);
  if (rc != GG_OK) return rc;
  auto kern = GG_SWEEP_KERNEL(mm, k_sweep_group<MM, G>);
  GG_CUDA(launch_chained(kern, blocks, kGroupThreads, st, a));
  return GG_OK;
}

bool sweep_lists(const gg_system* S) { return S->g.nl_idx && S->tune.sweep_variant == 0; }
bool sweep_sums_residual(const gg_system* S) {
  return sweep_lists(S) && !S->P.math_mode && S->n > 0;
}

gg_status sweep(gg_system* S, int it, cudaStream_t st, ResidualSlot* res) {
  if (S->n <= 0) return GG_OK;
  SweepArgs a;
  a.g = S->grid;
  a.n = (int)S->n;
  a.it = it;
  a.xs = S->g.xs;
  a.inv_m = S->g.inv_m;
  a.keys = S->g.keys;
  a.cs = S->g.cell_start;
  a.bcs = S->b.cell_start;
  a.bpos = S->b.pos;
  a.delta = S->g.delta;
  a.s_extra = S->g.s_extra;
  a.scal = S->scal;
  a.brad = S->P.boundary_radius;
  a.fcap = S->P.friction_cap;
  a.fcapf = (float)S->P.friction_cap;
  a.bradf = (float)S->P.boundary_radius;
  a.window = S->window;
  a.scene_fcap = S->scene_fcap;
  a.scene_inv_w = S->scene_width > 0.0f ? 1.0f / S->scene_width : 0.0f;
  a.n_scenes = S->n_scenes;
  a.minr = S->P.boundary_min_radius;
  const bool coulomb = S->P.contact_law == 1;
  a.pos0 = coulomb ? S->g.pos[S->g.cur] : nullptr;
  a.fdelta = coulomb ? S->g.fdelta : nullptr;
  const int mm = (S->P.math_mode ? 1 : 0) | (coulomb ? 2 : 0) | (res ? 4 : 0);  // the kernels' template argument
  a.res = res;
  a.nl_idx = S->g.nl_idx;
  a.nl_meta = S->g.nl_meta;
  a.nl_acc = S->g.nl_acc;
  a.nl_queue = S->g.nl_queue;
  a.cell_inc = S->g.cell_inc[(it & 1) ^ 1];
  a.cell_clear = S->g.cell_inc[it & 1];
  a.nl_over = S->g.split_slot;  // (scratch of the split, free during the sweeps)
  a.nl_long = S->g.nl_long;
  a.long_rows = (int)std::min<int64_t>(kLongInts * S->cap / kLongMax, INT_MAX);
  a.li_row = a.li_step = 0;
  a.group_queue = 0;
  a.skin = S->nl_skin;
  a.div_yz = make_udiv((uint32_t)(S->grid.ny * S->grid.nz));
  a.div_z = make_udiv((uint32_t)S->grid.nz);
  {
    // half an ulp of the largest in-grid coordinate, with a margin
    const float ext = S->grid.L * (float)std::max(S->grid.nx, std::max(S->grid.ny, S->grid.nz));
    a.eabs = 2.5e-7f * (1.0f + ext);
  }
  prof_begin(S, PC_SWEEP, st);
  // the sweep kernel: contact lists when they are allocated (the default),
  // else one thread per particle over all 27 cells with its candidates
  // listed in order; gg_tuning.sweep_variant = 1 picks the pruned
  // one-thread-per-particle stencil sweep instead (same results)
  if (S->tune.sweep_variant == 1) {
    auto kern = (mm == 0 ? k_sweep<0> : mm == 1 ? k_sweep<1> : mm == 2 ? k_sweep<2> : k_sweep<3>);
    kern<<<blocks_for(S->n, 256), 256, 0, st>>>(a);
  } else if (S->g.nl_idx && S->n <= kGroupMax) {
    a.li_row = kNlistMax;
    a.li_step = 1;
    gg_status rc = S->n <= kGroup32Max   ? launch_group<32>(S, a, mm, st)
                   : S->n <= kGroup16Max ? launch_group<16>(S, a, mm, st)
                                         : launch_group<8>(S, a, mm, st);
    if (rc != GG_OK) return rc;
  } else if (S->g.nl_idx) {
    a.li_row = 1;
    a.li_step = (size_t)S->cap;
    a.group_queue = kGroupQueue;
    gg_status rc = clear_by_memset(S, a, S->n, st);
    if (rc != GG_OK) return rc;
    auto build = GG_SWEEP_KERNEL(mm, k_sweep_nlist_build<MM>);
    if (it == 0) {
      GG_CUDA(launch_chained(build, blocks_for(S->n, kBuildThreads), kBuildThreads, st, a, 0));
    } else {
      auto keep = S->n > kKeepWide ? GG_SWEEP_KERNEL(mm, k_sweep_nlist_keep<MM, (MM & 2) ? 5 : 4>)
                                   : GG_SWEEP_KERNEL(mm, k_sweep_nlist_keep<MM, 4>);
      const int tk = S->tune.keep_threads;
      GG_CUDA(launch_chained(keep, blocks_for(S->n, tk), tk, st, a));
      const int nb = std::min(blocks_for(S->n, kBuildThreads), S->num_sms * S->tune.build_blocks_per_sm);
      GG_CUDA(launch_chained(build, nb, kBuildThreads, st, a, 1));
      count_launches(S, 1);
    }
    // short queues, and what a list does not hold
    auto rest = GG_SWEEP_KERNEL(mm, k_sweep_rest<MM>);
    GG_CUDA(launch_chained(rest, S->num_sms * 3, kGroupThreads, st, a));
    count_launches(S, 1);
  } else {
    auto kern = (mm == 0 ? k_sweep_list<0> : mm == 1 ? k_sweep_list<1> : mm == 2 ? k_sweep_list<2> : k_sweep_list<3>);
    kern<<<blocks_for(S->n, kWarpThreads), kWarpThreads, 0, st>>>(a);
  }
  count_launches(S, 1);
  prof_end(S, PC_SWEEP, S->n, st);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

}  // namespace gg
