// Particle/grid transfer kernels of the adaptive GIMP substep.
//
// Reference steps (adaptive_gimp.py, g1n0st/adaptive-gimp):
//   230-250 p2g               -> k_p2g      (all levels in one launch)
//   289-301 grid_restriction  -> k_restrict (one launch per level, fine->coarse)
//   277-287 grid_op           -> level 0 in the last k_restrict, level l in
//                                k_prolong(l); k_gridop (all levels) only
//                                when every scene has one level
//   303-321 grid_prolongation -> k_prolong  (one launch per level, coarse->fine)
//   252-275 g2p               -> k_g2p      (all levels in one launch)
//
// P2G: one warp per work item = some tens of particles of one bin (one 4^d
// block of one level).  A bin's particles touch only the (4+2)^d nodes from the
// block origin, so P2G accumulates into that tile in shared memory and flushes
// it with one float4 atomic per touched node.  G2P: one thread per particle
// slot in bin order; 3D reads the nodes from a tile staged per block, 2D
// gathers them through L1.
//
// Every kernel serves a batch of scenes (a single simulator is a batch of
// one): each CTA works for the scene its launch range assigns it to.
//
// Restriction and prolongation are written as gathers (each destination node
// sums its sources) instead of the reference's scatters, so they need no
// atomics; the set of terms and their weights are the reference's.
#include "common.cuh"
#include "umma.cuh"

namespace agimp {

// first stored cell of block `blk` (block indices are 32-bit: 32-bit division)
template <int D>
__device__ __forceinline__ void chunk_origin(const LevelDev& V, long long blk, int* O) {
  unsigned b = (unsigned)blk;
  const unsigned nb = (unsigned)V.nb;
#pragma unroll
  for (int d = D - 1; d >= 0; --d) {
    O[d] = (int)(b % nb) * 4 - HALO;
    b /= nb;
  }
}

// ---------------------------------------------------------------------------
// P2G (adaptive_gimp.py:230-250).  Each warp works alone on a contiguous range
// of work items (k_bins): an item is up to TASKS tasks of one 4^d block
// of one level, a task up to T particles of one base cell (bins store their
// particles sorted by cell, so an item's particles are contiguous).
//  1. Rounds of 32 particles, one per lane: the scaled Kirchhoff stress S
//     (utils.py:11-16, adaptive_gimp.py:240; symmetric, kirchhoff_sym), m,
//     a = m (v - C (tc+1)), B = m C and tc go to shared memory, at [place in
//     its task][task].
//  2. The tasks' contributions to their cell's 3^d nodes are summed in registers
//     (packed f32x2), by three lanes per task, one per plane (3D) or row (2D) of
//     nodes along the first axis: all 27 nodes' sums in one lane leave room for
//     8 warps on an SM (200 instead of 132 us for 1.9M particles), and in 2D
//     the three lanes make a small scene's items shorter.
//  3. The sums go through shared memory to one lane per node, which adds the
//     tasks of one cell and updates the warp's (4+2)^d node tile.
// The tile goes to the grid with one float4 atomic per touched node when the
// warp's next item is another block.  There are no atomics on shared memory
// (an f32 add there is a compare-and-swap loop) and no CTA barriers.
//
// What bounds it: instruction issue (41 warp instructions per 3D particle, half
// of them multiply-adds, at 53 percent of the issue slots) and, between, the
// latency of step 1's reads at 16 warps per SM.  Before (one lane per row of
// three nodes, a 52-float record read by nine lanes, shared-memory atomics at
// every change of cell) it took 53.  1.9M 3D particles on three levels 172 (182
// before the particles' rows) -> 129 us, 15.5M 1210 -> 900, 0.6M at 8 per cell 70 -> 53, 50,000 16.6 -> 11.3;
// 4.1M 2D particles at 4 per cell 254 (at the best of its CTA sizes, 613 at the
// default) -> 213 us.  Also measured: long tasks in dense cells (up to 32
// particles: 273 us, a warp's range of items then differs in cost), the next
// round's rows in registers (152: spills), 5 CTAs of 96 registers (176).
template <int D>
struct P2GLayout {
  static constexpr int WARPS = 4;                 // warps of a CTA
  static constexpr int CTAS = D == 2 ? 8 : 4;     // CTAs an SM should hold
  static constexpr int NN = (D == 2) ? 9 : 27;    // stencil nodes
  static constexpr int SPLIT = 3;                 // lanes of a task
  static constexpr int PN = NN / SPLIT;           // their nodes
  static constexpr int TN = (D == 2) ? 36 : 216;  // nodes of the (4+2)^d tile
  static constexpr int TASKS = P2G_TASKS, TMAX = 1 << P2G_LOG_TMAX;
  // step 3: groups of node lanes, each with its share of the tasks and its own
  // tile (3D 27 lanes, 2D 3 x 9 lanes)
  static constexpr int GROUPS = 32 / NN;
  // record (floats): 3D  0 a m | 4 B0 t0 | 8 B1 t1 | 12 B2 t2 | 16 Sxx Sxy Sxz Syz | 20 Syy Szz
  //                  2D  0 a m t0 | 4 B0 B1 | 8 Sxx Sxy Syy t1
  // (B_d: column d of m C).  REC and ROW put the float4 accesses of eight
  // neighbouring lanes in distinct banks, by task (step 2) and by place (step
  // 1, where consecutive particles are consecutive places of a task).
  static constexpr int REC = (D == 2) ? 12 : 28;
  static constexpr int ROW = TASKS * REC + (D == 2 ? 12 : 4);
  static constexpr int RECS = TMAX * ROW, SUMS = TASKS * NN * 4;  // records, then the lanes' sums
  static constexpr int AREA = RECS > SUMS ? RECS : SUMS;
  static constexpr int WARP_FLOATS = AREA + GROUPS * TN * 4;
  static constexpr size_t bytes() { return sizeof(float) * (size_t)WARPS * WARP_FLOATS; }
};

// Step 1: the record of particle p of a level (inv = 1 / dx) at R.  The stress
// carries sc = 2 (-dt 0.5^d) / (radius^d dx): the factor kg / kw = 2 of the
// gradient weights; the sums get kw when they leave the tile.
template <int D>
__device__ __forceinline__ void p2g_record(const Ctx& c, int p, float inv, float sc, float* R) {
  using W = PWord<D>;
  float4 q[W::NQ];
  const float4* src = c.P.s + prow<D>(p);
#pragma unroll
  for (int k = 0; k < W::NQ; ++k) q[k] = src[32 * k];
  float t[D], F[D * D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float xs = qword(q, W::X + d) * inv;
    const int base = (int)(xs + 0.5f) - 1;
    t[d] = xs - (float)(base + 1);
  }
#pragma unroll
  for (int k = 0; k < D * D; ++k) F[k] = qword(q, W::F + k);
  const float m = qword(q, W::M);
  float mu = c.mu, la = c.la;
  if (c.plast == 1) {
    const float h = expf(c.xi * (1.f - qword(q, W::JP)));
    mu *= h;
    la *= h;
  }
  const float J = det<D>(F);
  float S[(D == 2) ? 3 : 6];
  kirchhoff_sym<D>(F, 2.f * mu, la * J * (J - 1.f), S);
  float a[D];
#pragma unroll
  for (int i = 0; i < D; ++i) {
    float cd = 0.f;
#pragma unroll
    for (int b = 0; b < D; ++b) cd += qword(q, W::C + i * D + b) * (t[b] + 1.f);
    a[i] = m * (qword(q, W::V + i) - cd);
  }
  auto B = [&](int i, int d) { return m * qword(q, W::C + i * D + d); };
  float4* R4 = (float4*)R;
  if constexpr (D == 3) {
    R4[0] = make_float4(a[0], a[1], a[2], m);
#pragma unroll
    for (int d = 0; d < 3; ++d) R4[1 + d] = make_float4(B(0, d), B(1, d), B(2, d), t[d]);
    R4[4] = make_float4(sc * S[0], sc * S[1], sc * S[3], sc * S[4]);
    *(float2*)(R4 + 5) = make_float2(sc * S[2], sc * S[5]);
  } else {
    R4[0] = make_float4(a[0], a[1], m, t[0]);
    R4[1] = make_float4(B(0, 0), B(1, 0), B(0, 1), B(1, 1));
    R4[2] = make_float4(sc * S[0], sc * S[1], sc * S[2], t[1]);
  }
}

// One axis's weights and gradients, each twice (packed operands); for radius
// 1/2 axis_weights_half's closed form.
__device__ __forceinline__ void p2g_axis(float t, float radius, bool half, f2* w, f2* g) {
  if (half) {
    const f2 t2 = f2_dup(t);
    g[0] = f2_add(t2, f2_dup(-0.5f));
    g[1] = f2_mul(t2, f2_dup(-2.f));
    g[2] = f2_add(t2, f2_dup(0.5f));
    w[0] = f2_mul(g[0], g[0]);
    w[1] = f2_fma(g[1], t2, f2_dup(1.5f));
    w[2] = f2_mul(g[2], g[2]);
  } else {
    float W[3], G[3];
    axis_weights(t, radius, W, G);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      w[k] = f2_dup(W[k]);
      g[k] = f2_dup(G[k]);
    }
  }
}

// Weight and gradient of node n0 of the first axis: for radius 1/2, with q = t
// + (n0 - 1) / 2, the gradient is b q and the weight b q^2 + e, (b, e) = (1, 0),
// (-2, 3/2), (1, 0).
__device__ __forceinline__ void p2g_axis_at(float t, float radius, bool half, int n0, f2& w, f2& g) {
  if (half) {
    const float q = t + 0.5f * (float)(n0 - 1);
    const float gs = n0 == 1 ? -2.f * q : q;
    g = f2_dup(gs);
    w = f2_dup(fmaf(gs, q, n0 == 1 ? 1.5f : 0.f));
  } else {
    float W[3], G[3];
    axis_weights(t, radius, W, G);
    g = f2_dup(n0 == 0 ? G[0] : n0 == 1 ? G[1] : G[2]);
    w = f2_dup(n0 == 0 ? W[0] : n0 == 1 ? W[1] : W[2]);
  }
}

// Step 2: one particle into the sums of plane n0.  A node's term (unscaled, see
// p2g_record) is
//   w (a + B n) + S grad w = Wz (A + k Bz') + Gz Sz',
//   A = Wy (P + n1 Wx By) + Gy Wx Sy,  P = Wx (a + n0 Bx) + Gx Sx,
//   Bz' = Wx Wy Bz,  Sz' = Wx Wy Sz   (B_d, S_d: columns)
// 3D node n = 3 n1 + k: xy[n] = (p_x, p_y), zm[n] = (p_z, m): the mass rides as
// the fourth component of a (B and S have none).
__device__ __forceinline__ void p2g_plane(const float* R, float radius, bool half, int n0, f2* xy, f2* zm) {
  const float4* R4 = (const float4*)R;
  const float4 a = R4[0], b0 = R4[1], b1 = R4[2], b2 = R4[3], s = R4[4];
  const float2 e = *(const float2*)(R4 + 5);  // Syy Szz
  f2 wx, gx, wy[3], gy[3], wz[3], gz[3];
  p2g_axis_at(b0.w, radius, half, n0, wx, gx);
  p2g_axis(b1.w, radius, half, wy, gy);
  p2g_axis(b2.w, radius, half, wz, gz);
  const f2 fn = f2_dup((float)n0);
  const f2 u = f2_fma(fn, f2_make(b0.x, b0.y), f2_make(a.x, a.y));
  const f2 z = f2_fma(fn, f2_make(b0.z, 0.f), f2_make(a.z, a.w));
  f2 P = f2_fma(wx, u, f2_mul(gx, f2_make(s.x, s.y))), Pz = f2_fma(wx, z, f2_mul(gx, f2_make(s.z, 0.f)));
  const f2 Q = f2_mul(wx, f2_make(b1.x, b1.y)), Qz = f2_mul(wx, f2_make(b1.z, 0.f));
  const f2 T = f2_mul(wx, f2_make(s.y, e.x)), Tz = f2_mul(wx, f2_make(s.w, 0.f));
  const f2 E = f2_mul(wx, f2_make(b2.x, b2.y)), Ez = f2_mul(wx, f2_make(b2.z, 0.f));
  const f2 H = f2_mul(wx, f2_make(s.z, s.w)), Hz = f2_mul(wx, f2_make(e.y, 0.f));
#pragma unroll
  for (int n1 = 0; n1 < 3; ++n1) {
    f2 A = f2_fma(wy[n1], P, f2_mul(gy[n1], T)), Az = f2_fma(wy[n1], Pz, f2_mul(gy[n1], Tz));
    const f2 b = f2_mul(wy[n1], E), bz = f2_mul(wy[n1], Ez), h = f2_mul(wy[n1], H), hz = f2_mul(wy[n1], Hz);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      xy[3 * n1 + k] = f2_fma(gz[k], h, f2_fma(wz[k], A, xy[3 * n1 + k]));
      zm[3 * n1 + k] = f2_fma(gz[k], hz, f2_fma(wz[k], Az, zm[3 * n1 + k]));
      if (k < 2) {
        A = f2_add(A, b);
        Az = f2_add(Az, bz);
      }
    }
    if (n1 < 2) {
      P = f2_add(P, Q);
      Pz = f2_add(Pz, Qz);
    }
  }
}

// 2D row n0: xy[k] = (p_x, p_y), m[k].
__device__ __forceinline__ void p2g_row(const float* R, float radius, bool half, int n0, f2* xy, float* m) {
  const float4* R4 = (const float4*)R;
  const float4 a = R4[0], b = R4[1], s = R4[2];
  f2 wx, gx, wy[3], gy[3];
  p2g_axis_at(a.w, radius, half, n0, wx, gx);
  p2g_axis(s.w, radius, half, wy, gy);
  const f2 u = f2_fma(f2_dup((float)n0), f2_make(b.x, b.y), f2_make(a.x, a.y));
  f2 A = f2_fma(wx, u, f2_mul(gx, f2_make(s.x, s.y)));
  const f2 e = f2_mul(wx, f2_make(b.z, b.w)), h = f2_mul(wx, f2_make(s.y, s.z));
  const float cm = f2_get(wx).x * a.z;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    xy[k] = f2_fma(gy[k], h, f2_fma(wy[k], A, xy[k]));
    m[k] = fmaf(f2_get(wy[k]).x, cm, m[k]);
    A = f2_add(A, e);
  }
}

template <int D>
__global__ void __launch_bounds__(32 * P2GLayout<D>::WARPS, P2GLayout<D>::CTAS) k_p2g(Batch B) {
  SCENE_CTA(B, MAP_P);
  using Y = P2GLayout<D>;
  constexpr int NN = Y::NN, PN = Y::PN, TN = Y::TN, NC = 1 << (2 * D);
  constexpr unsigned ALL = 0xffffffffu;
  extern __shared__ float4 dsm4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* area = (float*)dsm4 + warp * Y::WARP_FLOATS;
  float4* sums = (float4*)area;               // [TASKS][NN]
  float4* tiles = (float4*)(area + Y::AREA);  // [GROUPS][TN]
  const int nitem = c.ctr[CTR_ITEMS];
  const long long nw = (long long)nblk_ * Y::WARPS, wid = (long long)bid_ * Y::WARPS + warp;
  const int i0 = (int)(wid * nitem / nw), i1 = (int)((wid + 1) * nitem / nw);
  if (i0 >= i1) return;
  const float radius = c.radius, r2 = 2.f * radius;
  const float kw = (D == 2) ? 1.f / (4.f * r2 * r2) : 1.f / (8.f * r2 * r2 * r2);
  const float pw = (D == 2) ? 0.25f : 0.125f;                            // 0.5**dim
  const float rd = (D == 2) ? radius * radius : radius * radius * radius;  // radius**dim
  const bool half = radius == 0.5f;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int t = lane; t < Y::GROUPS * TN; t += 32) tiles[t] = zero;
  // step 2: this lane's task and plane
  const int mytask = lane / Y::SPLIT, n0 = lane % Y::SPLIT;
  // step 3: this lane's node and task group
  const int grp = lane / NN, node = lane % NN;
  const unsigned gmask = grp < Y::GROUPS ? ((1u << NN) - 1u) << (grp * NN) : 0u;
  int toff = 0;  // the node's offset in the tile
#pragma unroll
  for (int d = 0, r = node, m = 1; d < D; ++d, r /= 3, m *= 6) toff += (r % 3) * m;
  float4* tile = tiles + (grp < Y::GROUPS ? grp : 0) * TN + toff;
  int bin = -1, excl = 0, nt0 = 0, off0 = 0, off1 = 0, c0 = 0, c1 = 0, tasks = 0;
  int4 it = c.items[i0];
  for (int i = i0; i < i1; ++i) {
    const int l = it.x & 15, lt = (it.x >> 4) & 15, first = (int)((unsigned)it.x >> 8) * Y::TASKS, blk = it.y;
    if (it.z != bin) {
      // the bin's cells: lane holds cells 2 lane, 2 lane + 1 (3D) or cell
      // lane (2D): their particles, and the tasks of the cells before them
      bin = it.z;
      const int* co = c.cell_off + (long long)bin * NC;
      if (D == 3) {
        const int2 o = *(const int2*)(co + 2 * lane);
        off0 = o.x;
        off1 = o.y;
      } else {
        off0 = off1 = lane < NC ? co[lane] : it.w;
      }
      int nx = __shfl_down_sync(ALL, off0, 1);
      if (lane == 31) nx = it.w;
      c0 = (D == 3 ? off1 : nx) - off0;
      c1 = D == 3 ? nx - off1 : 0;
      nt0 = (c0 + (1 << lt) - 1) >> lt;
      const int nt = nt0 + ((c1 + (1 << lt) - 1) >> lt);
      int inc = nt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(ALL, inc, o);
        if (lane >= o) inc += y;
      }
      excl = inc - nt;
      tasks = __shfl_sync(ALL, inc, 31);
    }
    const int bend = it.w;  // the end of the bin's particles
    if (i + 1 < i1) it = c.items[i + 1];
    // lane t < TASKS holds task first + t: its cell, first particle and particles
    const int k = first + lane;
    int own = 0;  // the last lane whose cells start at or before task k
#pragma unroll
    for (int s = 16; s; s >>= 1)
      if (__shfl_sync(ALL, excl, own + s) <= k) own += s;
    int j = k - __shfl_sync(ALL, excl, own);
    const int ont0 = __shfl_sync(ALL, nt0, own);
    int off = __shfl_sync(ALL, off0, own), n = __shfl_sync(ALL, c0, own), cell = own;
    if (D == 3) {
      const int o1 = __shfl_sync(ALL, off1, own), m1 = __shfl_sync(ALL, c1, own);
      cell = 2 * own;
      if (j >= ont0) {
        j -= ont0;
        off = o1;
        n = m1;
        ++cell;
      }
    }
    const int nv = min(Y::TASKS, tasks - first);  // tasks of this item
    const int start = lane < nv ? off + (j << lt) : 0x7fffffff;
    const int cnt = lane < nv ? min(1 << lt, n - (j << lt)) : 0;
    const int s0 = __shfl_sync(ALL, start, 0), e0 = __shfl_sync(ALL, start + cnt, nv - 1);
    // place in the tile of the cell's first node
    const int place = D == 3 ? ((cell >> 4) * 6 + ((cell >> 2) & 3)) * 6 + (cell & 3) : (cell >> 2) * 6 + (cell & 3);
    // the next item's particles follow this one's in the bin, or start the next
    // bin; 3D asks for them ahead of the sums (2 to 3 percent; 2D items are over
    // before it helps)
    int ahead[2] = {-1, -1};
    if (D == 3 && i + 1 < i1) {
      const int from = it.z != bin ? c.cell_off[(long long)it.z * NC] : e0, left = (it.z != bin ? it.w : bend) - from;
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (32 * r + lane < left) ahead[r] = c.perm[from + 32 * r + lane];
    }
    // -- 1. records -------------------------------------------------------------
    {
      const float inv = (float)(c.coarsest << l);
      const float sc = 2.f * ((-c.dt * pw) / (rd * (1.f / inv)));
#pragma unroll 1
      for (int p0 = s0; p0 < e0; p0 += 32) {
        const int q = p0 + lane;
        int task = 0;  // the last task that starts at or before q
#pragma unroll
        for (int s = 8; s; s >>= 1)
          if (__shfl_sync(ALL, start, task + s) <= q) task += s;
        const int ts = __shfl_sync(ALL, start, task);
        if (q < e0) p2g_record<D>(c, c.perm[q], inv, sc, area + (q - ts) * Y::ROW + task * Y::REC);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
      if (D == 3 && ahead[r] >= 0) {
        const float4* src = c.P.s + prow<D>(ahead[r]);
#pragma unroll
        for (int k = 0; k < PWord<D>::NQ; ++k) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + 32 * k));
      }
    __syncwarp();
    // -- 2. sums of the lane's plane ------------------------------------------------
    {
      const int count = __shfl_sync(ALL, cnt, mytask);
      const float* R = area + mytask * Y::REC;
      f2 xy[PN], zm[D == 3 ? PN : 1];
      float m[D == 2 ? PN : 1];
#pragma unroll
      for (int a = 0; a < PN; ++a) {
        xy[a] = 0ull;
        if (D == 3) zm[a % (D == 3 ? PN : 1)] = 0ull;
        if (D == 2) m[a % (D == 2 ? PN : 1)] = 0.f;
      }
#pragma unroll 1
      for (int p = 0; p < count; ++p, R += Y::ROW) {
        if constexpr (D == 3)
          p2g_plane(R, radius, half, n0, xy, zm);
        else
          p2g_row(R, radius, half, n0, xy, m);
      }
      __syncwarp();  // the records have been read: the sums take their place
      if (mytask < nv)
#pragma unroll
        for (int a = 0; a < PN; ++a) {
          const float2 u = f2_get(xy[a]);
          float2 w;
          if constexpr (D == 3)
            w = f2_get(zm[a]);
          else
            w = make_float2(0.f, m[a]);
          sums[mytask * NN + n0 * PN + a] = make_float4(u.x, u.y, w.x, w.y);
        }
    }
    __syncwarp();
    // -- 3. lane <-> node: the tasks of one cell, then the tile ---------------------
    {
      const int per = (nv + Y::GROUPS - 1) / Y::GROUPS;
      const int j0 = grp * per;
      float4 acc = zero;
      int at = -1;  // place of the cell being summed
      auto flush = [&]() {
        float4 o = tile[at];
        o.x += acc.x;
        o.y += acc.y;
        if (D == 3) o.z += acc.z;
        o.w += acc.w;
        tile[at] = o;
        __syncwarp(gmask);  // the lanes of one tile stay together
      };
#pragma unroll 2
      for (int e = 0; e < per; ++e) {
        const int tj = j0 + e;
        const int pj = __shfl_sync(ALL, place, tj & 31);
        if (grp >= Y::GROUPS || tj >= nv) continue;
        const float4 v = sums[tj * NN + node];
        if (pj != at) {
          if (at >= 0) flush();
          at = pj;
          acc = v;
        } else {
          acc.x += v.x;
          acc.y += v.y;
          if (D == 3) acc.z += v.z;
          acc.w += v.w;
        }
      }
      if (at >= 0) flush();
    }
    __syncwarp();
    // the same block follows: keep summing into the tile
    if (i + 1 < i1 && it.y == blk && (it.x & 15) == l) continue;
    const LevelDev& V = c.lev[l];
    int O[D];
    chunk_origin<D>(V, blk, O);
    for (int t = lane; t < TN; t += 32) {
      float4 val = tiles[t];
      tiles[t] = zero;
#pragma unroll
      for (int g = 1; g < Y::GROUPS; ++g) {
        const float4 o = tiles[g * TN + t];
        tiles[g * TN + t] = zero;
        val.x += o.x;
        val.y += o.y;
        val.w += o.w;
      }
      if (val.x == 0.f && val.y == 0.f && val.z == 0.f && val.w == 0.f) continue;
      int I[D], tt = t;
#pragma unroll
      for (int d = D - 1; d >= 0; --d) {
        I[d] = O[d] + tt % 6;
        tt /= 6;
      }
      if (!in_store<D>(V, I)) {
        set_err(c, ERR_OOB);
        continue;
      }
      atomicAdd(&V.node[elem_of<D>(V, I)], make_float4(val.x * kw, val.y * kw, val.z * kw, val.w * kw));
    }
    __syncwarp();
  }
}

// Node mask of node I of level l stored at idx: 3D scenes read the level's
// own copy (k_level_masks), which the staged transfers copy by whole blocks;
// 2D scenes, whose transfers gather node by node, read the node mask itself.
template <int D>
__device__ __forceinline__ uint32_t level_mask(const Ctx& c, int l, const int* I, long long idx) {
  if (D == 3) return c.lev[l].nm[idx];
  return nm_get<D>(c, l, I);
}

// grid_op (adaptive_gimp.py:277-287) of node I of level l with mask nm and value
// nd: an activated node's momentum becomes its velocity (gravity, walls,
// colliders); with inv_norm the other nodes with mass are divided by it.  I lies
// in [0, size]^d.
template <int D>
__device__ __forceinline__ float4 gridop_value(const Ctx& c, int l, const int* I, uint32_t nm, const float4 nd) {
  if (!(nd.w > 0.f)) return nd;
  if (!is_activated(nm)) {
    if (c.inv_norm) return make_float4(nd.x / nd.w, nd.y / nd.w, D == 3 ? nd.z / nd.w : nd.z, nd.w);
    return nd;
  }
  float vv[3] = {nd.x, nd.y, nd.z};
  const int s = c.L - 1 - l;
  bool band = false;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    vv[d] = vv[d] / nd.w;
    vv[d] = vv[d] + c.grav[d] * c.dt;
    const int P = I[d] * (1 << s);
    if (P < c.gap || P > c.sz - c.gap) {
      band = true;
      if (c.bmode == 0) vv[d] = 0.f;
    }
  }
  if (c.bmode == 1 && band)
#pragma unroll
    for (int d = 0; d < D; ++d) vv[d] = 0.f;
  if (c.ncol) {
    const double ldx = 1.0 / (double)(c.coarsest << l);
    for (int k = 0; k < c.ncol; ++k) {
      bool in = true;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double pos = (double)I[d] * ldx;
        in = in && pos >= c.col[k][d] && pos <= c.col[k][3 + d];
      }
      if (in)
#pragma unroll
        for (int d = 0; d < D; ++d) vv[d] = 0.f;
    }
  }
  return make_float4(vv[0], vv[1], vv[2], nd.w);
}

template <int D>
__device__ __forceinline__ void gridop_node(const Ctx& c, int l, const int* I, long long idx) {
  float4& node = c.lev[l].node[idx];
  const uint32_t nm = level_mask<D>(c, l, I, idx);
  node = gridop_value<D>(c, l, I, nm, node);
}

// ---------------------------------------------------------------------------
// Level transfers staged through shared memory by the TMA engine.  A CTA takes
// one destination block at a time; one thread issues bulk copies
// (cp.async.bulk, global -> shared, completion counted in bytes on an
// mbarrier) of the source level's node blocks and node-mask blocks the
// destination block reads, every thread waits on the mbarrier (bounded), and
// the gather then reads shared memory only.  Blocks are contiguous in HBM
// (PER nodes of 16 B, PER masks of 4 B), so every copy is one aligned run.
template <int D>
struct Stage {
  static constexpr int PER = 1 << (2 * D);
  static constexpr uint32_t NODE_BYTES = PER * 16, MASK_BYTES = PER * 4;
  // the lanes of the first warp (a 2D CTA has 16 threads)
  static constexpr unsigned WARP0 = PER >= 32 ? 0xffffffffu : ((1u << PER) - 1u);
};

__device__ __forceinline__ void mbar_expect_tx(uint64_t* m, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(umma::smem_u32(m)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void bulk_to_shared(void* dst, const void* src, uint32_t bytes, uint64_t* m) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   umma::smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(umma::smem_u32(m))
               : "memory");
}

// Wait for the staged copies of this phase.  When the bounded wait gives up,
// the CTA records ERR_MLP (a bounded device wait gave up), waits once more
// (bounded) for its copies in flight and returns false.
__device__ __forceinline__ bool stage_wait(const Ctx& c, uint64_t* m, uint32_t phase) {
  if (umma::mbar_wait(m, phase)) return true;
  if (threadIdx.x == 0) set_err(c, ERR_MLP);
  umma::mbar_wait(m, phase);
  return false;
}

__device__ __forceinline__ void stage_init(uint64_t* m) {
  if (threadIdx.x == 0) {
    umma::mbar_init(m, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}

// stored block coordinates of linear block index b (first axis slowest)
template <int D>
__device__ __forceinline__ void block_coords(unsigned b, unsigned nb, int* Bc) {
#pragma unroll
  for (int d = D - 1; d >= 0; --d) {
    Bc[d] = (int)(b % nb);
    b /= nb;
  }
}

// grid_restriction(l) (adaptive_gimp.py:289-301) as a gather over the coarse
// nodes K of level l-1: the restricted sum onto K of the fine nodes 2K - dI
// that are (activated and even), T-junctions or ghosts, weight 0.5^|dI|_1.
// The fine nodes of a coarse block lie in the 3^d fine blocks 2B-2 .. 2B (B:
// the coarse block's stored coordinates).  The last restriction (into level
// 0) also applies grid_op to level 0, whose momentum no later pass reads; in a
// scene of one level it only does that.
template <int D>
__global__ void __launch_bounds__(Stage<D>::PER) k_restrict(Batch B, int l) {
  SCENE_CTA(B, MAP_T);
  using S = Stage<D>;
  constexpr int NB = (D == 2) ? 9 : 27;
  __shared__ __align__(128) float4 fn[NB][S::PER];
  __shared__ __align__(128) uint32_t fm[NB][S::PER];
  __shared__ int fok[NB];
  __shared__ __align__(8) uint64_t mbar;
  const bool restrict_l = l < c.L;
  if (!restrict_l && l != 1) return;
  const LevelDev& Vc = c.lev[l - 1];
  const LevelDev& Vf = c.lev[restrict_l ? l : l - 1];
  const int nblk = c.ctr[CTR_LEVEL + l - 1];
  const int lsz = Vf.size, l0sz = Vc.size;
  const int loc = threadIdx.x;
  stage_init(&mbar);
  uint32_t phase = 0;
  for (int bi = bid_; bi < nblk; bi += nblk_) {
    const unsigned blk = (unsigned)Vc.blist[bi];
    int Bc[D];
    block_coords<D>(blk, (unsigned)Vc.nb, Bc);
    if (restrict_l) {
      if (threadIdx.x < 32) {
        // lane t of the first warp stages fine block t (NB <= 32)
        const int t = threadIdx.x;
        uint32_t bytes = 0;
        if (t < NB) {
          bool ok = true;
          unsigned fb = 0;
          int tt = t, fc[D];
#pragma unroll
          for (int d = D - 1; d >= 0; --d) {
            fc[d] = 2 * Bc[d] - 2 + tt % 3;
            tt /= 3;
            ok = ok && fc[d] >= 0 && fc[d] < Vf.nb;
          }
#pragma unroll
          for (int d = 0; d < D; ++d) fb = fb * (unsigned)Vf.nb + (unsigned)fc[d];
          fok[t] = ok ? (int)fb : -1;
          if (ok) bytes = S::NODE_BYTES + S::MASK_BYTES;
        }
        bytes = __reduce_add_sync(S::WARP0, bytes);
        // earlier generic reads of the tile finished at the barrier that
        // ended the previous block; order them before the async writes
        umma::fence_proxy_async();
        if (t == 0) mbar_expect_tx(&mbar, bytes);
        __syncwarp(S::WARP0);
        if (t < NB && fok[t] >= 0) {
          bulk_to_shared(fn[t], Vf.node + ((long long)fok[t] << (2 * D)), S::NODE_BYTES, &mbar);
          bulk_to_shared(fm[t], Vf.nm + ((long long)fok[t] << (2 * D)), S::MASK_BYTES, &mbar);
        }
      }
      __syncthreads();  // fok
      const bool ok = stage_wait(c, &mbar, phase);
      phase ^= 1;
      if (!ok) return;
    }
    int K[D];
#pragma unroll
    for (int d = D - 1, t = loc; d >= 0; --d, t >>= 2) K[d] = ((Bc[d] - 1) << 2) + (t & 3);
    bool inr = true;
#pragma unroll
    for (int d = 0; d < D; ++d) inr = inr && K[d] >= 0 && K[d] <= l0sz;
    const long long cidx = ((long long)blk << (2 * D)) | loc;
    if (inr && restrict_l && is_valid(Vc.nm[cidx])) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      bool any = false;
#pragma unroll
      for (int a = 0; a < ((D == 2) ? 9 : 27); ++a) {
        int t = a, nrm = 0, tile = 0, li = 0;
        bool okI = true;
#pragma unroll
        for (int d = D - 1; d >= 0; --d) {
          const int dI = t % 3 - 1;
          t /= 3;
          const int I = 2 * K[d] - dI;
          nrm += dI != 0;
          okI = okI && I >= 0 && I <= lsz;
        }
        if (!okI) continue;
        // tile and local index of fine node 2K - dI
        t = a;
        int mul = 1, lmul = 1;
#pragma unroll
        for (int d = D - 1; d >= 0; --d) {
          const int dI = t % 3 - 1;
          t /= 3;
          const int q = 2 * K[d] - dI + HALO;
          tile += ((q >> 2) - (2 * Bc[d] - 2)) * mul;
          li += (q & 3) * lmul;
          mul *= 3;
          lmul *= 4;
        }
        if (fok[tile] < 0) continue;
        const uint32_t nm = fm[tile][li];
        if (!((is_activated(nm) && nrm == 0) || is_tj(nm) || is_ghost(nm))) continue;
        const float w = (nrm == 0) ? 1.f : (nrm == 1) ? 0.5f : (nrm == 2) ? 0.25f : 0.125f;
        const float4 f = fn[tile][li];
        acc.x += f.x * w;
        acc.y += f.y * w;
        acc.z += f.z * w;
        acc.w += f.w * w;
        any = true;
      }
      if (any) {
        float4 o = Vc.node[cidx];
        o.x += acc.x;
        o.y += acc.y;
        o.z += acc.z;
        o.w += acc.w;
        Vc.node[cidx] = o;
      }
    }
    if (inr && l == 1) gridop_node<D>(c, 0, K, cidx);
    __syncthreads();  // the tile is free for the next block's copies
  }
}

// ---------------------------------------------------------------------------
// The same two transfers as direct gathers through L1 (one thread per
// destination node): used for 2D scenes, whose 16-node blocks are too small
// for a staging round trip per block to pay.  Bound by the latency of L2
// reads: a node's masks are loaded together, then the nodes they select
// (before, each weight's mask and then its node: 20,000 particles restriction
// 6.7 -> 4.4 us, prolongation 5.3 -> 4.0; 256 scenes 26 and 31, as before).
// Three CTAs an SM: with two the batch's restriction takes 31 us.
template <int D>
__global__ void __launch_bounds__(256, 3) k_restrict_gather(Batch B, int l) {
  static_assert(D == 2, "3D transfers are staged");
  SCENE_CTA(B, MAP_G);
  const bool restrict_l = l < c.L;
  if (!restrict_l && l != 1) return;
  const LevelDev& Vc = c.lev[l - 1];
  const LevelDev& Vf = c.lev[restrict_l ? l : l - 1];
  const long long tot = (long long)c.ctr[CTR_LEVEL + l - 1] << (2 * D);
  const int lsz = Vf.size, l0sz = Vc.size;
  SCENE_LOOP(e, tot) {
    const long long blk = Vc.blist[e >> (2 * D)];
    const int loc = (int)(e & ((1 << (2 * D)) - 1));
    int K[D];
    elem_coords<D>(Vc, blk, loc, K);
    bool inr = true;
#pragma unroll
    for (int d = 0; d < D; ++d) inr = inr && K[d] >= 0 && K[d] <= l0sz;
    if (!inr) continue;
    const long long cidx = (blk << (2 * D)) | loc;
    const uint32_t cm = level_mask<D>(c, l - 1, K, cidx);
    float4 o = Vc.node[cidx];
    bool any = false;
    if (restrict_l && is_valid(cm)) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      // the nine sources' masks are read together, then the nodes that count (two
      // memory latencies)
      unsigned fidx[9], use = 0;
      uint32_t nm[9];
      auto weight = [&](int a, int* I) {  // source a's node and weight
        int nrm = 0;
#pragma unroll
        for (int d = D - 1; d >= 0; --d) {
          const int dI = a % 3 - 1;
          a /= 3;
          I[d] = 2 * K[d] - dI;
          nrm += dI != 0;
        }
        return (nrm == 0) ? 1.f : (nrm == 1) ? 0.5f : 0.25f;
      };
#pragma unroll
      for (int a = 0; a < 9; ++a) {
        int I[D];
        weight(a, I);
        bool ok = true;
#pragma unroll
        for (int d = 0; d < D; ++d) ok = ok && I[d] >= 0 && I[d] <= lsz;
        fidx[a] = (unsigned)elem_of<D>(Vf, I);
        nm[a] = ok ? level_mask<D>(c, l, I, fidx[a]) : 0u;
      }
      float4 f[9];
#pragma unroll
      for (int a = 0; a < 9; ++a) {
        int I[D];
        if ((is_activated(nm[a]) && weight(a, I) == 1.f) || is_tj(nm[a]) || is_ghost(nm[a])) {
          f[a] = Vf.node[fidx[a]];
          use |= 1u << a;
        }
      }
      any = use != 0;
#pragma unroll
      for (int a = 0; a < 9; ++a) {
        if (!(use >> a & 1u)) continue;
        int I[D];
        const float w = weight(a, I);
        acc.x += f[a].x * w;
        acc.y += f[a].y * w;
        acc.w += f[a].w * w;
      }
      if (any) o = make_float4(o.x + acc.x, o.y + acc.y, o.z + acc.z, o.w + acc.w);
    }
    if (l == 1)
      Vc.node[cidx] = gridop_value<D>(c, 0, K, cm, o);
    else if (any)
      Vc.node[cidx] = o;
  }
}

template <int D>
__global__ void k_prolong_gather(Batch B, int l) {
  static_assert(D == 2, "3D transfers are staged");
  SCENE_CTA(B, MAP_G);
  if (l >= c.L) return;
  const LevelDev& Vc = c.lev[l - 1];
  const LevelDev& Vf = c.lev[l];
  const long long tot = (long long)c.ctr[CTR_LEVEL + l] << (2 * D);
  const int lsz = Vf.size;
  SCENE_LOOP(e, tot) {
    const long long blk = Vf.blist[e >> (2 * D)];
    const int loc = (int)(e & ((1 << (2 * D)) - 1));
    int J[D];
    elem_coords<D>(Vf, blk, loc, J);
    bool inr = true, even = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      inr = inr && J[d] >= 0 && J[d] <= lsz;
      even = even && (J[d] & 1) == 0;
    }
    if (!inr) continue;
    const long long fidx = (blk << (2 * D)) | loc;
    // the node and its mask are read together (even nodes: with the mask of the
    // coarse node they take), then the masks of the coarse nodes around a T or
    // ghost node, then the coarse nodes
    const float4 nd = Vf.node[fidx];
    const uint32_t nm = level_mask<D>(c, l, J, fidx);
    const bool tg = is_tj(nm) || is_ghost(nm);
    // node J lies between the coarse nodes J / 2 (and + 1 on its odd axes)
    unsigned cidx[1 << D];
    uint32_t cm[1 << D];
    int nodd = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) nodd += J[d] & 1;
#pragma unroll
    for (int a = 0; a < (1 << D); ++a) {
      int K[D];
      bool use = true;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const int bit = (a >> d) & 1;
        K[d] = (J[d] >> 1) + bit;
        use = use && (bit == 0 || (J[d] & 1));
      }
      cidx[a] = (unsigned)elem_of<D>(Vc, K);
      cm[a] = use && (even || tg) ? level_mask<D>(c, l - 1, K, cidx[a]) : 0u;
    }
    float4 o = gridop_value<D>(c, l, J, nm, nd);
    if (tg || even) {
      const bool take = tg || is_activated(nm);  // (an even node's only source is a = 0)
      const float w = (nodd == 0) ? 1.f : (nodd == 1) ? 0.5f : 0.25f;
      float4 cv[1 << D];
#pragma unroll
      for (int a = 0; a < (1 << D); ++a)
        if (take && is_valid(cm[a])) cv[a] = Vc.node[cidx[a]];
      float acc[2] = {0.f, 0.f};
#pragma unroll
      for (int a = 0; a < (1 << D); ++a)
        if (take && is_valid(cm[a])) {
          acc[0] += cv[a].x * w;
          acc[1] += cv[a].y * w;
        }
      o.x = acc[0];
      o.y = acc[1];
      o.z = 0.f;
    }
    Vf.node[fidx] = o;
  }
}

// 3D scenes stage their transfers through shared memory, 2D scenes gather
template <int D>
constexpr bool staged_transfers() {
  return D == 3;
}

// ---------------------------------------------------------------------------
// grid_op for every level at once.  Only substeps whose scenes all have one
// level launch it; otherwise the last restriction applies grid_op to level 0
// and each prolongation to its own level (see there).
template <int D>
__global__ void k_gridop(Batch B) {
  SCENE_CTA(B, MAP_G);
  __shared__ BlockRanges br;
  load_block_ranges(c, br);
  const long long tot = total_elems_r(br, 0, c.L, D);
  SCENE_LOOP(e, tot) {
    int l, loc;
    long long blk;
    decode_elem_r<D>(c, br, 0, c.L, e, l, blk, loc);
    const LevelDev& V = c.lev[l];
    int I[D];
    elem_coords<D>(V, blk, loc, I);
    bool inr = true;
#pragma unroll
    for (int d = 0; d < D; ++d) inr = inr && I[d] >= 0 && I[d] <= V.size;
    if (inr) gridop_node<D>(c, l, I, (blk << (2 * D)) | loc);
  }
}

// ---------------------------------------------------------------------------
// grid_prolongation(l) (adaptive_gimp.py:303-321) as a gather over the fine
// nodes J of level l: T-junction and ghost nodes take the weighted sum of
// their valid coarse neighbours, other all-even nodes take the coincident
// coarse velocity if they are activated and it is valid, else 0; the rest keep
// their value.  The coarse nodes of a fine block B lie in the 2^d coarse
// blocks (2B + 1) / 4 .. (2B + 1) / 4 + 1 per axis, staged like the
// restriction's.  Level l's grid_op runs first on each node: its momentum is
// no longer read (the restrictions are done) and its coarser neighbour is
// final.
template <int D>
__global__ void __launch_bounds__(Stage<D>::PER) k_prolong(Batch B, int l) {
  SCENE_CTA(B, MAP_T);
  using S = Stage<D>;
  constexpr int NB = 1 << D;
  __shared__ __align__(128) float4 cn[NB][S::PER];
  __shared__ __align__(128) uint32_t cm[NB][S::PER];
  __shared__ int cok[NB];
  __shared__ __align__(8) uint64_t mbar;
  if (l >= c.L) return;
  const LevelDev& Vc = c.lev[l - 1];
  const LevelDev& Vf = c.lev[l];
  const int nblk = c.ctr[CTR_LEVEL + l];
  const int lsz = Vf.size;
  const int loc = threadIdx.x;
  stage_init(&mbar);
  uint32_t phase = 0;
  for (int bi = bid_; bi < nblk; bi += nblk_) {
    const unsigned blk = (unsigned)Vf.blist[bi];
    int Bf[D], C0[D];
    block_coords<D>(blk, (unsigned)Vf.nb, Bf);
#pragma unroll
    for (int d = 0; d < D; ++d) C0[d] = (2 * Bf[d] + 1) >> 2;
    if (threadIdx.x < 32) {
      // lane t of the first warp stages coarse block t
      const int t = threadIdx.x;
      uint32_t bytes = 0;
      if (t < NB) {
        bool ok = true;
        unsigned cb = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const int q = C0[d] + ((t >> (D - 1 - d)) & 1);
          ok = ok && q < Vc.nb;
          cb = cb * (unsigned)Vc.nb + (unsigned)q;
        }
        cok[t] = ok ? (int)cb : -1;
        if (ok) bytes = S::NODE_BYTES + S::MASK_BYTES;
      }
      bytes = __reduce_add_sync(S::WARP0, bytes);
      umma::fence_proxy_async();
      if (t == 0) mbar_expect_tx(&mbar, bytes);
      __syncwarp(S::WARP0);
      if (t < NB && cok[t] >= 0) {
        bulk_to_shared(cn[t], Vc.node + ((long long)cok[t] << (2 * D)), S::NODE_BYTES, &mbar);
        bulk_to_shared(cm[t], Vc.nm + ((long long)cok[t] << (2 * D)), S::MASK_BYTES, &mbar);
      }
    }
    __syncthreads();  // cok
    const bool okw = stage_wait(c, &mbar, phase);
    phase ^= 1;
    if (!okw) return;
    int J[D];
#pragma unroll
    for (int d = D - 1, t = loc; d >= 0; --d, t >>= 2) J[d] = ((Bf[d] - 1) << 2) + (t & 3);
    bool inr = true, even = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      inr = inr && J[d] >= 0 && J[d] <= lsz;
      even = even && (J[d] & 1) == 0;
    }
    const long long fidx = ((long long)blk << (2 * D)) | loc;
    if (inr) {
      gridop_node<D>(c, l, J, fidx);
      const uint32_t nm = Vf.nm[fidx];
      const bool tg = is_tj(nm) || is_ghost(nm);
      if (tg || even) {
        // coarse node K: staged tile and local index
        auto coarse = [&](const int* K, float4& v) -> bool {
          int tile = 0, li = 0;
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const int q = K[d] + HALO;
            tile = tile * 2 + ((q >> 2) - C0[d]);
            li = li * 4 + (q & 3);
          }
          if (cok[tile] < 0 || !is_valid(cm[tile][li])) return false;
          v = cn[tile][li];
          return true;
        };
        float acc[3] = {0.f, 0.f, 0.f};
        if (tg) {
          int nodd = 0;
#pragma unroll
          for (int d = 0; d < D; ++d) nodd += J[d] & 1;
          const float w = (nodd == 0) ? 1.f : (nodd == 1) ? 0.5f : (nodd == 2) ? 0.25f : 0.125f;
#pragma unroll
          for (int a = 0; a < (1 << D); ++a) {
            int K[D];
            bool use = true;
#pragma unroll
            for (int d = 0; d < D; ++d) {
              const int bit = (a >> d) & 1;
              if (J[d] & 1)
                K[d] = (J[d] - 1) / 2 + bit;
              else {
                K[d] = J[d] / 2;
                use = use && bit == 0;
              }
            }
            float4 cv;
            if (!use || !coarse(K, cv)) continue;
            acc[0] += cv.x * w;
            acc[1] += cv.y * w;
            acc[2] += cv.z * w;
          }
        } else if (is_activated(nm)) {
          int K[D];
#pragma unroll
          for (int d = 0; d < D; ++d) K[d] = J[d] / 2;
          float4 cv;
          if (coarse(K, cv)) {
            acc[0] = cv.x;
            acc[1] = cv.y;
            acc[2] = cv.z;
          }
        }
        float4 o = Vf.node[fidx];
        o.x = acc[0];
        o.y = acc[1];
        o.z = acc[2];
        Vf.node[fidx] = o;
      }
    }
    __syncthreads();  // the tile is free for the next block's copies
  }
}

// ---------------------------------------------------------------------------
// g2p (adaptive_gimp.py:252-275), plus the snow return map (extension).
template <int D>
__device__ __forceinline__ void svd_d(const float* F, float* U, float* sg, float* V) {
  if (D == 2)
    svd2(F, U, sg, V);
  else
    svd3(F, U, sg, V);
}

// Exact snow return map (Stomakhin et al. 2013) on an SVD: clamp the singular
// values to [1-theta_c, 1+theta_s], update Jp, rebuild F.  Written with
// explicitly rounded operations (no contraction choices left to the compiler)
// so that every inlined copy, in G2P and in the surrogate's finishing kernel,
// gives the same bits for the same SVD.
template <int D>
__device__ __forceinline__ void snow_clamp_rebuild(const Ctx& c, const float* U, const float* sg, const float* V,
                                                   float* F, float& jp) {
  const float lo = 1.f - c.theta_c, hi = 1.f + c.theta_s;
  float Jo = 1.f, Jn = 1.f, sc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float cl = fminf(fmaxf(sg[d], lo), hi);
    Jo = __fmul_rn(Jo, sg[d]);
    Jn = __fmul_rn(Jn, cl);
    sc[d] = cl;
  }
  jp = __fdiv_rn(__fmul_rn(jp, Jo), Jn);
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) {
      float a = 0.f;
#pragma unroll
      for (int k = 0; k < D; ++k) a = __fmaf_rn(__fmul_rn(U[i * D + k], sc[k]), V[j * D + k], a);
      F[i * D + j] = a;
    }
}


// The surrogate's domain: a non-inverted trial state with positive singular
// values and plastic ratio.
template <int D>
__device__ __forceinline__ bool sur_domain(const float* F, const float* sg, float jp) {
  bool ok = jp > 0.f && det<D>(F) > 0.f;
#pragma unroll
  for (int d = 0; d < D; ++d) ok = ok && sg[d] > 0.f;
  return ok;
}

// Recorder: the surrogate's training pair (features, exact projected state)
// of a trial state with singular values sg and plastic ratio jp.
template <int D>
__device__ __forceinline__ void record_pair(const Ctx& c, const float* sg, float jp) {
  float x[7], y[4];
  snow_features<D>(sg, jp, c.xi, c.theta_c, c.theta_s, x);
  float Jo = 1.f, Jn = 1.f;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (d < D) {
      const float cl = fminf(fmaxf(sg[d], 1.f - c.theta_c), 1.f + c.theta_s);
      Jo *= sg[d];
      Jn *= cl;
      y[d] = (cl - sg[d]) / SUR_DSIG;
    } else {
      y[d] = 0.f;
    }
  }
  y[3] = logf(Jo / Jn) / SUR_DLJ;
  const int slot = reserve_slot(&c.ctr[CTR_REC]);
  if ((long long)slot >= c.rec_cap) return;
#pragma unroll
  for (int k = 0; k < 7; ++k) c.rec_X[(long long)slot * 7 + k] = x[k];
#pragma unroll
  for (int k = 0; k < 4; ++k) c.rec_T[(long long)slot * 4 + k] = y[k];
}

// Surrogate hand-off of a trial state with SVD (U, sg, V): its features go to
// the MLP's input buffer and U, V, sig, jp to the metadata buffer, and
// k_sur_finish writes F and Jp.  Returns false when the features leave the
// trained range (the caller then applies the exact return map).
template <int D>
__device__ __forceinline__ bool sur_handoff(const Ctx& c, const float* U, const float* sg, const float* V, float jp,
                                            int j) {
  float x[7];
  snow_features<D>(sg, jp, c.xi, c.theta_c, c.theta_s, x);
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 7; ++k) ok = ok && fabsf(x[k]) <= c.sur_xmax[k];
  if (!ok) return false;
  const int slot = reserve_slot(c.sur_ctr);
  float* meta = c.sur_meta + (long long)slot * SUR_META;
  meta[0] = __int_as_float(j);
  meta[23] = __int_as_float(c.scene);
#pragma unroll
  for (int k = 0; k < D * D; ++k) {
    meta[1 + k] = U[k];
    meta[10 + k] = V[k];
  }
#pragma unroll
  for (int d = 0; d < D; ++d) meta[19 + d] = sg[d];
  meta[22] = jp;
#pragma unroll
  for (int k = 0; k < 7; ++k) c.sur_X[(long long)slot * 7 + k] = x[k];
  return true;
}

// Snow return map of G2P's trial state F (in place): states whose singular
// values are provably inside the clamp interval are unchanged; the others get
// an SVD, are recorded when the recorder samples this particle, and are
// projected exactly or handed to the surrogate.  In 3D without a surrogate the
// states near a rotation take snow_clamp_near, as in G2P, which lists them here
// only for a recorder: recording changes no result, and a state that is not
// sampled needs no SVD.
template <int D>
__device__ __forceinline__ void snow_return_map(const Ctx& c, float* F, float& jp, int j) {
  const float lo = 1.f - c.theta_c, hi = 1.f + c.theta_s;
  bool within = singular_values_within<D>(F, lo, hi), near = false;
  float Fn[D * D], jn = jp;
  if constexpr (D == 3) {
    if (c.rec_X && !c.sur) {
#pragma unroll
      for (int k = 0; k < D * D; ++k) Fn[k] = F[k];
      near = snow_clamp_near(Fn, jn, lo, hi);
      within = within || (near && j % c.rec_stride != 0);  // no SVD wanted
    }
  }
  if (!within) {
    float U[D * D], sg[D], V[D * D];
    svd_d<D>(F, U, sg, V);
    const bool dom = (c.rec_X || c.sur) && sur_domain<D>(F, sg, jp);
    if (c.rec_X && dom && j % c.rec_stride == 0) record_pair<D>(c, sg, jp);
    if (c.sur && dom && sur_handoff<D>(c, U, sg, V, jp, j)) return;
    if (!near) snow_clamp_rebuild<D>(c, U, sg, V, F, jp);
  }
  if (near) {
#pragma unroll
    for (int k = 0; k < D * D; ++k) F[k] = Fn[k];
    jp = jn;
  }
}

// F and Jp of particle j of a state (the rows' other words stay as they are).
template <int D>
__device__ __forceinline__ void store_elastic(const Particles& Q, int j, const float* F, float jp) {
  using W = PWord<D>;
  float4* q = Q.s + prow<D>(j);
  __stwb(q + 32, make_float4(F[0], F[1], F[2], F[3]));
  if (D == 3) {
    __stwb(q + 64, make_float4(F[4 % (D * D)], F[5 % (D * D)], F[6 % (D * D)], F[7 % (D * D)]));
    __stwb((float*)(q + 96), F[D * D - 1]);
  }
  __stwb((float*)Q.s + pword<D>(j, W::JP), jp);
}

// Apply the MLP's predictions: decode the projected singular values sig' and
// the change of log Jp, reject them when sig' leaves the clamp interval (the
// yield surface) or the change breaks the plastic-volume balance
// log Jp' - log Jp = sum log sig - sum log sig' by more than sur_tol (then the
// exact return map is used), and write F and Jp.
template <int D>
__global__ void k_sur_finish(Batch B, const float* __restrict__ meta_all, const float* __restrict__ Y,
                             const int32_t* __restrict__ n_dev) {
  const int n = *n_dev;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    const float* meta = meta_all + (long long)s * SUR_META;
    const int j = __float_as_int(meta[0]);
    const Ctx& c = B.ctx[__float_as_int(meta[23])];  // the slot's scene
    float U[D * D], V[D * D], sg[D];
#pragma unroll
    for (int k = 0; k < D * D; ++k) {
      U[k] = meta[1 + k];
      V[k] = meta[10 + k];
    }
#pragma unroll
    for (int d = 0; d < D; ++d) sg[d] = meta[19 + d];
    float jp = meta[22];
    const float* y = Y + (long long)s * 4;
    const float ts = c.theta_s, tcr = c.theta_c;
    float sp[D], r = 0.f, lsum = 0.f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      sp[d] = sg[d] + SUR_DSIG * y[d];
      r = fmaxf(r, fmaxf(sp[d] - (1.f + ts), (1.f - tcr) - sp[d]));
      lsum += logf(sg[d]) - logf(fmaxf(sp[d], 1e-6f));
    }
    const float dljp = SUR_DLJ * y[3];
    r = fmaxf(r, fabsf(dljp - lsum));
    float F[D * D];
    if (!(r <= c.sur_tol)) {
      snow_clamp_rebuild<D>(c, U, sg, V, F, jp);
      atomicAdd(&c.ctr[CTR_SURFB], 1);
    } else {
      jp = jp * expf(dljp);
#pragma unroll
      for (int a = 0; a < D; ++a)
#pragma unroll
        for (int b = 0; b < D; ++b) {
          float acc = 0.f;
#pragma unroll
          for (int k = 0; k < D; ++k) acc += U[a * D + k] * sp[k] * V[b * D + k];
          F[a * D + b] = acc;
        }
    }
    store_elastic<D>(c.Q, j, F, jp);
  }
}

// G2P writes the updated particles into Q in this substep's bin order, so the
// next substep reads every particle array with contiguous loads.  m, g and id
// travel with the particle; fl records the level used; particles without a
// level (the extra bin, level -1) are copied unchanged.
template <int D>
__device__ __forceinline__ void copy_particle(const Ctx& c, int p, int j) {
  const float4* src = c.P.s + prow<D>(p);
  float4* dst = c.Q.s + prow<D>(j);
#pragma unroll
  for (int k = 0; k < PWord<D>::NQ; ++k) __stwb(dst + 32 * k, src[32 * k]);
  __stwb(&c.Q.id[j], c.P.id[p]);
  __stwb(&c.Q.fl[j], -1);
}

// Factors of G2P that depend only on the scene and the level, computed once a
// CTA (they hold four divisions, 5 % of G2P's time: 256 2D scenes 154 -> 141
// us): s of F' = (I + s G) F per level, and the scale of the weights (kw) and
// of their gradients (kg).
struct G2PScale {
  float s[MAXL], kw, kg;
};
template <int D>
__device__ __forceinline__ void g2p_scale(const Ctx& c, G2PScale& sc) {
  if ((int)threadIdx.x < c.L) {
    const float pw = (D == 2) ? 0.25f : 0.125f;
    const float rd = (D == 2) ? c.radius * c.radius : c.radius * c.radius * c.radius;
    const float dx = 1.f / (float)(c.coarsest << (int)threadIdx.x);
    sc.s[threadIdx.x] = (c.dt * pw) / (rd * dx);
  }
  if (threadIdx.x == 32) {
    const float r2 = 2.f * c.radius;
    sc.kw = (D == 2) ? 1.f / (4.f * r2 * r2) : 1.f / (8.f * r2 * r2 * r2);
    sc.kg = (D == 2) ? 1.f / (2.f * r2 * r2) : 1.f / (4.f * r2 * r2 * r2);
  }
  __syncthreads();
}

// The end of G2P for particle p (slot j of this substep's bin order, level l):
// the new state from its position, node velocity nv and velocity gradient G
// (F' = (I + s G) F, whose Gram matrix decides whether the snow return map
// may change it).  st holds the rows of p before V (x, g, F, m, Jp).
template <int D>
__device__ __forceinline__ void g2p_finish(const Ctx& c, const G2PScale& sc, int l, int p, int j, const float4* st,
                                           const float* nv, const float* G) {
  using W = PWord<D>;
  const float s = sc.s[l];
  float F[D * D], A[D * D], Fn[D * D], Sg[(D == 2) ? 3 : 6];
#pragma unroll
  for (int k = 0; k < D * D; ++k) F[k] = qword(st, W::F + k);
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int k = 0; k < D; ++k) A[i * D + k] = (i == k ? 1.f : 0.f) + s * G[i * D + k];
#pragma unroll
  for (int k = 0; k < ((D == 2) ? 3 : 6); ++k) Sg[k] = 0.f;
#pragma unroll
  for (int i = 0; i < D; ++i) {
#pragma unroll
    for (int q = 0; q < D; ++q) {
      float a = 0.f;
#pragma unroll
      for (int k = 0; k < D; ++k) a += A[i * D + k] * F[k * D + q];
      Fn[i * D + q] = a;
    }
    int u = 0;
#pragma unroll
    for (int a = 0; a < D; ++a)
#pragma unroll
      for (int b = a; b < D; ++b) Sg[u++] += Fn[i * D + a] * Fn[i * D + b];
  }
  float w[4 * W::NQ];
#pragma unroll
  for (int k = 0; k < 4 * W::NQ; ++k) w[k] = 0.f;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    w[W::X + d] = qword(st, W::X + d) + c.dt * nv[d];
    w[W::V + d] = nv[d];
  }
#pragma unroll
  for (int k = 0; k < D * D; ++k) w[W::C + k] = G[k];
  w[W::M] = qword(st, W::M);
  w[W::G] = qword(st, W::G);
  float4* dst = c.Q.s + prow<D>(j);
  auto row = [&](int k) { __stwb(dst + 32 * k, make_float4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3])); };
  // the rows without F, Jp first: the return map needs the registers
#pragma unroll
  for (int k = 0; k < W::NQ; ++k)
    if (D == 3 && (k == 0 || k > 3)) row(k);
  __stwb(&c.Q.id[j], c.P.id[p]);
  __stwb(&c.Q.fl[j], l);
  // Trial states that may leave the elastic interval.  In 3D the ones near a
  // rotation are projected here: it takes some 150 operations in the registers
  // at hand.  Through the list and k_project it took another trip through
  // memory and, with the SVD, 1000 operations (1.9M particles: G2P 97 + SVD 94
  // us; G2P 98 + this projection in k_project 46; G2P with it 117, now 103).  The rest
  // is listed for k_project, whose SVD would halve G2P's occupancy.
  float jp = 1.f;
  if (c.plast == 1) {
    jp = qword(st, W::JP);
    const float lo = 1.f - c.theta_c, hi = 1.f + c.theta_s;
    // det F' = det(I + s G) det F
    if (!gram_within<D>(Sg, det<D>(A) * det<D>(F), lo, hi)) {
      bool done = false;
      if constexpr (D == 3) done = !c.rec_X && !c.sur && snow_clamp_near(Fn, jp, lo, hi);
      if (!done) c.proj[reserve_slot(&c.ctr[CTR_PROJ])] = j;
    }
  }
  w[W::JP] = jp;
#pragma unroll
  for (int k = 0; k < D * D; ++k) w[W::F + k] = Fn[k];
#pragma unroll
  for (int k = 0; k < W::NQ; ++k)
    if (!(D == 3 && (k == 0 || k > 3))) row(k);
}

// One particle, slot j of this substep's bin order; the 3^d nodes come
// through L1 (particles of a bin share a (4+2)^d node tile).
template <int D>
__device__ __forceinline__ void g2p_one(const Ctx& c, const G2PScale& sc, int j) {
  const int p = c.perm[j];
  const int l = c.P.fl[p];
  if (l < 0) {
    copy_particle<D>(c, p, j);
    return;
  }
  float4 st[4];  // the rows before V (2D: and the row of Jp)
  const float4* src = c.P.s + prow<D>(p);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (D == 3 || k != 2) st[k] = src[32 * k];
  float xp[D];
#pragma unroll
  for (int d = 0; d < D; ++d) xp[d] = qword(st, d);
  const LevelDev& V = c.lev[l];
  const float inv = (float)(c.coarsest << l);
  int base[D];
  float tc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float xs = xp[d] * inv;
    base[d] = (int)(xs + 0.5f) - 1;
    tc[d] = xs - (float)(base[d] + 1);
  }
  // Gather by rows along the last axis: the weights are products of per-axis
  // terms, so a row's nodes are first summed with the last axis's weight (S)
  // and gradient (T), and the other axes' factors are applied once per row.
  // Only the last axis's factors are kept; the others are formed when their
  // row starts (closed form for radius 1/2), which keeps G2P inside 64
  // registers with a slab of nodes in flight.
  const bool half = c.radius == 0.5f;
  float W2[3], G2[3];
  if (half)
    axis_weights_half(tc[D - 1], W2, G2);
  else
    axis_weights(tc[D - 1], c.radius, W2, G2);
  auto axis_factor = [&](float t, int k, float& w, float& g) {
    if (half) {
      const float a = 0.5f - t, b = 0.5f + t;
      w = k == 0 ? a * a : (k == 1 ? fmaf(-2.f * t, t, 1.5f) : b * b);
      g = k == 0 ? -a : (k == 1 ? -2.f * t : b);
    } else {
      float Wk[3], Gk[3];
      axis_weights(t, c.radius, Wk, Gk);
      w = k == 0 ? Wk[0] : (k == 1 ? Wk[1] : Wk[2]);
      g = k == 0 ? Gk[0] : (k == 1 ? Gk[1] : Gk[2]);
    }
  };
  const float kw = sc.kw, kg = sc.kg;
  float nv[D], G[D * D];
#pragma unroll
  for (int i = 0; i < D; ++i) nv[i] = 0.f;
#pragma unroll
  for (int i = 0; i < D * D; ++i) G[i] = 0.f;
#pragma unroll(D == 3 ? 1 : 3)
  for (int n0 = 0; n0 < 3; ++n0) {
    float w0, g0;
    axis_factor(tc[0], n0, w0, g0);
    // one row (3 nodes) in flight at a time: measured faster than a slab of
    // 9 gathers, which does not fit the 64-register budget
#pragma unroll 1
    for (int n1 = 0; n1 < ((D == 2) ? 1 : 3); ++n1) {
      float S[D], T[D];
#pragma unroll
      for (int i = 0; i < D; ++i) S[i] = T[i] = 0.f;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        int I[D];
        I[0] = base[0] + n0;
        if (D == 3) I[1] = base[1] + n1;
        I[D - 1] = base[D - 1] + k;
        // base lies in [-1, size-1] for an in-domain particle: always in store
        const float4 nd = V.node[elem_of<D>(V, I)];
        const float gv[3] = {nd.x, nd.y, nd.z};
#pragma unroll
        for (int i = 0; i < D; ++i) {
          S[i] += gv[i] * W2[k];
          T[i] += gv[i] * G2[k];
        }
      }
      // row factors: weight, and the gradient components of the other axes
      float cw, cg[D];
      if (D == 2) {
        cw = w0 * kw;
        cg[0] = g0 * kg;
        cg[1] = w0 * kg;
      } else {
        float w1, g1;
        axis_factor(tc[1], n1, w1, g1);
        const float wxy = w0 * w1;
        cw = wxy * kw;
        cg[0] = g0 * w1 * kg;
        cg[1] = w0 * g1 * kg;
        cg[D - 1] = wxy * kg;
      }
#pragma unroll
      for (int i = 0; i < D; ++i) {
        nv[i] += cw * S[i];
#pragma unroll
        for (int q = 0; q < D - 1; ++q) G[i * D + q] += cg[q] * S[i];
        G[i * D + D - 1] += cg[D - 1] * T[i];
      }
    }
  }
  g2p_finish<D>(c, sc, l, p, j, st, nv, G);
}

// 2D G2P: one thread per particle slot, grid-stride (a 2D block holds about
// one work item, too little to pay for staging its nodes).
template <int D>
__global__ void __launch_bounds__(256, 4) k_g2p_gather(Batch B) {
  SCENE_CTA(B, MAP_W);
  __shared__ G2PScale sc;
  g2p_scale<D>(c, sc);
  SCENE_LOOP(j, c.N) g2p_one<D>(c, sc, (int)j);
}

// The new state of particle p (slot j of this substep's bin order) whose
// base cell lies in the block with first node O, from the block's staged
// node velocities: txy[t] = (v_x, v_y), tz[t] = v_z of tile node t (the
// (4+2)^d nodes O..O+5, last axis fastest).
template <int D>
__device__ __forceinline__ void g2p_staged(const Ctx& c, const G2PScale& sc, int l, int p, int j, const float4* st,
                                           const int* O, const float2* txy, const float* tz) {
  const float inv = (float)(c.coarsest << l);
  float tc[D];
  int t0 = 0;
  bool inside = true;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float xs = qword(st, d) * inv;
    const int base = (int)(xs + 0.5f) - 1;
    tc[d] = xs - (float)(base + 1);
    // the binning put the base cell in this block; a cell outside it would
    // read another tile's nodes, so it is clamped and reported
    int r = base - O[d];
    inside = inside && r >= 0 && r <= 3;
    r = min(max(r, 0), 3);
    t0 = t0 * 6 + r;
  }
  if (!inside) set_err(c, ERR_OOB);
  const bool half = c.radius == 0.5f;
  float W2[3], G2[3];
  if (half)
    axis_weights_half(tc[D - 1], W2, G2);
  else
    axis_weights(tc[D - 1], c.radius, W2, G2);
  auto axis_factor = [&](float t, int k, float& w, float& g) {
    if (half) {
      const float a = 0.5f - t, b = 0.5f + t;
      w = k == 0 ? a * a : (k == 1 ? fmaf(-2.f * t, t, 1.5f) : b * b);
      g = k == 0 ? -a : (k == 1 ? -2.f * t : b);
    } else {
      float Wk[3], Gk[3];
      axis_weights(t, c.radius, Wk, Gk);
      w = k == 0 ? Wk[0] : (k == 1 ? Wk[1] : Wk[2]);
      g = k == 0 ? Gk[0] : (k == 1 ? Gk[1] : Gk[2]);
    }
  };
  const float kw = sc.kw, kg = sc.kg;
  float nv[D], G[D * D];
#pragma unroll
  for (int i = 0; i < D; ++i) nv[i] = 0.f;
#pragma unroll
  for (int i = 0; i < D * D; ++i) G[i] = 0.f;
  // Rows along the last axis: a row's nodes are summed with the last axis's
  // weight (S) and gradient (T) first; the other axes' factors are applied
  // once per row.  (Summing planes before the first axis as well saves a third
  // of the multiply-adds, but its partial sums do not fit the 64 registers:
  // 114 against 111 us for 1.9M particles, 34.6 against 30.7 for 600,000.)
#pragma unroll
  for (int n0 = 0; n0 < 3; ++n0) {
    float w0, g0;
    axis_factor(tc[0], n0, w0, g0);
#pragma unroll
    for (int n1 = 0; n1 < ((D == 2) ? 1 : 3); ++n1) {
      const int tr = t0 + n0 * ((D == 2) ? 6 : 36) + ((D == 2) ? 0 : n1 * 6);
      float2 Sxy = make_float2(0.f, 0.f), Txy = make_float2(0.f, 0.f);
      float Sz = 0.f, Tz = 0.f;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float2 v = txy[tr + k];
        Sxy = ffma2(v, dup2(W2[k]), Sxy);
        Txy = ffma2(v, dup2(G2[k]), Txy);
        if (D == 3) {
          const float vz = tz[tr + k];
          Sz = fmaf(vz, W2[k], Sz);
          Tz = fmaf(vz, G2[k], Tz);
        }
      }
      const float S[3] = {Sxy.x, Sxy.y, Sz}, T[3] = {Txy.x, Txy.y, Tz};
      // row factors: weight, and the gradient components of the other axes
      float cw, cg[D];
      if (D == 2) {
        cw = w0 * kw;
        cg[0] = g0 * kg;
        cg[1] = w0 * kg;
      } else {
        float w1, g1;
        axis_factor(tc[1], n1, w1, g1);
        const float wxy = w0 * w1;
        cw = wxy * kw;
        cg[0] = g0 * w1 * kg;
        cg[1] = w0 * g1 * kg;
        cg[D - 1] = wxy * kg;
      }
#pragma unroll
      for (int i = 0; i < D; ++i) {
        nv[i] = fmaf(cw, S[i], nv[i]);
#pragma unroll
        for (int q = 0; q < D - 1; ++q) G[i * D + q] = fmaf(cg[q], S[i], G[i * D + q]);
        G[i * D + D - 1] = fmaf(cg[D - 1], T[i], G[i * D + D - 1]);
      }
    }
  }
  g2p_finish<D>(c, sc, l, p, j, st, nv, G);
}

// 3D G2P (adaptive_gimp.py:289-321) over its work items (k_bins): a CTA takes a
// contiguous range of them (up to CH particles of one 4^3 block each); when
// the block changes it stages the block's 6^3 node velocities in shared
// memory (two tiles alternate, so one barrier per block suffices: a thread
// that passed the previous barrier has finished reading the tile from two
// blocks ago), and each thread then computes one particle from the tile.
// Particles without a level (the extra bin) are copied unchanged.
template <int D, int CH>
__global__ void __launch_bounds__(CH, 1024 / CH) k_g2p(Batch B) {
  SCENE_CTA(B, MAP_W);
  constexpr int TN = 216;
  __shared__ float2 txy[2][TN];
  __shared__ float tz[2][TN];
  __shared__ G2PScale sc;
  g2p_scale<D>(c, sc);
  __shared__ int4 item[32];
  const int nch = c.ctr[CTR_CHUNKS];
  const int q = nch / nblk_, extra = nch - q * nblk_;
  const int c0 = bid_ * q + min(bid_, extra), c1 = c0 + q + (bid_ < extra);
  const int i = threadIdx.x;
  // The items of this CTA come 32 at a time through shared memory and a
  // particle's source slot is read one item ahead, so an item starts with the
  // reads of its particles' rows (600,000 static particles 27.4 -> 25.3 us).
  // Items of 128 particles, not 256, halve the lanes idle in a block's last
  // item (30.7 -> 27.4; 1.9M particles 111 -> 107); 64 load a tile for too few
  // (33, 138).
  auto source = [&](const int4& w) { return i < w.w ? c.perm[w.z + i] : 0; };
  int tb = 1, tl = -1, tk = -1, next = 0;
  for (int ch = c0; ch < c1; ++ch) {
    const int k0 = (ch - c0) & 31;
    if (k0 == 0) {
      __syncthreads();
      if (i < 32 && ch + i < c1) item[i] = c.chunks[ch + i];
      __syncthreads();
      next = source(item[0]);
    }
    const int4 wd = item[k0];
    const int p = next, j = wd.z + i;
    const bool mine = i < wd.w;
    if (wd.x < 0) {  // uniform over the CTA
      if (mine) copy_particle<D>(c, p, j);
      if (k0 < 31 && ch + 1 < c1) next = source(item[k0 + 1]);
      continue;
    }
    const int l = wd.x;
    const LevelDev& V = c.lev[l];
    int O[D];
    chunk_origin<D>(V, wd.y, O);
    // the particle's rows before V are requested before the tile load, so both
    // latencies overlap
    float4 st[4];
    if (mine) {
      const float4* src = c.P.s + prow<D>(p);
#pragma unroll
      for (int k = 0; k < 4; ++k) st[k] = src[32 * k];
    }
    if (k0 < 31 && ch + 1 < c1) next = source(item[k0 + 1]);
    if (l != tl || wd.y != tk) {  // uniform over the CTA
      tb ^= 1;
      tl = l;
      tk = wd.y;
      for (int t = threadIdx.x; t < TN; t += CH) {
        int I[D], r = t;
#pragma unroll
        for (int d = D - 1; d >= 0; --d) {
          I[d] = O[d] + r % 6;
          r /= 6;
        }
        float4 nd = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in_store<D>(V, I)) nd = V.node[elem_of<D>(V, I)];
        txy[tb][t] = make_float2(nd.x, nd.y);
        tz[tb][t] = nd.z;
      }
      __syncthreads();
    }
    if (mine) g2p_staged<D>(c, sc, l, p, j, st, O, txy[tb], tz[tb]);
  }
}

// Snow return map (extension) of the particles G2P listed (2D: all that may
// leave the elastic interval; 3D: those far from a rotation, or all when a
// recorder or surrogate wants their SVD): the trial state written to Q is
// projected in place (or handed to the surrogate).
template <int D>
__global__ void __launch_bounds__(256) k_project(Batch B) {
  SCENE_CTA(B, MAP_G);
  if (c.plast != 1) return;
  const int n = c.ctr[CTR_PROJ];
  using W = PWord<D>;
  SCENE_LOOP(s, n) {
    const int j = c.proj[s];
    const float4* src = c.Q.s + prow<D>(j);
    float4 st[4];
#pragma unroll
    for (int k = 1; k < 4; ++k)
      if (D == 3 || k != 2) st[k] = src[32 * k];
    float F[D * D];
#pragma unroll
    for (int k = 0; k < D * D; ++k) F[k] = qword(st, W::F + k);
    float jp = qword(st, W::JP);
    snow_return_map<D>(c, F, jp, j);
    store_elastic<D>(c.Q, j, F, jp);
  }
}

// ---------------------------------------------------------------------------
template <int D>
static void set_p2g_smem() {
  cudaFuncSetAttribute(k_p2g<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P2GLayout<D>::bytes());
}

// CTAs of k_p2g that one SM holds at once
int p2g_resident(int dim) {
  int n = 0;
  if (dim == 2)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_p2g<2>, 32 * P2GLayout<2>::WARPS, P2GLayout<2>::bytes());
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_p2g<3>, 32 * P2GLayout<3>::WARPS, P2GLayout<3>::bytes());
  return n > 0 ? n : 1;
}

void prepare_transfer_kernels() {
  set_p2g_smem<2>();
  set_p2g_smem<3>();
}

template <int D>
static void launch_p2g(const BatchLaunch& bl, cudaStream_t s, bool pdl) {
  using Y = P2GLayout<D>;
  launch_k(pdl, k_p2g<D>, bl.nct[MAP_P], 32 * Y::WARPS, Y::bytes(), s, bl.b);
}

template <int D>
static void launch_g2p(const BatchLaunch& bl, cudaStream_t s, bool pdl) {
  const int W = bl.nct[MAP_W];
  if constexpr (D == 2) {
    launch_k(pdl, k_g2p_gather<D>, W, 256, 0, s, bl.b);
  } else {
    switch (bl.chunk) {
      case 64: launch_k(pdl, k_g2p<D, 64>, W, 64, 0, s, bl.b); break;
      case 128: launch_k(pdl, k_g2p<D, 128>, W, 128, 0, s, bl.b); break;
      case 512: launch_k(pdl, k_g2p<D, 512>, W, 512, 0, s, bl.b); break;
      default: launch_k(pdl, k_g2p<D, 256>, W, 256, 0, s, bl.b); break;
    }
  }
}

template <int D>
void launch_transfer(const BatchLaunch& bl, cudaStream_t s, cudaEvent_t* ev) {
  const int G = bl.nct[MAP_G];
  const bool pdl = bl.pdl && !ev;
  launch_p2g<D>(bl, s, pdl);
  if (bl.side) cudaStreamWaitEvent(s, bl.join, 0);  // k_ghost_tj's node mask
  if (ev) cudaEventRecord(ev[4], s);
  // the first launch after the join is a plain one
  bool first = true;
  for (int l = bl.maxL - 1; l >= 1; --l, first = false) {
    if constexpr (staged_transfers<D>())
      launch_k(pdl && !(first && bl.side), k_restrict<D>, bl.nct[MAP_T], Stage<D>::PER, 0, s, bl.b, l);
    else
      launch_k(pdl && !(first && bl.side), k_restrict_gather<D>, G, 256, 0, s, bl.b, l);
  }
  if (ev) cudaEventRecord(ev[5], s);
  // with more than one level grid_op runs inside the restriction into level 0
  // and the prolongations
  if (bl.maxL == 1) launch_k(pdl && !bl.side, k_gridop<D>, G, 256, 0, s, bl.b);
  if (ev) cudaEventRecord(ev[6], s);
  for (int l = 1; l < bl.maxL; ++l) {
    if constexpr (staged_transfers<D>())
      launch_k(pdl, k_prolong<D>, bl.nct[MAP_T], Stage<D>::PER, 0, s, bl.b, l);
    else
      launch_k(pdl, k_prolong_gather<D>, G, 256, 0, s, bl.b, l);
  }
  if (ev) cudaEventRecord(ev[7], s);
  launch_g2p<D>(bl, s, pdl);
  if (bl.any_plastic) launch_k(pdl, k_project<D>, G, 256, 0, s, bl.b);
  if (bl.sur) {
    launch_mlp_forward_dev(bl.mlp_packed, bl.mlp_P, bl.sur_X, bl.sur_Y, bl.sur_n, bl.sur_cap, bl.sur_err, bl.sms, s);
    k_sur_finish<D><<<G, 256, 0, s>>>(bl.b, bl.sur_meta, bl.sur_Y, bl.sur_n);
  }
  if (ev) cudaEventRecord(ev[8], s);
}

template void launch_transfer<2>(const BatchLaunch&, cudaStream_t, cudaEvent_t*);
template void launch_transfer<3>(const BatchLaunch&, cudaStream_t, cudaEvent_t*);

}  // namespace agimp
