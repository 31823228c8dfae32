// mpm_world.cu -- the MPM substep on sm_100a: kernels and the world driver.
//
// Substep (every scene of a world at once):
//   sort     counts per grid node -> places (radix sort of cell keys where the grid is huge for its
//            particles) -> perm (sorted position -> storage slot)
//   grid     one pass over the blocks P2G touched: momentum -> velocity, gravity, walls;
//            clears the accumulator and the touched flags for the next substep
//   G2P      one thread per sorted particle: gather, APIC C, F update and material return
//            mapping, written to the other particle buffer in sorted order (the reorder costs
//            nothing extra), plus the next substep's cell key
//   P2G      sums per cell run of a warp, added to the grid with 16-byte vector atomics
//            (red.global.add.v4.f32).  In physics mode the G2P kernel scatters its particles for
//            the next substep while they are in registers; P2G alone is the first substep's
// Deterministic mode replaces P2G's float atomics with per-cell fixed-order sums and a per-node
// fixed-order gather (no float atomics anywhere), so two runs are bitwise identical.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <memory>

#include "device_util.cuh"
#include "mpm_world.cuh"

namespace aemp {

// ============================================================================================
// device helpers
// ============================================================================================
template <class T>
struct Bits;
template <>
struct Bits<float> {
  static __device__ __forceinline__ float pack(uint32_t u) { return __uint_as_float(u); }
  static __device__ __forceinline__ uint32_t unpack(float f) { return __float_as_uint(f); }
};
template <>
struct Bits<double> {
  static __device__ __forceinline__ double pack(uint32_t u) { return __longlong_as_double((long long)u); }
  static __device__ __forceinline__ uint32_t unpack(double d) { return uint32_t(__double_as_longlong(d)); }
};

__device__ __forceinline__ float4 ld4(const float4* p) { return __ldg(p); }
__device__ __forceinline__ double4 ld4(const double4* p) {
  const double2* q = reinterpret_cast<const double2*>(p);
  double2 a = __ldg(q), b = __ldg(q + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 mk4(float a, float b, float c, float d) { return make_float4(a, b, c, d); }
__device__ __forceinline__ double4 mk4(double a, double b, double c, double d) { return make_double4(a, b, c, d); }

__device__ __forceinline__ void atomic_add4(float4* p, float a, float b, float c, float d) {
  atomicAdd(p, make_float4(a, b, c, d));  // one 16-byte vector reduction (sm_90+)
}
__device__ __forceinline__ void atomic_add4(double4* p, double a, double b, double c, double d) {
  atomicAdd(&p->x, a);
  atomicAdd(&p->y, b);
  atomicAdd(&p->z, c);
  atomicAdd(&p->w, d);
}

// asynchronous 16-byte global -> shared copies (cp.async, no registers held while in flight)
__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}
// A work counter that an earlier kernel wrote and that no thread of this kernel changes, read by
// every thread: an ordinary load, which each SM's L1 serves after the first.  (A volatile or L2-only
// load would send every warp of the grid to the same L2 slice before any of them could start.  The
// read-only path is for data that does not change while the kernel runs, and a kernel launched
// dependently runs before its predecessor has written.)
__device__ __forceinline__ uint32_t launch_count(const uint32_t* p) { return *p; }

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }
template <class V4>
__device__ __forceinline__ void cp_async_v4(V4* sdst, const V4* gsrc) {
#pragma unroll
  for (int k = 0; k < int(sizeof(V4) / 16); ++k)
    cp_async16(reinterpret_cast<char*>(sdst) + 16 * k, reinterpret_cast<const char*>(gsrc) + 16 * k);
}

template <class T>
__device__ __forceinline__ int floor_to_int(T v) {
  if (v != v) return 0;  // NaN -> 0, as Rust's `as isize`
  v = t_clamp(v, T(-1.0e9), T(1.0e9));
  return int(t_floor(v));
}

template <class T>
__device__ __forceinline__ uint32_t node_index(const SceneDev<T>& sc, int i, int j, int k) {
  uint32_t b = (uint32_t(k >> 2) * uint32_t(sc.nb[1]) + uint32_t(j >> 2)) * uint32_t(sc.nb[0]) + uint32_t(i >> 2);
  return (sc.blk_off + b) * 64u + ((uint32_t(k & 3) << 4) | (uint32_t(j & 3) << 2) | uint32_t(i & 3));
}

template <class T>
__device__ __forceinline__ T sel3(const T* a, int i) {
  return i == 0 ? a[0] : (i == 1 ? a[1] : a[2]);
}

// cell key of a position: physics mode base clamped into the grid; reference modes base clamped
// at 0 (Grid::pos_to_grid, mpm_solver.rs:161-175) and the dead key when the stencil is off-grid
template <class T>
__device__ __forceinline__ uint32_t cell_key(const SceneDev<T>& sc, int mode, T x, T y, T z) {
  T p[3] = {x, y, z};
  int b[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int g = floor_to_int((p[a] - sc.origin[a]) * sc.inv_dx - T(0.5));
    if (mode == AE_MPM_MODE_PHYSICS) {
      g = min(max(g, 0), sc.n[a] - 1);
    } else {
      g = max(g, 0);
      if (g >= sc.n[a]) return sc.dead_key;
    }
    b[a] = g;
  }
  return node_index(sc, b[0], b[1], b[2]);
}

// The chunk a CTA works on: {scene, first slot, end of the live particles, end of capacity}.
// A world of one scene needs no table (its chunks are consecutive ranges of blockDim.x slots),
// so its CTAs start their particle loads without first waiting for a descriptor load.
template <class T>
__device__ __forceinline__ int4 chunk_at(const WorldDev<T>& w, uint32_t chunk, uint32_t slots) {
  if (w.one_scene) {
    const uint64_t lo = uint64_t(w.one_off) + uint64_t(chunk) * slots;
    const uint64_t live = lo + slots < w.one_live_end ? lo + slots : w.one_live_end;
    const uint64_t cap = lo + slots < w.one_cap_end ? lo + slots : w.one_cap_end;
    return make_int4(0, int(lo), int(live > lo ? live : lo), int(cap));
  }
  return w.chunks[chunk];
}
template <class T>
__device__ __forceinline__ int4 cta_chunk(const WorldDev<T>& w) {
  return chunk_at(w, blockIdx.x, blockDim.x);
}

template <class T>
__device__ __forceinline__ void mark_block(const WorldDev<T>& w, uint32_t gb) {
  volatile uint32_t* f = w.blk_flag + gb;
  if (*f == 0u && atomicExch(w.blk_flag + gb, 1u) == 0u) {
    uint32_t slot = atomicAdd(w.touched_count, 1u);
    w.touched[slot] = gb;
  }
}

// Deterministic sums: marks block `corner` (0..7) of the at most two blocks per axis that the stencil
// based at (g0, g1, g2) spans.  A particle uploaded outside the grid has that base unclamped until its
// first G2P, wherever it lies: both ends are clamped into the grid (a block marked without need is an
// update of unchanged nodes).
template <class T>
__device__ __forceinline__ void mark_stencil_corner(const WorldDev<T>& w, const SceneDev<T>& sc, int corner, int g0,
                                                    int g1, int g2) {
  const int X = min(max(g0 + 2 * (corner & 1), 0), sc.n[0] - 1);
  const int Y = min(max(g1 + (corner & 2), 0), sc.n[1] - 1);
  const int Z = min(max(g2 + ((corner & 4) >> 1), 0), sc.n[2] - 1);
  mark_block(w, sc.blk_off + (uint32_t(Z >> 2) * sc.nb[1] + (Y >> 2)) * sc.nb[0] + (X >> 2));
}

template <class T>
__device__ __forceinline__ const MatDev& mat_of(const WorldDev<T>& w, const SceneDev<T>& sc, uint32_t m) {
  return w.mats[sc.mat_off + (m < sc.n_mat ? m : sc.n_mat)];
}

// MLS-MPM affine momentum matrix (Hu et al. 2018): A = m C - k tau(F, J) with
// k = 4 dt V0 / dx^2, V0 = m / rho.  Physics mode stores A in the particle's C slot between
// substeps (G2P computes it while F is in registers), so P2G needs neither F nor the stress;
// pack/unpack convert to and from the caller's C at the boundary.
template <class T>
__device__ __forceinline__ T affine_k(const SceneDev<T>& sc, const MatDev& md, T m) {
  return T(4) * sc.dt * (m / T(md.rho)) * sc.inv_dx * sc.inv_dx;
}
template <class T>
__device__ __forceinline__ void affine_from_c(const SceneDev<T>& sc, const MatDev& md, T m, const T* C, const T* F, T J,
                                              T* A) {
  T tau[9];
  phys_tau(md, F, J, tau);
  const T k = affine_k(sc, md, m);
#pragma unroll
  for (int i = 0; i < 9; ++i) A[i] = m * C[i] - k * tau[i];
}

// ============================================================================================
// per-particle P2G setup
// ============================================================================================
template <class T>
struct P2GPart {
  int g[3];     // stencil base node per axis (nodes g..g+2)
  T w[3][3];    // per-axis weights
  T o[3][3];    // physics: (k - fx) dx;  reference: node position - particle position
  T fx[3];      // physics: position relative to the base node, in cells (in [0.5, 1.5))
  T dw[3][3];   // reference: N'(k - fx) / dx
  T m;
  T v[3];       // physics: m v;  reference/velonly: v
  T A[9];       // physics: m C - 4 dt V0/dx^2 tau;  reference: C
  T sv[9];      // reference: dt * V * sigma
};

template <class T, int MODE>
__device__ __forceinline__ void p2g_setup(const WorldDev<T>& w, const SceneDev<T>& sc, uint32_t src, P2GPart<T>& p) {
  using V4 = typename V4T<T>::type;
  const V4 a0 = ld4(w.in[0] + src);
  const V4 a4 = ld4(w.in[4] + src);
  T x[3] = {a0.x, a0.y, a0.z};
  p.m = a0.w;
  if (MODE == AE_MPM_MODE_VELOCITY_ONLY) {
    p.v[0] = a4.x;
    p.v[1] = a4.y;
    p.v[2] = a4.z;
  } else if (MODE == AE_MPM_MODE_PHYSICS) {
    const V4 a5 = ld4(w.in[5] + src), a6 = ld4(w.in[6] + src);
    const T A[9] = {a4.w, a5.x, a5.y, a5.z, a5.w, a6.x, a6.y, a6.z, a6.w};
#pragma unroll
    for (int k = 0; k < 9; ++k) p.A[k] = A[k];
    p.v[0] = p.m * a4.x;
    p.v[1] = p.m * a4.y;
    p.v[2] = p.m * a4.z;
  } else {
    const V4 a1 = ld4(w.in[1] + src), a2 = ld4(w.in[2] + src), a3 = ld4(w.in[3] + src);
    const V4 a5 = ld4(w.in[5] + src), a6 = ld4(w.in[6] + src);
    T F[9] = {a1.x, a1.y, a1.z, a1.w, a2.x, a2.y, a2.z, a2.w, a3.x};
    T C[9] = {a4.w, a5.x, a5.y, a5.z, a5.w, a6.x, a6.y, a6.z, a6.w};
    T J = a3.y;
    const MatDev& md = mat_of(w, sc, Bits<T>::unpack(a3.z) & 0xffffu);
    {
      T st[9];
      ref_stress(md, F, J, st);
      T vol = p.m / T(md.rho);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        p.sv[k] = sc.dt * (vol * st[k]);
        p.A[k] = C[k];
      }
      p.v[0] = a4.x;
      p.v[1] = a4.y;
      p.v[2] = a4.z;
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T X = (x[a] - sc.origin[a]) * sc.inv_dx;
    if (MODE == AE_MPM_MODE_PHYSICS) {
      int b = floor_to_int(X - T(0.5));
      T fx = X - T(b);
      p.g[a] = b;
      p.fx[a] = fx;
      T t0 = T(1.5) - fx, t1 = fx - T(1), t2 = fx - T(0.5);
      p.w[a][0] = T(0.5) * t0 * t0;
      p.w[a][1] = T(0.75) - t1 * t1;
      p.w[a][2] = T(0.5) * t2 * t2;
#pragma unroll
      for (int k = 0; k < 3; ++k) p.o[a][k] = (T(k) - fx) * sc.dx;
    } else {
      int gu = floor_to_int(X - T(0.5));
      T fx = X - T(0.5) - T(gu);
      int g = max(gu, 0);
      p.g[a] = g;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p.w[a][k] = b_spline(T(k) - fx);
        if (MODE == AE_MPM_MODE_REFERENCE) {
          p.dw[a][k] = b_spline_deriv(T(k) - fx) * sc.inv_dx;
          p.o[a][k] = (T(g + k) + T(0.5)) * sc.dx + sc.origin[a] - x[a];
        }
      }
    }
  }
}

// Contribution of a particle to stencil node (a,b,c); returns false when the node is skipped.
template <class T, int MODE>
__device__ __forceinline__ bool p2g_contrib(const SceneDev<T>& sc, const P2GPart<T>& p, int a, int b, int c, T& cm,
                                            T& cx, T& cy, T& cz) {
  int X = p.g[0] + a, Y = p.g[1] + b, Z = p.g[2] + c;
  if (X < 0 || Y < 0 || Z < 0 || X >= sc.n[0] || Y >= sc.n[1] || Z >= sc.n[2]) return false;
  T wx = sel3(p.w[0], a), wy = sel3(p.w[1], b), wz = sel3(p.w[2], c);
  if (MODE == AE_MPM_MODE_PHYSICS) {
    T w = wx * wy * wz;
    T d0 = sel3(p.o[0], a), d1 = sel3(p.o[1], b), d2 = sel3(p.o[2], c);
    cm = w * p.m;
    cx = w * (p.v[0] + p.A[0] * d0 + p.A[1] * d1 + p.A[2] * d2);
    cy = w * (p.v[1] + p.A[3] * d0 + p.A[4] * d1 + p.A[5] * d2);
    cz = w * (p.v[2] + p.A[6] * d0 + p.A[7] * d1 + p.A[8] * d2);
    return true;
  } else if (MODE == AE_MPM_MODE_REFERENCE) {
    T w = wx * wy * wz;
    if (w < T(1e-10)) return false;
    T d0 = sel3(p.o[0], a), d1 = sel3(p.o[1], b), d2 = sel3(p.o[2], c);
    T vx = p.v[0] + p.A[0] * d0 + p.A[1] * d1 + p.A[2] * d2;
    T vy = p.v[1] + p.A[3] * d0 + p.A[4] * d1 + p.A[5] * d2;
    T vz = p.v[2] + p.A[6] * d0 + p.A[7] * d1 + p.A[8] * d2;
    T e0 = sel3(p.dw[0], a), e1 = sel3(p.dw[1], b), e2 = sel3(p.dw[2], c);
    T wm = w * p.m;
    cm = wm;
    cx = wm * vx + (p.sv[0] * e0 + p.sv[1] * e1 + p.sv[2] * e2);
    cy = wm * vy + (p.sv[3] * e0 + p.sv[4] * e1 + p.sv[5] * e2);
    cz = wm * vz + (p.sv[6] * e0 + p.sv[7] * e1 + p.sv[8] * e2);
    return true;
  } else {
    if (wz < T(1e-10) || wy < T(1e-10)) return false;
    T w = wx * (wy * wz);
    if (w < T(1e-10)) return false;
    T wm = w * p.m;
    cm = wm;
    cx = wm * p.v[0];
    cy = wm * p.v[1];
    cz = wm * p.v[2];
    return true;
  }
}

// ============================================================================================
// P2G
// ============================================================================================
enum { kVarTile = 1, kVarWarpAgg = 2, kVarGlobal = 3, kVarLanes = 4 };

template <class T>
__device__ __forceinline__ void shared_add4(typename V4T<T>::type* t, T a, T b, T c, T d) {
  T* q = reinterpret_cast<T*>(t);
  atomicAdd(q + 0, a);
  atomicAdd(q + 1, b);
  atomicAdd(q + 2, c);
  atomicAdd(q + 3, d);
}

template <class T, int MODE, int VAR>
__global__ void __launch_bounds__(512) p2g_kernel(WorldDev<T> w) {
  using V4 = typename V4T<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  V4* tile = reinterpret_cast<V4*>(smem);
  __shared__ int s_lo[3], s_hi[3];
  const int tid = threadIdx.x, lane = tid & 31;
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  if (tid < 3) {
    s_lo[tid] = INT_MAX;
    s_hi[tid] = INT_MIN;
  }
  __syncthreads();
  const int j = ch.y + tid;
  const bool live = j < ch.z;
  P2GPart<T> p;
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
  bool has = false;
  if (live) {
    const uint32_t src = w.perm ? w.perm[j] : uint32_t(j);
    p2g_setup<T, MODE>(w, sc, src, p);
    has = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = max(p.g[a], 0);
      hi[a] = min(p.g[a] + 2, sc.n[a] - 1);
      if (lo[a] > hi[a]) has = false;
    }
  }
  // block bounding box of all in-grid stencil nodes
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int l = __reduce_min_sync(0xffffffffu, has ? lo[a] : INT_MAX);
    int h = __reduce_max_sync(0xffffffffu, has ? hi[a] : INT_MIN);
    if (lane == 0 && l != INT_MAX) {
      atomicMin(&s_lo[a], l);
      atomicMax(&s_hi[a], h);
    }
  }
  __syncthreads();
  const int L0 = s_lo[0], L1 = s_lo[1], L2 = s_lo[2];
  const bool any = L0 != INT_MAX;
  const int D0 = any ? s_hi[0] - L0 + 1 : 0, D1 = any ? s_hi[1] - L1 + 1 : 0, D2 = any ? s_hi[2] - L2 + 1 : 0;
  const int vol = D0 * D1 * D2;
  const bool use_tile = VAR != kVarGlobal && any && vol <= w.max_tile_nodes;
  if (!any) return;
  if (use_tile) {
    for (int t = tid; t < vol; t += blockDim.x) tile[t] = mk4(T(0), T(0), T(0), T(0));
    __syncthreads();
    if (VAR == kVarWarpAgg) {
      // lanes of one cell are one run in sorted order: reduce each run with shuffles and let its
      // first lane add the run's sum to the tile
      uint32_t key = has ? uint32_t(((p.g[2] - L2 + 2) * (D1 + 4) + (p.g[1] - L1 + 2)) * (D0 + 4) + (p.g[0] - L0 + 2))
                         : (0x80000000u | uint32_t(lane));
      uint32_t peers = __match_any_sync(0xffffffffu, key);
      int first = __ffs(peers) - 1;
      int cnt = __popc(peers);
      uint32_t run = (cnt == 32) ? 0xffffffffu : (((1u << cnt) - 1u) << first);
      bool contiguous = peers == run;
      int last = first + cnt - 1;
      int gmax = __reduce_max_sync(0xffffffffu, cnt);
      if (__all_sync(0xffffffffu, contiguous)) {
#pragma unroll 1
        for (int o = 0; o < 27; ++o) {
          const int a = o % 3, b = (o / 3) % 3, c = o / 9;
          T cm = T(0), cx = T(0), cy = T(0), cz = T(0);
          bool ok = has && p2g_contrib<T, MODE>(sc, p, a, b, c, cm, cx, cy, cz);
          if (!ok) cm = cx = cy = cz = T(0);
          for (int off = 1; off < gmax; off <<= 1) {
            T tm = __shfl_down_sync(0xffffffffu, cm, off);
            T tx = __shfl_down_sync(0xffffffffu, cx, off);
            T ty = __shfl_down_sync(0xffffffffu, cy, off);
            T tz = __shfl_down_sync(0xffffffffu, cz, off);
            if (lane + off <= last) {
              cm += tm;
              cx += tx;
              cy += ty;
              cz += tz;
            }
          }
          if (has && lane == first) {
            int X = p.g[0] + a, Y = p.g[1] + b, Z = p.g[2] + c;
            if (X >= 0 && Y >= 0 && Z >= 0 && X < sc.n[0] && Y < sc.n[1] && Z < sc.n[2] && cm != T(0))
              shared_add4<T>(tile + ((Z - L2) * D1 + (Y - L1)) * D0 + (X - L0), cm, cx, cy, cz);
          }
        }
      } else if (has) {
        for (int o = 0; o < 27; ++o) {
          const int a = o % 3, b = (o / 3) % 3, c = o / 9;
          T cm, cx, cy, cz;
          if (p2g_contrib<T, MODE>(sc, p, a, b, c, cm, cx, cy, cz))
            shared_add4<T>(tile + ((p.g[2] + c - L2) * D1 + (p.g[1] + b - L1)) * D0 + (p.g[0] + a - L0), cm, cx, cy, cz);
        }
      }
    } else if (has) {
      // lanes of one cell start at different stencil nodes so their shared atomics do not collide
      const int rot = lane % 27;
#pragma unroll 3
      for (int k = 0; k < 27; ++k) {
        int o = k + rot;
        o = (o >= 27) ? o - 27 : o;
        const int a = o % 3, b = (o / 3) % 3, c = o / 9;
        T cm, cx, cy, cz;
        if (p2g_contrib<T, MODE>(sc, p, a, b, c, cm, cx, cy, cz))
          shared_add4<T>(tile + ((p.g[2] + c - L2) * D1 + (p.g[1] + b - L1)) * D0 + (p.g[0] + a - L0), cm, cx, cy, cz);
      }
    }
    __syncthreads();
    for (int t = tid; t < vol; t += blockDim.x) {
      V4 v = tile[t];
      if (v.x != T(0)) {
        int X = L0 + t % D0, Y = L1 + (t / D0) % D1, Z = L2 + t / (D0 * D1);
        atomic_add4(w.acc + node_index(sc, X, Y, Z), v.x, v.y, v.z, v.w);
      }
    }
    const int B0 = L0 >> 2, B1 = L1 >> 2, B2 = L2 >> 2;
    const int E0 = (L0 + D0 - 1) >> 2, E1 = (L1 + D1 - 1) >> 2, E2 = (L2 + D2 - 1) >> 2;
    const int nbx = E0 - B0 + 1, nby = E1 - B1 + 1, nbz = E2 - B2 + 1;
    for (int t = tid; t < nbx * nby * nbz; t += blockDim.x) {
      int bx = B0 + t % nbx, by = B1 + (t / nbx) % nby, bz = B2 + t / (nbx * nby);
      mark_block(w, sc.blk_off + (uint32_t(bz) * sc.nb[1] + by) * sc.nb[0] + bx);
    }
  } else {
    if (VAR != kVarGlobal && tid == 0) atomicAdd(w.err + 4 * ch.x + 3, 1u);
    if (has) {
#pragma unroll 1
      for (int o = 0; o < 27; ++o) {
        const int a = o % 3, b = (o / 3) % 3, c = o / 9;
        T cm, cx, cy, cz;
        if (p2g_contrib<T, MODE>(sc, p, a, b, c, cm, cx, cy, cz))
          atomic_add4(w.acc + node_index(sc, p.g[0] + a, p.g[1] + b, p.g[2] + c), cm, cx, cy, cz);
      }
      for (int t = 0; t < 8; ++t) {
        int bx = (t & 1) ? (hi[0] >> 2) : (lo[0] >> 2);
        int by = (t & 2) ? (hi[1] >> 2) : (lo[1] >> 2);
        int bz = (t & 4) ? (hi[2] >> 2) : (lo[2] >> 2);
        mark_block(w, sc.blk_off + (uint32_t(bz) * sc.nb[1] + by) * sc.nb[0] + bx);
      }
    }
  }
}

// --------------------------------------------------------------------------------------------
// P2G, physics mode, lanes as stencil columns.  Particles are sorted by cell, so a warp's 32
// particles form a few runs of equal cells (about 30 particles per cell in a dense snow block).
// Lanes 0..26 are 3 particle groups x 9 (y,z) columns of the 3x3x3 stencil: lane (G, b + 3c)
// takes particles s0+G, s0+G+3, ... of a run and keeps the sums of nodes (0..2, b, c) of the
// run's cell in 12 registers.  At the end of the run the three groups are summed with shuffles
// and lanes 0..8 add the run's 27 node sums to the grid with 16-byte vector reductions, one per
// node and run instead of one per node and particle.  Warps never wait for one another: each
// stages its own particles and marks the grid blocks its own stencils touch.
//
// Everything that depends on one particle only is computed by the particle's own thread (in
// parallel over particles) and staged particle-major in shared memory:
//   col[q*9 + b + 3c] = (u, wy[b] wz[c])    u = m v + A d, d = node (0,b,c) - particle
//   wxm[q]            = (wx[0], wx[1], wx[2], m)
//   acol[q]           = (dx A[.][0], 0)      node (a+1,b,c) has u + dx A[.][0]
// so a lane's work per particle is 3 shared loads (the 27 column loads are consecutive vectors,
// conflict-free), 3 weight products, 12 FMAs and 6 adds.
// --------------------------------------------------------------------------------------------
constexpr int kLaneVecs = 11;  // shared vectors per particle: 9 columns, x weights + mass, x column

template <class T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) p2g_lanes_kernel(WorldDev<T> w) {
  using V4 = typename V4T<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  const int nt = blockDim.x;
  V4* col = reinterpret_cast<V4*>(smem);          // col[q * 9 + j]
  V4* wxm = col + 9 * nt;                         // wxm[q]
  V4* acol = wxm + nt;                            // acol[q]
  int4* gk = reinterpret_cast<int4*>(acol + nt);  // gk[q] = (stencil base, cell key)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const int n0 = sc.n[0], n1 = sc.n[1], n2 = sc.n[2];
  const int j = ch.y + tid;
  const bool live = j < ch.z;
  bool has = false;
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
  P2GPart<T> p;
  p.g[0] = p.g[1] = p.g[2] = 0;
  if (live) {
    const uint32_t src = w.perm ? w.perm[j] : uint32_t(j);
    p2g_setup<T, AE_MPM_MODE_PHYSICS>(w, sc, src, p);
    has = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = max(p.g[a], 0);
      hi[a] = min(p.g[a] + 2, sc.n[a] - 1);
      if (lo[a] > hi[a]) has = false;
    }
  }
  // cell key: unique per cell (a stencil with any node in the grid has g in [-2, n-1] per axis)
  const uint32_t key = has ? uint32_t(p.g[0] + 2) + uint32_t(n0 + 2) * (uint32_t(p.g[1] + 2) + uint32_t(n1 + 2) * uint32_t(p.g[2] + 2))
                           : 0xffffffffu;
  // Group equal keys anywhere in the warp (not only adjacent ones: particles that crossed into a
  // neighbouring cell since the last sort rejoin it): groups in order of their first lane, lanes
  // within a group in lane order.  pos is this particle's slot in that grouped order.
  const uint32_t peers = __match_any_sync(0xffffffffu, key);
  const int leader = __ffs(peers) - 1;
  const uint32_t lead_cnt = lane == leader ? uint32_t(__popc(peers)) : 0u;
  uint32_t incl = lead_cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t lead_off = incl - lead_cnt;
  const int pos = int(__shfl_sync(0xffffffffu, lead_off, leader)) + __popc(peers & ((1u << lane) - 1u));
  uint32_t starts = __reduce_or_sync(0xffffffffu, lane == leader ? (1u << lead_off) : 0u);
  const int q = warp * 32 + pos;
  if (live) {
    const T dx = sc.dx;
    T c0[3], c1[3], c2[3], qv[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      c0[r] = dx * p.A[3 * r + 0];
      c1[r] = dx * p.A[3 * r + 1];
      c2[r] = dx * p.A[3 * r + 2];
      qv[r] = p.v[r] - (c0[r] * p.fx[0] + c1[r] * p.fx[1] + c2[r] * p.fx[2]);
    }
    V4* cq = col + q * 9;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const T ux = qv[0] + T(b) * c1[0] + T(c) * c2[0];
        const T uy = qv[1] + T(b) * c1[1] + T(c) * c2[1];
        const T uz = qv[2] + T(b) * c1[2] + T(c) * c2[2];
        cq[b + 3 * c] = mk4(ux, uy, uz, p.w[1][b] * p.w[2][c]);
      }
    }
    wxm[q] = mk4(p.w[0][0], p.w[0][1], p.w[0][2], p.m);
    acol[q] = mk4(c0[0], c0[1], c0[2], T(0));
  }
  gk[q] = make_int4(p.g[0], p.g[1], p.g[2], int(key));
  __syncwarp();
  // lanes 27..31 mirror the columns of lanes 22..26 (in-bounds reads, results never used)
  const int grp = lane < 27 ? lane / 9 : 2;
  const int jc = lane < 27 ? lane - 9 * grp : lane - 23;
  const int nb = jc % 3, nc = jc / 3;
  const uint32_t nb0u = uint32_t(sc.nb[0]), nb1u = uint32_t(sc.nb[1]);
  const V4* colw = col + warp * 32 * 9 + jc;
  const V4* wxw = wxm + warp * 32;
  const V4* acw = acol + warp * 32;
  while (starts) {
    const int s0 = __ffs(starts) - 1;
    starts &= starts - 1u;
    const int e0 = starts ? __ffs(starts) - 1 : 32;
    const int4 run = gk[warp * 32 + s0];
    if (uint32_t(run.w) == 0xffffffffu) continue;
    const int X = run.x, Y = run.y + nb, Z = run.z + nc;
    T m0 = 0, x0 = 0, y0 = 0, z0 = 0, m1 = 0, x1 = 0, y1 = 0, z1 = 0, m2 = 0, x2 = 0, y2 = 0, z2 = 0;
    if constexpr (sizeof(T) == 4) {  // x and y of each node as one packed pair
      float2 q0 = make_float2(0.f, 0.f), q1 = q0, q2 = q0;
#pragma unroll 2
      for (int i = s0 + grp; i < e0; i += 3) {
        const float4 u = colw[i * 9];
        const float4 r = wxw[i];
        const float4 a = acw[i];
        const float W0 = r.x * u.w, W1 = r.y * u.w, W2 = r.z * u.w;
        const float2 axy = make_float2(a.x, a.y), u0 = make_float2(u.x, u.y);
        const float2 u1 = __fadd2_rn(u0, axy), u2 = __fadd2_rn(u1, axy);
        m0 += W0 * r.w;
        m1 += W1 * r.w;
        m2 += W2 * r.w;
        q0 = __ffma2_rn(make_float2(W0, W0), u0, q0);
        q1 = __ffma2_rn(make_float2(W1, W1), u1, q1);
        q2 = __ffma2_rn(make_float2(W2, W2), u2, q2);
        const float uz1 = u.z + a.z;
        z0 += W0 * u.z;
        z1 += W1 * uz1;
        z2 += W2 * (uz1 + a.z);
      }
      x0 = q0.x, y0 = q0.y, x1 = q1.x, y1 = q1.y, x2 = q2.x, y2 = q2.y;
    } else
#pragma unroll 2
    for (int i = s0 + grp; i < e0; i += 3) {
      const V4 u = colw[i * 9];
      const V4 r = wxw[i];
      const V4 a = acw[i];
      const T W0 = r.x * u.w, W1 = r.y * u.w, W2 = r.z * u.w;
      m0 += W0 * r.w;
      x0 += W0 * u.x;
      y0 += W0 * u.y;
      z0 += W0 * u.z;
      const T ux = u.x + a.x, uy = u.y + a.y, uz = u.z + a.z;
      m1 += W1 * r.w;
      x1 += W1 * ux;
      y1 += W1 * uy;
      z1 += W1 * uz;
      m2 += W2 * r.w;
      x2 += W2 * (ux + a.x);
      y2 += W2 * (uy + a.y);
      z2 += W2 * (uz + a.z);
    }
    if (e0 - s0 > 1) {
      auto groups = [](T v) { return v + __shfl_down_sync(0xffffffffu, v, 9) + __shfl_down_sync(0xffffffffu, v, 18); };
      m0 = groups(m0), x0 = groups(x0), y0 = groups(y0), z0 = groups(z0);
      m1 = groups(m1), x1 = groups(x1), y1 = groups(y1), z1 = groups(z1);
      m2 = groups(m2), x2 = groups(x2), y2 = groups(y2), z2 = groups(z2);
    }
    if (lane < 9 && Y >= 0 && Z >= 0 && Y < n1 && Z < n2) {
      // block-major node index, the (y,z) part once: ((blk_off + (bz nb1 + by) nb0 + bx) << 6) | local
      const uint32_t row = ((sc.blk_off + (uint32_t(Z >> 2) * nb1u + uint32_t(Y >> 2)) * nb0u) << 6) |
                           (uint32_t(Z & 3) << 4) | (uint32_t(Y & 3) << 2);
      auto node = [row](int xa) { return row + ((uint32_t(xa >> 2) << 6) | uint32_t(xa & 3)); };
      if (m0 != T(0) && X >= 0 && X < n0) atomic_add4(w.acc + node(X), m0, x0, y0, z0);
      if (m1 != T(0) && X + 1 >= 0 && X + 1 < n0) atomic_add4(w.acc + node(X + 1), m1, x1, y1, z1);
      if (m2 != T(0) && X + 2 >= 0 && X + 2 < n0) atomic_add4(w.acc + node(X + 2), m2, x2, y2, z2);
    }
  }
  // grid blocks of this warp's stencil bounding box
  int B[3], NB[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int l = __reduce_min_sync(0xffffffffu, has ? lo[a] : INT_MAX);
    const int h = __reduce_max_sync(0xffffffffu, has ? hi[a] : INT_MIN);
    B[a] = l >> 2;
    NB[a] = l == INT_MAX ? 0 : (h >> 2) - (l >> 2) + 1;
  }
  const int nblk = NB[0] * NB[1] * NB[2];
  if (NB[0] <= 4 && NB[1] <= 4 && NB[2] <= 2) {
    const int bx = lane & 3, by = (lane >> 2) & 3, bz = lane >> 4;
    if (bx < NB[0] && by < NB[1] && bz < NB[2])
      mark_block(w, sc.blk_off + (uint32_t(B[2] + bz) * sc.nb[1] + (B[1] + by)) * sc.nb[0] + (B[0] + bx));
  } else {
    for (int t = lane; t < nblk; t += 32) {
      const int bx = B[0] + t % NB[0], by = B[1] + (t / NB[0]) % NB[1], bz = B[2] + t / (NB[0] * NB[1]);
      mark_block(w, sc.blk_off + (uint32_t(bz) * sc.nb[1] + by) * sc.nb[0] + bx);
    }
  }
}

// Column-lane P2G of the velocity-only mode (mpm_substep_velocity_only, mpm_solver.rs:1377-1449):
// per node w m and w m v, w = wx (wy wz), skipping a (y,z) column whose wy or wz is below 1e-10
// and a node whose w is, and nodes past the grid's upper faces.  The structure is
// p2g_lanes_kernel's: the warp groups its particles by cell, stages per particle the nine
// w_y w_z column products, the x weights with the mass and the velocity, and lanes 0..26
// (3 particle groups x 9 columns) sum the three x nodes of their column over each cell's run,
// one vector reduction per node and run.
template <class T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) p2g_lanes_velonly_kernel(WorldDev<T> w) {
  using V4 = typename V4T<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  const int nt = blockDim.x;
  V4* wxm = reinterpret_cast<V4*>(smem);          // wxm[q] = (wx0, wx1, wx2, m)
  V4* vel = wxm + nt;                             // vel[q] = (vx, vy, vz, -)
  int4* gk = reinterpret_cast<int4*>(vel + nt);   // gk[q] = (stencil base, cell key)
  T* cw = reinterpret_cast<T*>(gk + nt);          // cw[q * 9 + column] = w_y w_z, 0 when skipped
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const int n0 = sc.n[0], n1 = sc.n[1], n2 = sc.n[2];
  const int j = ch.y + tid;
  const bool live = j < ch.z;
  bool has = false;
  P2GPart<T> p;
  p.g[0] = p.g[1] = p.g[2] = 0;
  if (live) {
    const uint32_t src = w.perm ? w.perm[j] : uint32_t(j);
    p2g_setup<T, AE_MPM_MODE_VELOCITY_ONLY>(w, sc, src, p);
    has = p.g[0] < n0 && p.g[1] < n1 && p.g[2] < n2;  // some stencil node inside the grid (g >= 0)
  }
  const uint32_t key = has ? uint32_t(p.g[0]) + uint32_t(n0) * (uint32_t(p.g[1]) + uint32_t(n1) * uint32_t(p.g[2]))
                           : 0xffffffffu;
  const uint32_t peers = __match_any_sync(0xffffffffu, key);
  const int leader = __ffs(peers) - 1;
  const uint32_t lead_cnt = lane == leader ? uint32_t(__popc(peers)) : 0u;
  uint32_t incl = lead_cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t lead_off = incl - lead_cnt;
  const int pos = int(__shfl_sync(0xffffffffu, lead_off, leader)) + __popc(peers & ((1u << lane) - 1u));
  uint32_t starts = __reduce_or_sync(0xffffffffu, lane == leader ? (1u << lead_off) : 0u);
  const int q = warp * 32 + pos;
  if (has) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int b = 0; b < 3; ++b)
        cw[q * 9 + b + 3 * c] = (p.w[2][c] < T(1e-10) || p.w[1][b] < T(1e-10)) ? T(0) : p.w[1][b] * p.w[2][c];
    wxm[q] = mk4(p.w[0][0], p.w[0][1], p.w[0][2], p.m);
    vel[q] = mk4(p.v[0], p.v[1], p.v[2], T(0));
  }
  gk[q] = make_int4(p.g[0], p.g[1], p.g[2], int(key));
  __syncwarp();
  const int grp = lane < 27 ? lane / 9 : 2;
  const int jc = lane < 27 ? lane - 9 * grp : lane - 23;
  const int nb = jc % 3, nc = jc / 3;
  const T* cww = cw + warp * 32 * 9 + jc;
  const V4* wxw = wxm + warp * 32;
  const V4* vw = vel + warp * 32;
  while (starts) {
    const int s0 = __ffs(starts) - 1;
    starts &= starts - 1u;
    const int e0 = starts ? __ffs(starts) - 1 : 32;
    const int4 run = gk[warp * 32 + s0];
    if (uint32_t(run.w) == 0xffffffffu) continue;
    const int X = run.x, Y = run.y + nb, Z = run.z + nc;
    T m0 = 0, x0 = 0, y0 = 0, z0 = 0, m1 = 0, x1 = 0, y1 = 0, z1 = 0, m2 = 0, x2 = 0, y2 = 0, z2 = 0;
    for (int i = s0 + grp; i < e0; i += 3) {
      const T wyz = cww[i * 9];
      const V4 r = wxw[i];
      const V4 v = vw[i];
      T W0 = r.x * wyz, W1 = r.y * wyz, W2 = r.z * wyz;
      W0 = W0 < T(1e-10) ? T(0) : W0;
      W1 = W1 < T(1e-10) ? T(0) : W1;
      W2 = W2 < T(1e-10) ? T(0) : W2;
      const T a0 = W0 * r.w, a1 = W1 * r.w, a2 = W2 * r.w;  // w m, as the reference forms it
      m0 += a0;
      x0 += a0 * v.x;
      y0 += a0 * v.y;
      z0 += a0 * v.z;
      m1 += a1;
      x1 += a1 * v.x;
      y1 += a1 * v.y;
      z1 += a1 * v.z;
      m2 += a2;
      x2 += a2 * v.x;
      y2 += a2 * v.y;
      z2 += a2 * v.z;
    }
    if (e0 - s0 > 1) {
      auto groups = [](T v) { return v + __shfl_down_sync(0xffffffffu, v, 9) + __shfl_down_sync(0xffffffffu, v, 18); };
      m0 = groups(m0), x0 = groups(x0), y0 = groups(y0), z0 = groups(z0);
      m1 = groups(m1), x1 = groups(x1), y1 = groups(y1), z1 = groups(z1);
      m2 = groups(m2), x2 = groups(x2), y2 = groups(y2), z2 = groups(z2);
    }
    if (lane < 9 && Y < n1 && Z < n2) {
      const uint32_t row = ((sc.blk_off + (uint32_t(Z >> 2) * uint32_t(sc.nb[1]) + uint32_t(Y >> 2)) * uint32_t(sc.nb[0])) << 6) |
                           (uint32_t(Z & 3) << 4) | (uint32_t(Y & 3) << 2);
      auto node = [row](int xa) { return row + ((uint32_t(xa >> 2) << 6) | uint32_t(xa & 3)); };
      if (m0 != T(0) && X < n0) atomic_add4(w.acc + node(X), m0, x0, y0, z0);
      if (m1 != T(0) && X + 1 < n0) atomic_add4(w.acc + node(X + 1), m1, x1, y1, z1);
      if (m2 != T(0) && X + 2 < n0) atomic_add4(w.acc + node(X + 2), m2, x2, y2, z2);
    }
  }
  // grid blocks of this warp's stencil bounding box (inside the grid)
  int B[3], NB[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int l = __reduce_min_sync(0xffffffffu, has ? p.g[a] : INT_MAX);
    const int h = __reduce_max_sync(0xffffffffu, has ? min(p.g[a] + 2, sc.n[a] - 1) : INT_MIN);
    B[a] = l >> 2;
    NB[a] = l == INT_MAX ? 0 : (h >> 2) - (l >> 2) + 1;
  }
  const int nblk = NB[0] * NB[1] * NB[2];
  for (int t = lane; t < nblk; t += 32) {
    const int bx = B[0] + t % NB[0], by = B[1] + (t / NB[0]) % NB[1], bz = B[2] + t / (NB[0] * NB[1]);
    mark_block(w, sc.blk_off + (uint32_t(bz) * uint32_t(sc.nb[1]) + uint32_t(by)) * uint32_t(sc.nb[0]) + uint32_t(bx));
  }
}
// Column-lane P2G of the reference mode (mpm_substep_serial_active / parallel_with_indices P2G,
// mpm_solver.rs:831-903, 1108-1193).  Per node (a,b,c) of a particle: w = (wx wy) wz, skipped below
// 1e-10 (mass, momentum and force alike); momentum w m (v + C d) with d the node minus the particle;
// the force sv . (N'(a), N'(b), N'(c)) / dx, not weighted by w, folded into momentum as dt sv (the
// grid update's v = p/m + g dt then equals the reference's p/m + (g + f/m) dt up to rounding).
// The particle's owner thread stages per (y,z) column u = v + C[.][1] d_y + C[.][2] d_z with wy,
// and f = sv[.][1] N'_y + sv[.][2] N'_z with wz; lanes 0..26 (3 particle groups x 9 columns) add
// the x part of each of their column's three nodes and sum over each cell's run, one vector
// reduction per node and run.
constexpr int kRefLaneVecs = 2 * 9 + 5;  // shared vectors per particle
// kPer particles per warp, 32 / kPer CTAs per chunk: the engine's near set is sparse (about one
// particle in twelve cells), so every particle is a run of its own and a warp sums its runs one
// after another; 10 000 particles with 32 per warp took 30 us on 40 of the SMs.
template <class T, int kPer>
__global__ void __launch_bounds__(256, 1) p2g_lanes_ref_kernel(WorldDev<T> w) {
  using V4 = typename V4T<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kSplit = 32 / kPer;
  const int nt = blockDim.x;
  V4* cu = reinterpret_cast<V4*>(smem);  // cu[q * 9 + j] = (u, wy)
  V4* cf = cu + 9 * nt;                  // cf[q * 9 + j] = (f, wz)
  V4* pw = cf + 9 * nt;                  // pw[q] = (wx0, wx1, wx2, m)
  V4* pc = pw + nt;                      // pc[q] = C[.][0]
  V4* po = pc + nt;                      // po[q] = (d_x of the three x nodes)
  V4* ps = po + nt;                      // ps[q] = dt sv[.][0]
  V4* pe = ps + nt;                      // pe[q] = (N'_x of the three x nodes) / dx
  int4* gk = reinterpret_cast<int4*>(pe + nt);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int4 ch = chunk_at(w, blockIdx.x / kSplit, blockDim.x);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const int n0 = sc.n[0], n1 = sc.n[1], n2 = sc.n[2];
  const int j = ch.y + int(blockIdx.x % kSplit) * int(blockDim.x / kSplit) + warp * kPer + lane;
  const bool live = (kPer == 32 || lane < kPer) && j < ch.z;
  bool has = false;
  P2GPart<T> p;
  p.g[0] = p.g[1] = p.g[2] = 0;
  if (live) {
    const uint32_t src = w.perm ? w.perm[j] : uint32_t(j);
    p2g_setup<T, AE_MPM_MODE_REFERENCE>(w, sc, src, p);
    has = p.g[0] < n0 && p.g[1] < n1 && p.g[2] < n2;  // some stencil node inside the grid (g >= 0)
  }
  const uint32_t key = has ? uint32_t(p.g[0]) + uint32_t(n0) * (uint32_t(p.g[1]) + uint32_t(n1) * uint32_t(p.g[2]))
                           : 0xffffffffu;
  const uint32_t peers = __match_any_sync(0xffffffffu, key);
  const int leader = __ffs(peers) - 1;
  const uint32_t lead_cnt = lane == leader ? uint32_t(__popc(peers)) : 0u;
  uint32_t incl = lead_cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t lead_off = incl - lead_cnt;
  const int pos = int(__shfl_sync(0xffffffffu, lead_off, leader)) + __popc(peers & ((1u << lane) - 1u));
  uint32_t starts = __reduce_or_sync(0xffffffffu, lane == leader ? (1u << lead_off) : 0u);
  const int q = warp * 32 + pos;
  if (has) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const T dy = p.o[1][b], dz = p.o[2][c], ey = p.dw[1][b], ez = p.dw[2][c];
        const T ux = p.v[0] + p.A[1] * dy + p.A[2] * dz;
        const T uy = p.v[1] + p.A[4] * dy + p.A[5] * dz;
        const T uz = p.v[2] + p.A[7] * dy + p.A[8] * dz;
        cu[q * 9 + b + 3 * c] = mk4(ux, uy, uz, p.w[1][b]);
        cf[q * 9 + b + 3 * c] =
            mk4(p.sv[1] * ey + p.sv[2] * ez, p.sv[4] * ey + p.sv[5] * ez, p.sv[7] * ey + p.sv[8] * ez, p.w[2][c]);
      }
    pw[q] = mk4(p.w[0][0], p.w[0][1], p.w[0][2], p.m);
    pc[q] = mk4(p.A[0], p.A[3], p.A[6], T(0));
    po[q] = mk4(p.o[0][0], p.o[0][1], p.o[0][2], T(0));
    ps[q] = mk4(p.sv[0], p.sv[3], p.sv[6], T(0));
    pe[q] = mk4(p.dw[0][0], p.dw[0][1], p.dw[0][2], T(0));
  }
  gk[q] = make_int4(p.g[0], p.g[1], p.g[2], int(key));
  __syncwarp();
  const int grp = lane < 27 ? lane / 9 : 2;
  const int jc = lane < 27 ? lane - 9 * grp : lane - 23;
  const int nb = jc % 3, nc = jc / 3;
  const int wb = warp * 32;
  while (starts) {
    const int s0 = __ffs(starts) - 1;
    starts &= starts - 1u;
    const int e0 = starts ? __ffs(starts) - 1 : 32;
    const int4 run = gk[wb + s0];
    if (uint32_t(run.w) == 0xffffffffu) continue;
    const int X = run.x, Y = run.y + nb, Z = run.z + nc;
    T acc[3][4];
#pragma unroll
    for (int a = 0; a < 3; ++a) acc[a][0] = acc[a][1] = acc[a][2] = acc[a][3] = T(0);
    for (int i = s0 + grp; i < e0; i += 3) {
      const V4 u = cu[(wb + i) * 9 + jc], f = cf[(wb + i) * 9 + jc];
      const V4 r = pw[wb + i], cx = pc[wb + i], dx = po[wb + i], sx = ps[wb + i], ex = pe[wb + i];
      const T wxs[3] = {r.x, r.y, r.z}, dxs[3] = {dx.x, dx.y, dx.z}, exs[3] = {ex.x, ex.y, ex.z};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const T wn = (wxs[a] * u.w) * f.w;  // (wx wy) wz, as the reference multiplies
        if (wn < T(1e-10)) continue;
        const T wm = wn * r.w;
        acc[a][0] += wm;
        acc[a][1] += wm * (u.x + cx.x * dxs[a]) + (f.x + sx.x * exs[a]);
        acc[a][2] += wm * (u.y + cx.y * dxs[a]) + (f.y + sx.y * exs[a]);
        acc[a][3] += wm * (u.z + cx.z * dxs[a]) + (f.z + sx.z * exs[a]);
      }
    }
    if (e0 - s0 > 1) {
      auto groups = [](T v) { return v + __shfl_down_sync(0xffffffffu, v, 9) + __shfl_down_sync(0xffffffffu, v, 18); };
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[a][k] = groups(acc[a][k]);
    }
    if (lane < 9 && Y < n1 && Z < n2) {
      const uint32_t row = ((sc.blk_off + (uint32_t(Z >> 2) * uint32_t(sc.nb[1]) + uint32_t(Y >> 2)) * uint32_t(sc.nb[0])) << 6) |
                           (uint32_t(Z & 3) << 4) | (uint32_t(Y & 3) << 2);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int xa = X + a;
        // a node every particle skipped has mass 0; one with a (skipped-weight) force only does not
        // exist: the force is added exactly where the mass is
        if (acc[a][0] != T(0) && xa < n0)
          atomic_add4(w.acc + (row + ((uint32_t(xa >> 2) << 6) | uint32_t(xa & 3))), acc[a][0], acc[a][1], acc[a][2],
                      acc[a][3]);
      }
    }
  }
  int B[3], NB[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int l = __reduce_min_sync(0xffffffffu, has ? p.g[a] : INT_MAX);
    const int h = __reduce_max_sync(0xffffffffu, has ? min(p.g[a] + 2, sc.n[a] - 1) : INT_MIN);
    B[a] = l >> 2;
    NB[a] = l == INT_MAX ? 0 : (h >> 2) - (l >> 2) + 1;
  }
  const int nblk = NB[0] * NB[1] * NB[2];
  for (int t = lane; t < nblk; t += 32) {
    const int bx = B[0] + t % NB[0], by = B[1] + (t / NB[0]) % NB[1], bz = B[2] + t / (NB[0] * NB[1]);
    mark_block(w, sc.blk_off + (uint32_t(bz) * uint32_t(sc.nb[1]) + uint32_t(by)) * uint32_t(sc.nb[0]) + uint32_t(bx));
  }
}

// shared bytes per particle of p2g_lanes_velonly_kernel
template <class T>
constexpr size_t velonly_lane_bytes() {
  return 2 * sizeof(typename V4T<T>::type) + sizeof(int4) + 9 * sizeof(T);
}

// ============================================================================================
// grid update (momentum -> velocity, gravity, walls); clears accumulator and touched flags
// ============================================================================================
template <class T, int MODE>
__device__ __forceinline__ void grid_velocity(const SceneDev<T>& sc, int i, int j, int k, T m, T px, T py, T pz,
                                              T& vx, T& vy, T& vz) {
  vx = vy = vz = T(0);
  if (MODE == AE_MPM_MODE_PHYSICS) {
    if (!(m > T(0))) return;
    vx = px / m + sc.dt * sc.grav[0];
    vy = py / m + sc.dt * sc.grav[1];
    vz = pz / m + sc.dt * sc.grav[2];
    const int mg = sc.wall_margin;
    const int id[3] = {i, j, k};
    if (sc.wall_mode == AE_MPM_WALL_STICKY) {
      bool wall = false;
#pragma unroll
      for (int a = 0; a < 3; ++a) wall = wall || id[a] < mg || id[a] >= sc.n[a] - mg;
      if (wall) vx = vy = vz = T(0);
    } else {
      T v[3] = {vx, vy, vz};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (id[a] < mg && v[a] < T(0)) v[a] = -v[a] * sc.restitution;
        if (id[a] >= sc.n[a] - mg && v[a] > T(0)) v[a] = -v[a] * sc.restitution;
      }
      vx = v[0];
      vy = v[1];
      vz = v[2];
    }
  } else {  // Grid::update_parallel (mpm_solver.rs:112-139), force folded into momentum
    if (!(m > T(1e-12))) return;
    vx = px / m + sc.grav[0] * sc.dt;
    vy = py / m + sc.grav[1] * sc.dt;
    vz = pz / m + sc.grav[2] * sc.dt;
    if (j == 0) {
      vy = t_max(vy, T(0));
      vx *= T(0.9);
      vz *= T(0.9);
    }
  }
}

template <class T>
__device__ __forceinline__ void block_coords(const SceneDev<T>& sc, uint32_t gb, int l, int& i, int& j, int& k) {
  uint32_t lb = gb - sc.blk_off;
  int bx = int(lb % uint32_t(sc.nb[0]));
  int by = int((lb / uint32_t(sc.nb[0])) % uint32_t(sc.nb[1]));
  int bz = int(lb / (uint32_t(sc.nb[0]) * uint32_t(sc.nb[1])));
  i = bx * 4 + (l & 3);
  j = by * 4 + ((l >> 2) & 3);
  k = bz * 4 + (l >> 4);
}

// by CTA `cta` of `ctas`
template <class T, int MODE>
__device__ __forceinline__ void grid_update(const WorldDev<T>& w, uint32_t* blk_epoch, const uint32_t* epoch,
                                            uint32_t* zero_count, uint32_t cta, uint32_t ctas) {
  using V4 = typename V4T<T>::type;
  const uint32_t count = launch_count(w.touched_count);
  const uint32_t ep = *epoch;
  if (cta == 0 && threadIdx.x == 0) {
    *w.clamp_count = 0u;  // G2P of this substep refills it
    // the fused G2P + P2G appends the next substep's blocks to the other list, whose previous
    // contents the grid update of the substep before consumed
    if (zero_count) *zero_count = 0u;
  }
  // each 64-thread group takes 4 touched blocks per iteration and issues their 4 accumulator loads
  // before using any, so a long touched list is not one latency-bound load after another
  constexpr int kU = 4;
  const int sub = threadIdx.x >> 6, l = threadIdx.x & 63;
  for (uint32_t t0 = (cta * 4 + sub) * kU; t0 < count; t0 += ctas * 4 * kU) {
    uint32_t gb[kU];
    V4 a[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) gb[u] = (t0 + u < count) ? w.touched[t0 + u] : 0xffffffffu;
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (gb[u] != 0xffffffffu) a[u] = w.acc[uint64_t(gb[u]) * 64u + l];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (gb[u] == 0xffffffffu) continue;
      const SceneDev<T>& sc = w.scenes[w.one_scene ? 0u : w.blk_scene[gb[u]]];  // one scene: no lookup
      int i, j, k;
      block_coords(sc, gb[u], l, i, j, k);
      const uint64_t gi = uint64_t(gb[u]) * 64u + l;
      w.acc[gi] = mk4(T(0), T(0), T(0), T(0));
      T vx, vy, vz;
      grid_velocity<T, MODE>(sc, i, j, k, a[u].x, a[u].y, a[u].z, a[u].w, vx, vy, vz);
      w.vel[gi] = mk4(vx, vy, vz, a[u].x);
      if (l == 0) {
        w.blk_flag[gb[u]] = 0u;
        blk_epoch[gb[u]] = ep;
      }
    }
  }
}

template <class T, int MODE>
__global__ void __launch_bounds__(256) grid_update_kernel(WorldDev<T> w, uint32_t* blk_epoch, const uint32_t* epoch,
                                                          uint32_t* zero_count) {
  let_next_start();
  dependency_wait();
  grid_update<T, MODE>(w, blk_epoch, epoch, zero_count, blockIdx.x, gridDim.x);
}

// ============================================================================================
// G2P
// ============================================================================================
template <class T>
struct G2POut {
  T x[3], v[3], C[9], F[9], J;
  uint32_t err;       // kErr* bits
  bool needs_clamp;   // snow: F left the elastic region; the clamp kernel finishes the update
  bool clamped;
};

// Node velocities for one block of particles: the block's bounding-box tile in shared memory
// (filled with coalesced loads before the gather), or the global array when the box is too big.
// The tile's x and y pitches are powers of two (2^p0 >= D0, 2^(sp-p0) >= D1), so slot indexes
// split into coordinates with shifts and masks.
template <class T>
struct VelTile {
  using V4 = typename V4T<T>::type;
  const V4* tile;
  const V4* vel;
  int L0, L1, L2, p0, sp;
  __device__ __forceinline__ V4 operator()(const SceneDev<T>& sc, int X, int Y, int Z) const {
    if (tile) return tile[((Z - L2) << sp) + ((Y - L1) << p0) + (X - L0)];
    return ld4(vel + node_index(sc, X, Y, Z));
  }
};

// Node velocities of the block-major grid by (y,z) row, through the read-only cache: row(Y, Z)
// once per stencil column, then at(row, X) for its three x nodes.  The block needs no bounding
// box, tile or barrier, so its warps never wait for one another.
template <class T>
struct GridRows {
  using V4 = typename V4T<T>::type;
  const V4* __restrict__ vel;
  uint32_t blk_off, nb0, nb1;
  __device__ __forceinline__ uint32_t row(int Y, int Z) const {
    return ((blk_off + (uint32_t(Z >> 2) * nb1 + uint32_t(Y >> 2)) * nb0) << 6) | (uint32_t(Z & 3) << 4) |
           (uint32_t(Y & 3) << 2);
  }
  __device__ __forceinline__ V4 at(uint32_t r, int X) const {
    return ld4(vel + (r + ((uint32_t(X >> 2) << 6) | uint32_t(X & 3))));
  }
  // row(Y, Z) == zpart(Z) + ypart(Y), and the node index of (X, Y, Z) == row + xpart(X)
  __device__ __forceinline__ uint32_t xpart(int X) const { return (uint32_t(X >> 2) << 6) | uint32_t(X & 3); }
  __device__ __forceinline__ uint32_t ypart(int Y) const {
    return ((uint32_t(Y >> 2) * nb0) << 6) | (uint32_t(Y & 3) << 2);
  }
  __device__ __forceinline__ uint32_t zpart(int Z) const {
    return ((blk_off + uint32_t(Z >> 2) * nb1 * nb0) << 6) | (uint32_t(Z & 3) << 4);
  }
  __device__ __forceinline__ V4 at_part(uint32_t r, uint32_t xp) const { return ld4(vel + (r + xp)); }
};
// Physics gather for a particle whose 27 stencil nodes are all inside the grid (every particle
// after its first substep: positions are clamped to [1, n-2] dx).  Separable: each (y,z) column
// is summed over x first,
//   S0 = sum_a wx[a] g(a,b,c),   S1 = sum_a wx[a] (a - fx) dx g(a,b,c),
// then v += wy wz S0, B[.][0] += wy wz S1, B[.][1] += wy (b - fy) dx wz S0,
// B[.][2] += wy wz (c - fz) dx S0: 36 instructions per column instead of 42 per node.
// Returns false (nothing written) when the particle does not qualify.
template <class T, class Rows>
__device__ __forceinline__ bool g2p_physics_gather_sep(const Rows& rows, const SceneDev<T>& sc, const T* x0, T* v,
                                                       T* C) {
  using V4 = typename V4T<T>::type;
  int b[3];
  T w[3][3], e[3][3];
  bool inside = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const T X = (x0[a] - sc.origin[a]) * sc.inv_dx;
    const int bb = floor_to_int(X - T(0.5));
    const T fx = X - T(bb);
    b[a] = bb;
    inside = inside && bb >= 0 && bb + 2 < sc.n[a];
    const T t0 = T(1.5) - fx, t1 = fx - T(1), t2 = fx - T(0.5);
    w[a][0] = T(0.5) * t0 * t0;
    w[a][1] = T(0.75) - t1 * t1;
    w[a][2] = T(0.5) * t2 * t2;
#pragma unroll
    for (int k = 0; k < 3; ++k) e[a][k] = w[a][k] * ((T(k) - fx) * sc.dx);
  }
  if (!inside) return false;
  T vv[3] = {0, 0, 0}, B[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int bb = 0; bb < 3; ++bb) {
      const uint32_t r = rows.row(b[1] + bb, b[2] + c);
      const V4 g0 = rows.at(r, b[0]), g1 = rows.at(r, b[0] + 1), g2 = rows.at(r, b[0] + 2);
      const T s0[3] = {w[0][0] * g0.x + w[0][1] * g1.x + w[0][2] * g2.x, w[0][0] * g0.y + w[0][1] * g1.y + w[0][2] * g2.y,
                       w[0][0] * g0.z + w[0][1] * g1.z + w[0][2] * g2.z};
      const T s1[3] = {e[0][0] * g0.x + e[0][1] * g1.x + e[0][2] * g2.x, e[0][0] * g0.y + e[0][1] * g1.y + e[0][2] * g2.y,
                       e[0][0] * g0.z + e[0][1] * g1.z + e[0][2] * g2.z};
      const T wbc = w[1][bb] * w[2][c], ebc = e[1][bb] * w[2][c], fbc = w[1][bb] * e[2][c];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        vv[k] += wbc * s0[k];
        B[k * 3 + 0] += wbc * s1[k];
        B[k * 3 + 1] += ebc * s0[k];
        B[k * 3 + 2] += fbc * s0[k];
      }
    }
  }
  const T cs = T(4) * sc.inv_dx * sc.inv_dx;
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = vv[k];
#pragma unroll
  for (int k = 0; k < 9; ++k) C[k] = cs * B[k];
  return true;
}

// The same separable gather in f32 with Blackwell's packed FMA (two lanes of a float2 per
// instruction): the x and y components of each column sum and accumulator travel as one pair, z
// alone.  Every pair op rounds like the scalar fused multiply-adds it replaces.
template <class Rows>
__device__ __forceinline__ bool g2p_physics_gather_sep_f2(const Rows& rows, const SceneDev<float>& sc, const float* x0,
                                                          float* v, float* C) {
  int b[3];
  float w[3][3], e[3][3];
  bool inside = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float X = (x0[a] - sc.origin[a]) * sc.inv_dx;
    const int bb = floor_to_int(X - 0.5f);
    const float fx = X - float(bb);
    b[a] = bb;
    inside = inside && bb >= 0 && bb + 2 < sc.n[a];
    const float t0 = 1.5f - fx, t1 = fx - 1.0f, t2 = fx - 0.5f;
    w[a][0] = 0.5f * t0 * t0;
    w[a][1] = 0.75f - t1 * t1;
    w[a][2] = 0.5f * t2 * t2;
#pragma unroll
    for (int k = 0; k < 3; ++k) e[a][k] = w[a][k] * ((float(k) - fx) * sc.dx);
  }
  if (!inside) return false;
  // only the x weights are kept as broadcast pairs; the y/z weight products are formed per
  // column and paired there (pairs of all six weight sets took 36 registers and spilled)
  float2 wx[3], ex[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    wx[k] = make_float2(w[0][k], w[0][k]);
    ex[k] = make_float2(e[0][k], e[0][k]);
  }
  float2 vxy = make_float2(0.f, 0.f), b0xy = vxy, b1xy = vxy, b2xy = vxy;
  float vz = 0.f, b0z = 0.f, b1z = 0.f, b2z = 0.f;
  // node index = z part + y part + x part: the three bit fields of the block-major index are
  // disjoint, so the 27 indexes come from 3 + 3 + 3 parts with one add each
  uint32_t xp[3], yp[3], zp[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    xp[k] = rows.xpart(b[0] + k);
    yp[k] = rows.ypart(b[1] + k);
    zp[k] = rows.zpart(b[2] + k);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int bb = 0; bb < 3; ++bb) {
      const uint32_t r = zp[c] + yp[bb];
      const float4 g0 = rows.at_part(r, xp[0]), g1 = rows.at_part(r, xp[1]), g2 = rows.at_part(r, xp[2]);
      const float2 g0xy = make_float2(g0.x, g0.y), g1xy = make_float2(g1.x, g1.y), g2xy = make_float2(g2.x, g2.y);
      const float2 s0xy = __ffma2_rn(wx[2], g2xy, __ffma2_rn(wx[1], g1xy, __fmul2_rn(wx[0], g0xy)));
      const float2 s1xy = __ffma2_rn(ex[2], g2xy, __ffma2_rn(ex[1], g1xy, __fmul2_rn(ex[0], g0xy)));
      const float s0z = w[0][0] * g0.z + w[0][1] * g1.z + w[0][2] * g2.z;
      const float s1z = e[0][0] * g0.z + e[0][1] * g1.z + e[0][2] * g2.z;
      const float wbs = w[1][bb] * w[2][c], ebs = e[1][bb] * w[2][c], fbs = w[1][bb] * e[2][c];
      const float2 wbc = make_float2(wbs, wbs), ebc = make_float2(ebs, ebs), fbc = make_float2(fbs, fbs);
      vxy = __ffma2_rn(wbc, s0xy, vxy);
      b0xy = __ffma2_rn(wbc, s1xy, b0xy);
      b1xy = __ffma2_rn(ebc, s0xy, b1xy);
      b2xy = __ffma2_rn(fbc, s0xy, b2xy);
      vz += wbc.x * s0z;
      b0z += wbc.x * s1z;
      b1z += ebc.x * s0z;
      b2z += fbc.x * s0z;
    }
  }
  const float cs = 4.0f * sc.inv_dx * sc.inv_dx;
  v[0] = vxy.x;
  v[1] = vxy.y;
  v[2] = vz;
  // B[k][col]: column col of the affine sum for velocity component k
  C[0] = cs * b0xy.x;
  C[1] = cs * b1xy.x;
  C[2] = cs * b2xy.x;
  C[3] = cs * b0xy.y;
  C[4] = cs * b1xy.y;
  C[5] = cs * b2xy.y;
  C[6] = cs * b0z;
  C[7] = cs * b1z;
  C[8] = cs * b2z;
  return true;
}

// gather half of the physics G2P: grid velocity and APIC C at the particle
template <class T>
__device__ __forceinline__ void g2p_physics_gather(const VelTile<T>& vt, const SceneDev<T>& sc, const T* x0, T* v,
                                                   T* C) {
  using V4 = typename V4T<T>::type;
  int b[3];
  T wt[3][3], dp[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T X = (x0[a] - sc.origin[a]) * sc.inv_dx;
    int bb = floor_to_int(X - T(0.5));
    T fx = X - T(bb);
    b[a] = bb;
    T t0 = T(1.5) - fx, t1 = fx - T(1), t2 = fx - T(0.5);
    wt[a][0] = T(0.5) * t0 * t0;
    wt[a][1] = T(0.75) - t1 * t1;
    wt[a][2] = T(0.5) * t2 * t2;
#pragma unroll
    for (int k = 0; k < 3; ++k) dp[a][k] = (T(k) - fx) * sc.dx;
  }
  T B[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  v[0] = v[1] = v[2] = T(0);
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int bb = 0; bb < 3; ++bb)
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        int X = b[0] + a, Y = b[1] + bb, Z = b[2] + c;
        if (X < 0 || Y < 0 || Z < 0 || X >= sc.n[0] || Y >= sc.n[1] || Z >= sc.n[2]) continue;
        T ww = wt[0][a] * wt[1][bb] * wt[2][c];
        V4 gv = vt(sc, X, Y, Z);
        T g3[3] = {gv.x, gv.y, gv.z};
        T d[3] = {dp[0][a], dp[1][bb], dp[2][c]};
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          v[r] += ww * g3[r];
#pragma unroll
          for (int k = 0; k < 3; ++k) B[r * 3 + k] += ww * g3[r] * d[k];
        }
      }
  const T cs = T(4) * sc.inv_dx * sc.inv_dx;
#pragma unroll
  for (int k = 0; k < 9; ++k) C[k] = cs * B[k];
}

// update half of the physics G2P: advection and the F or J update.  Snow whose F left the elastic
// region (needs_clamp) has its trial F and old J_p here; everything else is final.  o.C keeps C.
template <class T>
__device__ __forceinline__ void g2p_physics_move(const SceneDev<T>& sc, const MatDev& md, const T* x0, const T* v,
                                                 const T* F, T J, G2POut<T>& o) {
  bool nan = false, clamped = false;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T nx = x0[a] + sc.dt * v[a];
    if (!t_finite(nx)) nan = true;
    T lo = sc.origin[a] + sc.dx, hi = sc.origin[a] + T(sc.n[a] - 2) * sc.dx;
    T cx = t_fclamp(nx, lo, hi);
    if (cx != nx) clamped = true;
    o.x[a] = cx;
    o.v[a] = v[a];
  }
  o.err = (nan ? kErrNaN : 0u) | (clamped ? kErrDomain : 0u);
  o.clamped = clamped;
  o.needs_clamp = false;
  if (md.model == kPhysFluid) {
    T Jn = J * (T(1) + sc.dt * (o.C[0] + o.C[4] + o.C[8]));
    o.J = t_max(Jn, T(0.01));
#pragma unroll
    for (int k = 0; k < 9; ++k) o.F[k] = F[k];
    return;
  }
  T G[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) G[k] = ((k % 4 == 0) ? T(1) : T(0)) + sc.dt * o.C[k];
  mm3(G, F, o.F);
  if (md.model == kPhysSnow) {
    // elastic region: every singular value provably inside the clamp interval, F_E and J_p are final
    o.J = J;
    o.needs_clamp = !clamp_is_identity(o.F, T(1) - T(md.theta_c), T(1) + T(md.theta_s));
  } else {
    o.J = det3(o.F);
  }
}

// the C slot carries A = m C - k tau from here on (not for particles that still need the clamp)
template <class T>
__device__ __forceinline__ void g2p_physics_affine(const SceneDev<T>& sc, const MatDev& md, T m, G2POut<T>& o) {
  T A[9];
  affine_from_c(sc, md, m, o.C, o.F, o.J, A);
#pragma unroll
  for (int k = 0; k < 9; ++k) o.C[k] = A[k];
}

// The FP64 redo of the snow return mapping's SVD, taken by few particles: a call of its own, so that
// its registers and stack stay out of the FP32 path.
__device__ __noinline__ void svd3_fp64(const float* F, float* U, float* s, float* V) {
  double Fd[9], Ud[9], sd[3], Vd[9];
  for (int i = 0; i < 9; ++i) Fd[i] = double(F[i]);
  svd3(Fd, Ud, sd, Vd);
  for (int i = 0; i < 9; ++i) {
    U[i] = float(Ud[i]);
    V[i] = float(Vd[i]);
  }
  for (int i = 0; i < 3; ++i) s[i] = float(sd[i]);
}

// Snow return mapping: F = U S V^T, singular values clamped to [1-theta_c, 1+theta_s],
// J_p *= prod(S)/prod(S_clamped) (ae_physics/src/mpm.rs:565-606 plus Stomakhin's J_p), with the FP64
// SVD redo where a near-degenerate pair straddles a threshold.  Returns whether it was redone.
template <class T>
__device__ __forceinline__ bool snow_return(const MatDev& md, bool redo, T* F, T& J) {
  const T lo = T(1) - T(md.theta_c), hi = T(1) + T(md.theta_s);
  T U[9], sg[3], V[9];
  svd3(F, U, sg, V);
  bool fb = false;
  if constexpr (sizeof(T) == 4) {
    if (redo && svd3_straddles(sg, lo, hi)) {
      float tF[9], tU[9], ts[3], tV[9];
      for (int i = 0; i < 9; ++i) tF[i] = F[i];
      svd3_fp64(tF, tU, ts, tV);
      for (int i = 0; i < 9; ++i) {
        U[i] = tU[i];
        V[i] = tV[i];
      }
      for (int i = 0; i < 3; ++i) sg[i] = ts[i];
      fb = true;
    }
  }
  T scl[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) scl[k] = t_min(t_max(sg[k], lo), hi);
  J = J * ((sg[0] * sg[1] * sg[2]) / (scl[0] * scl[1] * scl[2]));
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      F[r * 3 + c] = U[r * 3 + 0] * scl[0] * V[c * 3 + 0] + U[r * 3 + 1] * scl[1] * V[c * 3 + 1] + U[r * 3 + 2] * scl[2] * V[c * 3 + 2];
  return fb;
}

// mpm_substep_serial_active / parallel_with_indices G2P (mpm_solver.rs:914-1053, 1206-1325).
// kAhead: the nine nodes of a plane are loaded before any is used, which hides their latency where the
// GPU holds few warps; at more registers per thread it has fewer of them where it could hold many (the
// kernel alone with and without: 20 000 particles 19.4 / 22.5 us, 30 000 19.1 / 21.4, 50 000 26.3 / 24.4,
// 400 000 99.6 / 78.3).
template <class T, bool kAhead>
__device__ __forceinline__ void g2p_reference(const VelTile<T>& vt, const SceneDev<T>& sc, const T* pos, const T* f,
                                              G2POut<T>& o) {
  using V4 = typename V4T<T>::type;
  int g[3];
  T fx[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T q = (pos[a] - sc.origin[a]) * sc.inv_dx - T(0.5);
    int gu = floor_to_int(q);
    fx[a] = q - T(gu);
    g[a] = max(gu, 0);
  }
  T nv[3] = {0, 0, 0}, nc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, gvm[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  // one node with mass: velocity, affine matrix and velocity gradient
  const auto add = [&](const V4& gv, int X, int Y, int Z, T ww, T dwx, T dwy, T dwz) {
    T g3[3] = {gv.x, gv.y, gv.z};
    nv[0] += ww * g3[0];
    nv[1] += ww * g3[1];
    nv[2] += ww * g3[2];
    T d3[3] = {(T(X) + T(0.5)) * sc.dx + sc.origin[0] - pos[0], (T(Y) + T(0.5)) * sc.dx + sc.origin[1] - pos[1],
               (T(Z) + T(0.5)) * sc.dx + sc.origin[2] - pos[2]};
    T scale = T(4) * sc.inv_dx * sc.inv_dx * ww;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) nc[r * 3 + c] += scale * g3[r] * d3[c];
    T dw[3] = {dwx, dwy, dwz};
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) gvm[r * 3 + c] -= ww * g3[r] * dw[c];
  };
  if constexpr (kAhead) {
    T wgt[3][3], dwg[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        wgt[a][k] = b_spline(T(k) - fx[a]);
        dwg[a][k] = b_spline_deriv(T(k) - fx[a]) * sc.inv_dx;
      }
#pragma unroll 1
    for (int dk = 0; dk < 3; ++dk) {
      V4 node[9];  // (a node outside the grid weighs 0)
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const int X = g[0] + q % 3, Y = g[1] + q / 3, Z = g[2] + dk;
        node[q] = (X < sc.n[0] && Y < sc.n[1] && Z < sc.n[2]) ? vt(sc, X, Y, Z) : mk4(T(0), T(0), T(0), T(0));
      }
      const T wz = dk == 0 ? wgt[2][0] : (dk == 1 ? wgt[2][1] : wgt[2][2]);
      const T dwz = dk == 0 ? dwg[2][0] : (dk == 1 ? dwg[2][1] : dwg[2][2]);
#pragma unroll
      for (int dj = 0; dj < 3; ++dj)
#pragma unroll
        for (int di = 0; di < 3; ++di) {
          const T ww = wgt[0][di] * wgt[1][dj] * wz;
          const V4 gv = node[dj * 3 + di];
          if (ww < T(1e-10) || gv.w < T(1e-12)) continue;
          add(gv, g[0] + di, g[1] + dj, g[2] + dk, ww, dwg[0][di], dwg[1][dj], dwz);
        }
    }
  } else {
#pragma unroll 1
    for (int dk = 0; dk < 3; ++dk)
#pragma unroll 1
      for (int dj = 0; dj < 3; ++dj)
#pragma unroll
        for (int di = 0; di < 3; ++di) {
          const T ww = b_spline(T(di) - fx[0]) * b_spline(T(dj) - fx[1]) * b_spline(T(dk) - fx[2]);
          const int X = g[0] + di, Y = g[1] + dj, Z = g[2] + dk;
          if (ww < T(1e-10) || X >= sc.n[0] || Y >= sc.n[1] || Z >= sc.n[2]) continue;
          const V4 gv = vt(sc, X, Y, Z);
          if (gv.w < T(1e-12)) continue;
          add(gv, X, Y, Z, ww, b_spline_deriv(T(di) - fx[0]) * sc.inv_dx, b_spline_deriv(T(dj) - fx[1]) * sc.inv_dx,
              b_spline_deriv(T(dk) - fx[2]) * sc.inv_dx);
        }
  }
  if (!t_finite(nv[0]) || !t_finite(nv[1]) || !t_finite(nv[2])) {
    nv[0] = nv[1] = nv[2] = T(0);
#pragma unroll
    for (int k = 0; k < 9; ++k) nc[k] = T(0);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) nv[a] = t_clamp(nv[a], T(-50), T(50));
  T np[3] = {t_add_mul_rn(pos[0], nv[0], sc.dt), t_add_mul_rn(pos[1], nv[1], sc.dt), t_add_mul_rn(pos[2], nv[2], sc.dt)};
  if (!t_finite(np[0]) || !t_finite(np[1]) || !t_finite(np[2])) {
    np[0] = T(6);
    np[1] = T(5);
    np[2] = T(6);
    nv[0] = nv[1] = nv[2] = T(0);
  }
  if (np[1] < T(0)) {
    np[1] = T(0);
    nv[1] = t_max(nv[1], T(0)) * T(0.5);
  }
  const T gmx = T(sc.n[0] - 1) * sc.dx, gmz = T(sc.n[2] - 1) * sc.dx;
  const T lox = sc.wall_origin ? sc.origin[0] : T(0), loz = sc.wall_origin ? sc.origin[2] : T(0);
  if (np[0] < lox) {
    np[0] = lox;
    nv[0] = t_max(nv[0], T(0)) * T(0.5);
  } else if (np[0] > gmx + lox) {
    np[0] = gmx + lox;
    nv[0] = t_min(nv[0], T(0)) * T(0.5);
  }
  if (np[2] < loz) {
    np[2] = loz;
    nv[2] = t_max(nv[2], T(0)) * T(0.5);
  } else if (np[2] > gmz + loz) {
    np[2] = gmz + loz;
    nv[2] = t_min(nv[2], T(0)) * T(0.5);
  }
  T nf[9];
  bool valid = true;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      T sum = T(0);
#pragma unroll
      for (int k = 0; k < 3; ++k) sum += (((r == k) ? T(1) : T(0)) + gvm[r * 3 + k] * sc.dt) * f[k * 3 + c];
      nf[r * 3 + c] = sum;
      if (!t_finite(sum) || t_abs(sum) > T(1e3)) valid = false;
    }
  if (valid) {
    o.J = t_clamp(det3(nf), T(0.1), T(10));
  } else {
    ident3(nf);
    o.J = T(1);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    o.v[a] = nv[a] * sc.damping;
    o.x[a] = np[a];
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    o.C[k] = nc[k];
    o.F[k] = nf[k];
  }
  o.err = 0;
  o.needs_clamp = o.clamped = false;
}

// mpm_substep_velocity_only G2P (mpm_solver.rs:1465-1571); C, F and J are carried unchanged
template <class T>
__device__ __forceinline__ void g2p_velonly(const VelTile<T>& vt, const SceneDev<T>& sc, const T* pos, G2POut<T>& o) {
  using V4 = typename V4T<T>::type;
  int g[3];
  T wx[3], wy[3], wz[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T q = (pos[a] - sc.origin[a]) * sc.inv_dx - T(0.5);
    int gu = floor_to_int(q);
    T fx = q - T(gu);
    g[a] = max(gu, 0);
    T* wa = a == 0 ? wx : (a == 1 ? wy : wz);
#pragma unroll
    for (int k = 0; k < 3; ++k) wa[k] = b_spline(T(k) - fx);
  }
  T nv[3] = {0, 0, 0};
#pragma unroll
  for (int dk = 0; dk < 3; ++dk) {
    if (wz[dk] < T(1e-10)) continue;
    int Z = g[2] + dk;
    if (Z >= sc.n[2]) continue;
#pragma unroll
    for (int dj = 0; dj < 3; ++dj) {
      if (wy[dj] < T(1e-10)) continue;
      int Y = g[1] + dj;
      if (Y >= sc.n[1]) continue;
      T wyz = wy[dj] * wz[dk];
#pragma unroll
      for (int di = 0; di < 3; ++di) {
        T ww = wx[di] * wyz;
        if (ww < T(1e-10)) continue;
        int X = g[0] + di;
        if (X >= sc.n[0]) continue;
        V4 gv = vt(sc, X, Y, Z);
        if (gv.w < T(1e-12)) continue;
        nv[0] += ww * gv.x;
        nv[1] += ww * gv.y;
        nv[2] += ww * gv.z;
      }
    }
  }
  if (!t_finite(nv[0]) || !t_finite(nv[1]) || !t_finite(nv[2])) nv[0] = nv[1] = nv[2] = T(0);
#pragma unroll
  for (int a = 0; a < 3; ++a) nv[a] = t_clamp(nv[a], T(-50), T(50));
  T np[3] = {t_add_mul_rn(pos[0], nv[0], sc.dt), t_add_mul_rn(pos[1], nv[1], sc.dt), t_add_mul_rn(pos[2], nv[2], sc.dt)};
  if (!t_finite(np[0]) || !t_finite(np[1]) || !t_finite(np[2])) {
    np[0] = pos[0];
    np[1] = pos[1];
    np[2] = pos[2];
    nv[0] = nv[1] = nv[2] = T(0);
  }
  if (np[1] < T(0)) {
    np[1] = T(0);
    nv[1] = t_max(nv[1], T(0)) * T(0.5);
  }
  const T gmx = T(sc.n[0] - 1) * sc.dx, gmz = T(sc.n[2] - 1) * sc.dx;
  if (np[0] < T(0)) {
    np[0] = T(0);
    nv[0] = t_max(nv[0], T(0)) * T(0.5);
  } else if (np[0] > gmx + sc.origin[0]) {
    np[0] = gmx + sc.origin[0];
    nv[0] = t_min(nv[0], T(0)) * T(0.5);
  }
  if (np[2] < T(0)) {
    np[2] = T(0);
    nv[2] = t_max(nv[2], T(0)) * T(0.5);
  } else if (np[2] > gmz + sc.origin[2]) {
    np[2] = gmz + sc.origin[2];
    nv[2] = t_min(nv[2], T(0)) * T(0.5);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    o.v[a] = nv[a] * sc.damping;
    o.x[a] = np[a];
  }
  o.err = 0;
  o.needs_clamp = o.clamped = false;
}

// in-grid stencil node range of a position along one axis (empty when lo > hi)
template <class T, int MODE>
__device__ __forceinline__ void stencil_range(const SceneDev<T>& sc, T x, int a, int& lo, int& hi) {
  int g = floor_to_int((x - sc.origin[a]) * sc.inv_dx - T(0.5));
  if (MODE != AE_MPM_MODE_PHYSICS) g = max(g, 0);
  lo = max(g, 0);
  hi = min(g + 2, sc.n[a] - 1);
}

template <class T, int MODE, bool kAhead>
__global__ void __launch_bounds__(256, (MODE == AE_MPM_MODE_PHYSICS && sizeof(T) == 4) ? 4 : 1) g2p_kernel(WorldDev<T> w, uint32_t* epoch,
                                                                                                    int write_keys) {
  using V4 = typename V4T<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  V4* tile = reinterpret_cast<V4*>(smem);
  // physics mode gathers straight from the grid (no block tile, no barriers)
  constexpr bool kTile = MODE != AE_MPM_MODE_PHYSICS;
  V4* stage = kTile ? tile + w.max_tile_nodes : tile;  // a1..a3 of this block's particles: stage[k * nt + tid]
  __shared__ int s_lo[3], s_hi[3];
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const int tid = threadIdx.x, lane = tid & 31, nt = blockDim.x;
  const int j = ch.y + tid;
  const bool live = j < ch.z;
  if (blockIdx.x == 0 && tid == 0) {
    *w.touched_count = 0u;
    if (w.cell_count) *w.cell_count = 0u;
    *epoch += 1u;
  }
  if (kTile) {
    if (tid < 3) {
      s_lo[tid] = INT_MAX;
      s_hi[tid] = INT_MIN;
    }
    __syncthreads();
  }
  uint32_t src = 0;
  V4 a0 = mk4(T(0), T(0), T(0), T(0));
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
  bool has = false;
  if (live) {
    src = w.perm ? w.perm[j] : uint32_t(j);
    // F, J and the material arrive in shared memory while the node velocities are gathered
#pragma unroll
    for (int k = 0; k < 3; ++k) cp_async_v4(stage + k * nt + tid, w.in[1 + k] + src);
    cp_async_commit();
    a0 = ld4(w.in[0] + src);
    const T x3[3] = {a0.x, a0.y, a0.z};
    has = true;
    if (kTile) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        stencil_range<T, MODE>(sc, x3[a], a, lo[a], hi[a]);
        if (lo[a] > hi[a]) has = false;
      }
    }
  }
  if (kTile) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      int l = __reduce_min_sync(0xffffffffu, has ? lo[a] : INT_MAX);
      int h = __reduce_max_sync(0xffffffffu, has ? hi[a] : INT_MIN);
      if (lane == 0 && l != INT_MAX) {
        atomicMin(&s_lo[a], l);
        atomicMax(&s_hi[a], h);
      }
    }
    __syncthreads();
  }
  VelTile<T> vt;
  vt.tile = nullptr;
  vt.vel = w.vel;
  vt.L0 = kTile ? s_lo[0] : INT_MAX;
  vt.L1 = kTile ? s_lo[1] : INT_MAX;
  vt.L2 = kTile ? s_lo[2] : INT_MAX;
  if (kTile && vt.L0 != INT_MAX) {
    const int D0 = s_hi[0] - vt.L0 + 1, D1 = s_hi[1] - vt.L1 + 1, D2 = s_hi[2] - vt.L2 + 1;
    const int p0 = 32 - __clz(D0 - 1), p1 = 32 - __clz(D1 - 1);
    vt.p0 = p0;
    vt.sp = p0 + p1;
    const int slots = D2 << vt.sp;
    if (slots <= w.max_tile_nodes) {
      const int mx = (1 << p0) - 1, my = (1 << p1) - 1;
      for (int t = tid; t < slots; t += blockDim.x) {
        const int X = t & mx, Y = (t >> p0) & my;
        if (X < D0 && Y < D1) tile[t] = ld4(w.vel + node_index(sc, vt.L0 + X, vt.L1 + Y, vt.L2 + (t >> vt.sp)));
      }
      vt.tile = tile;
    }
  }
  if (kTile) __syncthreads();
  uint32_t err = 0;
  bool cl = false, need = false, off = false;
  const uint32_t live_mask = __ballot_sync(0xffffffffu, live);
  if (live) {
    const T x0[3] = {a0.x, a0.y, a0.z};
    G2POut<T> o;
    T pv[3] = {0, 0, 0};
    if (MODE == AE_MPM_MODE_PHYSICS) {
      bool done;
      const GridRows<T> rows{w.vel, sc.blk_off, uint32_t(sc.nb[0]), uint32_t(sc.nb[1])};
      if constexpr (sizeof(T) == 4)
        done = g2p_physics_gather_sep_f2(rows, sc, x0, pv, o.C);
      else
        done = g2p_physics_gather_sep<T>(rows, sc, x0, pv, o.C);
      if (!done) g2p_physics_gather<T>(vt, sc, x0, pv, o.C);  // stencil partly outside the grid
    }
    cp_async_wait_all();
    const V4 a1 = stage[tid], a2 = stage[nt + tid], a3 = stage[2 * nt + tid];
    const T F[9] = {a1.x, a1.y, a1.z, a1.w, a2.x, a2.y, a2.z, a2.w, a3.x};
    if (MODE == AE_MPM_MODE_PHYSICS) {
      const MatDev& md = mat_of(w, sc, Bits<T>::unpack(a3.z) & 0xffffu);
      g2p_physics_move<T>(sc, md, x0, pv, F, a3.y, o);
      if (!o.needs_clamp) g2p_physics_affine<T>(sc, md, a0.w, o);
    } else if (MODE == AE_MPM_MODE_REFERENCE) {
      g2p_reference<T, kAhead>(vt, sc, x0, F, o);
    } else {
      const V4 a4 = ld4(w.in[4] + src), a5 = ld4(w.in[5] + src), a6 = ld4(w.in[6] + src);
      g2p_velonly<T>(vt, sc, x0, o);
#pragma unroll
      for (int k = 0; k < 9; ++k) o.F[k] = F[k];
      o.J = a3.y;
      o.C[0] = a4.w;
      o.C[1] = a5.x;
      o.C[2] = a5.y;
      o.C[3] = a5.z;
      o.C[4] = a5.w;
      o.C[5] = a6.x;
      o.C[6] = a6.y;
      o.C[7] = a6.z;
      o.C[8] = a6.w;
    }
    w.out[0][j] = mk4(o.x[0], o.x[1], o.x[2], a0.w);
    w.out[1][j] = mk4(o.F[0], o.F[1], o.F[2], o.F[3]);
    w.out[2][j] = mk4(o.F[4], o.F[5], o.F[6], o.F[7]);
    w.out[3][j] = mk4(o.F[8], o.J, a3.z, a3.w);
    w.out[4][j] = mk4(o.v[0], o.v[1], o.v[2], o.C[0]);
    w.out[5][j] = mk4(o.C[1], o.C[2], o.C[3], o.C[4]);
    w.out[6][j] = mk4(o.C[5], o.C[6], o.C[7], o.C[8]);
    // the next substep's cell key, only when the next substep sorts (the world tracks this); with
    // dense grouping counted in its cell too
    if (write_keys) {
      const uint32_t key = cell_key(sc, MODE, o.x[0], o.x[1], o.x[2]);
      w.keys[j] = key;
      if (w.bins) {
        const uint32_t peers = __match_any_sync(live_mask, key);
        if (lane == __ffs(peers) - 1) atomicAdd(w.bins + key, uint32_t(__popc(peers)));
      }
      off = key == sc.dead_key;
    }
    err = o.err;
    cl = o.clamped;
    need = o.needs_clamp;
  } else if (j < ch.w && write_keys && !w.bins) {
    w.keys[j] = sc.dead_key;
  }
  if (kTile && write_keys && w.dead_cnt) {
    const int c = __syncthreads_count(off);
    if (tid == 0) w.dead_cnt[blockIdx.x] = uint32_t(c);
  }
  // warp-aggregated error words, counters and clamp-queue appends
  const uint32_t e = __reduce_or_sync(0xffffffffu, err);
  const uint32_t ncl = __popc(__ballot_sync(0xffffffffu, cl));
  const uint32_t qmask = __ballot_sync(0xffffffffu, need);
  uint32_t qbase = 0;
  if (lane == 0) {
    if (e) atomicOr(w.err + 4 * ch.x, e);
    if (ncl) atomicAdd(w.err + 4 * ch.x + 2, ncl);
    if (qmask) qbase = atomicAdd(w.clamp_count, uint32_t(__popc(qmask)));
  }
  qbase = __shfl_sync(0xffffffffu, qbase, 0);
  if (need) w.clamp_queue[qbase + __popc(qmask & ((1u << lane) - 1u))] = make_uint2(uint32_t(j), uint32_t(ch.x));
}

// Snow return mapping for the particles G2P queued, then A from the returned F.
// 64 registers, 8 blocks of 128 per SM.
template <class T>
__global__ void __launch_bounds__(128, 8) snow_clamp_kernel(WorldDev<T> w) {
  using V4 = typename V4T<T>::type;
  // the particle's mass and C slots arrive here while its SVD runs (each thread its own column)
  __shared__ V4 pre[4][128];
  const int tid = threadIdx.x;
  const uint32_t count = launch_count(w.clamp_count);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint2 q = w.clamp_queue[i];
    cp_async_v4(&pre[0][tid], w.out[0] + q.x);
    cp_async_v4(&pre[1][tid], w.out[4] + q.x);
    cp_async_v4(&pre[2][tid], w.out[5] + q.x);
    cp_async_v4(&pre[3][tid], w.out[6] + q.x);
    cp_async_commit();
    const SceneDev<T>& sc = w.scenes[q.y];
    V4 a1 = w.out[1][q.x], a2 = w.out[2][q.x], a3 = w.out[3][q.x];
    const MatDev& md = mat_of(w, sc, Bits<T>::unpack(a3.z) & 0xffffu);
    T nF[9] = {a1.x, a1.y, a1.z, a1.w, a2.x, a2.y, a2.z, a2.w, a3.x}, J = a3.y;
    const bool fb = snow_return<T>(md, w.svd_fallback != 0, nF, J);
    w.out[1][q.x] = mk4(nF[0], nF[1], nF[2], nF[3]);
    w.out[2][q.x] = mk4(nF[4], nF[5], nF[6], nF[7]);
    w.out[3][q.x] = mk4(nF[8], J, a3.z, a3.w);
    // G2P left C in the C slot of queued particles: turn it into A with the returned F and J_p
    cp_async_wait_all();
    const V4 a0 = pre[0][tid], a4 = pre[1][tid], a5 = pre[2][tid], a6 = pre[3][tid];
    const T C[9] = {a4.w, a5.x, a5.y, a5.z, a5.w, a6.x, a6.y, a6.z, a6.w};
    T A[9];
    affine_from_c(sc, md, a0.w, C, nF, J, A);
    w.out[4][q.x] = mk4(a4.x, a4.y, a4.z, A[0]);
    w.out[5][q.x] = mk4(A[1], A[2], A[3], A[4]);
    w.out[6][q.x] = mk4(A[5], A[6], A[7], A[8]);
    if (fb) atomicAdd(w.err + 4 * q.y + 1, 1u);
  }
}

// ============================================================================================
// fused G2P + P2G for physics mode (grid -> particle -> grid in one pass over the particles)
// ============================================================================================
// G2P of substep s computes each particle's new position, mass-weighted velocity and affine
// matrix A = m C - k tau; those are exactly the inputs of P2G for substep s + 1, so the same
// kernel scatters them into the (already cleared) accumulator of the next substep while they are
// still in registers.  P2G then never re-reads the particle state.  Snow particles whose F left
// the elastic region get A only after the return mapping: the clamp kernel scatters them.
//
// Per-warp shared staging of the column-lane scatter (the layout of p2g_lanes_kernel, one
// contiguous region per warp): 32 particles x (9 column vectors, x weights + mass, dx times A's x
// column) and 32 run records.  Per-thread data the warp stages before the scatter (the cp.async
// prefetch of F, J and the material) lives in the same region.
template <class T>
struct WarpStage {
  using V4 = typename V4T<T>::type;
  V4* col;   // col[pos * 9 + column]
  V4* wxm;   // wxm[pos] = (wx0, wx1, wx2, m)
  V4* acol;  // acol[pos] = dx * A[.][0]
  int4* gk;  // gk[pos] = (cell key, block row pitch and plane pitch of its scene, -)
};
template <class T>
__host__ __device__ constexpr size_t warp_stage_bytes() {
  return sizeof(typename V4T<T>::type) * 32 * kLaneVecs + sizeof(int4) * 32;
}
template <class T>
__device__ __forceinline__ WarpStage<T> warp_stage(unsigned char* smem, int warp) {
  using V4 = typename V4T<T>::type;
  unsigned char* base = smem + size_t(warp) * warp_stage_bytes<T>();
  WarpStage<T> s;
  s.col = reinterpret_cast<V4*>(base);
  s.wxm = s.col + 32 * 9;
  s.acol = s.wxm + 32;
  s.gk = reinterpret_cast<int4*>(s.acol + 32);
  return s;
}

// The column-lane scatter of one warp (p2g_lanes_kernel's grouping, runs and vector reductions)
// for particles whose 27 stencil nodes all lie inside their scene's grid, which G2P's domain clamp
// guarantees.  Every lane of the warp calls it; has = false lanes contribute nothing.  x is the
// position, mv = m v, A = m C - k tau.  The cell key is the global index of the stencil's base
// node, unique across scenes.  kMixed: lanes may belong to different scenes (sc is the lane's own);
// otherwise every lane belongs to scene sc.  write_keys: the
// next substep sorts, so each particle's key goes to its slot and, with dense grouping, each group
// of equal keys is counted in its cell with one atomic (the grouping is needed here anyway).
// runs of at most this many particles are summed one node per lane; longer ones by the column lanes
constexpr int kShortRun = 6;

template <class T, bool kMixed>
__device__ __forceinline__ void p2g_warp_scatter(const WorldDev<T>& w, const SceneDev<T>& sc, bool has, const T* x,
                                                 T m, const T* mv, const T* A, const WarpStage<T>& st, uint32_t slot,
                                                 int write_keys) {
  using V4 = typename V4T<T>::type;
  const int lane = threadIdx.x & 31;
  int g[3] = {0, 0, 0};
  T fx[3] = {0, 0, 0}, wt[3][3];
  if (has) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const T X = (x[a] - sc.origin[a]) * sc.inv_dx;
      const int b = floor_to_int(X - T(0.5));
      fx[a] = X - T(b);
      g[a] = b;
      const T t0 = T(1.5) - fx[a], t1 = fx[a] - T(1), t2 = fx[a] - T(0.5);
      wt[a][0] = T(0.5) * t0 * t0;
      wt[a][1] = T(0.75) - t1 * t1;
      wt[a][2] = T(0.5) * t2 * t2;
    }
  }
  const uint32_t key = has ? node_index(sc, g[0], g[1], g[2]) : 0xffffffffu;
  // equal keys anywhere in the warp form one group: groups in order of their first lane, lanes
  // within a group in lane order; pos is this particle's slot in that grouped order
  const uint32_t peers = __match_any_sync(0xffffffffu, key);
  const int leader = __ffs(peers) - 1;
  if (write_keys && has) {
    w.keys[slot] = key;
    if (w.bins && lane == leader) atomicAdd(w.bins + key, uint32_t(__popc(peers)));
  }
  const uint32_t lead_cnt = lane == leader ? uint32_t(__popc(peers)) : 0u;
  uint32_t incl = lead_cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t lead_off = incl - lead_cnt;
  const int pos = int(__shfl_sync(0xffffffffu, lead_off, leader)) + __popc(peers & ((1u << lane) - 1u));
  uint32_t starts = __reduce_or_sync(0xffffffffu, lane == leader ? (1u << lead_off) : 0u);
  if (has) {
    const T dx = sc.dx;
    T c0[3], c1[3], c2[3], qv[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      c0[r] = dx * A[3 * r + 0];
      c1[r] = dx * A[3 * r + 1];
      c2[r] = dx * A[3 * r + 2];
      qv[r] = mv[r] - (c0[r] * fx[0] + c1[r] * fx[1] + c2[r] * fx[2]);
    }
    V4* cq = st.col + pos * 9;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const T ux = qv[0] + T(b) * c1[0] + T(c) * c2[0];
        const T uy = qv[1] + T(b) * c1[1] + T(c) * c2[1];
        const T uz = qv[2] + T(b) * c1[2] + T(c) * c2[2];
        cq[b + 3 * c] = mk4(ux, uy, uz, wt[1][b] * wt[2][c]);
      }
    }
    st.wxm[pos] = mk4(wt[0][0], wt[0][1], wt[0][2], m);
    st.acol[pos] = mk4(c0[0], c0[1], c0[2], T(0));
  }
  st.gk[pos] = make_int4(int(key), sc.nb[0], sc.nb[0] * sc.nb[1], 0);
  if (kMixed && has) {
    // the stencil's blocks (at most 2 per axis), every lane its own particle's at once: marked run by
    // run, each run would wait for its flags in turn
    uint32_t gb[8];
    uint32_t set[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const int bx = (g[0] + 2 * (o & 1)) >> 2, by = (g[1] + (o & 2)) >> 2, bz = (g[2] + ((o >> 1) & 2)) >> 2;
      gb[o] = sc.blk_off + (uint32_t(bz) * uint32_t(sc.nb[1]) + uint32_t(by)) * uint32_t(sc.nb[0]) + uint32_t(bx);
    }
#pragma unroll
    for (int o = 0; o < 8; ++o) set[o] = *static_cast<volatile uint32_t*>(w.blk_flag + gb[o]);
#pragma unroll
    for (int o = 0; o < 8; ++o)
      if (set[o] == 0u) mark_block(w, gb[o]);
  }
  __syncwarp();
  // lanes 0..26 are 3 particle groups x 9 (y,z) columns; lanes 27..31 mirror lanes 22..26
  // (in-bounds reads, results never used)
  const int grp = lane < 27 ? lane / 9 : 2;
  const int jc = lane < 27 ? lane - 9 * grp : lane - 23;
  const int nb = jc % 3, nc = jc / 3;
  const V4* colw = st.col + jc;
  while (starts) {
    const int s0 = __ffs(starts) - 1;
    starts &= starts - 1u;
    const int e0 = starts ? __ffs(starts) - 1 : 32;
    const int4 run = st.gk[s0];
    const uint32_t rk = uint32_t(run.x);
    if (rk == 0xffffffffu) continue;
    // node index of the run's stencil node (X, Y, Z) = base + x part + y part + z part, each part the
    // distance of that axis from the base node in the block-major order
    const int r0 = int(rk & 3u), r1 = int((rk >> 2) & 3u), r2 = int((rk >> 4) & 3u);
    const uint32_t row64 = uint32_t(run.y) << 6, plane64 = uint32_t(run.z) << 6;
    const uint32_t rb = rk & ~63u;
    if (e0 - s0 <= kShortRun) {
      // a short run: one lane per stencil node (27 lanes), each summing every particle of the run
      // for its node; no combine across lane groups, one vector reduction per lane
      const int ln = lane < 27 ? lane : 26;
      const int xa = ln % 3, jn = ln / 3;
      const T fa = T(xa);
      const V4* cn = st.col + jn;
      T m = 0, px = 0, py = 0, pz = 0;
      if constexpr (sizeof(T) == 4) {  // x and y as one packed pair
        float2 pxy = make_float2(0.f, 0.f);
        const float2 fa2 = make_float2(fa, fa);
        for (int i = s0; i < e0; ++i) {
          const float4 u = cn[i * 9];
          const float4 r = st.wxm[i];
          const float4 a = st.acol[i];
          const float W = (xa == 0 ? r.x : (xa == 1 ? r.y : r.z)) * u.w;
          m += W * r.w;
          pxy = __ffma2_rn(make_float2(W, W), __ffma2_rn(fa2, make_float2(a.x, a.y), make_float2(u.x, u.y)), pxy);
          pz += W * (u.z + fa * a.z);
        }
        px = pxy.x;
        py = pxy.y;
      } else {
        for (int i = s0; i < e0; ++i) {
          const V4 u = cn[i * 9];
          const V4 r = st.wxm[i];
          const V4 a = st.acol[i];
          const T W = (xa == 0 ? r.x : (xa == 1 ? r.y : r.z)) * u.w;
          m += W * r.w;
          px += W * (u.x + fa * a.x);
          py += W * (u.y + fa * a.y);
          pz += W * (u.z + fa * a.z);
        }
      }
      if (lane < 27 && m != T(0)) {
        const uint32_t Xl = uint32_t(r0 + xa), Yl = uint32_t(r1 + jn % 3), Zl = uint32_t(r2 + jn / 3);
        const uint32_t node = rb + ((Xl >> 2) << 6) + (Yl >> 2) * row64 + (Zl >> 2) * plane64 +
                              ((Zl & 3u) << 4 | (Yl & 3u) << 2 | (Xl & 3u));
        atomic_add4(w.acc + node, m, px, py, pz);
      }
      continue;
    }
    T m0 = 0, x0 = 0, y0 = 0, z0 = 0, m1 = 0, x1 = 0, y1 = 0, z1 = 0, m2 = 0, x2 = 0, y2 = 0, z2 = 0;
    if constexpr (sizeof(T) == 4) {  // x and y of each node as one packed pair
      float2 q0 = make_float2(0.f, 0.f), q1 = q0, q2 = q0;
#pragma unroll 2
      for (int i = s0 + grp; i < e0; i += 3) {
        const float4 u = colw[i * 9];
        const float4 r = st.wxm[i];
        const float4 a = st.acol[i];
        const float W0 = r.x * u.w, W1 = r.y * u.w, W2 = r.z * u.w;
        const float2 axy = make_float2(a.x, a.y), u0 = make_float2(u.x, u.y);
        const float2 u1 = __fadd2_rn(u0, axy), u2 = __fadd2_rn(u1, axy);
        m0 += W0 * r.w;
        m1 += W1 * r.w;
        m2 += W2 * r.w;
        q0 = __ffma2_rn(make_float2(W0, W0), u0, q0);
        q1 = __ffma2_rn(make_float2(W1, W1), u1, q1);
        q2 = __ffma2_rn(make_float2(W2, W2), u2, q2);
        const float uz1 = u.z + a.z;
        z0 += W0 * u.z;
        z1 += W1 * uz1;
        z2 += W2 * (uz1 + a.z);
      }
      x0 = q0.x, y0 = q0.y, x1 = q1.x, y1 = q1.y, x2 = q2.x, y2 = q2.y;
    } else
#pragma unroll 2
    for (int i = s0 + grp; i < e0; i += 3) {
      const V4 u = colw[i * 9];
      const V4 r = st.wxm[i];
      const V4 a = st.acol[i];
      const T W0 = r.x * u.w, W1 = r.y * u.w, W2 = r.z * u.w;
      m0 += W0 * r.w;
      x0 += W0 * u.x;
      y0 += W0 * u.y;
      z0 += W0 * u.z;
      const T ux = u.x + a.x, uy = u.y + a.y, uz = u.z + a.z;
      m1 += W1 * r.w;
      x1 += W1 * ux;
      y1 += W1 * uy;
      z1 += W1 * uz;
      m2 += W2 * r.w;
      x2 += W2 * (ux + a.x);
      y2 += W2 * (uy + a.y);
      z2 += W2 * (uz + a.z);
    }
    if (e0 - s0 > 1) {
      auto groups = [](T v) { return v + __shfl_down_sync(0xffffffffu, v, 9) + __shfl_down_sync(0xffffffffu, v, 18); };
      m0 = groups(m0), x0 = groups(x0), y0 = groups(y0), z0 = groups(z0);
      m1 = groups(m1), x1 = groups(x1), y1 = groups(y1), z1 = groups(z1);
      m2 = groups(m2), x2 = groups(x2), y2 = groups(y2), z2 = groups(z2);
    }
    if (lane < 9) {
      const uint32_t Yl = uint32_t(r1 + nb), Zl = uint32_t(r2 + nc);
      const uint32_t row = rb + (Yl >> 2) * row64 + (Zl >> 2) * plane64 + ((Zl & 3u) << 4 | (Yl & 3u) << 2);
      auto node = [row](uint32_t xl) { return row + ((xl >> 2) << 6 | (xl & 3u)); };
      if (m0 != T(0)) atomic_add4(w.acc + node(uint32_t(r0)), m0, x0, y0, z0);
      if (m1 != T(0)) atomic_add4(w.acc + node(uint32_t(r0 + 1)), m1, x1, y1, z1);
      if (m2 != T(0)) atomic_add4(w.acc + node(uint32_t(r0 + 2)), m2, x2, y2, z2);
    }
  }
  if (!kMixed) {  // grid blocks of the warp's stencil bounding box (all inside the grid)
    int B[3], NB[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int l = __reduce_min_sync(0xffffffffu, has ? g[a] : INT_MAX);
      const int h = __reduce_max_sync(0xffffffffu, has ? g[a] + 2 : INT_MIN);
      B[a] = l >> 2;
      NB[a] = l == INT_MAX ? 0 : (h >> 2) - (l >> 2) + 1;
    }
    const int nblk = NB[0] * NB[1] * NB[2];
    for (int t = lane; t < nblk; t += 32) {
      const int bx = B[0] + t % NB[0], by = B[1] + (t / NB[0]) % NB[1], bz = B[2] + t / (NB[0] * NB[1]);
      mark_block(w, sc.blk_off + (uint32_t(bz) * uint32_t(sc.nb[1]) + uint32_t(by)) * uint32_t(sc.nb[0]) + uint32_t(bx));
    }
  }
  __syncwarp();  // the staging region is free again
}

// snow_return on F (park[0..8]) and J_p (park[9]) at a stride of 32 in the warp's shared staging: a
// call of its own, so that the fused kernel's other particles keep their registers
template <class T>
__device__ __noinline__ bool snow_return_parked(const MatDev* md, bool redo, T* park) {
  T F[9], J = park[9 * 32];
#pragma unroll
  for (int k = 0; k < 9; ++k) F[k] = park[k * 32];
  const bool fb = snow_return<T>(*md, redo, F, J);
#pragma unroll
  for (int k = 0; k < 9; ++k) park[k * 32] = F[k];
  park[9 * 32] = J;
  return fb;
}

// Yielding snow particles of a warp from which on the fused kernel maps them back itself.  Where they
// come in whole warps this saves the clamp kernel's pass over them (512 scenes: fused + clamp 846 + 401 ->
// 1077 + 25 us; 8.4 M dam break from a yielding start 734 + 134 -> 827 + 23).  The call costs a world with
// snow 2 % of the kernel while nothing yields (dam break 711 -> 727 us; 9.4 -> 10.0 us for 2 000 to 20 000
// particles).  The mapping behind the scatter,
// as a function or as a second turn of a loop around it, cost more in both states (752 / 837 us).
constexpr int kInlineClamp = 8;

// G2P of substep s and P2G of substep s + 1 (physics mode).  The grid update of substep s ran
// before; w.touched / w.touched_count are the touched-block list of substep s + 1.
// kSnow: the world has snow materials.  kPer: particles per warp; a chunk of blockDim slots takes
// 32 / kPer CTAs.
template <class T, bool kSnow, int kPer>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) g2p2g_kernel(WorldDev<T> w, uint32_t* epoch,
                                                                              int write_keys) {
  using V4 = typename V4T<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kSplit = 32 / kPer;
  const int4 ch = chunk_at(w, blockIdx.x / kSplit, blockDim.x);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const int tid = threadIdx.x, lane = tid & 31;
  const WarpStage<T> st = warp_stage<T>(smem, tid >> 5);
  V4* pre = st.col;  // F, J and the material of the warp's particles (pre[k * 32 + lane]) until the scatter
  const int j = ch.y + int(blockIdx.x % kSplit) * int(blockDim.x / kSplit) + (tid >> 5) * kPer + lane;
  const bool slot = kPer == 32 || lane < kPer, live = slot && j < ch.z;
  if (blockIdx.x == 0 && tid == 0) *epoch += 1u;
  uint32_t err = 0;
  bool cl = false, need = false, has = false;
  T xs[3] = {0, 0, 0}, m = 0, mv[3] = {0, 0, 0}, A[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  const uint32_t live_mask = __ballot_sync(0xffffffffu, live);
  if (live) {
    const uint32_t src = w.perm ? w.perm[j] : uint32_t(j);
#pragma unroll
    for (int k = 0; k < 3; ++k) cp_async_v4(pre + k * 32 + lane, w.in[1 + k] + src);
    cp_async_commit();
    const V4 a0 = ld4(w.in[0] + src);
    const T x0[3] = {a0.x, a0.y, a0.z};
    G2POut<T> o;
    T pv[3] = {0, 0, 0};
    bool done;
    if constexpr (sizeof(T) == 4)
      done = g2p_physics_gather_sep_f2(GridRows<T>{w.vel, sc.blk_off, uint32_t(sc.nb[0]), uint32_t(sc.nb[1])}, sc, x0,
                                       pv, o.C);
    else
      done = g2p_physics_gather_sep<T>(GridRows<T>{w.vel, sc.blk_off, uint32_t(sc.nb[0]), uint32_t(sc.nb[1])}, sc, x0,
                                       pv, o.C);
    if (!done) {  // stencil partly outside the grid (a particle's first substep)
      VelTile<T> vt;
      vt.tile = nullptr;
      vt.vel = w.vel;
      g2p_physics_gather<T>(vt, sc, x0, pv, o.C);
    }
    cp_async_wait_all();
    const V4 a1 = pre[lane], a2 = pre[32 + lane], a3 = pre[64 + lane];
    const T F[9] = {a1.x, a1.y, a1.z, a1.w, a2.x, a2.y, a2.z, a2.w, a3.x};
    const MatDev& md = mat_of(w, sc, Bits<T>::unpack(a3.z) & 0xffffu);
    g2p_physics_move<T>(sc, md, x0, pv, F, a3.y, o);
    need = kSnow && o.needs_clamp;
    // Yielding snow: a warp with many such particles maps them back here; a few are left to the
    // clamp kernel, which packs 32 of them from all over into a warp.
    m = a0.w;
    if (kSnow && __popc(__ballot_sync(live_mask, need)) >= kInlineClamp) {
      // the particle waits in the warp's staging region (past the prefetched F) during the call
      T* park = reinterpret_cast<T*>(pre + 96) + lane;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        park[k * 32] = o.F[k];
        park[(10 + k) * 32] = o.C[k];
      }
      park[9 * 32] = o.J;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        park[(19 + a) * 32] = o.x[a];
        park[(22 + a) * 32] = o.v[a];
      }
      park[25 * 32] = m;
      if (need && snow_return_parked<T>(&md, w.svd_fallback != 0, park)) atomicAdd(w.err + 4 * ch.x + 1, 1u);
      need = false;
      const T volatile* back = park;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        o.F[k] = back[k * 32];
        o.C[k] = back[(10 + k) * 32];
      }
      o.J = back[9 * 32];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        o.x[a] = back[(19 + a) * 32];
        o.v[a] = back[(22 + a) * 32];
      }
      m = back[25 * 32];
    }
    if (!need) g2p_physics_affine<T>(sc, md, m, o);
    w.out[0][j] = mk4(o.x[0], o.x[1], o.x[2], m);
    w.out[1][j] = mk4(o.F[0], o.F[1], o.F[2], o.F[3]);
    w.out[2][j] = mk4(o.F[4], o.F[5], o.F[6], o.F[7]);
    w.out[3][j] = mk4(o.F[8], o.J, a3.z, a3.w);
    w.out[4][j] = mk4(o.v[0], o.v[1], o.v[2], o.C[0]);
    w.out[5][j] = mk4(o.C[1], o.C[2], o.C[3], o.C[4]);
    w.out[6][j] = mk4(o.C[5], o.C[6], o.C[7], o.C[8]);
    err = o.err;
    cl = o.clamped;
    has = !need;  // the queued particles are scattered (and keyed) by the clamp kernel
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      xs[a] = o.x[a];
      mv[a] = m * o.v[a];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) A[k] = o.C[k];
  } else if (slot && j < ch.w && write_keys && !w.bins) {
    w.keys[j] = sc.dead_key;
  }
  const uint32_t e = __reduce_or_sync(0xffffffffu, err);
  const uint32_t ncl = __popc(__ballot_sync(0xffffffffu, cl));
  const uint32_t qmask = kSnow ? __ballot_sync(0xffffffffu, need) : 0u;
  uint32_t qbase = 0;
  if (lane == 0) {
    if (e) atomicOr(w.err + 4 * ch.x, e);
    if (ncl) atomicAdd(w.err + 4 * ch.x + 2, ncl);
    if (kSnow && qmask) qbase = atomicAdd(w.clamp_count, uint32_t(__popc(qmask)));
  }
  if (kSnow) {
    qbase = __shfl_sync(0xffffffffu, qbase, 0);
    if (need) w.clamp_queue[qbase + __popc(qmask & ((1u << lane) - 1u))] = make_uint2(uint32_t(j), uint32_t(ch.x));
  }
  __syncwarp();  // every lane has read its F, J and material: the scatter may reuse the region
  p2g_warp_scatter<T, false>(w, sc, has, xs, m, mv, A, st, uint32_t(j), write_keys);
}

// The snow return mapping of snow_clamp_kernel for the particles the fused kernel queued, each
// then scattered into the next substep's accumulator with its final A.  A warp takes consecutive
// queue entries (possibly of several scenes of a world): as many as spread the queue over all warps,
// between 4 and 32, because scattered particles are runs of their own that a warp sums one after
// another (a short queue took 16 us with 32 entries per warp).  80 registers and 6 CTAs per SM: at 64
// and 8 the return mapping spills (16.7 against 19.3 us a launch in a batch of snow and other scenes).
// Launched with those 6 per SM; with 8, the last two waited for a second wave (20 000 quiet particles
// sorted every substep: 19.3 -> 18.8 us).
template <class T>
__global__ void __launch_bounds__(128, 6) snow_clamp_scatter_kernel(WorldDev<T> w, int write_keys) {
  using V4 = typename V4T<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const WarpStage<T> st = warp_stage<T>(smem, threadIdx.x >> 5);
  V4* pre = st.col;  // position+mass, velocity+A of the queued particle: pre[k * 32 + lane], until the scatter
  const uint32_t count = launch_count(w.clamp_count);
  const uint32_t warps = gridDim.x * (blockDim.x >> 5), warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t per = min(32u, max(4u, (count + warps - 1) / warps));
  for (uint32_t base = warp * per; base < count; base += warps * per) {
    const uint32_t i = base + lane;
    const bool valid = uint32_t(lane) < per && i < count;
    const uint2 q = valid ? w.clamp_queue[i] : make_uint2(0u, 0u);
    const SceneDev<T>& sc = w.scenes[q.y];
    T xs[3] = {0, 0, 0}, m = 0, mv[3] = {0, 0, 0}, A[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (valid) {
      cp_async_v4(pre + lane, w.out[0] + q.x);
      cp_async_v4(pre + 32 + lane, w.out[4] + q.x);
      cp_async_v4(pre + 64 + lane, w.out[5] + q.x);
      cp_async_v4(pre + 96 + lane, w.out[6] + q.x);
      cp_async_commit();
      const V4 a1 = w.out[1][q.x], a2 = w.out[2][q.x], a3 = w.out[3][q.x];
      const MatDev& md = mat_of(w, sc, Bits<T>::unpack(a3.z) & 0xffffu);
      T nF[9] = {a1.x, a1.y, a1.z, a1.w, a2.x, a2.y, a2.z, a2.w, a3.x}, J = a3.y;
      T* park = reinterpret_cast<T*>(pre + 128) + lane;
#pragma unroll
      for (int k = 0; k < 9; ++k) park[k * 32] = nF[k];
      park[9 * 32] = J;
      const bool fb = snow_return_parked<T>(&md, w.svd_fallback != 0, park);
      const T volatile* back = park;
#pragma unroll
      for (int k = 0; k < 9; ++k) nF[k] = back[k * 32];
      J = back[9 * 32];
      w.out[1][q.x] = mk4(nF[0], nF[1], nF[2], nF[3]);
      w.out[2][q.x] = mk4(nF[4], nF[5], nF[6], nF[7]);
      w.out[3][q.x] = mk4(nF[8], J, a3.z, a3.w);
      cp_async_wait_all();
      const V4 a0 = pre[lane], a4 = pre[32 + lane], a5 = pre[64 + lane], a6 = pre[96 + lane];
      const T C[9] = {a4.w, a5.x, a5.y, a5.z, a5.w, a6.x, a6.y, a6.z, a6.w};
      affine_from_c(sc, md, a0.w, C, nF, J, A);
      w.out[4][q.x] = mk4(a4.x, a4.y, a4.z, A[0]);
      w.out[5][q.x] = mk4(A[1], A[2], A[3], A[4]);
      w.out[6][q.x] = mk4(A[5], A[6], A[7], A[8]);
      if (fb) atomicAdd(w.err + 4 * q.y + 1, 1u);
      m = a0.w;
      xs[0] = a0.x, xs[1] = a0.y, xs[2] = a0.z;
      mv[0] = m * a4.x, mv[1] = m * a4.y, mv[2] = m * a4.z;
    }
    __syncwarp();  // prefetched data consumed: the scatter may reuse the region
    p2g_warp_scatter<T, true>(w, sc, valid, xs, m, mv, A, st, q.x, write_keys);
  }
}

// Drops a scatter that was queued for the next substep (the particle state it came from changed):
// zeroes the accumulator and the flags of the blocks on its touched list.
template <class T>
__global__ void discard_scatter_kernel(typename V4T<T>::type* acc, uint32_t* blk_flag, const uint32_t* list,
                                       const uint32_t* count) {
  const uint32_t n = launch_count(count);
  for (uint32_t t = blockIdx.x; t < n; t += gridDim.x) {
    const uint32_t gb = list[t];
    if (threadIdx.x < 64) acc[uint64_t(gb) * 64u + threadIdx.x] = mk4(T(0), T(0), T(0), T(0));
    if (threadIdx.x == 0) blk_flag[gb] = 0u;
  }
}

// dense grouping (bin_scan_kernel): nodes per scan CTA
constexpr int kBinSeg = 4096;
constexpr int kBinThreads = 256;

// ============================================================================================
// deterministic mode: per-cell fixed-order sums, per-node fixed-order gather
// ============================================================================================
__global__ void det_heads_kernel(const uint32_t* __restrict__ skeys, uint64_t n, const uint32_t* __restrict__ dead_flag,
                                 uint32_t* cell_slot, uint32_t* seg_start, uint32_t* cell_count) {
  uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t k = skeys[i];
  if (dead_flag[k >> 6]) return;  // spare blocks hold dead and off-grid particles
  if (i > 0 && skeys[i - 1] == k) return;
  uint32_t s = atomicAdd(cell_count, 1u);
  cell_slot[k] = s;
  seg_start[s] = uint32_t(i);
}

template <class T, int MODE>
__global__ void __launch_bounds__(128) det_cellsum_kernel(WorldDev<T> w, uint64_t n_sorted) {
  using V4 = typename V4T<T>::type;
  const uint32_t count = launch_count(w.cell_count);
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < count; s += gridDim.x * blockDim.x) {
    const uint32_t start = w.seg_start[s];
    const uint32_t key = w.sorted_keys[start];
    const SceneDev<T>& sc = w.scenes[w.blk_scene[key >> 6]];
    T acc[27][4];
#pragma unroll
    for (int o = 0; o < 27; ++o) acc[o][0] = acc[o][1] = acc[o][2] = acc[o][3] = T(0);
    int g0 = 0, g1 = 0, g2 = 0;
    for (uint64_t i = start; i < n_sorted && w.sorted_keys[i] == key; ++i) {
      P2GPart<T> p;
      p2g_setup<T, MODE>(w, sc, w.perm[i], p);
      g0 = p.g[0];
      g1 = p.g[1];
      g2 = p.g[2];
#pragma unroll
      for (int o = 0; o < 27; ++o) {
        T cm, cx, cy, cz;
        if (p2g_contrib<T, MODE>(sc, p, o % 3, (o / 3) % 3, o / 9, cm, cx, cy, cz)) {
          acc[o][0] += cm;
          acc[o][1] += cx;
          acc[o][2] += cy;
          acc[o][3] += cz;
        }
      }
    }
#pragma unroll
    for (int o = 0; o < 27; ++o) w.cell_rec[uint64_t(s) * 27 + o] = mk4(acc[o][0], acc[o][1], acc[o][2], acc[o][3]);
    for (int t = 0; t < 8; ++t) mark_stencil_corner(w, sc, t, g0, g1, g2);
  }
}

template <class T, int MODE>
__global__ void __launch_bounds__(256) det_gather_kernel(WorldDev<T> w, uint32_t* blk_epoch, const uint32_t* epoch) {
  using V4 = typename V4T<T>::type;
  const uint32_t count = launch_count(w.touched_count);
  const uint32_t ep = *epoch;
  if (blockIdx.x == 0 && threadIdx.x == 0) *w.clamp_count = 0u;
  const int sub = threadIdx.x >> 6, l = threadIdx.x & 63;
  for (uint32_t t = blockIdx.x * 4 + sub; t < count; t += gridDim.x * 4) {
    const uint32_t gb = w.touched[t];
    const SceneDev<T>& sc = w.scenes[w.blk_scene[gb]];
    int i, j, k;
    block_coords(sc, gb, l, i, j, k);
    T m = 0, px = 0, py = 0, pz = 0;
    if (i < sc.n[0] && j < sc.n[1] && k < sc.n[2]) {
      // node (i,j,k) receives offset (a,b,c) of the cell based at (i-a, j-b, k-c), in fixed order
#pragma unroll 1
      for (int o = 0; o < 27; ++o) {
        const int a = o % 3, b = (o / 3) % 3, c = o / 9;
        int X = i - a, Y = j - b, Z = k - c;
        if (X < 0 || Y < 0 || Z < 0) continue;
        const uint32_t ck = node_index(sc, X, Y, Z);
        uint32_t s;
        if (w.cells) {
          const uint2 cell = w.cells[ck];
          if (cell.y == 0u) continue;
          s = cell.x + w.seg_off[ck / kBinSeg];
        } else {
          s = w.cell_slot[ck];
          if (s == 0xffffffffu) continue;
        }
        V4 r = w.cell_rec[uint64_t(s) * 27 + o];
        m += r.x;
        px += r.y;
        py += r.z;
        pz += r.w;
      }
    }
    T vx, vy, vz;
    grid_velocity<T, MODE>(sc, i, j, k, m, px, py, pz, vx, vy, vz);
    w.vel[uint64_t(gb) * 64u + l] = mk4(vx, vy, vz, m);
    if (l == 0) {
      w.blk_flag[gb] = 0u;
      blk_epoch[gb] = ep;
    }
  }
}

// ---- deterministic sums with dense grouping ----
// After the grouping a cell's particles stand together but in no defined order.  The warp whose 32
// sorted places hold a cell's first place puts them in slot order (as the stable radix sort does),
// writes the final order and adds them up in it: lanes 0..26 are the 27 stencil nodes, every lane
// adds its node's contributions particle by particle.  One thread per cell with 108 accumulators
// (det_cellsum_kernel) left the chip to a few spilling warps: 211 us for 1 M particles at 8 per cell.
//
// Slot order: up to 32 particles rank each other by shuffles, up to kCellRankMax by comparing with
// the whole cell; a larger cell is radix-sorted by its warp, at a cost per particle below that of the sum
// that follows, which one warp walks too.  The off-grid particles of the reference modes come in slot order
// from their placement (bin_scatter_kernel).  1 M particles, one cell of 500 / 600 / 5 000: 372 / 13 800 /
// 14 300 us a substep while cells above 512 were collected in a walk over the scene's keys, 302 / 301 / 843
// now (2 360 / 16 700 with one thread per cell over radix-sorted particles).  The line: 1 000 cells of 200
// take 352 us ranked and 331 sorted, 2 000 cells of 64 the same either way.
constexpr uint32_t kCellRankMax = 128;

// Sorts the k slots at run into out by one warp: 8 bits of slot - base per pass, each pass counted, scanned
// and placed 32 slots at a time in input order.  tmp: k entries, hist: 256 counters of the warp's own.
// out and tmp take the passes in turn so that the last one ends in out; run is only read.
__device__ __noinline__ void warp_sort_slots(const uint32_t* run, uint32_t* out, uint32_t* tmp, uint32_t k,
                                                uint32_t base, uint32_t slots, uint32_t* hist, int lane) {
  const int passes = slots > 1u ? (39 - __clz(slots - 1u)) / 8 : 1;
  const uint32_t* src = run;
  constexpr uint32_t kAhead = 4;  // loads in flight per lane
  for (int p = 0; p < passes; ++p) {
    uint32_t* dst = ((passes - 1 - p) & 1) ? tmp : out;
    const int shift = 8 * p;
    __syncwarp();
    for (int q = 0; q < 8; ++q) hist[q * 32 + lane] = 0u;
    __syncwarp();
    for (uint32_t b0 = 0; b0 < k; b0 += 32 * kAhead) {
      uint32_t v[kAhead];
#pragma unroll
      for (uint32_t q = 0; q < kAhead; ++q) {
        const uint32_t i = b0 + 32 * q + lane;
        v[q] = i < k ? src[i] : 0u;
      }
#pragma unroll
      for (uint32_t q = 0; q < kAhead; ++q)
        if (b0 + 32 * q + lane < k) atomicAdd(hist + ((v[q] - base) >> shift & 255u), 1u);
    }
    __syncwarp();
    uint32_t c[8], sum = 0;
    for (int q = 0; q < 8; ++q) {
      c[q] = sum;
      sum += hist[lane * 8 + q];
    }
    const uint32_t before = warp_scan_incl(sum, lane) - sum;
    for (int q = 0; q < 8; ++q) hist[lane * 8 + q] = before + c[q];
    __syncwarp();
    for (uint32_t b0 = 0; b0 < k; b0 += 32 * kAhead) {
      uint32_t v[kAhead];
#pragma unroll
      for (uint32_t q = 0; q < kAhead; ++q) {
        const uint32_t i = b0 + 32 * q + lane;
        v[q] = i < k ? src[i] : 0u;
      }
#pragma unroll
      for (uint32_t q = 0; q < kAhead; ++q) {
        const bool in = b0 + 32 * q + lane < k;
        const uint32_t d = in ? (v[q] - base) >> shift & 255u : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t at = in ? hist[d] + uint32_t(__popc(peers & ((1u << lane) - 1u))) : 0u;
        __syncwarp();
        if (in) {
          if (lane == __ffs(peers) - 1) hist[d] += uint32_t(__popc(peers));
          dst[at] = v[q];
        }
        __syncwarp();
      }
    }
    src = dst;
  }
  __syncwarp();
}

// Physics mode stages what the column-lane scatter stages: per (y,z) column u = m v + A d and w_y w_z,
// the x weights with the mass, dx times A's x column (3 shared loads per particle and node; weights,
// offsets and A's rows staged as they are took 7, and the kernel was bound by shared memory: 95 us
// against 88 for 1 M particles).
template <class T, int MODE>
struct CellStage {
  P2GPart<T> p[32];
};
template <class T>
struct CellStage<T, AE_MPM_MODE_PHYSICS> {
  using V4 = typename V4T<T>::type;
  V4 col[32 * 9], wxm[32], acol[32];
  int4 g[32];
};

template <class T>
__device__ __forceinline__ void cell_stage_put(CellStage<T, AE_MPM_MODE_PHYSICS>& st, const SceneDev<T>& sc, int i,
                                               const P2GPart<T>& p) {
  const T dx = sc.dx;
  T c0[3], c1[3], c2[3], qv[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    c0[r] = dx * p.A[3 * r + 0];
    c1[r] = dx * p.A[3 * r + 1];
    c2[r] = dx * p.A[3 * r + 2];
    qv[r] = p.v[r] - (c0[r] * p.fx[0] + c1[r] * p.fx[1] + c2[r] * p.fx[2]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      st.col[i * 9 + b + 3 * c] = mk4(qv[0] + T(b) * c1[0] + T(c) * c2[0], qv[1] + T(b) * c1[1] + T(c) * c2[1],
                                      qv[2] + T(b) * c1[2] + T(c) * c2[2], p.w[1][b] * p.w[2][c]);
  st.wxm[i] = mk4(p.w[0][0], p.w[0][1], p.w[0][2], p.m);
  st.acol[i] = mk4(c0[0], c0[1], c0[2], T(0));
  st.g[i] = make_int4(p.g[0], p.g[1], p.g[2], 0);
}
template <class T, int MODE>
__device__ __forceinline__ void cell_stage_put(CellStage<T, MODE>& st, const SceneDev<T>&, int i, const P2GPart<T>& p) {
  st.p[i] = p;
}
// adds staged particle i's contribution to the node at offset (a, b, c); `inside`: every staged
// stencil lies in the grid
template <class T>
__device__ __forceinline__ void cell_add(const CellStage<T, AE_MPM_MODE_PHYSICS>& st, const SceneDev<T>& sc, int i,
                                         int a, int b, int c, bool inside, T& am, T& ax, T& ay, T& az) {
  if (!inside) {
    const int4 g = st.g[i];
    const int X = g.x + a, Y = g.y + b, Z = g.z + c;
    if (X < 0 || Y < 0 || Z < 0 || X >= sc.n[0] || Y >= sc.n[1] || Z >= sc.n[2]) return;
  }
  const auto u = st.col[i * 9 + b + 3 * c], r = st.wxm[i], s = st.acol[i];
  const T fa = T(a), ww = (a == 0 ? r.x : (a == 1 ? r.y : r.z)) * u.w;
  am += ww * r.w;
  ax += ww * (u.x + fa * s.x);
  ay += ww * (u.y + fa * s.y);
  az += ww * (u.z + fa * s.z);
}
template <class T, int MODE>
__device__ __forceinline__ void cell_add(const CellStage<T, MODE>& st, const SceneDev<T>& sc, int i, int a, int b, int c,
                                         bool, T& am, T& ax, T& ay, T& az) {
  T cm, cx, cy, cz;
  if (!p2g_contrib<T, MODE>(sc, st.p[i], a, b, c, cm, cx, cy, cz)) return;
  am += cm;
  ax += cx;
  ay += cy;
  az += cz;
}

template <class T, int MODE>
__global__ void __launch_bounds__(256) det_cells_kernel(WorldDev<T> w, const uint32_t* __restrict__ grouped,
                                                        uint32_t* __restrict__ ordered) {
  using V4 = typename V4T<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  auto& st = reinterpret_cast<CellStage<T, MODE>*>(smem)[threadIdx.x >> 5];
  static_assert(sizeof(st) >= 256 * sizeof(uint32_t), "warp_sort_slots counts in the staging");
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const int lane = threadIdx.x & 31;
  const uint32_t pos = uint32_t(ch.y) + threadIdx.x;
  bool live = int(pos) < ch.z;
  const uint32_t mine = live ? grouped[pos] : 0u;
  const uint32_t key = live ? w.keys[mine] : 0u;
  if (MODE != AE_MPM_MODE_PHYSICS && live && key == sc.dead_key) {  // off the grid: in order, not summed
    ordered[pos] = mine;
    live = false;
  }
  uint32_t first = 0xffffffffu, cnt = 0;
  if (live) {
    const uint2 cell = w.cells[key];
    first = cell.x + w.seg_off[key / kBinSeg];
    cnt = cell.y;
  }
  const int na = lane % 3, nb = (lane / 3) % 3, nc = min(lane / 9, 2);
  T am, ax, ay, az;
  auto add_staged = [&](int i0, int i1, bool inside) {  // staged particles in order, this lane's node
    for (int i = i0; i < i1; ++i) cell_add(st, sc, i, na, nb, nc, inside, am, ax, ay, az);
  };
  auto finish = [&](uint32_t start, int g0, int g1, int g2) {
    if (lane < 27) w.cell_rec[uint64_t(start) * 27 + lane] = mk4(am, ax, ay, az);
    if (lane < 8) mark_stencil_corner(w, sc, lane, g0, g1, g2);
  };
  auto inside_grid = [&](const P2GPart<T>& p) {
    return p.g[0] >= 0 && p.g[1] >= 0 && p.g[2] >= 0 && p.g[0] + 2 < sc.n[0] && p.g[1] + 2 < sc.n[1] &&
           p.g[2] + 2 < sc.n[2];
  };
  uint32_t heads = __ballot_sync(0xffffffffu, live && first == pos);
  const uint32_t base = pos - lane;

  // cells that lie in the warp's 32 places: ordered and staged together, one particle per lane
  const bool batch = live && first >= base && first + cnt <= base + 32u;
  const uint32_t in_batch = __ballot_sync(0xffffffffu, batch);
  if (in_batch) {
    const uint32_t most = __reduce_max_sync(0xffffffffu, batch ? cnt : 0u);
    const int l0 = batch ? int(first - base) : 0;
    uint32_t rank = 0;
    for (uint32_t t = 0; t < most; ++t) {
      const uint32_t other = __shfl_sync(0xffffffffu, mine, (l0 + int(t)) & 31);
      if (t < cnt && other < mine) ++rank;
    }
    P2GPart<T> p;
    p.g[0] = p.g[1] = p.g[2] = 0;
    bool in = true;
    if (batch) {
      ordered[first + rank] = mine;
      p2g_setup<T, MODE>(w, sc, mine, p);
      cell_stage_put(st, sc, l0 + int(rank), p);
      in = inside_grid(p);
    }
    const bool inside = __all_sync(0xffffffffu, in);
    __syncwarp();
    for (uint32_t todo = heads & in_batch; todo; todo &= todo - 1u) {
      const int h = __ffs(todo) - 1;
      const int k = int(__shfl_sync(0xffffffffu, cnt, h));
      am = ax = ay = az = T(0);
      add_staged(h, h + k, inside);
      finish(base + uint32_t(h), __shfl_sync(0xffffffffu, p.g[0], h), __shfl_sync(0xffffffffu, p.g[1], h),
             __shfl_sync(0xffffffffu, p.g[2], h));
    }
    heads &= ~in_batch;
    __syncwarp();
  }

  // the others one by one: the cell that runs past the places, or cells of more than 32 particles
  while (heads) {
    const int h = __ffs(heads) - 1;
    heads &= heads - 1u;
    const uint32_t start = __shfl_sync(0xffffffffu, first, h), k = __shfl_sync(0xffffffffu, cnt, h);
    const uint32_t* run = grouped + start;
    uint32_t* out = ordered + start;
    uint32_t slot = 0, rank = 0;
    if (k <= 32u) {
      slot = uint32_t(lane) < k ? run[lane] : 0xffffffffu;
      for (uint32_t i = 0; i < k; ++i) rank += __shfl_sync(0xffffffffu, slot, int(i)) < slot ? 1u : 0u;
      if (uint32_t(lane) < k) out[rank] = slot;
    } else if (k <= kCellRankMax) {
      for (uint32_t b0 = 0; b0 < k; b0 += 32) {
        const uint32_t s = b0 + lane < k ? run[b0 + lane] : 0xffffffffu;
        uint32_t r = 0;
        for (uint32_t i = 0; i < k; ++i) r += run[i] < s ? 1u : 0u;
        if (s != 0xffffffffu) out[r] = s;
      }
    } else {
      // the clamp queue is empty until this substep's G2P
      warp_sort_slots(run, out, reinterpret_cast<uint32_t*>(w.clamp_queue) + start, k, sc.p_off, sc.p_cap,
                      reinterpret_cast<uint32_t*>(&st), lane);
    }
    __syncwarp();
    am = ax = ay = az = T(0);
    int g0 = 0, g1 = 0, g2 = 0;
    for (uint32_t b0 = 0; b0 < k; b0 += 32) {
      const uint32_t n = min(32u, k - b0);
      bool in = true;
      if (uint32_t(lane) < n) {
        P2GPart<T> p;
        if (k > 32u) {
          slot = out[b0 + lane];
          rank = uint32_t(lane);
        }
        p2g_setup<T, MODE>(w, sc, slot, p);
        cell_stage_put(st, sc, int(rank), p);
        g0 = p.g[0], g1 = p.g[1], g2 = p.g[2];
        in = inside_grid(p);
      }
      const bool inside = __all_sync(0xffffffffu, in);
      __syncwarp();
      add_staged(0, int(n), inside);
      __syncwarp();
    }
    finish(start, __shfl_sync(0xffffffffu, g0, 0), __shfl_sync(0xffffffffu, g1, 0), __shfl_sync(0xffffffffu, g2, 0));
  }
}

__global__ void det_reset_kernel(const uint32_t* __restrict__ seg_start, const uint32_t* __restrict__ skeys,
                                 const uint32_t* cell_count, uint32_t* cell_slot) {
  const uint32_t count = launch_count(cell_count);
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < count; s += gridDim.x * blockDim.x)
    cell_slot[skeys[seg_start[s]]] = 0xffffffffu;
}

// ============================================================================================
// keys, pack/unpack, totals, grid export
// ============================================================================================
// Cell keys of the current positions; with dense grouping also the live particles per cell (one
// atomic per cell and warp), and no keys for the dead slots, which that grouping never reads.
template <class T, int MODE>
__global__ void init_keys_kernel(WorldDev<T> w) {
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const int j = ch.y + threadIdx.x;
  const bool live = j < ch.z;
  uint32_t key = sc.dead_key;
  if (live) {
    auto a0 = ld4(w.in[0] + j);
    key = cell_key(sc, MODE, a0.x, a0.y, a0.z);
  }
  if (!w.bins) {
    if (j < ch.w) w.keys[j] = key;
    return;
  }
  const uint32_t peers = __match_any_sync(0xffffffffu, live ? key : 0xffffffffu);
  if (live) {
    w.keys[j] = key;
    if (int(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(w.bins + key, uint32_t(__popc(peers)));
  }
  if (MODE != AE_MPM_MODE_PHYSICS && w.dead_cnt) {
    const int c = __syncthreads_count(live && key == sc.dead_key);
    if (threadIdx.x == 0) w.dead_cnt[blockIdx.x] = uint32_t(c);
  }
}

// ============================================================================================
// dense grouping: particles in ascending cell order through one counter per grid node
// ============================================================================================
// The kernels that write the keys count the live particles of every cell (w.bins).  bin_scan turns
// the counts into offsets and bin_scatter claims a place per particle with them: two launches and
// 12 bytes per node + 12 per particle, where the radix sort takes 3 launches and 20 bytes per key
// for each 8 bits of key.  Equal keys land in no defined order, so only the modes whose results do
// not depend on it (anything but deterministic) use it.  Sorted places of a scene are its slot
// range: the dead key's cell holds the off-grid particles of the reference modes first and then,
// without entries, the scene's empty slots.
//
// One CTA scans 4096 nodes (64 blocks) and zeroes the counts it read, so the array is clean for
// the next count; offsets are written only where a count is not zero.  The CTA that finishes last
// scans the segment totals (no CTA waits for another).

template <class T>
__device__ __forceinline__ void bin_scan(const WorldDev<T>& w, uint64_t nodes, const uint32_t* __restrict__ dead_blk,
                                         uint32_t* seg_total, uint32_t* done, uint32_t cta, uint32_t ctas) {
  __shared__ uint32_t wsum[kBinThreads / 32];
  __shared__ uint32_t s_last, s_carry;
  const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5;
  const uint64_t base = uint64_t(cta) * kBinSeg + uint64_t(wi) * 512u;
  uint4* bins4 = reinterpret_cast<uint4*>(w.bins);
  uint4* off4 = reinterpret_cast<uint4*>(w.bin_off);
  uint4 c[4];
  uint32_t pad[4], any[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint64_t i = base + r * 128 + lane * 4;
    c[r] = make_uint4(0u, 0u, 0u, 0u);
    pad[r] = 0u;
    if (i < nodes) {
      c[r] = bins4[i >> 2];
      if ((i & 63u) == 0 && dead_blk[i >> 6]) {  // the scene's empty slots follow the dead key's particles
        const SceneDev<T>& sc = w.scenes[w.blk_scene[i >> 6]];
        pad[r] = sc.p_cap - sc.p_count;
      }
    }
  }
  uint32_t ex[4], run = 0;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    any[r] = c[r].x | c[r].y | c[r].z | c[r].w;
    const uint32_t t = c[r].x + c[r].y + c[r].z + c[r].w + pad[r];
    const uint32_t incl = warp_scan_incl(t, lane);
    ex[r] = run + incl - t;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) wsum[wi] = run;
  __syncthreads();
  uint32_t off = 0, total = 0;
#pragma unroll
  for (int k = 0; k < kBinThreads / 32; ++k) {
    const uint32_t v = wsum[k];
    if (k < wi) off += v;
    total += v;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint64_t i = base + r * 128 + lane * 4, q = i >> 2;
    uint4 o;
    o.x = off + ex[r];
    o.y = o.x + c[r].x + pad[r];
    o.z = o.y + c[r].y;
    o.w = o.z + c[r].z;
    if (any[r]) {
      off4[q] = o;
      bins4[q] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (w.cells && i < nodes) {  // occupied now, or at the last sort
      uint4* cq = reinterpret_cast<uint4*>(w.cells) + (i >> 1);
      const uint4 a = cq[0], b = cq[1];
      if (any[r] | a.y | a.w | b.y | b.w) {
        cq[0] = make_uint4(o.x, c[r].x, o.y, c[r].y);
        cq[1] = make_uint4(o.z, c[r].z, o.w, c[r].w);
      }
    }
  }
  if (tid == 0) {
    seg_total[cta] = total;
    __threadfence();
    s_last = atomicAdd(done, 1u) == ctas - 1 ? 1u : 0u;
    s_carry = 0u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (uint32_t s0 = 0; s0 < ctas; s0 += kBinThreads * 4) {
    uint32_t v[4], t = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t i = s0 + tid * 4 + k;
      v[k] = i < ctas ? __ldcg(seg_total + i) : 0u;
      t += v[k];
    }
    const uint32_t incl = warp_scan_incl(t, lane);
    __syncthreads();  // the previous round's wsum and carry have been read
    if (lane == 31) wsum[wi] = incl;
    __syncthreads();
    uint32_t o = s_carry + incl - t, sum = 0;
#pragma unroll
    for (int k = 0; k < kBinThreads / 32; ++k) {
      if (k < wi) o += wsum[k];
      sum += wsum[k];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t i = s0 + tid * 4 + k;
      if (i < ctas) w.seg_off[i] = o;
      o += v[k];
    }
    __syncthreads();
    if (tid == 0) s_carry += sum;
  }
  if (tid == 0) *done = 0u;
}

template <class T>
__global__ void __launch_bounds__(kBinThreads) bin_scan_kernel(WorldDev<T> w, uint64_t nodes,
                                                               const uint32_t* __restrict__ dead_blk,
                                                               uint32_t* seg_total, uint32_t* done) {
  bin_scan(w, nodes, dead_blk, seg_total, done, blockIdx.x, gridDim.x);
}

// The scan of the next order and the grid update read nothing of each other: one launch, the first
// `scan_ctas` CTAs scan.  Small worlds are bound by the number of dependent launches (2 300
// particles on a 32^3 grid: 20.2 us a substep with four launches).
template <class T>
__global__ void __launch_bounds__(kBinThreads) scan_and_grid_kernel(WorldDev<T> w, uint64_t nodes,
                                                                    const uint32_t* __restrict__ dead_blk,
                                                                    uint32_t* seg_total, uint32_t* done,
                                                                    uint32_t scan_ctas, uint32_t* blk_epoch,
                                                                    const uint32_t* epoch, uint32_t* zero_count) {
  let_next_start();
  dependency_wait();
  if (blockIdx.x < scan_ctas)
    bin_scan(w, nodes, dead_blk, seg_total, done, blockIdx.x, scan_ctas);
  else
    grid_update<T, AE_MPM_MODE_PHYSICS>(w, blk_epoch, epoch, zero_count, blockIdx.x - scan_ctas, gridDim.x - scan_ctas);
}

// kOff: the deterministic reference modes, whose particles off the grid, any number of them on one key,
// are placed in slot order: after those of the scene's earlier chunks, in order within their own.
template <class T, bool kOff>
__global__ void __launch_bounds__(256) bin_scatter_kernel(WorldDev<T> w, uint32_t* __restrict__ perm,
                                                          uint32_t n_slots) {
  let_next_start();
  const int4 ch = cta_chunk(w);
  dependency_wait();
  const int j = ch.y + threadIdx.x, lane = threadIdx.x & 31;
  const bool live = j < ch.z;
  const uint32_t key = live ? w.keys[j] : 0xffffffffu;
  const bool count_off = kOff && w.dead_cnt[blockIdx.x] != 0u;  // uniform over the CTA
  bool off = false;
  uint32_t pos = 0;
  if (count_off) {
    __shared__ uint32_t warp_off[8], earlier;
    const SceneDev<T>& sc = w.scenes[ch.x];
    off = key == sc.dead_key;
    if (threadIdx.x == 0) earlier = 0u;
    const uint32_t mask = __ballot_sync(0xffffffffu, off);
    if (lane == 0) warp_off[threadIdx.x >> 5] = uint32_t(__popc(mask));
    uint32_t sum = 0;
    for (uint32_t c = blockIdx.x - (uint32_t(ch.y) - sc.p_off) / blockDim.x + threadIdx.x; c < blockIdx.x; c += blockDim.x)
      sum += w.dead_cnt[c];
    sum = __reduce_add_sync(0xffffffffu, sum);
    __syncthreads();
    if (lane == 0 && sum) atomicAdd(&earlier, sum);
    __syncthreads();
    pos = earlier + uint32_t(__popc(mask & ((1u << lane) - 1u)));
    for (uint32_t k = 0; k < (threadIdx.x >> 5); ++k) pos += warp_off[k];
    if (off) pos += w.bin_off[key] + w.seg_off[key / kBinSeg];
  }
  const uint32_t peers = __match_any_sync(0xffffffffu, key);
  const int leader = __ffs(peers) - 1;
  uint32_t at = 0;
  if (live && !off && lane == leader) at = atomicAdd(w.bin_off + key, uint32_t(__popc(peers))) + w.seg_off[key / kBinSeg];
  at = __shfl_sync(0xffffffffu, at, leader) + __popc(peers & ((1u << lane) - 1u));
  if (!off) pos = at;
  if (live && pos < n_slots) perm[pos] = uint32_t(j);
}

// One scene's particles in the caller's layout: arrays of the caller on this device, or a staging
// area (pos 3n | vel 3n | F 9n | J n | C 9n | mass n, then n u16 material indices).
template <class T>
struct XferDev {
  T* f[6];  // pos, vel, F, J, C, mass
  uint16_t* mat;
  uint32_t n, pad;
};
// The scenes of one transfer: a single one by value, or a table over the scenes s0, s0 + 1, ... (n = 0
// for scenes that do not take part).
template <class T>
struct XferSet {
  const XferDev<T>* tab;
  uint32_t s0;
  XferDev<T> one;
  __device__ __forceinline__ XferDev<T> of(uint32_t s) const { return tab ? tab[s - s0] : one; }
};

// Caller's layout -> slots, one launch for all scenes of a transfer (a launch per scene, 4.6 us each
// for 19 000 particles, took 2.4 ms for 512 scenes against 0.4 together).  Bound by memory: 106 bytes
// read and 112 written per particle run at the copy rate.  kMotion: position, velocity and mass only.
template <class T, bool kMotion>
__global__ void __launch_bounds__(256) pack_kernel(WorldDev<T> w, XferSet<T> xs) {
  using V4 = typename V4T<T>::type;
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const XferDev<T> d = xs.of(uint32_t(ch.x));
  const uint32_t s = uint32_t(ch.y) + threadIdx.x;
  const uint64_t i = s - sc.p_off;
  if (i >= d.n) return;
  V4* const* dst = const_cast<V4* const*>(w.in);
  const T *pos = d.f[0], *vel = d.f[1], *F = d.f[2], *C = d.f[4];
  const T J = kMotion ? T(1) : d.f[3][i], m = d.f[5][i];
  const uint32_t mi = kMotion ? 0u : d.mat[i];
  T f[9], c[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    f[k] = kMotion ? T(k % 4 == 0 ? 1 : 0) : F[9 * i + k];
    c[k] = kMotion ? T(0) : C[9 * i + k];
  }
  dst[0][s] = mk4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], m);
  dst[1][s] = mk4(f[0], f[1], f[2], f[3]);
  dst[2][s] = mk4(f[4], f[5], f[6], f[7]);
  dst[3][s] = mk4(f[8], J, Bits<T>::pack(mi), Bits<T>::pack(uint32_t(i)));
  if (!kMotion && sc.mode == AE_MPM_MODE_PHYSICS) {  // the C slot holds A = m C - k tau on the device
    const MatDev& md = w.mats[sc.mat_off + (mi < sc.n_mat ? mi : sc.n_mat)];
    T a[9];
    affine_from_c(sc, md, m, c, f, J, a);
#pragma unroll
    for (int k = 0; k < 9; ++k) c[k] = a[k];
  }
  dst[4][s] = mk4(vel[3 * i], vel[3 * i + 1], vel[3 * i + 2], c[0]);
  dst[5][s] = mk4(c[1], c[2], c[3], c[4]);
  dst[6][s] = mk4(c[5], c[6], c[7], c[8]);
}

// Slots -> caller's layout in two launches: the slot of each original index (inv), then a gather
// that writes every array in order.  Scattering from the slots instead (one launch) sends each
// particle's 12- and 36-byte rows to lines of their own: 3.46 ms for 8.4 M particles whose order is
// not the caller's, 0.14 for 1 M that nearly kept it.
template <class T>
__global__ void __launch_bounds__(256) unpack_index_kernel(WorldDev<T> w, XferSet<T> xs, uint32_t* __restrict__ inv) {
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const uint32_t n = xs.of(uint32_t(ch.x)).n;
  const uint32_t s = uint32_t(ch.y) + threadIdx.x;
  if (s - sc.p_off >= n) return;
  const uint32_t o = Bits<T>::unpack(w.in[3][s].w);
  if (o < n) inv[sc.p_off + o] = s;
}

// rows of K values per lane -> K consecutive values per particle at dst[i0 * K], through the warp's
// shared row buffer, so that each store instruction writes consecutive values
template <int K, class T>
__device__ __forceinline__ void store_rows(T* dst, uint64_t i0, uint64_t n, const T* v, T* buf, bool has, int lane) {
  if (has) {
#pragma unroll
    for (int k = 0; k < K; ++k) buf[lane * K + k] = v[k];
  }
  __syncwarp();
  const uint64_t end = n * K;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint64_t q = i0 * K + uint64_t(k * 32 + lane);
    if (q < end) dst[q] = buf[k * 32 + lane];
  }
  __syncwarp();
}

template <class T, bool kMotion>
__global__ void __launch_bounds__(256) unpack_kernel(WorldDev<T> w, XferSet<T> xs, const uint32_t* __restrict__ inv) {
  using V4 = typename V4T<T>::type;
  __shared__ T rows[8][32 * 9];
  const int4 ch = cta_chunk(w);
  const SceneDev<T>& sc = w.scenes[ch.x];
  const XferDev<T> d = xs.of(uint32_t(ch.x));
  const int lane = threadIdx.x & 31;
  T* buf = rows[threadIdx.x >> 5];
  const uint64_t i = uint32_t(ch.y) + threadIdx.x - sc.p_off, i0 = i - lane;
  if (i0 >= d.n) return;  // warp-uniform
  bool has = i < d.n;
  uint32_t s = 0;
  if (has) {
    s = inv[sc.p_off + i];
    has = s - sc.p_off < d.n;
  }
  if constexpr (kMotion) {
    T x[3], v[3];
    if (has) {
      const V4 a0 = ld4(w.in[0] + s), a4 = ld4(w.in[4] + s);
      x[0] = a0.x, x[1] = a0.y, x[2] = a0.z;
      v[0] = a4.x, v[1] = a4.y, v[2] = a4.z;
    }
    store_rows<3>(d.f[0], i0, d.n, x, buf, has, lane);
    store_rows<3>(d.f[1], i0, d.n, v, buf, has, lane);
    return;
  }
  T f[9], c[9], x[3], v[3], J = T(0), m = T(0);
  uint32_t mi = 0;
  if (has) {
    const V4 a0 = ld4(w.in[0] + s), a1 = ld4(w.in[1] + s), a2 = ld4(w.in[2] + s), a3 = ld4(w.in[3] + s);
    const V4 a4 = ld4(w.in[4] + s), a5 = ld4(w.in[5] + s), a6 = ld4(w.in[6] + s);
    x[0] = a0.x, x[1] = a0.y, x[2] = a0.z, m = a0.w;
    v[0] = a4.x, v[1] = a4.y, v[2] = a4.z;
    J = a3.y;
    mi = Bits<T>::unpack(a3.z) & 0xffffu;
    f[0] = a1.x, f[1] = a1.y, f[2] = a1.z, f[3] = a1.w, f[4] = a2.x, f[5] = a2.y, f[6] = a2.z, f[7] = a2.w, f[8] = a3.x;
    c[0] = a4.w, c[1] = a5.x, c[2] = a5.y, c[3] = a5.z, c[4] = a5.w, c[5] = a6.x, c[6] = a6.y, c[7] = a6.z, c[8] = a6.w;
    if (sc.mode == AE_MPM_MODE_PHYSICS) {  // C = (A + k tau) / m
      const MatDev& md = w.mats[sc.mat_off + (mi < sc.n_mat ? mi : sc.n_mat)];
      T tau[9];
      phys_tau(md, f, J, tau);
      const T k = affine_k(sc, md, m);
#pragma unroll
      for (int q = 0; q < 9; ++q) c[q] = (c[q] + k * tau[q]) / m;
    }
    d.f[3][i] = J;
    d.f[5][i] = m;
    d.mat[i] = uint16_t(mi);
  }
  store_rows<3>(d.f[0], i0, d.n, x, buf, has, lane);
  store_rows<3>(d.f[1], i0, d.n, v, buf, has, lane);
  store_rows<9>(d.f[2], i0, d.n, f, buf, has, lane);
  store_rows<9>(d.f[4], i0, d.n, c, buf, has, lane);
}

// per-chunk FP64 partial sums [mass, px, py, pz, ke]; fixed reduction order (deterministic)
template <class T>
__global__ void __launch_bounds__(256) totals_kernel(WorldDev<T> w, double* partial) {
  __shared__ double sm[8][5];
  const int4 ch = cta_chunk(w);
  const int j = ch.y + threadIdx.x;
  double v[5] = {0, 0, 0, 0, 0};
  if (j < ch.z) {
    auto a0 = ld4(w.in[0] + j);
    auto a4 = ld4(w.in[4] + j);
    double m = double(a0.w), vx = double(a4.x), vy = double(a4.y), vz = double(a4.z);
    v[0] = m;
    v[1] = m * vx;
    v[2] = m * vy;
    v[3] = m * vz;
    v[4] = 0.5 * m * (vx * vx + vy * vy + vz * vz);
  }
#pragma unroll
  for (int k = 0; k < 5; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  if (lane == 0)
    for (int k = 0; k < 5; ++k) sm[wi][k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = (blockDim.x + 31) / 32;
    for (int k = 0; k < 5; ++k) {
      double s = 0;
      for (int q = 0; q < nw; ++q) s += sm[q][k];
      partial[uint64_t(blockIdx.x) * 5 + k] = s;
    }
  }
}

// dense reference-order grid export of scene 0's last substep (mass, velocity)
template <class T>
__global__ void grid_export_kernel(const typename V4T<T>::type* vel, const SceneDev<T>* scp, const uint32_t* blk_epoch,
                                   const uint32_t* epoch, float* mass_out, float* vel_out) {
  const SceneDev<T>& sc = *scp;
  uint64_t idx = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  uint64_t nn = uint64_t(sc.n[0]) * sc.n[1] * sc.n[2];
  if (idx >= nn) return;
  int i = int(idx % sc.n[0]), j = int((idx / sc.n[0]) % sc.n[1]), k = int(idx / (uint64_t(sc.n[0]) * sc.n[1]));
  uint32_t gi = node_index(sc, i, j, k);
  bool fresh = blk_epoch[gi >> 6] + 1u == *epoch;
  auto v = vel[gi];
  mass_out[idx] = fresh ? float(v.w) : 0.0f;
  vel_out[3 * idx] = fresh ? float(v.x) : 0.0f;
  vel_out[3 * idx + 1] = fresh ? float(v.y) : 0.0f;
  vel_out[3 * idx + 2] = fresh ? float(v.z) : 0.0f;
}

// ============================================================================================
// host side
// ============================================================================================
int device_sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (!cached[dev]) {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    cached[dev] = v > 0 ? v : 148;
  }
  return cached[dev];
}

static MatDev mat_dev(const ae_mpm_material& m, int model) {
  MatDev d{};
  float nu = std::min(std::max(m.poisson_ratio, -0.999f), 0.4999f);
  d.model = model;
  d.lambda = m.young_modulus * nu / ((1.0f + nu) * (1.0f - 2.0f * nu));
  d.mu = m.young_modulus / (2.0f * (1.0f + nu));
  d.bulk = m.young_modulus / (3.0f * (1.0f - 2.0f * nu));
  if (model >= kPhysJelly && m.bulk_modulus > 0.0f) d.bulk = m.bulk_modulus;
  d.rho = m.density;
  d.yield_stress = m.yield_stress;
  d.friction_angle = m.friction_angle;
  d.cohesion = m.cohesion;
  d.theta_c = m.theta_c;
  d.theta_s = m.theta_s;
  d.xi = m.hardening_xi;
  return d;
}

static uint64_t blocks_of(const ae_mpm_scene_desc& d) {
  return uint64_t((d.n[0] + 3) / 4) * ((d.n[1] + 3) / 4) * ((d.n[2] + 3) / 4) + 1;  // + spare block
}

#define AE_TRY(call)                                                                           \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) {                                                                   \
      err = std::string(#call) + ": " + cudaGetErrorString(e_);                                \
      cudaGetLastError(); /* reported here: the next call's check must not find it again */    \
      return (e_ == cudaErrorMemoryAllocation) ? AE_MPM_ENOMEM : AE_MPM_ECUDA;                 \
    }                                                                                          \
  } while (0)

// the caller's arrays, from an ae_mpm_particles (f32) or ae_mpm_particles_f64 (f64) view
template <class T>
struct HostView {
  T* f[6];  // pos, vel, strain, jacobian, c, mass
  uint16_t* mat;
};
template <class T>
HostView<T> host_view(const void* host);
template <>
HostView<float> host_view<float>(const void* host) {
  const auto* h = static_cast<const ae_mpm_particles*>(host);
  return HostView<float>{{h->pos, h->vel, h->strain, h->jacobian, h->c, h->mass}, h->material_idx};
}
template <>
HostView<double> host_view<double>(const void* host) {
  const auto* h = static_cast<const ae_mpm_particles_f64*>(host);
  return HostView<double>{{h->pos, h->vel, h->strain, h->jacobian, h->c, h->mass}, h->material_idx};
}

// Whether two arrays of k views share memory.  Results copied out of a staging area one after another
// leave the later one there; kernels that write both in place would leave a mixture.
template <class T>
static bool arrays_overlap(const HostView<T>* views, const uint64_t* counts, uint32_t k) {
  typedef std::pair<uintptr_t, uintptr_t> Range;  // begin, end
  const auto array = [&](uint32_t i, int q) {
    static const uint64_t bytes[7] = {3 * sizeof(T), 3 * sizeof(T), 9 * sizeof(T), sizeof(T), 9 * sizeof(T), sizeof(T), 2};
    const uintptr_t a = reinterpret_cast<uintptr_t>(q < 6 ? static_cast<const void*>(views[i].f[q]) : views[i].mat);
    return Range(a, a + bytes[q] * counts[i]);
  };
  const auto apart = [](Range* r, size_t n) {
    std::sort(r, r + n);
    for (size_t q = 1; q < n; ++q)
      if (r[q].first < r[q - 1].second) return false;
    return true;
  };
  // the usual view sets need no sort of all arrays: one buffer per array, its scenes one after another
  Range span[7] = {};
  bool in_order = true;
  for (int q = 0; q < 7 && in_order; ++q) {
    bool any = false;
    for (uint32_t i = 0; i < k && in_order; ++i) {
      if (counts[i] == 0) continue;
      const Range r = array(i, q);
      in_order = !any || r.first >= span[q].second;
      if (!any) span[q].first = r.first;
      span[q].second = r.second;
      any = true;
    }
  }
  if (in_order && apart(span, 7)) return false;
  std::vector<Range> used;
  used.reserve(7 * size_t(k));
  for (uint32_t i = 0; i < k; ++i)
    for (int q = 0; q < 7 && counts[i] > 0; ++q) used.push_back(array(i, q));
  return !apart(used.data(), used.size());
}

bool views_overlap(const ae_mpm_particles* views, const uint64_t* counts, uint32_t k) {
  std::vector<HostView<float>> v(k);
  for (uint32_t i = 0; i < k; ++i) v[i] = host_view<float>(&views[i]);
  return arrays_overlap(v.data(), counts, k);
}

// [lo, hi) of the device allocation that address a lies in, as the driver knows it
static bool device_allocation(uintptr_t a, uintptr_t& lo, uintptr_t& hi) {
  typedef int (*RangeFn)(unsigned long long*, size_t*, unsigned long long);
  static const RangeFn range = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<RangeFn>(fn);
  }();
  unsigned long long base = 0;
  size_t size = 0;
  if (!range || range(&base, &size, a) != 0) return false;
  lo = uintptr_t(base);
  hi = lo + size;
  return true;
}

template <class T>
class World final : public WorldBase {
 public:
  using V4 = typename V4T<T>::type;

  ~World() override { release(); }

  int init(const ae_mpm_scene_desc* sc, uint32_t n, const ae_mpm_exec_opts& o) {
    opts_ = o;
    if (n == 0) {
      err = "a world needs at least one scene";
      return AE_MPM_EINVAL;
    }
    mode_ = sc[0].mode;
    if (mode_ < AE_MPM_MODE_PHYSICS || mode_ > AE_MPM_MODE_VELOCITY_ONLY) {
      err = "unknown substep mode";
      return AE_MPM_EINVAL;
    }
    uint64_t blk = 0, cap = 0;
    for (uint32_t s = 0; s < n; ++s) {
      const ae_mpm_scene_desc& d = sc[s];
      if (d.mode != mode_) {
        err = "all scenes of a world must use the same substep mode";
        return AE_MPM_EINVAL;
      }
      const uint32_t nmin = mode_ == AE_MPM_MODE_PHYSICS ? 4u : 1u;
      if (d.n[0] < nmin || d.n[1] < nmin || d.n[2] < nmin || !(d.dx > 0.0f) || !(d.dt >= 0.0f)) {
        err = "scene " + std::to_string(s) + ": grid needs >= " + std::to_string(nmin) +
              " nodes per axis, dx > 0 and dt >= 0";
        return AE_MPM_EINVAL;
      }
      if (d.n_materials == 0 || !d.materials) {
        err = "scene " + std::to_string(s) + ": material table is empty";
        return AE_MPM_EINVAL;
      }
      if (mode_ == AE_MPM_MODE_PHYSICS && d.wall_margin < 1) {
        err = "physics mode needs wall_margin >= 1";
        return AE_MPM_EINVAL;
      }
      if (mode_ == AE_MPM_MODE_PHYSICS && (d.n[0] > 1024 || d.n[1] > 1024 || d.n[2] > 1024)) {
        err = "physics-mode grids are limited to 1024 nodes per axis";
        return AE_MPM_EINVAL;
      }
      descs_.push_back(d);
      mats_.emplace_back(d.materials, d.materials + d.n_materials);
      blk += blocks_of(d);
      cap += d.max_particles;
    }
    if (blk * 64 >= (1ull << 31) || cap >= (1ull << 31)) {
      err = "world too large for 32-bit keys";
      return AE_MPM_EINVAL;
    }
    total_blocks_ = blk;
    total_cap_ = cap;
    key_bits_ = 1;
    while ((1ull << key_bits_) < blk * 64) ++key_bits_;
    if (opts_.precision != 32 && opts_.precision != 64) opts_.precision = sizeof(T) == 8 ? 64 : 32;
    if (opts_.sort_interval < 1) opts_.sort_interval = 1;
    if (opts_.block_threads != 128 && opts_.block_threads != 256) opts_.block_threads = 256;
    if (opts_.p2g_variant < kVarTile || opts_.p2g_variant > kVarLanes) opts_.p2g_variant = kVarLanes;
    AE_TRY(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    // scene table and materials
    uint64_t mat_off = 0, boff = 0, poff = 0;
    std::vector<uint32_t> blk_scene(blk), dead(blk, 0u);
    for (uint32_t s = 0; s < n; ++s) {
      const ae_mpm_scene_desc& d = descs_[s];
      SceneDev<T> h{};
      h.mode = d.mode;
      h.wall_mode = d.wall_mode;
      h.wall_margin = d.wall_margin;
      h.wall_origin = d.wall_origin;
      for (int a = 0; a < 3; ++a) {
        h.n[a] = int(d.n[a]);
        h.nb[a] = int((d.n[a] + 3) / 4);
      }
      h.blk_off = uint32_t(boff);
      uint64_t nbk = blocks_of(d);
      h.dead_key = uint32_t((boff + nbk - 1) * 64);
      for (uint64_t b = 0; b < nbk; ++b) blk_scene[boff + b] = s;
      dead[boff + nbk - 1] = 1u;
      boff += nbk;
      h.mat_off = uint32_t(mat_off);
      h.n_mat = d.n_materials;
      for (uint32_t k = 0; k < d.n_materials; ++k) {
        h_mats_.push_back(mat_dev(d.materials[k], d.materials[k].model));
        if (d.materials[k].model == kPhysSnow) has_snow_ = true;
      }
      // out-of-range material index: materials[0]'s parameters; the reference pairs them with
      // the neo-Hookean model (mpm_solver.rs:840-841)
      h_mats_.push_back(mat_dev(d.materials[0], mode_ == AE_MPM_MODE_PHYSICS ? d.materials[0].model : kNeoHookean));
      mat_off += d.n_materials + 1;
      h.p_off = uint32_t(poff);
      h.p_cap = uint32_t(d.max_particles);
      h.p_count = 0;
      poff += d.max_particles;
      fill_scene_params(h, d);
      h_scenes_.push_back(h);
    }
    // One allocation carries every array of the world, the ones that start at zero side by side (one
    // clear): thirty allocations and a dozen clears took most of a world's creation.
    const uint64_t pc = std::max<uint64_t>(cap, 1), nodes = blk * 64;
    // Dense grouping reads every node's counter; the radix sort moves 20 bytes per key and pass.
    // The grid decides: up to 16 nodes per particle slot (or 8 M nodes, 5 us of scan) the dense
    // grouping wins, a huge grid with few particles in it keeps the radix sort.
    dense_sort_ = nodes <= 16 * cap + (uint64_t(8) << 20);
    if (dense_sort_) n_segs_ = uint32_t((nodes + kBinSeg - 1) / kBinSeg);
    n_chunks_alloc_ = 0;
    for (const ae_mpm_scene_desc& d : descs_) n_chunks_alloc_ += int((d.max_particles + 127) / 128);  // smallest chunks
    std::vector<Region> regions =
        plan(this, {n, h_mats_.size(), blk, pc, uint64_t(n_chunks_alloc_), dense_sort_, opts_.deterministic != 0});
    std::stable_sort(regions.begin(), regions.end(), [](const Region& x, const Region& y) { return x.fill < y.fill; });
    size_t total = 0, end[2] = {0, 0};
    for (const Region& r : regions) {
      total += r.rounded();
      if (r.fill != kNone) end[r.fill] = total;
    }
    if (end[kOnes] == 0) end[kOnes] = end[kZero];
    AE_TRY(dmalloc(&arena_, total));
    size_t off = 0;
    for (const Region& r : regions) {
      *r.p = arena_ + off;
      off += r.rounded();
    }
    AE_TRY(cudaMemsetAsync(arena_, 0, end[kZero], stream_));
    AE_TRY(cudaMemsetAsync(arena_ + end[kZero], 0xff, end[kOnes] - end[kZero], stream_));
    AE_TRY(cudaMemcpyAsync(d_mats_, h_mats_.data(), sizeof(MatDev) * h_mats_.size(), cudaMemcpyHostToDevice, stream_));
    AE_TRY(cudaMemcpyAsync(blk_scene_, blk_scene.data(), sizeof(uint32_t) * blk, cudaMemcpyHostToDevice, stream_));
    AE_TRY(cudaMemcpyAsync(dead_blk_, dead.data(), sizeof(uint32_t) * blk, cudaMemcpyHostToDevice, stream_));
    if (!dense_sort_) AE_TRY(sort_scratch_alloc(sort_, pc, alloc_ ? &World::sort_alloc : nullptr, alloc_));
    AE_TRY(cudaStreamSynchronize(stream_));
    return AE_MPM_OK;
  }

  // The arrays of a world: where each goes (null without a world), its bytes and what it starts with.
  enum { kZero, kOnes, kNone };
  struct Region {
    void** p;
    size_t bytes;
    int fill;
    size_t rounded() const { return (bytes + 255) & ~size_t(255); }
  };
  struct Extent {
    uint64_t scenes, mats, blk, pc, chunks;
    bool dense, deterministic;
  };
  static std::vector<Region> plan(World* w, const Extent& x) {
    std::vector<Region> regions;
    const uint64_t nodes = x.blk * 64, segs = (nodes + kBinSeg - 1) / kBinSeg;
    auto reserve = [&](auto World::*m, size_t bytes, int fill) {
      regions.push_back({w ? reinterpret_cast<void**>(&(w->*m)) : nullptr, bytes, fill});
    };
    reserve(&World::d_scenes_, sizeof(SceneDev<T>) * x.scenes, kNone);
    reserve(&World::d_mats_, sizeof(MatDev) * x.mats, kNone);
    reserve(&World::blk_scene_, sizeof(uint32_t) * x.blk, kNone);
    reserve(&World::dead_blk_, sizeof(uint32_t) * x.blk, kNone);
    // particle slots past a scene's count are never read (every kernel gates on the live range),
    // so the particle arrays need no clearing
    for (int k = 0; k < 7; ++k) {
      regions.push_back({w ? reinterpret_cast<void**>(&w->bufA_[k]) : nullptr, sizeof(V4) * x.pc, kNone});
      regions.push_back({w ? reinterpret_cast<void**>(&w->bufB_[k]) : nullptr, sizeof(V4) * x.pc, kNone});
    }
    reserve(&World::keys_, sizeof(uint32_t) * x.pc, kNone);
    reserve(&World::clamp_queue_, sizeof(uint2) * x.pc, kNone);
    if (x.dense) {
      reserve(&World::bins_, sizeof(uint32_t) * nodes, kZero);
      reserve(&World::bin_off_, sizeof(uint32_t) * nodes, kNone);
      reserve(&World::seg_, sizeof(uint32_t) * 2 * segs, kNone);
      reserve(&World::bin_perm_, sizeof(uint32_t) * x.pc, kZero);
      if (x.deterministic) {
        reserve(&World::cells_, sizeof(uint2) * nodes, kZero);
        reserve(&World::ordered_, sizeof(uint32_t) * x.pc, kZero);
        reserve(&World::dead_cnt_, sizeof(uint32_t) * std::max<uint64_t>(x.chunks, 1), kNone);
      }
    } else if (x.deterministic) {
      reserve(&World::cell_slot_, sizeof(uint32_t) * nodes, kOnes);
      reserve(&World::seg_start_, sizeof(uint32_t) * x.pc, kNone);
    }
    if (x.deterministic) reserve(&World::cell_rec_, sizeof(V4) * 27 * x.pc, kNone);
    reserve(&World::acc_, sizeof(V4) * nodes, kZero);
    reserve(&World::vel_, sizeof(V4) * nodes, kZero);
    reserve(&World::blk_flag_, sizeof(uint32_t) * x.blk, kZero);
    reserve(&World::blk_epoch_, sizeof(uint32_t) * x.blk, kOnes);
    // two touched-block lists: the fused G2P + P2G fills the next substep's while the grid update
    // consumes the current one's
    reserve(&World::touched_, sizeof(uint32_t) * 2 * x.blk, kNone);
    reserve(&World::counters_, sizeof(uint32_t) * 8, kZero);
    reserve(&World::err_, sizeof(uint32_t) * 4 * x.scenes, kZero);
    reserve(&World::d_xfer_, sizeof(XferDev<T>) * x.scenes, kNone);
    reserve(&World::d_chunks_, sizeof(int4) * std::max<uint64_t>(x.chunks, 1), kNone);
    return regions;
  }

  // Device bytes that a scene adds to a world at most: its share of the world's arrays, of the radix
  // sort's scratch where the world may sort so (its other scenes decide), and of the transfer staging.
  static uint64_t device_bytes_of(const ae_mpm_scene_desc& d, bool deterministic) {
    const uint64_t pc = std::max<uint64_t>(d.max_particles, 1), chunks = (d.max_particles + 127) / 128;
    uint64_t most = 0;
    for (const bool dense : {false, true}) {
      uint64_t sum = dense ? 0 : sort_scratch_bytes(pc);
      for (const Region& r : plan(nullptr, {1, uint64_t(d.n_materials) + 1, blocks_of(d), pc, chunks, dense, deterministic}))
        sum += r.rounded();
      most = std::max(most, sum);
    }
    return most + pc * (26 * sizeof(T) + sizeof(uint16_t)) + 64;
  }

  void fill_scene_params(SceneDev<T>& h, const ae_mpm_scene_desc& d) {
    h.dx = T(d.dx);
    h.inv_dx = T(1) / T(d.dx);
    h.dt = T(d.dt);
    h.restitution = T(d.restitution);
    h.damping = T(d.damping);
    h.wall_mode = d.wall_mode;
    h.wall_margin = d.wall_margin;
    h.wall_origin = d.wall_origin;
    for (int a = 0; a < 3; ++a) {
      h.origin[a] = T(d.origin[a]);
      h.grav[a] = T(d.gravity[a]);
    }
    if (sizeof(T) == 4) h.inv_dx = T(1.0f / d.dx);  // f32: the reference's `1.0 / dx` in f32
  }

  int set_scene_params(uint32_t s, const ae_mpm_scene_desc& d) override {
    if (s >= h_scenes_.size()) {
      err = "unknown scene";
      return AE_MPM_ENOTFOUND;
    }
    if (d.n[0] != uint32_t(h_scenes_[s].n[0]) || d.n[1] != uint32_t(h_scenes_[s].n[1]) || d.n[2] != uint32_t(h_scenes_[s].n[2])) {
      err = "grid size of a resident scene cannot change";
      return AE_MPM_EINVAL;
    }
    if (d.n_materials != h_scenes_[s].n_mat || !d.materials) {
      err = "material count of a resident scene cannot change";
      return AE_MPM_EINVAL;
    }
    if (d.mode != mode_ || !(d.dx > 0.0f) || !(d.dt >= 0.0f) || (mode_ == AE_MPM_MODE_PHYSICS && d.wall_margin < 1)) {
      err = "scene update needs the world's mode, dx > 0, dt >= 0 and (physics) wall_margin >= 1";
      return AE_MPM_EINVAL;
    }
    // physics mode stores A = m C - k tau, which depends on dt and the materials: convert the
    // resident particles back to C with the old tables and again to A with the new ones
    const uint64_t cnt = h_scenes_[s].p_count;
    const bool rebase = mode_ == AE_MPM_MODE_PHYSICS && cnt > 0;
    if (rebase) {
      int rc = ensure_stage(cnt);
      if (rc) return rc;
      const XferDev<T> x = stage_xfer(stage_, cnt);
      if ((rc = launch_unpack(1, &s, &x))) return rc;
    }
    fill_scene_params(h_scenes_[s], d);
    for (uint32_t k = 0; k < d.n_materials; ++k) {
      h_mats_[h_scenes_[s].mat_off + k] = mat_dev(d.materials[k], d.materials[k].model);
      if (d.materials[k].model == kPhysSnow && !has_snow_) {
        has_snow_ = true;  // the substep gains the clamp kernel: recapture
        invalidate_graph();
      }
    }
    h_mats_[h_scenes_[s].mat_off + d.n_materials] =
        mat_dev(d.materials[0], mode_ == AE_MPM_MODE_PHYSICS ? d.materials[0].model : kNeoHookean);
    dirty_scene(s);
    dirty_mats(s);
    keys_stale_ = true;  // dx or origin may have moved the cells
    scatter_invalid_ = true;
    if (rebase) {
      const XferDev<T> x = stage_xfer(stage_, cnt);
      const int rc = launch_pack(1, &s, &x);
      if (rc) return rc;
      keys_stale_ = true;
    }
    return AE_MPM_OK;
  }

  static XferDev<T> stage_xfer(T* st, uint64_t n) {
    return XferDev<T>{{st, st + 3 * n, st + 6 * n, st + 15 * n, st + 16 * n, st + 25 * n},
                      reinterpret_cast<uint16_t*>(st + 26 * n), uint32_t(n), 0u};
  }
  static XferDev<T> view_xfer(const HostView<T>& hv, uint64_t n) {
    return XferDev<T>{{hv.f[0], hv.f[1], hv.f[2], hv.f[3], hv.f[4], hv.f[5]}, hv.mat, uint32_t(n), 0u};
  }

  // Which views of one transfer the kernels may use in place.  Every array has to be ordinary memory of
  // the world's device, aligned for its type, and to end inside its allocation: a copy of too short an
  // array is refused by the driver, a kernel would run past it.  Anything else (host, managed or another
  // device's memory, odd addresses, short arrays) travels through the staging area.
  struct DirectViews {
    struct {
      uintptr_t lo, hi;
    } known[8] = {};  // allocations found in this call, the last 8: one per array of the views and one more
    uint32_t next = 0;

    bool array(const void* p, size_t bytes, size_t align) {
      const uintptr_t a = reinterpret_cast<uintptr_t>(p);
      if (a % align != 0) return false;
      for (const auto& k : known)
        if (a >= k.lo && a < k.hi) return bytes <= k.hi - a;
      int dev = 0;
      cudaPointerAttributes at{};
      if (cudaGetDevice(&dev) != cudaSuccess || cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      uintptr_t lo = 0, hi = 0;
      if (at.type != cudaMemoryTypeDevice || at.device != dev || !device_allocation(a, lo, hi)) return false;
      known[next++ % 8] = {lo, hi};
      return a >= lo && a < hi && bytes <= hi - a;
    }
    bool takes(const HostView<T>& hv, uint64_t n) {
      const uint64_t len[6] = {3, 3, 9, 1, 9, 1};
      bool ok = array(hv.mat, sizeof(uint16_t) * n, sizeof(uint16_t));
      for (int k = 0; k < 6 && ok; ++k) ok = array(hv.f[k], sizeof(T) * len[k] * n, sizeof(T));
      return ok;
    }
  };

  // Launch range and description of a transfer of k scenes (x[i] describes scene scenes[i]); false
  // when no particle moves.  A single scene travels as a launch parameter, several as a table.
  int xfer_range(uint32_t k, const uint32_t* scenes, const XferDev<T>* x, WorldDev<T>& w, XferSet<T>& xs, int& blocks) {
    blocks = 0;
    int rc = prepare();
    if (rc) return rc;
    w = dev(false);
    xs = XferSet<T>{};
    int c0 = 0;
    if (k == 1) {
      xs.one = x[0];
      c0 = chunk_first_[scenes[0]];
      blocks = int((x[0].n + uint32_t(chunk_threads_) - 1) / uint32_t(chunk_threads_));
    } else {
      uint32_t lo = scenes[0], hi = scenes[0];
      for (uint32_t i = 1; i < k; ++i) {
        lo = std::min(lo, scenes[i]);
        hi = std::max(hi, scenes[i]);
      }
      h_xfer_.assign(hi - lo + 1, XferDev<T>{});
      for (uint32_t i = 0; i < k; ++i) h_xfer_[scenes[i] - lo] = x[i];
      AE_TRY(cudaMemcpyAsync(d_xfer_, h_xfer_.data(), sizeof(XferDev<T>) * h_xfer_.size(), cudaMemcpyHostToDevice,
                             stream_));
      xs.tab = d_xfer_;
      xs.s0 = lo;
      c0 = chunk_first_[lo];
      blocks = chunk_first_[hi + 1] - c0;
    }
    if (!w.one_scene) w.chunks = d_chunks_ + c0;
    return AE_MPM_OK;
  }

  // a scene named twice in one call is transferred twice, in order
  static bool has_repeats(uint32_t k, const uint32_t* scenes) {
    std::vector<uint32_t> v(scenes, scenes + k);
    std::sort(v.begin(), v.end());
    return std::adjacent_find(v.begin(), v.end()) != v.end();
  }

  int launch_pack(uint32_t k, const uint32_t* scenes, const XferDev<T>* x, bool motion = false) {
    if (k > 1 && has_repeats(k, scenes)) {
      int rc = AE_MPM_OK;
      for (uint32_t i = 0; i < k && rc == AE_MPM_OK; ++i) rc = launch_pack(1, scenes + i, x + i);
      return rc;
    }
    WorldDev<T> w{};
    XferSet<T> xs{};
    int blocks = 0;
    const int rc = xfer_range(k, scenes, x, w, xs, blocks);
    if (rc || blocks == 0) return rc;
    const auto pack = motion ? pack_kernel<T, true> : pack_kernel<T, false>;
    pack<<<unsigned(blocks), chunk_threads_, 0, stream_>>>(w, xs);
    AE_TRY(cudaGetLastError());
    return AE_MPM_OK;
  }

  // the slot index lives in the clamp queue, which is empty between substeps
  int launch_unpack(uint32_t k, const uint32_t* scenes, const XferDev<T>* x, bool motion = false) {
    if (k > 1 && has_repeats(k, scenes)) {
      int rc = AE_MPM_OK;
      for (uint32_t i = 0; i < k && rc == AE_MPM_OK; ++i) rc = launch_unpack(1, scenes + i, x + i);
      return rc;
    }
    WorldDev<T> w{};
    XferSet<T> xs{};
    int blocks = 0;
    const int rc = xfer_range(k, scenes, x, w, xs, blocks);
    if (rc || blocks == 0) return rc;
    uint32_t* inv = reinterpret_cast<uint32_t*>(clamp_queue_);
    unpack_index_kernel<T><<<unsigned(blocks), chunk_threads_, 0, stream_>>>(w, xs, inv);
    const auto unpack = motion ? unpack_kernel<T, true> : unpack_kernel<T, false>;
    unpack<<<unsigned(blocks), chunk_threads_, 0, stream_>>>(w, xs, inv);
    AE_TRY(cudaGetLastError());
    return AE_MPM_OK;
  }

  // whether a particle view's seven arrays lie back to back in the staging order (pos, vel, F, J,
  // C, mass at 0, 3n, 6n, 15n, 16n, 25n elements, the material indices at 26n)
  static bool staging_layout(const HostView<T>& hv, uint64_t n) {
    const uintptr_t b = reinterpret_cast<uintptr_t>(hv.f[0]);
    const uint64_t at[6] = {0, 3, 6, 15, 16, 25};
    for (int k = 1; k < 6; ++k)
      if (reinterpret_cast<uintptr_t>(hv.f[k]) != b + sizeof(T) * at[k] * n) return false;
    return reinterpret_cast<uintptr_t>(hv.mat) == b + sizeof(T) * 26 * n;
  }

  int upload(uint32_t s, const void* host, uint64_t n, bool f64) override {
    if (s >= h_scenes_.size()) {
      err = "unknown scene";
      return AE_MPM_ENOTFOUND;
    }
    if ((sizeof(T) == 8) != f64) {
      err = "particle view precision does not match the world precision";
      return AE_MPM_EINVAL;
    }
    if (n > h_scenes_[s].p_cap) {
      err = "scene " + std::to_string(s) + ": " + std::to_string(n) + " particles exceed max_particles " +
            std::to_string(h_scenes_[s].p_cap);
      return AE_MPM_EINVAL;
    }
    const HostView<T> hv = host_view<T>(host);
    const T* const* f = hv.f;
    if (n > 0 && (!f[0] || !f[1] || !f[2] || !f[3] || !f[4] || !f[5] || !hv.mat)) {
      err = "particle view has a null array";
      return AE_MPM_EINVAL;
    }
    if (n > 0) {
      XferDev<T> x = view_xfer(hv, n);
      if (!DirectViews().takes(hv, n)) {
        const int rs = ensure_stage(n);
        if (rs) return rs;
        const int rc = stage_in(stage_, hv, n, stream_);
        if (rc) return rc;
        x = stage_xfer(stage_, n);
      }
      const int rc = launch_pack(1, &s, &x);
      if (rc) return rc;
    }
    uploaded(s, n);
    return AE_MPM_OK;
  }

  // the same count keeps the scene table, the chunks and the captured graph (which replays from
  // the upload's buffers); the cell keys are recomputed before the next substep either way
  void uploaded(uint32_t s, uint64_t n) {
    scatter_invalid_ = true;
    if (h_scenes_[s].p_count != uint32_t(n)) {
      h_scenes_[s].p_count = uint32_t(n);
      count_changed(s);
    }
    keys_stale_ = true;
  }

  int upload_motion(const float* pos, const float* vel, const float* mass, uint64_t n) override {
    if constexpr (sizeof(T) == 4) {
      if (mode_ == AE_MPM_MODE_VELOCITY_ONLY && n <= h_scenes_[0].p_cap) {
        XferDev<T> x{};
        x.f[0] = const_cast<float*>(pos);
        x.f[1] = const_cast<float*>(vel);
        x.f[5] = const_cast<float*>(mass);
        x.n = uint32_t(n);
        const uint32_t s = 0;
        const int rc = n > 0 ? launch_pack(1, &s, &x, true) : AE_MPM_OK;
        if (rc) return rc;
        uploaded(0, n);
        return AE_MPM_OK;
      }
    }
    err = "not a velocity-only FP32 world of that capacity";
    return AE_MPM_EINVAL;
  }

  int download_motion(float* pos, float* vel) override {
    if constexpr (sizeof(T) == 4) {
      if (mode_ == AE_MPM_MODE_VELOCITY_ONLY) {
        XferDev<T> x{};
        x.f[0] = pos;
        x.f[1] = vel;
        x.n = h_scenes_[0].p_count;
        const uint32_t s = 0;
        return x.n > 0 ? launch_unpack(1, &s, &x, true) : AE_MPM_OK;
      }
    }
    err = "not a velocity-only FP32 world";
    return AE_MPM_EINVAL;
  }

  int download(uint32_t s, void* host, bool f64) override {
    if (s >= h_scenes_.size()) {
      err = "unknown scene";
      return AE_MPM_ENOTFOUND;
    }
    if ((sizeof(T) == 8) != f64) {
      err = "particle view precision does not match the world precision";
      return AE_MPM_EINVAL;
    }
    const uint64_t n = h_scenes_[s].p_count;
    HostView<T> hv = host_view<T>(host);
    T* const* f = hv.f;
    if (n == 0) return AE_MPM_OK;
    if (!f[0] || !f[1] || !f[2] || !f[3] || !f[4] || !f[5] || !hv.mat) {
      err = "particle view has a null array";
      return AE_MPM_EINVAL;
    }
    const bool direct = DirectViews().takes(hv, n) && !arrays_overlap(&hv, &n, 1);
    XferDev<T> x = view_xfer(hv, n);
    if (!direct) {
      const int rs = ensure_stage(n);
      if (rs) return rs;
      x = stage_xfer(stage_, n);
    }
    int rc = launch_unpack(1, &s, &x);
    if (rc) return rc;
    if (!direct && (rc = stage_out(stage_, hv, n, stream_))) return rc;
    AE_TRY(cudaStreamSynchronize(stream_));
    return AE_MPM_OK;
  }

  // a view's arrays into a staging area and back (unified addressing picks the direction); a view
  // laid out as the staging itself travels in one copy
  int stage_in(T* st, const HostView<T>& hv, uint64_t n, cudaStream_t cs) {
    if (staging_layout(hv, n)) {
      AE_TRY(cudaMemcpyAsync(st, hv.f[0], sizeof(T) * 26 * n + sizeof(uint16_t) * n, cudaMemcpyDefault, cs));
      return AE_MPM_OK;
    }
    const uint64_t at[6] = {0, 3, 6, 15, 16, 25}, len[6] = {3, 3, 9, 1, 9, 1};
    for (int f = 0; f < 6; ++f)
      AE_TRY(cudaMemcpyAsync(st + at[f] * n, hv.f[f], sizeof(T) * len[f] * n, cudaMemcpyDefault, cs));
    AE_TRY(cudaMemcpyAsync(st + 26 * n, hv.mat, sizeof(uint16_t) * n, cudaMemcpyDefault, cs));
    return AE_MPM_OK;
  }
  int stage_out(const T* st, const HostView<T>& hv, uint64_t n, cudaStream_t cs) {
    if (staging_layout(hv, n)) {
      AE_TRY(cudaMemcpyAsync(hv.f[0], st, sizeof(T) * 26 * n + sizeof(uint16_t) * n, cudaMemcpyDefault, cs));
      return AE_MPM_OK;
    }
    const uint64_t at[6] = {0, 3, 6, 15, 16, 25}, len[6] = {3, 3, 9, 1, 9, 1};
    for (int f = 0; f < 6; ++f)
      AE_TRY(cudaMemcpyAsync(hv.f[f], st + at[f] * n, sizeof(T) * len[f] * n, cudaMemcpyDefault, cs));
    AE_TRY(cudaMemcpyAsync(hv.mat, st + 26 * n, sizeof(uint16_t) * n, cudaMemcpyDefault, cs));
    return AE_MPM_OK;
  }

  // byte offset of each scene's region in a many-scene staging area (16-byte aligned regions in the
  // staging layout of upload)
  static uint64_t stage_region(uint64_t n) { return (sizeof(T) * 26 * n + sizeof(uint16_t) * n + 15) / 16 * 16; }

  // orders `later` after the work queued so far on `earlier`
  int stream_after(cudaStream_t later, cudaStream_t earlier) {
    if (!xfer_ev_) AE_TRY(cudaEventCreateWithFlags(&xfer_ev_, cudaEventDisableTiming));
    AE_TRY(cudaEventRecord(xfer_ev_, earlier));
    AE_TRY(cudaStreamWaitEvent(later, xfer_ev_, 0));
    return AE_MPM_OK;
  }

  int upload_many(uint32_t k, const uint32_t* scenes, const ae_mpm_particles* views, const uint64_t* counts,
                  cudaStream_t copy) override {
    if (sizeof(T) != 4) {
      err = "many-scene transfers are for f32 worlds";
      return AE_MPM_EINVAL;
    }
    if (k == 0) return AE_MPM_OK;
    if (!scenes || !views || !counts) {
      err = "null scene, view or count array";
      return AE_MPM_EINVAL;
    }
    uint64_t total = 0;
    for (uint32_t i = 0; i < k; ++i) {
      const uint32_t s = scenes[i];
      if (s >= h_scenes_.size()) {
        err = "unknown scene";
        return AE_MPM_ENOTFOUND;
      }
      if (counts[i] > h_scenes_[s].p_cap) {
        err = "scene " + std::to_string(s) + ": " + std::to_string(counts[i]) + " particles exceed max_particles " +
              std::to_string(h_scenes_[s].p_cap);
        return AE_MPM_EINVAL;
      }
      const ae_mpm_particles& v = views[i];
      if (counts[i] > 0 && (!v.pos || !v.vel || !v.strain || !v.jacobian || !v.c || !v.mass || !v.material_idx)) {
        err = "particle view has a null array";
        return AE_MPM_EINVAL;
      }
    }
    // views in device memory are read in place; the others get a region of the staging area each
    std::vector<XferDev<T>> x(k);
    std::vector<uint8_t> staged(k, 0);
    DirectViews in_place;
    for (uint32_t i = 0; i < k; ++i) {
      const HostView<T> hv = host_view<T>(&views[i]);
      x[i] = view_xfer(hv, counts[i]);
      staged[i] = counts[i] > 0 && !in_place.takes(hv, counts[i]);
      if (staged[i]) total += stage_region(counts[i]);
    }
    if (total > 0) {
      const int rs = ensure_stage_bytes(total);
      if (rs) return rs;
      // all copies first, back to back on the copy stream (the world's own by default), then the pack
      const cudaStream_t cs = copy ? copy : stream_;
      if (copy) {  // the staging area is free once the world's queued work is done with it
        const int r = stream_after(cs, stream_);
        if (r) return r;
      }
      uint64_t off = 0;
      for (uint32_t i = 0; i < k; ++i) {
        if (!staged[i]) continue;
        T* st = reinterpret_cast<T*>(reinterpret_cast<char*>(stage_) + off);
        const int r = stage_in(st, host_view<T>(&views[i]), counts[i], cs);
        if (r) return r;
        x[i] = stage_xfer(st, counts[i]);
        off += stage_region(counts[i]);
      }
      if (copy) {
        const int r = stream_after(stream_, cs);
        if (r) return r;
      }
    }
    for (uint32_t i = 0; i < k; ++i) {
      const uint32_t s = scenes[i];
      if (h_scenes_[s].p_count != uint32_t(counts[i])) {
        h_scenes_[s].p_count = uint32_t(counts[i]);
        count_changed(s);
      }
    }
    const int rc = launch_pack(k, scenes, x.data());
    if (rc) return rc;
    keys_stale_ = true;
    scatter_invalid_ = true;
    return AE_MPM_OK;
  }

  int download_many(uint32_t k, const uint32_t* scenes, ae_mpm_particles* views, cudaStream_t copy,
                    bool in_place) override {
    if (sizeof(T) != 4) {
      err = "many-scene transfers are for f32 worlds";
      return AE_MPM_EINVAL;
    }
    if (k == 0) return AE_MPM_OK;
    if (!scenes || !views) {
      err = "null scene or view array";
      return AE_MPM_EINVAL;
    }
    uint64_t total = 0;
    for (uint32_t i = 0; i < k; ++i) {
      if (scenes[i] >= h_scenes_.size()) {
        err = "unknown scene";
        return AE_MPM_ENOTFOUND;
      }
      const ae_mpm_particles& v = views[i];
      if (h_scenes_[scenes[i]].p_count > 0 &&
          (!v.pos || !v.vel || !v.strain || !v.jacobian || !v.c || !v.mass || !v.material_idx)) {
        err = "particle view has a null array";
        return AE_MPM_EINVAL;
      }
    }
    std::vector<XferDev<T>> x(k);
    std::vector<uint64_t> counts(k), at(k, UINT64_MAX);  // at: offset of a staged scene's region
    DirectViews direct;
    for (uint32_t i = 0; i < k; ++i) counts[i] = h_scenes_[scenes[i]].p_count;
    in_place = in_place && !views_overlap(views, counts.data(), k);
    for (uint32_t i = 0; i < k; ++i) {
      const HostView<T> hv = host_view<T>(&views[i]);
      x[i] = view_xfer(hv, counts[i]);
      if (counts[i] == 0 || (in_place && direct.takes(hv, counts[i]))) continue;
      at[i] = total;
      total += stage_region(counts[i]);
    }
    if (total > 0) {
      const int rs = ensure_stage_bytes(total);
      if (rs) return rs;
    }
    for (uint32_t i = 0; i < k; ++i)
      if (at[i] != UINT64_MAX)
        x[i] = stage_xfer(reinterpret_cast<T*>(reinterpret_cast<char*>(stage_) + at[i]), x[i].n);
    const int rc = launch_unpack(k, scenes, x.data());
    if (rc) return rc;
    const cudaStream_t cs = copy ? copy : stream_;
    if (copy) {
      const int r = stream_after(cs, stream_);
      if (r) return r;
    }
    for (uint32_t i = 0; i < k; ++i) {
      if (at[i] == UINT64_MAX) continue;
      const int r = stage_out(x[i].f[0], host_view<T>(&views[i]), x[i].n, cs);
      if (r) return r;
    }
    if (copy) {  // the next use of the staging area on the world's stream waits for these reads
      const int r = stream_after(stream_, cs);
      if (r) return r;
      return AE_MPM_OK;
    }
    AE_TRY(cudaStreamSynchronize(stream_));
    return AE_MPM_OK;
  }

  int step(uint32_t n) override {
    launches_ = 0;
    int rc = prepare();
    if (rc) return rc;
    if (n == 0) return AE_MPM_OK;
    if ((rc = settle_order())) return rc;
    if ((rc = sync_scatter())) return rc;
    const uint32_t interval = sort_interval();
    const uint32_t period = (interval % 2 == 0) ? interval : 2 * interval;
    uint32_t left = n;
    while (left > 0) {
      if (opts_.use_graph && phase_ == 0 && left >= period && n_chunks_ > 0 && graph_now()) {
        rc = ensure_graph(period);
        if (rc) return rc;
        Graph& g = graphs_[substep_ & 1][graph_entry()];
        AE_TRY(cudaGraphLaunch(g.exec, stream_));
        sorted_ = g.sorted_out;
        keys_fresh_ = g.fresh_out;
        launches_ += g.launches;
        substep_ += period;
        left -= period;
      } else {
        substep_eager(left == 1);
        --left;
      }
    }
    AE_TRY(cudaGetLastError());
    return AE_MPM_OK;
  }

  int sync() override {
    AE_TRY(cudaStreamSynchronize(stream_));
    std::vector<uint32_t> e(4 * h_scenes_.size());
    AE_TRY(cudaMemcpy(e.data(), err_, sizeof(uint32_t) * e.size(), cudaMemcpyDeviceToHost));
    uint32_t any = 0;
    for (size_t s = 0; s < h_scenes_.size(); ++s) any |= e[4 * s];
    if (any & kErrNaN) {
      err = "a particle position became non-finite";
      return AE_MPM_ENAN;
    }
    if (any & kErrDomain) {
      err = "particles reached the grid's outer ring and were clamped back";
      return AE_MPM_EDOMAIN;
    }
    return AE_MPM_OK;
  }

  int totals(uint32_t s, double out[5]) override {
    if (s >= h_scenes_.size()) {
      err = "unknown scene";
      return AE_MPM_ENOTFOUND;
    }
    int rc = prepare();
    if (rc) return rc;
    if (n_chunks_ == 0) {
      for (int k = 0; k < 5; ++k) out[k] = 0;
      return AE_MPM_OK;
    }
    if (!partial_) AE_TRY(dmalloc(&partial_, sizeof(double) * 5 * n_chunks_alloc_));
    WorldDev<T> w = dev(false);
    totals_kernel<T><<<n_chunks_, chunk_threads_, 0, stream_>>>(w, partial_);
    AE_TRY(cudaGetLastError());
    std::vector<double> h(5 * size_t(n_chunks_));
    AE_TRY(cudaMemcpyAsync(h.data(), partial_, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, stream_));
    AE_TRY(cudaStreamSynchronize(stream_));
    for (int k = 0; k < 5; ++k) out[k] = 0;
    for (int c = 0; c < n_chunks_; ++c)
      if (uint32_t(h_chunks_[c].x) == s)
        for (int k = 0; k < 5; ++k) out[k] += h[5 * size_t(c) + k];
    return AE_MPM_OK;
  }

  int errors(uint32_t s, uint32_t* word, uint64_t counters[3]) override {
    if (s >= h_scenes_.size()) {
      err = "unknown scene";
      return AE_MPM_ENOTFOUND;
    }
    uint32_t e[4];
    AE_TRY(cudaStreamSynchronize(stream_));
    AE_TRY(cudaMemcpy(e, err_ + 4 * s, sizeof(e), cudaMemcpyDeviceToHost));
    AE_TRY(cudaMemset(err_ + 4 * s, 0, sizeof(e)));
    if (word) *word = e[0];
    if (counters) {
      counters[0] = e[1];
      counters[1] = e[2];
      counters[2] = e[3];
    }
    return AE_MPM_OK;
  }

  int grid_download(uint32_t s, float* mass, float* vel, uint64_t n_nodes) override {
    if (s >= h_scenes_.size()) {
      err = "unknown scene";
      return AE_MPM_ENOTFOUND;
    }
    const SceneDev<T>& h = h_scenes_[s];
    uint64_t nn = uint64_t(h.n[0]) * h.n[1] * h.n[2];
    if (n_nodes != nn || !mass || !vel) {
      err = "grid download needs nx*ny*nz nodes";
      return AE_MPM_EINVAL;
    }
    float *dm = nullptr, *dv = nullptr;
    AE_TRY(dmalloc(&dm, sizeof(float) * nn));
    AE_TRY(dmalloc(&dv, sizeof(float) * 3 * nn));
    grid_export_kernel<T><<<unsigned((nn + 255) / 256), 256, 0, stream_>>>(vel_, d_scenes_ + s, blk_epoch_, counters_ + 2,
                                                                           dm, dv);
    cudaError_t e1 = cudaMemcpyAsync(mass, dm, sizeof(float) * nn, cudaMemcpyDeviceToHost, stream_);
    cudaError_t e2 = cudaMemcpyAsync(vel, dv, sizeof(float) * 3 * nn, cudaMemcpyDeviceToHost, stream_);
    cudaError_t e3 = cudaStreamSynchronize(stream_);
    dfree(dm);
    dfree(dv);
    if (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess) {
      err = "grid download failed";
      return AE_MPM_ECUDA;
    }
    return AE_MPM_OK;
  }

  int snapshot(bool restore) override {
    const uint64_t pc = std::max<uint64_t>(total_cap_, 1);
    if (!restore) {
      for (int k = 0; k < 7; ++k) {
        if (!snap_[k]) AE_TRY(dmalloc(&snap_[k], sizeof(V4) * pc));
        AE_TRY(cudaMemcpyAsync(snap_[k], in_buf()[k], sizeof(V4) * pc, cudaMemcpyDeviceToDevice, stream_));
      }
      snap_substep_ = substep_;
    } else {
      if (!snap_[0]) {
        err = "no snapshot";
        return AE_MPM_EINVAL;
      }
      for (int k = 0; k < 7; ++k)
        AE_TRY(cudaMemcpyAsync(in_buf()[k], snap_[k], sizeof(V4) * pc, cudaMemcpyDeviceToDevice, stream_));
      keys_stale_ = true;
      scatter_invalid_ = true;
      AE_TRY(cudaMemsetAsync(err_, 0, sizeof(uint32_t) * 4 * h_scenes_.size(), stream_));
    }
    AE_TRY(cudaStreamSynchronize(stream_));
    return AE_MPM_OK;
  }

  uint64_t last_launches() const override { return launches_; }
  uint64_t particles() const override {
    uint64_t s = 0;
    for (auto& h : h_scenes_) s += h.p_count;
    return s;
  }
  cudaStream_t stream() const override { return stream_; }
  int set_stream_priority(int priority) override {
    drop_graphs();
    AE_TRY(cudaStreamSynchronize(stream_));
    cudaStream_t s = nullptr;
    AE_TRY(cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, priority));
    cudaStreamDestroy(stream_);
    stream_ = s;
    return AE_MPM_OK;
  }
  ae_mpm_exec_opts& opts() override { return opts_; }
  void invalidate_graph() override {
    drop_graphs();
    chunks_dirty_ = true;
  }
  uint64_t device_bytes() const override { return device_bytes_; }

  int copy_scene_from(uint32_t dst, WorldBase* srcb, uint32_t s) override {
    auto* src = dynamic_cast<World<T>*>(srcb);
    if (!src || dst >= h_scenes_.size() || s >= src->h_scenes_.size()) {
      err = "scene copy between incompatible worlds";
      return AE_MPM_EINVAL;
    }
    const SceneDev<T>& a = src->h_scenes_[s];
    SceneDev<T>& b = h_scenes_[dst];
    if (a.n[0] != b.n[0] || a.n[1] != b.n[1] || a.n[2] != b.n[2] || a.p_count > b.p_cap) {
      err = "scene copy needs the same grid and enough particle capacity";
      return AE_MPM_EINVAL;
    }
    for (int k = 0; k < 7; ++k)
      if (a.p_count)
        AE_TRY(cudaMemcpyAsync(in_buf()[k] + b.p_off, src->in_buf()[k] + a.p_off, sizeof(V4) * a.p_count,
                               cudaMemcpyDeviceToDevice, stream_));
    // the scene's error word and counters move with it
    AE_TRY(cudaMemcpyAsync(err_ + 4 * dst, src->err_ + 4 * s, sizeof(uint32_t) * 4, cudaMemcpyDeviceToDevice, stream_));
    b.p_count = a.p_count;
    count_changed(dst);
    keys_stale_ = scatter_invalid_ = true;
    return AE_MPM_OK;
  }
  uint32_t scene_count(uint32_t s) const override { return s < h_scenes_.size() ? h_scenes_[s].p_count : 0; }

  int assign_scene(uint32_t s, const ae_mpm_scene_desc& d, const void* host, uint64_t n) override {
    if (s >= h_scenes_.size()) {
      err = "unknown scene";
      return AE_MPM_ENOTFOUND;
    }
    SceneDev<T>& h = h_scenes_[s];
    const uint32_t nmin = mode_ == AE_MPM_MODE_PHYSICS ? 4u : 1u;
    if (d.mode != mode_ || d.n[0] < nmin || d.n[1] < nmin || d.n[2] < nmin || !(d.dx > 0.0f) || !(d.dt >= 0.0f) ||
        (mode_ == AE_MPM_MODE_PHYSICS && d.wall_margin < 1) || d.n_materials == 0 || !d.materials) {
      err = "slot scene needs the world's mode, >= " + std::to_string(nmin) +
            " nodes per axis, dx > 0, dt >= 0, materials and (physics) wall_margin >= 1";
      return AE_MPM_EINVAL;
    }
    if (blocks_of(d) > blocks_of(descs_[s]) || d.n_materials > descs_[s].n_materials || n > h.p_cap) {
      err = "scene does not fit slot " + std::to_string(s) + " (grid blocks, materials or particles)";
      return AE_MPM_EINVAL;
    }
    for (int a = 0; a < 3; ++a) {
      h.n[a] = int(d.n[a]);
      h.nb[a] = int((d.n[a] + 3) / 4);
    }
    h.mode = d.mode;
    h.n_mat = d.n_materials;  // the out-of-range fallback entry follows the scene's materials
    fill_scene_params(h, d);
    for (uint32_t k = 0; k < d.n_materials; ++k) {
      h_mats_[h.mat_off + k] = mat_dev(d.materials[k], d.materials[k].model);
      if (d.materials[k].model == kPhysSnow && !has_snow_) {
        has_snow_ = true;  // the substep gains the clamp kernel: recapture
        invalidate_graph();
      }
    }
    h_mats_[h.mat_off + d.n_materials] =
        mat_dev(d.materials[0], mode_ == AE_MPM_MODE_PHYSICS ? d.materials[0].model : kNeoHookean);
    dirty_scene(s);
    dirty_mats(s);
    keys_stale_ = true;
    AE_TRY(cudaMemsetAsync(err_ + 4 * s, 0, sizeof(uint32_t) * 4, stream_));
    if (!host) {
      h.p_count = 0;
      count_changed(s);
      return AE_MPM_OK;
    }
    // with the P2G of the next substep already queued for the other scenes (fused flow), add
    // only this scene's scatter instead of redoing everyone's
    const bool keep_queued = scatter_pending_ && !scatter_invalid_ && fused();
    int rc = upload(s, host, n, sizeof(T) == 8);
    if (rc || !keep_queued) return rc;
    scatter_invalid_ = false;
    // the slot's blocks may hold the last scatter of the scene that vacated it: zero them (their
    // flags stay set, so the touched list keeps each block once); the next step() scatters the new
    // particles once it has put them in cell order
    AE_TRY(cudaMemsetAsync(acc_ + uint64_t(h.blk_off) * 64u, 0, sizeof(V4) * 64 * blocks_of(descs_[s]), stream_));
    if (std::find(late_slots_.begin(), late_slots_.end(), s) == late_slots_.end()) late_slots_.push_back(s);
    return AE_MPM_OK;
  }

  int vacate_scene(uint32_t s) override {
    if (s >= h_scenes_.size()) {
      err = "unknown scene";
      return AE_MPM_ENOTFOUND;
    }
    // a scatter queued for the next substep may still hold the scene's contributions: they land in
    // the slot's own blocks, which the next grid update consumes and no particle reads
    h_scenes_[s].p_count = 0;
    count_changed(s);
    keys_stale_ = true;
    return AE_MPM_OK;
  }
  int precision() const override { return sizeof(T) == 8 ? 64 : 32; }

  int stage_times(uint32_t n, double out_us[6]) override {
    for (int k = 0; k < 6; ++k) out_us[k] = 0;
    int rc = prepare();
    if (rc) return rc;
    if (n == 0 || n_chunks_ == 0) return AE_MPM_OK;
    if ((rc = settle_order()) || (rc = sync_scatter())) return rc;
    // all substeps are queued before the one wait, so that (past the first) the stream is never
    // idle waiting for the host and the events measure device time, not launch latency
    // per substep: start, after the sort, after P2G, after the grid update, end, and after the
    // G2P (or fused) kernel alone, before the snow clamp (recorded between the last two)
    std::vector<cudaEvent_t> ev(6 * size_t(n), nullptr);
    int rc2 = AE_MPM_OK;
    for (auto& e : ev)
      if (cudaEventCreate(&e) != cudaSuccess) rc2 = AE_MPM_ECUDA;
    if (rc2 == AE_MPM_OK) {
      for (uint32_t i = 0; i < n; ++i) {
        stage_events_ = ev.data() + 6 * size_t(i);
        substep_eager();
      }
      stage_events_ = nullptr;
      if (cudaEventSynchronize(ev[6 * size_t(n - 1) + 4]) != cudaSuccess) rc2 = AE_MPM_ECUDA;
    }
    double acc[6] = {0, 0, 0, 0, 0, 0};
    // the first substep starts on an idle stream: skip it when there is more than one
    const uint32_t first = n > 1 ? 1u : 0u;
    for (uint32_t i = first; i < n && rc2 == AE_MPM_OK; ++i) {
      const cudaEvent_t* e = ev.data() + 6 * size_t(i);
      float ms;
      for (int k = 0; k < 4; ++k) {
        cudaEventElapsedTime(&ms, e[k], e[k + 1]);
        acc[k] += ms;
      }
      cudaEventElapsedTime(&ms, e[0], e[4]);
      acc[4] += ms;
      cudaEventElapsedTime(&ms, e[3], e[5]);
      acc[5] += ms;
    }
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
    if (rc2 != AE_MPM_OK) {
      err = "stage timing events failed";
      return rc2;
    }
    for (int k = 0; k < 6; ++k) out_us[k] = 1000.0 * acc[k] / (n - first);
    return AE_MPM_OK;
  }

 private:
  template <class P>
  cudaError_t dmalloc(P** p, size_t bytes) {
    void* q = nullptr;
    cudaError_t e = alloc_ ? alloc_->alloc(&q, bytes) : cudaMalloc(&q, bytes);
    *p = static_cast<P*>(q);
    return e;
  }
  void dfree(const void* p) {
    if (!p) return;
    if (alloc_)
      alloc_->release(const_cast<void*>(p));
    else
      cudaFree(const_cast<void*>(p));
  }
  static cudaError_t sort_alloc(void* user, void** p, size_t bytes) { return static_cast<DevAlloc*>(user)->alloc(p, bytes); }
  static void sort_free(void* user, void* p) { static_cast<DevAlloc*>(user)->release(p); }

  V4** in_buf() { return a_in_ ? bufA_ : bufB_; }
  V4** out_buf() { return a_in_ ? bufB_ : bufA_; }

  int ensure_stage(uint64_t n) { return ensure_stage_bytes(sizeof(T) * 26 * n + sizeof(uint16_t) * n + 64); }
  int ensure_stage_bytes(size_t need) {
    if (need <= stage_bytes_) return AE_MPM_OK;
    // queued work may still read the old staging area
    AE_TRY(cudaStreamSynchronize(stream_));
    dfree(stage_);
    stage_ = nullptr;
    stage_bytes_ = 0;
    AE_TRY(dmalloc(&stage_, need));
    stage_bytes_ = need;
    return AE_MPM_OK;
  }

  int prepare() {
    if (opts_.block_threads != 128 && opts_.block_threads != 256) opts_.block_threads = 256;
    if (opts_.sort_interval < 1) opts_.sort_interval = 1;
    if (opts_.p2g_variant < kVarTile || opts_.p2g_variant > kVarLanes) opts_.p2g_variant = kVarLanes;
    if (opts_.block_threads != chunk_threads_) {
      chunks_dirty_ = true;
      if (dead_cnt_) keys_stale_ = true;  // counted per chunk
    }
    if (chunks_dirty_) {
      chunk_threads_ = opts_.block_threads;
      h_chunks_.clear();
      chunk_first_.assign(h_scenes_.size() + 1, 0);
      for (size_t s = 0; s < h_scenes_.size(); ++s) {
        chunk_first_[s] = int(h_chunks_.size());
        const SceneDev<T>& h = h_scenes_[s];
        for (uint64_t lo = h.p_off; lo < uint64_t(h.p_off) + h.p_cap; lo += chunk_threads_) {
          uint64_t hl = std::min<uint64_t>(lo + chunk_threads_, uint64_t(h.p_off) + h.p_count);
          uint64_t hc = std::min<uint64_t>(lo + chunk_threads_, uint64_t(h.p_off) + h.p_cap);
          h_chunks_.push_back(make_int4(int(s), int(lo), int(std::max(hl, lo)), int(hc)));
        }
      }
      n_chunks_ = int(h_chunks_.size());
      chunk_first_[h_scenes_.size()] = n_chunks_;
      count_dirty_.assign(h_scenes_.size(), 0);
      any_count_dirty_ = false;
      if (n_chunks_ > 0)
        AE_TRY(cudaMemcpyAsync(d_chunks_, h_chunks_.data(), sizeof(int4) * n_chunks_, cudaMemcpyHostToDevice, stream_));
      drop_graphs();
      chunks_dirty_ = false;
    } else if (any_count_dirty_) {
      // particle counts changed, the chunk layout (by capacity) did not: rewrite those scenes'
      // slices of the chunk table only
      for (size_t s = 0; s < h_scenes_.size(); ++s) {
        if (!count_dirty_[s]) continue;
        const SceneDev<T>& h = h_scenes_[s];
        const int c0 = chunk_first_[s], c1 = chunk_first_[s + 1];
        for (int c = c0; c < c1; ++c) {
          const uint64_t lo = uint64_t(h_chunks_[c].y);
          const uint64_t hl = std::min<uint64_t>(lo + chunk_threads_, uint64_t(h.p_off) + h.p_count);
          h_chunks_[c].z = int(std::max(hl, lo));
        }
        if (c1 > c0)
          AE_TRY(cudaMemcpyAsync(d_chunks_ + c0, h_chunks_.data() + c0, sizeof(int4) * (c1 - c0), cudaMemcpyHostToDevice,
                                 stream_));
        count_dirty_[s] = 0;
      }
      any_count_dirty_ = false;
      drop_graphs();  // a one-scene world's graphs carry the count in their launch parameters
    }
    int rc = sync_tables();
    if (rc) return rc;
    // the tables are copied from pageable host memory, which the copy stages before returning
    return AE_MPM_OK;
  }

  // scene and material tables to the device (copied from pageable memory, staged at the call)
  int sync_tables() {
    if (scenes_dirty_) {
      const size_t lo = std::min(scene_lo_, h_scenes_.size()), hi = std::min(scene_hi_, h_scenes_.size());
      if (hi > lo)
        AE_TRY(cudaMemcpyAsync(d_scenes_ + lo, h_scenes_.data() + lo, sizeof(SceneDev<T>) * (hi - lo),
                               cudaMemcpyHostToDevice, stream_));
      scenes_dirty_ = false;
      scene_lo_ = SIZE_MAX;
      scene_hi_ = 0;
    }
    if (mats_dirty_) {
      const size_t lo = std::min(mat_lo_, h_mats_.size()), hi = std::min(mat_hi_, h_mats_.size());
      if (hi > lo)
        AE_TRY(cudaMemcpyAsync(d_mats_ + lo, h_mats_.data() + lo, sizeof(MatDev) * (hi - lo), cudaMemcpyHostToDevice,
                               stream_));
      mats_dirty_ = false;
      mat_lo_ = SIZE_MAX;
      mat_hi_ = 0;
    }
    return AE_MPM_OK;
  }

  WorldDev<T> dev(bool sorted) {
    WorldDev<T> w{};
    w.scenes = d_scenes_;
    w.mats = d_mats_;
    w.chunks = d_chunks_;
    if (h_scenes_.size() == 1) {
      const SceneDev<T>& h = h_scenes_[0];
      w.one_scene = 1u;
      w.one_off = h.p_off;
      w.one_live_end = h.p_off + h.p_count;
      w.one_cap_end = h.p_off + h.p_cap;
    }
    for (int k = 0; k < 7; ++k) {
      w.in[k] = in_buf()[k];
      w.out[k] = out_buf()[k];
    }
    w.perm = sorted ? perm_ : nullptr;
    w.keys = keys_;
    w.bins = bins_;
    w.bin_off = bin_off_;
    w.seg_off = seg_ ? seg_ + n_segs_ : nullptr;
    w.cells = cells_;
    w.dead_cnt = mode_ == AE_MPM_MODE_PHYSICS ? nullptr : dead_cnt_;
    w.acc = acc_;
    w.vel = vel_;
    w.blk_flag = blk_flag_;
    w.touched = touched_;
    w.touched_count = counters_;
    w.blk_scene = blk_scene_;
    w.err = err_;
    w.svd_fallback = opts_.svd_fp64_fallback;
    w.max_tile_nodes = max_tile_nodes();
    w.sorted_keys = sorted ? sorted_keys_ : nullptr;
    w.cell_slot = cell_slot_;
    w.cell_rec = cell_rec_;
    w.cell_count = opts_.deterministic ? counters_ + 1 : nullptr;
    w.seg_start = seg_start_;
    w.clamp_queue = clamp_queue_;
    w.clamp_count = counters_ + 3;
    return w;
  }

  int max_tile_nodes() const { return sizeof(T) == 4 ? 1024 : 512; }

  void launch_init_keys(WorldDev<T>& w) {
    if (n_chunks_ == 0) return;
    switch (mode_) {
      case AE_MPM_MODE_PHYSICS: init_keys_kernel<T, AE_MPM_MODE_PHYSICS><<<n_chunks_, chunk_threads_, 0, stream_>>>(w); break;
      case AE_MPM_MODE_REFERENCE: init_keys_kernel<T, AE_MPM_MODE_REFERENCE><<<n_chunks_, chunk_threads_, 0, stream_>>>(w); break;
      default: init_keys_kernel<T, AE_MPM_MODE_VELOCITY_ONLY><<<n_chunks_, chunk_threads_, 0, stream_>>>(w); break;
    }
    ++launches_;
  }

  void launch_p2g_lanes(WorldDev<T>& w, int chunks) {
    const size_t per = sizeof(V4) * kLaneVecs + sizeof(int4);
    if (!lanes_smem_set_) {  // sized for the largest block (256 threads) the world accepts
      cudaFuncSetAttribute(p2g_lanes_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(per * 256));
      lanes_smem_set_ = true;
    }
    p2g_lanes_kernel<T><<<chunks, chunk_threads_, per * chunk_threads_, stream_>>>(w);
  }

  template <int MODE>
  void launch_p2g(WorldDev<T>& w) {
    const size_t sm = sizeof(V4) * max_tile_nodes();
    if (MODE == AE_MPM_MODE_PHYSICS && opts_.p2g_variant == kVarLanes) {
      launch_p2g_lanes(w, n_chunks_);
      return;
    }
    if (MODE == AE_MPM_MODE_REFERENCE && opts_.p2g_variant == kVarLanes) {
      const size_t per = sizeof(V4) * kRefLaneVecs + sizeof(int4);
      if (!ref_lanes_smem_set_) {  // sized for the largest block (256 threads) the world accepts
        for (auto fn : {p2g_lanes_ref_kernel<T, 8>, p2g_lanes_ref_kernel<T, 32>})
          cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(per * 256));
        ref_lanes_smem_set_ = true;
      }
      // one CTA of 256 threads per SM (shared memory): 8 particles per warp while all of them run at once
      if (total_cap_ <= uint64_t(device_sm_count()) * 128)
        p2g_lanes_ref_kernel<T, 8><<<n_chunks_ * 4, chunk_threads_, per * chunk_threads_, stream_>>>(w);
      else
        p2g_lanes_ref_kernel<T, 32><<<n_chunks_, chunk_threads_, per * chunk_threads_, stream_>>>(w);
      return;
    }
    if (MODE == AE_MPM_MODE_VELOCITY_ONLY && opts_.p2g_variant == kVarLanes) {
      p2g_lanes_velonly_kernel<T><<<n_chunks_, chunk_threads_, velonly_lane_bytes<T>() * chunk_threads_, stream_>>>(w);
      return;
    }
    switch (opts_.p2g_variant) {
      case kVarWarpAgg: p2g_kernel<T, MODE, kVarWarpAgg><<<n_chunks_, chunk_threads_, sm, stream_>>>(w); break;
      case kVarGlobal: p2g_kernel<T, MODE, kVarGlobal><<<n_chunks_, chunk_threads_, 0, stream_>>>(w); break;
      default: p2g_kernel<T, MODE, kVarTile><<<n_chunks_, chunk_threads_, sm, stream_>>>(w); break;
    }
  }

  template <int MODE>
  void substep_mode(WorldDev<T>& w, bool write_keys) {
    const int sms = device_sm_count();
    if (opts_.deterministic && dense_sort_) {
      const size_t sm = sizeof(CellStage<T, MODE>) * size_t(chunk_threads_ / 32);
      if (!det_smem_set_) {  // sized for the largest block (256 threads) the world accepts
        cudaFuncSetAttribute(det_cells_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(sizeof(CellStage<T, MODE>) * 8));
        det_smem_set_ = true;
      }
      det_cells_kernel<T, MODE><<<n_chunks_, chunk_threads_, sm, stream_>>>(w, bin_perm_, ordered_);
      det_gather_kernel<T, MODE><<<sms * 8, 256, 0, stream_>>>(w, blk_epoch_, counters_ + 2);
      mark(2);
      launches_ += 2;
    } else if (opts_.deterministic) {
      det_heads_kernel<<<unsigned((total_cap_ + 255) / 256), 256, 0, stream_>>>(w.sorted_keys, total_cap_, dead_blk_,
                                                                                 cell_slot_, seg_start_, counters_ + 1);
      det_cellsum_kernel<T, MODE><<<sms * 8, 128, 0, stream_>>>(w, total_cap_);
      det_gather_kernel<T, MODE><<<sms * 8, 256, 0, stream_>>>(w, blk_epoch_, counters_ + 2);
      mark(2);
      det_reset_kernel<<<sms * 4, 256, 0, stream_>>>(seg_start_, w.sorted_keys, counters_ + 1, cell_slot_);
      launches_ += 4;
    } else {
      launch_p2g<MODE>(w);
      mark(2);
      grid_update_kernel<T, MODE><<<sms * 4, 256, 0, stream_>>>(w, blk_epoch_, counters_ + 2, nullptr);
      launches_ += 2;
    }
    mark(3);
    const size_t g2p_smem = sizeof(V4) * ((MODE == AE_MPM_MODE_PHYSICS ? 0 : max_tile_nodes()) + 3 * chunk_threads_);
    // node loads ahead of their use in the reference mode while a CTA of 256 threads per SM holds all slots
    const bool ahead = MODE == AE_MPM_MODE_REFERENCE && total_cap_ <= uint64_t(sms) * 256;
    const auto g2p = ahead ? g2p_kernel<T, MODE, MODE == AE_MPM_MODE_REFERENCE> : g2p_kernel<T, MODE, false>;
    g2p<<<n_chunks_, chunk_threads_, g2p_smem, stream_>>>(w, counters_ + 2, write_keys ? 1 : 0);
    ++launches_;
    mark(5);  // the G2P kernel alone ends here
    if (MODE == AE_MPM_MODE_PHYSICS && has_snow_) {
      snow_clamp_kernel<T><<<sms * 8, 128, 0, stream_>>>(w);
      ++launches_;
    }
    mark(4);
  }

  void mark(int k) {
    if (stage_events_) cudaEventRecord(stage_events_[k], stream_);
  }

  // ranges of the scene and material tables to copy to the device before the next launch
  void dirty_scene(size_t s) {
    scene_lo_ = std::min(scene_lo_, s);
    scene_hi_ = std::max(scene_hi_, s + 1);
    scenes_dirty_ = true;
  }
  void dirty_mats(size_t s) {
    const size_t lo = h_scenes_[s].mat_off, hi = lo + descs_[s].n_materials + 1;
    mat_lo_ = std::min(mat_lo_, lo);
    mat_hi_ = std::max(mat_hi_, hi);
    mats_dirty_ = true;
  }

  void count_changed(uint32_t s) {
    dirty_scene(s);
    if (count_dirty_.size() != h_scenes_.size()) {
      chunks_dirty_ = true;  // no table yet: the next prepare() builds it whole
      return;
    }
    count_dirty_[s] = 1;
    any_count_dirty_ = true;
  }

  // ---- fused G2P + P2G (physics mode, column-lane P2G, not deterministic) ----
  // The P2G of substep s + 1 is done by the G2P of substep s, so between substeps the grid
  // accumulator holds the scatter of the current particle state ("queued"), on touched list
  // (s + 1) & 1.  Anything that changes the particles or the flow drops it; the next step()
  // scatters the current state once with the stand-alone P2G before its first substep.
  bool fused() const {
    return mode_ == AE_MPM_MODE_PHYSICS && !opts_.deterministic && opts_.p2g_variant == kVarLanes;
  }
  uint32_t* touched_list(int par) { return touched_ + size_t(par) * total_blocks_; }
  uint32_t* touched_count(int par) { return counters_ + (par ? 4 : 0); }
  WorldDev<T> with_list(WorldDev<T> w, int par) {
    w.touched = touched_list(par);
    w.touched_count = touched_count(par);
    return w;
  }
  static size_t fused_smem(int threads) { return warp_stage_bytes<T>() * size_t(threads / 32); }

  int sync_scatter() {
    const int par = int(substep_ & 1);
    if (fused() && !fused_smem_set_) {  // sized for the largest block (256 threads) the world accepts
      for (auto fn : {g2p2g_kernel<T, false, 8>, g2p2g_kernel<T, false, 16>, g2p2g_kernel<T, false, 32>,
                      g2p2g_kernel<T, true, 32>})
        AE_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(fused_smem(256))));
      AE_TRY(cudaFuncSetAttribute(snow_clamp_scatter_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(fused_smem(128))));
      fused_smem_set_ = true;
    }
    if (scatter_pending_ && (!fused() || scatter_invalid_)) {
      discard_scatter_kernel<T><<<device_sm_count() * 8, 64, 0, stream_>>>(acc_, blk_flag_, touched_list(par),
                                                                            touched_count(par));
      AE_TRY(cudaMemsetAsync(counters_, 0, sizeof(uint32_t), stream_));
      AE_TRY(cudaMemsetAsync(counters_ + 4, 0, sizeof(uint32_t), stream_));
      ++launches_;
      scatter_pending_ = false;
    }
    scatter_invalid_ = false;
    // In cell order: particles as the caller stored them would each be a run of their own, 27 vector
    // reductions per particle instead of per cell and warp (dam break, 8.4 M particles in random
    // order: 7.3 ms of P2G against 0.8 with the sort the first substep does anyway).
    if (fused() && !scatter_pending_ && n_chunks_ > 0) {
      if (phase_ == 0 && !sorted_) sort_particles();
      AE_TRY(cudaMemsetAsync(touched_count(par), 0, sizeof(uint32_t), stream_));
      WorldDev<T> w = with_list(dev(sorted_), par);
      launch_p2g<AE_MPM_MODE_PHYSICS>(w);
      ++launches_;
      scatter_pending_ = true;
    } else if (fused() && !late_slots_.empty()) {  // only the slots assigned since the last step
      if (phase_ == 0 && !sorted_) sort_particles();
      for (uint32_t s : late_slots_) {
        const int c0 = chunk_first_[s], c1 = chunk_first_[s + 1];
        if (c1 == c0 || h_scenes_[s].p_count == 0) continue;
        WorldDev<T> w = with_list(dev(sorted_), par);
        if (!w.one_scene) w.chunks = d_chunks_ + c0;
        launch_p2g_lanes(w, c1 - c0);
        ++launches_;
      }
    }
    late_slots_.clear();
    AE_TRY(cudaGetLastError());
    return AE_MPM_OK;
  }

  // The fused kernel of this world: without the snow code where no material needs it, and with fewer
  // particles per warp where the warps are too few to hide one another's latency (a warp sums its
  // runs one after another).  Water at 8 per cell, us per substep with 32 / 16 / 8 per warp: 2 309
  // particles 16.8 / 15.4 / 14.6, 9 000 17.9 / 16.5 / 15.6, 24 000 18.4 / 17.9 / 18.5, 40 000 22.6 /
  // 20.2 / 24.5, 64 000 20.2 / 21.7 / 26.9: 8 up to 10 such warps per SM, 16 up to 20.  With snow's
  // return mapping in the warp 32 is the fastest from 4 600 particles on (27.6 / 30.3 / 32.7).
  struct FusedKernel {
    void (*fn)(WorldDev<T>, uint32_t*, int);
    int per;
  };
  FusedKernel fused_kernel() const {
    const uint64_t sms = uint64_t(device_sm_count());
    if (has_snow_) return {g2p2g_kernel<T, true, 32>, 32};
    if (total_cap_ <= sms * 80) return {g2p2g_kernel<T, false, 8>, 8};
    if (total_cap_ <= sms * 320) return {g2p2g_kernel<T, false, 16>, 16};
    return {g2p2g_kernel<T, false, 32>, 32};
  }

  // A small kernel between the fused ones.  In a world whose particles fit the GPU at once it may start
  // while its predecessor drains; in a larger one, whose CTAs fill the GPU anyway, early CTAs would
  // only hold room that other streams' worlds can use.  (The fused kernel itself starts after the
  // others: early CTAs crowd on the first free SMs, 9.3 -> 18 us for 128 CTAs.)
  template <class... P, class... A>
  void launch_dependent(void (*kernel)(P...), unsigned ctas, unsigned threads, size_t smem, A&&... args) {
    launch_after(total_cap_ <= uint64_t(device_sm_count()) * 1024, kernel, ctas, threads, smem, stream_,
                 std::forward<A>(args)...);
    ++launches_;
  }

  // sort_first: the substep starts with the sort, whose keys and counts are there
  void substep_fused(bool sort_first, bool write_keys) {
    const unsigned sms = unsigned(device_sm_count());
    const int par = int(substep_ & 1);
    mark(2);  // no stand-alone P2G: the previous substep's G2P scattered this one
    WorldDev<T> wg = with_list(dev(sorted_), par);
    if (sort_first) {
      launch_dependent(scan_and_grid_kernel<T>, n_segs_ + sms * 4, kBinThreads, 0, wg, total_blocks_ * 64, dead_blk_,
                       seg_, counters_ + 5, n_segs_, blk_epoch_, counters_ + 2, touched_count(par ^ 1));
      launch_dependent(bin_scatter_kernel<T, false>, unsigned(n_chunks_), unsigned(chunk_threads_), 0, wg, bin_perm_,
                       uint32_t(total_cap_));
      perm_ = bin_perm_;
      sorted_ = true;
      keys_fresh_ = false;
    } else {
      launch_dependent(grid_update_kernel<T, AE_MPM_MODE_PHYSICS>, sms * 4, 256, 0, wg, blk_epoch_, counters_ + 2,
                       touched_count(par ^ 1));
    }
    mark(3);
    WorldDev<T> wf = with_list(dev(sorted_), par ^ 1);
    const FusedKernel k = fused_kernel();
    k.fn<<<unsigned(n_chunks_) * (32 / k.per), unsigned(chunk_threads_), fused_smem(chunk_threads_), stream_>>>(
        wf, counters_ + 2, write_keys ? 1 : 0);
    ++launches_;
    mark(5);  // the fused kernel alone ends here
    if (has_snow_) {
      snow_clamp_scatter_kernel<T><<<sms * 6, 128, fused_smem(128), stream_>>>(wf, write_keys ? 1 : 0);
      ++launches_;
    }
    mark(4);
  }

  uint32_t sort_interval() const { return opts_.deterministic ? 1u : uint32_t(opts_.sort_interval); }

  // The particles changed since their order was established (upload, scene change, ...): the next
  // substep sorts, and the sort interval counts from there, so a run never starts on particles in
  // the caller's order.
  int settle_order() {
    if (phase_ >= sort_interval()) phase_ = 0;  // the interval was shortened
    if (!keys_stale_) return AE_MPM_OK;
    // cells counted for the dropped state
    if (dense_sort_ && keys_fresh_) AE_TRY(cudaMemsetAsync(bins_, 0, sizeof(uint32_t) * 64 * total_blocks_, stream_));
    keys_stale_ = keys_fresh_ = sorted_ = false;
    phase_ = 0;
    return AE_MPM_OK;
  }

  // perm_: sorted position -> storage slot of the current particle state
  void sort_particles() {
    if (!keys_fresh_) {
      WorldDev<T> wk = dev(false);
      launch_init_keys(wk);
    }
    if (dense_sort_) {
      WorldDev<T> w = dev(false);
      bin_scan_kernel<T><<<n_segs_, kBinThreads, 0, stream_>>>(w, total_blocks_ * 64, dead_blk_, seg_, counters_ + 5);
      const auto scatter = w.dead_cnt ? bin_scatter_kernel<T, true> : bin_scatter_kernel<T, false>;
      scatter<<<n_chunks_, chunk_threads_, 0, stream_>>>(w, bin_perm_, uint32_t(total_cap_));
      // a deterministic substep orders each cell (det_cells_kernel) before anything reads the order
      perm_ = opts_.deterministic ? ordered_ : bin_perm_;
      launches_ += 2;
    } else {
      launches_ += radix_sort_pairs(keys_, total_cap_, key_bits_, sort_, stream_, &sorted_keys_, &perm_);
    }
    keys_fresh_ = false;  // the counts (or the keys) are used up
    sorted_ = true;
  }

  void substep_eager(bool last = false) {
    // the keys of the next sort are written by the G2P just before it; a sort without them (first
    // substep, changed interval) computes them first.  Only the fused G2P counts cells too.
    const uint32_t next = phase_ + 1 >= sort_interval() ? 0u : phase_ + 1;
    const bool write_keys = next == 0 && (!dense_sort_ || fused() || opts_.deterministic || !last);
    if (n_chunks_ > 0) {
      mark(0);
      const bool sort_now = phase_ == 0 && !sorted_;
      // the scan shares its launch with the grid update, except where stages are timed one by one
      const bool joined = sort_now && fused() && dense_sort_ && keys_fresh_ && !stage_events_;
      if (sort_now && !joined) sort_particles();
      mark(1);
      WorldDev<T> w = dev(sorted_);
      switch (mode_) {
        case AE_MPM_MODE_PHYSICS:
          if (fused())
            substep_fused(joined, write_keys);
          else
            substep_mode<AE_MPM_MODE_PHYSICS>(w, write_keys);
          break;
        case AE_MPM_MODE_REFERENCE: substep_mode<AE_MPM_MODE_REFERENCE>(w, write_keys); break;
        default: substep_mode<AE_MPM_MODE_VELOCITY_ONLY>(w, write_keys); break;
      }
      keys_fresh_ = write_keys;
      sorted_ = false;
      a_in_ = !a_in_;
    }
    phase_ = next;
    ++substep_;
  }

  // What a graph starts from, once the phase is 0: particles in order (their sort ran for the first scatter
  // after an upload), their keys and cell counts written by the substep before, or neither.  The sort is
  // then part of the graph: two launches and a wait for them before each period took 4 us (20 000 particles
  // sorted every 4th substep: 16.4 -> 14.4 us a substep).
  enum { kEntrySorted, kEntryFresh, kEntryBare, kEntries };
  int graph_entry() const { return sorted_ ? kEntrySorted : (keys_fresh_ ? kEntryFresh : kEntryBare); }
  // With a sort every substep the one substep that starts in order runs on its own, without a graph of
  // its own.
  bool graph_now() const { return !(sort_interval() == 1 && fused() && dense_sort_ && sorted_); }

  // A graph holds one period of substeps: lcm(2, sort interval), since buffers and touched lists
  // alternate.  A period may start on either parity (the interval counts from the last upload), so
  // there is one graph for each and for what it starts from.
  int ensure_graph(uint32_t period) {
    Graph& gr = graphs_[substep_ & 1][graph_entry()];
    if (gr.exec && gr.period == period && gr.variant == opts_.p2g_variant && gr.a_in == a_in_) return AE_MPM_OK;
    if (gr.exec) {
      cudaGraphExecDestroy(gr.exec);
      gr.exec = nullptr;
    }
    const bool a_in0 = a_in_;
    const uint64_t sub0 = substep_, l0 = launches_;
    AE_TRY(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
    const bool sorted0 = sorted_, fresh0 = keys_fresh_;
    for (uint32_t k = 0; k < period; ++k) substep_eager();
    gr.sorted_out = sorted_;
    gr.fresh_out = keys_fresh_;
    sorted_ = sorted0;
    keys_fresh_ = fresh0;
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(stream_, &g);
    a_in_ = a_in0;
    substep_ = sub0;
    gr.launches = launches_ - l0;
    launches_ = l0;
    if (e != cudaSuccess) {
      err = std::string("stream capture failed: ") + cudaGetErrorString(e);
      return AE_MPM_ECUDA;
    }
    e = cudaGraphInstantiate(&gr.exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
      err = std::string("graph instantiation failed: ") + cudaGetErrorString(e);
      gr.exec = nullptr;
      return AE_MPM_ECUDA;
    }
    gr.period = period;
    gr.variant = opts_.p2g_variant;
    gr.a_in = a_in0;
    return AE_MPM_OK;
  }
  void drop_graphs() {
    for (auto& by_entry : graphs_)
      for (Graph& g : by_entry) {
        if (g.exec) cudaGraphExecDestroy(g.exec);
        g.exec = nullptr;
      }
  }

  void release() {
    drop_graphs();
    if (stream_) cudaStreamSynchronize(stream_);
    if (xfer_ev_) cudaEventDestroy(xfer_ev_);
    for (int k = 0; k < 7; ++k) dfree(snap_[k]);
    sort_scratch_free(sort_, alloc_ ? &World::sort_free : nullptr, alloc_);
    dfree(arena_);
    dfree(partial_);
    dfree(stage_);
    if (stream_) cudaStreamDestroy(stream_);
  }

 public:
  DevAlloc* alloc_ = nullptr;
  unsigned char* arena_ = nullptr;  // the world's arrays
  int mode_ = 0;
  ae_mpm_exec_opts opts_{};
  std::vector<ae_mpm_scene_desc> descs_;
  std::vector<std::vector<ae_mpm_material>> mats_;
  std::vector<SceneDev<T>> h_scenes_;
  std::vector<MatDev> h_mats_;
  std::vector<int4> h_chunks_;
  std::vector<int> chunk_first_;  // first chunk of each scene (and the chunk count at the end)
  std::vector<uint8_t> count_dirty_;  // scenes whose particle count changed since the table was written
  bool any_count_dirty_ = false;
  SceneDev<T>* d_scenes_ = nullptr;
  MatDev* d_mats_ = nullptr;
  int4* d_chunks_ = nullptr;
  int n_chunks_ = 0, n_chunks_alloc_ = 0, chunk_threads_ = 0;
  V4* bufA_[7] = {};
  V4* bufB_[7] = {};
  V4* snap_[7] = {};
  bool a_in_ = true;
  uint32_t* keys_ = nullptr;
  SortScratch sort_;
  bool dense_sort_ = false;  // particles are grouped by counting (bins_), not by the radix sort
  uint32_t *bins_ = nullptr, *bin_off_ = nullptr, *seg_ = nullptr, *bin_perm_ = nullptr;
  uint2* cells_ = nullptr;        // deterministic dense grouping: each cell's places
  uint32_t* dead_cnt_ = nullptr;  // ... the off-grid particles of each chunk
  uint32_t* ordered_ = nullptr;   // ... and the sorted places in slot order within each cell
  uint32_t n_segs_ = 0;
  const uint32_t* perm_ = nullptr;
  const uint32_t* sorted_keys_ = nullptr;
  V4* acc_ = nullptr;
  V4* vel_ = nullptr;
  uint32_t *blk_flag_ = nullptr, *blk_epoch_ = nullptr, *touched_ = nullptr, *blk_scene_ = nullptr, *dead_blk_ = nullptr;
  uint32_t* counters_ = nullptr;  // [touched count, cell count, epoch, snow clamp queue count]
  uint32_t* err_ = nullptr;
  uint32_t *cell_slot_ = nullptr, *seg_start_ = nullptr;
  V4* cell_rec_ = nullptr;
  uint2* clamp_queue_ = nullptr;
  bool has_snow_ = false;
  T* stage_ = nullptr;
  size_t stage_bytes_ = 0;
  std::vector<XferDev<T>> h_xfer_;  // many-scene transfer table
  XferDev<T>* d_xfer_ = nullptr;
  double* partial_ = nullptr;
  cudaStream_t stream_ = nullptr;
  struct Graph {
    cudaGraphExec_t exec = nullptr;
    uint32_t period = 0;
    uint64_t launches = 0;
    int variant = -1;
    bool a_in = true;
    bool sorted_out = false, fresh_out = false;  // the world's state after it
  };
  Graph graphs_[2][kEntries];  // by the parity of the period's first substep and what it starts from
  bool lanes_smem_set_ = false, fused_smem_set_ = false, ref_lanes_smem_set_ = false, det_smem_set_ = false;
  bool scatter_pending_ = false;  // the accumulator holds the P2G of the current particle state
  bool scatter_invalid_ = false;  // the particles changed since that scatter
  std::vector<uint32_t> late_slots_;  // slots assigned into a queued scatter, not scattered themselves yet
  uint64_t substep_ = 0, snap_substep_ = 0, launches_ = 0;
  cudaEvent_t* stage_events_ = nullptr;
  cudaEvent_t xfer_ev_ = nullptr;  // orders copy streams against the world's stream
  uint64_t total_cap_ = 0, total_blocks_ = 0, device_bytes_ = 0;
  int key_bits_ = 1;
  bool keys_stale_ = true, chunks_dirty_ = true, scenes_dirty_ = true, mats_dirty_ = false;
  size_t scene_lo_ = 0, scene_hi_ = SIZE_MAX;  // dirty range of the scene table (all of it at first)
  size_t mat_lo_ = SIZE_MAX, mat_hi_ = 0;       // dirty range of the material table
  bool keys_fresh_ = false;  // keys_ (and the cell counts) are those of the current positions
  bool sorted_ = false;      // perm_ orders the current particle state
  uint32_t phase_ = 0;       // substeps since the last sort was due
};

uint64_t scene_device_bytes(const ae_mpm_scene_desc& d, const ae_mpm_exec_opts& opts) {
  return opts.precision == 64 ? World<double>::device_bytes_of(d, opts.deterministic != 0)
                              : World<float>::device_bytes_of(d, opts.deterministic != 0);
}

WorldBase* make_world(const ae_mpm_scene_desc* scenes, uint32_t n_scenes, const ae_mpm_exec_opts& opts, std::string& why,
                      int* status, DevAlloc* alloc) {
  size_t free0 = 0, total = 0;
  cudaMemGetInfo(&free0, &total);
  WorldBase* w = nullptr;
  int rc;
  if (opts.precision == 64) {
    auto* x = new World<double>();
    x->alloc_ = alloc;
    rc = x->init(scenes, n_scenes, opts);
    w = x;
  } else {
    auto* x = new World<float>();
    x->alloc_ = alloc;
    rc = x->init(scenes, n_scenes, opts);
    w = x;
  }
  if (rc != AE_MPM_OK) {
    why = w->err;
    delete w;
    if (status) *status = rc;
    return nullptr;
  }
  size_t free1 = 0;
  cudaMemGetInfo(&free1, &total);
  if (opts.precision == 64)
    static_cast<World<double>*>(w)->device_bytes_ = free0 > free1 ? free0 - free1 : 0;
  else
    static_cast<World<float>*>(w)->device_bytes_ = free0 > free1 ? free0 - free1 : 0;
  if (status) *status = AE_MPM_OK;
  return w;
}

}  // namespace aemp
