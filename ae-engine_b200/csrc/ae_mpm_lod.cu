// ae_mpm_lod.cu -- the engine tick's particle passes around the MPM substep, on the device
// (ae_engine/src/managers/simulation.rs).  Every pass restates the reference's f32 arithmetic
// operation by operation with explicitly rounded intrinsics (__fmul_rn / __fadd_rn / __fdiv_rn are
// never fused into FMAs), so results match the CPU path bit for bit:
//
//   classify      stable 3-way partition of the particles by squared distance to the player
//                 (count per 2048-particle tile, scan of the tile counts, scatter in index order).
//                 When more than max_near fall within near_dist, a one-block radix select over
//                 the near candidates' squared distances (non-negative floats, so their bit patterns
//                 order like the values) flags the max_near closest, and a second partition splits
//                 the candidates into the kept near list and the tail appended to the mid list.
//   far_field     one thread per far particle: gravity on y, position, nearest-cell sample.
//   coarse_field  the near particles' cells are radix-sorted (stable, so each cell keeps the
//                 reference's index order), each cell's run is located, and one lane per cell
//                 sums its run sequentially, which reproduces the reference's serial accumulation
//                 exactly, and relaxes the cell; then one FTCS step, one thread per cell.
#include "ae_mpm_lod.cuh"

#include <algorithm>
#include <cmath>

#include "device_util.cuh"

namespace aemp {

namespace {

constexpr int kPT = 256, kPItems = 8, kPTile = kPT * kPItems;  // partition: 2048 items per tile
constexpr int kPWarps = kPT / 32;

__device__ __forceinline__ int64_t as_isize(float v) {  // Rust `f32 as isize`
  if (v != v) return 0;
  if (v >= 9.2233720368547758e18f) return INT64_MAX;
  if (v <= -9.2233720368547758e18f) return INT64_MIN;
  return static_cast<int64_t>(v);
}

// class of particle idx: 0 near, 1 mid, 2 far, 3 skipped (inactive); simulation.rs:499-513
struct PosClass {
  const float* pos;
  const uint8_t* active;
  float px, py, pz, near2, mid2;
  __device__ __forceinline__ int operator()(uint64_t idx, uint64_t& item, float& d2) const {
    item = idx;
    const bool on = !active || active[idx];
    const float dx = __fsub_rn(pos[3 * idx], px), dy = __fsub_rn(pos[3 * idx + 1], py), dz = __fsub_rn(pos[3 * idx + 2], pz);
    d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    return !on ? 3 : (d2 < near2 ? 0 : (d2 < mid2 ? 1 : 2));  // NaN compares false: far
  }
};

// near candidate k: 0 kept, 1 culled to mid
struct KeepClass {
  const uint64_t* near;
  const uint8_t* keep;  // null: none is kept
  __device__ __forceinline__ int operator()(uint64_t k, uint64_t& item, float& d2) const {
    item = near[k];
    d2 = 0.0f;
    return keep && keep[k] ? 0 : 1;
  }
};

// The items of a partition: n, or *n_dev where an earlier kernel found it, none of them up to `cap`
// (the near candidates are where they belong then).  CTAs without items leave at once.
struct Items {
  uint64_t n;
  const uint32_t* n_dev;
  uint32_t cap;
  __device__ __forceinline__ uint64_t count() const {
    if (!n_dev) return n;
    const uint32_t v = *n_dev;
    return v > cap ? v : 0u;
  }
};

template <class Cls>
__global__ void __launch_bounds__(kPT) part_count(Cls cls, Items items, uint32_t* tile_counts, uint32_t tiles) {
  __shared__ uint32_t wc[kPWarps][3];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  let_next_start();
  dependency_wait();
  const uint64_t n = items.count();
  if (uint64_t(blockIdx.x) * kPTile >= n) return;
  const uint64_t base = uint64_t(blockIdx.x) * kPTile + uint64_t(w) * (32 * kPItems);
  uint32_t c0 = 0, c1 = 0, c2 = 0;
  int k[kPItems];
#pragma unroll
  for (int r = 0; r < kPItems; ++r) {  // no branch or vote between the 8 items' loads (1 M: 5.9 -> 3.7 us)
    const uint64_t idx = base + uint64_t(r) * 32 + lane;
    uint64_t item;
    float d2;
    k[r] = cls(min(idx, n - 1), item, d2);
    if (idx >= n) k[r] = 3;
  }
#pragma unroll
  for (int r = 0; r < kPItems; ++r) {
    c0 += __popc(__ballot_sync(0xffffffffu, k[r] == 0));
    c1 += __popc(__ballot_sync(0xffffffffu, k[r] == 1));
    c2 += __popc(__ballot_sync(0xffffffffu, k[r] == 2));
  }
  if (lane == 0) {
    wc[w][0] = c0;
    wc[w][1] = c1;
    wc[w][2] = c2;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    uint32_t s = 0;
    for (int ww = 0; ww < kPWarps; ++ww) s += wc[ww][threadIdx.x];
    tile_counts[uint64_t(threadIdx.x) * tiles + blockIdx.x] = s;
  }
}

// one block: exclusive scan of the three classes' tile counts together, and the class totals
__global__ void __launch_bounds__(1024) part_scan(const uint32_t* tile_counts, uint32_t* tile_offs, uint32_t tiles,
                                                  Items items, uint32_t* totals) {
  __shared__ uint32_t ws[3][32];
  __shared__ uint32_t carry[3];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  let_next_start();
  dependency_wait();
  const uint32_t used = uint32_t((items.count() + kPTile - 1) / kPTile);
  if (tid < 3) carry[tid] = 0;
  __syncthreads();
  for (uint32_t start = 0; start < used; start += 1024) {
    const uint32_t i = start + tid;
    uint32_t x[3], incl[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) x[c] = i < used ? tile_counts[uint64_t(c) * tiles + i] : 0u;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      incl[c] = warp_scan_incl(x[c], lane);
      if (lane == 31) ws[c][w] = incl[c];
    }
    __syncthreads();
    if (w < 3) {
      const uint32_t v = ws[w][lane];
      ws[w][lane] = warp_scan_incl(v, lane) - v;
    }
    __syncthreads();
    uint32_t at[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      at[c] = carry[c] + ws[c][w] + incl[c];
      if (i < used) tile_offs[uint64_t(c) * tiles + i] = at[c] - x[c];
    }
    __syncthreads();
    if (tid == 1023)
      for (int c = 0; c < 3; ++c) carry[c] = at[c];
    __syncthreads();
  }
  if (tid < 3) totals[tid] = carry[tid];
}

// writes each item at its class's tile offset + rank in index order; class 1 lands at *out1_from +
// position.  The first cap0 items of class 0 go to out0 (nothing is written past them), all of them
// optionally to a second list, with their squared distances to a third
template <class Cls>
__global__ void __launch_bounds__(kPT) part_scatter(Cls cls, Items items, const uint32_t* tile_offs,
                                                    uint32_t tiles, uint64_t* out0, uint64_t* all0, uint32_t cap0, float* d2_0,
                                                    uint64_t* out1, const uint32_t* out1_from, uint64_t* out2) {
  __shared__ uint32_t wc[kPWarps][3];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  let_next_start();
  dependency_wait();
  const uint64_t n = items.count();
  if (uint64_t(blockIdx.x) * kPTile >= n) return;
  const uint64_t out1_base = out1_from ? *out1_from : 0;
  const uint64_t base = uint64_t(blockIdx.x) * kPTile + uint64_t(w) * (32 * kPItems);
  int k[kPItems];
  uint64_t item[kPItems];
  float d2[kPItems];
  uint32_t c0 = 0, c1 = 0, c2 = 0;
#pragma unroll
  for (int r = 0; r < kPItems; ++r) {
    const uint64_t idx = base + uint64_t(r) * 32 + lane;
    k[r] = cls(min(idx, n - 1), item[r], d2[r]);
    if (idx >= n) k[r] = 3;
  }
#pragma unroll
  for (int r = 0; r < kPItems; ++r) {
    c0 += __popc(__ballot_sync(0xffffffffu, k[r] == 0));
    c1 += __popc(__ballot_sync(0xffffffffu, k[r] == 1));
    c2 += __popc(__ballot_sync(0xffffffffu, k[r] == 2));
  }
  if (lane == 0) {
    wc[w][0] = c0;
    wc[w][1] = c1;
    wc[w][2] = c2;
  }
  __syncthreads();
  uint32_t wb[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    uint32_t s = tile_offs[uint64_t(q) * tiles + blockIdx.x];
    for (int ww = 0; ww < w; ++ww) s += wc[ww][q];
    wb[q] = s;
  }
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < kPItems; ++r) {
    const uint32_t m0 = __ballot_sync(0xffffffffu, k[r] == 0);
    const uint32_t m1 = __ballot_sync(0xffffffffu, k[r] == 1);
    const uint32_t m2 = __ballot_sync(0xffffffffu, k[r] == 2);
    if (k[r] == 0) {
      const uint32_t p = wb[0] + __popc(m0 & lt);
      if (p < cap0) out0[p] = item[r];
      if (all0) all0[p] = item[r];
      if (d2_0) d2_0[p] = d2[r];
    } else if (k[r] == 1) {
      out1[out1_base + wb[1] + __popc(m1 & lt)] = item[r];
    } else if (k[r] == 2) {
      out2[wb[2] + __popc(m2 & lt)] = item[r];
    }
    wb[0] += __popc(m0);
    wb[1] += __popc(m1);
    wb[2] += __popc(m2);
  }
}

// One block: flags the k smallest of *n_dev keys (k >= 1), equal keys by position; nothing when
// there are no more than k.  Radix-select passes of 11 bits, from the highest bit in which the
// keys differ, find the k-th smallest key T and how many of the keys equal to T are kept; the keys
// below T and the first of those equal to T (each warp ranks a contiguous part, a scan over the
// warps' counts) are flagged.
// One SM's shared-memory atomics are the time.  With 8-bit digits from bit 31 the first digit of
// 31 000 squared distances was two or three values (their exponents), so nearly all atomics of a
// warp hit one counter: 26 us, 15.5 now.  Counting a warp's equal digits first (match) took 51 us.
constexpr uint32_t kSelectSmemKeys = 40960;  // 160 KB: candidates up to this count are read once
constexpr int kSelectBits = 11, kSelectBins = 1 << kSelectBits;
__global__ void __launch_bounds__(1024) select_keep(const uint32_t* gkeys, const uint32_t* n_dev, uint32_t k,
                                                    uint8_t* keep) {
  extern __shared__ uint32_t skeys[];  // kSelectSmemKeys keys
  let_next_start();
  dependency_wait();
  const uint32_t n = *n_dev;
  if (n <= k) return;
  __shared__ uint32_t hist[kSelectBins];
  __shared__ uint32_t s_prefix, s_rem, s_min, s_max;
  __shared__ uint32_t wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const bool cached = n <= kSelectSmemKeys;
  if (tid == 0) {
    s_min = 0xffffffffu;
    s_max = 0;
    s_rem = k;
  }
  __syncthreads();
  uint32_t lo = 0xffffffffu, hi = 0;
#pragma unroll 8
  for (uint32_t i = tid; i < n; i += 1024) {
    const uint32_t key = gkeys[i];
    if (cached) skeys[i] = key;
    lo = min(lo, key);
    hi = max(hi, key);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) {
    atomicMin(&s_min, lo);
    atomicMax(&s_max, hi);
  }
  __syncthreads();
  const uint32_t* keys = cached ? skeys : gkeys;
  int top = 32 - __clz(s_min ^ s_max);  // bits below this one differ
  if (tid == 0) s_prefix = top < 32 ? s_min >> top << top : 0u;
  __syncthreads();
  while (top > 0) {
    const int shift = max(0, top - kSelectBits);
    const uint32_t digits = (1u << (top - shift)) - 1u, mask = top < 32 ? ~0u << top : 0u, prefix = s_prefix;
    hist[tid] = hist[tid + 1024] = 0;
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = tid; i < n; i += 1024) {
      const uint32_t key = keys[i];
      if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & digits], 1u);
    }
    __syncthreads();
    // the digit whose bucket holds the s_rem-th smallest remaining key: two buckets per thread
    const uint32_t h0 = hist[2 * tid], h1 = hist[2 * tid + 1], rem = s_rem;
    const uint32_t incl = warp_scan_incl(h0 + h1, lane);
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
      const uint32_t v = wsum[lane];
      wsum[lane] = warp_scan_incl(v, lane) - v;
    }
    __syncthreads();
    const uint32_t below = wsum[w] + incl - h0 - h1;
    if (below < rem && rem <= below + h0 + h1) {
      const bool second = rem > below + h0;
      s_prefix = prefix | ((2u * tid + second) << shift);
      s_rem = rem - below - (second ? h0 : 0u);
    }
    __syncthreads();
    top = shift;
  }
  const uint32_t T = s_prefix, rem = s_rem;
  const uint32_t chunk = (n + 1023) / 1024 * 32, c0 = w * chunk;
  uint32_t eq = 0;
  for (uint32_t r = 0; r < chunk; r += 32) {
    const uint32_t i = c0 + r + lane;
    eq += __popc(__ballot_sync(0xffffffffu, i < n && keys[i] == T));
  }
  if (lane == 0) wsum[w] = eq;
  __syncthreads();
  uint32_t before = 0;
  for (int ww = 0; ww < w; ++ww) before += wsum[ww];
  for (uint32_t r = 0; r < chunk; r += 32) {
    const uint32_t i = c0 + r + lane;
    const uint32_t key = i < n ? keys[i] : 0xffffffffu;
    const uint32_t same = __ballot_sync(0xffffffffu, i < n && key == T);
    if (i < n) keep[i] = key < T || (key == T && before + __popc(same & ((1u << lane) - 1u)) < rem) ? 1 : 0;
    before += __popc(same);
  }
}

// simulation.rs:626-650 per far particle
__global__ void far_field_kernel(float* pos, float* vel, float* temp, const uint64_t* idx, uint64_t n,
                                 const float* coarse, uint32_t cn, float cdx, float ox, float oy, float oz, float far_dt) {
  for (uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; k < n; k += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t i = idx ? idx[k] : k;
    // every input is loaded before the first store, so that the loads are in flight together (about
    // 900 000 of 1 M particles: 11.6 -> 8.4 us)
    const float vy0 = vel[3 * i + 1], px = pos[3 * i], py0 = pos[3 * i + 1], pz = pos[3 * i + 2], t = temp[i];
    const float vy = __fsub_rn(vy0, __fmul_rn(9.81f, far_dt));
    vel[3 * i + 1] = vy;
    const float py = __fadd_rn(py0, __fmul_rn(vy, far_dt));
    pos[3 * i + 1] = py;
    const int64_t gx = as_isize(__fdiv_rn(__fsub_rn(px, ox), cdx));
    const int64_t gy = as_isize(__fdiv_rn(__fsub_rn(py, oy), cdx));
    const int64_t gz = as_isize(__fdiv_rn(__fsub_rn(pz, oz), cdx));
    if (gx >= 0 && gy >= 0 && gz >= 0 && gx < int64_t(cn) && gy < int64_t(cn) && gz < int64_t(cn)) {
      const float field = coarse[gx + gy * int64_t(cn) + gz * int64_t(cn) * int64_t(cn)];
      temp[i] = __fadd_rn(t, __fmul_rn(__fmul_rn(__fsub_rn(field, t), 0.02f), far_dt));
    }
  }
}

// cell key of near particle k (simulation.rs:889-905), or `dead` when skipped; empties every cell's run
__global__ void coarse_keys(const float* pos, const uint8_t* active, const uint64_t* idx, uint64_t n, uint32_t cn,
                            float inv_dx, float ox, float oy, float oz, uint32_t dead, uint32_t* keys,
                            uint32_t* run_start, uint32_t* run_end) {
  for (uint64_t c = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; c < dead; c += uint64_t(gridDim.x) * blockDim.x)
    run_start[c] = run_end[c] = 0u;
  for (uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; k < n; k += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t i = idx ? idx[k] : k;
    uint32_t key = dead;
    if (!active || active[i]) {
      const int64_t gx = as_isize(__fmul_rn(__fsub_rn(pos[3 * i], ox), inv_dx));
      const int64_t gy = as_isize(__fmul_rn(__fsub_rn(pos[3 * i + 1], oy), inv_dx));
      const int64_t gz = as_isize(__fmul_rn(__fsub_rn(pos[3 * i + 2], oz), inv_dx));
      if (gx >= 0 && gy >= 0 && gz >= 0 && gx < int64_t(cn) && gy < int64_t(cn) && gz < int64_t(cn))
        key = uint32_t(gx + gy * int64_t(cn) + gz * int64_t(cn) * int64_t(cn));
    }
    keys[k] = key;
  }
}

// the near particles' (temperature x mass, mass) in cell order (simulation.rs:906-908), and each
// cell's run [start, end) in that order (cells without particles keep start == end == 0)
__global__ void coarse_gather(const float* mass, const float* temp, const uint64_t* idx, const uint32_t* perm,
                              const uint32_t* skeys, uint64_t n, uint32_t dead, float2* tm_m, uint32_t* run_start,
                              uint32_t* run_end) {
  for (uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; k < n; k += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t kk = perm[k];
    const uint64_t i = idx ? idx[kk] : kk;
    const float mi = fmaxf(mass[i], 1e-6f);
    tm_m[k] = make_float2(__fmul_rn(temp[i], mi), mi);
    const uint32_t key = skeys[k];
    if (key == dead) continue;
    if (k == 0 || skeys[k - 1] != key) run_start[key] = uint32_t(k);
    if (k + 1 == n || skeys[k + 1] != key) run_end[key] = uint32_t(k + 1);
  }
}

// One warp per cell: the warp stages its cell's run in shared memory 256 entries at a time
// (coalesced loads) and lane 0 adds them in order, as the reference's serial loop does; then the
// cell relaxes toward the injected temperature (simulation.rs:914-923).  The order is the
// reference's, so the two chains of additions are the time: 8 entries are loaded ahead of them.
constexpr int kSumBatch = 256;
__global__ void __launch_bounds__(256) coarse_sums(const uint32_t* run_start, const uint32_t* run_end, const float2* tm_m,
                                                   uint64_t cells, const float* coarse, float blend, float* blended) {
  __shared__ float2 st[8][kSumBatch];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint64_t c = blockIdx.x * 8ull + w; c < cells; c += uint64_t(gridDim.x) * 8) {
    const uint32_t s0 = run_start ? run_start[c] : 0u, e0 = run_start ? run_end[c] : 0u;
    float a = 0.0f, b = 0.0f;
    for (uint32_t base = s0; base < e0; base += kSumBatch) {
      const uint32_t cnt = min(uint32_t(kSumBatch), e0 - base);
      for (uint32_t t = lane; t < cnt; t += 32) st[w][t] = tm_m[base + t];
      __syncwarp();
      if (lane == 0) {
        uint32_t t = 0;
        for (; t + 8 <= cnt; t += 8) {
          float2 q[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) q[u] = st[w][t + u];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            a = __fadd_rn(a, q[u].x);
            b = __fadd_rn(b, q[u].y);
          }
        }
        for (; t < cnt; ++t) {
          a = __fadd_rn(a, st[w][t].x);
          b = __fadd_rn(b, st[w][t].y);
        }
      }
      __syncwarp();
    }
    if (lane == 0) {
      float t = coarse[c];
      if (b > 1e-6f) t = __fadd_rn(t, __fmul_rn(__fsub_rn(__fdiv_rn(a, b), t), blend));
      blended[c] = t;
    }
  }
}

// one FTCS step over the 6 neighbours, neighbours summed in the reference's order (:929-964)
__global__ void coarse_diffuse(const float* f, uint32_t cn, float coef, float* out) {
  const uint64_t n = cn, nn = n * n, cells = nn * n;
  for (uint64_t g = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; g < cells; g += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t i = g % n, j = (g / n) % n, k = g / nn;
    float lap = 0.0f;
    int count = 0;
    if (i > 0) lap = __fadd_rn(lap, f[g - 1]), ++count;
    if (i + 1 < n) lap = __fadd_rn(lap, f[g + 1]), ++count;
    if (j > 0) lap = __fadd_rn(lap, f[g - n]), ++count;
    if (j + 1 < n) lap = __fadd_rn(lap, f[g + n]), ++count;
    if (k > 0) lap = __fadd_rn(lap, f[g - nn]), ++count;
    if (k + 1 < n) lap = __fadd_rn(lap, f[g + nn]), ++count;
    float t = f[g];
    if (count > 0) {
      const float avg = __fdiv_rn(lap, float(count));
      t = __fadd_rn(t, __fmul_rn(__fmul_rn(coef, __fsub_rn(avg, t)), float(count)));
    }
    out[g] = t;
  }
}

// MpssPhase (mpss.rs:67-75): Solid 0, Liquid 1, Gas 2, Plasma 3, Granular 4, Crystal 5, Amorphous 6.
// One hop of apply_phase_transitions' table (mpss.rs:512-524): the arms in order, a failing guard
// falling through to the next arm.
__device__ __forceinline__ uint8_t phase_hop(uint16_t m, uint8_t cur, float t) {
  if (m == 1 && cur == 0 && t >= 273.0f) return 1;
  if (m == 1 && cur == 1 && t >= 373.0f) return 2;
  if (m == 1 && cur == 2 && t < 373.0f) return 1;
  if (m == 1 && cur == 1 && t < 273.0f) return 0;
  if (m == 3 && cur == 0 && t >= 1811.0f) return 1;
  if (m == 3 && cur == 1 && t >= 3134.0f) return 2;
  if (m == 3 && cur == 2 && t < 3134.0f) return 1;
  if (m == 3 && cur == 1 && t < 1811.0f) return 0;
  if (m == 0 && cur == 0 && t >= 500.0f) return 2;
  if (m == 2 && cur == 0 && t >= 1923.0f) return 2;
  return cur;
}

// MpssBuffer housekeeping after the substep (ae_engine/src/lib.rs:347-358): per active particle,
// reflecting world bounds (mpss.rs:449-476), temperature clamp (:479-497), phase transitions with
// up to 3 hops (:500-548), in that order; passes selects them (1, 2, 4).  Each CTA adds its
// transitions with one atomic: one per warp, 31 000 on one address, took longer
// than the passes (1 M particles, most of them in transition: 30 -> 14.6 us).  As many CTAs as run at
// once: with a CTA of its own for every 512 particles the bounds or the clamp alone took 53.7 and 44.7 us
// for 8 M particles, 37.8 and 31.0 so (all three passes 79.2 -> 67.1).
__global__ void housekeeping_kernel(float* pos, float* vel, float* temp, uint8_t* phase, const uint16_t* mat,
                                    const uint8_t* active, uint64_t n, float x0, float y0, float z0, float x1, float y1,
                                    float z1, float tmin, float tmax, uint32_t passes, uint32_t* transitions) {
  // a particle's inputs are all loaded before anything is decided, the velocity components once the
  // bounds are known: two memory latencies per particle instead of one per component and pass
  const float lo[3] = {x0, y0, z0}, hi[3] = {x1, y1, z1};
  uint32_t changed = 0;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    const bool on = !active || active[i];
    float p[3] = {0.0f, 0.0f, 0.0f}, v[3] = {0.0f, 0.0f, 0.0f}, t = 0.0f;
    uint16_t m = 0;
    uint8_t cur = 0;
    if (passes & 1u)
#pragma unroll
      for (int d = 0; d < 3; ++d) p[d] = pos[3 * i + d];
    if (passes & 6u) t = temp[i];
    if (passes & 4u) {
      m = mat[i];
      cur = phase[i];
    }
    if (on) {
      if (passes & 1u) {
        bool below[3], above[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          below[d] = p[d] < lo[d];
          above[d] = !below[d] && p[d] > hi[d];
          if (below[d] || above[d]) v[d] = vel[3 * i + d];
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (!(below[d] || above[d])) continue;
          pos[3 * i + d] = below[d] ? lo[d] : hi[d];
          if (below[d] ? v[d] < 0.0f : v[d] > 0.0f) vel[3 * i + d] = __fmul_rn(-v[d], 0.5f);
        }
      }
      if (passes & 2u) {
        const float before = t;
        if (t > tmax)
          t = tmax;
        else if (t < tmin)
          t = tmin;
        if (t != before) temp[i] = t;
      }
      if (passes & 4u) {
        uint8_t next = cur;
        for (int hop = 0; hop < 3; ++hop) {
          const uint8_t h = phase_hop(m, next, t);
          if (h == next) break;
          next = h;
        }
        if (next != cur) {
          phase[i] = next;
          ++changed;
        }
      }
    }
  }
  if (!(passes & 4u)) return;
  __shared__ uint32_t sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  changed = __reduce_add_sync(0xffffffffu, changed);
  if ((threadIdx.x & 31) == 0 && changed) atomicAdd(&sum, changed);
  __syncthreads();
  if (threadIdx.x == 0 && sum) atomicAdd(transitions, sum);
}

inline unsigned grid_for(uint64_t n, int threads) {
  const uint64_t b = (n + threads - 1) / threads;
  return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(b, 148ull * 16)));
}

int bits_for(uint64_t v) {  // bits needed to hold values 0..v
  int b = 1;
  while (b < 32 && (uint64_t(1) << b) <= v) ++b;
  return b;
}

}  // namespace

#define LOD_TRY(x)                          \
  do {                                      \
    cudaError_t e_ = (x);                   \
    if (e_ != cudaSuccess) return e_;       \
  } while (0)

LodWork::~LodWork() {
  if (items_) cudaFree(items_);
  if (cells_) cudaFree(cells_);
  sort_scratch_free(sort_);
}

// One allocation for the arrays per particle and one for those per cell: an allocation of its own for
// each of the ten was a third of a new context's first tick (3.2 -> 2.0 ms).
cudaError_t LodWork::grow(uint64_t count, uint64_t cells) {
  if (count > cap_ || !items_) {
    const uint64_t cap = std::max<uint64_t>(count, std::max<uint64_t>(cap_ * 2, 4096));
    if (items_) cudaFree(items_);
    items_ = nullptr;
    cap_ = 0;
    const uint64_t tiles = (cap + kPTile - 1) / kPTile;
    uint64_t at = 0;
    const auto place = [&](uint64_t bytes) {
      const uint64_t here = at;
      at += (bytes + 255) / 256 * 256;
      return here;
    };
    const uint64_t o_totals = place(sizeof(uint32_t) * 8), o_counts = place(sizeof(uint32_t) * 3 * tiles),
                   o_offs = place(sizeof(uint32_t) * 3 * tiles), o_tmp = place(sizeof(uint64_t) * cap),
                   o_key = place(sizeof(uint32_t) * cap), o_keep = place(cap), o_tm = place(sizeof(float2) * cap);
    LOD_TRY(cudaMalloc(&items_, at));
    char* const base = static_cast<char*>(items_);
    totals_ = reinterpret_cast<uint32_t*>(base + o_totals);
    tile_counts_ = reinterpret_cast<uint32_t*>(base + o_counts);
    tile_offs_ = reinterpret_cast<uint32_t*>(base + o_offs);
    near_tmp_ = reinterpret_cast<uint64_t*>(base + o_tmp);
    near_key_ = reinterpret_cast<uint32_t*>(base + o_key);
    keep_ = reinterpret_cast<uint8_t*>(base + o_keep);
    tm_m_ = reinterpret_cast<float2*>(base + o_tm);
    LOD_TRY(sort_scratch_alloc(sort_, cap));
    cap_ = cap;
  }
  if (cells > cells_cap_) {
    if (cells_) cudaFree(cells_);
    cells_ = nullptr;
    cells_cap_ = 0;
    LOD_TRY(cudaMalloc(&cells_, sizeof(uint32_t) * 3 * cells));
    field_tmp_ = static_cast<float*>(cells_);
    run_start_ = reinterpret_cast<uint32_t*>(field_tmp_ + cells);
    run_end_ = run_start_ + cells;
    cells_cap_ = cells;
  }
  return cudaSuccess;
}

cudaError_t LodWork::classify(const float* pos, const uint8_t* active, uint64_t count, const float player[3],
                              float near_dist, float mid_dist, uint64_t max_near, uint64_t* near_out, uint64_t* mid_out,
                              uint64_t* far_out, uint64_t counts[3], cudaStream_t s) {
  counts[0] = counts[1] = counts[2] = 0;
  if (count == 0) return cudaSuccess;
  LOD_TRY(grow(count, 0));
  const uint32_t tiles = uint32_t((count + kPTile - 1) / kPTile);
  // squared distances as the reference computes them (simulation.rs:484-485)
  const PosClass pc{pos, active, player[0], player[1], player[2], near_dist * near_dist, mid_dist * mid_dist};
  // Each kernel after the first is launched dependently and waits for the one before it: the kernels are
  // short, up to seven in a row.
  const Items all{count, nullptr, 0u};
  const uint32_t cap = uint32_t(std::min<uint64_t>(max_near, 0xffffffffu));
  part_count<PosClass><<<tiles, kPT, 0, s>>>(pc, all, tile_counts_, tiles);
  LOD_TRY(launch_after(true, part_scan, 1, 1024, 0, s, tile_counts_, tile_offs_, tiles, all, totals_));
  LOD_TRY(launch_after(true, part_scatter<PosClass>, tiles, kPT, 0, s, pc, all, tile_offs_, tiles, near_out, near_tmp_,
                       cap, reinterpret_cast<float*>(near_key_), mid_out, nullptr, far_out));
  // cap (simulation.rs:519-530): the max_near smallest squared distances stay near, ties by index.
  // The number of candidates stays on the device: the host waits once, for the final counts, and the
  // kernels of the cap leave at once where the candidates do not exceed it (3 000 particles, 100 near ones
  // under a cap of 1 000: 37 us, 53 with the kernels launched one after another and working through them).
  if (cap < count) {
    if (!select_smem_set_) {
      LOD_TRY(cudaFuncSetAttribute(select_keep, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(sizeof(uint32_t) * kSelectSmemKeys)));
      select_smem_set_ = true;
    }
    if (cap) LOD_TRY(launch_after(true, select_keep, 1, 1024, sizeof(uint32_t) * kSelectSmemKeys, s, near_key_, totals_, cap,
                                  keep_));
    const KeepClass kc{near_tmp_, cap ? keep_ : nullptr};
    const Items near{0, totals_, cap};
    LOD_TRY(launch_after(true, part_count<KeepClass>, tiles, kPT, 0, s, kc, near, tile_counts_, tiles));
    LOD_TRY(launch_after(true, part_scan, 1, 1024, 0, s, tile_counts_, tile_offs_, tiles, near, totals_ + 4));
    LOD_TRY(launch_after(true, part_scatter<KeepClass>, tiles, kPT, 0, s, kc, near, tile_offs_, tiles, near_out, nullptr,
                         cap, nullptr, mid_out, totals_ + 1, nullptr));
  }
  LOD_TRY(cudaGetLastError());
  uint32_t tot[3] = {0, 0, 0};
  LOD_TRY(cudaMemcpyAsync(tot, totals_, sizeof(tot), cudaMemcpyDeviceToHost, s));
  LOD_TRY(cudaStreamSynchronize(s));
  counts[0] = std::min<uint64_t>(tot[0], max_near);
  counts[1] = tot[1] + (tot[0] - counts[0]);
  counts[2] = tot[2];
  return cudaSuccess;
}

cudaError_t LodWork::housekeeping(float* pos, float* vel, float* temp, uint8_t* phase, const uint16_t* material,
                                  const uint8_t* active, uint64_t n, const float bmin[3], const float bmax[3],
                                  float min_temp, float max_temp, uint32_t passes, uint32_t* transitions,
                                  cudaStream_t s) {
  *transitions = 0;
  if (n == 0) return cudaSuccess;
  LOD_TRY(grow(1, 0));
  LOD_TRY(cudaMemsetAsync(totals_ + 3, 0, sizeof(uint32_t), s));
  housekeeping_kernel<<<std::min(grid_for(n, 256), 148u * 8u), 256, 0, s>>>(pos, vel, temp, phase, material, active, n, bmin[0],
                                                               bmin[1], bmin[2], bmax[0], bmax[1], bmax[2], min_temp,
                                                               max_temp, passes, totals_ + 3);
  LOD_TRY(cudaGetLastError());
  LOD_TRY(cudaMemcpyAsync(transitions, totals_ + 3, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  return cudaStreamSynchronize(s);
}

cudaError_t LodWork::far_field(float* pos, float* vel, float* temp, const uint64_t* far_idx, uint64_t n,
                               const float* coarse, uint32_t cn, float cdx, const float origin[3], float far_dt,
                               cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  far_field_kernel<<<grid_for(n, 256), 256, 0, s>>>(pos, vel, temp, far_idx, n, coarse, cn, cdx, origin[0], origin[1],
                                                   origin[2], far_dt);
  return cudaGetLastError();
}

cudaError_t LodWork::coarse_field(const float* pos, const float* mass, const float* temp, const uint8_t* active,
                                  const uint64_t* near_idx, uint64_t n, float* coarse, uint32_t cn, float cdx,
                                  const float origin[3], float dt, cudaStream_t s) {
  const uint64_t cells = uint64_t(cn) * cn * cn;
  if (cells == 0) return cudaSuccess;
  LOD_TRY(grow(std::max<uint64_t>(n, 1), cells));
  const float inject_rate = 0.1f;
  const float blend = std::fmin(inject_rate * dt, 1.0f);
  const float alpha = 10.0f;
  const float coef = std::fmin(alpha * dt / (cdx * cdx), 0.16f);
  if (n > 0) {
    const uint32_t dead = uint32_t(cells);
    const float inv_dx = 1.0f / cdx;
    coarse_keys<<<grid_for(std::max(n, cells), 256), 256, 0, s>>>(pos, active, near_idx, n, cn, inv_dx, origin[0],
                                                                 origin[1], origin[2], dead, near_key_, run_start_,
                                                                 run_end_);
    const uint32_t *sorted = nullptr, *perm = nullptr;
    radix_sort_pairs(near_key_, n, bits_for(cells), sort_, s, &sorted, &perm);
    coarse_gather<<<grid_for(n, 256), 256, 0, s>>>(mass, temp, near_idx, perm, sorted, n, dead, tm_m_, run_start_,
                                                  run_end_);
  }
  // without particles the injection adds nothing
  coarse_sums<<<unsigned(std::min<uint64_t>((cells + 7) / 8, 148 * 16)), 256, 0, s>>>(
      n > 0 ? run_start_ : nullptr, run_end_, tm_m_, cells, coarse, blend, field_tmp_);
  coarse_diffuse<<<grid_for(cells, 256), 256, 0, s>>>(field_tmp_, cn, coef, coarse);
  return cudaGetLastError();
}

}  // namespace aemp
