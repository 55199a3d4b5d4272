// mg_kernels.cu -- sm_100a kernels of the per-server PIR answer path.
//
// scan_kernel<G>: persistent CTAs walk a list of (tile, key group) work items.
// For one item (an aligned subtree of 2^S rows and g <= G keys):
//   1. each key's node at the tile root is read from a frontier, or, when a CTA
//      has one item only, walked to from the key's root by threads 0..g-1 (d - S
//      levels; the prefix walk of dpf.rs:183-203).  The walk's 16 serial levels
//      and the barriers around them took 27k cycles per item, 10% of the time
//      of a 512-page tile: 1300021 x 4 KB 940 us with it, 887 without (0.92 of
//      the measured copy rate);
//   2. the CTA expands U levels breadth-first in shared memory, giving every
//      thread one node 2^M leaves above the rows (the GGM tree of
//      dpf.rs:210-246 in breadth-first order);
//   3. each thread walks its node depth-first with a per-thread stack in
//      shared memory, one leaf pair per step; the 16-byte leaf outputs
//      (masks) of all g keys go to shared memory;
//   4. the CTA scans the step's rows with coalesced 128-bit loads and
//      XOR-accumulates row & mask per key in registers (kernel.rs:1243-1256);
//   5. after the last step the per-thread accumulators are XOR-reduced with
//      warp shuffles and shared memory and folded into this CTA's own row of
//      the partial buffer (no atomics).
// reduce_kernel XORs the partial rows (per CTA, or per warp for the warp
// kernel) into the shares: slices of the rows in parallel, combined with
// 64-bit XOR atomics into the zeroed shares.  XOR is
// associative and commutative, so the shares are bit-exact whatever the
// schedule.  The kernels contain no waits on other CTAs or on the host.
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "mg_device.cuh"
#include "mg_internal.h"
#include "morphogen_gpu.h"

namespace mg {

// Every kernel of a pass begins with one of these two: chain_wait waits until
// the kernel before it has completed and its writes are visible, chain_begin
// before that lets the pass's next kernel be launched while this one runs (its
// CTAs take their places as these leave).
//
// The frontier only waits.  A scan launched beside it would hold SMs idle, with
// most of their shared memory, and any other pass on the device would wait for
// them; and the CTAs of a narrow scan would crowd onto the SMs that the frontier
// leaves free.  Launched as the frontier's CTAs end, they spread over the SMs by
// themselves.  3 keys, two workspaces replaying at once, us per pair of passes
// with the scan beside its frontier (narrow CTAs padded to one per SM) and
// after it: 140000 x 128 B 89 and 60, 30000 x 64 B 46 and 28, 175056 x 256 B 100
// and 70, 2^20 x 256 B 261 and 241; a pass alone: 39.0 and 38.4, 23.0 and 22.8,
// 43.3 and 43.1, 132.8 and 132.9.
//
// Nothing in global memory is touched earlier, and what a kernel of
// the pass writes (keys, frontier, partial rows, shares) or the host may write
// beside it (a delta buffer) is read with plain loads: the read-only path and
// __restrict__ promise data that nothing writes while the kernel lives, and its
// life now begins before that of its predecessors ends.  Only the table's rows,
// which no kernel of a pass writes, are read through __ldg.  See launch_chained.
__device__ __forceinline__ void chain_wait() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void chain_begin() {
  cudaTriggerProgrammaticLaunchCompletion();
  chain_wait();
}

// Up to 4 keys per CTA the kernel is held to 80 registers so that three
// CTAs share an SM (page mode: more bytes in flight per SM).
// FMA: node expansions balanced over both integer pipes, or all-ALU (see
// launch_scan).
template <int G, bool FMA>
__global__ void __launch_bounds__(kThreads, (G <= 4 ? 3 : 2)) scan_kernel(const __grid_constant__ ScanParams p) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KeyDev* s_keys = reinterpret_cast<KeyDev*>(smem_raw);
  uint4* s_mask = reinterpret_cast<uint4*>(smem_raw + G * sizeof(KeyDev));  // [G][2*T]
  uint4* s_seed = s_mask + G * 2 * kThreads;                                 // [G][slots][T]
  uint8_t* s_t = reinterpret_cast<uint8_t*>(s_seed + (size_t)G * p.slots * kThreads);
  const uint32_t tid = threadIdx.x;
  const uint32_t slots = p.slots;

  uint4* my_partial = p.partial + (size_t)blockIdx.x * p.cols;
  for (uint32_t c = tid; c < p.cols; c += kThreads) my_partial[c] = make_uint4(0u, 0u, 0u, 0u);

  for (uint64_t item = blockIdx.x; item < p.items; item += gridDim.x) {
    uint32_t si = 0;
    while (si + 1 < p.nsegs && item >= p.seg[si + 1].item_begin) ++si;
    const Segment& sg = p.seg[si];
    const uint64_t local = item - sg.item_begin;
    const uint32_t group = (uint32_t)(local % sg.groups);
    const uint32_t g = sg.g, V = sg.V, d = sg.d, S = sg.S, U = sg.U, M = sg.M;
    const uint32_t L0 = d - S;
    // Global index of the tile at level L0 (row-range tables start mid-domain).
    const uint32_t tile = (uint32_t)(local / sg.groups + (sg.first >> S));

    __syncthreads();  // the previous item is done with shared memory
    {
      const uint4* src = reinterpret_cast<const uint4*>(p.keys + sg.key_base + (size_t)group * g);
      uint4* dst = reinterpret_cast<uint4*>(s_keys);
      const uint32_t n = g * (uint32_t)(sizeof(KeyDev) / 16);
      for (uint32_t i = tid; i < n; i += kThreads) dst[i] = src[i];
    }
    // 1. the tile's root, from the frontier or by the prefix walk; the
    //    breadth-first ping-pong below starts in slot (U & 1) so that it ends
    //    in slot 0.
    const uint32_t start_slot = U & 1u;
    if (p.fr_seed) {
      if (tid < g) {
        const uint64_t at = sg.fr_base + ((uint64_t)group * g + tid) * sg.tiles + local / sg.groups;
        s_seed[(tid * slots + start_slot) * kThreads] = p.fr_seed[at];
        s_t[(tid * slots + start_slot) * kThreads] = p.fr_t[at];
      }
      __syncthreads();
    } else {
      __syncthreads();
      if (tid < g) {
        const KeyDev& K = s_keys[tid];
        uint4 s = K.root_seed;
        uint32_t t = K.root_t;
        for (uint32_t lvl = 0; lvl < L0; ++lvl) {
          uint4 Lc, Rc;
          uint32_t tl, tr;
          expand_cw<false>(s, t, K, lvl, Lc, tl, Rc, tr);
          const uint32_t bit = (tile >> (L0 - 1 - lvl)) & 1u;
          s = bit ? Rc : Lc;
          t = bit ? tr : tl;
        }
        s_seed[(tid * slots + start_slot) * kThreads] = s;
        s_t[(tid * slots + start_slot) * kThreads] = (uint8_t)t;
      }
      __syncthreads();
    }

    // 2. breadth-first expansion of U levels below the tile root.
    uint32_t cur = start_slot;
    for (uint32_t j = 0; j < U; ++j) {
      const uint32_t nxt = cur ^ 1u;
      const uint32_t work = g << j;
      for (uint32_t it = tid; it < work; it += kThreads) {
        const uint32_t k = it >> j, i = it & ((1u << j) - 1u);
        const size_t src = (k * slots + cur) * kThreads + i;
        const size_t dst = (k * slots + nxt) * kThreads + 2 * i;
        uint4 Lc, Rc;
        uint32_t tl, tr;
        expand_cw<FMA>(s_seed[src], s_t[src], s_keys[k], L0 + j, Lc, tl, Rc, tr);
        s_seed[dst] = Lc;
        s_seed[dst + 1] = Rc;
        s_t[dst] = (uint8_t)tl;
        s_t[dst + 1] = (uint8_t)tr;
      }
      __syncthreads();
      cur = nxt;
    }

    // 3-4. depth-first leaf pairs + scan of the step's rows.
    uint4 acc[G];
#pragma unroll
    for (int k = 0; k < G; ++k) acc[k] = make_uint4(0u, 0u, 0u, 0u);
    const uint32_t NR = 1u << U;
    const uint32_t pairs = M ? (1u << (M - 1)) : 1u;
    const uint64_t tile_row0 = ((uint64_t)tile << S) - sg.first;  // table row of the tile's first leaf (may wrap)
    const uint32_t rpi = kThreads / V;  // rows per scan sweep
    const uint32_t lane = tid % V, rslot = tid / V;
    const bool scan_thread = tid < rpi * V;
    const uint4* __restrict__ tbl = sg.table;
    const uint64_t nrows = sg.rows;
    const uint32_t abs0 = d - M;  // tree level of the depth-first roots
    // Every row of the tile inside the table and every sweep of 8 rows full:
    // loads need no bounds checks.
    const bool full_tile = tile_row0 < nrows && nrows - tile_row0 >= (1ull << S) &&
                           (2 * NR) % (8 * rpi) == 0 && M > 0;

    for (uint32_t pi = 0; pi < pairs; ++pi) {
      if (tid < NR) {
#pragma unroll 1
        for (uint32_t k = 0; k < g; ++k) {
          const KeyDev& K = s_keys[k];
          uint4* col_seed = s_seed + (size_t)k * slots * kThreads + tid;
          uint8_t* col_t = s_t + (size_t)k * slots * kThreads + tid;
          uint4* mk = s_mask + (size_t)k * 2 * kThreads + 2 * tid;
          if (M == 0) {
            mk[0] = leaf_mask(col_seed[0], col_t[0], K);
            mk[1] = make_uint4(0u, 0u, 0u, 0u);
            continue;
          }
          // Pair pi's parent path re-joins the stack at relative level
          // M - 1 - ctz(pi) (root for pi == 0).
          uint32_t lvl = pi ? (M - (uint32_t)__ffs((int)pi)) : 0u;
          uint4 s = col_seed[lvl * kThreads];
          uint32_t t = col_t[lvl * kThreads];
          for (;; ++lvl) {
            uint4 Lc, Rc;
            uint32_t tl, tr;
            expand_cw<FMA>(s, t, K, abs0 + lvl, Lc, tl, Rc, tr);
            if (lvl == M - 1) {
              mk[0] = leaf_mask(Lc, tl, K);
              mk[1] = leaf_mask(Rc, tr, K);
              break;
            }
            col_seed[(lvl + 1) * kThreads] = Rc;
            col_t[(lvl + 1) * kThreads] = (uint8_t)tr;
            s = Lc;
            t = tl;
          }
        }
      }
      __syncthreads();
      if (scan_thread && full_tile) {
        const uint4* __restrict__ bp = tbl + (tile_row0 + 2u * pi) * V + lane;
        for (uint32_t rb = rslot; rb < 2 * NR; rb += 8 * rpi) {
          uint4 dat[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const uint32_t r = rb + (uint32_t)u * rpi;
            dat[u] = __ldg(bp + (size_t)(((r >> 1) << M) + (r & 1u)) * V);
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const uint32_t r = rb + (uint32_t)u * rpi;
#pragma unroll
            for (int k = 0; k < G; ++k)
              if ((uint32_t)k < g) acc[k] = xor_and(acc[k], dat[u], s_mask[(size_t)k * 2 * kThreads + r]);
          }
        }
      } else if (scan_thread) {
        // Eight independent 128-bit loads in flight per thread before any
        // is consumed (wide rows leave one lane position per thread, so
        // this is what keeps enough bytes in flight for HBM).
        for (uint32_t rb = rslot; rb < 2 * NR; rb += 8 * rpi) {
          uint4 dat[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const uint32_t r = rb + (uint32_t)u * rpi;
            // Leaves before the table's first row wrap to huge values and fail the check.
            const uint64_t row = tile_row0 + ((uint64_t)(r >> 1) << M) + 2u * pi + (r & 1u);
            dat[u] = (r < 2 * NR && row < nrows) ? __ldg(tbl + row * V + lane) : make_uint4(0u, 0u, 0u, 0u);
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const uint32_t r = rb + (uint32_t)u * rpi;
            if (r < 2 * NR) {
#pragma unroll
              for (int k = 0; k < G; ++k)
                if ((uint32_t)k < g) acc[k] = xor_and(acc[k], dat[u], s_mask[(size_t)k * 2 * kThreads + r]);
            }
          }
        }
      }
      __syncthreads();
    }

    // 5. reduce the accumulators of threads holding the same lane.
    uint4* s_red = s_mask;  // G * T uint4 fit in the mask buffer
    const bool pow2 = (V & (V - 1)) == 0;
    if (pow2 && V < 32) {
#pragma unroll
      for (int k = 0; k < G; ++k) {
        uint4 v = acc[k];
        for (uint32_t off = 16; off >= V; off >>= 1) {
          v.x ^= __shfl_xor_sync(0xFFFFFFFFu, v.x, off);
          v.y ^= __shfl_xor_sync(0xFFFFFFFFu, v.y, off);
          v.z ^= __shfl_xor_sync(0xFFFFFFFFu, v.z, off);
          v.w ^= __shfl_xor_sync(0xFFFFFFFFu, v.w, off);
        }
        if ((tid & 31u) < V) s_red[(size_t)k * kThreads + (tid >> 5) * V + (tid & 31u)] = v;
      }
      __syncthreads();
      for (uint32_t o = tid; o < g * V; o += kThreads) {
        const uint32_t k = o / V, ln = o % V;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t w = 0; w < kThreads / 32; ++w) v = xor4(v, s_red[(size_t)k * kThreads + w * V + ln]);
        const size_t col = sg.col_base + ((size_t)group * g + k) * V + ln;
        my_partial[col] = xor4(my_partial[col], v);
      }
    } else {
#pragma unroll
      for (int k = 0; k < G; ++k)
        s_red[(size_t)k * kThreads + tid] = scan_thread ? acc[k] : make_uint4(0u, 0u, 0u, 0u);
      __syncthreads();
      for (uint32_t o = tid; o < g * V; o += kThreads) {
        const uint32_t k = o / V, ln = o % V;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t j = 0; j < rpi; ++j) v = xor4(v, s_red[(size_t)k * kThreads + ln + j * V]);
        const size_t col = sg.col_base + ((size_t)group * g + k) * V + ln;
        my_partial[col] = xor4(my_partial[col], v);
      }
    }
  }
}

// ---- warp-independent path -------------------------------------------------

// Frontier chain step: CTA (x, key) takes node x of level L_in (level index
// in_first + x) of key `blockIdx.y` c levels down and stores the nodes of level
// L_in + c that intersect the table, at slot (level index - out_first).
//
// The levels are a serial chain, so what bounds a small frontier is the time of
// one node expansion (0.57 us a level), and a large one the share of full warps
// (26 G nodes/s: ALU pipe 81% busy at 3 x 2^20 nodes, 118 us; 151 us with every
// level breadth first and one lane per node).  The path to the CTA's node (with
// walk) and the first min(c, 8) levels below it go breadth first in shared
// memory: up to 4 nodes with eight lanes per node, up to 128 with two, the even
// one computing block 0 (both children's seeds), the odd one block 1 (their t
// bits).  Levels of up to 16 nodes run in warp 0 without a CTA barrier.  The
// last c - 8 levels are walked depth first, one of the 256 nodes per thread,
// with no barrier at all.
__global__ void __launch_bounds__(kThreads) frontier_kernel(const __grid_constant__ FrontierStep f) {
  chain_wait();
  constexpr uint32_t kWide = 1u << kFrontierWide;  // nodes of the widest breadth-first level
  static_assert(kWide == kThreads, "one node per thread for the depth-first levels");
  __shared__ uint4 sa[kWide], sb[kWide];
  __shared__ uint8_t ta[kWide], tb[kWide];
  __shared__ uint4 stk[kFrontierLevels - kFrontierWide - 1][kWide];
  __shared__ uint8_t stk_t[kFrontierLevels - kFrontierWide - 1][kWide];
  __shared__ uint4 s_cw[kMaxLevels];
  __shared__ uint32_t s_cwt[2][kMaxLevels];  // t correction bytes: left, right
  const uint32_t tid = threadIdx.x, half = tid & 1u;
  const uint64_t node = blockIdx.x, j = blockIdx.y;
  // The pass's shares start at zero: the scan CTAs XOR into them.
  if (f.zero_out && blockIdx.x == 0 && blockIdx.y == 0)
    for (uint64_t i = tid; i < f.zero_n; i += kThreads) f.zero_out[i] = make_uint4(0u, 0u, 0u, 0u);
  const uint64_t a = f.in_first + node;  // level index of the CTA's node
  const uint64_t g_out0 = a << f.c;      // level index of its first descendant
  if (g_out0 + (1ull << f.c) <= f.out_first || g_out0 >= f.out_first + f.n_out) return;  // uniform per CTA
  const KeyDev* K = f.keys + j;
  const uint32_t walk = f.walk ? f.L_in : 0u;  // levels above the CTA's node
  const uint32_t top = f.L_in - walk;          // level of the first node expanded
  const uint32_t wide = f.c < kFrontierWide ? f.c : kFrontierWide;
  const uint32_t deep = f.c - wide;
  if (tid < kMaxLevels) {
    // Correction words of the step's levels, and its root.
    const uint32_t lvl = top + tid;
    if (tid < walk + f.c) {
      s_cw[tid] = K->cw_seed[lvl];
      s_cwt[0][tid] = K->cw_tl[lvl];
      s_cwt[1][tid] = K->cw_tr[lvl];
    }
    if (tid == 0) {
      sa[0] = top == 0 ? K->root_seed : f.in_seed[j * f.n_in + node];
      ta[0] = (uint8_t)(top == 0 ? K->root_t : f.in_t[j * f.n_in + node]);
    }
  }
  uint4* cs = sa; uint8_t* ct = ta;
  uint4* ns = sb; uint8_t* nt = tb;
  auto swap = [&]() {
    uint4* x = cs; cs = ns; ns = x;
    uint8_t* y = ct; ct = nt; nt = y;
  };
  // Levels of at most 4 nodes: eight lanes of warp 0 per node (block, column).
  const uint32_t tiny = walk + (wide < 3u ? wide : 3u);
  if (tid < 32) {
    const uint32_t i = tid >> 3, blk = (tid >> 2) & 1u, col = tid & 3u;
#pragma unroll 1
    for (uint32_t lv = 0; lv < tiny; ++lv) {
      __syncwarp();
      const uint32_t n = lv < walk ? 1u : 1u << (lv - walk);  // nodes of the level
      const uint32_t s = reinterpret_cast<const uint32_t*>(cs)[(i < n ? 4 * i : 0u) + col];
      // dpf.rs:221-239: correction word on both children when t == 1.
      const uint32_t m = ct[i < n ? i : 0u] == 1 ? 0xFFFFFFFFu : 0u;
      uint32_t l, r;
      prg_block_quad(col, s, blk, l, r);
      if (i < n) {
        // On the path (dpf.rs:103-142) only the child towards node a is kept.
        const bool path = lv < walk;
        const uint32_t bit = path ? (uint32_t)(a >> (walk - 1 - lv)) & 1u : 0u;
        if (blk == 0) {
          const uint32_t cw = reinterpret_cast<const uint32_t*>(s_cw)[4 * lv + col] & m;
          uint32_t* const dst = reinterpret_cast<uint32_t*>(ns) + (path ? 0u : 8 * i) + col;
          dst[0] = (bit ? r : l) ^ cw;
          if (!path) dst[4] = r ^ cw;
        } else if (col < 2 && (!path || col == bit)) {
          nt[path ? 0u : 2 * i + col] = (uint8_t)((l & 1u) ^ (s_cwt[col][lv] & m));
        }
      }
      swap();
    }
  } else if (tiny & 1u) {
    swap();
  }
  // Levels of 8 to 128 nodes: two lanes per node, those of warp 0 without a
  // CTA barrier.
#pragma unroll 1
  for (uint32_t lv = tiny; lv < walk + wide; ++lv) {
    const uint32_t n = 1u << (lv - walk);
    if (n > 16)
      __syncthreads();
    else if (tid < 32)
      __syncwarp();
    if (tid < 2 * n) {
      const uint32_t i = tid >> 1;
      const uint32_t m = ct[i] == 1 ? 0xFFFFFFFFu : 0u;
      uint4 L, R;
      prg_block(cs[i], half, L, R);
      if (half == 0) {
        const uint4 cw = s_cw[lv];
        ns[2 * i] = make_uint4(L.x ^ (cw.x & m), L.y ^ (cw.y & m), L.z ^ (cw.z & m), L.w ^ (cw.w & m));
        ns[2 * i + 1] = make_uint4(R.x ^ (cw.x & m), R.y ^ (cw.y & m), R.z ^ (cw.z & m), R.w ^ (cw.w & m));
      } else {
        nt[2 * i] = (uint8_t)((L.x & 1u) ^ (s_cwt[0][lv] & m));
        nt[2 * i + 1] = (uint8_t)((L.y & 1u) ^ (s_cwt[1][lv] & m));
      }
    }
    swap();
  }
  __syncthreads();
  if (tid >= (1u << wide)) return;
  // Thread tid's node and its 2^deep descendants.
  uint4* const out_seed = f.out_seed + f.out_base + j * f.out_stride;
  uint8_t* const out_t = f.out_t + f.out_base + j * f.out_stride;
  auto store = [&](uint32_t i, const uint4 s, uint32_t t) {
    const uint64_t o = g_out0 + i - f.out_first;  // wraps for nodes before the range
    if (o < f.n_out) {
      out_seed[o] = s;
      out_t[o] = (uint8_t)t;
    }
  };
  uint4 s = cs[tid];
  uint32_t t = ct[tid];
  if (deep == 0) {
    store(tid, s, t);
    return;
  }
#pragma unroll 1
  for (uint32_t pi = 0; pi < (1u << (deep - 1)); ++pi) {
    uint32_t lvl = 0;
    if (pi) {
      lvl = deep - (uint32_t)__ffs((int)pi);
      s = stk[lvl - 1][tid];
      t = stk_t[lvl - 1][tid];
    }
    for (;; ++lvl) {
      uint4 L, R;
      uint32_t tl, tr;
      prg_expand(s, L, R, tl, tr);
      const uint32_t m = t == 1u ? 0xFFFFFFFFu : 0u;
      const uint4 cw = s_cw[walk + wide + lvl];
      L.x ^= cw.x & m; L.y ^= cw.y & m; L.z ^= cw.z & m; L.w ^= cw.w & m;
      R.x ^= cw.x & m; R.y ^= cw.y & m; R.z ^= cw.z & m; R.w ^= cw.w & m;
      tl ^= s_cwt[0][walk + wide + lvl] & m;
      tr ^= s_cwt[1][walk + wide + lvl] & m;
      if (lvl + 1 == deep) {
        const uint32_t i = (tid << deep) + 2 * pi;
        store(i, L, tl);
        store(i + 1, R, tr);
        break;
      }
      stk[lvl][tid] = R;
      stk_t[lvl][tid] = (uint8_t)tr;
      s = L;
      t = tl;
    }
  }
}

// out ^= v with two 64-bit XOR atomics.
__device__ __forceinline__ void xor_out(uint4* out, const uint4 v) {
  unsigned long long* o = reinterpret_cast<unsigned long long*>(out);
  atomicXor(o, ((unsigned long long)v.y << 32) | v.x);
  atomicXor(o + 1, ((unsigned long long)v.w << 32) | v.z);
}

// Warp-independent fused expansion + scan.  A CTA of W warps owns a
// contiguous range of the pass's work items, in (tile, key group) order with
// the groups of a tile next to each other; its warps take the items one at a
// time (ItemQueue).  Per item each lane takes one frontier node and walks its
// 2^M leaves depth-first (stack in the warp's shared-memory slice), one leaf
// pair per step.  Accumulators stay in registers and are flushed (warp shuffle
// XOR) into the warp's own partial row when the group or segment changes.
//
// scan_pair_kernel (one key per warp; rows of 16, 32 or 64 B): a step's rows
// are loaded before its leaf pair is expanded and stay in registers meanwhile.
// Rows of 16 and 32 B: each lane ANDs its own pair's rows (whole sectors) with
// its own masks.  64 B: the lanes exchange the step's 64 masks through shared
// memory and the row loads are coalesced.  Two copies of the PRG code, one for
// internal nodes and one for leaf pairs (about 25 KB); a third copy runs into
// the instruction cache: 2^25 x 32 B, 3 keys 2.80 ms with three copies, 2.65
// with one and a stack round trip per step, 2.61 with two; 2.52 with 20 warps.
// Bound by integer issue: 90.4% of the issue slots, ALU pipe 91.2%, FMA 86.2%.
//
// scan_block_kernel (other row sizes, or several keys per warp): a step's rows
// are too many for registers.  Its masks, for each of the warp's keys, go to
// shared memory, and its 64 rows are scanned with coalesced 16-byte copies while
// the next step's nodes are expanded: before each node expansion a chunk of the
// earlier step's rows is copied towards shared memory (cp.async, no register
// held), after it the chunk is used, so hardly a load is waited for and the
// table is read at an even rate.  One copy of the PRG code, since the chunk code
// beside it would take two past the instruction cache (no-instruction stalls
// 0.38 per issue with two, 0.08 with one).  3 keys: 2^20 x 256 B 135 us a pass
// (148 with the rows loaded in batches between the expansions), 10^6 x 48 B 115
// (242 on the CTA kernel), 2^22 x 128 B 412 (475).

// Stack of a lane: levels 1 .. M - 2 of its walk (stride 32 between levels).
struct LaneStack {
  uint4* seed;
  int8_t* t;  // masks, one byte each (0 or 0xFF; sign-extended on load)
};

// Walk to the node of leaf pair pi (pi even) of the lane's subtree (root at
// tree level F, M levels deep) and, when M >= 2, its sibling, the node of pair
// pi + 1: s0, m0 and s1, m1.  For pi == 0 the caller passes the root in s0, m0;
// otherwise the path re-joins the stack at relative level M - ffs(pi).  The
// right children it passes are pushed, the last one staying in registers.
__device__ __forceinline__ void walk_to_pairs(const KeyDev* K, const KeyAux* A,
                                              const LaneStack st, const uint32_t pi, const uint32_t M,
                                              const uint32_t F, uint4& s0, uint32_t& m0, uint4& s1, uint32_t& m1) {
  uint32_t lvl = 0;
  if (pi) {
    lvl = M - (uint32_t)__ffs((int)pi);
    s0 = st.seed[(lvl - 1) * 32];
    m0 = (uint32_t)(int32_t)st.t[(lvl - 1) * 32];
  }
#pragma unroll 1
  for (; lvl + 1 < M; ++lvl) {
    uint4 Lc;
    uint32_t mlc;
    expand_cw_m(s0, m0, K, A, F + lvl, Lc, mlc, s1, m1);
    if (lvl + 2 < M) {
      st.seed[lvl * 32] = s1;
      st.t[lvl * 32] = (int8_t)m1;
    }
    s0 = Lc;
    m0 = mlc;
  }
}

// 16 bytes copied to shared memory past the L1 cache, without a register.
__device__ __forceinline__ void copy_async(uint4* dst, const uint4* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// The items of a CTA's contiguous range, taken one at a time by its warps: from
// one queue, or from four, each served by the warps of one scheduler (warp w
// issues on scheduler w mod 4) and holding every fourth item, so that a CTA of
// as many warps as items has one for each (contiguous quarters gave some queues
// more items than warps: 175056 x 256 B with 3 keys 44.5 us against 50.8, 60000
// x 32 B 31.4 against 34.2, 20000 x 256 B with 24 keys 43.4 against 50.8).  The
// step is read from the launch parameters: in a register it cost the pair scan
// 0.4% (2^22 x 32 B: 349.6 us against 347.9).  See WarpScanParams.
struct ItemQueue {
  uint64_t first, end;
  uint32_t* next;
  __device__ __forceinline__ ItemQueue(const WarpScanParams& p, uint32_t* s_next, uint32_t warp) {
    const uint32_t q = warp % p.queues;
    first = (uint64_t)blockIdx.x * p.items / gridDim.x + q;
    end = (uint64_t)(blockIdx.x + 1) * p.items / gridDim.x;
    next = s_next + q;
  }
  __device__ __forceinline__ bool take(const WarpScanParams& p, const uint32_t lane, uint64_t& item) const {
    uint32_t rel = 0;
    if (lane == 0) rel = atomicAdd(next, p.queues);
    item = first + __shfl_sync(0xFFFFFFFFu, rel, 0);
    return item < end;
  }
};

__device__ __forceinline__ uint4 shfl_xor4(uint4 v, const uint32_t off) {
  v.x ^= __shfl_xor_sync(0xFFFFFFFFu, v.x, off);
  v.y ^= __shfl_xor_sync(0xFFFFFFFFu, v.y, off);
  v.z ^= __shfl_xor_sync(0xFFFFFFFFu, v.z, off);
  v.w ^= __shfl_xor_sync(0xFFFFFFFFu, v.w, off);
  return v;
}

// Cross-block reduction at the end of a kernel: the CTA XORs its warps' partial
// rows (written by this CTA, visible after the barrier; plain loads, not the
// read-only path) and folds the result into the zeroed shares with 64-bit XOR
// atomics.  XOR is associative and commutative, so the shares do not depend on
// the order.  (The pair scan of rows up to 32 B leaves this to reduce_kernel:
// the extra code changed its register allocation and cost 0.5% on the 31-bit
// pass.)
__device__ __forceinline__ void fold_partials(const WarpScanParams& p, const uint32_t nw) {
  __syncthreads();
  const uint4* const cta_part = p.partial + (uint64_t)blockIdx.x * nw * p.cols;
  for (uint32_t c = threadIdx.x; c < p.cols; c += blockDim.x) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t w = 0; w < nw; ++w) v = xor4(v, cta_part[(size_t)w * p.cols + c]);
    xor_out(p.out + c, v);
  }
}

// VT: uint4 per row (1, 2 or 4).
template <int VT>
__global__ void __launch_bounds__(warp_cta_warps(1) * 32, 1) scan_pair_kernel(const __grid_constant__ WarpScanParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t s_next[4];  // next item of each scheduler's queue
  constexpr bool OWN = VT <= 2;
  constexpr int AV = OWN ? VT : 1;         // accumulators per lane
  constexpr uint32_t RPL = 32 / VT;        // rows of one warp-wide load (exchange)
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t nw = blockDim.x >> 5;
  const uint32_t pos = lane % VT, r0 = lane / VT;
  // Shared memory: leaf masks [nw][64] (exchange only), stacks [nw][slots][32],
  // then the stacks' t masks.
  constexpr uint32_t nm = OWN ? 0u : 64u;
  uint4* const w_mask = reinterpret_cast<uint4*>(smem_raw) + (size_t)warp * nm;
  uint4* const stk4 = reinterpret_cast<uint4*>(smem_raw) + (size_t)nw * nm;
  const LaneStack st = {stk4 + (size_t)warp * p.slots * 32 + lane,
                        reinterpret_cast<int8_t*>(stk4 + (size_t)nw * p.slots * 32) + (size_t)warp * p.slots * 32 + lane};
  uint4* const my_partial = p.partial + ((uint64_t)blockIdx.x * nw + warp) * p.cols;
  const ItemQueue queue(p, s_next, warp);
  if (threadIdx.x < 4) s_next[threadIdx.x] = 0;
  __syncthreads();
  chain_begin();
  for (uint32_t c = lane; c < p.cols; c += 32) my_partial[c] = make_uint4(0u, 0u, 0u, 0u);

  uint4 acc[AV];
#pragma unroll
  for (int v = 0; v < AV; ++v) acc[v] = make_uint4(0u, 0u, 0u, 0u);
  int cur_seg = -1;
  uint32_t cur_group = 0;
  auto flush = [&](const WarpSeg& sg, uint32_t group) {
#pragma unroll
    for (int v = 0; v < AV; ++v) {
      uint4 x = acc[v];
#pragma unroll
      for (uint32_t off = 16; off >= (OWN ? 1u : (uint32_t)VT); off >>= 1) x = shfl_xor4(x, off);
      if (OWN ? lane == (uint32_t)v : lane < (uint32_t)VT) {
        const size_t col = sg.col_base + (size_t)group * VT + (OWN ? (uint32_t)v : lane);
        my_partial[col] = xor4(my_partial[col], x);
      }
      acc[v] = make_uint4(0u, 0u, 0u, 0u);
    }
  };

  for (uint64_t item; queue.take(p, lane, item);) {
    uint32_t si = 0;
    while (si + 1 < p.nsegs && item >= p.seg[si + 1].item_begin) ++si;
    const WarpSeg& sg = p.seg[si];
    const uint64_t local = item - sg.item_begin;
    const uint32_t tile = (uint32_t)(local / sg.groups);
    const uint32_t group = (uint32_t)(local % sg.groups);
    if ((int)si != cur_seg || group != cur_group) {
      if (cur_seg >= 0) flush(p.seg[cur_seg], cur_group);
      cur_seg = (int)si;
      cur_group = group;
    }
    const uint32_t M = sg.M, F = sg.d - M;
    const uint64_t node = (uint64_t)tile * 32 + lane;
    const bool valid = node < sg.nF;
    const KeyDev* K = p.keys + sg.key_base + group;
    const KeyAux* A = p.aux + sg.key_base + group;
    const uint64_t idx = sg.fr_base + (uint64_t)group * sg.nF + node;
    uint4 s0 = valid ? p.fr_seed[idx] : make_uint4(0u, 0u, 0u, 0u);
    uint32_t m0 = (valid && p.fr_t[idx] == 1) ? 0xFFFFFFFFu : 0u;
    const uint4* __restrict__ tbl = sg.table;
    const uint64_t nrows = sg.rows;
    // Table row of the warp tile's first leaf (wraps below the first row).
    const uint64_t row0 = (((sg.first >> M) + (uint64_t)tile * 32) << M) - sg.first;
    const uint32_t pairs = 1u << (M - 1);
    // A warp tile whose 32 x 2^M rows all lie in the table needs no bounds checks.
    const bool full = row0 < nrows && nrows - row0 >= ((uint64_t)32 << M);
    // Row of load j of a step: the lane's own pair, or row r = r0 + j * RPL of
    // the warp's 64 (leaf r mod 2 of lane r / 2; RPL is even).
    auto row_of = [&](int j) {
      return OWN ? ((uint64_t)lane << M) + (uint32_t)(j / VT)
                 : ((uint64_t)((r0 + (uint32_t)j * RPL) >> 1) << M) + (r0 & 1u);
    };
    const uint4* const lp = full ? tbl + (row0 + row_of(0)) * VT + (OWN ? 0u : pos) : tbl;
    const size_t jstep = ((size_t)(RPL >> 1) << M) * VT;  // exchange: from load j to j + 1
    auto run = [&](auto full_tag) {
      constexpr bool FULL = decltype(full_tag)::value;
      for (uint32_t pi = 0; pi < pairs; pi += 2) {
        uint4 s1 = make_uint4(0u, 0u, 0u, 0u);
        uint32_t m1 = 0u;
        walk_to_pairs(K, A, st, pi, M, F, s0, m0, s1, m1);
#pragma unroll 1
        for (uint32_t h = 0; h < 2u && pi + h < pairs; ++h) {
          // The step's rows, loaded before the ChaCha work.
          uint4 dat[2 * VT];
#pragma unroll
          for (int j = 0; j < 2 * VT; ++j) {
            if constexpr (FULL) {
              dat[j] = __ldg(lp + (size_t)(pi + h) * (2 * VT) + (OWN ? (size_t)j : (size_t)j * jstep));
            } else {
              const uint64_t row = row0 + row_of(j) + 2u * (pi + h);
              dat[j] = row < nrows ? __ldg(tbl + row * VT + (OWN ? (uint32_t)(j % VT) : pos))
                                   : make_uint4(0u, 0u, 0u, 0u);
            }
          }
          uint4 ml, mr;
          leaf_pair_m(s0, m0, A, ml, mr);
          if constexpr (OWN) {
#pragma unroll
            for (int v = 0; v < AV; ++v) {
              acc[v] = xor_and(acc[v], dat[v], ml);
              acc[v] = xor_and(acc[v], dat[VT + v], mr);
            }
          } else {
            w_mask[2 * lane] = ml;
            w_mask[2 * lane + 1] = mr;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 2 * VT; ++j) acc[0] = xor_and(acc[0], dat[j], w_mask[r0 + (uint32_t)j * RPL]);
            __syncwarp();
          }
          s0 = s1;
          m0 = m1;
        }
      }
    };
    if (full)
      run(std::true_type{});
    else
      run(std::false_type{});
  }
  if (cur_seg >= 0) flush(p.seg[cur_seg], cur_group);
  if constexpr (!OWN) fold_partials(p, nw);
}

// VT: uint4 per row when it is a power of two (4..32), 0 for any other V up to
// 32 (p.V).  RPL = 32 / V rows are covered by one warp-wide load; V * RPL
// lanes take part and a lane always holds the same 16-byte position of a row.
// Row r of a step (0..63) is leaf r mod 2 of lane r / 2; its mask lies at
// r ^ ((r >> 3) mod 2), so that the lanes' stores of one leaf and the loads of
// consecutive rows both touch all banks.
template <int G, int VT>
__global__ void __launch_bounds__(warp_cta_warps(G) * 32, 1)
    scan_block_kernel(const __grid_constant__ WarpScanParams p) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t s_next[4];  // next item of each scheduler's queue
  constexpr uint32_t kRows = 32u * kBlockLeaves;
  constexpr int CH = block_chunk(VT);  // loads per lane and chunk
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t nw = blockDim.x >> 5;
  const uint32_t V = VT ? (uint32_t)VT : p.V;
  const uint32_t RPL = 32u / V;
  const uint32_t pos = lane % V, r0 = lane / V;
  const bool scans = VT ? true : lane < V * RPL;
  const uint32_t nload = (kRows + RPL - 1) / RPL;  // loads per lane and block
  // Shared memory: masks of two steps [nw][2][G][kRows], the stages of the row
  // chunks [nw][CH][32], stacks [nw][G][slots][32], then the stacks' t masks.
  constexpr uint32_t nm = 2u * G * kRows;
  const uint32_t ns = G * p.slots * 32u;
  uint4* const sm4 = reinterpret_cast<uint4*>(smem_raw);
  uint4* const w_mask = sm4 + (size_t)warp * nm;
  uint4* const w_stage = sm4 + (size_t)nw * nm + (size_t)warp * CH * 32 + lane;
  uint4* const w_stk = sm4 + (size_t)nw * (nm + CH * 32) + (size_t)warp * ns + lane;
  int8_t* const w_stk_t = reinterpret_cast<int8_t*>(sm4 + (size_t)nw * (nm + CH * 32 + ns)) + (size_t)warp * ns + lane;

  uint4* const my_partial = p.partial + ((uint64_t)blockIdx.x * nw + warp) * p.cols;
  for (uint32_t c = lane; c < p.cols; c += 32) my_partial[c] = make_uint4(0u, 0u, 0u, 0u);
  const ItemQueue queue(p, s_next, warp);
  if (threadIdx.x < 4) s_next[threadIdx.x] = 0;
  __syncthreads();

  uint4 acc[G];
#pragma unroll
  for (int k = 0; k < G; ++k) acc[k] = make_uint4(0u, 0u, 0u, 0u);
  int cur_seg = -1;
  uint32_t cur_group = 0, M = 2;

  // Load j of a lane is row r = r0 + j * RPL of the block, off(r) rows below
  // its first row, with its mask at mask_at(r).  When V is a power of two the
  // bits of r0 and j * RPL are disjoint and both maps split into a lane part
  // (r0) and a part of j that is the same for all lanes.
  auto row_off = [&](uint32_t r) { return ((r / kBlockLeaves) << M) + r % kBlockLeaves; };
  auto mask_at = [&](uint32_t r) { return r ^ ((r >> 3) % kBlockLeaves); };
  const uint32_t lane_mask = mask_at(r0);
  auto use_rows = [&](const uint4* masks, const uint4* stage, uint32_t j0) {
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      uint32_t at;
      if constexpr (VT != 0) {
        at = lane_mask ^ mask_at(j0 * RPL) ^ mask_at((uint32_t)j * RPL);
      } else {
        const uint32_t r = r0 + (j0 + (uint32_t)j) * RPL;
        at = mask_at(r < kRows ? r : kRows - 1u);  // past the block the data is zero
      }
      const uint4 row = stage[j * 32];
#pragma unroll
      for (int k = 0; k < G; ++k) acc[k] = xor_and(acc[k], row, masks[k * kRows + at]);
    }
  };

  // The step whose rows are being scanned (all of them in the table): its rows
  // are copied a chunk at a time before, and used after, the node expansions of
  // the next step.
  const uint4* pend_row = nullptr;    // the lane's row 0
  const uint4* pend_mask = w_mask;
  uint32_t pend_j = nload;            // next load; nload: nothing pending
  uint32_t buf_at = 0;                // mask buffer of the next step
  auto load_chunk = [&]() {
    if (pend_j >= nload) return;
    if constexpr (VT != 0) {
      const uint4* const q = pend_row + (size_t)row_off(pend_j * RPL) * V;
#pragma unroll
      for (int j = 0; j < CH; ++j) copy_async(w_stage + j * 32, q + row_off((uint32_t)j * RPL) * V);
    } else {
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const uint32_t r = r0 + (pend_j + (uint32_t)j) * RPL;
        if (scans && r < kRows)
          copy_async(w_stage + j * 32, pend_row + (size_t)row_off(r) * V);
        else
          w_stage[j * 32] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };
  auto use_chunk = [&]() {
    if (pend_j >= nload) return;
    asm volatile("cp.async.wait_all;" ::: "memory");
    use_rows(pend_mask, w_stage, pend_j);
    pend_j += CH;
  };
  auto drain = [&]() {
#pragma unroll 1
    while (pend_j < nload) {
      load_chunk();
      use_chunk();
    }
  };
  auto flush = [&](const WarpSeg& sg, uint32_t group) {
#pragma unroll
    for (int k = 0; k < G; ++k) {
      uint4 v = acc[k];
      if constexpr (VT != 0) {
#pragma unroll
        for (uint32_t off = 16; off >= (uint32_t)VT; off >>= 1) v = shfl_xor4(v, off);
      } else {
        const uint4 x = v;
        for (uint32_t i = 1; i < RPL; ++i) {
          const uint32_t src = (lane + i * V) & 31u;
          v.x ^= __shfl_sync(0xFFFFFFFFu, x.x, src);
          v.y ^= __shfl_sync(0xFFFFFFFFu, x.y, src);
          v.z ^= __shfl_sync(0xFFFFFFFFu, x.z, src);
          v.w ^= __shfl_sync(0xFFFFFFFFu, x.w, src);
        }
      }
      if ((uint32_t)k < sg.g && lane < V) {
        const size_t col = sg.col_base + ((size_t)group * sg.g + k) * V + lane;
        my_partial[col] = xor4(my_partial[col], v);
      }
      acc[k] = make_uint4(0u, 0u, 0u, 0u);
    }
  };

  for (uint64_t item; queue.take(p, lane, item);) {
    uint32_t si = 0;
    while (si + 1 < p.nsegs && item >= p.seg[si + 1].item_begin) ++si;
    const WarpSeg& sg = p.seg[si];
    const uint64_t local = item - sg.item_begin;
    const uint32_t tile = (uint32_t)(local / sg.groups);
    const uint32_t group = (uint32_t)(local % sg.groups);
    const uint32_t g = sg.g;
    if ((int)si != cur_seg || group != cur_group) {
      if (cur_seg >= 0) {
        drain();
        flush(p.seg[cur_seg], cur_group);
      }
      // A segment of fewer than G keys: the other keys' masks are zero, so the
      // row scan needs no test of the key count.
      if ((int)si != cur_seg) {
        __syncwarp();
        for (uint32_t i = lane; i < nm; i += 32) w_mask[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
      }
      cur_seg = (int)si;
      cur_group = group;
      M = sg.M;
    }
    const uint32_t F = sg.d - M;
    const uint64_t node = (uint64_t)tile * 32 + lane;
    const bool valid = node < sg.nF;
    const KeyDev* kp = p.keys + sg.key_base + (size_t)group * g;
    const KeyAux* ap = p.aux + sg.key_base + (size_t)group * g;
    // A key's root waits in its stack's first slot, which level 1 takes over
    // once the walk has read it.
    for (uint32_t k = 0; k < g; ++k) {
      const uint64_t idx = sg.fr_base + ((uint64_t)group * g + k) * sg.nF + node;
      w_stk[k * p.slots * 32] = valid ? p.fr_seed[idx] : make_uint4(0u, 0u, 0u, 0u);
      w_stk_t[k * p.slots * 32] = (valid && p.fr_t[idx] == 1) ? (int8_t)-1 : (int8_t)0;
    }
    const uint4* __restrict__ tbl = sg.table;
    const uint64_t nrows = sg.rows;
    // Table row of the warp tile's first leaf (wraps below the first row).
    const uint64_t row0 = (((sg.first >> M) + (uint64_t)tile * 32) << M) - sg.first;
    // A warp tile whose 32 x 2^M rows all lie in the table needs no bounds
    // checks.
    const bool full = row0 < nrows && nrows - row0 >= ((uint64_t)32 << M);
    const uint32_t pairs = 1u << (M - 1);
    for (uint32_t pi = 0; pi < pairs; ++pi) {
      // The step's masks, key by key.
      uint4* const masks = w_mask + buf_at * (G * kRows);
#pragma unroll 1
      for (uint32_t k = 0; k < g; ++k) {
        uint4* const st_seed = w_stk + k * p.slots * 32;
        int8_t* const st_t = w_stk_t + k * p.slots * 32;
        const KeyDev* K = kp + k;
        const KeyAux* A = ap + k;
        uint32_t lvl = pi ? M - (uint32_t)__ffs((int)pi) : 0u;
        uint4 s = st_seed[(pi ? lvl - 1 : 0u) * 32];
        uint32_t m = (uint32_t)(int32_t)st_t[(pi ? lvl - 1 : 0u) * 32];
        for (bool leaf = false; !leaf;) {
          load_chunk();
          uint4 Lc, Rc;
          uint32_t bl, br;
          prg_expand(s, Lc, Rc, bl, br);
          leaf = lvl + 1 >= M;
          if (!leaf) {
            uint32_t mr;
            apply_cw_m(Lc, Rc, bl, br, m, K, A, F + lvl, m, mr);
            st_seed[lvl * 32] = Rc;
            st_t[lvl * 32] = (int8_t)mr;
            s = Lc;
            ++lvl;
          } else {
            uint4 ml, mr;
            leaf_terms_m(Lc, Rc, bl, br, m, A, ml, mr);
            masks[k * kRows + mask_at(lane * 2u)] = ml;
            masks[k * kRows + mask_at(lane * 2u + 1u)] = mr;
          }
          use_chunk();
        }
      }
      drain();
      __syncwarp();  // the masks are written, and the other buffer's are read
      const uint64_t blk_row0 = row0 + 2u * pi;
      if (full) {
        pend_row = tbl + (blk_row0 + (VT ? row_off(r0) : 0u)) * V + pos;
        pend_mask = masks;
        pend_j = 0;
        buf_at ^= 1u;
      } else {
#pragma unroll 1
        for (uint32_t j0 = 0; j0 < nload; j0 += CH) {
#pragma unroll
          for (int j = 0; j < CH; ++j) {
            const uint32_t r = r0 + (j0 + (uint32_t)j) * RPL;
            const uint64_t row = blk_row0 + row_off(r);
            const bool in = scans && r < kRows && row < nrows;
            w_stage[j * 32] = in ? __ldg(tbl + row * V + pos) : make_uint4(0u, 0u, 0u, 0u);
          }
          use_rows(masks, w_stage, j0);
        }
        __syncwarp();
      }
    }
  }
  if (cur_seg >= 0) {
    drain();
    flush(p.seg[cur_seg], cur_group);
  }
  fold_partials(p, nw);
}

// Whether the warp kernel reduces its partial rows into the shares itself
// or leaves them to reduce_kernel (the pair scan of rows up to 32 B).
bool warp_reduces_in_kernel(int G, uint32_t V) { return G > 1 || V > 2; }

// out[c] ^= XOR over the nparts partial rows (launch_reduce zeroes out first).
// Block (x, y) = cpb columns x (kThreads / cpb) slices over the partial rows
// [y * per_block, (y + 1) * per_block); slices combine in shared memory and
// each block folds its result into out with XOR atomics.
__global__ void __launch_bounds__(kThreads) reduce_kernel(const uint4* partial,
                                                          uint32_t nparts, uint32_t cols,
                                                          uint32_t per_block, uint4* out) {
  chain_begin();
  __shared__ uint4 red[kThreads];
  const uint32_t cpb = cols < 32u ? cols : 32u;
  const uint32_t slices = kThreads / cpb;
  const uint32_t cl = threadIdx.x % cpb, sl = threadIdx.x / cpb;
  const uint32_t c = blockIdx.x * cpb + cl;
  const uint32_t j0 = blockIdx.y * per_block;
  const uint32_t j1 = min(nparts, j0 + per_block);
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (c < cols && sl < slices)
    for (uint32_t j = j0 + sl; j < j1; j += slices) v = xor4(v, partial[(size_t)j * cols + c]);
  red[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < cpb && c < cols) {
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t s = 0; s < slices; ++s) r = xor4(r, red[s * cpb + threadIdx.x]);
    xor_out(out + c, r);
  }
}

// ChaChaKey::eval (dpf.rs:103-142) of one index from its ancestor (s, t) `below`
// levels above the leaves.
__device__ __forceinline__ uint4 eval_below(const KeyDev* K, uint4 s, uint32_t t, uint32_t below,
                                            uint64_t x) {
  const uint32_t d = K->domain_bits;
#pragma unroll 1
  for (uint32_t i = below; i-- > 0;) {
    uint4 Lc, Rc;
    uint32_t tl, tr;
    expand_cw_g(s, t, K, d - 1 - i, Lc, tl, Rc, tr);
    const uint32_t bit = (uint32_t)(x >> i) & 1u;
    s = bit ? Rc : Lc;
    t = bit ? tr : tl;
  }
  return leaf_mask_g(s, t, K);
}

// Pending epoch delta of a table folded into the shares of the pass
// (scan_delta_for_gpu, crates/morphogen-server/src/scan.rs:434-485, in row
// mode): out[col_j] ^= XOR_e diff_e & eval_j(row_e) for every job j (a key
// scanned over this table).  One thread per entry evaluates its row, from the
// row's ancestor in the pass's frontier where there is one (3 keys, 2^22 x 32 B,
// 2^16 entries: 5 levels per entry instead of 22, a call 400 us instead of 497).
// Each 16-byte position is XOR-reduced across the warp with shuffles, then across
// the CTA in shared memory, and the CTA's result is XORed into the share
// with one atomic per word (XOR is order-independent, so the result is
// deterministic).  The entry count is read on the device so that pushes are
// seen by replayed graphs.
__global__ void __launch_bounds__(kThreads) delta_kernel(const KeyDev* keys, const DeltaJob* jobs,
                                                         const uint4* fr_seed, const uint8_t* fr_t,
                                                         const uint64_t* idx, const uint4* diffs,
                                                         const uint32_t* count, uint32_t V, uint64_t first,
                                                         uint4* out) {
  chain_begin();
  __shared__ uint4 s_acc[MG_MAX_ROW_BYTES / 16];
  const uint32_t n = *count;
  const uint64_t e0 = (uint64_t)blockIdx.x * kThreads;
  if (e0 >= n) return;  // uniform per CTA
  const DeltaJob job = jobs[blockIdx.y];
  const KeyDev* K = keys + job.key;
  for (uint32_t v = threadIdx.x; v < V; v += kThreads) s_acc[v] = make_uint4(0u, 0u, 0u, 0u);
  const uint64_t e = e0 + threadIdx.x;
  const bool live = e < n;
  uint4 m = make_uint4(0u, 0u, 0u, 0u);
  if (live) {
    const uint64_t x = first + idx[e];
    if (job.below != ~0u) {
      const uint64_t at = job.fr_base + ((x >> job.below) - job.fr_first);
      m = eval_below(K, fr_seed[at], fr_t[at], job.below, x);
    } else {
      m = eval_below(K, K->root_seed, K->root_t, K->domain_bits, x);
    }
  }
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t v = 0; v < V; ++v) {
    uint4 c = live ? diffs[e * V + v] : make_uint4(0u, 0u, 0u, 0u);
    c.x &= m.x; c.y &= m.y; c.z &= m.z; c.w &= m.w;
#pragma unroll
    for (uint32_t off = 16; off >= 1; off >>= 1) {
      c.x ^= __shfl_xor_sync(0xFFFFFFFFu, c.x, off);
      c.y ^= __shfl_xor_sync(0xFFFFFFFFu, c.y, off);
      c.z ^= __shfl_xor_sync(0xFFFFFFFFu, c.z, off);
      c.w ^= __shfl_xor_sync(0xFFFFFFFFu, c.w, off);
    }
    if (lane == 0 && (c.x | c.y | c.z | c.w)) {
      atomicXor(&s_acc[v].x, c.x);
      atomicXor(&s_acc[v].y, c.y);
      atomicXor(&s_acc[v].z, c.z);
      atomicXor(&s_acc[v].w, c.w);
    }
  }
  __syncthreads();
  for (uint32_t v = threadIdx.x; v < V; v += kThreads) {
    const uint4 a = s_acc[v];
    if (a.x | a.y | a.z | a.w) {
      unsigned int* o = reinterpret_cast<unsigned int*>(out + job.col + v);
      atomicXor(o + 0, a.x);
      atomicXor(o + 1, a.y);
      atomicXor(o + 2, a.z);
      atomicXor(o + 3, a.w);
    }
  }
}

// SplitMix64 output `w` of the stream seeded with `seed` (Steele, Lea, Flood 2014).
__device__ __forceinline__ uint64_t splitmix_word(uint64_t seed, uint64_t w) {
  uint64_t z = seed + (w + 1) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void fill_splitmix_kernel(uint2* __restrict__ dst, uint64_t words, uint64_t seed, uint64_t word0) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += stride) {
    const uint64_t z = splitmix_word(seed, word0 + w);
    dst[w] = make_uint2((uint32_t)z, (uint32_t)(z >> 32));
  }
}

// dst[i] = src[i] for n 16-byte words, and zero[i] = 0 for nz.  Used
// inside the one-call path's graph to move the keys in (clearing the shares
// at the same time) and the shares out through the pinned host buffers'
// device-mapped addresses: a kernel node of a few hundred threads finishes
// sooner than a copy-engine transfer of a few KB.
__global__ void copy_u4_kernel(const uint4* src, uint4* dst, uint32_t n, uint4* zero, uint32_t nz) {
  chain_begin();
  const uint32_t m = n > nz ? n : nz;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    if (i < n) dst[i] = src[i];
    if (i < nz) zero[i] = make_uint4(0u, 0u, 0u, 0u);
  }
}

// table[row_idx[e]] ^= diff[e]; XOR atomics make duplicate rows in one batch
// order-independent.
__global__ void xor_rows_kernel(uint4* __restrict__ table, uint32_t V, const uint64_t* __restrict__ idx,
                                const uint4* __restrict__ diffs, uint64_t n) {
  const uint64_t total = n * V;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const uint64_t e = i / V;
    const uint32_t ln = (uint32_t)(i % V);
    const uint4 dv = diffs[i];
    unsigned int* t = reinterpret_cast<unsigned int*>(table + idx[e] * V + ln);
    atomicXor(t + 0, dv.x);
    atomicXor(t + 1, dv.y);
    atomicXor(t + 2, dv.z);
    atomicXor(t + 3, dv.w);
  }
}

// ChaChaKey::eval (dpf.rs:103-142) at n indices, one thread per index.
__global__ void eval_points_kernel(const KeyDev* key, const uint64_t* __restrict__ idx,
                                   uint64_t n, uint4* __restrict__ out) {
  __shared__ KeyDev sk;
  {
    const uint4* src = reinterpret_cast<const uint4*>(key);
    uint4* dst = reinterpret_cast<uint4*>(&sk);
    for (uint32_t i = threadIdx.x; i < sizeof(KeyDev) / 16; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint64_t x = idx[i];
    uint4 s = sk.root_seed;
    uint32_t t = sk.root_t;
    const uint32_t d = sk.domain_bits;
    for (uint32_t lvl = 0; lvl < d; ++lvl) {
      uint4 Lc, Rc;
      uint32_t tl, tr;
      expand_cw(s, t, sk, lvl, Lc, tl, Rc, tr);
      const uint32_t bit = (uint32_t)(x >> (d - 1 - lvl)) & 1u;
      s = bit ? Rc : Lc;
      t = bit ? tr : tl;
    }
    out[i] = leaf_mask(s, t, sk);
  }
}

// PRG-only ceiling: every thread chains `iters` node expansions (left child,
// t folded in) with no memory traffic -- the best the ChaCha8 code above can
// do on this GPU, the ALU roofline of the scan kernel.
__global__ void __launch_bounds__(256) prg_peak_kernel(uint32_t* __restrict__ out, uint32_t iters) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  uint4 s = make_uint4(tid, tid * 0x9E3779B9u, ~tid, 0x01234567u);
  uint32_t acc = 0;
  for (uint32_t i = 0; i < iters; ++i) {
    uint4 L, R;
    uint32_t tl, tr;
    prg_expand(s, L, R, tl, tr);
    s = make_uint4(L.x ^ R.w, L.y ^ tl, L.z ^ tr, L.w ^ R.x);
    acc += R.y;
  }
  out[tid] = s.x ^ s.y ^ s.z ^ s.w ^ acc;
}

// ---- host-side launchers --------------------------------------------------

// Launch a kernel that begins with chain_begin() or chain_wait(): when the work
// before it on the stream is such a kernel too, it need not have completed for
// this one's launch to be processed (programmatic stream serialization; a
// captured graph gets programmatic edges).  One call, 3 keys, without and with:
// 4099 x 32 B 47.9 and 47.5 us, 1000003 x 48 B 146.0 and 144.3, 1300021 x 4 KB
// pages 1020 and 1016; calls of milliseconds take the same.
template <class... P, class... A>
static cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, uint32_t threads, size_t smem, cudaStream_t st,
                                  A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// The dynamic shared memory limit of a kernel (cudaFuncAttributeMax-
// DynamicSharedMemorySize) belongs to the kernel function on its device, for
// the whole process: every context, workspace and the allocation-free entry
// point see the same value.  It is therefore kept here as one high-water mark
// per (device, kernel) under one mutex and only ever raised, so that a caller
// preparing a small launch can never lower the limit under another caller's
// larger launch.
namespace {
std::mutex g_smem_mu;
std::map<std::pair<int, const void*>, size_t> g_smem_limit;

cudaError_t raise_smem_limit(const void* fn, size_t smem) {
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  std::lock_guard<std::mutex> lk(g_smem_mu);
  size_t& have = g_smem_limit[{dev, fn}];
  if (have >= smem) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) have = smem;
  return e;
}
}  // namespace

cudaError_t prg_peak_shape(int sms, uint32_t* blocks, uint32_t* threads) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, prg_peak_kernel, 256, 0);
  if (e != cudaSuccess) return e;
  *threads = 256;
  *blocks = (uint32_t)(per_sm > 0 ? per_sm : 1) * (uint32_t)sms * 4;
  return cudaSuccess;
}

cudaError_t launch_prg_peak(uint32_t* out, uint32_t iters, uint32_t blocks, uint32_t threads,
                            cudaStream_t st) {
  prg_peak_kernel<<<blocks, threads, 0, st>>>(out, iters);
  return cudaGetLastError();
}

size_t scan_smem_bytes(int G, uint32_t slots) {
  return (size_t)G * (sizeof(KeyDev) + 2 * kThreads * 16 + (size_t)slots * kThreads * 17);
}

using ScanKernel = void (*)(const ScanParams);
template <bool FMA>
static ScanKernel scan_kernel_of(int G) {
  switch (G) {
    case 1: return scan_kernel<1, FMA>;
    case 2: return scan_kernel<2, FMA>;
    case 3: return scan_kernel<3, FMA>;
    case 4: return scan_kernel<4, FMA>;
    case 8: return scan_kernel<8, FMA>;
    default: return nullptr;
  }
}
static ScanKernel scan_kernel_of(int G, bool fma) { return fma ? scan_kernel_of<true>(G) : scan_kernel_of<false>(G); }

bool scan_g_supported(int G) { return G == 1 || G == 2 || G == 3 || G == 4 || G == 8; }

cudaError_t scan_prepare(int G, bool fma, size_t smem) {
  const ScanKernel k = scan_kernel_of(G, fma);
  return k ? raise_smem_limit(reinterpret_cast<const void*>(k), smem) : cudaErrorInvalidValue;
}

int scan_occupancy(int G, bool fma, size_t smem) {
  const ScanKernel k = scan_kernel_of(G, fma);
  int n = 0;
  if (!k || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kThreads, smem) != cudaSuccess) return 0;
  return n;
}

// Rows under 2 KB leave the pass bound by its node expansions as much as by
// memory, and the balanced PRG is faster: 3 keys, 10^6 x 528 B 239 us against
// 252 all-ALU.  So it is for the rows of 16 to 512 B that come here with the
// kernel pinned or from mg_scan_noalloc (pinned, then noalloc): 2^20 x 16 B 180
// against 193 and 224 against 240, 2^23 x 32 B 900 against 986 and 974 against
// 1061, 2^20 x 256 B 187 against 198 and 278 against 296, 12 keys over 2^19 x
// 512 B 351 against 367 and 561 against 590; tables of one wave (20000 rows)
// take either.  Wider rows are bound by HBM and its power, where the all-ALU
// form with fewer instructions wins (1300021 x 4 KB: 887 us against 925).
bool scan_fma(uint32_t V) { return V < 128; }

cudaError_t launch_scan(int G, bool fma, const ScanParams& p, uint32_t grid, size_t smem, cudaStream_t st) {
  const ScanKernel k = scan_kernel_of(G, fma);
  if (!k) return cudaErrorInvalidValue;
  // Not launched early: beside a kernel that still holds some of the SMs, its
  // three CTAs per SM are placed unevenly for the whole pass (beside its
  // frontier, 3 keys, 10^6 x 528 B: 269 us against 239; 48 keys, 100000 x 4 KB:
  // 1010 against 885).
  k<<<grid, kThreads, smem, st>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_reduce(const uint4* partial, uint32_t nparts, uint32_t cols, uint4* out,
                          cudaStream_t st, bool out_zeroed) {
  if (cols == 0) return cudaSuccess;
  if (!out_zeroed)
    if (cudaError_t e = cudaMemsetAsync(out, 0, (size_t)cols * 16, st)) return e;
  const uint32_t cpb = cols < 32u ? cols : 32u;
  const uint32_t slices = kThreads / cpb;
  const uint32_t per_block = slices * 4;  // at most 4 partial rows per thread
  const dim3 grid((cols + cpb - 1) / cpb, nparts ? (nparts + per_block - 1) / per_block : 1);
  return launch_chained(reduce_kernel, grid, kThreads, 0, st, partial, nparts, cols, per_block, out);
}

cudaError_t launch_copy_u4(const void* src, void* dst, uint32_t n, cudaStream_t st, void* zero, uint32_t nz) {
  const uint32_t m = n > nz ? n : nz;
  if (m == 0) return cudaSuccess;
  const uint32_t blocks = (m + kThreads - 1) / kThreads < 32u ? (m + kThreads - 1) / kThreads : 32u;
  return launch_chained(copy_u4_kernel, dim3(blocks), kThreads, 0, st, static_cast<const uint4*>(src),
                        static_cast<uint4*>(dst), n, static_cast<uint4*>(zero), nz);
}

cudaError_t launch_fill_splitmix(void* dst, uint64_t words, uint64_t seed, uint64_t word0, int sms, cudaStream_t st) {
  if (words == 0) return cudaSuccess;
  uint64_t blocks = (words + 255) / 256;
  const uint64_t cap = (uint64_t)sms * 16;
  if (blocks > cap) blocks = cap;
  fill_splitmix_kernel<<<(unsigned)blocks, 256, 0, st>>>(reinterpret_cast<uint2*>(dst), words, seed, word0);
  return cudaGetLastError();
}

cudaError_t launch_xor_rows(void* table, uint32_t V, const uint64_t* idx, const void* diffs,
                            uint64_t n, int sms, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  uint64_t blocks = (n * V + 255) / 256;
  const uint64_t cap = (uint64_t)sms * 16;
  if (blocks > cap) blocks = cap;
  xor_rows_kernel<<<(unsigned)blocks, 256, 0, st>>>(reinterpret_cast<uint4*>(table), V, idx,
                                                     reinterpret_cast<const uint4*>(diffs), n);
  return cudaGetLastError();
}

cudaError_t launch_eval_points(const KeyDev* key, const uint64_t* idx, uint64_t n, void* out, int sms,
                               cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  uint64_t blocks = (n + 127) / 128;
  const uint64_t cap = (uint64_t)sms * 8;
  if (blocks > cap) blocks = cap;
  eval_points_kernel<<<(unsigned)blocks, 128, 0, st>>>(key, idx, n, reinterpret_cast<uint4*>(out));
  return cudaGetLastError();
}

// ---- warp-path launchers --------------------------------------------------

// Levels of a lane's stack: 1 .. M - 2 (the last right child stays in
// registers); the block scan keeps a key's root in the first slot too.
uint32_t warp_slots(int G, uint32_t V, uint32_t M) { const uint32_t top = pair_scan(G, V) ? 2 : 1; return M > top ? M - top : 1; }

// Dynamic shared memory of a warp-kernel CTA of nw warps.  Pair scan: a stack
// per warp, and for 64-B rows a step's masks.  Block scan: a stage per warp, and
// two steps' masks and a stack per key and warp.
size_t warp_smem_bytes(int G, uint32_t V, uint32_t slots, uint32_t nw) {
  if (pair_scan(G, V)) return (size_t)nw * 32 * ((V > 2 ? 2 * 16 : 0) + (size_t)slots * 17);
  return (size_t)nw * 32 * ((size_t)block_chunk(V) * 16 + (size_t)G * (2 * kBlockLeaves * 16 + (size_t)slots * 17));
}

bool warp_vt_supported(uint32_t V) { return V >= 1 && V <= 32; }

using WarpKernel = void (*)(const WarpScanParams);
template <int G>
static WarpKernel block_kernel(uint32_t V) {
  switch (V) {
    case 4: return scan_block_kernel<G, 4>;
    case 8: return scan_block_kernel<G, 8>;
    case 16: return scan_block_kernel<G, 16>;
    case 32: return scan_block_kernel<G, 32>;
    default: return scan_block_kernel<G, 0>;
  }
}
static WarpKernel warp_kernel(int G, uint32_t V) {
  if (!warp_vt_supported(V)) return nullptr;
  if (pair_scan(G, V)) return V == 1 ? scan_pair_kernel<1> : V == 2 ? scan_pair_kernel<2> : scan_pair_kernel<4>;
  switch (G) {
    case 1: return block_kernel<1>(V);
    case 2: return block_kernel<2>(V);
    case 3: return block_kernel<3>(V);
    case 4: return block_kernel<4>(V);
    default: return nullptr;
  }
}

bool warp_g_supported(int G) { return G >= 1 && G <= 4; }

cudaError_t warp_prepare(int G, uint32_t V, size_t smem) {
  const WarpKernel k = warp_kernel(G, V);
  return k ? raise_smem_limit(reinterpret_cast<const void*>(k), smem) : cudaErrorInvalidValue;
}
int warp_occupancy(int G, uint32_t V, size_t smem, uint32_t nw) {
  const WarpKernel k = warp_kernel(G, V);
  int n = 0;
  if (!k || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, (int)(nw * 32), smem) != cudaSuccess) return 0;
  return n;
}
cudaError_t launch_scan_warp(int G, uint32_t V, const WarpScanParams& p, uint32_t grid, uint32_t nw, size_t smem,
                             cudaStream_t st) {
  const WarpKernel k = warp_kernel(G, V);
  if (!k) return cudaErrorInvalidValue;
  return launch_chained(k, dim3(grid), nw * 32, smem, st, p);
}

cudaError_t launch_delta(const KeyDev* keys, const DeltaJob* jobs, uint32_t njobs, const uint4* fr_seed,
                         const uint8_t* fr_t, const uint64_t* idx,
                         const void* diffs, const uint32_t* count, uint32_t capacity, uint32_t V, uint64_t first,
                         uint4* out, cudaStream_t st) {
  if (njobs == 0 || capacity == 0) return cudaSuccess;
  dim3 grid((capacity + kThreads - 1) / kThreads, njobs);
  return launch_chained(delta_kernel, grid, kThreads, 0, st, keys, jobs, fr_seed, fr_t, idx,
                        static_cast<const uint4*>(diffs), count, V, first, out);
}

cudaError_t launch_frontier(const FrontierStep& f, uint32_t nkeys, cudaStream_t st) {
  if (f.n_in == 0 || nkeys == 0) return cudaSuccess;
  if (f.c > kFrontierLevels || f.L_in + f.c > (uint32_t)kMaxLevels) return cudaErrorInvalidValue;
  dim3 grid((unsigned)f.n_in, nkeys);
  return launch_chained(frontier_kernel, grid, kThreads, 0, st, f);
}

}  // namespace mg
