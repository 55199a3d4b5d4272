// mg_device.cuh -- device-side ChaCha8 GGM PRG and DPF key layout (sm_100a).
//
// The PRG is the reference's ChaCha8Prg::expand
// (crates/morphogen-gpu-dpf/src/chacha_prg.rs:153-178): ChaCha key = seed||seed,
// nonce 0, two blocks with counters 0 and 1 (RFC 8439 state layout, 4 double
// rounds, feed-forward add, chacha_prg.rs:112-144).  Children: L = block0[0..4],
// R = block0[4..8], tL = block1[0] & 1, tR = block1[1] & 1.
//
// B200 notes: the path is bound by integer issue.  XOR/AND (LOP3), funnel
// shifts (SHF) and byte permutes (PRMT) go to the ALU pipe and two-input adds
// to the FMA pipe, both at 16 lanes per clock per scheduler, so a node
// expansion written with one instruction per operation keeps the ALU pipe full
// (456 instructions) and the FMA pipe half idle (227).  Rotations by 16 and 8
// are whole bytes, and a byte-wise dot product plus a multiply-add does one on
// the FMA pipe (rotl_bytes): with 70 of them there, about 387 ALU and 366 FMA
// instructions, 40.2 -> 45.2 G node expansions/s for the PRG alone
// (mg_prg_peak).  More of them loses to the issue rate (one instruction per
// clock and scheduler, 755 per expansion), fewer to the ALU pipe.  Both blocks
// are written out in one straight-line function so the compiler shares the
// three counter-independent column quarter rounds of round 1 and drops the
// parts of block 1 that do not reach bit 0 of words 0 and 1.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace mg {

constexpr int kThreads = 256;    // CTA size of the scan kernel
constexpr int kMaxLevels = 32;   // MG_MAX_DOMAIN_BITS
constexpr int kMaxSegs = 8;      // (table, domain) segments per launch
constexpr uint32_t kSigma0 = 0x61707865u;  // "expand 32-byte k"
constexpr uint32_t kSigma1 = 0x3320646eu;
constexpr uint32_t kSigma2 = 0x79622d32u;
constexpr uint32_t kSigma3 = 0x6b206574u;

// Device key: the wire key (dpf.rs:259-274) re-laid out for 16-byte loads.
// t bytes keep the reference's byte semantics (a node applies its correction
// word iff t == 1, dpf.rs:122,192,228).
struct alignas(16) KeyDev {
  uint4 root_seed;
  uint4 final_cw;
  uint4 cw_seed[kMaxLevels];
  uint8_t cw_tl[kMaxLevels];
  uint8_t cw_tr[kMaxLevels];
  uint32_t root_t;
  uint32_t domain_bits;
  uint32_t pad[2];
};
static_assert(sizeof(KeyDev) == 624, "KeyDev layout");

// Per-key constants of the warp-independent kernel, derived on the host from
// the key.  That kernel carries a node's t as a mask (all ones iff t == 1);
// for a parent mask m and the PRG's child bit b, the child's mask is
//   (-b ^ (one & m)) & ~(big & m)
// where, per level and side, one = all ones iff the t correction byte is 1
// and big = all ones iff it is 2..255 (the child's t byte is then >= 2 and
// never corrects).  This equals the byte rule of dpf.rs:122,192,228 exactly.
// A last-level child's mask is only needed to pick its leaf's XOR term, so
// that step is a table lookup by the parent's bit p and the child's PRG bit b:
// leaf[4 * side + 2 * p + b] = (p ? cw_seed[d - 1] : 0) ^ (c ? final_cw : 0)
// with c the child's corrected bit (side 0 left, 1 right); the leaf mask is
// the PRG seed XOR that entry.
struct alignas(16) KeyAux {
  uint4 cw_tm[kMaxLevels];  // x: tl one, y: tl big, z: tr one, w: tr big (0 or ~0)
  uint4 leaf[8];
};
static_assert(sizeof(KeyAux) == 640, "KeyAux layout");

__device__ __forceinline__ uint32_t rotl12(uint32_t x) { return __funnelshift_l(x, x, 12); }
__device__ __forceinline__ uint32_t rotl7(uint32_t x) { return __funnelshift_l(x, x, 7); }

// 2^16 and 2^8 read from constant memory: a multiplier the compiler cannot
// see stays an integer multiply-add (with an immediate power of two it may
// become a shift, which is back on the ALU pipe).
static __constant__ uint32_t kRotMul[2] = {1u << 16, 1u << 8};

// rotl by 16 or 8, on the ALU pipe (one byte permute) or, with FMA set, as two
// multiply-adds on the otherwise half-idle FMA pipe: the part shifted down is
// a dot product with a one-hot byte vector (dp2a selects the upper half-word,
// dp4a the top byte), and a multiply-add places the part shifted up above it.
template <int N, bool FMA>
__device__ __forceinline__ uint32_t rotl_bytes(uint32_t x) {
  static_assert(N == 16 || N == 8, "whole bytes");
  if constexpr (!FMA) return __byte_perm(x, 0, N == 16 ? 0x1032 : 0x2103);
  const uint32_t down = N == 16 ? __dp2a_lo(x, 0x00000100u, 0u) : __dp4a(x, 0x01000000u, 0u);
  return x * kRotMul[N == 16 ? 0 : 1] + down;
}

template <bool F16, bool F8>
__device__ __forceinline__ void quarter_round(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  a += b; d ^= a; d = rotl_bytes<16, F16>(d);
  c += d; b ^= c; b = rotl12(b);
  a += b; d ^= a; d = rotl_bytes<8, F8>(d);
  c += d; b ^= c; b = rotl7(b);
}

// Which of a block's rotations by 16 and 8 run on the FMA pipe (FMA set), by
// round and quarter round: the 16s of quarter rounds 0..2 and the 8s of the
// diagonal rounds, about 70 of the 114 that matter.  Which ones matters little
// for the PRG alone; of 72 such choices this was the best over the pair scan's
// three kernels (between 2.51 and 2.63 ms for 3 keys over 2^25 x 32 B).
template <bool FMA, int RD, int C>
__device__ __forceinline__ void qr_at(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  quarter_round<FMA && C != 3, FMA && (RD & 1) != 0>(a, b, c, d);
}

template <bool FMA, int DR>
__device__ __forceinline__ void double_round(uint32_t (&x)[16]) {
  qr_at<FMA, 2 * DR, 0>(x[0], x[4], x[8], x[12]);
  qr_at<FMA, 2 * DR, 1>(x[1], x[5], x[9], x[13]);
  qr_at<FMA, 2 * DR, 2>(x[2], x[6], x[10], x[14]);
  qr_at<FMA, 2 * DR, 3>(x[3], x[7], x[11], x[15]);
  qr_at<FMA, 2 * DR + 1, 0>(x[0], x[5], x[10], x[15]);
  qr_at<FMA, 2 * DR + 1, 1>(x[1], x[6], x[11], x[12]);
  qr_at<FMA, 2 * DR + 1, 2>(x[2], x[7], x[8], x[13]);
  qr_at<FMA, 2 * DR + 1, 3>(x[3], x[4], x[9], x[14]);
}

// ChaCha8Prg::expand.  tl/tr are 0 or 1.  FMA balances the two integer pipes
// (throughput); without it every rotation is one ALU instruction, a shorter
// dependent chain for code that walks a path with few warps at work.
template <bool FMA = true>
__device__ __forceinline__ void prg_expand(const uint4 s, uint4& L, uint4& R, uint32_t& tl,
                                           uint32_t& tr) {
  uint32_t x[16] = {kSigma0, kSigma1, kSigma2, kSigma3, s.x, s.y, s.z, s.w, s.x, s.y, s.z, s.w, 0u, 0u, 0u, 0u};
  uint32_t y[16] = {kSigma0, kSigma1, kSigma2, kSigma3, s.x, s.y, s.z, s.w, s.x, s.y, s.z, s.w, 1u, 0u, 0u, 0u};
  double_round<FMA, 0>(x); double_round<FMA, 0>(y);
  double_round<FMA, 1>(x); double_round<FMA, 1>(y);
  double_round<FMA, 2>(x); double_round<FMA, 2>(y);
  double_round<FMA, 3>(x); double_round<FMA, 3>(y);
  L = make_uint4(x[0] + kSigma0, x[1] + kSigma1, x[2] + kSigma2, x[3] + kSigma3);
  R = make_uint4(x[4] + s.x, x[5] + s.y, x[6] + s.z, x[7] + s.w);
  tl = (y[0] + kSigma0) & 1u;
  tr = (y[1] + kSigma1) & 1u;
}

// One of a node expansion's two blocks: L, R hold its words 0-3 and 4-7 (block
// 0: the children's seeds; block 1: their t bits in bit 0 of L.x and L.y).
// Two lanes expand a node together where the dependent chain counts and not
// the throughput: about 1000 cycles, where both blocks in a lane take 1700.
__device__ __forceinline__ void prg_block(const uint4 s, const uint32_t counter, uint4& L, uint4& R) {
  uint32_t x[16] = {kSigma0, kSigma1, kSigma2, kSigma3, s.x, s.y, s.z, s.w, s.x, s.y, s.z, s.w, counter, 0u, 0u, 0u};
  double_round<false, 0>(x);
  double_round<false, 1>(x);
  double_round<false, 2>(x);
  double_round<false, 3>(x);
  L = make_uint4(x[0] + kSigma0, x[1] + kSigma1, x[2] + kSigma2, x[3] + kSigma3);
  R = make_uint4(x[4] + s.x, x[5] + s.y, x[6] + s.z, x[7] + s.w);
}

// The same block over four neighbouring lanes, one column of the state each
// (all 32 lanes call it): lane `col` of four passes word `col` of the seed and
// gets words col and 4 + col of the block.  The diagonal rounds cost three
// shuffles on either side, so the chain is no shorter than prg_block's, but it
// issues a quarter of the instructions.
__device__ __forceinline__ void prg_block_quad(const uint32_t col, const uint32_t s, const uint32_t counter, uint32_t& l,
                                               uint32_t& r) {
  const uint32_t sigma = col == 0 ? kSigma0 : col == 1 ? kSigma1 : col == 2 ? kSigma2 : kSigma3;
  uint32_t a = sigma, b = s, c = s, d = col == 0 ? counter : 0u;
#pragma unroll
  for (int dr = 0; dr < 4; ++dr) {
    quarter_round<false, false>(a, b, c, d);
    b = __shfl_sync(0xFFFFFFFFu, b, (int)(col + 1u) & 3, 4);
    c = __shfl_sync(0xFFFFFFFFu, c, (int)(col + 2u) & 3, 4);
    d = __shfl_sync(0xFFFFFFFFu, d, (int)(col + 3u) & 3, 4);
    quarter_round<false, false>(a, b, c, d);
    b = __shfl_sync(0xFFFFFFFFu, b, (int)(col + 3u) & 3, 4);
    c = __shfl_sync(0xFFFFFFFFu, c, (int)(col + 2u) & 3, 4);
    d = __shfl_sync(0xFFFFFFFFu, d, (int)(col + 1u) & 3, 4);
  }
  l = a + sigma;
  r = b + s;
}

// One GGM node expansion with the level's correction word applied to both
// children when t == 1 (dpf.rs:221-239).
template <bool FMA = true>
__device__ __forceinline__ void expand_cw(const uint4 s, const uint32_t t, const KeyDev& k,
                                          const uint32_t level, uint4& L, uint32_t& tl, uint4& R,
                                          uint32_t& tr) {
  const uint4 cw = k.cw_seed[level];
  const uint32_t cwl = k.cw_tl[level];
  const uint32_t cwr = k.cw_tr[level];
  prg_expand<FMA>(s, L, R, tl, tr);
  const uint32_t m = (t == 1u) ? 0xFFFFFFFFu : 0u;
  L.x ^= cw.x & m; L.y ^= cw.y & m; L.z ^= cw.z & m; L.w ^= cw.w & m;
  R.x ^= cw.x & m; R.y ^= cw.y & m; R.z ^= cw.z & m; R.w ^= cw.w & m;
  tl ^= cwl & m;
  tr ^= cwr & m;
}

// Leaf output: seed, XOR final_cw when t == 1 (dpf.rs:136-139, 211-218).
__device__ __forceinline__ uint4 leaf_mask(const uint4 s, const uint32_t t, const KeyDev& k) {
  const uint32_t m = (t == 1u) ? 0xFFFFFFFFu : 0u;
  const uint4 f = k.final_cw;
  return make_uint4(s.x ^ (f.x & m), s.y ^ (f.y & m), s.z ^ (f.z & m), s.w ^ (f.w & m));
}

// Same as expand_cw with the key in global memory (it is uniform across a
// warp, so every load is a broadcast L1 hit).  Keys and their constants are
// read with plain loads: the pass's first kernel writes them, and a kernel of
// the pass may have been launched before that one has ended.
template <bool FMA = true>
__device__ __forceinline__ void expand_cw_g(const uint4 s, const uint32_t t, const KeyDev* k,
                                            const uint32_t level, uint4& L, uint32_t& tl, uint4& R,
                                            uint32_t& tr) {
  const uint4 cw = k->cw_seed[level];
  const uint32_t cwl = k->cw_tl[level];
  const uint32_t cwr = k->cw_tr[level];
  prg_expand<FMA>(s, L, R, tl, tr);
  const uint32_t m = (t == 1u) ? 0xFFFFFFFFu : 0u;
  L.x ^= cw.x & m; L.y ^= cw.y & m; L.z ^= cw.z & m; L.w ^= cw.w & m;
  R.x ^= cw.x & m; R.y ^= cw.y & m; R.z ^= cw.z & m; R.w ^= cw.w & m;
  tl ^= cwl & m;
  tr ^= cwr & m;
}

__device__ __forceinline__ uint4 leaf_mask_g(const uint4 s, const uint32_t t, const KeyDev* k) {
  const uint32_t m = (t == 1u) ? 0xFFFFFFFFu : 0u;
  const uint4 f = k->final_cw;
  return make_uint4(s.x ^ (f.x & m), s.y ^ (f.y & m), s.z ^ (f.z & m), s.w ^ (f.w & m));
}

// The level's correction word on a node's children as prg_expand gives them
// (seeds L, R, bits bl, br), with t carried as a mask (KeyAux): m is all ones
// iff the parent's t == 1; ml / mr are the children's masks.
__device__ __forceinline__ void apply_cw_m(uint4& L, uint4& R, const uint32_t bl, const uint32_t br, const uint32_t m,
                                           const KeyDev* k, const KeyAux* a,
                                           const uint32_t level, uint32_t& ml, uint32_t& mr) {
  const uint4 cw = k->cw_seed[level];
  const uint4 tm = a->cw_tm[level];
  L.x ^= cw.x & m; L.y ^= cw.y & m; L.z ^= cw.z & m; L.w ^= cw.w & m;
  R.x ^= cw.x & m; R.y ^= cw.y & m; R.z ^= cw.z & m; R.w ^= cw.w & m;
  ml = ((0u - bl) ^ (tm.x & m)) & ~(tm.y & m);
  mr = ((0u - br) ^ (tm.z & m)) & ~(tm.w & m);
}

// Last level (level d - 1): both children's leaf masks straight from the PRG
// seeds, with the level's correction word and the final correction word
// folded into one table entry per child.
__device__ __forceinline__ void leaf_terms_m(const uint4 L, const uint4 R, const uint32_t bl, const uint32_t br,
                                             const uint32_t m, const KeyAux* a, uint4& mask_l,
                                             uint4& mask_r) {
  const uint32_t p2 = m & 2u;  // 2 * parent bit
  const uint4 cl = a->leaf[p2 | bl];
  const uint4 cr = a->leaf[4u + (p2 | br)];
  mask_l = make_uint4(L.x ^ cl.x, L.y ^ cl.y, L.z ^ cl.z, L.w ^ cl.w);
  mask_r = make_uint4(R.x ^ cr.x, R.y ^ cr.y, R.z ^ cr.z, R.w ^ cr.w);
}

// One node expansion with the level's correction word, t carried as a mask.
__device__ __forceinline__ void expand_cw_m(const uint4 s, const uint32_t m, const KeyDev* k,
                                            const KeyAux* a, const uint32_t level, uint4& L,
                                            uint32_t& ml, uint4& R, uint32_t& mr) {
  uint32_t bl, br;
  prg_expand(s, L, R, bl, br);
  apply_cw_m(L, R, bl, br, m, k, a, level, ml, mr);
}

// The leaf pair below node s of level d - 1.
__device__ __forceinline__ void leaf_pair_m(const uint4 s, const uint32_t m, const KeyAux* a,
                                            uint4& mask_l, uint4& mask_r) {
  uint4 L, R;
  uint32_t bl, br;
  prg_expand(s, L, R, bl, br);
  leaf_terms_m(L, R, bl, br, m, a, mask_l, mask_r);
}

__device__ __forceinline__ uint4 xor_and(uint4 acc, const uint4 d, const uint4 m) {
  acc.x ^= d.x & m.x; acc.y ^= d.y & m.y; acc.z ^= d.z & m.z; acc.w ^= d.w & m.w;
  return acc;
}
__device__ __forceinline__ uint4 xor4(uint4 a, const uint4 b) {
  a.x ^= b.x; a.y ^= b.y; a.z ^= b.z; a.w ^= b.w;
  return a;
}

// One (table, domain) segment of a pass.  Work items of the segment are
// (tile, group) pairs, tile-major so that CTAs running at the same time
// share row tiles through L2.
struct Segment {
  const uint4* table;   // rows * V uint4, row-major
  uint64_t first;       // logical index of table row 0 (row-range tables)
  uint64_t rows;        // rows scanned (first + rows <= 2^d)
  uint64_t item_begin;  // first global item index of the segment
  uint32_t tiles;       // 2^S-leaf tiles intersecting [first, first + rows)
  uint32_t groups;      // key groups
  uint32_t V;           // uint4 per row (row_bytes / 16), 1..256
  uint32_t d;           // domain bits of every key in the segment
  uint32_t S;           // tile depth: 2^S leaves per item (S <= d)
  uint32_t U;           // breadth-first levels below the tile root (2^U DFS roots)
  uint32_t M;           // depth-first levels per thread (S - U)
  uint32_t g;           // keys per group (<= kernel G)
  uint32_t key_base;    // KeyDev index of group 0, key 0
  uint32_t col_base;    // partial column of group 0, key 0, lane 0
  uint64_t fr_base;     // frontier index of group 0, key 0 (key j at fr_base + j * tiles)
};

struct ScanParams {
  Segment seg[kMaxSegs];
  const KeyDev* keys;
  uint4* partial;       // [gridDim.x][cols]
  uint64_t items;
  uint32_t nsegs;
  uint32_t cols;        // total share uint4s of the pass
  uint32_t slots;       // stack slots per key per thread allocated in smem
  const uint4* fr_seed; // frontier holding every key's tile roots, or null: CTAs walk to them
  const uint8_t* fr_t;
};

// ---- warp-independent scan ------------------------------------------------
//
// A frontier holds, for every key, the tree nodes at level F = d - M whose
// subtrees intersect the table's rows [first, first + rows).  A warp work
// item is 32 consecutive frontier nodes of one key group ("warp tile", 32 x
// 2^M rows); each lane walks its node's 2^M leaves depth-first.

// One key per warp and rows of 16, 32 or 64 B: the pair scan (a step is one
// leaf pair per lane, its rows in registers beside the ChaCha state).  Other
// row sizes up to 512 B, or several keys per warp: the block scan.
__host__ __device__ constexpr bool pair_scan(int G, uint32_t V) { return G == 1 && (V == 1 || V == 2 || V == 4); }

// Widest CTA of the warp-independent kernels, one CTA per SM; four warps fewer
// at a time when the shared memory does not hold it.  One key per warp: 20
// warps, whose registers fit 96.  With the ALU and FMA pipes both near their
// limit a fifth warp per scheduler hides what is left of the fixed-latency
// waits (3 keys, 2^28 x 32 B: 19.8-20.0 ms against 20.1-20.3 with 16; 12 keys,
// 3000000 x 64 B: 0.99 against 1.02).  Several keys: 16 warps, 128 registers.
__host__ __device__ constexpr int warp_cta_warps(int G) { return G == 1 ? 20 : 16; }

// Leaves per lane of a step (one pair).
constexpr uint32_t kBlockLeaves = 2;

// Loads per lane and chunk of the block scan's rows.  8 (with 3 keys a 256-B
// row pair's 32 loads pass in 4 of its 5-6 node expansions); 512-B rows take 16.
__host__ __device__ constexpr int block_chunk(uint32_t V) { return V == 32 ? 16 : 8; }

struct WarpSeg {
  const uint4* table;   // rows * V uint4
  uint64_t first;       // logical index of table row 0
  uint64_t rows;
  uint64_t item_begin;  // first global item of the segment
  uint64_t fr_base;     // frontier index of the segment's key 0 (key j at fr_base + j * nF)
  uint64_t nF;          // frontier nodes per key (level d - M nodes meeting the rows)
  uint32_t tiles;       // warp tiles per key group = ceil(nF / 32)
  uint32_t groups;      // key groups (items are tile-major: the groups of a tile lie side by side)
  uint32_t d;           // domain bits
  uint32_t M;           // depth-first levels per lane (>= 1)
  uint32_t g;           // keys per group
  uint32_t key_base;    // KeyDev index of the segment's key 0
  uint32_t col_base;    // first share column of the segment
  uint32_t pad;
};

struct WarpScanParams {
  WarpSeg seg[kMaxSegs];
  const KeyDev* keys;
  const KeyAux* aux;    // one per key, same index as keys
  const uint4* fr_seed;
  const uint8_t* fr_t;
  uint4* partial;       // [gridDim.x * warps per CTA][cols]
  uint4* out;           // the launch's cols shares (wide rows: zeroed before the launch, CTAs XOR into them)
  uint64_t items;
  uint32_t nsegs;
  uint32_t cols;
  uint32_t V;           // uint4 per row of every segment of the launch
  uint32_t slots;       // stack levels per lane and key
  uint32_t queues;      // item queues per CTA: 1, or one per warp scheduler (up to 4, at most the CTA's warps)
};

// A key whose table has a pending delta: its key slot, its first share column
// and, when the pass holds a frontier for it, where that is.
struct DeltaJob {
  uint32_t key;
  uint32_t col;
  uint32_t below;      // levels from the frontier's nodes to the leaves; ~0: no frontier
  uint32_t pad;
  uint64_t fr_base;    // frontier index of the key's node 0
  uint64_t fr_first;   // level index of node 0
};

// Most levels one frontier-chain step expands: breadth first up to
// kFrontierWide (one node per thread of its CTA), the rest depth first.
constexpr uint32_t kFrontierWide = 8;
constexpr uint32_t kFrontierLevels = 11;

// One step of the frontier chain: every CTA expands one node of
// level L_in of key blockIdx.y by c <= kFrontierLevels levels and stores the
// nodes of level L_in + c that meet the table.  With `walk` set the CTA's root
// is not read from in_seed: the CTA derives it from the key's root by the
// L_in-level path walk of ChaCha::eval, so the first step of a chain needs no
// narrow one-CTA-per-key launch above it.
struct FrontierStep {
  const KeyDev* keys;     // the segment's keys
  const uint4* in_seed;   // level L_in (unused when L_in == 0): key j at j * n_in
  const uint8_t* in_t;
  uint4* out_seed;        // key j at out_base + j * out_stride
  uint8_t* out_t;
  uint64_t in_first;      // level index of input slot 0
  uint64_t out_first;     // level index of output slot 0
  uint64_t n_in;
  uint64_t n_out;
  uint64_t out_base;
  uint64_t out_stride;
  uint32_t L_in;
  uint32_t c;
  uint32_t walk;          // 1: each CTA walks from the key's root to its level-L_in node
  uint4* zero_out;        // CTA (0, 0) zeroes these zero_n shares first (or null)
  uint64_t zero_n;
};

}  // namespace mg
