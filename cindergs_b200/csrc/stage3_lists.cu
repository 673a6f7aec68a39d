// Stage 3 on sm_100a: the screen tiles' depth-sorted splat lists through
// screen blocks of 8x4 tiles, without forming or sorting one key per entry.
//
// Reference semantics: count_tiles_kernel, gpu_exclusive_scan, emit_tile_keys,
// the radix sort by (tile, depth) and identify_tile_ranges
// (render/kernels/binning.rs:37-417, scan.rs:198-333, radix_sort.rs:292-477).
// The lists equal theirs entry for entry: the splats arrive in (depth key,
// splat index) order, and every step below keeps that order.
//
//   k_list_pairs: a slot's tile box touches a few 8x4-tile blocks (3 on
//                 average at 1080p, where it touches 24 tiles); one
//                 (block, splat) pair per touched block is written in slot order;
//   (pair sort):  stable radix sort of the pairs by block;
//   k_list_count: a warp takes 32 pairs of one block, one per lane, and runs
//                 the exact ellipse-vs-tile test against the block's 32 tiles
//                 in turn: the ballot of tile t's tests is tile t's list of
//                 these 32 splats, already in depth order;
//   k_list_place: each chunk's first entry per tile inside its block, the
//                 tiles' first entries and their [start, end) ranges;
//   k_list_write: every ballot's splats are stored at their places.
//
// An entry costs one ballot bit and one 4-byte store instead of a 4-byte key
// and a 4-byte index written by the binning and moved by two or three radix
// passes; the tests need no owner search, no tables and no look-back. The
// block shape balances the tests wasted on tiles outside a splat's box (32
// per pair) against the pairs: 8x8-tile blocks tested 1.7 times as many.
#include <algorithm>

#include "kernels.h"
#include "tile_test.cuh"

namespace cgs {
namespace {

constexpr int kPairThreads = 256;
constexpr int kPairItems = kListSlots / kPairThreads;
constexpr int kListThreads = 256;
constexpr int kListWarps = kListThreads / 32;

// Exclusive scans of the block counts (pairs, chunks, placing segments) and
// the digit counts of the pair sort, by the last pairing block to finish.
__device__ void list_plan(const ListArgs& a, uint32_t* s_hist, uint32_t* s_red) {
  const uint32_t nb = a.num_blocks;
  const uint32_t pairs = __ldcg(&a.fc->pairs);
  const bool over = pairs > a.pair_cap;
  const uint32_t groups = pairs <= kListSmallPairs ? 1u : kListGroups;
  const uint32_t per = (nb + kPairThreads - 1) / kPairThreads;
  const uint32_t b0 = min(nb, threadIdx.x * per), b1 = min(nb, b0 + per);
  const uint32_t radix = 1u << a.radix_bits;
  for (uint32_t k = threadIdx.x; k < a.passes * radix; k += kPairThreads) s_hist[k] = 0u;
  __syncthreads();
  auto chunks_of = [&](uint32_t c) { return over ? 0u : (c + 32u * groups - 1u) / (32u * groups); };
  // every block has a segment: it writes the block's ranges
  auto segs_of = [](uint32_t ch) { return max(1u, (ch + kListSegChunks - 1u) / kListSegChunks); };
  uint32_t sum = 0, csum = 0, ssum = 0;
  for (uint32_t b = b0; b < b1; ++b) {
    const uint32_t c = __ldcg(a.block_count + b);
    sum += c;
    csum += chunks_of(c);
    ssum += segs_of(chunks_of(c));
    for (uint32_t p = 0; p < a.passes; ++p)
      if (c) atomicAdd(&s_hist[p * radix + ((b >> (p * a.radix_bits)) & (radix - 1u))], c);
  }
  uint32_t tot, ctot, stot;
  uint32_t run = block_exclusive_sum(sum, s_red, &tot);
  uint32_t crun = block_exclusive_sum(csum, s_red, &ctot);
  uint32_t srun = block_exclusive_sum(ssum, s_red, &stot);
  for (uint32_t b = b0; b < b1; ++b) {
    const uint32_t c = __ldcg(a.block_count + b);
    a.block_start[b] = run;
    a.chunk_first[b] = crun;
    a.seg_first[b] = srun;
    run += c;
    crun += chunks_of(c);
    srun += segs_of(chunks_of(c));
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < a.passes * radix; k += kPairThreads) a.hist[k] = s_hist[k];
  if (threadIdx.x == 0) {
    a.block_start[nb] = tot;
    a.chunk_first[nb] = ctot;
    a.seg_first[nb] = stot;
    a.plan->sort_n = over ? 0u : tot;
    a.plan->chunks = ctot;
    a.plan->segs = stot;
    a.plan->groups = groups;
    if (over) atomicOr(&a.fc->status, kStatusCapacity);
  }
}

// (block, splat) pairs in slot order. Persistent blocks take tiles of 1,024
// slots from a counter; a tile's pair count goes through a chained look-back
// and its pairs are written by the whole block, one per thread (the slot by a
// binary search over the tile's prefix), so a splat over hundreds of blocks
// costs no more per pair than a small one. The boxes come from Stage 2 (4
// bytes gathered per splat instead of its record). More pairs than the buffers
// hold are counted but not written: the plan is then empty and the capacity
// bit set. Bound by the latency of the gathers and the block's barriers.
__global__ void __launch_bounds__(kPairThreads) k_list_pairs(const ListArgs a, uint32_t look_words) {
  extern __shared__ __align__(16) uint32_t s_dyn[];  // block counters [num_blocks], then digits
  __shared__ uint32_t s_first[kListSlots + 1];
  __shared__ uint32_t s_box[kListSlots];
  __shared__ uint32_t s_sid[kListSlots];
  __shared__ uint32_t s_red[32];
  __shared__ uint32_t s_tile, s_base;
  __shared__ bool s_last;
  const uint32_t tid = threadIdx.x;
  const uint32_t active = min(a.n_rest + (a.split_count ? *a.split_count : 0u), a.max_n);
  const uint32_t num_tiles = (a.max_n + kListSlots - 1) / kListSlots;
  for (uint32_t k = tid; k < a.num_blocks; k += kPairThreads) s_dyn[k] = 0u;
  // the placing kernel's look-back words
  for (uint32_t k = blockIdx.x * kPairThreads + tid; k < look_words; k += gridDim.x * kPairThreads)
    a.seg_look[k] = 0ull;
  for (;;) {
    if (tid == 0) s_tile = atomicAdd(&a.plan->slot_ctr, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= num_tiles) break;
    // four consecutive slots per thread
    const uint32_t first = tile * kListSlots + tid * kPairItems;
    uint32_t sid[kPairItems], box[kPairItems];
#pragma unroll
    for (int k = 0; k < kPairItems; ++k) sid[k] = first + k < active ? a.order_ids[first + k] : kInvalid;
#pragma unroll
    for (int k = 0; k < kPairItems; ++k) box[k] = sid[k] < active ? a.boxes[sid[k]] : 0u;
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kPairItems; ++k) {
      sum += ((box[k] >> 14) & 511u) * (box[k] >> 23);
      s_sid[tid * kPairItems + k] = sid[k];
      s_box[tid * kPairItems + k] = box[k];
    }
    uint32_t total;
    uint32_t run = block_exclusive_sum(sum, s_red, &total);
#pragma unroll
    for (int k = 0; k < kPairItems; ++k) {
      s_first[tid * kPairItems + k] = run;
      run += ((box[k] >> 14) & 511u) * (box[k] >> 23);
    }
    if (tid < 32) {
      const uint32_t base = chained_scan_warp<true>(a.lookback, tile, total, &a.fc->status);
      if (tid == 0) {
        s_base = base;
        if (tile == num_tiles - 1) a.fc->pairs = sat_add_u32(base, total);
      }
    }
    __syncthreads();
    const uint32_t base = s_base;
    for (uint32_t i = tid; i < total; i += kPairThreads) {
      uint32_t o = 0;  // the last slot whose first pair is at most i
#pragma unroll
      for (uint32_t step = kListSlots / 2; step >= 1; step >>= 1)
        if (s_first[o + step] <= i) o += step;
      const uint32_t k = i - s_first[o], b = s_box[o], w = (b >> 14) & 511u;
      const uint32_t r = k / w, c = k - r * w;
      const uint32_t block = (b & 16383u) + r * a.blocks_x + c;
      atomicAdd(&s_dyn[block], 1u);
      const uint64_t pos = (uint64_t)base + i;
      if (pos < a.pair_cap) {
        a.pair_blocks[pos] = block;
        a.pair_ids[pos] = s_sid[o];
      }
    }
    __syncthreads();
  }
  for (uint32_t k = tid; k < a.num_blocks; k += kPairThreads)
    if (s_dyn[k]) atomicAdd(&a.block_count[k], s_dyn[k]);
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&a.plan->done, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  list_plan(a, s_dyn, s_red);
}

// The last of nb blocks whose first chunk (or segment) is at most c (blocks
// without any share the next one's first and are skipped by "last").
__device__ __forceinline__ uint32_t block_of(const uint32_t* first, uint32_t nb, uint32_t c) {
  uint32_t lo = 0, hi = nb;  // first[lo] <= c < first[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(first + mid) <= c)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// Two binary32 values in one register pair: sm_100's packed products and sums
// round each half as the scalar instructions do. A packed product that feeds
// a packed sum is contracted into one fused operation whatever its rounding
// qualifier and -fmad say, which changes the test's result now and then (one
// entry in 3 million of a 2400x1800 frame with 8x8 tiles). Such products are
// written as a b + z instead, z = -0 from a kernel argument the compiler
// cannot see through: exactly the rounded product, and nothing to contract.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// n / d in both halves, correctly rounded to binary32, from y = RN(1 / d):
// Markstein's division (IBM J. Res. Dev. 34(1), 1990). One step makes q
// faithful; from a faithful q and a correctly rounded reciprocal the second
// gives the correctly rounded quotient, as long as nothing under- or
// overflows (3 x 10^9 operand pairs equal n / d). The sign of a zero is lost.
__device__ __forceinline__ f2 div2(f2 n, f2 neg_d, f2 y) {
  const f2 q = mul2(n, y);
  const f2 q1 = fma2(fma2(neg_d, q, n), y, q);
  return fma2(fma2(neg_d, q1, n), y, q1);
}
__device__ __noinline__ f2 div2_ieee(f2 n, f2 neg_d) {
  float a, b, c, d;
  unpack2(n, a, b);
  unpack2(neg_d, c, d);
  return pack2(__fdiv_rn(a, -c), __fdiv_rn(b, -d));
}

// The tests of 32 pairs of a block against its 32 tiles, one pair per lane
// (ellipse_intersects_tile_gpu, binning.rs:37-96, term for term). Per lane the
// four rows' terms stay in registers and the eight columns are walked two at a
// time; a tile takes two clamps, a compare pair and half of 11 packed products
// and sums, then one ballot. A tile outside the lane's own tile box fails: its
// row's limit is NaN, its column's predicate false. Bound by instruction issue
// (clamps and compares run at half the products' rate).
__global__ void __launch_bounds__(kListThreads, 3) k_list_count(const ListArgs a, float neg_zero) {
  __shared__ __align__(16) uint32_t s_mask[kListWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunks = a.plan->chunks, groups = a.plan->groups;
  const uint32_t active = min(a.n_rest + (a.split_count ? *a.split_count : 0u), a.max_n);
  const float x_last = pixel_center(a.width - 1u), y_last = pixel_center(a.height - 1u);
  const uint32_t lw = a.tile_w_log2, lh = a.tile_h_log2;
  const float tw = (float)(1u << lw), th = (float)(1u << lh);
  uint32_t* sm = s_mask[warp];
  const f2 nz = pack2(neg_zero, neg_zero);
  for (uint32_t c = blockIdx.x * kListWarps + warp; c < chunks; c += gridDim.x * kListWarps) {
    const uint32_t b = block_of(a.chunk_first, a.num_blocks, c);
    const uint32_t tx0 = (b % a.blocks_x) << kListBlockW, ty0 = (b / a.blocks_x) << kListBlockH;
    const uint32_t i0 = a.block_start[b] + (c - a.chunk_first[b]) * 32u * groups;
    const uint32_t end = min(a.block_start[b + 1], a.pair_cap);
    // pixel centres are half-integers below 2^22: these sums are exact
    const float px0 = pixel_center(tx0 << lw), py0 = pixel_center(ty0 << lh);
    uint32_t cnt = 0;
    uint32_t sid = i0 + lane < end ? a.sorted_pairs[i0 + lane] : kInvalid;
    for (uint32_t j = 0; j < groups && i0 + 32u * j < end; ++j) {
      const SplatBox bx = load_box(a, sid, active);
      const float lim = bx.valid ? a.recs[sid].rgb.w : 0.0f;
      const uint32_t nxt = i0 + 32u * (j + 1) + lane;
      sid = j + 1 < groups && nxt < end ? a.sorted_pairs[nxt] : kInvalid;
      const float nan = __int_as_float(0x7FC00000);
      const float ca_ = fmaxf(bx.ca, 1e-12f), cc_ = fmaxf(bx.cc, 1e-12f);
      const float cb2 = __fmul_rn(2.0f, bx.cb);
      const float ya = __frcp_rn(ca_), yc = __frcp_rn(cc_);
      // a nonzero distance to a pixel centre is at least 2^-25 and below 2^24,
      // so with these bounds no quotient or residue leaves the normal range
      const bool ok = (bx.cb == 0.0f || fabsf(bx.cb) >= 0x1p-30f) && fabsf(bx.cb) < 0x1p40f &&
                      ca_ <= 0x1p20f && cc_ <= 0x1p20f;
      const bool fast = __all_sync(0xffffffffu, ok || !bx.valid);
      const f2 ca2 = pack2(bx.ca, bx.ca), cc2 = pack2(bx.cc, bx.cc), cb22 = pack2(cb2, cb2);
      const f2 nb2 = pack2(-bx.cb, -bx.cb);
      float y0[4], y1[4], rz[4], rl[4];
      f2 yn[4], rw[4];
      {
        const f2 nmu = pack2(-bx.mu_y, -bx.mu_y), nd = pack2(-ca_, -ca_), y2 = pack2(ya, ya);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float f0 = py0 + (float)(2 * h) * th, f1 = f0 + th;
          unpack2(add2(pack2(f0, f1), nmu), y0[2 * h], y0[2 * h + 1]);
          unpack2(add2(pack2(fminf(f0 + (th - 1.0f), y_last), fminf(f1 + (th - 1.0f), y_last)), nmu),
                  y1[2 * h], y1[2 * h + 1]);
          const float na = clampf(0.0f, y0[2 * h], y1[2 * h]);
          const float nb = clampf(0.0f, y0[2 * h + 1], y1[2 * h + 1]);
          const f2 n = pack2(na, nb), num = mul2(nb2, n);
          unpack2(fast ? div2(num, nd, y2) : div2_ieee(num, nd), rz[2 * h], rz[2 * h + 1]);
          float wa, wb;
          unpack2(mul2(mul2(cc2, n), n), wa, wb);
          yn[2 * h] = pack2(na, na);
          yn[2 * h + 1] = pack2(nb, nb);
          rw[2 * h] = pack2(wa, wa);
          rw[2 * h + 1] = pack2(wb, wb);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
          rl[k] = bx.valid && ty0 + k >= bx.y0 && ty0 + k <= bx.y1 ? lim : nan;
      }
      const f2 nmu = pack2(-bx.mu_x, -bx.mu_x), nd = pack2(-cc_, -cc_), y2 = pack2(yc, yc);
#pragma unroll 1
      for (uint32_t k = 0; k < 8; k += 2) {
        const uint32_t tx = tx0 + k;
        const bool in0 = tx >= bx.x0 && tx <= bx.x1, in1 = tx + 1 >= bx.x0 && tx + 1 <= bx.x1;
        const float f0 = px0 + (float)k * tw, f1 = f0 + tw;
        float x0a, x0b, x1a, x1b;
        unpack2(add2(pack2(f0, f1), nmu), x0a, x0b);
        unpack2(add2(pack2(fminf(f0 + (tw - 1.0f), x_last), fminf(f1 + (tw - 1.0f), x_last)), nmu), x1a,
                x1b);
        const f2 xn = pack2(clampf(0.0f, x0a, x1a), clampf(0.0f, x0b, x1b));
        const f2 num = mul2(nb2, xn);
        float cza, czb;
        unpack2(fast ? div2(num, nd, y2) : div2_ieee(num, nd), cza, czb);
        const f2 cw = fma2(mul2(ca2, xn), xn, nz);
        const f2 cp = mul2(cb22, xn);
        uint32_t m0[4], m1[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const f2 y = pack2(clampf(cza, y0[r], y1[r]), clampf(czb, y0[r], y1[r]));
          const f2 q1 = add2(add2(cw, fma2(cp, y, nz)), fma2(mul2(cc2, y), y, nz));
          const f2 x = pack2(clampf(rz[r], x0a, x1a), clampf(rz[r], x0b, x1b));
          const f2 q2 = add2(add2(fma2(mul2(ca2, x), x, nz), fma2(mul2(cb22, x), yn[r], nz)), rw[r]);
          float q1a, q1b, q2a, q2b;
          unpack2(q1, q1a, q1b);
          unpack2(q2, q2a, q2b);
          // fminf(q1, q2) <= limit: either is (a NaN never is)
          m0[r] = __ballot_sync(0xffffffffu, in0 && (q1a <= rl[r] || q2a <= rl[r]));
          m1[r] = __ballot_sync(0xffffffffu, in1 && (q1b <= rl[r] || q2b <= rl[r]));
        }
        if (lane == 0) {
          *reinterpret_cast<uint4*>(sm + 4 * k) = make_uint4(m0[0], m0[1], m0[2], m0[3]);
          *reinterpret_cast<uint4*>(sm + 4 * k + 4) = make_uint4(m1[0], m1[1], m1[2], m1[3]);
        }
      }
      __syncwarp();
      // lane t holds tile t (row-major in the block)
      const uint32_t mt = sm[(lane & 7) * 4 + (lane >> 3)];
      a.masks[((size_t)c * groups + j) * 32 + lane] = mt;
      cnt += __popc(mt);
      __syncwarp();
    }
    a.chunk_base[(size_t)c * 32 + lane] = cnt;
  }
}

// A placing segment is up to 64 consecutive chunks of one block: its per-tile
// sums go through a look-back over the block's earlier segments (vectors of 32
// words), and its chunks' counts become exclusive sums over the block's
// chunks. The block's last segment knows the tiles' totals: it takes the
// block's entries from a counter and writes the tiles' first entries and
// ranges. 32 tiles x 8 parts of 8 chunks.
__global__ void __launch_bounds__(256) k_list_place(const ListArgs a) {
  __shared__ uint32_t s_part[8][32];
  __shared__ uint32_t s_excl[32];
  __shared__ uint32_t s_seg;
  const uint32_t t = threadIdx.x & 31u, g = threadIdx.x >> 5;
  const uint32_t segs = a.plan->segs;
  for (;;) {
    if (threadIdx.x == 0) s_seg = atomicAdd(&a.plan->seg_ctr, 1u);
    __syncthreads();
    const uint32_t seg = s_seg;
    if (seg >= segs) break;
    const uint32_t b = block_of(a.seg_first, a.num_blocks, seg);
    const uint32_t s0 = a.seg_first[b], s1 = a.seg_first[b + 1];
    const uint32_t end = a.chunk_first[b + 1];
    const uint32_t c0 = min(end, a.chunk_first[b] + (seg - s0) * kListSegChunks + g * 8u);
    const uint32_t c1 = min(end, c0 + 8u);
    uint32_t v[8], sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k] = c0 + k < c1 ? a.chunk_base[(size_t)(c0 + k) * 32 + t] : 0u;
      sum += v[k];
    }
    s_part[g][t] = sum;
    __syncthreads();
    if (g == 0) {
      uint32_t agg = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) agg += s_part[k][t];
      // look-back, a lane per tile
      uint32_t excl = 0;
      unsigned long long* look = a.seg_look + (size_t)seg * 32 + t;
      if (seg == s0) {
        st_relaxed_u64(look, (2ull << 32) | agg);
      } else {
        st_relaxed_u64(look, (1ull << 32) | agg);
        const unsigned long long* p = look - 32;
        bool done = false;
        for (uint32_t spins = 0; !done;) {
          const unsigned long long w = ld_relaxed_u64(p);
          if ((w >> 32) == 0ull) {
            if (++spins > kSpinLimit) {
              atomicOr(&a.fc->status, kStatusLookbackTimeout);
              break;
            }
            __nanosleep(32);
            continue;
          }
          excl += (uint32_t)w;
          done = (w >> 32) == 2ull;
          p -= 32;
        }
        st_relaxed_u64(look, (2ull << 32) | (excl + agg));
      }
      s_excl[t] = excl;
      __syncwarp();
      if (seg + 1 == s1) {
        const uint32_t n = excl + agg;  // the tile's entries
        unsigned long long incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
          if (t >= (uint32_t)o) incl += y;
        }
        unsigned long long at = 0;
        const unsigned long long cap = a.entry_cap;
        if (t == 31) {
          at = incl ? atomicAdd(&a.fc->stage_ctr, incl) : 0ull;
          if (at + incl > cap) atomicOr(&a.fc->status, kStatusCapacity);
        }
        at = __shfl_sync(0xffffffffu, at, 31) + incl - n;
        a.tile_base[(size_t)b * 32 + t] = (uint32_t)min(at, cap);  // at the capacity: not written
        const uint32_t tx = ((b % a.blocks_x) << kListBlockW) + (t & 7u);
        const uint32_t ty = ((b / a.blocks_x) << kListBlockH) + (t >> 3);
        if (tx < a.tiles_x && ty < a.tiles_y)
          reinterpret_cast<uint2*>(a.ranges)[(size_t)ty * a.tiles_x + tx] =
              n ? make_uint2((uint32_t)min(at, cap), (uint32_t)min(at + n, cap)) : make_uint2(0u, 0u);
      }
    }
    __syncthreads();
    uint32_t run = s_excl[t];
    for (uint32_t k = 0; k < g; ++k) run += s_part[k][t];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (c0 + k < c1) a.chunk_base[(size_t)(c0 + k) * 32 + t] = run;
      run += v[k];
    }
    __syncthreads();
  }
}

// Entries. A warp takes two groups of 32 pairs at a time: lane t walks the set
// bits of tile t's two ballots and lists them in shared memory, tile after
// tile; then the warp copies that list out, one entry per lane, so that a
// tile's entries of the 64 pairs (about 14 at 1080p) are stored together.
__global__ void __launch_bounds__(kListThreads) k_list_write(const ListArgs a) {
  __shared__ uint16_t s_stage[kListWarps][64 * 32];  // tile << 6 | pair
  __shared__ uint32_t s_sid[kListWarps][64];
  __shared__ uint32_t s_delta[kListWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunks = a.plan->chunks, groups = a.plan->groups;
  const uint32_t cap = a.entry_cap;
  if (blockIdx.x == 0 && threadIdx.x == 0)
    a.fc->entries = (uint32_t)min(a.fc->stage_ctr, 0xFFFFFFFFull);
  uint16_t* stage = s_stage[warp];
  for (uint32_t c = blockIdx.x * kListWarps + warp; c < chunks; c += gridDim.x * kListWarps) {
    const uint32_t b = block_of(a.chunk_first, a.num_blocks, c);
    const uint32_t i0 = a.block_start[b] + (c - a.chunk_first[b]) * 32u * groups;
    const uint32_t end = min(a.block_start[b + 1], a.pair_cap);
    uint64_t at = (uint64_t)a.tile_base[(size_t)b * 32 + lane] + a.chunk_base[(size_t)c * 32 + lane];
    uint32_t p = (uint32_t)min(at, (uint64_t)cap);  // at the capacity: not written
    for (uint32_t j = 0; j < groups && i0 + 32u * j < end; j += 2) {
      const uint32_t i = i0 + 32u * j + lane;
      const bool two = j + 1 < groups && i0 + 32u * (j + 1) < end;
      const uint32_t* in = a.masks + ((size_t)c * groups + j) * 32 + lane;
      const uint32_t m0 = in[0], m1 = two ? in[32] : 0u;
      s_sid[warp][lane] = i < end ? a.sorted_pairs[i] : 0u;
      if (two) s_sid[warp][lane + 32] = i + 32 < end ? a.sorted_pairs[i + 32] : 0u;
      const uint32_t n = __popc(m0) + __popc(m1);
      uint32_t incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
      s_delta[warp][lane] = p - (incl - n);
      // from the highest bit down, backwards from the tile's end
      uint16_t* at_s = stage + incl;
      const uint32_t tile = (uint32_t)lane << 6;
      for (uint32_t m = m1; m;) {
        const uint32_t bit = 31u - __clz(m);
        m ^= 1u << bit;
        *--at_s = (uint16_t)(tile + 32u + bit);
      }
      for (uint32_t m = m0; m;) {
        const uint32_t bit = 31u - __clz(m);
        m ^= 1u << bit;
        *--at_s = (uint16_t)(tile + bit);
      }
      __syncwarp();
      for (uint32_t k = lane; k < total; k += 32) {
        const uint32_t e = stage[k];
        const uint32_t pos = s_delta[warp][e >> 6] + k;
        if (pos < cap) a.ids[pos] = s_sid[warp][e & 63u];
      }
      p = min(p + n, cap);
      __syncwarp();
    }
  }
}

// Resident blocks of kernel K on the current device.
template <typename K>
uint32_t resident_blocks(K kernel, int threads) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) != cudaSuccess)
    return 148u;
  return (uint32_t)std::max(1, sms * std::max(per_sm, 1));
}

}  // namespace

cudaError_t launch_list_pairs(const ListArgs& a, cudaStream_t s) {
  if (a.num_blocks == 0 || a.num_blocks > kListMaxBlocks) return cudaErrorInvalidValue;
  const size_t fixed = 4 * (3 * (size_t)kListSlots + 64);
  const size_t smem = sizeof(uint32_t) * std::max<uint32_t>(a.num_blocks, a.passes << a.radix_bits);
  if (fixed + smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_list_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  // eight blocks of 256 threads per SM, fewer where the block counters are large
  const uint32_t per_sm = (uint32_t)std::min<size_t>(8, 227 * 1024 / (fixed + smem + 1024));
  const uint32_t tiles = (a.max_n + kListSlots - 1) / kListSlots;
  k_list_pairs<<<std::max(1u, std::min(148u * per_sm, tiles)), kPairThreads, smem, s>>>(
      a, list_seg_cap(a.pair_cap, a.num_blocks) * 32u);
  return cudaGetLastError();
}

cudaError_t launch_list_count(const ListArgs& a, cudaStream_t s) {
  static const uint32_t grid = resident_blocks(k_list_count, kListThreads);
  const uint32_t most = (list_chunk_cap(a.pair_cap, a.num_blocks) + kListWarps - 1) / kListWarps;
  k_list_count<<<std::min(most, grid), kListThreads, 0, s>>>(a, -0.0f);
  return cudaGetLastError();
}

cudaError_t launch_list_place(const ListArgs& a, cudaStream_t s) {
  static const uint32_t grid = resident_blocks(k_list_place, 256);
  k_list_place<<<std::min(list_seg_cap(a.pair_cap, a.num_blocks), grid), 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_list_write(const ListArgs& a, cudaStream_t s) {
  static const uint32_t grid = resident_blocks(k_list_write, kListThreads);
  const uint32_t most = (list_chunk_cap(a.pair_cap, a.num_blocks) + kListWarps - 1) / kListWarps;
  k_list_write<<<std::min(most, grid), kListThreads, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace cgs
