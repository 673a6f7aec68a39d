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
//   k_list_count: a warp takes 32 pairs of one block, one per lane, finds the
//                 tiles of the block each hits (an interval of columns per
//                 row) and transposes the 32 words: tile t's word is its list
//                 of these 32 splats, already in depth order;
//   k_list_place: each chunk's first entry per tile inside its block, the
//                 tiles' first entries and counts;
//   k_list_write: the words' splats are stored at their places, the front-most
//                 1,024 of every tile (the compositor takes the rest from the
//                 words, if it ever gets there).
//
// An entry costs one bit and one 4-byte store instead of a 4-byte key
// and a 4-byte index written by the binning and moved by two or three radix
// passes, and nothing is evaluated per tile.
#include <algorithm>

#include "kernels.h"
#include "tile_span.h"
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

// ellipse_intersects_tile_gpu (binning.rs:37-96) for tile (tx, ty), every
// operation rounded separately in the reference's operand order (a call: only
// the tiles that tile_span.h leaves undecided come here).
__device__ __noinline__ bool tile_exact(uint32_t tx, uint32_t ty, uint32_t lw, uint32_t lh, uint32_t wm1,
                                        uint32_t hm1, float mu_x, float mu_y, float a, float b, float c,
                                        float lim) {
  const uint32_t xs = tx << lw, ys = ty << lh;
  const float dx0 = __fsub_rn(pixel_center(xs), mu_x);
  const float dx1 = __fsub_rn(pixel_center(min(xs + ((1u << lw) - 1u), wm1)), mu_x);
  const float dy0 = __fsub_rn(pixel_center(ys), mu_y);
  const float dy1 = __fsub_rn(pixel_center(min(ys + ((1u << lh) - 1u), hm1)), mu_y);
  const float b2 = __fmul_rn(2.0f, b);
  const float xn = clampf(0.0f, dx0, dx1), yn = clampf(0.0f, dy0, dy1);
  const float y1 = clampf(__fdiv_rn(__fmul_rn(-b, xn), fmaxf(c, 1e-12f)), dy0, dy1);
  const float q1 = __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(a, xn), xn), __fmul_rn(__fmul_rn(b2, xn), y1)),
                             __fmul_rn(__fmul_rn(c, y1), y1));
  const float x2 = clampf(__fdiv_rn(__fmul_rn(-b, yn), fmaxf(a, 1e-12f)), dx0, dx1);
  const float q2 = __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(a, x2), x2), __fmul_rn(__fmul_rn(b2, x2), yn)),
                             __fmul_rn(__fmul_rn(c, yn), yn));
  return fminf(q1, q2) <= lim;
}

// Transpose of a 32x32 bit matrix, a row per lane: lane t gets bit t of every
// lane's word, lane l's at bit l.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
  uint32_t m = 0x0000FFFFu;
#pragma unroll
  for (int j = 16; j >= 1; j >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
    m ^= m << (j >> 1);
  }
  return x;
}

// The tiles that 32 pairs of a block hit, one pair per lane: for each of the
// block's four rows the columns the splat's ellipse reaches (tile_span.h), and
// the test itself for the few tiles that lie within the rounding margin of
// an end; the 32 lanes' words are then transposed into the 32 tiles' lists.
// One interval per row instead of eight tests: 880 -> 590 instructions per 32
// pairs, 168 -> 113 us at 4.4M pairs (1.1M splats, 1080p). Bound by
// instruction issue.
__global__ void __launch_bounds__(kListThreads) k_list_count(const ListArgs a) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunks = a.plan->chunks, groups = a.plan->groups;
  const uint32_t active = min(a.n_rest + (a.split_count ? *a.split_count : 0u), a.max_n);
  const uint32_t wm1 = a.width - 1u, hm1 = a.height - 1u;
  const float x_last = pixel_center(wm1), y_last = pixel_center(hm1);
  const uint32_t lw = a.tile_w_log2, lh = a.tile_h_log2;
  const float tw = (float)(1u << lw), th = (float)(1u << lh);
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
      const float dx00 = px0 - bx.mu_x;
      const SplatSpan sp = splat_span(bx.ca, bx.cb, bx.cc, lim, dx00, (px0 + (tw - 1.0f)) - bx.mu_x,
                                      x_last - bx.mu_x, tw);
      // the splat's tile box in this block
      const int c0 = max((int)bx.x0 - (int)tx0, 0), c1 = min((int)bx.x1 - (int)tx0, 7);
      const uint32_t cols = bx.valid && c1 >= c0 ? ((2u << c1) - 1u) & ~((1u << c0) - 1u) : 0u;
      uint32_t hits = 0, open = 0;
#pragma unroll
      for (uint32_t r = 0; r < 4; ++r) {
        const float f = py0 + (float)r * th;
        uint32_t in, out;
        row_span(sp, f - bx.mu_y, fminf(f + (th - 1.0f), y_last) - bx.mu_y, in, out);
        const uint32_t row = ty0 + r >= bx.y0 && ty0 + r <= bx.y1 ? cols : 0u;
        hits |= (sp.ok ? in & row : 0u) << (8u * r);
        open |= (sp.ok ? out & ~in & row : row) << (8u * r);
      }
      while (open) {
        const uint32_t t = (uint32_t)__ffs(open) - 1u;
        open &= open - 1u;
        if (tile_exact(tx0 + (t & 7u), ty0 + (t >> 3), lw, lh, wm1, hm1, bx.mu_x, bx.mu_y, bx.ca, bx.cb,
                       bx.cc, lim))
          hits |= 1u << t;
      }
      __syncwarp();
      const uint32_t mt = transpose_bits(hits, lane);
      a.masks[((size_t)c * groups + j) * 32 + lane] = mt;
      cnt += __popc(mt);
    }
    a.chunk_base[(size_t)c * 32 + lane] = cnt;
  }
}

// A placing segment is up to 64 consecutive chunks of one block: its per-tile
// sums go through a look-back over the block's earlier segments (vectors of 32
// words), and its chunks' counts become exclusive sums over the block's
// chunks. The block's last segment knows the tiles' totals: it takes the
// block's places from a counter and writes the tiles' first entries and
// counts. 32 tiles x 8 parts of 8 chunks.
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
        const uint32_t n = excl + agg;  // the tile's entries, the first `held` of them written
        const uint32_t held = min(n, kListLimit);
        unsigned long long all = n;
        uint32_t incl = held;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long y = __shfl_up_sync(0xffffffffu, all, o);
          const uint32_t z = __shfl_up_sync(0xffffffffu, incl, o);
          if (t >= (uint32_t)o) {
            all += y;
            incl += z;
          }
        }
        // at most 32 x kListLimit entries in each of kListMaxBlocks blocks
        static_assert((unsigned long long)kListLimit * 32 * kListMaxBlocks < (1ull << 32), "32-bit places");
        uint32_t at = 0;
        const uint32_t cap = a.entry_cap;
        if (t == 31) {
          if (all) atomicAdd(&a.fc->stage_ctr, all);
          at = incl ? atomicAdd(&a.fc->written, incl) : 0u;
          if (at + incl > cap) atomicOr(&a.fc->status, kStatusCapacity);
        }
        at = __shfl_sync(0xffffffffu, at, 31) + incl - held;
        a.tile_base[(size_t)b * 32 + t] = min(at, cap);  // at the capacity: not written
        const uint32_t tx = ((b % a.blocks_x) << kListBlockW) + (t & 7u);
        const uint32_t ty = ((b / a.blocks_x) << kListBlockH) + (t >> 3);
        if (tx < a.tiles_x && ty < a.tiles_y)
          reinterpret_cast<uint2*>(a.ranges)[(size_t)ty * a.tiles_x + tx] = make_uint2(min(at, cap), n);
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

// Entries, the first kListLimit of every tile. A warp takes two groups of 32
// pairs at a time: lane t walks the set bits of tile t's two words and lists
// them in shared memory, tile after tile; then the warp copies that list out,
// one entry per lane, so that a tile's entries of the 64 pairs (about 14 at
// 1080p) are stored together. Chunks whose tiles all have their kListLimit
// entries are passed over: at 26M entries 72 -> 22 us.
__global__ void __launch_bounds__(kListThreads) k_list_write(const ListArgs a) {
  __shared__ uint16_t s_stage[kListWarps][64 * 32];  // tile << 6 | pair
  __shared__ uint32_t s_sid[kListWarps][64];
  __shared__ uint32_t s_delta[kListWarps][32], s_end[kListWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunks = a.plan->chunks, groups = a.plan->groups;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const unsigned long long all = a.fc->stage_ctr;
    a.fc->entries = (uint32_t)min(all, 0xFFFFFFFFull);
    if (all > kMaxEntryCap) atomicOr(&a.fc->status, kStatusCapacity);  // as the entry sorts
  }
  uint16_t* stage = s_stage[warp];
  for (uint32_t c = blockIdx.x * kListWarps + warp; c < chunks; c += gridDim.x * kListWarps) {
    uint32_t rank = a.chunk_base[(size_t)c * 32 + lane];
    if (!__any_sync(0xffffffffu, rank < kListLimit)) continue;
    const uint32_t b = block_of(a.chunk_first, a.num_blocks, c);
    const uint32_t i0 = a.block_start[b] + (c - a.chunk_first[b]) * 32u * groups;
    const uint32_t end = min(a.block_start[b + 1], a.pair_cap);
    const uint32_t first = a.tile_base[(size_t)b * 32 + lane];
    s_end[warp][lane] = min(first + kListLimit, a.entry_cap);
    for (uint32_t j = 0; j < groups && i0 + 32u * j < end; j += 2) {
      const uint32_t i = i0 + 32u * j + lane;
      const bool two = j + 1 < groups && i0 + 32u * (j + 1) < end;
      const bool on = rank < kListLimit;
      if (!__any_sync(0xffffffffu, on)) break;
      const uint32_t* in = a.masks + ((size_t)c * groups + j) * 32 + lane;
      const uint32_t m0 = on ? in[0] : 0u, m1 = on && two ? in[32] : 0u;
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
      s_delta[warp][lane] = first + rank - (incl - n);
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
        const uint32_t e = stage[k], t = e >> 6;
        const uint32_t pos = s_delta[warp][t] + k;
        if (pos < s_end[warp][t]) a.ids[pos] = s_sid[warp][e & 63u];
      }
      rank += n;
      __syncwarp();
    }
    __syncwarp();
  }
}

// Every entry of every tile at its place in the reference's order, and how
// many entries each splat has, from the blocks' hit words: a warp per chunk, a
// lane per tile. For readbacks only (26M entries put together on the host took
// 160 ms).
__global__ void __launch_bounds__(kListThreads) k_list_export(const ListArgs a, const ListExport e) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunks = a.chunk_first[a.num_blocks];
  const uint32_t groups = a.block_start[a.num_blocks] <= kListSmallPairs ? 1u : kListGroups;
  for (uint32_t c = blockIdx.x * kListWarps + warp; c < chunks; c += gridDim.x * kListWarps) {
    const uint32_t b = block_of(a.chunk_first, a.num_blocks, c);
    const uint32_t tx = ((b % a.blocks_x) << kListBlockW) + (lane & 7u);
    const uint32_t ty = ((b / a.blocks_x) << kListBlockH) + (lane >> 3);
    const bool on = tx < a.tiles_x && ty < a.tiles_y;
    const uint32_t tile = ty * a.tiles_x + tx;
    const uint32_t i0 = a.block_start[b] + (c - a.chunk_first[b]) * 32u * groups;
    const uint32_t end = min(a.block_start[b + 1], a.pair_cap);
    uint32_t at = on ? e.tile_at[tile] + a.chunk_base[(size_t)c * 32 + lane] : 0u;
    for (uint32_t j = 0; j < groups && i0 + 32u * j < end; ++j) {
      const uint32_t i = i0 + 32u * j;
      uint32_t m = on ? a.masks[((size_t)c * groups + j) * 32 + lane] : 0u;
      if (e.counts) {
        const uint32_t tiles = __popc(transpose_bits(m, lane));  // of pair i + lane
        const uint32_t sid = i + lane < end ? a.sorted_pairs[i + lane] : kInvalid;
        if (tiles && sid < a.max_n) atomicAdd(&e.counts[sid], tiles);
      }
      if (!e.ids && !e.keys) continue;
      for (; m; m &= m - 1u, ++at) {
        if (at >= e.entries) break;
        const uint32_t sid = a.sorted_pairs[i + (uint32_t)__ffs(m) - 1u];
        if (e.ids) e.ids[at] = sid;
        if (e.keys) {
          const uint32_t d = sid < a.max_n ? e.depths[sid] : 0u;
          if (e.key64)
            static_cast<unsigned long long*>(e.keys)[at] = ((unsigned long long)tile << 32) | d;
          else
            static_cast<uint32_t*>(e.keys)[at] = (e.depth_bits >= 32u ? 0u : tile << e.depth_bits) | d;
        }
      }
      __syncwarp();
    }
  }
}

__global__ void k_list_depths(const uint32_t* __restrict__ ids, const uint32_t* __restrict__ keys,
                              uint32_t n, uint32_t* __restrict__ depths) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n && ids[j] < n) depths[ids[j]] = keys[j];
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

cudaError_t launch_list_export(const ListArgs& a, const ListExport& e, cudaStream_t s) {
  static const uint32_t grid = resident_blocks(k_list_export, kListThreads);
  const uint32_t most = (list_chunk_cap(a.pair_cap, a.num_blocks) + kListWarps - 1) / kListWarps;
  k_list_export<<<std::min(most, grid), kListThreads, 0, s>>>(a, e);
  return cudaGetLastError();
}

cudaError_t launch_list_depths(const uint32_t* ids, const uint32_t* keys, uint32_t n, uint32_t* depths,
                               cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_list_depths<<<(n + 255) / 256, 256, 0, s>>>(ids, keys, n, depths);
  return cudaGetLastError();
}

cudaError_t launch_list_pairs(const ListArgs& a, cudaStream_t s) {
  if (a.num_blocks == 0 || a.num_blocks > kListMaxBlocks) return cudaErrorInvalidValue;
  const size_t fixed = 4 * (3 * (size_t)kListSlots + 64);
  const size_t smem = sizeof(uint32_t) * std::max<uint32_t>(a.num_blocks, a.passes << a.radix_bits);
  // the same value for every viewport: another thread's launch may come between
  const cudaError_t e = cudaFuncSetAttribute(k_list_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(sizeof(uint32_t) * kListMaxBlocks));
  if (e != cudaSuccess) return e;
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
  k_list_count<<<std::min(most, grid), kListThreads, 0, s>>>(a);
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
