// Stage 4: tile compositor on sm_100a (tile_compositor_v2_kernel,
// render/kernels/compositor.rs:727-883) for 16x16 tiles (the reference's)
// and 8x8 or 32x16 tiles (the autotuner's other shapes).
//
// One block per screen tile (or for several, where a viewport has very many),
// one pixel per thread (64, 256 or 512 threads), a warp per 8x4 pixels. A tile
// without entries gets the background at once. The tile's depth-sorted splat
// list is consumed in batches of 128: each batch's 48-byte splat records are
// gathered from the Stage 2 record array into shared memory by the whole block,
// three 16-byte cp.async copies per record (measured faster than one
// cp.async.bulk per record completing on an mbarrier: 6.5 vs 6.3 x 10^11
// pixel-entry pairs/s on the 1080p frame), double buffered so the next batch is
// in flight while the current one is blended. Blending follows the reference:
// skip opacity <= 1/255; q = -(a dx^2 + 2 b dx dy + c dy^2)/2 clamped to <= 0;
// skip q < -4; alpha = min(0.99, op e^q); skip alpha < 1/255; front-to-back
// accumulate; a pixel stops at T < 1e-3 (T := 0). The q cut and the alpha cut
// are evaluated exactly as the host restatement does (IEEE-rounded q, the
// deterministic exp near the cut), so the only differences are last-bit colour
// sums and the rare pixel whose transmittance lands within an ulp of 1e-3
// (bounded by that 1e-3).
//
// A tile's lists are walked warp by warp: when a batch has landed, each of its
// entries is tested once against the warps' pixel blocks with the splat's
// extents (a bound on where it can pass the cuts, with a margin for the
// rounding of q), the ballots give every warp the entries that can touch it,
// and the warp evaluates only those, four at a time without a branch: the four
// opacities are independent, an entry that fails a cut blends with opacity 0
// (which leaves the sums and T as they are, bit for bit, as does any entry
// once T is 0), and only the transmittance is serial. One entry at a time, a
// relevant entry took 300-400 cycles of dependent latency, and a frame waits
// for its heaviest tiles: 128 us of a 20,000-splat 640x360 frame. The block stops
// when no pixel is still accumulating (the reference's double-buffered
// tile_alive vote), a warp when none of its own is. Output is RGBA8 packed in
// u32 rows padded to 64 pixels, optionally also RGBA f32. A block never exits
// with a copy still in flight into its shared memory.
#include <cmath>

#include "kernels.h"

namespace cgs {
namespace {

constexpr int kBatch = 128;
constexpr float kCut = 0.003921569f;  // 1/255

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait for a phase; returns false (and the caller flags it) on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          uint32_t limit = kSpinLimit) {
  for (uint32_t i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Wait drill: an mbarrier expecting one arrival that never comes; the bounded
// wait gives up after `limit` tries and the timeout bit is set.
__global__ void k_drill_mbarrier(uint32_t* status_word, uint32_t limit) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0 && !mbar_wait(&bar, 0u, limit)) atomicOr(status_word, kStatusBarrierTimeout);
}

// The pixel blocks (8x4 pixels, BX by BY of them from pixel (x0, y0)) that a
// splat can touch, one bit each: those that overlap the box of its extents.
// Outside that box the quadratic exceeds the splat's cut; the margin of a
// pixel plus the rounding of its three terms relative to their sum (they
// cancel for long diagonal splats: kappa = a c / (a c - b^2)) covers the
// computed value. Extents clamped to 1,024 bound nothing, and a conic that is
// not finite and positive definite may pass anywhere: all blocks.
template <uint32_t BX, uint32_t BY>
__device__ __forceinline__ uint32_t block_mask(const float4 geo, const float4 cc, float x0, float y0) {
  if (!(cc.y > kCut)) return 0u;  // the opacity cut
  constexpr uint32_t kAll = BX * BY >= 32 ? 0xffffffffu : (1u << (BX * BY)) - 1u;
  const uint32_t p = __float_as_uint(cc.w);
  const float ex = (float)(p & 0xFFFFu), ey = (float)((p >> 16) & 0xFFFFu);
  const float ac = geo.z * cc.x, det = ac - geo.w * geo.w;
  const float rel = 2e-6f * (ac / fmaxf(det, 1e-7f * ac));
  const bool fin = fabsf(geo.x) < 1e9f && fabsf(geo.y) < 1e9f && geo.z > 0.0f && cc.x > 0.0f &&
                   det > 0.0f && ac < 1e30f;
  if (!fin) return kAll;
  const float hx = ex + 1.0f + ex * rel + 1e-6f * fabsf(geo.x);
  const float hy = ey + 1.0f + ey * rel + 1e-6f * fabsf(geo.y);
  // blocks i with x0 + 8 i + 7.5 >= mu - h and x0 + 8 i + 0.5 <= mu + h
  const float rx = geo.x - x0, ry = geo.y - y0;
  int i0 = max(0, __float2int_ru((rx - hx - 7.5f) * 0.125f));
  int i1 = min((int)BX - 1, __float2int_rd((rx + hx - 0.5f) * 0.125f));
  int j0 = max(0, __float2int_ru((ry - hy - 3.5f) * 0.25f));
  int j1 = min((int)BY - 1, __float2int_rd((ry + hy - 0.5f) * 0.25f));
  if (ex >= 1024.0f) i0 = 0, i1 = (int)BX - 1;
  if (ey >= 1024.0f) j0 = 0, j1 = (int)BY - 1;
  if (i0 > i1 || j0 > j1) return 0u;
  const uint32_t row = ((2u << i1) - 1u) & ~((1u << i0) - 1u);
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < (int)BY; ++j)
    if (j >= j0 && j <= j1) m |= row << (j * BX);
  return m;
}

// Splats of entries [r0, r1) of tile (tx, ty), past those that the lists hold:
// from the hit words of the tile's screen block (stage3_lists.cu), a group of
// 32 pairs per thread and step. *cur is the chunk to start from (0 at first: a
// search over the chunks' exclusive counts); the steps go on from the chunk
// where the last entries were found. Called by the whole block.
__device__ __forceinline__ void ids_beyond(const CompositeArgs& a, uint32_t tx, uint32_t ty, uint32_t r0,
                                        uint32_t r1, uint32_t* cur, uint32_t* s_ids, uint32_t* s_red) {
  const uint32_t blk = (ty >> kListBlockH) * a.blocks_x + (tx >> kListBlockW);
  const uint32_t t = ((ty & ((1u << kListBlockH) - 1u)) << kListBlockW) | (tx & ((1u << kListBlockW) - 1u));
  const uint32_t groups = a.block_start[a.num_blocks] <= kListSmallPairs ? 1u : kListGroups;
  const uint32_t c0 = a.chunk_first[blk], c1 = a.chunk_first[blk + 1];
  const uint32_t p0 = a.block_start[blk], p1 = a.block_start[blk + 1];
  uint32_t c = *cur;
  if (c < c0) {
    uint32_t lo = c0, hi = c1;  // base[lo] <= r0
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (a.chunk_base[(size_t)mid * 32 + t] <= r0)
        lo = mid;
      else
        hi = mid;
    }
    c = lo;
  }
  for (uint32_t k = threadIdx.x; k < r1 - r0; k += blockDim.x) s_ids[k] = kInvalid;
  while (c < c1) {
    const uint32_t g = threadIdx.x % groups, ci = c + threadIdx.x / groups;
    const uint32_t i0 = p0 + (ci - c0) * 32u * groups + 32u * g;
    uint32_t m = 0;
    if (ci < c1 && i0 < p1) m = a.masks[((size_t)ci * groups + g) * 32 + t];
    uint32_t total;
    uint32_t rank = a.chunk_base[(size_t)c * 32 + t];
    const uint32_t first = rank;
    rank += block_exclusive_sum(__popc(m), s_red, &total);
    for (; m; m &= m - 1u, ++rank)
      if (rank >= r0 && rank < r1) s_ids[rank - r0] = a.sorted_pairs[i0 + (uint32_t)__ffs(m) - 1u];
    if (first + total >= r1) break;
    c += blockDim.x / groups;
  }
  *cur = c;
  __syncthreads();
}

template <int LW, int LH, bool STRIDED>
__global__ void __launch_bounds__(1 << (LW + LH)) k_composite(const CompositeArgs a) {
  constexpr uint32_t TW = 1u << LW, TH = 1u << LH, kCompThreads = TW * TH;
  constexpr uint32_t BX = TW / 8, BY = TH / 4, NW = kCompThreads / 32;
  static_assert(BX * BY == NW, "a warp per 8x4 pixels");
  // [kBatch]: a record of opacity 0 that fills up a group of four
  __shared__ __align__(128) SplatRec s_rec[2][kBatch + 1];
  __shared__ uint32_t s_bits[kBatch / 32][NW];  // entries of a batch per warp
  __shared__ uint32_t s_ids[kBatch], s_red[32];  // entries beyond the lists
  static_assert(kListLimit % kBatch == 0, "a batch is in the lists or beyond them");

  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid < 2) {
    const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    s_rec[tid][kBatch].geo = s_rec[tid][kBatch].cc = s_rec[tid][kBatch].rgb = z;
  }
  const uint2* ranges = reinterpret_cast<const uint2*>(a.ranges);
  const uint32_t tiles = a.tiles_x * a.tiles_y;
  uint32_t tile_id = blockIdx.x, tx = tile_id % a.tiles_x, ty = tile_id / a.tiles_x;
  const uint32_t step_x = gridDim.x % a.tiles_x, step_y = gridDim.x / a.tiles_x;
  uint2 range = ranges[tile_id];
  // STRIDED: a block takes every gridDim.x-th tile, its range loaded while the
  // one before is blended
  do {
    uint2 next{};
    if (STRIDED && tile_id + gridDim.x < tiles) next = ranges[tile_id + gridDim.x];
    const uint32_t px = tx * TW + (warp % BX) * 8u + (lane & 7u);
    const uint32_t py = ty * TH + (warp / BX) * 4u + (lane >> 3);
    const bool inside = px < a.width && py < a.height;
    const bool lists = a.masks != nullptr;
    const uint32_t rs = min(range.x, a.num_entries);
    const uint32_t re = min(range.y, a.num_entries);
    // what overflowed the entry buffer (flagged, rendered again) is left out
    const uint32_t n = !lists ? re - min(rs, re)
                       : a.num_entries - rs < min(range.y, kListLimit) ? a.num_entries - rs : range.y;
    const uint32_t beyond = lists ? kListLimit / kBatch : 0xFFFFFFFFu;  // first batch past the lists
    uint32_t cur = 0;  // chunk of the entries beyond the lists
    const uint32_t nb = (n + kBatch - 1) / kBatch;
    if (n == 0u) {  // empty: the background, two rows of the tile per warp
      const uint32_t ex = tx * TW + (tid & (TW - 1u)), ey = ty * TH + (tid >> LW);
      if (ex < a.width && ey < a.height) {
        a.out_rgba8[(size_t)ey * a.pitch_px + ex] = a.bg_rgba8;
        if (a.out_f32) a.out_f32[(size_t)ey * a.width + ex] = a.bg_f32;
      }
    } else {
      auto issue = [&](uint32_t b) {
        const uint32_t stage = b & 1u;
        const uint32_t cnt = min((uint32_t)kBatch, n - b * kBatch);
        for (uint32_t c = tid; c < cnt * 3u; c += kCompThreads) {
          const uint32_t k = c / 3u, part = c - 3u * k;
          uint32_t id = b >= beyond ? s_ids[k] : a.sorted_ids[rs + b * kBatch + k];
          if (id >= a.num_recs) {  // never let a bad id become an out-of-bounds copy
            if (a.fc) atomicOr(&a.fc->status, kStatusCapacity);
            id = 0;
          }
          const float4* src = reinterpret_cast<const float4*>(a.recs + id) + part;
          float4* dst = reinterpret_cast<float4*>(&s_rec[stage][k]) + part;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
                       : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };

      // T = 0: saturated, or no pixel of the frame
      float cr = 0.0f, cg = 0.0f, cb = 0.0f, t = inside ? 1.0f : 0.0f;
      const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
      const float bx0 = (float)(tx * TW), by0 = (float)(ty * TH);

      uint32_t issued = 0;
      if (nb > 0) {
        issue(0);
        issued = 1;
      }
      for (uint32_t b = 0; b < nb; ++b) {
        const uint32_t stage = b & 1u;
        if (b + 1 < nb) {
          if (b + 1 >= beyond)
            ids_beyond(a, tx, ty, (b + 1) * kBatch, min((b + 2) * kBatch, n), &cur, s_ids, s_red);
          issue(b + 1);
          issued = b + 2;
        }
        // this thread's copies of batch b have landed; the barrier makes every
        // thread's visible
        if (b + 1 < nb)
          asm volatile("cp.async.wait_group 1;" ::: "memory");
        else
          asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const uint32_t cnt = min((uint32_t)kBatch, n - b * kBatch);
        const uint32_t chunks = (cnt + 31u) / 32u;
        const SplatRec* recs = s_rec[stage];
        for (uint32_t c = warp; c < chunks; c += NW) {
          const uint32_t k = 32u * c + lane;
          const uint32_t m = k < cnt ? block_mask<BX, BY>(recs[k].geo, recs[k].cc, bx0, by0) : 0u;
          uint32_t mine = 0;
    #pragma unroll
          for (uint32_t w = 0; w < NW; ++w) {
            const uint32_t v = __ballot_sync(0xffffffffu, (m >> w) & 1u);
            if (lane == w) mine = v;
          }
          if (lane < NW) s_bits[c][lane] = mine;
        }
        __syncthreads();
        // a lane leaves once its pixel has saturated, a warp with its last
        for (uint32_t c = 0; c < chunks && t > 0.0f; ++c) {
          uint32_t bits = s_bits[c][warp];
          while (bits && t > 0.0f) {
            uint32_t k[4];
            float s[4], q[4], raw[4];
            bool near = false;
    #pragma unroll
            for (int i = 0; i < 4; ++i) {
              k[i] = bits ? 32u * c + (uint32_t)__ffs(bits) - 1u : (uint32_t)kBatch;
              bits &= bits - 1u;
            }
    #pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 cc4 = recs[k[i]].cc, geo = recs[k[i]].geo;
              // The quadratic rounded term by term in the reference's order, so
              // that the q >= -4 cut (q = -quad / 2, clamped to <= 0: a quad above
              // 8 fails) agrees exactly with the host restatement.
              const float dx = pcx - geo.x, dy = pcy - geo.y;
              const float qa = __fmul_rn(__fmul_rn(geo.z, dx), dx);
              const float qb = __fmul_rn(__fmul_rn(__fmul_rn(2.0f, geo.w), dx), dy);
              const float qc = __fmul_rn(__fmul_rn(cc4.x, dy), dy);
              s[i] = __fadd_rn(__fadd_rn(qa, qb), qc);
              q[i] = fminf(__fmul_rn(-0.5f, s[i]), 0.0f);
              raw[i] = cc4.y * __expf(q[i]);
              near = near || fabsf(raw[i] - kCut) < 4e-7f;
            }
            // Near the 1/255 visibility cut, re-evaluate with the deterministic
            // exp so the keep/skip decision matches the host restatement.
            if (near) {
    #pragma unroll
              for (int i = 0; i < 4; ++i)
                if (fabsf(raw[i] - kCut) < 4e-7f) raw[i] = __fmul_rn(recs[k[i]].cc.y, cgs_expf(q[i]));
            }
    #pragma unroll
            for (int i = 0; i < 4; ++i) {
              float alpha = fminf(0.99f, raw[i]);
              alpha = alpha >= kCut && !(s[i] > 8.0f) ? alpha : 0.0f;
              const float4 rgb = recs[k[i]].rgb;
              const float w = alpha * t;
              cr += w * rgb.x;
              cg += w * rgb.y;
              cb += w * rgb.z;
              t *= 1.0f - alpha;
              if (t < 0.001f) t = 0.0f;
            }
          }
        }
        // Batch boundary: stop when no pixel is left (also orders this batch's
        // reads before the copies that refill its buffer).
        if (!__syncthreads_or(t > 0.0f)) break;
      }
      // Never leave with a copy still writing into this block's shared memory.
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (tid == 0 && a.fc && issued > 0) atomicAdd(&a.fc->fetched, min(n, issued * (uint32_t)kBatch));
      if (inside) {
        const float fr = clampf(cr + t * a.bg[0], 0.0f, 1.0f);
        const float fg = clampf(cg + t * a.bg[1], 0.0f, 1.0f);
        const float fb = clampf(cb + t * a.bg[2], 0.0f, 1.0f);
        const float fa = clampf(1.0f - t, 0.0f, 1.0f);
        const uint32_t r8 = (uint32_t)clampf(rintf(fr * 255.0f), 0.0f, 255.0f);
        const uint32_t g8 = (uint32_t)clampf(rintf(fg * 255.0f), 0.0f, 255.0f);
        const uint32_t b8 = (uint32_t)clampf(rintf(fb * 255.0f), 0.0f, 255.0f);
        const uint32_t a8 = (uint32_t)clampf(rintf(fa * 255.0f), 0.0f, 255.0f);
        a.out_rgba8[(size_t)py * a.pitch_px + px] = r8 | (g8 << 8) | (b8 << 16) | (a8 << 24);
        if (a.out_f32) a.out_f32[(size_t)py * a.width + px] = make_float4(fr, fg, fb, fa);
      }
    }
    range = next;
    tile_id += gridDim.x;
    tx += step_x;
    ty += step_y;
    if (tx >= a.tiles_x) tx -= a.tiles_x, ++ty;
  } while (STRIDED && tile_id < tiles);
}

}  // namespace

cudaError_t launch_drill_mbarrier(uint32_t* status_word, uint32_t limit, cudaStream_t s) {
  k_drill_mbarrier<<<1, 32, 0, s>>>(status_word, limit);
  return cudaGetLastError();
}

// Tiles per resident block from which a block takes several tiles, and the
// grid it then has. Short lists and empty tiles are bound by what a tile costs
// whatever its length, and by the four blocks of 64 registers a thread that an
// SM holds; a block that goes on to its next tile saves the launch and the
// range's latency (16x16 tiles, 8K, 219 tiles a resident block: 1,000 splats
// 229 -> 188 us, 1.5M splats 510 -> 486). Below, blocks of several tiles
// balance worse than the launches cost (4K, 55 tiles: 300,000 splats 128 us
// with one tile a block, 136 with several; 1080p, 14 tiles: 45 and 57).
constexpr uint32_t kStridedWaves = 64, kStridedGrid = 16;

template <int LW, int LH>
cudaError_t composite_tiles(const CompositeArgs& a, cudaStream_t s) {
  constexpr int threads = 1 << (LW + LH);
  static const uint32_t resident = [] {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_composite<LW, LH, true>, threads, 0) !=
            cudaSuccess)
      return 592u;
    return (uint32_t)(sms > 0 && per_sm > 0 ? sms * per_sm : 592);
  }();
  const uint32_t tiles = a.tiles_x * a.tiles_y;
  if (tiles > kStridedWaves * resident)
    k_composite<LW, LH, true><<<kStridedGrid * resident, threads, 0, s>>>(a);
  else
    k_composite<LW, LH, false><<<tiles, threads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_composite(const CompositeArgs& args, cudaStream_t s) {
  CompositeArgs a = args;
  if (a.tiles_x == 0 || a.tiles_y == 0) return cudaSuccess;
  // what a pixel without entries gets (T = 1, the background's own alpha)
  auto clamp = [](float x, float lo, float hi) { return std::fmin(std::fmax(x, lo), hi); };
  const float bg[4] = {clamp(0.0f + a.bg[0], 0.0f, 1.0f), clamp(0.0f + a.bg[1], 0.0f, 1.0f),
                       clamp(0.0f + a.bg[2], 0.0f, 1.0f), a.bg[3]};
  a.bg_f32 = make_float4(bg[0], bg[1], bg[2], bg[3]);
  a.bg_rgba8 = 0;
  for (int k = 0; k < 4; ++k)
    a.bg_rgba8 |= (uint32_t)clamp(std::rint(bg[k] * 255.0f), 0.0f, 255.0f) << (8 * k);
  if (a.tile_w_log2 == 3 && a.tile_h_log2 == 3) return composite_tiles<3, 3>(a, s);
  if (a.tile_w_log2 == 5 && a.tile_h_log2 == 4) return composite_tiles<5, 4>(a, s);
  if (a.tile_w_log2 == 4 && a.tile_h_log2 == 4) return composite_tiles<4, 4>(a, s);
  return cudaErrorInvalidValue;
}

}  // namespace cgs
