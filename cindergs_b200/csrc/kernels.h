// Host-side launchers for the sm_100a kernels (one per .cu translation unit).
// All launchers enqueue on `stream` and return the launch error code.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace cgs {

// Launch that may overlap the end of the stream's previous kernel: every
// thread of k calls wait_for_previous_kernel before its first access to global
// memory, and no thread leaves before that. Used between short kernels of
// one shared-memory size, where it hides about 1.2 us of each launch: the
// training step (13 launches, 184 -> 167 us) and the sort's passes. Between
// the frame's other kernels it costs more than it gives in large frames (12
// views of 2M splats 6.8 -> 8.6 ms, 1.1M splats 556 -> 605 us), probably
// because blocks that wait take shared memory from the L1 cache of the kernel
// still running.
template <typename... P, typename... A>
cudaError_t launch_dependent(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, P(args)...);
}

// ---- Stage 1 (stage1_deform.cu) --------------------------------------------
struct DeformArgs {
  uint32_t n;                 // rest Gaussians
  uint32_t num_tets;
  const float* verts;         // [V*3] current cage vertices
  const uint4* elems;         // [T]
  const float* inv_dm;        // [T*9]
  float* tet_J;               // [T*9] out (column-major)
  float* tet_R;               // [T*9] out (column-major)
  float* tet_stretch;         // [T] out
  const uint32_t* bind_tet;   // [n]
  const float4* bind_w;       // [n]
  const float4* rest_pos;     // [n] xyz + opacity
  const float4* rest_cova;    // [n] xx, xy, xz, yy
  const float2* rest_covb;    // [n] yz, zz
  float4* def_pos;            // [2n]
  float4* def_cova;           // [2n]
  float2* def_covb;           // [2n]
  uint2* split_meta;          // [n] (parent, tet)
  uint32_t* split_count;      // persistent device word
  unsigned long long* status; // [ceil(n/256)] chained-scan status, zeroed
  FrameCounters* fc;
  float split_threshold;
  float mip;
  // MVC-bound Gaussians (bind_tet == kMvcBound): per slot the deformed
  // position and gradient (3 float4, k_mvc_jacobian) in, the polar rotation
  // (9 floats, column-major) out for Stage 2's SH directions
  const float4* mvc_xf;
  float* mvc_R;
  // 1: the deform launch also computes the tet transforms (its first blocks
  // take the tets; the Gaussian blocks wait for them), instead of a separate
  // launch_tet_transforms
  uint32_t fuse_tets;
};
// FrameCounters::tile_ctr slot counting the finished tet blocks of a fused
// deform launch.
constexpr int kTetsDoneCtr = 8;
cudaError_t launch_tet_transforms(const DeformArgs& a, cudaStream_t s);

// ---- MVC (stage1_mvc.cu) -----------------------------------------------------
// bind_tet value of a Gaussian bound to the polygon (MVC) cage; its bind_w.x
// holds the bits of its MVC slot.
constexpr uint32_t kMvcBound = 0xFFFFFFFEu;
struct MvcCage {
  uint32_t V, F;
  const float4* verts;      // [V] rest (binding) or current vertices
  const uint4* tris;        // [F] outward triangles
  const uint32_t* vf_off;   // [V + 1] incident faces per vertex (CSR)
  const uint32_t* vf_list;  // face << 2 | corner, ascending faces per vertex
};
bool mvc_cage_fits(uint32_t V, uint32_t F);
cudaError_t launch_mvc_weights(const MvcCage& c, uint32_t n, const float* pts, float* w,
                               cudaStream_t s);
cudaError_t launch_mvc_inside(const MvcCage& c, uint32_t n, const float4* rest_pos,
                              const uint32_t* bind_tet, uint32_t* flag, cudaStream_t s);
cudaError_t launch_mvc_compact(uint32_t n, const uint32_t* flag, const uint32_t* slot_of,
                               uint32_t* bind_tet, float4* bind_w, uint32_t* list, cudaStream_t s);
cudaError_t launch_mvc_bind_weights(const MvcCage& c, uint32_t nb, const uint32_t* list,
                                    const float4* rest_pos, float h, float4* wg, cudaStream_t s);
cudaError_t launch_mvc_jacobian(uint32_t V, const float4* verts, uint32_t nb, const float4* wg,
                                float4* xf, cudaStream_t s);
// Linear-precision residual |x' - x| / s at each listed rest position, where
// x' (xf, 3 float4 per slot) is the learned field's position on the rest
// cage; flag = residual > threshold.
cudaError_t launch_mvc_residual(uint32_t nb, const uint32_t* list, const float4* rest_pos,
                                const float4* xf, float inv_scale, float threshold, float* resid,
                                uint32_t* flag, cudaStream_t s);

// ---- learned MVC field (mvc_field.cu) ------------------------------------------
constexpr uint32_t kMvcMaxVerts = 1024;  // vertices of a polygon cage (mvc_cage_fits)
constexpr int kFieldBands = 8;
constexpr int kFieldIn = 64;    // 3 + 6 * bands, zero-padded
constexpr int kFieldHid = 128;
// epilogues of the training GEMMs: bias (C), bias and SiLU (C, D and its
// transpose), SiLU slope of the layer below (C, D and its transpose), split
// partial sums
constexpr int kEpiBias = 1, kEpiBiasSilu = 2, kEpiBack = 3, kEpiSplit = 4;
// per-frame projection: Pc (128 x 3), pc (3), A3 (3 x 3)
constexpr int kFieldProj = 3 * kFieldHid + 3 + 9;
struct FieldMat {  // M = (Vb Vb^T)^-1, row-major 4 x 4
  float m[16];
};

struct FieldNet {  // device pointers into one parameter block
  const __nv_bfloat16 *W1b, *W2b, *W3b, *W4b, *W5b;
  const float *b1, *b2, *b3, *b4, *b5;
};
struct GemmArgs {  // C = A B^T; tcgen05 (mvc_field_tc.cu)
  const __nv_bfloat16* A;
  const __nv_bfloat16* B;
  uint32_t M, N, K, lda, ldb;
  float* C;              // fp32 result (+ bias, times silu'(pre)), or the splits' [z][M][N]
  uint32_t ldc;
  const float* bias;     // [N]
  __nv_bfloat16* D;      // bf16(silu(C)), or bf16(C silu'(pre)); or null
  uint32_t ldd;
  __nv_bfloat16* DT;     // D transposed [N][ldt], or null
  uint32_t ldt;
  const float* pre;      // [M][ldc] (kEpiBack)
  uint32_t* status;      // kStatusBarrierTimeout / kStatusPoisoned on a failed wait, or null
};
// The weight gradients of all layers in one launch: problem p's tiles are
// [first[p], first[p + 1]) of 128 x 64, K split into `splits` ranges; and the
// bias gradients, the column sums over the batch's rows of sum[p] [K][ld].
constexpr int kGradProblems = 5;
struct GemmBatch {
  GemmArgs g[kGradProblems];
  uint32_t first[kGradProblems + 1];
  uint32_t splits;
  const float* sum[kGradProblems];
  float* sum_out[kGradProblems];
  uint32_t sum_n[kGradProblems], sum_ld[kGradProblems];
};
uint32_t grad_splits(uint32_t B);  // ranges of K = B
struct FieldBatch {
  const float* points;   // [n*3]
  uint32_t n, B;
  uint32_t seed;         // 0: rows r % n in order
  const float* enc;      // [4] centre xyz, 1/s
  float* x;              // [B*3]
  uint32_t* idx;         // [B] the point of each row
  __nv_bfloat16* a0;     // [B*64]
  __nv_bfloat16* a0T;    // [64*B] or null
};
struct FieldLoss {
  const float* z;        // [B*ldz]
  const float* target;   // [n*V] exact weights
  const uint32_t* idx;   // [B] row -> point
  const float* x;        // [B*3]
  const float4* verts;   // [V] rest vertices
  uint32_t B, V, ldz;
  float lambda, s2;
  float M[16];           // (Vb Vb^T)^-1 of the rest cage
  __nv_bfloat16* dzb;    // [B*ldz]
  __nv_bfloat16* dzT;    // [V*B]
  float* dz;             // [B*ldz]
  float* loss;           // [2] accumulated (weight term, residual term)
};
constexpr uint32_t kLossRows = 16;  // rows of one loss block
// Weight gradients from the split partial sums, and Adam on all gradients
// (adam = 0: gradients only); refreshes the bf16 weights and the transposed
// copies that the backward products read.
struct FieldUpdate {
  uint32_t off[11];      // parameter offsets (FieldParam), total
  uint32_t V, ldV, splits;
  const float* ws[5];    // W1..W5 partial sums [splits][rows][cols]
  float *p, *g, *m, *v;  // g: the bias gradients in, all gradients out
  __nv_bfloat16* pb;
  __nv_bfloat16* wT[4];  // W2..W4 transposed [128][128], W5 transposed [128][ldV]
  int adam;
  float lr, b1, b2, eps, c1, c2;
};
struct FieldInfer {
  FieldNet net;
  const float* enc;      // [4]
  const float* proj;     // [kFieldProj]
  const uint32_t* gauss; // item -> point index, or null (identity)
  const float4* points4; // rest positions (xyz), or null
  const float* points3;  // packed xyz when points4 is null
  uint32_t first, count, out_first;
  float4* xf;            // [(out_first + count) * 3]
  // cached codes [count][4][128] bf16 and the items' rest positions
  // [count]: written by launch_field_infer when codes is set (instead of
  // xf), read by launch_field_apply
  __nv_bfloat16* codes;
  float4* code_pos;
  uint32_t* status;      // kStatusBarrierTimeout when a bounded wait gave up, or null
};
cudaError_t launch_field_gather(const FieldBatch& b, cudaStream_t s);
cudaError_t launch_gemm_nt(const GemmArgs& g, int epi, cudaStream_t s);
cudaError_t launch_gemm_grads(const GemmBatch& g, cudaStream_t s);
// out = bf16(in), and W2..W5 transposed into wT (null: not wanted)
cudaError_t launch_field_refresh(const uint32_t* off, uint32_t V, uint32_t ldV, const float* p,
                                 __nv_bfloat16* pb, __nv_bfloat16* const* wT, cudaStream_t s);
cudaError_t launch_field_loss(const FieldLoss& l, cudaStream_t s);
cudaError_t launch_field_update(const FieldUpdate& u, cudaStream_t s);
// verts null: the network's own rest position (no linear-precision
// projection); otherwise the projected weights on current vertices verts.
cudaError_t launch_field_project(const FieldNet& net, uint32_t V, const float4* rest,
                                 const float4* verts, const float* M, float* proj,
                                 cudaStream_t s);
cudaError_t launch_field_infer(const FieldInfer& fi, cudaStream_t s);
// The same on the tcgen05 tensor cores (mvc_field_tc.cu).
cudaError_t launch_field_infer_tc(const FieldInfer& fi, cudaStream_t s);
// Output layer over cached codes (needs codes, points4): position + gradient.
cudaError_t launch_field_apply(const FieldInfer& fi, cudaStream_t s);

cudaError_t launch_deform(const DeformArgs& a, cudaStream_t s);

struct BindArgs {
  uint32_t n;
  uint32_t num_tets;
  const float4* points;   // [n] xyz (+ unused w)
  const float* tet_x0;    // [T*3] rest position of each tet's first vertex
  const float* inv_dm;    // [T*9]
  int use_bounds;
  float bmin[3], bmax[3];
  uint32_t* bind_tet;     // [n] out
  float4* bind_w;         // [n] out
};
cudaError_t launch_bind(const BindArgs& a, cudaStream_t s);

// ---- Stage 2 (stage2_project.cu) -------------------------------------------
struct ProjectArgs {
  uint32_t threads;           // block size: 128, 256 (0) or 512
  const float4* pos;          // [max_n] xyz + opacity
  const float4* cova;         // [max_n]
  const float2* covb;         // [max_n]
  const void* sh;             // SH planes: f32 -> float4 [12][sh_stride]; f16 -> uint4 [6][sh_stride]
  int sh_f16;
  uint32_t sh_stride;         // plane stride (rest Gaussian count)
  const uint32_t* bind_tet;   // [n_rest] or null
  const float4* bind_w;       // [n_rest] (MVC slot bits in .x for kMvcBound) or null
  const float* tet_R;         // [T*9] or null
  uint32_t num_tets;
  const float* mvc_R;         // [MVC slots * 9] or null
  const uint2* split_meta;    // [n_rest] or null
  const uint32_t* split_count;  // device word or null (no splitting)
  uint32_t n_rest;
  uint32_t max_n;             // grid covers max_n splats
  float cam[24];
  float cam_pos[3];
  float mip, min_opacity, min_radius;
  uint32_t sh_degree;
  SplatRec* out;              // [max_n]
  FrameCounters* fc;
  // Stage 3's per-splat depth keys and slot ids (null when the frame reuses
  // an earlier frame's Stage 3): 32-bit keys get the quantised depth of the
  // packed (tile, depth) key, 64-bit keys the raw depth bits; culled splats
  // get 0xFFFFFFFF, which sorts after every visible depth.
  uint32_t* depth_keys;       // [max_n]
  uint32_t* depth_ids;        // [max_n]
  int key64;
  uint32_t depth_base_bits;   // near-plane exponent bits (32-bit keys)
  uint32_t depth_bits;        // depth bits in a 32-bit key
  // screen-block lists: the blocks each splat's tile box touches (list_box),
  // or null
  uint32_t* boxes;            // [max_n]
  uint32_t tiles_x, tiles_y, tile_w_log2, tile_h_log2, blocks_x;
};
cudaError_t launch_project(const ProjectArgs& a, cudaStream_t s);

// QuantizedGaussianSceneSoa words (f16 covariance pairs, degree-trimmed f16
// SH) into the resident layout with f16 SH planes.
cudaError_t launch_scene_decode_quantized(uint32_t n, const float* pos, const uint32_t* cov_words,
                                          const float* opa, const uint32_t* sh_words,
                                          uint32_t sh_degree, float4* out_pos, float4* out_cova,
                                          float2* out_covb, void* out_sh, cudaStream_t s);
// Rest-scene layout conversion from the reference's interleaved SoA.
cudaError_t launch_scene_layout(uint32_t n, const float* pos, const float* cov, const float* opa,
                                const void* sh, int sh_f16, float4* out_pos, float4* out_cova,
                                float2* out_covb, void* out_sh, cudaStream_t s);

// ---- Stage 3 (stage3_bin.cu) -------------------------------------------------
struct BinArgs {
  const SplatRec* recs;
  // Splats in depth-key order (the stable radix sort of Stage 2's depth keys):
  // slot s of the binning grid is splat order_ids[s] with depth key
  // order_keys[s]; its entries are emitted in this order.
  const uint32_t* order_keys;
  const uint32_t* order_ids;
  const uint32_t* split_count;  // null when no splitting
  uint32_t n_rest;
  uint32_t max_n;
  uint32_t width, height, tiles_x, tiles_y;
  uint32_t tile_w_log2, tile_h_log2;  // screen tile shape (8x8, 16x16 or 32x16 pixels)
  // per slot (depth order): the first entry (direct mode), or the tile count
  // that a scan turns into the first entry in place (record mode)
  uint32_t* offsets;            // [max_n]
  // direct mode: look-back words of the 32-slot tiles' hit counts, zeroed
  unsigned long long* lookback; // [ceil(max_n/32)]
  // record mode: staging start and records of each 32-slot tile and group
  uint32_t* tile_stage;
  uint32_t* tile_count;
  uint32_t blocks_per_sm;       // resident blocks per SM of the count kernel (0: all that fit)
  FrameCounters* fc;
  int key64;
  uint32_t depth_bits;          // depth bits in a 32-bit key
  // record mode: the staged records; direct mode: the entries in depth order
  uint32_t* stage_keys;
  uint32_t* keys;               // 32-bit: packed keys; 64-bit: tile ids
  uint32_t* depths;             // 64-bit: raw depth bits
  uint32_t* ids;
  uint32_t* hist;               // [passes][1 << radix_bits] tile-digit histograms, zeroed
  uint32_t radix_bits;
  uint32_t tile_bits;           // tile id bits (the entry sort's key bits)
  uint32_t entry_cap;           // capacity of every entry buffer
  // Record mode (the tile transpose): stage one word per hit, tile << 5 |
  // slot lane, instead of keys and ids; no histograms. Each 32-slot tile
  // stages one run per group of 2^group_shift screen tiles, so tile_stage /
  // tile_count are [ceil(max_n/32)][groups].
  int records;
  uint32_t groups;              // <= 8
  uint32_t group_shift;
};
// Counts each slot's tiles and, in direct mode, writes the scanned offsets,
// the entry total (fc->entries) and every entry at its place in depth order
// and accumulates the tile-digit histograms (k_bin_count, one launch); in
// record mode it stages one record per hit and leaves the per-slot counts
// for a scan (launch_scan_u32).
cudaError_t launch_bin_count(const BinArgs& a, cudaStream_t s);
// Tile transpose (the entry sort when the tiles fit shared memory): a
// one-pass stable counting sort of the staged records by tile. Chunk k is the
// 32-slot tiles [k * chunk_wtiles, (k + 1) * chunk_wtiles); warp w of a chunk
// block owns the w-th eighth of them.
struct TransposeArgs {
  const uint32_t* records;      // staged tile << 5 | slot lane
  const uint32_t* tile_stage;   // [num_wtiles][groups] staging start of each run
  const uint32_t* tile_count;   // [num_wtiles][groups] records of each run
  const uint32_t* order_ids;    // slot -> splat index
  uint32_t num_wtiles;
  uint32_t chunk_wtiles;        // multiple of 8, at most 2040
  uint32_t num_chunks;
  uint32_t num_tiles;           // screen tiles
  uint32_t groups;              // tile groups (runs per 32-slot tile)
  uint32_t group_tiles;         // screen tiles per group (a power of two)
  uint32_t* cmat;               // [num_tiles][num_chunks] counts -> first entries (in place)
  uint32_t* totals;             // [num_tiles] entries per tile, zeroed
  const uint32_t* tile_base;    // [num_tiles] exclusive scan of totals
  uint32_t* ranges;             // [num_tiles] (start, end), (0, 0) when empty
  uint32_t* ids_out;            // [capacity] sorted splat indices
  uint32_t capacity;
  uint32_t* status_word;
};
constexpr uint32_t kTransposeGroupTiles = 2048;  // screen tiles per group (2^11)
cudaError_t launch_chunk_counts(const TransposeArgs& a, cudaStream_t s);
cudaError_t launch_column_scan(const TransposeArgs& a, cudaStream_t s);
cudaError_t launch_chunk_place(const TransposeArgs& a, cudaStream_t s);

// ---- Stage 3, screen-block lists (stage3_lists.cu) -----------------------------
// A screen block is 8x4 screen tiles. Splats in depth order are paired with
// the blocks their tile boxes touch, the pairs are sorted by block, and every
// block's pairs are turned into its 32 tiles' lists.
constexpr uint32_t kListBlockW = 3, kListBlockH = 2;  // log2 of a block's tiles
constexpr uint32_t kListMaxBlocks = 16384;  // block counters in shared memory, 14-bit block ids
constexpr uint32_t kListSlots = 1024;       // slots of one pairing tile
constexpr uint32_t kListSmallPairs = 1u << 18;  // up to here a chunk is one group of 32 pairs
constexpr uint32_t kListGroups = 4;         // groups of 32 pairs per chunk beyond
constexpr uint32_t kListSegChunks = 64;     // chunks of one placing segment
// Entries of a tile that are written out: its front-most ones. A tile's pixels
// saturate long before its list ends (after at most 420 of up to 32,000 entries
// in a 100,000-splat 720p frame), and the compositor takes what lies beyond
// from the blocks' hit words. A multiple of its batch.
constexpr uint32_t kListLimit = 1024;
// The screen blocks a splat's tile box touches: first block | width << 14 |
// height << 23, 0 when the splat has no entries (a box spans at most 1024 + 1
// + 1024 pixels: 34 x 66 blocks of 8x8-pixel tiles).
__host__ __device__ inline uint32_t list_box(uint32_t first, uint32_t w, uint32_t h) {
  return first | (w << 14) | (h << 23);
}
// Control words of a frame's lists (zeroed with the frame's scratch).
struct ListPlan {
  uint32_t sort_n;        // pairs to sort (0 when they exceed the buffers)
  uint32_t chunks;        // chunks of all blocks
  uint32_t groups;        // groups of 32 pairs per chunk
  uint32_t segs;          // placing segments of all blocks
  uint32_t done;          // pairing thread blocks that have finished
  uint32_t slot_ctr;      // pairing tiles taken
  uint32_t seg_ctr;       // placing segments taken
  uint32_t pad;
};
struct ListArgs {
  const SplatRec* recs;
  const uint32_t* order_ids;    // slot -> splat (depth order)
  const uint32_t* boxes;        // [max_n] list_box of each splat (Stage 2)
  const uint32_t* split_count;  // null when no splitting
  uint32_t n_rest, max_n;
  uint32_t width, height, tiles_x, tiles_y, tile_w_log2, tile_h_log2;
  uint32_t blocks_x, num_blocks;
  FrameCounters* fc;
  ListPlan* plan;
  unsigned long long* lookback; // [ceil(max_n / kListSlots)] zeroed
  uint32_t* block_count;        // [num_blocks] pairs per block, zeroed
  uint32_t* block_start;        // [num_blocks + 1] first pair of each block
  uint32_t* chunk_first;        // [num_blocks + 1] first chunk of each block
  uint32_t* seg_first;          // [num_blocks + 1] first placing segment of each block
  uint32_t* hist;               // pair sort's digit counts [passes][1 << radix_bits]
  uint32_t radix_bits, passes;
  uint32_t* pair_blocks;        // [pair_cap] block of each pair, slot order
  uint32_t* pair_ids;           // [pair_cap] splat of each pair, slot order
  uint32_t pair_cap;
  const uint32_t* sorted_pairs; // [pair_cap] splats sorted by (block, slot)
  uint32_t* masks;              // [chunks * groups][32] ballots of 32 pairs per tile
  uint32_t* chunk_base;         // [chunks][32] entries per tile -> exclusive over the block's chunks
  unsigned long long* seg_look; // [segs][32] placing look-back words
  uint32_t* tile_base;          // [num_blocks][32] first entry of each tile
  uint32_t* ranges;             // [tiles] (first written entry, entries of the tile)
  uint32_t* ids;                // [entry_cap] splat indices, up to kListLimit of every tile
  uint32_t entry_cap;
};
// Readback of whole lists in the reference's order: tile by tile over the screen.
struct ListExport {
  const uint32_t* tile_at;  // [tiles] first entry of each tile
  const uint32_t* depths;   // [max_n] depth key of each splat (keys)
  uint32_t entries;         // of all tiles
  uint32_t* ids;            // [entries] splat indices, or null
  void* keys;               // [entries] (tile, depth key), 32 or 64 bits each, or null
  uint32_t key64, depth_bits;
  uint32_t* counts;         // [max_n] zeroed: entries of each splat, or null
};
// Chunks, ballot groups and placing segments of a frame of at most pair_cap pairs.
inline uint32_t list_chunk_cap(uint32_t pair_cap, uint32_t blocks) {
  const uint32_t all = pair_cap / 32 + 1, most = kListSmallPairs / 32;
  const uint32_t large = pair_cap / (32 * kListGroups) + 1;
  const uint32_t small = most < all ? most : all;
  return (small > large ? small : large) + blocks;
}
inline uint32_t list_group_cap(uint32_t pair_cap, uint32_t blocks) {
  return pair_cap / 32 + 1 + kListGroups * blocks;
}
inline uint32_t list_seg_cap(uint32_t pair_cap, uint32_t blocks) {
  return list_chunk_cap(pair_cap, blocks) / kListSegChunks + 1 + blocks;
}
cudaError_t launch_list_pairs(const ListArgs& a, cudaStream_t s);
cudaError_t launch_list_count(const ListArgs& a, cudaStream_t s);
cudaError_t launch_list_place(const ListArgs& a, cudaStream_t s);
cudaError_t launch_list_write(const ListArgs& a, cudaStream_t s);
cudaError_t launch_list_export(const ListArgs& a, const ListExport& e, cudaStream_t s);
// depths[ids[j]] = keys[j] for j < n
cudaError_t launch_list_depths(const uint32_t* ids, const uint32_t* keys, uint32_t n, uint32_t* depths,
                               cudaStream_t s);

// Per-tile [start, end) from sorted words: tile = word >> shift, over
// min(*n_ptr, capacity) words. ranges zeroed.
// Turns the last sort pass's range words (complemented first entries, ends)
// into [first, end) per screen tile; empty tiles stay (0, 0).
cudaError_t launch_ranges_fixup(uint32_t* ranges, uint32_t num_tiles, cudaStream_t s);
cudaError_t launch_tile_ranges(const uint32_t* sorted, uint32_t shift, const uint32_t* n_ptr,
                               uint32_t capacity, uint32_t total_tiles, uint32_t* ranges,
                               uint32_t blocks, cudaStream_t s);
// Generic exclusive scan of n u32 (chained scan); total -> *d_total.
cudaError_t launch_scan_u32(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* d_total,
                            unsigned long long* status, uint32_t* tile_ctr, uint32_t* status_word,
                            cudaStream_t s);
uint32_t scan_tiles(uint32_t n);

// ---- radix sort (radix_sort.cu) ----------------------------------------------
struct SortArgs {
  uint32_t* keys[2];     // ping-pong key buffers
  uint32_t* vals[2];     // ping-pong payload word 0
  uint32_t* vals2[2];    // ping-pong payload word 1 (null for one-word payloads)
  const uint32_t* n_ptr; // device element count (may exceed capacity -> capacity flag), or
                         // null: capacity elements
  uint32_t capacity;     // elements the buffers hold; grid is sized for it
  uint32_t first_bit;    // lowest key bit to sort on
  uint32_t num_bits;     // bits to sort on (from first_bit)
  uint32_t radix_bits;   // digit width, 4..8
  uint32_t* hist;        // [passes][radix] counts of the digits, filled before the passes
                         // (each block of a pass scans its pass's counts)
  // optional: the last pass also finds the [first, end) entries of every
  // screen tile (key >> tile_shift) into ranges[2 t], ranges[2 t + 1]
  // (zeroed before the sort; finish with launch_ranges_fixup)
  uint32_t* ranges = nullptr;
  uint32_t tile_shift = 0;
  uint32_t num_tiles = 0;
  void* status;          // [passes][tiles][radix] zeroed look-back words (when status2 is null)
  void* status2[2];      // optional: two [tiles][radix] look-back buffers used
                         // alternately; each pass clears the one it does not
                         // use for the next pass, so no per-frame memset is needed
  int* parity;           // in/out: buffer index the next pass uses (with status2)
  // look-back words of 64 bits (any 32-bit count; required above 2^30
  // elements) instead of 32 bits (counts below 2^30)
  bool wide_lookback = false;
  // words per tile that each pass clears in the status2 buffer it does not
  // use (0: the radix). A pair shared by sorts of different digit widths sets
  // the widest radix (256), so that a narrow sort leaves no stale word for a
  // later wide one to read.
  uint32_t lb_stride = 0;
  // 4,096-key tiles whatever the capacity: for callers with a line of their own
  // or a look-back area of a fixed size
  bool large_tiles = false;
  uint32_t* tile_ctr;    // [passes] zeroed
  uint32_t* status_word;
  int src;               // index of the buffer holding the input
  // bit p: pass p finds the lanes sharing a digit with one ballot per digit
  // bit (a fixed cost) instead of __match_any_sync (cheap when a warp's keys
  // share few digits, expensive when they are all different)
  uint32_t ballot_mask = ~0u;
  // bit p: pass p uses shared-memory peer masks instead (one atomicOr and
  // one warp barrier per key: cheapest for many distinct 8-bit digits)
  uint32_t smem_mask = 0u;
};
// Wait drills (cgs_ctx_wait_drill): each runs one of the library's bounded
// device waits against a predecessor or barrier that nothing completes, with
// `limit` polls, so that it gives up and sets its status bit in *status_word.
// The look-back arrays must hold two zeroed tiles.
cudaError_t launch_drill_chained_scan(unsigned long long* status, uint32_t* status_word,
                                      uint32_t limit, cudaStream_t s);
cudaError_t launch_drill_digit_lookback(const uint32_t* status, uint32_t radix,
                                        uint32_t* status_word, uint32_t limit, cudaStream_t s);
cudaError_t launch_drill_mbarrier(uint32_t* status_word, uint32_t limit, cudaStream_t s);
// Runs the passes; returns in *out_src the index of the buffer with the result.
cudaError_t run_radix_sort(const SortArgs& a, int* out_src, cudaStream_t s);
cudaError_t launch_histogram(const uint32_t* keys, const uint32_t* n_ptr, uint32_t capacity,
                             uint32_t first_bit, uint32_t num_bits, uint32_t radix_bits,
                             uint32_t* hist, cudaStream_t s);
uint32_t sort_tiles(uint32_t capacity, bool large_tiles = false);  // tiles of a sort
uint32_t sort_passes(uint32_t num_bits, uint32_t radix_bits);

// ---- Cage springs (springs.cu) -----------------------------------------------
struct SpringCageDev {
  float kim;        // stiffness / max(mass, 0.001)
  float gamma;      // velocity factor exp(-c dt) of one step
  float dt;         // min(dt, 0.033); a step is skipped unless > 0
  float pad;
  float cx, cy, cz; // rest centroid (jiggle impulse)
  uint32_t planes;  // first plane | count << 16
};
struct SpringArgs {
  uint32_t V, num_cages, steps;
  const float4* rest;          // [V] xyz + cage index bits (>= num_cages: no cage)
  float4* vel;                 // [V]
  const uint8_t* pinned;       // [V]
  float* verts;                // [V*3] the resident cage vertices, stepped in place
  const SpringCageDev* cages;  // [num_cages]
  const float4* planes;        // [2 per plane] (nx, ny, nz, offset), (restitution, friction, -, -)
};
cudaError_t launch_springs_step(const SpringArgs& a, cudaStream_t s);
cudaError_t launch_springs_impulse(const SpringArgs& a, float magnitude, cudaStream_t s);

// ---- SH coefficient rotation and export (sh_rotate.cu) ------------------------
// Floats per rotation in the band-matrix table: M1 (9), M2 (25), M3 (49), pad.
constexpr uint32_t kShRotStride = 84;
struct ExportArgs {
  uint32_t n_rest;            // rest Gaussians (splats at or above are split children)
  uint32_t first, count;      // the chunk of splats to write
  const float4* pos;          // [first + count] xyz + opacity (deformed or rest)
  const float4* cova;         // xx, xy, xz, yy
  const float2* covb;         // yz, zz
  const void* sh;             // resident SH planes (f32 [12][sh_stride] or f16 [6][sh_stride])
  int sh_f16;
  uint32_t sh_stride;
  const uint32_t* bind_tet;   // [n_rest] or null (no rotation)
  const float4* bind_w;       // [n_rest] (MVC slot bits in .x)
  const uint2* split_meta;    // [children] (parent, tet)
  uint32_t num_tets;          // table rows [0, num_tets) are tet rotations
  int mvc;                    // table rows num_tets + slot are MVC rotations
  const float* table;         // [rotations * kShRotStride] or null
  uint32_t degree;
  float* out_pos;             // [count * 3] or null
  float* out_cov;             // [count * 6] or null
  float* out_opa;             // [count] or null
  float* out_sh;              // [count * 48] or null
};
size_t sh_basis_bytes();
cudaError_t launch_sh_basis(void* basis, cudaStream_t s);
cudaError_t launch_sh_rotators(uint32_t count, const float* rot, const void* basis, uint32_t degree,
                               float* table, cudaStream_t s);
cudaError_t launch_sh_apply(uint64_t n, float* sh, const float* table, uint32_t num_rot,
                            const uint32_t* index, uint32_t degree, uint32_t* bad, cudaStream_t s);
cudaError_t launch_export(const ExportArgs& a, cudaStream_t s);

// ---- Stage 4 (stage4_composite.cu) -------------------------------------------
struct CompositeArgs {
  const SplatRec* recs;
  const uint32_t* sorted_ids;
  const uint32_t* ranges;
  uint32_t width, height, tiles_x, tiles_y;
  uint32_t tile_w_log2, tile_h_log2;  // screen tile shape: 8x8, 16x16 or 32x16 pixels
  uint32_t pitch_px;        // RGBA8 row pitch in pixels
  float bg[4];
  uint32_t* out_rgba8;
  float4* out_f32;          // null when not requested
  FrameCounters* fc;
  uint32_t num_recs;        // splat records (ids at or above are rejected)
  uint32_t num_entries;     // sorted ids (ranges beyond are clamped)
  // Screen-block lists (masks set): ranges hold (start, count) and sorted_ids
  // the first kListLimit entries of each tile; the others come from the
  // blocks' hit words.
  const uint32_t* masks;
  const uint32_t* chunk_base;
  const uint32_t* chunk_first;
  const uint32_t* block_start;
  const uint32_t* sorted_pairs;
  uint32_t blocks_x, num_blocks;
  // set by launch_composite: a pixel without entries
  uint32_t bg_rgba8;
  float4 bg_f32;
};
cudaError_t launch_composite(const CompositeArgs& a, cudaStream_t s);

}  // namespace cgs
