// Parameter blocks and host launchers of the prefill path (grouped.cu, route.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/umaq_b200.h"

namespace umaq {

constexpr int kTileCapMin = 64, kTileCapMax = 256;   // routes of a tile: transposed kernel (grouped_ts.cu), the others
constexpr int kTileCapWide = 192;                    // wide transposed kernel (grouped_wide.cu)

// The choice between the one-CTA and the transposed kernel when routes concentrate on some experts: see grouped.cu.
struct TileChoice {
  int cols_gate, cols_down;   // column tiles of a row tile of the one-CTA kernel in either GEMM; the transposed one has twice as many
  int sms;
  int num, den;               // transposed tiles while den * their waves < num * the waves of one-CTA tiles
};
#ifdef __CUDACC__
__host__ __device__ inline bool transposed_is_faster(const TileChoice& c, int tiles64, int tiles256) {
  auto waves = [&](int t) { return 2 * ((t * c.cols_gate + c.sms - 1) / c.sms) + (t * c.cols_down + c.sms - 1) / c.sms; };
  return c.den * waves(2 * tiles64) < c.num * 2 * waves(tiles256);        // in half waves: two transposed CTAs share an SM
}
#endif

// Device-side view handed to the grouped GEMM kernel.
struct GroupedParams {
  int k;                      // contraction length
  int n_rows;                 // weight rows per expert in this projection
  const float* scales0;       // [E * n_rows, k/128] (gate or down)
  const float* scales1;       // up (mode 0)
  const int* num_tiles;       // device: entries of the tile table, of up to 64 or 256 routes (SortArgs::tile_cap)
  const int* tile_expert;     // device [max_tiles]
  const int* tile_row0;       // first sorted route row of the tile
  const int* tile_rows;       // valid rows
  int max_tiles;
  int subs;                   // grouped_ts.cu: parts a table entry may be cut into
  int part_major;             // grouped_ts.cu: order of the parts
  int k_splits;               // BF16 down GEMM: the contraction is cut into this many parts, each a tile of its own
  float* part;                // k_splits > 1: float32 sums [k_splits, total rows, n_rows] instead of `out`
  long long part_stride;      // elements of one split
  __nv_bfloat16* out;         // mode 0: intermediate [routes, n_rows]; mode 1: weighted outputs [routes, n_rows]
  long long out_stride;       // elements
  const float* route_weight;  // mode 1: routing weight per sorted route
  int permute_out;            // mode 0: write the [k0,k4,k1,k5,k2,k6,k3,k7] order a quantised GEMM 2 expects
  unsigned* status;           // sticky error word
  // mode 0, optional: fetch the activation rows by index instead of reading pre-gathered rows.  Sorted route r
  // is row gather_route[r] / gather_top_k of gather_src ([tokens, k] BF16, k already in the order the encoding wants)
  const int* gather_route;
  int gather_top_k;
  const __nv_bfloat16* gather_src;
  // 1: this launch runs if transposed tiles are wanted, 2: if one-CTA tiles are, 0: always.  The answer is *use_ts, or
  // follows from the tile table (entries of up to 256 routes) where use_ts is null
  int conditional;
  const int* use_ts;
  TileChoice choice;
  int debug;
  int tma_out;                // mode 1, staged results: map_b1 describes `out` and whole 32-row groups leave by tensor store
};

struct GroupedGemmArgs {
  int mode;                   // 0 gate/up + SwiGLU, 1 down + routing weight
  int enc;
  int num_experts;
  int n_rows;                 // I (mode 0) or H (mode 1)
  int k;                      // H (mode 0) or I (mode 1)
  const void* act;            // bf16 [total_rows, k], sorted by expert
  long long total_rows;
  const void* w0; const float* s0;   // gate or down
  const void* w1; const float* s1;   // up
  const int* num_tiles; const int* tile_expert; const int* tile_row0; const int* tile_rows;
  int max_tiles;
  int tile_cap;               // most routes of a table entry
  long long most;             // most routes an expert can have (0: total_rows)
  const int* use_ts;          // device word of the sort whose table was cut for either kernel (null: decided from the table)
  int conditional;            // 1: transposed tiles, 2: one-CTA tiles, if the device picks them (see GroupedParams); 0: not conditional
  int k_splits;               // > 1 (BF16 down GEMM without routing weights): partial sums into `part`, `out` is not written
  float* part;                // [k_splits, total_rows, n_rows] float32
  __nv_bfloat16* out; long long out_stride;
  const float* route_weight;
  int permute_out;
  unsigned* status;
  int variant;                // 0: by size; 1: one CTA per tile (grouped.cu); 2: persistent CTA pairs (grouped_pair.cu);
                              // 3: transposed tiles (grouped_ts.cu)
  // mode 0 on the one-CTA and the transposed kernel, optional: act = [tokens, k] and the kernel fetches row sorted_route[r] / top_k
  // for sorted route r itself (no gathered copy of the activations)
  const int* gather_route;
  int gather_top_k;
};

// true if launch_grouped_gemm would run the kernel that can fetch its activation rows by index
bool grouped_gemm_can_gather(const GroupedGemmArgs& a);

int launch_grouped_gemm(const GroupedGemmArgs& a, cudaStream_t stream);        // picks the variant
int launch_grouped_gemm_single(const GroupedGemmArgs& a, cudaStream_t stream);
int launch_grouped_gemm_pair(const GroupedGemmArgs& a, cudaStream_t stream);
int launch_grouped_gemm_ts(const GroupedGemmArgs& a, cudaStream_t stream);
int launch_grouped_gemm_wide(const GroupedGemmArgs& a, cudaStream_t stream);   // only when asked for: the table is cut for it

// Whether both GEMMs of a quantised layer run on wide transposed tiles (grouped_wide.cu), the sort cutting its table for them
bool grouped_gemm_takes_wide(int enc, long long rows, int experts, int hidden, int inter);
// Routes per tile that suit the kernel launch_grouped_gemm picks for a layer: the cap to build the tile table with.
int grouped_gemm_tile_cap(int enc, long long rows, int num_experts, int variant);
// Whether that pick has to be made on the device, from the routes that the experts have; `most`: the most one can have
bool grouped_gemm_choice_on_device(int enc, long long rows, int num_experts, long long most, int variant);
TileChoice grouped_gemm_choice(int enc, int inter, int hidden);
// Parts the contraction of a dense BF16 down GEMM (the shared expert's) is cut into
int grouped_gemm_dense_splits(long long rows, int n_rows, int k);
// ... and the room they need, in rows of n_rows float32 sums, for every call of up to `rows` rows (0: never more than one part)
long long grouped_gemm_dense_part_rows(long long rows, int n_rows, int k);
constexpr int kMaxDenseSplits = 8;

// ---- routing (route.cu) ---------------------------------------------------------------------------
struct RouterArgs {
  const __nv_bfloat16* x;        // [tokens, hidden]
  const __nv_bfloat16* weight;   // [experts, hidden]
  int tokens, hidden, experts, top_k, renormalize;
  float* out_weights;            // [tokens, top_k] float32
  long long* out_indices;        // [tokens, top_k] int64
  __nv_bfloat16* out_logits;     // optional [tokens, experts]
};
int launch_router_topk(const RouterArgs& a, cudaStream_t stream);

struct SortArgs {
  const void* indices; int idx64;  // [tokens, top_k]
  const float* weights;            // [tokens, top_k]
  int tokens, top_k, experts;
  int* counts;                     // [experts]
  int* offsets;                    // [experts + 1]
  int* sorted_route;               // [routes] token * top_k + slot, stable by expert
  int* route_pos;                  // [routes] inverse permutation
  float* sorted_weight;            // [routes]
  int* num_tiles; int* tile_expert; int* tile_row0; int* tile_rows;   // tiles of up to tile_cap routes
  int max_tiles;
  int tile_cap;                    // routes per tile, unless use_ts is given
  int* use_ts; TileChoice choice;  // optional: the sort picks the kernel, cuts the table for it and writes 1 (transposed) or 0
  unsigned* status;
  // optional: rows of x in the k order of the quantised GEMMs, written by further CTAs of the first launch
  const __nv_bfloat16* permute_src; __nv_bfloat16* permute_dst; long long permute_chunks;   // 16-byte chunks
  // optional: the tile table of dense_rows rows of a single further expert (the shared one), in tiles of dense_cap
  int dense_rows, dense_cap;
  int* dense_num_tiles; int* dense_expert; int* dense_row0; int* dense_tile_rows;
  int* scratch;                    // optional: ceil(routes / 2048) * experts ints for sorts of more than 16,384 routes in two launches
  long long scratch_ints;
};
int launch_route_sort(const SortArgs& a, cudaStream_t stream);

// rows of x gathered into sorted order; `permute` writes each run of 8 as [0,4,1,5,2,6,3,7]
// valid_rows (device, may be null): only the first *valid_rows sorted routes exist
int launch_gather_rows(const __nv_bfloat16* x, const int* sorted_route, int top_k, long long routes, int hidden,
                       int permute, __nv_bfloat16* out, const int* valid_rows, cudaStream_t stream);
int launch_ep_local_ids(const void* indices, int idx64, long long n, int ranks, int rank, int per_rank, int placement,
                        int* out, cudaStream_t stream);
// expert-parallel exchange over peer memory (ep_peer.cu)
int launch_ep_push(const __nv_bfloat16* x, const void* indices, int idx64, const float* weights, int tokens, int top_k,
                   int hidden, int per_rank, int placement, int flags, const umaq_ep_peers& peers, size_t rows_offset,
                   size_t ids_offset, size_t weights_offset, int* present, cudaStream_t stream);
int launch_ep_barrier(const umaq_ep_peers& peers, size_t flags_offset, unsigned* epoch, unsigned* status,
                      cudaStream_t stream);
int launch_ep_pack(const __nv_bfloat16* x, const int* sorted_route, const int* sorted_key, const float* sorted_weight,
                   const int* offsets, int routes, int top_k, int hidden, int ranks, int per_rank, int capacity,
                   __nv_bfloat16* send_rows, int* send_meta, int* route_slot, int* overflow, cudaStream_t stream);
// Where the combine writes: by default row t of `out`.  With rows > 0 the tokens come in segments of `rows`
// (one per source rank of an expert-parallel exchange) and token t goes to row row0 + t % rows of
// ptr[t / rows] -- a buffer that may live on another GPU (plain peer stores); skip_empty leaves the rows
// of tokens without any present route unwritten.
constexpr int kMaxPeers = 8;
struct SegmentedOut {
  __nv_bfloat16* ptr[kMaxPeers];
  int rows;
  int row0;
  int skip_empty;
};
// experts: ids outside [0, experts) are treated as absent routes.  The shared expert's rows come as BF16 (shared_out) or
// as shared_parts float32 partial sums [shared_parts, tokens, hidden] that are added here and rounded once.
// The sticky status word and where the host looks at it (mapped host memory, null: nowhere).  The last kernel of a call copies
// the word there if it is set, so that a call without an error moves nothing.
struct StatusMirror {
  const unsigned* status;
  unsigned* host;
};
int launch_combine(const __nv_bfloat16* weighted, const void* indices, int idx64, const int* route_pos, int tokens,
                   int top_k, int hidden, int experts, const __nv_bfloat16* shared_out, const float* shared_part,
                   int shared_parts, const __nv_bfloat16* x, const __nv_bfloat16* gate_vec, __nv_bfloat16* out, cudaStream_t stream,
                   const SegmentedOut* segments = nullptr, StatusMirror mirror = {nullptr, nullptr});

}  // namespace umaq
