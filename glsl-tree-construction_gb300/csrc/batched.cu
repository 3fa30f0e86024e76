// batched.cu - many point clouds of uneven size in one stream-ordered build.
//
// No counterpart in the reference (its pipeline builds one cloud,
// main.rs:60-170).  Every cloud's outputs are defined to equal the
// single-cloud 32-bit build of that cloud alone, with cloud-local indices,
// so each cloud is checked against the oracle on its own.
//
// One launch per stage for the whole batch, every size read on the device, so
// the batch captures into one CUDA graph:
//   1. tiles:   each cloud is cut into its own tiles; tile_start[c] is the
//               first tile of cloud c (a device work list, block b taking tile b);
//   2. morton:  32-bit codes, cloud-local point index payload, per-cloud
//               digit histograms of the 4 passes;
//   3. segmented onesweep, 4 passes: a tile's digit bases come from its own
//               cloud's histogram and its decoupled look-back runs only over
//               earlier tiles of the same cloud (a cloud's first tile
//               publishes an inclusive prefix at once);
//   4. unique:  compaction that restarts at every cloud start; cloud c's
//               unique codes land at [U_c, U_{c+1});
//   5. radix tree of each cloud (the window kernel of tree_window.cuh, with
//               pairs that straddle two clouds as boundaries; karras_node
//               under the per-node method) with the edge counts, and a zero
//               edge in each cloud's last slot;
//   6. one inclusive scan of all edge counts; cloud c's node offsets are the
//               scan minus its value just before U_c (the bias);
//   7. octree of each cloud (octree_window.cuh; octree_warp_batch under the
//               per-node method) into its node range starting at O_c =
//               (non-empty clouds before c) + bias.

#include <atomic>
#include <utility>

#include "karras.cuh"
#include "octree_window.cuh"
#include "scan_dev.cuh"
#include "tree_window.cuh"

namespace gtc {

Launch context_launch(gtc_ctx* ctx, gtc_stream_t stream);
gtc_status context_error(gtc_ctx* ctx, gtc_status s, const char* msg, cudaError_t e);
cudaEvent_t context_stage_begin(gtc_ctx* ctx, gtc_stream_t stream);
bool context_stage_idle(const gtc_ctx* ctx);
void context_stage_end(gtc_ctx* ctx, gtc_stream_t stream, cudaEvent_t a, int stage);

namespace {

// Brackets one stage's launches with events while profiling is on.
struct Stage {
  gtc_ctx* ctx;
  gtc_stream_t s;
  int stage;
  cudaEvent_t a;
  Stage(gtc_ctx* c, gtc_stream_t st, int sg) : ctx(c), s(st), stage(sg), a(context_stage_begin(c, st)) {}
  ~Stage() { context_stage_end(ctx, s, a, stage); }
};

constexpr int BRADIX = 256;
constexpr int BPASSES = 4;  // 30-bit codes in 8-bit digits
constexpr int BM_THREADS = 512;  // Morton kernel: one block per tile
// Segmented onesweep tile shapes (threads x keys per thread), compiled as
// variants: pinned with gtc_batched_set_variant, else the autotuner's pick
// for the batch's size (gtc_autotune_batched), else by size (below).  Every tile
// division of the batch (tile list, Morton blocks, sort tiles) uses the
// chosen shape's tile.
struct BtVariant {
  int threads, kpt;
};
constexpr BtVariant kBtVariants[] = {{512, 12}, {256, 16}, {384, 16}, {512, 8}, {256, 24}, {512, 4}, {256, 16}};
constexpr int kBtNumVariants = sizeof(kBtVariants) / sizeof(kBtVariants[0]);
// Variant 6 is 256 x 16 held to 64 registers (four blocks per SM), as sort.cu's
// variant 7; variant 5 has short tiles for small batches, where a pass is one
// chain of dependent steps, and is limited to BT_SMALL_MAX points, which bounds
// the workspace's descriptors.  Whole builds (us):
//   points, clouds         512 x 12   512 x 4   256 x 16 at 4 blocks per SM
//   9,293, 16                  55.5      48.3      56.5
//   300,125, 64                90.3      74.8      81.6
//   422,794, 200               93.5      83.3      94.9
//   598,201, 16                98.7      89.7     101.7
//   1,562,588, 20             154.5        -      172.3
//   3,211,561, 200            257.7        -      247.3
//   74,044,652, 512          3640.1        -     3552.9
// (512 x 4 took over from 256 x 8: 77.0 -> 74.6 us for 64 clouds of 300 to
// 20,000 points as a graph, the same tile with half the ranking steps.)
constexpr int BT_SMALL = 5, BT_LARGE = 6;
constexpr uint32_t BT_SMALL_MAX = 600000;
constexpr uint32_t BT_LARGE_MIN = 2000000;  // untuned batches from here on take variant 6
// Most whole tiles of any variant for n points, and for up to n points: a
// workspace made for n also serves fewer, which may have more (short) tiles.
constexpr uint32_t bt_tiles(uint32_t n) {
  const uint32_t tile = n <= BT_SMALL_MAX ? 2048 : 4096;
  return ((n > 0 ? n : 1) + tile - 1) / tile;
}
constexpr uint32_t bt_tiles_up_to(uint32_t n) {
  return n > BT_SMALL_MAX && bt_tiles(n) < bt_tiles(BT_SMALL_MAX) ? bt_tiles(BT_SMALL_MAX) : bt_tiles(n);
}
constexpr uint32_t MAX_CLOUDS = 1u << 20;

// Tiles per cloud and non-empty clouds, both scanned (one block).  The
// offsets must partition [0, n): off[0] = 0, non-decreasing, off[S] = n.
// Otherwise the batch is flagged bad, every later kernel returns at once and
// the outputs say zero unique codes and zero nodes.  Blocks past the first
// clear the words that must start at zero (the clouds' digit histograms and
// the scans' descriptors), in place of a memset each; the first clears the
// counters, the bad flag among them.
__global__ void __launch_bounds__(1024) bt_tiles_kernel(const uint32_t* off, uint32_t S, uint32_t n, uint32_t tile,
                                                        uint32_t* tile_start, uint32_t* ne_start, uint32_t* counters,
                                                        uint32_t* bad, uint32_t* uoff, uint4* zero, size_t zero_vecs,
                                                        uint32_t* status) {
  griddep_wait();
  if (blockIdx.x > 0) {
    for (size_t i = (size_t)(blockIdx.x - 1) * 1024 + threadIdx.x; i < zero_vecs; i += (size_t)(gridDim.x - 1) * 1024)
      zero[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  __shared__ uint32_t s_t[1024], s_n[1024];
  if (threadIdx.x < 64) counters[threadIdx.x] = 0;
  const uint32_t per = (S + 1023) / 1024;
  const uint32_t first = threadIdx.x * per, last = min(first + per, S);
  bool ok = threadIdx.x != 0 || (off[0] == 0 && off[S] == n);
  for (uint32_t c = first; c < last; ++c) ok = ok && off[c + 1] >= off[c];
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) {
      *bad = 1;
      tile_start[S] = 0;
      uoff[S] = 0;
      atomicOr(status, DEV_BAD_INPUT);
    }
    return;
  }
  uint32_t t = 0, ne = 0;
  for (uint32_t c = first; c < last; ++c) {
    const uint32_t len = off[c + 1] - off[c];
    t += (len + tile - 1) / tile;
    ne += len > 0;
  }
  s_t[threadIdx.x] = t;
  s_n[threadIdx.x] = ne;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const uint32_t a = threadIdx.x >= (unsigned)o ? s_t[threadIdx.x - o] : 0u;
    const uint32_t b = threadIdx.x >= (unsigned)o ? s_n[threadIdx.x - o] : 0u;
    __syncthreads();
    s_t[threadIdx.x] += a;
    s_n[threadIdx.x] += b;
    __syncthreads();
  }
  t = threadIdx.x ? s_t[threadIdx.x - 1] : 0u;
  ne = threadIdx.x ? s_n[threadIdx.x - 1] : 0u;
  for (uint32_t c = first; c < last; ++c) {
    const uint32_t len = off[c + 1] - off[c];
    tile_start[c] = t;
    ne_start[c] = ne;
    t += (len + tile - 1) / tile;
    ne += len > 0;
  }
  if (threadIdx.x == 1023) {
    tile_start[S] = s_t[1023];
    ne_start[S] = s_n[1023];
  }
}

struct TileRange {
  uint32_t cloud, local, base, valid;
};

// Tile t of the batch, its cloud given.
__device__ __forceinline__ TileRange tile_range(uint32_t t, uint32_t cloud, const uint32_t* tile_start,
                                                const uint32_t* off, uint32_t tile) {
  TileRange r;
  r.cloud = cloud;
  r.local = t - tile_start[r.cloud];
  r.base = off[r.cloud] + r.local * tile;
  r.valid = min(tile, off[r.cloud + 1] - r.base);
  return r;
}

// Morton codes (10 bits per axis) and per-cloud digit histograms; also clears
// the look-back descriptors of all passes and records every tile's cloud for
// the sort.  (No payload is written: the first sort pass makes it.)  A block
// takes `group` consecutive tiles and adds its histogram to the cloud's only
// when the cloud changes: the 1,024 global atomics of a flush cost as much as
// the tile's points.
template <int Q>
__global__ void __launch_bounds__(BM_THREADS) bt_morton_kernel(const float4* pts, const uint32_t* off,
                                                               uint32_t S, const uint32_t* tile_start, uint32_t tile,
                                                               uint32_t group, float mn, float rg, float inv_rg,
                                                               uint32_t* __restrict__ keys, uint32_t* tile_cloud,
                                                               uint32_t* seg_hist, uint4* desc, size_t desc_vecs) {
  griddep_wait();
  __shared__ uint32_t s_hist[BPASSES * BRADIX];
  __shared__ uint32_t s_cloud;
  const int tid = threadIdx.x;
  for (int i = tid; i < BPASSES * BRADIX; i += BM_THREADS) s_hist[i] = 0;
  const size_t stride = (size_t)gridDim.x * BM_THREADS;
  for (size_t i = (size_t)blockIdx.x * BM_THREADS + tid; i < desc_vecs; i += stride) desc[i] = make_uint4(0, 0, 0, 0);
  const uint32_t tiles = tile_start[S];
  const uint32_t t0 = blockIdx.x * group;
  if (t0 >= tiles) return;
  if (tid < 32) {
    const uint32_t c = warp_upper_bound_u32(tile_start, S + 1, t0) - 1;
    if (tid == 0) s_cloud = c;
  }
  __syncthreads();
  uint32_t cloud = s_cloud;
  auto flush = [&] {
    __syncthreads();
    uint32_t* h = seg_hist + (size_t)cloud * BPASSES * BRADIX;
    for (int i = tid; i < BPASSES * BRADIX; i += BM_THREADS) {
      const uint32_t c = s_hist[i];
      if (c) atomicAdd(h + i, c);
      s_hist[i] = 0;
    }
    __syncthreads();
  };
  for (uint32_t t = t0; t < min(t0 + group, tiles); ++t) {  // block-uniform
    if (t >= tile_start[cloud + 1]) {
      flush();
      ++cloud;
      if (t >= tile_start[cloud + 1]) cloud = warp_upper_bound_u32(tile_start, S + 1, t) - 1;  // empty clouds between
    }
    if (tid == 0) tile_cloud[t] = cloud;
    const TileRange r = tile_range(t, cloud, tile_start, off, tile);
    for (uint32_t i0 = tid; i0 < r.valid; i0 += 4 * BM_THREADS) {  // four points in flight
      float4 p[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t i = i0 + q * BM_THREADS;
        p[q] = i < r.valid ? __ldcs(pts + r.base + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t i = i0 + q * BM_THREADS;
        if (i < r.valid) {
          const uint32_t k = encode_point<uint32_t, Q>(p[q], mn, rg, inv_rg);
          keys[r.base + i] = k;
#pragma unroll
          for (int d = 0; d < BPASSES; ++d) atomicAdd(&s_hist[d * BRADIX + ((k >> (8 * d)) & 255u)], 1u);
        }
      }
    }
  }
  flush();
}

// Per cloud and pass: digit counts -> global digit bases, in place.  Only the
// 64-register tiles of large batches want it (bt_onesweep_kernel).
__global__ void __launch_bounds__(BRADIX) bt_seg_scan_kernel(uint32_t* seg_hist, const uint32_t* off) {
  griddep_wait();
  __shared__ uint32_t s_w[BRADIX / 32];
  const uint32_t c = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int p = 0; p < BPASSES; ++p) {
    uint32_t* h = seg_hist + ((size_t)c * BPASSES + p) * BRADIX;
    const uint32_t v = h[tid];
    const uint32_t incl = warp_inclusive_sum(v);
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    uint32_t pre = 0;
    for (int w = 0; w < warp; ++w) pre += s_w[w];
    h[tid] = off[c] + pre + incl - v;
    __syncthreads();
  }
}

template <int THREADS, int KPT>
struct BtSmem {
  static constexpr int WARPS = THREADS / 32;
  static constexpr int TILE = THREADS * KPT;
  uint32_t keys[TILE];
  uint32_t vals[TILE];
  uint32_t warp_hist[WARPS][BRADIX];
  uint32_t gbase[BRADIX];
  uint32_t hist_sums[BRADIX / 32];
  uint32_t warp_sums[WARPS + 1];
};

// One segmented onesweep pass: the single-cloud pass of sort.cu with tiles
// confined to one cloud and digit bases from that cloud's histogram.  Every
// tile scans that for itself, behind its keys' loads, which saves a launch:
// 64 clouds of 300 to 20,000 points 74.6 -> 71.5 us.  SCANNED takes the bases
// from bt_seg_scan_kernel: in variant 6 the scan in the tile spills, and
// 512 clouds of 74M points took 3641 us against 3566.  A
// cloud's last tile is padded with all-ones keys, which rank last in the tile
// and are never stored.  Its descriptor counts them, but no tile reads it:
// the next tile starts another cloud and does not look back.  FIRST: the
// payload is the point's index in its cloud, made here.
template <int THREADS, int KPT, int MINB, bool FIRST, bool SCANNED>
__global__ void __launch_bounds__(THREADS, MINB) bt_onesweep_kernel(const uint32_t* kin,
                                                                 const uint32_t* vin,
                                                                 uint32_t* __restrict__ kout,
                                                                 uint32_t* __restrict__ vout, const uint32_t* off,
                                                                 uint32_t S, const uint32_t* tile_start,
                                                                 const uint32_t* tile_cloud, int shift,
                                                                 const uint32_t* seg_hist, int pass, uint32_t* desc,
                                                                 uint32_t* status) {
  griddep_wait();
  using Sm = BtSmem<THREADS, KPT>;
  constexpr int WARPS = Sm::WARPS;
  static_assert(THREADS >= BRADIX, "one thread per digit");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Sm& s = *reinterpret_cast<Sm*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t tile = blockIdx.x;  // sort.cu has what that assumes
  if (tile >= tile_start[S]) return;
  const TileRange r = tile_range(tile, tile_cloud[tile], tile_start, off, Sm::TILE);

  uint32_t key[KPT], val[KPT];
  const uint32_t wbase = warp * 32 * KPT + lane;
#pragma unroll
  for (int j = 0; j < KPT; ++j) {
    const uint32_t i = wbase + j * 32;
    key[j] = (i < r.valid) ? kin[r.base + i] : 0xffffffffu;
    if (FIRST) val[j] = r.local * Sm::TILE + i;
    else val[j] = (i < r.valid) ? vin[r.base + i] : 0u;
  }
  if (!SCANNED && tid < BRADIX) {  // the cloud's keys of smaller digits, but for earlier warps' digits
    const uint32_t h = seg_hist[((size_t)r.cloud * BPASSES + pass) * BRADIX + tid];
    const uint32_t incl = warp_inclusive_sum(h);
    s.gbase[tid] = incl - h;
    if (lane == 31) s.hist_sums[warp] = incl;
  }
  uint32_t* my_hist = s.warp_hist[warp];
#pragma unroll
  for (int i = 0; i < BRADIX / 32; ++i) my_hist[i * 32 + lane] = 0;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < KPT; ++j) {
    const uint32_t d = (key[j] >> shift) & 255u;
    const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
    if (__all_sync(0xffffffffu, d == d0)) {
      if (lane == 0) atomicAdd(&my_hist[d], 32u);
    } else {
      atomicAdd(&my_hist[d], 1u);
    }
  }
  __syncthreads();
  uint32_t count = 0;
  if (tid < BRADIX) {
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const uint32_t c = s.warp_hist[w][tid];
      s.warp_hist[w][tid] = count;
      count += c;
    }
    st_relaxed(desc + (size_t)tile * BRADIX + tid, (count << 2) | (r.local == 0 ? FLAG_INCLUSIVE : FLAG_AGGREGATE));
  }
  // Exclusive scan of the 256 digit counts (threads past 256 add zeros).
  uint32_t total;
  const uint32_t doff = block_exclusive<THREADS>(tid < BRADIX ? count : 0u, s.warp_sums, &total);
  if (tid < BRADIX) {
#pragma unroll
    for (int w = 0; w < WARPS; ++w) s.warp_hist[w][tid] += doff;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < KPT; ++j) {
    const uint32_t d = (key[j] >> shift) & 255u;
    const uint32_t peers = warp_peers<8>(d);
    const int leader = 31 - __clz(peers);
    uint32_t b0 = 0;
    if (lane == leader) b0 = atomicAdd(&my_hist[d], (uint32_t)__popc(peers));
    b0 = __shfl_sync(0xffffffffu, b0, leader);
    const uint32_t local = b0 + __popc(peers & lt_mask);
    s.keys[local] = key[j];
    s.vals[local] = val[j];
  }
  if (tid < BRADIX) {
    uint32_t excl = 0;
    if (r.local > 0) {  // look back only over this cloud's earlier tiles
      excl = lookback_window<8, BRADIX>(desc, tile, tid, status);
      st_relaxed(desc + (size_t)tile * BRADIX + tid, ((excl + count) << 2) | FLAG_INCLUSIVE);
    }
    if constexpr (SCANNED) {
      s.gbase[tid] = seg_hist[((size_t)r.cloud * BPASSES + pass) * BRADIX + tid] + excl - doff;
    } else {
      uint32_t base = r.base - r.local * Sm::TILE + excl - doff;
      for (int w = 0; w < warp; ++w) base += s.hist_sums[w];
      s.gbase[tid] += base;
    }
  }
  __syncthreads();
  // o stays inside the cloud while every look-back completes; after one ran
  // out (DEV_TIMEOUT) a later pass may see digit counts that disagree with
  // the cloud's histogram, and the check keeps its writes in bounds.
  const uint32_t end = off[r.cloud + 1];
  for (uint32_t i = tid; i < r.valid; i += THREADS) {
    const uint32_t k = s.keys[i];
    const uint32_t o = s.gbase[(k >> shift) & 255u] + i;
    if (o >= end) continue;
    kout[o] = k;
    vout[o] = s.vals[i];
  }
}

// Unique with a restart at every cloud start (a cloud's first code is always
// kept): scan.cu's two resident forms, out of place, on rows of 32 codes per
// warp.  A warp steps through the clouds that start in its rows, in order, so
// a row's cloud starts come as a bit mask, and every cloud's U_c is recorded
// where it starts - an empty cloud's too, which starts where the next one
// does.  BtStarts is that position: the next cloud to start and its offset.
struct BtStarts {
  uint32_t cloud, at;
};
// The first cloud that starts at or after position r (whole warp).
__device__ __forceinline__ BtStarts bt_starts_from(const uint32_t* off, uint32_t S, uint32_t r) {
  const uint32_t c = r > 0 ? warp_upper_bound_u32(off, S + 1, r - 1) : 0u;
  return BtStarts{c, c <= S ? off[c] : ~0u};
}
// The cloud starts in rows [r0, end) as masks, row j's in lane j; steps past
// them, 32 clouds at a time, and past the rest of a long run of empty clouds by
// search (whole warp).  RECORD: writes their U_c instead, with row j's kept
// mask and first output position in lane j.  One loop over the rows that clouds
// start in, outside the caller's unrolled ones, which it would fill with code.
template <bool RECORD>
__device__ __forceinline__ uint32_t bt_starts(const uint32_t* off, uint32_t S, uint32_t r0, uint32_t end, BtStarts& st,
                                              uint32_t bals, uint32_t runs, uint32_t* uoff) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t masks = 0;
#pragma unroll 1
  while (st.cloud < S && st.at < end) {  // warp-uniform
    const uint32_t j = (st.at - r0) / 32, r = r0 + 32 * j;
    const uint32_t c = st.cloud + lane;
    const uint32_t p = off[min(c, S)];
    const bool in = c < S && p < r + 32;
    const uint32_t k = __popc(__ballot_sync(0xffffffffu, in));  // a prefix of the lanes, of one at least
    uint32_t bal = 0, run = 0;
    if (RECORD) {
      bal = __shfl_sync(0xffffffffu, bals, j);
      run = __shfl_sync(0xffffffffu, runs, j);
      if (in) uoff[c] = run + __popc(bal & ((1u << (p - r)) - 1u));
    } else {
      const uint32_t m = __reduce_or_sync(0xffffffffu, in ? 1u << (p - r) : 0u);
      if (lane == j) masks |= m;
    }
    st.cloud += k;
    if (k < 32) {
      st.at = __shfl_sync(0xffffffffu, p, k);
    } else {
      const uint32_t last = __shfl_sync(0xffffffffu, p, 31);
      st.at = off[st.cloud];
      if (st.at == last) {
        const uint32_t c0 = st.cloud;
        st.cloud += warp_upper_bound_u32(off + c0, S - c0, last);
        if (RECORD) {
          for (uint32_t q = c0 + lane; q < st.cloud; q += 32) uoff[q] = run + __popc(bal & ((1u << (last - r)) - 1u));
        }
        st.at = off[st.cloud];
      }
    }
  }
  return masks;
}
// Past the last row: the empty clouds behind it, from cloud c on, and U_S (whole warp).
__device__ __forceinline__ void bt_record_end(uint32_t c, uint32_t S, uint32_t run, uint32_t* uoff) {
  for (c += threadIdx.x & 31; c <= S; c += 32) uoff[c] = run;
}

template <int ROWS>
__global__ void __launch_bounds__(CS_THREADS) bt_row_unique_kernel(const uint32_t* kin, const uint32_t* vin,
                                                                   uint32_t* __restrict__ kout,
                                                                   uint32_t* __restrict__ vout, uint32_t n,
                                                                   const uint32_t* off, uint32_t S, uint32_t* uoff,
                                                                   uint32_t* ws, const uint32_t* bad,
                                                                   uint32_t* status) {
  griddep_wait();
  __shared__ uint32_t s_seg[CS_WARPS];
  __shared__ uint32_t s_red[CS_WARPS];
  if (*bad) return;  // the same word for every block
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t r0 = (blockIdx.x * CS_WARPS + warp) * (ROWS * 32);
  uint32_t k[ROWS], v[ROWS];
#pragma unroll
  for (int j = 0; j < ROWS; ++j) {
    const uint32_t i = r0 + j * 32 + lane;
    k[j] = i < n ? kin[i] : 0u;
    v[j] = i < n ? vin[i] : 0u;
  }
  uint32_t carry = (lane == 0 && r0 > 0 && r0 < n) ? kin[r0 - 1] : 0u;
  const BtStarts first = bt_starts_from(off, S, min(r0, n));
  BtStarts st = first;
  const uint32_t masks = bt_starts<false>(off, S, r0, min(r0 + ROWS * 32, n), st, 0u, 0u, nullptr);
  uint32_t keep = 0, cnt = 0;
#pragma unroll
  for (int j = 0; j < ROWS; ++j) {
    const uint32_t i = r0 + j * 32 + lane;
    const uint32_t smask = __shfl_sync(0xffffffffu, masks, j);
    uint32_t prev = __shfl_up_sync(0xffffffffu, k[j], 1);
    if (lane == 0) prev = carry;
    const bool kp = i < n && (k[j] != prev || ((smask >> lane) & 1u));
    keep |= (uint32_t)kp << j;
    cnt += __popc(__ballot_sync(0xffffffffu, kp));
    carry = __shfl_sync(0xffffffffu, k[j], 31);
  }
  if (lane == 0) s_seg[warp] = cnt;
  uint32_t run = cs_block_prefix(ws + 64, s_seg, s_red, status) + s_seg[warp];
  uint32_t bals = 0, runs = 0;
#pragma unroll
  for (int j = 0; j < ROWS; ++j) {
    const bool kp = (keep >> j) & 1u;
    const uint32_t bal = __ballot_sync(0xffffffffu, kp);
    if (kp) {
      const uint32_t o = run + __popc(bal & lt);
      kout[o] = k[j];
      vout[o] = v[j];
    }
    if (lane == j) {
      bals = bal;
      runs = run;
    }
    run += __popc(bal);
  }
  st = first;
  bt_starts<true>(off, S, r0, min(r0 + ROWS * 32, n), st, bals, runs, uoff);
  if (blockIdx.x == gridDim.x - 1 && warp == CS_WARPS - 1) bt_record_end(st.cloud, S, run, uoff);
}

// Segments of any length, read twice (scan.cu's chunk_unique_kernel), eight
// rows in flight per warp, three blocks per SM (512 clouds, 74M points: 263 of
// 3,515 us).
__global__ void __launch_bounds__(CS_THREADS, 3) bt_chunk_unique_kernel(const uint32_t* kin, const uint32_t* vin,
                                                                        uint32_t* __restrict__ kout,
                                                                        uint32_t* __restrict__ vout, uint32_t n,
                                                                        const uint32_t* off, uint32_t S,
                                                                        uint32_t* uoff, uint32_t* ws,
                                                                        const uint32_t* bad, uint32_t* status) {
  griddep_wait();
  __shared__ uint32_t s_seg[CS_WARPS];
  __shared__ uint32_t s_red[CS_WARPS];
  if (*bad) return;  // the same word for every block
  constexpr int R = 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t nseg = gridDim.x * CS_WARPS;
  const uint64_t SL = (((uint64_t)n + nseg - 1) / nseg + 31) & ~(uint64_t)31;
  const uint64_t beg64 = (uint64_t)(blockIdx.x * CS_WARPS + warp) * SL;
  const uint32_t beg = (uint32_t)min(beg64, (uint64_t)n);
  const uint32_t end = (uint32_t)min(beg64 + SL, (uint64_t)n);
  const uint32_t first_prev = (beg > 0 && beg < end) ? kin[beg - 1] : 0u;
  const BtStarts first = bt_starts_from(off, S, beg);
  const uint64_t keep_pol = l2_keep_policy(), drop_pol = l2_drop_policy();

  // 1. kept codes per segment (codes tagged to stay in L2 for step 3)
  uint32_t cnt = 0;
  {
    uint32_t carry = first_prev;
    BtStarts st = first;
    for (uint32_t r0 = beg; r0 < end; r0 += 32 * R) {
      uint32_t k[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const uint32_t i = r0 + 32 * j + lane;
        k[j] = i < end ? ld_hint(kin + i, keep_pol) : 0u;
      }
      const uint32_t masks = bt_starts<false>(off, S, r0, min(r0 + 32 * R, end), st, 0u, 0u, nullptr);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const uint32_t i = r0 + 32 * j + lane;
        const uint32_t smask = __shfl_sync(0xffffffffu, masks, j);
        uint32_t prev = __shfl_up_sync(0xffffffffu, k[j], 1);
        if (lane == 0) prev = carry;
        cnt += __popc(__ballot_sync(0xffffffffu, i < end && (k[j] != prev || ((smask >> lane) & 1u))));
        carry = __shfl_sync(0xffffffffu, k[j], 31);
      }
    }
  }
  if (lane == 0) s_seg[warp] = cnt;

  // 2. block prefix
  uint32_t run = cs_block_prefix(ws + 64, s_seg, s_red, status);
  run += s_seg[warp];

  // 3. rescan and write, recording every cloud's U_c
  BtStarts st = first;
  {
    uint32_t carry = first_prev;
    for (uint32_t r0 = beg; r0 < end; r0 += 32 * R) {
      uint32_t k[R], v[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const uint32_t i = r0 + 32 * j + lane;
        k[j] = i < end ? ld_hint(kin + i, drop_pol) : 0u;
        v[j] = i < end ? ld_hint(vin + i, drop_pol) : 0u;
      }
      BtStarts here = st;
      const uint32_t masks = bt_starts<false>(off, S, r0, min(r0 + 32 * R, end), here, 0u, 0u, nullptr);
      uint32_t bals = 0, runs = 0;
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const uint32_t i = r0 + 32 * j + lane;
        const uint32_t smask = __shfl_sync(0xffffffffu, masks, j);
        uint32_t prev = __shfl_up_sync(0xffffffffu, k[j], 1);
        if (lane == 0) prev = carry;
        const bool kp = i < end && (k[j] != prev || ((smask >> lane) & 1u));
        const uint32_t bal = __ballot_sync(0xffffffffu, kp);
        if (kp) {
          const uint32_t o = run + __popc(bal & lt);
          kout[o] = k[j];
          vout[o] = v[j];
        }
        if (lane == j) {
          bals = bal;
          runs = run;
        }
        run += __popc(bal);
        carry = __shfl_sync(0xffffffffu, k[j], 31);
      }
      bt_starts<true>(off, S, r0, min(r0 + 32 * R, end), st, bals, runs, uoff);
    }
  }
  // The last warp of the last block ends at n: its running count is U.
  if (blockIdx.x == gridDim.x - 1 && warp == CS_WARPS - 1) bt_record_end(st.cloud, S, run, uoff);
}

// Radix tree of every cloud, one thread per unique code.
__global__ void __launch_bounds__(256) bt_tree_kernel(const uint32_t* codes, const uint32_t* uoff,
                                                      uint32_t S, uint8_t* prefix_n, uint8_t* hll, uint8_t* hlr,
                                                      int32_t* left, int32_t* parent, uint32_t* edge) {
  griddep_wait();
  const uint32_t U = uoff[S];
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < U; g += stride) {
    const uint32_t c = owner(uoff, S, g);
    const uint32_t U0 = uoff[c];
    const int i = (int)(g - U0);
    const int m = (int)(uoff[c + 1] - U0) - 1;
    if (i == 0 && m > 0) {
      parent[U0] = 0;
      edge[U0] = 0;
    }
    if (i < m)
      karras_node<uint32_t>(codes + U0, m, i, prefix_n + U0, hll + U0, hlr + U0, left + U0, parent + U0,
                            edge + U0);
    else
      edge[g] = 0;  // the cloud's last slot adds nothing to the scan
  }
}

// Per cloud: u, m, o and the first node slot O_c, from the global scan; and
// the cloud's (U0, U1, bias, O_c) for the octree kernel.
__global__ void bt_cloud_offsets_kernel(uint32_t* uoff, const uint32_t* ne_start, const uint32_t* ps, uint32_t S,
                                        uint32_t* node_off, uint32_t* cloud_counts, uint4* cinfo,
                                        const uint32_t* bad) {
  griddep_wait();
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= S) return;
  if (*bad) {
    uoff[c] = 0;
    node_off[c] = 0;
    cloud_counts[3 * c + 0] = cloud_counts[3 * c + 1] = cloud_counts[3 * c + 2] = 0;
    if (c == S - 1) node_off[S] = 0;
    return;
  }
  const uint32_t U0 = uoff[c], U1 = uoff[c + 1];
  const uint32_t u = U1 - U0;
  const uint32_t bias = U0 > 0 ? ps[U0 - 1] : 0u;
  const uint32_t O = ne_start[c] + bias;
  const uint32_t o = u > 0 ? 1 + ps[U1 - 1] - bias : 0u;
  node_off[c] = O;
  cinfo[c] = make_uint4(U0, U1, bias, O);
  cloud_counts[3 * c + 0] = u;
  cloud_counts[3 * c + 1] = u > 0 ? u - 1 : 0u;
  cloud_counts[3 * c + 2] = o;
  if (c == S - 1) node_off[S] = O + o;
}

// Octree of every cloud, and the cloud-local node offsets (what the
// single-cloud node-offset scan gives each cloud).  Warp slices of 32 codes:
// the slice's cloud comes from one binary search (then a step or two per
// lane), every lane writes its node offset, and the codes that own octree
// nodes are compacted, with their clouds, into a per-warp queue and run 32
// at a time through the single-cloud kernel's breadth-first warp batch
// (octree_warp_batch), each lane with its own cloud.
constexpr int BT_OCT_THREADS = 256;

__global__ void __launch_bounds__(BT_OCT_THREADS) bt_octree_kernel(const uint32_t* codes,
                                                                   const uint32_t* uoff, uint32_t S,
                                                                   const uint4* cinfo, const uint8_t* prefix_n,
                                                                   const uint8_t* hll, const uint8_t* hlr,
                                                                   const int32_t* left, const uint32_t* edge,
                                                                   const uint32_t* ps, uint32_t* node_offsets,
                                                                   float mn, float rg, gtc_octnode* nodes,
                                                                   uint32_t capacity, uint32_t lmask_keep,
                                                                   uint32_t* status) {
  griddep_wait();
  constexpr int WARPS = BT_OCT_THREADS / 32;
  constexpr int A = KeyTraits<uint32_t>::A;
  __shared__ OctWarp s_warp[WARPS];
  __shared__ uint32_t s_cloud[WARPS][64];
  const uint32_t U = uoff[S];
  const int lane = threadIdx.x & 31;
  OctWarp& Wq = s_warp[threadIdx.x >> 5];
  uint32_t* qc = s_cloud[threadIdx.x >> 5];
  uint32_t qn = 0;  // warp-uniform
  const uint32_t warps = gridDim.x * WARPS;
  auto run_batch = [&](uint32_t cnt) {
    const bool valid = (uint32_t)lane < cnt;
    const uint32_t g = valid ? Wq.q[lane] : 0u;
    const uint32_t c = valid ? qc[lane] : 0u;
    const uint32_t rest_g = (lane + 32 < qn) ? Wq.q[lane + 32] : 0u;
    const uint32_t rest_c = (lane + 32 < qn) ? qc[lane + 32] : 0u;
    __syncwarp();
    if (lane + 32 < qn) {
      Wq.q[lane] = rest_g;
      qc[lane] = rest_c;
    }
    qn -= cnt;
    OctCloud cl{0u, 0u, 0u, 0, nodes, 0u};
    bool ok = valid;
    if (valid) {
      const uint4 ci = cinfo[c];
      cl.u0 = ci.x;
      cl.mend = ci.y - 1;
      cl.bias = ci.z;
      cl.root_level = (prefix_n[ci.x] - A) / 3;
      if (ci.w >= capacity) {
        if (g == ci.x) atomicOr(status, DEV_CAPACITY);
        ok = false;
      } else {
        cl.nodes = nodes + ci.w;
        cl.capacity = capacity - ci.w;
      }
    }
    octree_warp_batch<uint32_t, true>(Wq, ok, g, cl, codes, prefix_n, hll, hlr, left, edge, ps, mn, rg, lmask_keep,
                                      status);
  };
  for (uint32_t base = (blockIdx.x * WARPS + (threadIdx.x >> 5)) * 32; base < U; base += warps * 32) {
    const uint32_t g = base + lane;
    bool act = false;
    uint32_t c = owner(uoff, S, base);  // the same address in every lane
    if (g < U) {
      while (g >= uoff[c + 1]) ++c;
      const uint4 ci = cinfo[c];
      const uint32_t k = g - ci.x, m = ci.y - ci.x - 1;
      node_offsets[g] = (k == 0) ? 0u : ps[g] - ci.z;
      if (m == 0) {  // a cloud of one distinct key: its root alone (D18)
        if (ci.w < capacity)
          octree_root_only<uint32_t>(nodes + ci.w, capacity - ci.w, mn, rg, status);
        else
          atomicOr(status, DEV_CAPACITY);
      } else {
        act = k < m && (k == 0 || edge[g] > 0);
      }
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, act);
    if (act) {
      const uint32_t pos = qn + __popc(bal & ((1u << lane) - 1u));
      Wq.q[pos] = g;
      qc[pos] = c;
    }
    qn += __popc(bal);
    __syncwarp();
    if (qn >= 32) run_batch(32u);
  }
  if (qn > 0) run_batch(qn);
}

struct BtPass {
  const uint32_t* kin;
  const uint32_t* vin;
  uint32_t* kout;
  uint32_t* vout;
  const uint32_t* off;
  uint32_t S;
  const uint32_t* tile_start;
  const uint32_t* tile_cloud;
  int pass;
  const uint32_t* seg_hist;
  uint32_t* desc;
};

template <int THREADS, int KPT, int MINB, bool SCANNED = false>
cudaError_t launch_bt_pass(const Launch& L, uint32_t grid, const BtPass& a) {
  using Sm = BtSmem<THREADS, KPT>;
  auto kern = a.pass == 0 ? bt_onesweep_kernel<THREADS, KPT, MINB, true, SCANNED>
                          : bt_onesweep_kernel<THREADS, KPT, MINB, false, SCANNED>;
  cudaError_t e = kernel_setup(kern, THREADS, sizeof(Sm));
  if (e != cudaSuccess) return e;
  return launch_kernel(L, kern, grid, THREADS, sizeof(Sm), a.kin, a.vin, a.kout, a.vout, a.off, a.S, a.tile_start,
                       a.tile_cloud, 8 * a.pass, a.seg_hist, a.pass, a.desc, L.status);
}

cudaError_t launch_bt_variant(int v, const Launch& L, uint32_t grid, const BtPass& a) {
  switch (v) {
    case 1: return launch_bt_pass<256, 16, 3>(L, grid, a);
    case 2: return launch_bt_pass<384, 16, 2>(L, grid, a);
    case 3: return launch_bt_pass<512, 8, 2>(L, grid, a);
    case 4: return launch_bt_pass<256, 24, 2>(L, grid, a);
    case BT_SMALL: return launch_bt_pass<512, 4, 2>(L, grid, a);
    case BT_LARGE: return launch_bt_pass<256, 16, 4, true>(L, grid, a);
    default: return launch_bt_pass<512, 12, 2>(L, grid, a);
  }
}

// Unique by the row kernel of the smallest ROWS whose blocks are all resident
// at one per SM (two at the most rows; scan.cu has the reason and times), or
// by segments read twice.
template <int ROWS>
cudaError_t launch_bt_unique(const Launch& L, const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout,
                             uint32_t n, const uint32_t* off, uint32_t S, uint32_t* uoff, uint32_t* ws,
                             uint32_t ws_blocks, const uint32_t* bad) {
  int occ = 1;
  if constexpr (ROWS <= 16) {
    auto kern = bt_row_unique_kernel<ROWS>;
    cudaError_t e = kernel_setup(kern, CS_THREADS, 0, &occ);
    if (e != cudaSuccess) return e;
    const uint32_t g = ceil_div(n, ROWS * CS_THREADS);
    if (g > min(occ, ROWS < 16 ? 1 : 2) * (uint32_t)L.num_sms || g > ws_blocks)
      return launch_bt_unique<ROWS * 2>(L, kin, vin, kout, vout, n, off, S, uoff, ws, ws_blocks, bad);
    return launch_kernel(L, kern, g, CS_THREADS, 0, kin, vin, kout, vout, n, off, S, uoff, ws, bad, L.status);
  } else {
    cudaError_t e = kernel_setup(bt_chunk_unique_kernel, CS_THREADS, 0, &occ);
    if (e != cudaSuccess) return e;
    const uint32_t g = max(1u, min(min((uint32_t)(occ * L.num_sms), ws_blocks), ceil_div(n, CS_THREADS)));
    return launch_kernel(L, bt_chunk_unique_kernel, g, CS_THREADS, 0, kin, vin, kout, vout, n, off, S, uoff, ws, bad,
                         L.status);
  }
}

std::atomic<int> g_bt_pinned{-1};  // gtc_batched_set_variant

struct BatchWs {
  uint32_t* tile_start;  // [S + 1]
  uint32_t* ne_start;    // [S + 1]
  uint32_t* tile_cloud;  // [tiles_max]
  uint32_t* seg_hist;    // [S][4][256], cleared per build, as are the next two
  void* unique_ws;
  void* scan_ws;
  size_t zero_vecs;      // 16-byte words from seg_hist on that are cleared
  uint32_t* counters;    // [8] bad batch
  uint32_t* desc;        // [4][tiles_max][256]
  uint32_t* keys_alt;    // [n]
  uint32_t* idx_alt;     // [n]
  uint32_t* ps;          // [n]
  size_t desc_words;
  uint32_t tiles_max;
};

// A cloud of len points has ceil(len / TILE) tiles, so the batch has at most
// n / TILE + S of them, for the smallest tile of any variant.  Room is taken
// for the tiles of up to n points, so the size never shrinks as n grows.
size_t batch_layout(uint32_t n, uint32_t S, BatchWs* W, char* p) {
  const uint32_t tiles_max = bt_tiles(n) + S;
  const uint32_t tiles_room = bt_tiles_up_to(n) + S;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    char* q = p ? p + o : nullptr;
    o += align_up(bytes, 256);
    return q;
  };
  BatchWs w;
  w.tile_start = reinterpret_cast<uint32_t*>(take(((size_t)S + 1) * 4));
  w.ne_start = reinterpret_cast<uint32_t*>(take(((size_t)S + 1) * 4));
  w.tile_cloud = reinterpret_cast<uint32_t*>(take((size_t)tiles_room * 4));
  const size_t zero_from = o;
  w.seg_hist = reinterpret_cast<uint32_t*>(take((size_t)S * BPASSES * BRADIX * 4));
  w.unique_ws = take(scan_workspace_bytes(n));
  w.scan_ws = take(scan_workspace_bytes(n));
  w.zero_vecs = (o - zero_from) / 16;
  w.counters = reinterpret_cast<uint32_t*>(take(256));
  w.desc_words = (size_t)BPASSES * tiles_max * BRADIX;
  w.desc = reinterpret_cast<uint32_t*>(take((size_t)BPASSES * tiles_room * BRADIX * 4));
  w.keys_alt = reinterpret_cast<uint32_t*>(take((size_t)n * 4));
  w.idx_alt = reinterpret_cast<uint32_t*>(take((size_t)n * 4));
  w.ps = reinterpret_cast<uint32_t*>(take((size_t)n * 4));
  w.tiles_max = tiles_max;
  if (W) *W = w;
  return o;
}

}  // namespace
}  // namespace gtc

using namespace gtc;

extern "C" {

GTC_API gtc_status gtc_batched_workspace_size(uint32_t n_total, uint32_t n_clouds, size_t* bytes) {
  if (!bytes || n_clouds == 0 || n_clouds > MAX_CLOUDS || n_total >= (1u << 30)) return GTC_ERR_INVALID_ARG;
  *bytes = batch_layout(n_total, n_clouds, nullptr, nullptr);
  return GTC_OK;
}

}  // extern "C"

namespace gtc {
int batched_select_variant(uint32_t n) {
  const int pinned = g_bt_pinned.load(std::memory_order_relaxed);
  if (pinned >= 0) return pinned;
  const int t = tuned_batched_variant(n);
  if (t >= 0 && t < kBtNumVariants) return t;
  return n <= BT_SMALL_MAX ? BT_SMALL : n >= BT_LARGE_MIN ? BT_LARGE : 0;
}
int batched_num_variants() { return kBtNumVariants; }

// The batched build with the segmented onesweep's tile shape given.
gtc_status build_octree_batched_variant(gtc_ctx* ctx, const float* pts, const uint32_t* d_offsets,
                                        uint32_t n_clouds, uint32_t n_total, float min_coord, float range,
                                        const gtc_batch_buffers* out, void* ws, size_t ws_bytes,
                                        gtc_stream_t stream, int variant) {
  if (!ctx) return GTC_ERR_INVALID_ARG;
  if (variant < 0 || variant >= kBtNumVariants)
    return context_error(ctx, GTC_ERR_INVALID_ARG, "no such batched variant", cudaSuccess);
  if (variant == BT_SMALL && n_total > BT_SMALL_MAX) variant = 0;
  const uint32_t tile = (uint32_t)(kBtVariants[variant].threads * kBtVariants[variant].kpt);
  if (!out || !d_offsets || n_clouds == 0 || n_clouds > MAX_CLOUDS)
    return context_error(ctx, GTC_ERR_INVALID_ARG, "need offsets, outputs and 1..2^20 clouds", cudaSuccess);
  if (n_total >= (1u << 30)) return context_error(ctx, GTC_ERR_INVALID_ARG, "n_total must be < 2^30", cudaSuccess);
  if (n_total > 0 && (!pts || (reinterpret_cast<uintptr_t>(pts) & 15)))
    return context_error(ctx, GTC_ERR_INVALID_ARG, "pts must be a 16-byte aligned float[n][4]", cudaSuccess);
  if (!out->keys || !out->idx || !out->prefix_n || !out->has_leaf_left || !out->has_leaf_right ||
      !out->left_child || !out->parent || !out->edge_count || !out->node_offsets || !out->nodes ||
      !out->key_offset || !out->node_offset || !out->cloud_counts)
    return context_error(ctx, GTC_ERR_INVALID_ARG, "null output buffer", cudaSuccess);
  const size_t need = batch_layout(n_total, n_clouds, nullptr, nullptr);
  if (!ws || ws_bytes < need || (reinterpret_cast<uintptr_t>(ws) & 255))
    return context_error(ctx, GTC_ERR_INVALID_ARG, "batched workspace missing, too small or not 256-byte aligned",
                         cudaSuccess);
  BatchWs W;
  batch_layout(n_total, n_clouds, &W, reinterpret_cast<char*>(ws));
  const Launch L = context_launch(ctx, stream);
  cudaStream_t s = L.stream;
  const uint32_t S = n_clouds;
  cudaError_t e;
#define BCHK(x)                                                                   \
  do {                                                                            \
    if ((e = (x)) != cudaSuccess) return context_error(ctx, GTC_ERR_CUDA, #x, e); \
  } while (0)
  if (n_total == 0) {
    BCHK(cudaMemsetAsync(out->key_offset, 0, ((size_t)S + 1) * 4, s));
    BCHK(cudaMemsetAsync(out->node_offset, 0, ((size_t)S + 1) * 4, s));
    BCHK(cudaMemsetAsync(out->cloud_counts, 0, (size_t)S * 12, s));
    return GTC_OK;
  }
  uint32_t* bad = W.counters + 8;
  // Every kernel after the first starts under a programmatic dependent launch
  // (not while stage events are being recorded between them).
  Launch Lp = L;
  Lp.pdl = context_stage_idle(ctx);
  Lp.ws_zeroed = true;
  {
    Stage t(ctx, stream, GTC_STAGE_MORTON);
    const uint32_t zgrid = (uint32_t)min((W.zero_vecs + 2047) / 2048, (size_t)L.num_sms);
    BCHK(launch_kernel(L, bt_tiles_kernel, 1 + zgrid, 1024, 0, d_offsets, S, n_total, tile, W.tile_start, W.ne_start,
                       W.counters, bad, out->key_offset, reinterpret_cast<uint4*>(W.seg_hist), W.zero_vecs, L.status));
    const float inv = pow2_reciprocal(range);
    auto kern = inv != 0.0f ? bt_morton_kernel<1> : bt_morton_kernel<2>;
    const uint32_t group = W.tiles_max > 16u * (uint32_t)L.num_sms ? 4u : 1u;
    BCHK(launch_kernel(Lp, kern, ceil_div(W.tiles_max, group), BM_THREADS, 0, reinterpret_cast<const float4*>(pts),
                       d_offsets, S, W.tile_start, tile, group, min_coord, range, inv, W.keys_alt, W.tile_cloud,
                       W.seg_hist, reinterpret_cast<uint4*>(W.desc), W.desc_words / 4));
    if (variant == BT_LARGE) BCHK(launch_kernel(Lp, bt_seg_scan_kernel, S, BRADIX, 0, W.seg_hist, d_offsets));
  }
  uint32_t* src_k = W.keys_alt;
  uint32_t* src_v = W.idx_alt;
  uint32_t* dst_k = out->keys;
  uint32_t* dst_v = out->idx;
  for (int p = 0; p < BPASSES; ++p) {
    Stage t(ctx, stream, GTC_STAGE_ONESWEEP);
    BCHK(launch_bt_variant(variant, Lp, W.tiles_max,
                           BtPass{src_k, src_v, dst_k, dst_v, d_offsets, S, W.tile_start, W.tile_cloud, p, W.seg_hist,
                                  W.desc + (size_t)p * W.tiles_max * BRADIX}));
    std::swap(src_k, dst_k);
    std::swap(src_v, dst_v);
  }
  // After 4 passes the sorted pairs are back in the alternate buffers.
  {
    Stage t(ctx, stream, GTC_STAGE_UNIQUE);
    BCHK(launch_bt_unique<2>(Lp, src_k, src_v, out->keys, out->idx, n_total, d_offsets, S, out->key_offset,
                             reinterpret_cast<uint32_t*>(W.unique_ws),
                             (uint32_t)(scan_workspace_bytes(n_total) / 4) - 64, bad));
  }
  // idx_alt is free after unique: the window tree leaves the split records
  // there for the octree.
  uint32_t* rec = tree_get_method() == 1 ? W.idx_alt : nullptr;
  {
    Stage t(ctx, stream, GTC_STAGE_RADIX_TREE);
    if (rec) {
      auto window = [&](auto shape) {
        using SH = decltype(shape);
        return launch_kernel(Lp, radix_tree_window_kernel<uint32_t, true, SH>, ceil_div(n_total, SH::T), TW_THREADS, 0,
                             out->keys, nullptr, 0u, out->key_offset, S, out->prefix_n, out->has_leaf_left,
                             out->has_leaf_right, out->left_child, out->parent, out->edge_count, nullptr, rec);
      };
      BCHK(n_total <= TW_TWO_MAX ? tw_window_two(n_total, window) : window(TwSegLarge{}));
    } else {
      const uint32_t grid = max(1u, min(ceil_div(n_total, 256), (uint32_t)L.num_sms * 8));
      BCHK(launch_kernel(Lp, bt_tree_kernel, grid, 256, 0, out->keys, out->key_offset, S, out->prefix_n,
                         out->has_leaf_left, out->has_leaf_right, out->left_child, out->parent, out->edge_count));
    }
  }
  {
    Stage t(ctx, stream, GTC_STAGE_PREFIX_SUM);
    BCHK(launch_inclusive_scan_dev(Lp, out->edge_count, W.ps, out->key_offset + S, n_total, W.scan_ws));
    // The per-cloud digit histograms are dead after the sort: their space
    // holds the per-cloud octree info.
    BCHK(launch_kernel(Lp, bt_cloud_offsets_kernel, ceil_div(S, 256), 256, 0, out->key_offset, W.ne_start, W.ps, S,
                       out->node_offset, out->cloud_counts, reinterpret_cast<uint4*>(W.seg_hist), bad));
  }
  {
    Stage t(ctx, stream, GTC_STAGE_OCTREE);
    if (rec) {
      BCHK((launch_octree_window<uint32_t, true>(Lp, out->keys, nullptr, out->key_offset, S,
                                                 reinterpret_cast<const uint4*>(W.seg_hist), n_total, rec,
                                                 out->prefix_n, out->has_leaf_left, out->has_leaf_right,
                                                 out->left_child, out->edge_count, W.ps, out->node_offsets, min_coord,
                                                 range, out->nodes, out->nodes_capacity)));
      return GTC_OK;
    }
    int occ = 4;  // resident blocks per SM
    if (kernel_setup(bt_octree_kernel, BT_OCT_THREADS, 0, &occ) != cudaSuccess) {
      cudaGetLastError();
      occ = 4;
    }
    const uint32_t ogrid = max(1u, min(ceil_div(n_total, BT_OCT_THREADS), (uint32_t)(L.num_sms * occ)));
    BCHK(launch_kernel(Lp, bt_octree_kernel, ogrid, BT_OCT_THREADS, 0, out->keys, out->key_offset, S,
                       reinterpret_cast<const uint4*>(W.seg_hist), out->prefix_n, out->has_leaf_left,
                       out->has_leaf_right, out->left_child, out->edge_count, W.ps, out->node_offsets, min_coord, range,
                       out->nodes, out->nodes_capacity, leaf_mask_keep(), L.status));
  }
#undef BCHK
  return GTC_OK;
}
}  // namespace gtc

extern "C" {

GTC_API gtc_status gtc_build_octree_batched(gtc_ctx* ctx, const float* pts, const uint32_t* d_offsets,
                                            uint32_t n_clouds, uint32_t n_total, float min_coord, float range,
                                            const gtc_batch_buffers* out, void* ws, size_t ws_bytes,
                                            gtc_stream_t stream) {
  return build_octree_batched_variant(ctx, pts, d_offsets, n_clouds, n_total, min_coord, range, out, ws, ws_bytes,
                                      stream, batched_select_variant(n_total));
}

GTC_API int gtc_batched_num_variants(void) { return kBtNumVariants; }

GTC_API gtc_status gtc_batched_variant_shape(int variant, int* threads, int* keys_per_thread) {
  if (variant < 0 || variant >= kBtNumVariants) return GTC_ERR_INVALID_ARG;
  if (threads) *threads = kBtVariants[variant].threads;
  if (keys_per_thread) *keys_per_thread = kBtVariants[variant].kpt;
  return GTC_OK;
}

GTC_API gtc_status gtc_batched_set_variant(int variant) {
  if (variant < -1 || variant >= kBtNumVariants) return GTC_ERR_INVALID_ARG;
  g_bt_pinned.store(variant, std::memory_order_relaxed);
  return GTC_OK;
}

GTC_API int gtc_batched_get_variant(uint32_t n_total) { return batched_select_variant(n_total); }

}  // extern "C"
