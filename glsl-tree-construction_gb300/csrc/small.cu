// small.cu - the whole build of a small cloud, and the whole sort of few keys,
// in one block.
//
// The stage kernels (morton.comp .. octree.comp, main.rs:60-170) each cost a
// launch and a chain of dependent global round trips however few points there
// are: eleven kernels, about 5 us each, for 4,096 points.  Up to
// SMALL_BUILD_MAX points one block holds the cloud in shared memory and does every
// stage there: Morton codes, stable LSD sort, unique, Karras tree, edge
// counts, node offsets and octree nodes, with the same outputs as the stage
// kernels.  One SM's issue rate bounds it (the sort's ranking above all), so
// its time grows with n where the stage kernels' does not yet.
// Per build, launched back to back (us):
//   points        32-bit: stages  one block     64-bit: stages  one block
//      256                  44         10                 52         11
//    1,024                  48         16                 56         17
//    4,096                  50         31                 63         35
// (The one block has no faster form at 8,192: its sort alone takes longer
// there than the stage kernels' passes.)
//
// The radix tree is kept by split (tree_window.cuh): split x has a parent
// split, an edge count and a Karras index.  The octree is pushed from the
// children: a leaf, or a split that owns octree nodes, walks up past splits
// of the same depth (at most two) to the split that owns its parent node and
// stores itself in that node's row of child slots in shared memory.

#include "octree_dev.cuh"
#include "scan_dev.cuh"
#include "tree_window.cuh"

namespace gtc {

constexpr int SB_HROW = 257;   // digit counters of one warp, padded so that a digit's counters of all warps
                               // fall in different banks
constexpr int SB_ROW = 5;      // words of a node's child slots (eight 16-bit slots), padded likewise
constexpr int SB_RUN = 16;     // longest run of equal high bits that one thread sorts
constexpr uint16_t SB_PRESENT = 1u << 15, SB_LEAF = 1u << 14, SB_ID = SB_LEAF - 1u;

template <class K, int THREADS_, int MAX_>
struct SbSmem {
  static constexpr int THREADS = THREADS_;
  static constexpr int WARPS = THREADS / 32;
  static constexpr int MAX = MAX_;
  static constexpr int KPT = MAX / THREADS;  // items per thread of the largest cloud
  using Shape = TwShape<MAX, 512, 1>;
  static_assert(THREADS % 256 == 0 && MAX % THREADS == 0, "whole digits and items per thread");
  static_assert(MAX <= 1 << 13, "a child's index and two flags fit 16 bits");
  K keys[MAX];
  union {
    struct {  // sort and unique
      uint32_t hist[WARPS][SB_HROW];
      uint16_t idx[MAX];
    };
    struct {  // from the node offsets on
      uint32_t ps[MAX];
      uint16_t crank[MAX];  // by split: rank among the splits that own octree nodes
    };
  };
  union {
    struct {  // by Karras index: the tree's output arrays
      uint16_t left[MAX];    // left child | left leaf << 14 | right leaf << 15
      uint16_t parent[MAX];
      uint8_t prefix[MAX];
      uint8_t edge[MAX];
    };
    uint32_t row[MAX][SB_ROW];  // child slots of the octree's branching nodes, by rank
  };
  uint16_t par[MAX];    // by split: parent split
  uint16_t kidx[MAX];   // by split: Karras index
  uint16_t owner[MAX];  // by rank: the split
  uint8_t cnt[MAX];     // by split: octree nodes owned (the root split owns its one beside these)
  TwSmem<Shape> tw;
  uint32_t wsum[2][WARPS];
  uint32_t root;
};

// Exclusive scan of one value per thread with one barrier (every warp scans
// the warp totals itself).  Consecutive calls alternate buf.
template <int WARPS>
__device__ __forceinline__ uint32_t sb_scan(uint32_t v, uint32_t (*wsum)[WARPS], int buf, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t incl = warp_inclusive_sum(v);
  if (lane == 31) wsum[buf][warp] = incl;
  __syncthreads();
  const uint32_t w = lane < WARPS ? wsum[buf][lane] : 0u;
  const uint32_t wi = warp_inclusive_sum(w);
  *total = __shfl_sync(0xffffffffu, wi, 31);
  return __shfl_sync(0xffffffffu, wi - w, warp) + incl - v;
}

// One stable 8-bit pass over the kpt * THREADS keys in shared memory (warp w
// holds keys [32 w kpt, 32 (w + 1) kpt) in rows of 32, so that rank order is
// position order).  Starts and ends with every thread past a barrier.
template <class S, class K>
__device__ __forceinline__ void sb_pass(S& s, int kpt, int shift, K*, uint32_t dmask = 255u) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t* my = s.hist[warp];
#pragma unroll
  for (int i = 0; i < 8; ++i) my[i * 32 + lane] = 0;
  K key[S::KPT];
  uint16_t val[S::KPT];
  uint32_t rank[S::KPT];
  const int base0 = warp * 32 * kpt + lane;
#pragma unroll
  for (int j = 0; j < S::KPT; ++j) {
    if (j < kpt) {
      key[j] = s.keys[base0 + j * 32];
      val[j] = s.idx[base0 + j * 32];
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < S::KPT; ++j) {
    if (j < kpt) {  // block-uniform
      const uint32_t d = (uint32_t)(key[j] >> shift) & dmask;
      const uint32_t peers = warp_peers<8>(d);
      const int leader = 31 - __clz(peers);
      uint32_t b = 0;
      if (lane == leader) b = atomicAdd(&my[d], (uint32_t)__popc(peers));
      b = __shfl_sync(0xffffffffu, b, leader);
      rank[j] = (b + __popc(peers & lt)) | (d << 16);
    }
  }
  __syncthreads();
  // Counts to positions, digit-major: THREADS / 256 threads per digit, eight
  // warps' counters each.
  {
    constexpr int TPD = S::THREADS / 256;
    const int d = tid / TPD, w0 = (tid % TPD) * 8;
    uint32_t c[8], sum = 0, total;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      c[w] = s.hist[w0 + w][d];
      sum += c[w];
    }
    uint32_t b = sb_scan<S::WARPS>(sum, s.wsum, 0, &total);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      s.hist[w0 + w][d] = b;
      b += c[w];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < S::KPT; ++j) {
    if (j < kpt) {
      const uint32_t pos = my[rank[j] >> 16] + (rank[j] & 0xffffu);
      s.keys[pos] = key[j];
      s.idx[pos] = val[j];
    }
  }
  __syncthreads();
}

template <class K>
__device__ __forceinline__ int sb_depth(uint32_t prefix) {
  return ((int)prefix - KeyTraits<K>::A) / 3;
}

template <class K, int THREADS, int MAX>
__global__ void __launch_bounds__(THREADS, 1) small_build_kernel(const float4* __restrict__ pts, uint32_t n, float mn,
                                                                 float rg, float inv_rg, gtc_octree_buffers out,
                                                                 uint32_t lmask_keep, uint32_t* status) {
  using S = SbSmem<K, THREADS, MAX>;
  using SH = typename S::Shape;
  constexpr int B = KeyTraits<K>::B;
  constexpr int KPT = S::KPT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S& s = *reinterpret_cast<S*>(smem_raw);
  K* const tag = nullptr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const int kpt = (int)((n + THREADS - 1) / THREADS);
  const int base0 = warp * 32 * kpt + lane;  // this lane's items: base0 + 32 j, j < kpt

  // 1. codes; padding past n sorts last (it starts last and has the largest digits).
  {
    float4 p[KPT];
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
      const int i = base0 + j * 32;
      p[j] = j < kpt && i < (int)n ? __ldcs(pts + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
      const int i = base0 + j * 32;
      if (j < kpt) {
        s.keys[i] = i < (int)n ? encode_point<K>(p[j], mn, rg, inv_rg) : ~K(0);
        s.idx[i] = (uint16_t)i;
      }
    }
  }
  __syncthreads();

  // 2. stable sort.  64-bit codes: the top 32 of the 63 bits first, then runs
  // that agree in them, as the large build does (run_fixup_kernel); if a run
  // is too long for one thread, eight passes over the whole code.  (The high
  // passes kept equal codes in index order, so the result is the same.)
  constexpr int LOW = sizeof(K) == 8 ? 3 * B - 32 : 0;
  for (int sh = LOW; sh < 3 * B; sh += 8) sb_pass(s, kpt, sh, tag);
  if (LOW) {
    uint32_t run[KPT];  // length of the run that starts at item j, 0 if none of two or more does
    bool too_long = false;
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
      run[j] = 0;
      const int i = base0 + j * 32;
      if (j < kpt && i + 1 < (int)n) {
        const K h = s.keys[i] >> LOW;
        if ((s.keys[i + 1] >> LOW) == h && (i == 0 || (s.keys[i - 1] >> LOW) != h)) {
          int g = 2;
          while (g <= SB_RUN && i + g < (int)n && (s.keys[i + g] >> LOW) == h) ++g;
          run[j] = (uint32_t)g;
          too_long |= g > SB_RUN;
        }
      }
    }
    if (__syncthreads_or(too_long)) {
      for (int sh = 0; sh < 3 * B; sh += 8) sb_pass(s, kpt, sh, tag);
    } else {
#pragma unroll
      for (int j = 0; j < KPT; ++j) {
        const int i = base0 + j * 32;
        for (int a = 1; a < (int)run[j]; ++a) {  // stable insertion
          const K k = s.keys[i + a];
          const uint16_t v = s.idx[i + a];
          int b = a;
          while (b > 0 && s.keys[i + b - 1] > k) {
            s.keys[i + b] = s.keys[i + b - 1];
            s.idx[i + b] = s.idx[i + b - 1];
            --b;
          }
          s.keys[i + b] = k;
          s.idx[i + b] = v;
        }
      }
      __syncthreads();
    }
  }

  // 3. unique: the first of each run of equal codes and its index.
  uint32_t u;
  {
    K key[KPT];
    uint32_t keep[KPT], kept = 0;  // ballots
    uint16_t val[KPT];
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
      keep[j] = 0;
      if (j < kpt) {
        const int i = base0 + j * 32;
        key[j] = s.keys[i];
        val[j] = s.idx[i];
        keep[j] = __ballot_sync(0xffffffffu, i < (int)n && (i == 0 || s.keys[i - 1] != key[j]));
        kept += __popc(keep[j]);
      }
    }
    // Past this scan's barrier everyone has read its keys.
    uint32_t at = sb_scan<S::WARPS>(lane == 0 ? kept : 0u, s.wsum, 1, &u);
    at = __shfl_sync(0xffffffffu, at, 0);
    K* gkeys = reinterpret_cast<K*>(out.keys);
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
      if ((keep[j] >> lane) & 1u) {
        const uint32_t o = at + __popc(keep[j] & lt);
        s.keys[o] = key[j];
        gkeys[o] = key[j];
        out.idx[o] = val[j];
      }
      at += __popc(keep[j]);
    }
  }
  const uint32_t m = u - 1;
  if (tid == 0) {
    out.counts[0] = u;
    out.counts[1] = m;
    out.counts[3] = 0;
  }
  if (m == 0) {  // D18: one distinct code
    if (tid == 0) {
      out.counts[2] = 1;
      out.node_offsets[0] = 0;
      octree_root_only<K>(out.nodes, out.nodes_capacity, mn, rg, status);
    }
    return;
  }
  __syncthreads();

  // 4. prefix lengths of adjacent codes with boundaries (0) before the first
  // and after the last, and the nearest-smaller tables over the warp-blocks
  // in use (tree_window.cuh; the window holds the whole cloud, so every
  // answer is in it).
  auto& T = s.tw;
  const int nwb = (SH::H + (int)m) / 512 + 1;  // warp-blocks holding positions 0 .. H + m
  for (int p = tid; p < nwb * 512; p += THREADS) {
    const int x = p - SH::H;
    T.d[p] = (x >= 0 && x < (int)m) ? (uint8_t)delta_key(s.keys[x], s.keys[x + 1]) : (uint8_t)0;
  }
  __syncthreads();
  for (int c = tid; c < nwb * 32; c += THREADS) T.cmin[c] = (uint8_t)tw_chunk_min(T.d + c * TW_C);
  for (int c = tid; c * TW_C < (int)m; c += THREADS) tw_chunk_stack(T, c);
  __syncthreads();
  for (int b = warp; b < nwb; b += S::WARPS) tw_table4(T, b);
  if (warp == S::WARPS - 1) tw_table9(T, nwb);
  __syncthreads();

  // 5. every split's node.
  for (int x = tid; x < (int)m; x += THREADS) {
    const int xi = x + SH::H, chunk = xi / TW_C, cstart = chunk * TW_C;
    const uint32_t lr = T.lr[x];
    const uint32_t t = T.d[xi];
    const int r = ((lr & 15) ? cstart + (int)(lr & 15) : tw_next_tab(T, chunk, t));
    const int l = ((lr >> 4) != 15 ? cstart + (int)(lr >> 4) : tw_prev_tab(T, chunk, t));
    const uint32_t dR = T.d[r], dL = T.d[l];
    const int hi = r - SH::H, lo = l - SH::H + 1;
    uint32_t k = 0, e = 0, p = 0;
    if (dL == 0 && dR == 0) {
      s.root = (uint32_t)x;
      s.parent[0] = 0;  // D13
    } else {
      k = (uint32_t)(dR > dL ? hi : lo);
      p = (uint32_t)(dR > dL ? hi : lo - 1);
      e = (uint32_t)(sb_depth<K>(t) - sb_depth<K>(max(dL, dR)));
    }
    s.par[x] = (uint16_t)p;
    s.kidx[x] = (uint16_t)k;
    s.cnt[x] = (uint8_t)e;
    s.left[k] = (uint16_t)(x | (lo == x ? 1 << 14 : 0) | (hi == x + 1 ? 1 << 15 : 0));
    s.prefix[k] = (uint8_t)t;
    s.edge[k] = (uint8_t)e;
    if (lo != x) s.parent[x] = (uint16_t)k;
    if (hi != x + 1) s.parent[x + 1] = (uint16_t)k;
  }
  __syncthreads();

  // 6. the tree's arrays, the node offsets (D3, D4) and the ranks of the
  // splits that own octree nodes.
  for (int k = tid; k < (int)m; k += THREADS) {
    const uint32_t l = s.left[k];
    out.prefix_n[k] = s.prefix[k];
    out.has_leaf_left[k] = (uint8_t)((l >> 14) & 1u);
    out.has_leaf_right[k] = (uint8_t)(l >> 15);
    out.left_child[k] = (int32_t)(l & 0x3fffu);
    out.parent[k] = (int32_t)s.parent[k];
    out.edge_count[k] = s.edge[k];
  }
  const uint32_t root = s.root;
  uint32_t owners;
  {
    // Both scans in one: edge counts below (a cloud owns < 2^18 octree nodes
    // beside its root), owners above.
    const int first = tid * kpt;
    uint32_t sum = 0, own = 0, total, total_own;
    for (int j = 0; j < kpt; ++j) {
      const int k = first + j;
      if (k < (int)m) {
        sum += s.edge[k];
        own += (s.cnt[k] > 0 || k == (int)root) ? 1u : 0u;
      }
    }
    uint32_t at = sb_scan<S::WARPS>(sum, s.wsum, 0, &total);
    uint32_t rk = sb_scan<S::WARPS>(own, s.wsum, 1, &total_own);
    owners = total_own;
    for (int j = 0; j < kpt; ++j) {
      const int k = first + j;
      if (k < (int)u) {
        if (k < (int)m) {
          at += s.edge[k];
          if (s.cnt[k] > 0 || k == (int)root) {
            s.owner[rk] = (uint16_t)k;
            s.crank[k] = (uint16_t)rk;
            ++rk;
          }
        }
        s.ps[k] = at;
      }
    }
    if (tid == 0) out.counts[2] = 1 + total;
  }
  __syncthreads();  // the output arrays are read: their space becomes the child rows
  for (int k = tid; k < (int)u; k += THREADS) out.node_offsets[k] = s.ps[k];
  for (uint32_t i = tid; i < owners * SB_ROW; i += THREADS) (&s.row[0][0])[i] = 0;
  __syncthreads();

  // 7. children: leaf x, and split x if it owns nodes, each into the row of
  // the split that owns its parent node (splits of the same depth between
  // them own nothing: at most two steps).
  for (int x = tid; x < (int)u; x += THREADS) {
    const uint32_t dl = T.d[SH::H + x - 1], dr = T.d[SH::H + x];
    const K code = s.keys[x];
    uint32_t p = (uint32_t)(dl > dr ? x - 1 : x);
    while (s.cnt[p] == 0 && p != root) p = s.par[p];
    reinterpret_cast<uint16_t*>(s.row[s.crank[p]])[child_slot<K>(code, sb_depth<K>(max(dl, dr)) + 1)] =
        (uint16_t)(x | SB_PRESENT | SB_LEAF);
    if (x < (int)m && s.cnt[x] != 0 && x != (int)root) {
      p = s.par[x];
      const uint32_t lev = (uint32_t)sb_depth<K>(T.d[SH::H + p]) + 1;
      while (s.cnt[p] == 0 && p != root) p = s.par[p];
      reinterpret_cast<uint16_t*>(s.row[s.crank[p]])[child_slot<K>(code, (int)lev)] = (uint16_t)(x | SB_PRESENT);
    }
  }
  __syncthreads();

  // 8. octree nodes: an owner's branching node, then the chain above it.
  const int root_level = sb_depth<K>(T.d[SH::H + root]);
  for (uint32_t o = tid; o < owners; o += THREADS) {
    const uint32_t x = s.owner[o];
    const uint32_t c = x == root ? 0u : s.cnt[x];
    const uint32_t top = x == root ? 0u : s.ps[s.kidx[x]];
    if (top >= out.nodes_capacity) {
      atomicOr(status, DEV_CAPACITY);
      continue;
    }
    uint32_t cv[8], nmask = 0, lmask = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const uint32_t v = (s.row[o][w >> 1] >> (16 * (w & 1))) & 0xffffu;
      const uint32_t id = v & SB_ID;
      cv[w] = id;
      if (v & SB_LEAF) lmask |= 1u << w;
      else if (v) {
        nmask |= 1u << w;
        cv[w] = s.ps[s.kidx[id]];
      }
    }
    lmask &= lmask_keep;
    const K code = s.keys[x];
    const int dk = sb_depth<K>(T.d[SH::H + x]);
    const uint32_t bottom = x == root ? 0u : top - c + 1;
    const uint3 qc = code_xyz<K>(code);
    store_node(out.nodes, bottom, make_int4((int)cv[0], (int)cv[1], (int)cv[2], (int)cv[3]),
               make_int4((int)cv[4], (int)cv[5], (int)cv[6], (int)cv[7]), corner_at<K>(qc, dk, mn, rg),
               __fmul_rn(rg, exp2_neg(dk - root_level)), (int32_t)nmask, (int32_t)lmask);
    for (uint32_t j = 1; j < c; ++j) {
      const int lv = dk - (int)j;
      int4 ca = make_int4(0, 0, 0, 0), cb = make_int4(0, 0, 0, 0);
      const int w = child_slot<K>(code, lv + 1);
      set_child(ca, cb, w, (int32_t)(bottom + j - 1));
      store_node(out.nodes, bottom + j, ca, cb, corner_at<K>(qc, lv, mn, rg), __fmul_rn(rg, exp2_neg(lv - root_level)),
                 1 << w, 0);
    }
  }
}

// ------------------------------------------------------- sort of few keys --
// The sort API's whole sort of at most SMALL_SORT_MAX keys in one launch of
// one block: the build's passes over bits [begin_bit, end_bit) on positions,
// then the values by position.  (The passes of sort.cu are a memset, a
// histogram and a launch per digit.)  Back to back, uniform pairs (us):
//   pairs    u32: passes  one block    u64: passes  one block
//   100           38.0        7.9           66.7        7.7
//   512           33.9        7.6           74.8        8.3
//   1,024         34.7        8.1           74.9       14.4
//   4,096         42.2       14.4           76.9       25.6
// (The passes as they were before the one-wave kernel; they take 21.5 and 34.8
// at 4,097 now.)
template <class K, int THREADS_, int MAX_>
struct SsSmem {
  static constexpr int THREADS = THREADS_;
  static constexpr int WARPS = THREADS / 32;
  static constexpr int KPT = MAX_ / THREADS;
  K keys[MAX_];
  uint32_t vals[MAX_];
  uint32_t hist[WARPS][SB_HROW];
  uint16_t idx[MAX_];
  uint32_t wsum[2][WARPS];
};

template <class K, int THREADS, int MAX>
__global__ void __launch_bounds__(THREADS, 1) small_sort_kernel(K* keys, uint32_t* vals, uint32_t n, int begin_bit,
                                                                int end_bit) {
  using S = SsSmem<K, THREADS, MAX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S& s = *reinterpret_cast<S*>(smem_raw);
  K* const tag = nullptr;
  const int tid = threadIdx.x;
  const int kpt = (int)((n + THREADS - 1) / THREADS);
#pragma unroll
  for (int j = 0; j < S::KPT; ++j) {
    const int i = j * THREADS + tid;
    if (j < kpt) {
      s.keys[i] = i < (int)n ? keys[i] : ~K(0);  // padding sorts last: it starts last and has the largest digits
      s.vals[i] = vals && i < (int)n ? vals[i] : 0u;
      s.idx[i] = (uint16_t)i;
    }
  }
  __syncthreads();
  for (int sh = begin_bit; sh < end_bit; sh += 8)
    sb_pass(s, kpt, sh, tag, end_bit - sh < 8 ? (1u << (end_bit - sh)) - 1u : 255u);
#pragma unroll
  for (int j = 0; j < S::KPT; ++j) {
    const int i = j * THREADS + tid;
    if (i < (int)n) {
      keys[i] = s.keys[i];
      if (vals) vals[i] = s.vals[s.idx[i]];
    }
  }
}

template <class K>
cudaError_t launch_small_sort(const Launch& L, K* keys, uint32_t* vals, uint32_t n, int begin_bit, int end_bit) {
  if (n == 0 || n > SMALL_SORT_MAX) return cudaErrorInvalidValue;
  auto run = [&](auto kern, int threads, size_t smem) {
    cudaError_t e = kernel_setup(kern, threads, smem);
    return e != cudaSuccess ? e : launch_kernel(L, kern, 1, threads, smem, keys, vals, n, begin_bit, end_bit);
  };
  if (n <= 512) return run(small_sort_kernel<K, 256, 512>, 256, sizeof(SsSmem<K, 256, 512>));
  return run(small_sort_kernel<K, 1024, (int)SMALL_SORT_MAX>, 1024, sizeof(SsSmem<K, 1024, (int)SMALL_SORT_MAX>));
}
template cudaError_t launch_small_sort<uint32_t>(const Launch&, uint32_t*, uint32_t*, uint32_t, int, int);
template cudaError_t launch_small_sort<uint64_t>(const Launch&, uint64_t*, uint32_t*, uint32_t, int, int);

template <class K, int THREADS, int MAX>
static cudaError_t launch_small(const Launch& L, const float4* pts, uint32_t n, float mn, float rg,
                                const gtc_octree_buffers& out) {
  using S = SbSmem<K, THREADS, MAX>;
  static_assert(sizeof(S) <= 227 * 1024, "one block's shared memory");
  auto kern = small_build_kernel<K, THREADS, MAX>;
  cudaError_t e = kernel_setup(kern, THREADS, sizeof(S));
  if (e != cudaSuccess) return e;
  return launch_kernel(L, kern, 1, THREADS, sizeof(S), pts, n, mn, rg, pow2_reciprocal(rg), out, leaf_mask_keep(),
                       L.status);
}

template <class K>
cudaError_t launch_small_build(const Launch& L, const float4* pts, uint32_t n, float mn, float rg,
                               const gtc_octree_buffers& out) {
  if (n == 0 || n > SMALL_BUILD_MAX) return cudaErrorInvalidValue;
  // Eight warps pay less at every barrier, thirty-two hide more: 12.6 against
  // 16.4 us at 256 points, 20.5 against 18.5 at 1,024.
  if (n <= 512) return launch_small<K, 256, 512>(L, pts, n, mn, rg, out);
  return launch_small<K, 1024, (int)SMALL_BUILD_MAX>(L, pts, n, mn, rg, out);
}
template cudaError_t launch_small_build<uint32_t>(const Launch&, const float4*, uint32_t, float, float,
                                                  const gtc_octree_buffers&);
template cudaError_t launch_small_build<uint64_t>(const Launch&, const float4*, uint32_t, float, float,
                                                  const gtc_octree_buffers&);

}  // namespace gtc
