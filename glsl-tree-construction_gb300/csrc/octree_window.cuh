// octree_window.cuh - octree nodes of a window of splits, pushed from the
// children (single cloud and batched clouds).
//
// octree_dev.cuh gathers a node's children by descending from its radix node:
// dependent gathers over the whole tree, about 450 thread instructions per
// radix node.  Here a child finds its parent instead, as the reference's walk
// does (octree.comp:126-222), but inside a block's window of the split-ordered
// tree, where the walk is a few shared-memory reads: the tree kernel leaves a
// record per split (SplitRec: key range, depth, octree nodes owned), a block
// loads the records of its T splits and H more on each side, and every leaf,
// and every split that owns octree nodes, walks up past splits of its own
// depth (at most two) to the split that owns its parent node and stores itself
// in that owner's row of child slots.  An owner whose key range lies inside
// the window has all its children there, and is written from its row; the
// others (two or three per block of the 10M clustered cloud) are gathered by
// octree_warp_batch in a warp of their own meanwhile.
//
// Instruction issue bounds it (ncu, 4M clustered points: 0.65 of the issue
// slots used, 25% of DRAM), so the pushes take no branches, owners and chain
// nodes are compacted to full warps, and child slots are 16-bit positions.
// Whole builds, gathering every owner -> this (us):
//   10M clustered, 64-bit codes            753 ->   726
//   1M uniform, 32-bit codes               124 ->   123
//   512 clouds, 74M points                4302 ->  3663
// Blocks of 512 threads at three per SM (40 registers): two or four per SM
// 727 and 728, 3775 and 3647.
#pragma once

#include "octree_dev.cuh"
#include "scan_dev.cuh"
#include "split_rec.cuh"
#include "tree_window.cuh"

namespace gtc {

constexpr int OW_THREADS = 480;       // workers; one more warp gathers the owners that reach past the window
constexpr int OW_WARPS = OW_THREADS / 32;
constexpr int OW_PER = 5;             // window positions per worker
constexpr int OW_W = OW_PER * OW_THREADS;
constexpr int OW_H = 256;             // halo on each side
constexpr int OW_T = OW_W - 2 * OW_H; // splits per block
constexpr int OW_ROWS = 1024;         // owners assembled at a time (on average 45% of the splits own nodes)
constexpr int OW_ROW = 5;             // words of an owner's eight 16-bit child slots, padded against bank conflicts
constexpr uint32_t OW_PRESENT = 1u << 15, OW_LEAF = 1u << 14, OW_ID = OW_LEAF - 1u;
// Owners not assembled here hold a key range that reaches past the window or
// past SPLIT_FAR positions on one side, so they are ancestors of a key at the
// window's edges or at one of the multiples of SPLIT_FAR inside it: at most
// four root paths of fewer than 64 splits.
constexpr int OW_LONG = 256;
constexpr int OW_CHAIN = 1024;        // chain nodes listed per round (more are written by their owner's lane)
static_assert(OW_ROWS <= 2048, "a row and a chain position fit 16 bits");
static_assert(OW_H % 32 == 0 && OW_T % 32 == 0, "whole warps in the core");
static_assert(OW_W <= 3 * SPLIT_FAR, "at most four root paths hold the long owners");

template <class K>
struct OwSmem {
  K code[OW_W + 1];
  uint32_t rec[OW_W + 1];      // one more: the position of every walk that leaves the window
  uint32_t ps[OW_W];
  uint16_t row_of[OW_W + 1];   // row rank of a core owner inside the window, else 0xffff
  uint16_t own[OW_T];          // by rank: window position of the owner
  uint32_t row[OW_ROWS + 1][OW_ROW];  // one more: takes what belongs to no row of this round
  OctWarp fb;
  uint32_t longk[OW_LONG];   // Karras indices of the other owners
  uint32_t wsum[OW_WARPS];
  uint16_t chain[OW_CHAIN];  // chain nodes to write: owner's row | position above the bottom << 11
  uint32_t long_n, chain_n, c_first, c_end;
};

// The octree node at `slot` whose one child is `child`, at level lv of code.
template <class K>
__device__ __forceinline__ void ow_chain_node(gtc_octnode* nodes, uint32_t slot, uint32_t child, K code, int lv,
                                              int root_level, float mn, float rg) {
  int4 ca = make_int4(0, 0, 0, 0), cb = make_int4(0, 0, 0, 0);
  const int w = child_slot<K>(code, lv + 1);
  set_child(ca, cb, w, (int32_t)child);
  store_node(nodes, slot, ca, cb, corner_at<K>(code_xyz<K>(code), lv, mn, rg),
             __fmul_rn(rg, exp2_neg(lv - root_level)), 1 << w, 0);
}

__device__ __forceinline__ void ow_sync() { asm volatile("bar.sync 1, 480;" ::: "memory"); }  // the workers

// One cloud of codes [0, u), or with SEG many: cloud c is [uoff[c], uoff[c + 1])
// with its octree at cinfo[c] = {U0, U1, bias, first node}, and its node
// offsets (ps minus the bias) are written here.
template <class K, bool SEG>
__global__ void __launch_bounds__(OW_THREADS + 32, 3) octree_window_kernel(
    const K* codes, const uint32_t* d_u, const uint32_t* uoff, uint32_t S,
    const uint4* cinfo, const uint32_t* rec, const uint8_t* prefix_n,
    const uint8_t* hll, const uint8_t* hlr, const int32_t* left,
    const uint32_t* edge, const uint32_t* ps, uint32_t* __restrict__ node_offsets, float mn,
    float rg, gtc_octnode* __restrict__ nodes, uint32_t capacity, uint32_t lmask_keep, uint32_t* status) {
  griddep_wait();
  constexpr int A = KeyTraits<K>::A;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Sm = OwSmem<K>;
  Sm& s = *reinterpret_cast<Sm*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t U = SEG ? uoff[S] : *d_u;
  const int m = (int)U - 1;  // SEG: splits at a cloud's last key carry SPLIT_NONE
  if (!SEG && m == 0) {
    if (blockIdx.x == 0 && tid == 0) octree_root_only<K>(nodes, capacity, mn, rg, status);
    return;
  }
  const int t0 = (int)blockIdx.x * OW_T;
  if (t0 >= (SEG ? (int)U : m)) return;
  const int w0 = t0 - OW_H;
  if (tid == 0) s.long_n = s.chain_n = 0;
  __syncthreads();

  if (warp == OW_WARPS) {
    // The gathering warp: the block's clouds (SEG), then the owners that
    // reach past the window, while the workers assemble the others.
    if (SEG) {
      const uint32_t a = warp_upper_bound_u32(uoff, S + 1, (uint32_t)t0) - 1;
      const uint32_t b = warp_upper_bound_u32(uoff, S + 1, (uint32_t)min(t0 + OW_T - 1, (int)U - 1));
      if (lane == 0) {
        s.c_first = a;
        s.c_end = b;
      }
    }
    __syncthreads();
    const uint32_t nl = min(s.long_n, (uint32_t)OW_LONG);
    for (uint32_t e0 = 0; e0 < nl; e0 += 32) {  // warp-uniform
      const bool have = e0 + lane < nl;
      const uint32_t k = have ? s.longk[e0 + lane] : 0u;
      OctCloud cl{0u, (uint32_t)m, 0u, 0, nodes, capacity};
      bool ok = have;
      if (have) {
        if (SEG) {  // k may lie in a neighbour block's core: search all clouds
          const uint4 ci = cinfo[owner(uoff, S, k)];
          cl.u0 = ci.x;
          cl.mend = ci.y - 1;
          cl.bias = ci.z;
          if (ci.w >= capacity) {
            atomicOr(status, DEV_CAPACITY);
            ok = false;
          } else {
            cl.nodes = nodes + ci.w;
            cl.capacity = capacity - ci.w;
          }
        }
        cl.root_level = ((int)prefix_n[cl.u0] - A) / 3;
        ok = ok && (k == cl.u0 || edge[k] > 0);
      }
      octree_warp_batch<K, true>(s.fb, ok, k, cl, codes, prefix_n, hll, hlr, left, edge, ps, mn, rg, lmask_keep,
                                 status);
    }
    return;
  }

  // 1. records, offsets and codes of the window (a warp's 32 positions lie
  // all in the core or all outside it), and the owners of the core: a row for
  // those inside the window, the list for the others.
  uint32_t mask[OW_PER], mine = 0;  // ballots of the owners with a row
  {
    uint32_t r[OW_PER], pv[OW_PER];
    K cx[OW_PER];
    if (w0 >= 0 && w0 + OW_W < (int)U - 1) {  // block-uniform: every position holds a key and a split
#pragma unroll
      for (int q = 0; q < OW_PER; ++q) {
        const uint32_t x = (uint32_t)(w0 + q * OW_THREADS + tid);
        r[q] = rec[x];
        pv[q] = ps[x];
        cx[q] = codes[x];
      }
    } else {
#pragma unroll
      for (int q = 0; q < OW_PER; ++q) {
        const int x = w0 + q * OW_THREADS + tid;
        const bool in = x >= 0 && x < (int)U;
        r[q] = in && (SEG || x < m) ? rec[x] : SPLIT_NONE;
        pv[q] = in ? ps[x] : 0u;
        cx[q] = in ? codes[x] : K(0);
      }
    }
    if (tid == 0) {
      s.rec[OW_W] = SPLIT_NONE;
      s.row_of[OW_W] = 0xffffu;
      if (w0 + OW_W < (int)U) s.code[OW_W] = codes[w0 + OW_W];  // the last position's next key
    }
#pragma unroll
    for (int q = 0; q < OW_PER; ++q) {
      const int i = q * OW_THREADS + tid;
      s.rec[i] = r[q];
      s.ps[i] = pv[q];
      s.code[i] = cx[q];
      bool in = false;
      if (i >= OW_H && i < OW_H + OW_T) {  // warp-uniform
        const bool near_in = !split_far(r[q]) && i - split_lo(r[q]) >= 0 && i + split_hi(r[q]) < OW_W;
        const bool owns = split_far(r[q]) ? r[q] != SPLIT_NONE : split_owned(r[q]) != 0;
        in = owns && near_in;
        if (owns && !near_in) {
          const uint32_t at = atomicAdd(&s.long_n, 1u);
          if (at < (uint32_t)OW_LONG)
            s.longk[at] = split_far(r[q]) ? r[q] & ~SPLIT_FAR_FLAG : (uint32_t)(w0 + i + split_kidx(r[q]));
          else
            atomicOr(status, DEV_INTERNAL);  // cannot happen on valid input
        }
      }
      mask[q] = __ballot_sync(0xffffffffu, in);
      mine += __popc(mask[q]);
    }
  }
  if (lane == 0) s.wsum[warp] = mine;
  __syncthreads();
  uint32_t owners, at;
  {
    const uint32_t w = lane < OW_WARPS ? s.wsum[lane] : 0u;
    const uint32_t wi = warp_inclusive_sum(w);
    owners = __shfl_sync(0xffffffffu, wi, 31);
    at = __shfl_sync(0xffffffffu, wi - w, warp);
  }
#pragma unroll
  for (int q = 0; q < OW_PER; ++q) {
    const int i = q * OW_THREADS + tid;
    const bool in = (mask[q] >> lane) & 1u;
    const uint32_t rank = at + __popc(mask[q] & lt);
    s.row_of[i] = in ? (uint16_t)rank : (uint16_t)0xffffu;
    if (in) s.own[rank] = (uint16_t)i;
    at += __popc(mask[q]);
  }

  // The cloud of core position x (SEG): the last one starting at or before it.
  auto cloud_of = [&](uint32_t x) -> uint32_t {
    uint32_t lo = s.c_first, hi = s.c_end;  // the first start past x is in (lo, hi]
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (uoff[mid] <= x) lo = mid;
      else hi = mid;
    }
    return lo;
  };
  // 2. node offsets (SEG), and the roots of single-code clouds (D18).
  if (SEG) {
#pragma unroll
    for (int q = 0; q < OW_PER; ++q) {
      const int i = q * OW_THREADS + tid;
      const uint32_t g = (uint32_t)(w0 + i);
      if (i >= OW_H && i < OW_H + OW_T && g < U) {
        const uint4 ci = cinfo[cloud_of(g)];
        node_offsets[g] = g == ci.x ? 0u : s.ps[i] - ci.z;
        if (ci.y - ci.x == 1) {
          if (ci.w < capacity) octree_root_only<K>(nodes + ci.w, capacity - ci.w, mn, rg, status);
          else atomicOr(status, DEV_CAPACITY);
        }
      }
    }
  }

  for (uint32_t r0 = 0; r0 < owners; r0 += OW_ROWS) {  // mostly once
    const uint32_t nrow = min((uint32_t)OW_ROWS, owners - r0);
    for (uint32_t i = tid; i < nrow * OW_ROW; i += OW_THREADS) (&s.row[0][0])[i] = 0;
    ow_sync();
    // 3. children push themselves: branch-free but for the stores, since some
    // lane of a warp takes every path.
    for (int i = tid; i < OW_W; i += OW_THREADS) {
      const uint32_t rq = s.rec[i];
      if (split_far(rq)) continue;
      // The owner above this split, past at most two splits of its own depth.
      // Far splits and the place outside the window count as owners without
      // a row: an owner that is one, or lies past one, is not assembled here.
      const bool own = split_owned(rq) != 0, root = split_root(rq);
      uint32_t p = root ? (uint32_t)OW_W : min((uint32_t)(i + split_parent(rq)), (uint32_t)OW_W);
      uint32_t rp = s.rec[p];
#pragma unroll
      for (int step = 0; step < 2; ++step) {
        if (split_owned(rp) == 0) {
          p = min(p + (uint32_t)split_parent(rp), (uint32_t)OW_W);
          rp = s.rec[p];
        }
      }
      const uint32_t row_up = min((uint32_t)s.row_of[p] - r0, (uint32_t)OW_ROWS);
      const uint32_t row_own = min((uint32_t)s.row_of[i] - r0, (uint32_t)OW_ROWS);
      const int level_up = (int)split_depth(rp) + 1;
      const int level_leaf = own ? (int)split_depth(rq) + 1 : level_up;
      uint16_t* leaf_row = reinterpret_cast<uint16_t*>(s.row[own ? row_own : row_up]);
      const K code = s.code[i];
      if (split_lo(rq) == 0)
        leaf_row[child_slot<K>(code, level_leaf)] = (uint16_t)(i | OW_PRESENT | OW_LEAF);
      if (split_hi(rq) == 1)
        leaf_row[child_slot<K>(s.code[i + 1], level_leaf)] = (uint16_t)((i + 1) | OW_PRESENT | OW_LEAF);
      if (own && !root)
        reinterpret_cast<uint16_t*>(s.row[row_up])[child_slot<K>(code, level_up)] =
            (uint16_t)((i + split_kidx(rq)) | OW_PRESENT);
    }
    ow_sync();
    // 4. nodes: an owner's branching node, then the chain above it.
    for (uint32_t o = tid; o < nrow; o += OW_THREADS) {
      const int i = s.own[r0 + o];
      const uint32_t ro = s.rec[i], x = (uint32_t)(w0 + i);
      const K code = s.code[i];
      uint32_t u0 = 0, bias = 0, first = 0, room = capacity;
      if (SEG) {
        const uint4 ci = cinfo[cloud_of(x)];
        u0 = ci.x;
        bias = ci.z;
        first = ci.w;
        room = first < capacity ? capacity - first : 0u;
      }
      const bool root = split_root(ro);
      const uint32_t c = root ? 0u : split_owned(ro);
      const uint32_t top = root ? 0u : s.ps[i + split_kidx(ro)] - bias;
      const int root_level = ((int)prefix_n[u0] - A) / 3;
      if (top >= room) {
        atomicOr(status, DEV_CAPACITY);
        continue;
      }
      // A slot holds a window position: a leaf's key, or the Karras index of
      // an internal child, whose offset is its top node.
      uint32_t cv[8], pm = 0, lm = 0;
      const uint32_t leaf0 = (uint32_t)w0 - u0;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t v = s.row[o][h];
        pm |= (((v >> 15) & 1u) | ((v >> 30) & 2u)) << (2 * h);
        lm |= (((v >> 14) & 1u) | ((v >> 29) & 2u)) << (2 * h);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const uint32_t id = (v >> (16 * b)) & OW_ID;
          const uint32_t t = (v >> (16 * b)) & OW_LEAF ? id + leaf0 : s.ps[id] - bias;
          cv[2 * h + b] = (v >> (16 * b)) & OW_PRESENT ? t : 0u;
        }
      }
      const int dk = (int)split_depth(ro);
      const uint32_t bottom = root ? 0u : top - c + 1;
      const uint3 qc = code_xyz<K>(code);
      store_node(nodes, first + bottom, make_int4((int)cv[0], (int)cv[1], (int)cv[2], (int)cv[3]),
                 make_int4((int)cv[4], (int)cv[5], (int)cv[6], (int)cv[7]), corner_at<K>(qc, dk, mn, rg),
                 __fmul_rn(rg, exp2_neg(dk - root_level)), (int32_t)(pm & ~lm), (int32_t)(lm & lmask_keep));
      // Chain nodes above the bottom: few owners have any, so they are listed
      // and written below by full warps.
      if (c > 1) {
        uint32_t q = atomicAdd(&s.chain_n, c - 1);
        for (uint32_t j = 1; j < c; ++j, ++q) {
          if (q < (uint32_t)OW_CHAIN) s.chain[q] = (uint16_t)(o | (j << 11));
          else ow_chain_node<K>(nodes, first + bottom + j, bottom + j - 1, code, dk - (int)j, root_level, mn, rg);
        }
      }
    }
    ow_sync();
    // 5. chain nodes (none of an owner refused for capacity is listed).
    const uint32_t nc = min(s.chain_n, (uint32_t)OW_CHAIN);
    for (uint32_t q = tid; q < nc; q += OW_THREADS) {
      const uint32_t j = s.chain[q] >> 11;
      const int i = s.own[r0 + (s.chain[q] & 2047u)];
      const uint32_t ro = s.rec[i];
      uint32_t u0 = 0, bias = 0, first = 0;
      if (SEG) {
        const uint4 ci = cinfo[cloud_of((uint32_t)(w0 + i))];
        u0 = ci.x;
        bias = ci.z;
        first = ci.w;
      }
      const uint32_t bottom = s.ps[i + split_kidx(ro)] - bias - split_owned(ro) + 1;
      ow_chain_node<K>(nodes, first + bottom + j, bottom + j - 1, s.code[i], (int)split_depth(ro) - (int)j,
                       ((int)prefix_n[u0] - A) / 3, mn, rg);
    }
    ow_sync();
    if (tid == 0) s.chain_n = 0;  // before the next round's first barrier
  }
}

// Launch over n_max codes (the count is on the device).
template <class K, bool SEG>
cudaError_t launch_octree_window(const Launch& L, const K* codes, const uint32_t* d_u, const uint32_t* uoff,
                                 uint32_t S, const uint4* cinfo, uint32_t n_max, const uint32_t* rec,
                                 const uint8_t* prefix_n, const uint8_t* hll, const uint8_t* hlr, const int32_t* left,
                                 const uint32_t* edge, const uint32_t* ps, uint32_t* node_offsets, float mn, float rg,
                                 gtc_octnode* nodes, uint32_t capacity) {
  auto kern = octree_window_kernel<K, SEG>;
  cudaError_t e = kernel_setup(kern, OW_THREADS + 32, sizeof(OwSmem<K>));
  if (e != cudaSuccess) return e;
  return launch_kernel(L, kern, max(1u, ceil_div(n_max, OW_T)), OW_THREADS + 32, sizeof(OwSmem<K>),
                       codes, d_u, uoff, S, cinfo,
                       rec, prefix_n, hll, hlr, left, edge, ps, node_offsets, mn, rg, nodes, capacity,
                       leaf_mask_keep(), L.status);
}

}  // namespace gtc
