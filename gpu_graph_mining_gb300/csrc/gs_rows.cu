// Extension kernels for packed rows (gs_device.hpp): count (support bitmaps,
// embedding counts, extension records) and materialise (children's rows), for
// one wave of DFS-tree nodes.  Same rules and results as the column kernels
// (gs_wave.cu), which serve graphs of more than 256 vertices, label alphabets
// too large for the 4-byte entries and the lists strategy.
//
// What the format is for: on columns a row cost a chain of k dependent 8-byte
// loads (a sector each), then two offsets and about 21 bytes of entries per
// right-most-path vertex, and every step of 32 entries searched owners and
// emitted few extensions.  250,000 graphs of 40 edges at minsup 0.5% (192 M
// rows, 760 M extensions, one stream): count kernels 33.3 ms on columns, 10.7
// here.  It is bound by issue now: a large launch of 390 M warp instructions
// in 0.45 ms issues in 70% of cycles, the integer pipe 64%, at 0.24 of the DRAM
// peak (0.73 GB).
#include <algorithm>

#include "gs_kernels.hpp"
#include "gs_stamp.cuh"

namespace gsgb {

namespace {

#ifndef GS_ROWS_WARPS
#define GS_ROWS_WARPS 4
#endif
#ifndef GS_ROWS_MINB
#define GS_ROWS_MINB 8
#endif
#ifndef GS_ROWS_GRID
#define GS_ROWS_GRID 64
#endif
constexpr int kWarps = GS_ROWS_WARPS;
constexpr unsigned kFull = 0xffffffffu;
#ifndef GS_ROWS_GROUP
#define GS_ROWS_GROUP 4  // tiles
#endif
constexpr int kRecBlocks = 4;  // record blocks a warp reserves at a time
constexpr int kShort = 6;      // entries of a block that every lane tests

struct RowsArgs {
  const PackedNode *nodes;
  const int32_t *tile0;   // first 32-row tile of each node
  int nnodes;
  int total_tiles;
  int group;              // consecutive tiles a warp takes at a time
  const SlotDesc *slots;
  uint32_t *bm;           // count: bitmaps to set; materialise: read
  const int32_t *bmx;     // materialise: prefix popcounts
  int32_t *cnt;           // count: embeddings per key, kRowsCopies copies cnt_stride apart
  long long cnt_stride;
  const uint32_t *chosen;   // materialise: a bit per key to materialise,
  const int32_t *childmap;  //   and such a key's child
  int32_t *cursor;
  const ChildOut *outs;
  uint32_t *rec;          // count, optional: record blocks
  int4 *hdr;
  int blk_cap;            // blocks of one region
  uint32_t *reg;          // blocks reserved in each region (may exceed blk_cap: none past it are written)
  unsigned int *err;
  unsigned long long *stamp;  // count: word for the kernel's start; materialise: the context's stamps
};

// One warp's shared memory; the right-most path has at most as many slots as
// the rows have pattern vertices.
template <int PL, bool WIDE> struct RowsSmem {
  static constexpr int kSlots = PL == 1 ? 8 : PL == 2 ? 24 : 64;
  uint32_t in[WIDE ? 8 * 32 : 1];  // WIDE: the rows' vertices, 8 words a lane (word w of lane l at 32 w + l)
  uint2 q[32 * 9];      // accepted items waiting for emission (31 and one block per lane):
                        // {entry, or backward item; owner row | slot << 5 | kBackItem}
  PackedNode nd;        // the tile's node and its right-most path
  SlotDesc slot[kSlots];
};

__device__ __forceinline__ unsigned lanemask_lt()
{
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

constexpr unsigned kBackItem = 1u << 11;

// Inclusive warp sum.
__device__ __forceinline__ int warp_incl(int x)
{
#pragma unroll
  for(int o = 1; o < 32; o <<= 1)
    asm volatile("{ .reg .s32 t; .reg .pred p; shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff; @p add.s32 %0, %0, t; }"
                 : "+r"(x)
                 : "r"(o));
  return x;
}

// 1 << n, 0 for n of 32 and more
__device__ __forceinline__ unsigned shl_one(unsigned n)
{
  unsigned x;
  asm("shl.b32 %0, 1, %1;" : "=r"(x) : "r"(n));
  return x;
}

// Graph-local id of pattern vertex t (the words' unused bytes are 0).
template <int NW> __device__ __forceinline__ unsigned id_of(const unsigned (&w)[NW], int t)
{
  unsigned x = w[0];
#pragma unroll
  for(int q = 1; q < NW; q++) x = (t >> 2) == q ? w[q] : x;
  return (x >> ((t & 3) * 8)) & 0xffu;
}

// The packed-row part of a child's outputs (three 16-byte loads).
struct RowsOut {
  uint4 *rows;
  long long word;
  int cap, kind, planes, k;
  const uint4 *prows;
  long long pnrows;
};
__device__ __forceinline__ RowsOut load_out(const ChildOut *o)
{
  const int4 *p = reinterpret_cast<const int4 *>(o);
  const int4 x = p[0], y = p[1], z = p[2];
  RowsOut r;
  r.rows = reinterpret_cast<uint4 *>(((unsigned long long)(unsigned)x.y << 32) | (unsigned)x.x);
  r.word = (long long)(((unsigned long long)(unsigned)x.w << 32) | (unsigned)x.z);
  r.cap = y.x;
  r.kind = y.y;
  r.planes = y.z;
  r.k = y.w;
  r.prows = reinterpret_cast<const uint4 *>(((unsigned long long)(unsigned)z.y << 32) | (unsigned)z.x);
  r.pnrows = (long long)(((unsigned long long)(unsigned)z.w << 32) | (unsigned)z.z);
  return r;
}

// A child's row: its parent's ids, and for a forward child the new vertex lv
// as pattern vertex k.
template <int PL, int NW>
__device__ __forceinline__ void store_row(const RowsOut &out, int pos, int gb, int rank, unsigned (&w)[NW], int k,
                                          unsigned lv)
{
  if(out.kind == 0) {
#pragma unroll
    for(int q = 0; q < NW; q++)
      if((k >> 2) == q) w[q] |= lv << ((k & 3) * 8);
  }
  out.rows[pos] = make_uint4((unsigned)gb, (unsigned)rank, w[0], w[1]);
#pragma unroll
  for(int p = 1; p < PL; p++)
    if(p < out.planes)
      out.rows[(long long)p * out.cap + pos] = make_uint4(w[4 * p - 2], w[4 * p - 1], w[4 * p], w[4 * p + 1]);
  // the new vertex is the first of a plane that no row of the wave has
  if(PL < 5 && out.planes > PL) out.rows[(long long)PL * out.cap + pos] = make_uint4(lv, 0, 0, 0);
}

// Work layout.  A warp owns a tile of 32 rows of one node, a row per lane: one
// 16-byte load (per plane) gives the whole embedding.  The right-most path is
// taken slot by slot; a lane's neighbour block is one aligned 32-byte sector,
// loaded while the slot before is decided, and its 8 entries are tested in
// registers: the forward rule and the empty entries are one compare, the
// embedding is a 64-bit set.  Accepted entries go, ranked by a warp scan, to a
// queue in shared memory, from which full batches of 32 are emitted: one
// counter add per distinct key, one bitmap OR per (key, graph), and the batch
// itself as a record block.
//
// WIDE (some database of the wave has graphs of more than 64 vertices): a node's
// ids have 6 or 8 bits, and a row's vertex set is 8 words of shared memory (as
// one 64-bit set in registers it costs less: the narrow kernel stays).  3,000
// graphs of 60 to 130 vertices, up to 5 edges: count 0.48 ms on columns, 0.33
// here, materialise 0.12 -> 0.08, the mine 0.86 -> 0.67.
//
// DENSE (count; some node of the wave has kDenseRows rows a graph and more): such
// a node's bitmap words are read before an OR, which is left out where the bit is
// set.  ORs to one word complete one after another, and when a graph has many
// rows nearly every OR sets a bit that is there; with few rows a graph the load
// is a trip to L2 for nothing.  Count kernels of a mine (ms; columns / an OR always /
// so): 300 stars of 200 leaves of 2 labels 29.5 / 80.9 / 11.5; 300 graphs of 40
// vertices and 240 edges, 2 labels 11.9 / 21.1 / 3.0; 3,000 trees with hubs, 60
// vertices, 2 labels 1.48 / 4.33 / 1.19.  With the load for every node 100,000
// molecule-like graphs at 5% 0.84 -> 1.06, 100,000 of 40 edges at 0.5% 4.37 -> 5.36;
// a test of the node alone costs those 1%, so it is an instance of its own.
template <int PL, bool MAT, bool WIDE, bool DENSE>
__global__ void __launch_bounds__(kWarps * 32, PL == 1 && !WIDE ? GS_ROWS_MINB : 7) k_rows(const RowsArgs a)
{
  if(!MAT) after_previous();
  constexpr int NW = 2 + 4 * (PL - 1);
  __shared__ RowsSmem<PL, WIDE> smem[kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  RowsSmem<PL, WIDE> &S = smem[warp];
  const int gwarp = blockIdx.x * kWarps + warp, nwarps = gridDim.x * kWarps;
  // the warp's reserved record blocks, and (lane 0) those reserved ahead: a
  // reservation made at the start of a tile arrives while its rows are loaded.
  // The warps reserve from kRecRegions counters on as many cache lines: adds
  // to one address complete at about one per 1.6 ns, which bounded the kernel
  // when one counter served all warps.
  if(!MAT) stamp_start(a.stamp);
  const int region = gwarp % kRecRegions;
  int blk = 0, blk_left = 0, blk_next = 0;  // within the region
  bool ahead = false;
  auto reserve = [&] {
    if(lane == 0) blk_next = (int)min(atomicAdd(&a.reg[region * kRecRegionStride], (unsigned)kRecBlocks), 0x7fffff00u);
    ahead = true;
  };

  // Groups of consecutive tiles: while the node stays the same, so do its
  // tables in shared memory (250,000 graphs: 12.3 ms in ones, 11.7 in twos,
  // 11.4 in fours, 11.5 in eights).
  int n = 0, n_first = 0, n_end = 0;  // the tables' node and its tiles
  for(int t0 = gwarp * a.group; t0 < a.total_tiles; t0 += nwarps * a.group)
  for(int tile = t0; tile < min(t0 + a.group, a.total_tiles); tile++) {
    if(!MAT && a.rec && blk_left < kRecBlocks && !ahead) reserve();
    // ---- the tile's node (tiles never span nodes): a 32-way search, whose last
    // round holds the node's first tile and the next one's.  The path tables and
    // the row are loaded side by side: waves of one node 6.0 -> 5.4 us a count.
    int4 table = make_int4(0, 0, 0, 0);
    const bool fresh = tile < n_first || tile >= n_end;
    if(fresh) {
      int lo = 0, hi = a.nnodes;  // the node is the last in [lo, hi) with tile0 <= tile
      n_first = 0;
      n_end = a.total_tiles;
      while(hi - lo > 1) {
        const int step = (hi - lo + 31) >> 5;
        const int probe = lo + lane * step;
        const int first = probe < hi ? a.tile0[probe] : 0;
        const unsigned ok = __ballot_sync(kFull, probe < hi && first <= tile);
        const int last = 31 - __clz(ok | 1u);
        n_first = __shfl_sync(kFull, first, last);
        const int next = __shfl_sync(kFull, first, (last + 1) & 31);
        if(last < 31 && lo + (last + 1) * step < hi) n_end = next;
        lo += last * step;
        hi = min(hi, lo + step);
      }
      n = lo;
      __syncwarp();  // the previous node's tables have been read
      constexpr int kNd = sizeof(PackedNode) / 16;
      if(lane < kNd) reinterpret_cast<int4 *>(&S.nd)[lane] = reinterpret_cast<const int4 *>(&a.nodes[n])[lane];
      __syncwarp();
      const int4 *sd = reinterpret_cast<const int4 *>(a.slots + S.nd.slot_off);
      const int pieces = 2 * min(S.nd.nslot, RowsSmem<PL, WIDE>::kSlots);
      if(lane < pieces) table = sd[lane];  // stored once the row's load is on its way too
      for(int t = lane + 32; t < pieces; t += 32) reinterpret_cast<int4 *>(S.slot)[t] = sd[t];
    }
    const int k = S.nd.k, nslot = S.nd.nslot, sh = S.nd.nb_shift;
    if(k > RowsSmem<PL, WIDE>::kSlots || nslot > RowsSmem<PL, WIDE>::kSlots || k < 2 || nslot < 2 || S.nd.planes > PL) {
      if(lane == 0) atomicOr(a.err, 2u);
      continue;
    }
    const int row0 = (tile - n_first) * 32;
    const int i = row0 + lane;
    bool valid = i < S.nd.nrows;
    unsigned w[NW];
#pragma unroll
    for(int q = 0; q < NW; q++) w[q] = 0;
    int gb = 0, g = 0;
    if(valid) {
      const uint4 r = __ldg(&S.nd.rows[i]);
      gb = (int)r.x;
      g = (int)r.y;
      w[0] = r.z;
      w[1] = r.w;
#pragma unroll
      for(int p = 1; p < PL; p++)
        if(p < S.nd.planes) {
          const uint4 x = __ldg(&S.nd.rows[(long long)p * S.nd.nrows + i]);
          w[4 * p - 2] = x.x;
          w[4 * p - 1] = x.y;
          w[4 * p] = x.z;
          w[4 * p + 1] = x.w;
        }
    }
    if(fresh) {
      if(lane < 2 * RowsSmem<PL, WIDE>::kSlots) reinterpret_cast<int4 *>(S.slot)[lane] = table;
      __syncwarp();
    }
    if(valid && ((unsigned)g >= (unsigned)S.nd.words * 32u || (unsigned)gb >= (unsigned)S.nd.n_vertices)) {
      atomicOr(a.err, (unsigned)g >= (unsigned)S.nd.words * 32u ? 1u : 2u);
      valid = false;
    }
    const int ids = WIDE ? S.nd.nb_ids : 6;
    const unsigned idm = (1u << ids) - 1u;
    unsigned m_lo = 0, m_hi = 0;  // the row's vertices
    if(WIDE) {
      __syncwarp();
#pragma unroll
      for(int q = 0; q < 8; q++) S.in[32 * q + lane] = 0;
      for(int t = 0; t < k; t++) {
        const unsigned lv = id_of(w, t);
        S.in[(lv >> 5) * 32 + lane] |= 1u << (lv & 31u);
      }
    } else if(PL == 1) {
#pragma unroll
      for(int t = 0; t < 8; t++)
        if(t < k) {
          const unsigned lv = (w[t >> 2] >> ((t & 3) * 8)) & 0xffu;
          m_lo |= shl_one(lv);
          m_hi |= shl_one(lv - 32u);
        }
    } else {
      for(int t = 0; t < k; t++) {
        const unsigned lv = id_of(w, t);
        m_lo |= shl_one(lv);
        m_hi |= shl_one(lv - 32u);
      }
    }
    auto in_row = [&](unsigned y) {  // entry y's vertex
      if(WIDE) return (S.in[((y & idm) >> 5) * 32 + lane] >> (y & 31u)) & 1u;
      return __funnelshift_r((y & 32u) ? m_hi : m_lo, 0u, y) & 1u;  // (bit y & 31 of the half)
    };
    const bool back = S.nd.back != 0;
    const uint4 *__restrict__ nb = S.nd.nb;
    const unsigned wlm = (1u << sh) - (1u << ids);  // the label field
    const unsigned minl = S.nd.minl;

    uint4 xa = make_uint4(0, 0, 0, 0), xb = xa;
    auto fetch = [&](int s) {
      if(valid) {
        const long long v = (long long)gb + id_of(w, S.slot[s].vertex);
        xa = __ldg(&nb[2 * v]);
        xb = __ldg(&nb[2 * v + 1]);
      }
    };
    int s_n = 0, qn = 0, hops = 0;
    fetch(0);
    bool more = true;
    while(more) {
      const int s = s_n;
      const unsigned x[8] = { xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w };
      // the next blocks: continuations of this slot's lists, then the next slot
      const unsigned cont = __ballot_sync(kFull, (int)x[7] < 0);
      if(cont && hops < (WIDE ? 40 : 16)) {  // (a list of 63 entries has 9 blocks, one of 255 has 37)
        hops++;
        const unsigned b = x[7] & 0x7fffffffu;
        const bool ok = (int)x[7] < 0 && b < (unsigned)S.nd.nb_blocks;
        xa = xb = make_uint4(0, 0, 0, 0);
        if(ok) {
          xa = __ldg(&nb[2ll * b]);
          xb = __ldg(&nb[2ll * b + 1]);
        }
      } else if(++s_n < nslot) {
        hops = 0;
        fetch(s_n);
      } else {
        more = false;
      }
      // ---- this block's entries that are forward extensions
      const int rule = S.slot[s].prule;
      unsigned acc = 0;
      // lists of more than kShort entries are few: the last words only where a
      // lane has one (10.91 -> 10.74 ms on 250,000 graphs; at 4 or 5 10.79)
      const bool tail = __any_sync(kFull, x[kShort] != 0);
      if(minl == 0) {
#pragma unroll
        for(int u = 0; u < kShort; u++) acc |= (int)x[u] >= rule && !in_row(x[u]) ? 1u << u : 0u;
        if(tail)
#pragma unroll
          for(int u = kShort; u < 8; u++) acc |= (int)x[u] >= rule && !in_row(x[u]) ? 1u << u : 0u;
      } else {
#pragma unroll
        for(int u = 0; u < kShort; u++)
          acc |= (int)x[u] >= rule && (x[u] & wlm) >= minl && !in_row(x[u]) ? 1u << u : 0u;
        if(tail)
#pragma unroll
          for(int u = kShort; u < 8; u++)
            acc |= (int)x[u] >= rule && (x[u] & wlm) >= minl && !in_row(x[u]) ? 1u << u : 0u;
      }
      const int c = __popc(acc);
      const int incl = warp_incl(c);
      uint2 *at = S.q + (qn + incl - c);
      qn += __shfl_sync(kFull, incl, 31);
      const unsigned meta = (unsigned)lane | ((unsigned)s << 5);
#pragma unroll
      for(int u = 0; u < kShort; u++)
        if((acc >> u) & 1u) *at++ = make_uint2(x[u], meta);
      if(tail)
#pragma unroll
        for(int u = kShort; u < 8; u++)
          if((acc >> u) & 1u) *at++ = make_uint2(x[u], meta);
      // ---- backward edges from the right-most vertex: entries whose vertex is
      // a right-most-path vertex of the row that takes one (not accepted above,
      // so the queue has room: 8 items per lane behind 31)
      if(back && s == nslot - 1) {
        // the row's vertices that a backward edge may go to (WIDE: all its vertices)
        unsigned long long bmask = 0;
        if(!WIDE)
          for(int t = 0; t + 2 < nslot; t++)
            if(S.slot[t].bkey_off >= 0) bmask |= 1ull << (id_of(w, S.slot[t].vertex) & 63u);
        unsigned bb = 0;
#pragma unroll
        for(int u = 0; u < 8; u++)
          bb |= (int)x[u] > 0 && (WIDE ? in_row(x[u]) : (unsigned)(bmask >> (x[u] & 63u)) & 1u) ? 1u << u : 0u;
        while(__ballot_sync(kFull, bb != 0)) {
          unsigned item = 0;
          bool ok = false;
          if(bb) {
            const int u = __ffs(bb) - 1;
            unsigned y = x[0];
#pragma unroll
            for(int q = 1; q < 8; q++) y = u == q ? x[q] : y;
            bb &= bb - 1;
            const int el = __ldg(&S.nd.pair_code[S.slot[s].pbase + (int)(y >> sh) - 1]) >> 16;
            for(int t = 0; t + 2 < nslot; t++)
              if(S.slot[t].bkey_off >= 0 && id_of(w, S.slot[t].vertex) == (y & idm) && el >= S.slot[t].bmin) {
                item = (unsigned)(S.slot[t].bkey_off + el) << (ids + 5);
                ok = true;
              }
          }
          const unsigned m = __ballot_sync(kFull, ok);
          if(ok) S.q[qn + __popc(m & lanemask_lt())] = make_uint2(item, (unsigned)lane | kBackItem);
          qn += __popc(m);
        }
      }
      // ---- emission, 32 queued items at a time (all that is left after the
      // tile's last block), warp converged
      while(qn >= 32 || (!more && qn > 0)) {
        __syncwarp();
        const int m = min(qn, 32);
        unsigned it = 0;  // the record item: (key << (ids + 5)) | (new vertex << 5) | row
        if(lane < m) {
          const uint2 e = S.q[qn - m + lane];
          it = e.y & 31u;
          if(e.y & kBackItem) it |= e.x;
          else it |= ((unsigned)S.slot[e.y >> 5].fkey_off - 1u + (e.x >> sh)) << (ids + 5) | (e.x & idm) << 5;
        }
        qn -= m;
        __syncwarp();
        const int key = lane < m ? (int)(it >> (ids + 5)) : -1;
        const int o = (int)(it & 31u);
        const int g_o = __shfl_sync(kFull, g, o);
        const int key_base = S.nd.key_base;
        if(!MAT) {
          // one counter add per distinct key, into this warp's copy of the
          // counters, and one bitmap OR unless a lane's graph differs from its key
          // group leader's (a tile's rows mostly share a graph)
          const unsigned peers = __match_any_sync(kFull, key);
          const int leader = __ffs(peers) - 1;
          const int g_lead = __shfl_sync(kFull, g_o, leader);
          if(key >= 0 && (lane == leader || g_o != g_lead)) {
            uint32_t *const word = &a.bm[S.nd.bm_base + (long long)key * S.nd.words + (g_o >> 5)];
            const uint32_t bit = 1u << (g_o & 31);
            if(!DENSE || !S.nd.dense || !(word_now(word) & bit)) atomicOr(word, bit);
          }
          if(key >= 0 && lane == leader) atomicAdd(&a.cnt[(gwarp % kRowsCopies) * a.cnt_stride + key_base + key], __popc(peers));
          if(a.rec) {
            if(blk_left == 0) {
              if(!ahead) reserve();
              blk = __shfl_sync(kFull, blk_next, 0);
              blk_left = kRecBlocks;
              ahead = false;
            }
            if(blk < a.blk_cap) {  // past the region's end nothing is written
              const unsigned b = (unsigned)region * (unsigned)a.blk_cap + (unsigned)blk;  // (below 2^26 blocks)
              a.rec[b * 32u + (unsigned)lane] = it;
              if(lane == 0) a.hdr[b] = make_int4(row0, 0, m | (gwarp % kRowsCopies) << 8 | (ids + 5) << 16, key_base);
            }
            blk++;
            blk_left--;
          }
        } else {
          const int wkey = key_base + key;
          const int c = key >= 0 && ((a.chosen[wkey >> 5] >> (wkey & 31)) & 1u) ? a.childmap[wkey] : -1;
          const unsigned peers = __match_any_sync(kFull, c);
          const int leader = __ffs(peers) - 1;
          int pos = 0;
          if(c >= 0 && lane == leader) pos = atomicAdd(&a.cursor[c], __popc(peers));
          pos = __shfl_sync(kFull, pos, leader) + __popc(peers & lanemask_lt());
          const int gb_o = __shfl_sync(kFull, gb, o);
          unsigned wo[NW];
#pragma unroll
          for(int q = 0; q < NW; q++) wo[q] = __shfl_sync(kFull, w[q], o);
          if(c >= 0) {
            const RowsOut out = load_out(&a.outs[c]);
            const long long wi = out.word + (g_o >> 5);
            const int rank = a.bmx[wi] + __popc(a.bm[wi] & ((1u << (g_o & 31)) - 1u));
            if(pos < out.cap) store_row<PL>(out, pos, gb_o, rank, wo, k, (it >> 5) & idm);
            else atomicOr(a.err, 4u);
          }
        }
      }
    }
  }
  // the reserved blocks that were not needed are empty
  if(!MAT && a.rec) {
    int4 *const hdr = a.hdr + (long long)region * a.blk_cap;
    if(lane < blk_left && blk + lane < a.blk_cap) hdr[blk + lane] = make_int4(0, 0, 0, 0);
    const int next = __shfl_sync(kFull, blk_next, 0);
    if(ahead && lane < kRecBlocks && next + lane < a.blk_cap) hdr[next + lane] = make_int4(0, 0, 0, 0);
  }
  if(MAT) stamp_mat_end(a.stamp);
}

// Materialise from the record blocks.  A warp takes B (kMatBlocks, or one in
// small waves) consecutive blocks of a region, their loads in flight together,
// tests the items' keys in the bit set of the chosen ones (a node's keys are a
// few words, one sector) and queues the items that are; 32 queued ones are then
// placed together: child map, child, and from there the parent's row, the graph
// rank's bitmap word and the cursor side by side.  A third of the items are
// chosen on 250,000 graphs of 40 edges, a tenth in the deep waves.  An item per
// lane with a child map entry gathered for every item took 5.7 ms a pass there,
// this 3.8 (100,000 graphs at 1%: 0.63 -> 0.43); latency and issue bound (61%),
// 0.4 of the DRAM peak in a large launch.  The child map gather was 13 to 15
// sectors a block.
constexpr int kMatWarps = 8, kMatBlocks = 4;
constexpr int kMatGrid = 16;  // thread blocks per SM: 8 are resident

template <int PL, bool WIDE, int B>
__global__ void __launch_bounds__(kMatWarps * 32) k_rows_mat(const uint32_t *__restrict__ rec,
                                                             const int4 *__restrict__ hdr,
                                                             const uint32_t *__restrict__ reg, int blk_cap,
                                                             const uint32_t *chosen, const int32_t *childmap,
                                                             const uint32_t *__restrict__ bm,
                                                             const int32_t *__restrict__ bmx, int32_t *cursor,
                                                             long long cursor_stride,
                                                             const ChildOut *outs, unsigned int *err,
                                                             unsigned long long *stamps)
{
  after_previous();
  constexpr int NW = 2 + 4 * (PL - 1);
  // queue entries: wave key (23 bits), counter copy (2), graph-local new vertex
  // (8), parent row (31)
  __shared__ unsigned long long queue[kMatWarps][32 * (B + 1)];
  unsigned long long *const q = queue[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  // a warp stays in one region (the number of warps is a multiple of theirs)
  const int b0 = blockIdx.x * kMatWarps + (threadIdx.x >> 5);
  const int region = b0 % kRecRegions;
  const int step = gridDim.x * kMatWarps / kRecRegions * B;
  const int used = min((int)min(__ldg(&reg[region * kRecRegionStride]), 0x7fffff00u), blk_cap);
  const int4 *const rh = hdr + (long long)region * blk_cap;
  const uint32_t *const ri = rec + (long long)region * blk_cap * 32 + lane;
  int qn = 0;
  for(int i = b0 / kRecRegions * B; i < used || qn > 0; i += step) {
    if(i < used) {
      int4 h = make_int4(0, 0, 0, 0);  // lane t: the header of block i + t
      if(lane < B && i + lane < used) h = __ldg(&rh[i + lane]);
      unsigned it[B];
      uint32_t w[B];
#pragma unroll
      for(int t = 0; t < B; t++) it[t] = i + t < used ? __ldg(&ri[(long long)(i + t) * 32]) : 0u;
#pragma unroll
      for(int t = 0; t < B; t++) {
        const int hz = __shfl_sync(kFull, h.z, t), m = hz & 0xff;
        const int key = __shfl_sync(kFull, h.w, t) + (int)(it[t] >> (WIDE ? hz >> 16 : 11));
        w[t] = lane < m ? chosen[key >> 5] : 0u;
      }
#pragma unroll
      for(int t = 0; t < B; t++) {
        const int hz = __shfl_sync(kFull, h.z, t), kb = WIDE ? hz >> 16 : 11;
        const int key = __shfl_sync(kFull, h.w, t) + (int)(it[t] >> kb);
        const bool on = (w[t] >> (key & 31)) & 1u;
        const unsigned m = __ballot_sync(kFull, on);
        if(m) {
          const int row0 = __shfl_sync(kFull, h.x, t), copy = (hz >> 8) & 0xff;
          if(on)
            q[qn + __popc(m & lanemask_lt())] = ((unsigned long long)(unsigned)(key * kRowsCopies + copy) << 39) |
                                                ((unsigned long long)((it[t] >> 5) & ((1u << (kb - 5)) - 1u)) << 31) |
                                                (unsigned)(row0 + (int)(it[t] & 31u));
          qn += __popc(m);
        }
      }
    }
    const bool last = i + step >= used;
    while(qn >= 32 || (last && qn > 0)) {
      __syncwarp();
      const int m = min(qn, 32);
      const bool has = lane < m;
      const unsigned long long e = has ? q[qn - m + lane] : 0ull;
      qn -= m;
      __syncwarp();
      const int kc = has ? (int)(e >> 39) : -1, key = kc / kRowsCopies, row = (int)(e & 0x7fffffffull);
      const unsigned lv = (unsigned)(e >> 31) & 0xffu;
      RowsOut out{};
      if(has) out = load_out(&outs[childmap[key]]);
      uint4 r = make_uint4(0, 0, 0, 0);
      unsigned w[NW];
#pragma unroll
      for(int t = 0; t < NW; t++) w[t] = 0;
      if(has) {
        r = __ldg(&out.prows[row]);
        w[0] = r.z;
        w[1] = r.w;
        const int planes = out.k <= 8 ? 1 : 1 + (out.k + 7) / 16;
#pragma unroll
        for(int p = 1; p < PL; p++)
          if(p < planes) {
            const uint4 x = __ldg(&out.prows[p * out.pnrows + row]);
            w[4 * p - 2] = x.x;
            w[4 * p - 1] = x.y;
            w[4 * p] = x.z;
            w[4 * p + 1] = x.w;
          }
      }
      const unsigned peers = __match_any_sync(kFull, kc);
      const int leader = __ffs(peers) - 1;
      int pos = 0;
      if(has && lane == leader) pos = atomicAdd(&cursor[(kc % kRowsCopies) * cursor_stride + key], __popc(peers));
      pos = __shfl_sync(kFull, pos, leader) + __popc(peers & lanemask_lt());
      if(has) {
        const int g = (int)r.y;
        const long long wi = out.word + (g >> 5);
        const int rank = bmx[wi] + __popc(bm[wi] & ((1u << (g & 31)) - 1u));
        if(pos < out.cap) store_row<PL>(out, pos, (int)r.x, rank, w, out.k, lv);
        else atomicOr(err, 4u);
      }
    }
  }
  stamp_mat_end(stamps);
}

// Neighbour blocks of a database (a thread per vertex, a warp's continuation
// blocks reserved together).
__global__ void __launch_bounds__(256) k_neighbour_blocks(const int32_t *__restrict__ adj_off, int V,
                                                          const unsigned long long *__restrict__ adj,
                                                          const int32_t *__restrict__ adj_pair,
                                                          const int32_t *__restrict__ vgbase, int sh, int ids, uint4 *nb,
                                                          int nb_blocks, int *used)
{
  const int lane = threadIdx.x & 31;
  // (64 bits: V is below 2^31, the step past the last vertex need not be)
  const long long stride = (long long)gridDim.x * blockDim.x;
  for(long long v0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) & ~31ll; v0 < V; v0 += stride) {
    const long long v = v0 + lane;
    int a0 = 0, d = 0, gb = 0;
    if(v < V) {
      a0 = __ldg(&adj_off[v]);
      d = __ldg(&adj_off[v + 1]) - a0;
      gb = __ldg(&vgbase[v]);
    }
    // continuation blocks: 7 entries and a link each, up to 8 in the last
    const int need = d <= 8 ? 0 : (d - 7 <= 8 ? 1 : 1 + (d - 7 - 8 + 6) / 7);
    int incl = need;
    for(int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kFull, incl, o);
      if(lane >= o) incl += t;
    }
    const int total = __shfl_sync(kFull, incl, 31);
    int first = 0;
    if(total > 0) {
      if(lane == 0) first = V + atomicAdd(used, total);
      first = __shfl_sync(kFull, first, 0) + incl - need;
    }
    if(v < V) {
      int at = a0, left = d, next = first;
      for(long long b = v;;) {
        const bool link = left > 8;
        const int here = link ? 7 : left;
        unsigned x[8];
#pragma unroll
        for(int u = 0; u < 8; u++) {
          x[u] = 0;
          if(u < here) {
            const unsigned long long e = __ldg(&adj[at + u]);
            x[u] = ((unsigned)(__ldg(&adj_pair[at + u]) + 1) << sh) | ((unsigned)((e >> 32) & 0xffffu) << ids) |
                   (((unsigned)e - (unsigned)gb) & ((1u << ids) - 1u));
          }
        }
        if(link) x[7] = 0x80000000u | (unsigned)next;
        if(b < nb_blocks) {
          nb[2 * b] = make_uint4(x[0], x[1], x[2], x[3]);
          nb[2 * b + 1] = make_uint4(x[4], x[5], x[6], x[7]);
        }
        if(!link) break;
        at += here;
        left -= here;
        b = next++;
      }
    }
  }
}

template <int PL, bool MAT, bool WIDE, bool DENSE> KernelCall rows_call(RowsArgs a, int grid_per_sm)
{
  const long long cap = (long long)sm_count() * (grid_per_sm > 0 ? grid_per_sm : GS_ROWS_GRID);
  // in groups once every warp of a full grid has one: below that the chip would idle
  a.group = (int)std::max(1ll, std::min((long long)GS_ROWS_GROUP, a.total_tiles / (cap * kWarps)));
  long long blocks = ((long long)a.total_tiles + kWarps * a.group - 1) / (kWarps * a.group);
  blocks = blocks > cap ? cap : blocks < 1 ? 1 : blocks;
  KernelCall c;
  c.func = (const void *)k_rows<PL, MAT, WIDE, DENSE>;
  c.early = !MAT;
  c.grid = dim3((unsigned)blocks);
  c.block = dim3(kWarps * 32);
  c.arg(a);
  return c;
}

template <bool MAT, bool DENSE> KernelCall rows_call(const RowsArgs &a, int planes, bool wide, int grid_per_sm)
{
  if(wide)
    return planes <= 1 ? rows_call<1, MAT, true, DENSE>(a, grid_per_sm)
         : planes <= 2 ? rows_call<2, MAT, true, DENSE>(a, grid_per_sm) : rows_call<5, MAT, true, DENSE>(a, grid_per_sm);
  return planes <= 1 ? rows_call<1, MAT, false, DENSE>(a, grid_per_sm)
       : planes <= 2 ? rows_call<2, MAT, false, DENSE>(a, grid_per_sm) : rows_call<5, MAT, false, DENSE>(a, grid_per_sm);
}

template <int B> auto *mat_kernel(int planes, bool wide)
{
  if(wide) return planes <= 1 ? k_rows_mat<1, true, B> : planes <= 2 ? k_rows_mat<2, true, B> : k_rows_mat<5, true, B>;
  return planes <= 1 ? k_rows_mat<1, false, B> : planes <= 2 ? k_rows_mat<2, false, B> : k_rows_mat<5, false, B>;
}

}  // namespace

KernelCall rows_count_call(const PackedNode *nodes, const int32_t *tile0, int32_t nnodes, int32_t total_tiles,
                           int32_t planes, bool wide, bool dense, const SlotDesc *slots, uint32_t *bm, int32_t *cnt,
                           long long cnt_stride, uint32_t *rec, int4 *hdr, int32_t blk_cap, uint32_t *reg,
                           unsigned long long *head, unsigned int *err, int32_t grid_per_sm)
{
  const RowsArgs a{ nodes, tile0, nnodes, total_tiles, 1, slots, bm, nullptr, cnt, cnt_stride, nullptr, nullptr,
                    nullptr, nullptr, rec, hdr, blk_cap, reg, err, head + kHeadCount0 };
  return dense ? rows_call<false, true>(a, planes, wide, grid_per_sm)
               : rows_call<false, false>(a, planes, wide, grid_per_sm);
}

void launch_rows_materialize(const PackedNode *nodes, const int32_t *tile0, int32_t nnodes, int32_t total_tiles,
                             int32_t planes, bool wide, const SlotDesc *slots, const uint32_t *bm, const int32_t *bmx,
                             const uint32_t *chosen, const int32_t *childmap, int32_t *cursor, const ChildOut *outs,
                             unsigned int *err, unsigned long long *stamps, cudaStream_t s)
{
  if(total_tiles <= 0) return;
  const RowsArgs a{ nodes, tile0, nnodes, total_tiles, 1, slots, const_cast<uint32_t *>(bm), bmx, nullptr, 0, chosen,
                    childmap, cursor, outs, nullptr, nullptr, 0, nullptr, err, stamps };
  KernelCall c = rows_call<true, false>(a, planes, wide, 0);
  c.run(s);
}

void launch_rows_records(const uint32_t *rec, const int4 *hdr, const uint32_t *reg, int32_t blk_cap, int32_t most,
                         int32_t planes, bool wide, const uint32_t *chosen, const int32_t *childmap, const uint32_t *bm,
                         const int32_t *bmx, int32_t *cursor, long long cursor_stride, const ChildOut *outs,
                         unsigned int *err, unsigned long long *stamps, cudaStream_t s)
{
  if(most <= 0) return;
  static_assert(kRecRegions % kMatWarps == 0, "thread blocks per set of regions");
  constexpr int kPer = kRecRegions / kMatWarps;
  const long long cap = (long long)kMatGrid * sm_count() / kPer * kPer;
  // a block a turn while every block has a warp of its own: four in turn were
  // 8 to 20% slower there (340 graphs: 33 -> 27 us a mine; larger waves equal)
  const bool one = (long long)most * kPer <= cap;
  const long long want = one ? (long long)most * kPer : ((long long)most + kMatBlocks - 1) / kMatBlocks * kPer;
  const int blocks = (int)(want < cap ? want : cap);
  auto *f = one ? mat_kernel<1>(planes, wide) : mat_kernel<kMatBlocks>(planes, wide);
  KernelCall c;
  c.func = (const void *)f;
  c.early = true;
  c.grid = dim3((unsigned)blocks);
  c.block = dim3(kMatWarps * 32);
  c.arg(rec);
  c.arg(hdr);
  c.arg(reg);
  c.arg(blk_cap);
  c.arg(chosen);
  c.arg(childmap);
  c.arg(bm);
  c.arg(bmx);
  c.arg(cursor);
  c.arg(cursor_stride);
  c.arg(outs);
  c.arg(err);
  c.arg(stamps);
  c.run(s);
}

void launch_neighbour_blocks(const DevDB &db, uint4 *nb, int32_t *used, cudaStream_t s)
{
  if(db.n_vertices <= 0) return;
  const long long want = ((long long)db.n_vertices + 255) / 256, cap = 64LL * sm_count();
  k_neighbour_blocks<<<(int)(want < cap ? want : cap), 256, 0, s>>>(db.adj_off, db.n_vertices, db.adj, db.adj_pair,
                                                                    db.vgbase, db.nb_shift, db.nb_ids, nb, db.nb_blocks, used);
}

}  // namespace gsgb
