// Device-side layouts shared by the kernels (gs_kernels.cu) and the host
// engine that fills them (gs_engine.cpp).
//
// Graph database in HBM (one per resident database):
//   adj[E2]      uint64: low 32 bits = neighbour (global vertex id),
//                high 32 bits = (edge label << 16) | neighbour vertex label;
//                with adj_sorted, ascending within each vertex's entries
//   adj_off[V+1] int32 CSR offsets, vlabel[V] dense vertex labels,
//   vgraph[V]    graph id of each vertex,
//   pair_idx[VL*EL*VL]  dense index of (elabel, tolabel) among the pairs that
//                occur next to a vertex of label fl, or -1.
// Labels are compacted order-preservingly to 0..VL-1 / 0..EL-1 (< 2^16).
//
// Embedding store: one column per pattern vertex, element = int2
// {graph vertex, row in the previous column}; an embedding is the chain
// from a row of the last column back to column 0 (the reference's
// embedding_list_columns, src/globals/embedding_lists.hpp:12-60).  A forward
// child appends a column; a backward child replaces the last column with a
// filtered copy.  Each DFS-tree node also carries gord[row]: the dense rank
// of the row's graph among the graphs that contain the node's pattern
// (0..support-1), the index into the node's support bitmaps.
//
// Packed rows (databases whose graphs have at most 256 vertices): a row is the
// embedding itself instead of a chain of back-links, the first graph vertex
// of its graph and one byte per pattern vertex (graph-local ids), with the
// row's graph rank: 16 bytes up to 8 pattern vertices, 16 more per further 16
// (planes of nrows uint4: plane 0 = {first vertex, graph rank, ids 0-3,
// ids 4-7}, plane p = ids 8 + 16(p - 1) ..).  Neighbour lists are 32-byte
// blocks, block v = vertex v's list, one DRAM sector: up to 8 entries of 4
// bytes, ((pair index + 1) << nb_shift) | (neighbour label << nb_ids) |
// graph-local neighbour, ascending, 0 = none; a list of more than 8 has 7 and
// in the last word 2^31 | the block that continues it (again up to 8 entries,
// or 7 and a link).  A wave's extension records are blocks of 32 four-byte
// items of one tile, (node's key << (nb_ids + 5)) | (graph-local new vertex << 5) | row
// in the tile, each with a header {first row of the tile, 0, items | counter
// copy << 8 | (nb_ids + 5) << 16, the node's first key}.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace gsgb {

struct DevDB {
  const unsigned long long *adj;
  const int32_t *adj_off;
  const int32_t *vlabel;
  const int32_t *vgraph;
  const int32_t *vgbase;    // [V] first global vertex of each vertex's graph
  const int32_t *vbase;     // [G+1] first global vertex of each graph
  const int32_t *adj_pair;  // [E2] pair index of each directed entry: pair_idx(label(source), el, label(nbr))
  const int32_t *pair_idx;
  int32_t VL, EL;
  int32_t n_graphs;
  int32_t n_vertices;
  int32_t max_graph_vertices;
  int32_t adj_sorted;  // 1: each vertex's entries ascend (adj as unsigned 64-bit values)
  const int32_t *root_off;   // [VL+1] first key of each vertex label's (elabel, tolabel) pairs
  const int32_t *pair_code;  // [root_off[VL]] (elabel << 16) | tolabel of each pair
  const uint4 *nb;           // neighbour blocks (two uint4 each), or nullptr: no packed rows
  int32_t nb_blocks;         // blocks there is room for
  int32_t nb_shift;          // nb_ids + bits of a vertex label
  int32_t nb_ids;            // bits of a graph-local vertex: 6, or 8 for graphs of more than 64
};

// Whether a database takes packed rows (nb_shift, else 0): its graphs' vertices
// as ids of packed_ids bits, neighbour entries below 2^31, and a node's keys (at
// most 64 slots of pairs and edge labels) in the items' other bits.
inline int32_t packed_ids(int64_t max_graph_vertices)
{
  return max_graph_vertices <= 64 ? 6 : max_graph_vertices <= 256 ? 8 : 0;
}
inline int32_t packed_shift(int64_t max_graph_vertices, int64_t VL, int64_t EL, int64_t pairs)
{
  int32_t bits = 0;
  while(((int64_t)1 << bits) < VL) bits++;
  const int32_t ids = packed_ids(max_graph_vertices), sh = ids + bits;
  if(!ids || sh > 30 || pairs + 1 >= ((int64_t)1 << (31 - sh)) || 64 * (pairs + EL) >= ((int64_t)1 << (27 - ids)))
    return 0;
  return sh;
}
// Neighbour blocks for V vertices and E2 entries: a list of d > 8 entries
// takes at most d / 7 blocks beside its first; ids of a row address up to 255
// blocks past its graph's first vertex.
inline int64_t packed_blocks(int64_t V, int64_t E2) { return V + E2 / 7 + 256; }
// 16-byte planes of a packed row of k pattern vertices.
inline int32_t packed_planes(int32_t k) { return k <= 8 ? 1 : 1 + (k - 8 + 15) / 16; }

// Per job of a root phase (the root level of a group of jobs, one launch per
// kernel): its vertices as 32-vertex warp tiles in the group's tile space, its
// bitmaps, counter copies and keys at their offsets in the group's buffers.
struct RootJob {
  long long tile_begin;  // first warp tile of the job (its vertex 0)
  long long bm_base;     // first bitmap word of the job's key 0
  long long cnt_base;    // first counter of the job's copy 0 (copy q at cnt_base + q * R)
  int32_t db;            // index into the resident-database table
  int32_t words;         // bitmap words per key = ceil(graphs / 32)
  int32_t R;             // root keys of the job's database
  int32_t copies;        // counter copies
  int32_t key_base;      // first key of the job in the group's key space
  int32_t pad;
};

// Per DFS-tree node of a wave (a batch of nodes extended together).
struct NodeDesc {
  long long tile_begin;  // first 32-row warp tile of the node (tiles never span two nodes)
  long long bm_base;     // first support-bitmap word of the node's key 0
  const int32_t *gord;   // [nrows]
  int32_t nrows;
  int32_t k;             // columns = pattern vertices; the right-most vertex is k-1
  int32_t col_off;       // first entry in the wave's column-pointer table
  int32_t slot_off;      // first entry in the wave's slot table
  int32_t vtab_off;      // first entry in the wave's vertex table (k entries)
  int32_t nslot;         // right-most path vertices; slot nslot-1 is the right-most vertex
  int32_t minlabel;      // label of pattern vertex 0: forward targets need label >= minlabel
  int32_t words;         // bitmap words per key = ceil(support / 32)
  int32_t key_base;      // first key of the node in the wave's key space
  int32_t nkeys;
  int32_t db;            // index into the resident-database table
  int32_t minsup;        // the node's job's minimum support (candidate selection)
  int32_t code_off;      // the node's DFS code: edges code_off.. of the wave's code table
  int32_t code_len;      //   (a uint2 per edge)
  int32_t nfwd;          // keys below nfwd are forward extensions
  int32_t dense;         // 1: many rows a graph (kDenseRows)
  // Lists strategy (extension by intersection): a forward child's extensions
  // from right-most-path vertices other than its new right-most vertex are
  // its parent's frequent forward extensions at the same parent row (minus
  // the child's new vertex), read from the parent's per-row lists instead of
  // the database; only the right-most vertex's adjacency is scanned.  The
  // child's right-most path up to the new edge's source u is the parent's, so
  // those slots have the parent's forward keys: a list entry's parent key lk
  // is the child's key when lk < join_hi (slots up to u) and, from u itself,
  // lk >= join_key (pairs at or after the new edge's).  csr_off == nullptr:
  // no join, every right-most-path vertex is scanned.
  const int32_t *csr_off;  // [csr_rows + 1] the parent rows' list offsets into csr_ent
  const int2 *csr_ent;     // list entries {neighbour, parent's forward key}
  int32_t csr_rows;        // parent rows
  int32_t join_lo;         // first forward key of u
  int32_t join_key;        // the new edge's key (in the parent)
  int32_t join_hi;         // one past u's forward keys
};

// One right-most-path vertex of a node.  The order rules of the
// right-most-path edge (el_u, tl_u) that leaves the vertex are single compares:
//   forward allowed iff (el_u, tl_u) <= (el, tl)  <=>  hi >= frule, with an
//     adjacency entry's high word hi = (el << 16) | nbr_label (INT32_MIN for
//     the right-most vertex: no rule), and for packed rows entry >= prule
//   backward allowed iff el_u < el || (el_u == el && tl_u <= label(right-most))
//     <=>  el >= bmin
struct alignas(16) SlotDesc {
  int32_t prule;     // packed rows: the least neighbour entry that the forward rule allows
  int32_t fkey_off;  // forward keys of this slot: fkey_off + pair_idx(vlab, el, tl)
  int32_t vertex;    // pattern vertex id
  int32_t bkey_off;  // backward keys to this vertex: bkey_off + el; -1 if not a target
  int32_t bmin;
  int32_t pbase;     // the first pair code of the vertex's label
  int32_t frule;
  int32_t vlab;      // its (dense) label
};

// What the packed-row count needs of a node, copied to shared memory whole.
struct alignas(16) PackedNode {
  const uint4 *rows;         // planes of nrows
  const uint4 *nb;           // its database's neighbour blocks
  int32_t nrows, k, nslot, planes;
  int32_t nb_shift, nb_ids;
  uint32_t minl;             // forward targets: entry label field >= minl
  int32_t back;              // 1: some slot takes a backward edge
  int32_t words;             // bitmap words per key
  long long bm_base;
  int32_t key_base;
  int32_t n_vertices;
  const int32_t *pair_code;
  int32_t nb_blocks, slot_off;
  int32_t dense;             // 1: many rows a graph (kDenseRows)
  int32_t pad[2];
};

// Output slots of a child node selected for materialisation.
struct alignas(16) ChildOut {
  uint4 *rows;    // packed rows: the child's planes of cap rows (else nullptr)
  long long word; // packed rows: the key's first support-bitmap word
  int32_t cap;    // rows allocated (the count pass's embedding count for the key)
  int32_t kind;   // 0 forward, 1 backward, 2 root
  int32_t planes; // packed rows: the child's
  int32_t k;      // packed rows: the parent's pattern vertices,
  const uint4 *prows;  // its planes
  long long pnrows;    //   of so many rows
  int2 *col;      // columns: the child's new last column
  int2 *col0;     // root children only: column 0
  int32_t *gord;  // the child's graph ranks
};

// A wave's (or root group's) results header, 8-byte words in device memory,
// written to pinned host memory by the wave's last kernel.  The time stamps are
// the device's nanosecond clock, taken by the first thread of a kernel: kernels
// of one stream start when the one before has finished.
enum HeadWord {
  kHeadRecords = 0,   // records (packed rows: blocks) reserved in the fullest region
  kHeadFlags = 1,     // consistency flags
  kHeadSelected = 2,  // selected candidates   } counters of
  kHeadExt = 3,       // embeddings of all keys } the support
  kHeadListed = 4,    // keys counted          } selection
  kHeadSelBytes = 5,  // algorithmic bytes     }
  kHeadDone = 6,      // blocks of the last kernel that have finished
  kHeadCount0 = 7,    // stamps: count,
  kHeadSel0 = 8,      //   selection,
  kHeadMin0 = 9,      //   canonicality,
  kHeadEnd = 10,      //   results written
  kHeadBytesCount = 11,  // algorithmic bytes so far: column count and materialise kernels
  kHeadBytesMat = 12,
  kHeadMat = 13,      // per wave context, the stamps of its last materialise pass: start, end
  kHeadSeq = 29,      // the wave's number, written last
  kHeadWords = 32,
};
constexpr int kMaxWaveCtx = 8;
// A context's materialise stamps: the start, and the ends of the blocks spread
// over kMatSlots cache lines (their maximum is the end).
constexpr int kMatSlots = 32, kMatStampWords = 16 * (kMatSlots + 1);

}  // namespace gsgb
