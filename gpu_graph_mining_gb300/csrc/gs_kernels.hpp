// Launchers for the mining kernels (gs_kernels.cu).  All launches go to the
// given stream; none synchronises.  `err` receives bit flags when a kernel's
// consistency checks fail (1: graph rank out of range, 2: back-link, vertex or
// label-pair index out of range, 4: more child rows than counted, 8: a key's
// embedding count past 2^31 - 1); the offending access is skipped, never
// performed.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

#include "gs_device.hpp"

namespace gsgb {

// SMs of device 0 (the library's device), read once; grid caps are per SM.
int sm_count();

// Extension records of the count pass, int4 {key field, x, y, graph rank}: the
// key field holds the wave key in bits 0-26 and the counter copy the
// extension was counted in in bits 27-30 (-1: an unused slot).  A forward
// extension has (x, y) = (new vertex, parent row), a backward one the copy of
// the parent row's last column element.
constexpr int kRecCopyShift = 27;
constexpr int kRecKeyMask = (1 << kRecCopyShift) - 1;

struct ListBuild;

// A kernel launch as data: function, shape and argument values.  run()
// launches it on a stream; params() gives the argument pointers a CUDA graph
// kernel node takes (the graph copies the values when the node is set).
struct KernelCall {
  const void *func = nullptr;
  dim3 grid, block;
  unsigned smem = 0;
  bool early = false;  // may start before the kernel ahead of it has finished (after_previous())
  template <class T> void arg(const T &v)
  {
    used_ = (used_ + alignof(T) - 1) & ~(alignof(T) - 1);
    std::memcpy(store_ + used_, &v, sizeof(T));
    off_[n_++] = (unsigned short)used_;
    used_ += sizeof(T);
  }
  void **params()
  {
    for(int i = 0; i < n_; i++) ptr_[i] = store_ + off_[i];
    return ptr_;
  }
  cudaError_t run(cudaStream_t s)
  {
    if(!early) return cudaLaunchKernel(func, grid, block, params(), smem, s);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelExC(&c, func, params());
  }

private:
  alignas(16) unsigned char store_[384];
  unsigned short off_[16];
  void *ptr_[16];
  int n_ = 0;
  size_t used_ = 0;
};

// First kernel of a wave or root group: copies its tables from pinned host
// memory (n16 16-byte pieces), clears its scratch (z16 pieces) and its header.
KernelCall begin_call(void *dst, const void *src, long long n16, void *zero, long long z16, unsigned long long *head);

// Root level of a group of jobs: a warp per 32 vertices of a job walks their
// adjacency; every directed entry (v -> w) with label(v) <= label(w) is a
// 1-edge embedding (get_forward_root, src/globals/graph_types.cpp:365-375).
// Sets support-bitmap bit [key][graph] and counts embeddings per key in the
// warp's counter copy.  tiles = the group's warp tiles.
void launch_root_count(const RootJob *jobs, int32_t njobs, long long tiles, const DevDB *dbs, uint32_t *bm,
                       int32_t *cnt, unsigned long long *head, cudaStream_t s);
// Per key of the group: sup[key] = its graphs (popcount of its bitmap words,
// whose exclusive prefixes go to bmx), tot[key] = its embeddings, counter copy
// q >= 1 = the count of copies 0..q-1 and copy 0 = 0 (the materialise pass's
// cursors; a job without copies has none).  total_keys = the group's keys.
void launch_root_support(const RootJob *jobs, int32_t njobs, int32_t total_keys, const uint32_t *bm, int32_t *bmx,
                         int32_t *cnt, int32_t *sup, int32_t *tot, cudaStream_t s);
// Copies n16 16-byte pieces to pinned host memory, then the header, *flags
// among it, to hhead with its sequence word last.
void launch_results(void *dst, const void *src, long long n16, unsigned long long *head, const unsigned int *flags,
                    unsigned long long *hhead, unsigned long long seq, cudaStream_t s);
// Writes the two columns and graph ranks of every selected root key of the
// group (childmap over the group's keys), with the counter copies as cursors.
void launch_root_materialize(const RootJob *jobs, int32_t njobs, long long tiles, const DevDB *dbs,
                             const uint32_t *bm, const int32_t *bmx, int32_t *cursor, const int32_t *childmap,
                             const ChildOut *outs, unsigned int *err, cudaStream_t s);

// Wave level (gs_wave.cu): a warp per 32 embedding rows of the wave's nodes.
// kmax = the largest column count of the wave's nodes (selects the instance
// sized for 8/16/32/64 pattern vertices); collen[] parallels coltab[]: the
// length of every column.
// small_graphs: every graph of the wave's databases has <= 64 vertices.
// rec (may be null): kRecRegions regions of rec_cap records, whole chunks of
// kRecChunk; reg: their counters, as for the packed rows (zeroed before).
// dense: some node has kDenseRows rows a graph and more (NodeDesc::dense).
// rule_skip: in databases with sorted adjacency (DevDB::adj_sorted), a
// right-most-path vertex's entries below its forward rule are bisected past
// instead of scanned.
KernelCall wave_count_call(const NodeDesc *nodes, int32_t nnodes, long long total_tiles, int32_t kmax,
                           bool small_graphs, const int2 *const *coltab, const int32_t *collen, const SlotDesc *slots,
                           const int32_t *vtab, const DevDB *dbs, uint32_t *bm, int32_t *cnt,
                           unsigned long long *bytes, unsigned int *err, int4 *rec, long long rec_cap,
                           uint32_t *reg, unsigned long long *head, int32_t grid_per_sm, int32_t cnt_copies,
                           long long cnt_stride, bool join, bool rule_skip, bool dense);
void launch_wave_materialize(const NodeDesc *nodes, int32_t nnodes, long long total_tiles, int32_t kmax,
                             bool small_graphs,
                             const int2 *const *coltab, const int32_t *collen, const SlotDesc *slots,
                             const int32_t *vtab, const DevDB *dbs, const uint32_t *bm, const int32_t *bmx,
                             const int32_t *childmap, int32_t *cursor, const ChildOut *outs,
                             unsigned long long *bytes, unsigned int *err, bool join, bool rule_skip,
                             unsigned long long *stamps, cudaStream_t s);

// Packed rows (gs_rows.cu).  nodes, tile0: every node's PackedNode and first
// 32-row tile; planes =
// the most planes of the wave's nodes' rows; wide: some node's database has
// nb_ids 8; dense: some node is dense; rec / hdr: record blocks (rec may
// be null) in kRecRegions regions of blk_cap blocks, reg[r * kRecRegionStride]
// counts the blocks reserved in region r (zeroed before).  cnt: kRowsCopies
// copies of the wave's counters, cnt_stride apart (a warp adds into one: 4 take
// the adds of a large node's few keys as well as 256 would, one makes the count
// 14% slower); the wave's keys stay below kRowsKeys.
constexpr int kRecRegions = 64, kRecRegionStride = 32;
#ifndef GS_REC_CHUNK
#define GS_REC_CHUNK 128
#endif
constexpr int kRecChunk = GS_REC_CHUNK;  // column records a warp reserves at a time
// Thread blocks for a kernel whose blocks each stay in one region, an item per
// thread of threads, the fullest region holding most.
inline int region_blocks(long long most, int threads)
{
  const long long per = std::min((most + threads - 1) / threads, (16ll * sm_count() + kRecRegions - 1) / kRecRegions);
  return (int)(std::max(per, 1ll) * kRecRegions);
}
constexpr int kRowsCopies = 4, kRowsKeys = 1 << 23;
// Rows a graph from which a node is dense (NodeDesc::dense, PackedNode::dense).  Count of 3,000 trees
// with hubs 1.19 ms with 8 to 24, 1.24 with 32 and 48, 1.80 with 64; a mine of 5,000
// stars (17 rows a graph) 0.27 ms with 12 and 16, 0.35 with 24; 2,000 graphs of 60 to 130
// vertices 0.157 ms with 8, 0.151 with 12 and more, as without.
constexpr int kDenseRows = 16;
KernelCall rows_count_call(const PackedNode *nodes, const int32_t *tile0, int32_t nnodes, int32_t total_tiles,
                           int32_t planes, bool wide, bool dense, const SlotDesc *slots, uint32_t *bm, int32_t *cnt,
                           long long cnt_stride, uint32_t *rec, int4 *hdr, int32_t blk_cap, uint32_t *reg,
                           unsigned long long *head, unsigned int *err, int32_t grid_per_sm);
// Materialise by enumerating again (cursor per child), and from the record
// blocks (cursor: the counter copies after selection, as for
// launch_materialize_records).
void launch_rows_materialize(const PackedNode *nodes, const int32_t *tile0, int32_t nnodes, int32_t total_tiles,
                             int32_t planes, bool wide, const SlotDesc *slots, const uint32_t *bm, const int32_t *bmx,
                             const uint32_t *chosen, const int32_t *childmap, int32_t *cursor, const ChildOut *outs,
                             unsigned int *err, unsigned long long *stamps, cudaStream_t s);
// most: the most blocks of a region; chosen: a bit per key to materialise
void launch_rows_records(const uint32_t *rec, const int4 *hdr, const uint32_t *reg, int32_t blk_cap, int32_t most,
                         int32_t planes, bool wide, const uint32_t *chosen, const int32_t *childmap, const uint32_t *bm,
                         const int32_t *bmx, int32_t *cursor, long long cursor_stride, const ChildOut *outs,
                         unsigned int *err, unsigned long long *stamps, cudaStream_t s);
// Fills a database's neighbour blocks from its adjacency (db.nb_blocks,
// db.nb_shift set; *used zeroed: receives the continuation blocks).
void launch_neighbour_blocks(const DevDB &db, uint4 *nb, int32_t *used, cudaStream_t s);

// Materialise from the count pass's records {wave key, x, y, graph rank}:
// children whose key is selected get column element (x, y) and their graph
// rank.  keyword[key] = the key's first support-bitmap word.
// cursor: the wave's counter copies after selection (copy q of a key starts
// at the count of copies 0..q-1), cursor_stride apart; a record's copy is in
// bits 27-30 of its key field.  reg, rec_cap: kRecRegions regions of rec_cap
// records and their fills, as for the packed rows; most: the largest fill.
// lists (may be null): also counts each list row's entries at list_cnt[row]
// (lists strategy, launch_fill_lists)
void launch_materialize_records(const int4 *rec, const uint32_t *reg, long long rec_cap, long long most,
                                const int32_t *childmap, const long long *keyword,
                                const uint32_t *bm, const int32_t *bmx, int32_t *cursor, long long cursor_stride,
                                const ChildOut *outs, unsigned long long *bytes, unsigned int *err,
                                const ListBuild *lists, int32_t *list_cnt, unsigned long long *stamps,
                                cudaStream_t s);

// Extension records given as (key, graph id) pairs: sets bit [key][graph].
// Keys and graph ids must be in range (checked by the caller).
void launch_records_bitmap(const int32_t *keys, const int32_t *gids, long long n, int32_t words, uint32_t *bm,
                           cudaStream_t s);

// Wave support with candidate selection (k_screen_keys, k_count_listed), into
// the header's counters; listed and sel hold total_keys entries.  The
// consistency flags after the count pass go to the header.
// lnode (lists strategy, may be null): reset to -1 for every key with extensions
// reg (may be null): kHeadRecords = the fullest region's records or blocks
KernelCall screen_keys_call(const NodeDesc *nodes, int32_t nnodes, int32_t total_keys, int32_t *cnt,
                            int32_t cnt_copies, long long cnt_stride, int32_t *childmap, int2 *listed,
                            unsigned long long *head, unsigned int *err, int32_t *lnode, const uint32_t *reg);
// lnode (lists strategy, may be null): lnode[key] = the key's node for every
// frequent forward key
KernelCall count_listed_call(const NodeDesc *nodes, const int2 *listed, const uint32_t *bm, int32_t *cnt,
                             int32_t *bmx, long long *keyword, int4 *sel, int32_t sel_cap,
                             unsigned long long *head, int32_t *lnode);
// Both in one kernel, for waves of at most kSelectWords bitmap words (8 MiB): a
// block counts its chunk's listed keys in turn, and keys with many embeddings
// stand together, so large waves are better spread by a list.  A wave of one
// node takes 5.0 us in two kernels, 3.0 in one; 250,000 graphs at 0.5% 17 us a
// wave in two, 50 when every wave takes one.  Selection of a mine with the line
// at 0, 2^17, 2^19, 2^21, 2^22 words: 100,000 graphs 163, 163, 157, 146, 153 us;
// 250,000 graphs 571, 560, 566, 553, 554.
constexpr int64_t kSelectWords = 1 << 21;
KernelCall select_call(const NodeDesc *nodes, int32_t nnodes, int32_t total_keys, int32_t *cnt, int32_t cnt_copies,
                       long long cnt_stride, int32_t *childmap, const uint32_t *bm, int32_t *bmx, long long *keyword,
                       int4 *sel, unsigned long long *head, unsigned int *err, int32_t *lnode, const uint32_t *reg);
// Canonicality of the selected candidates (gs_ismin.cu) and the wave's results:
// the low two bits of sel[i].w (above them the candidate's node) = 1 minimal, 0
// not minimal, 2 left to the host (all of them when !check).  codes = the
// wave's code table (a uint2 per edge: from | to << 8 | edge label << 16, from
// label | to label << 16).  The first hcap candidates and then the header go to
// pinned host memory (hsel, hhead), with bytes = the column kernels' byte
// counters and stamps = every context's materialise stamps, the sequence word
// last.
struct ResultsOut {
  int4 *hsel;
  long long hcap;
  unsigned long long *hhead;
  unsigned long long seq;
  const unsigned long long *bytes;
  const unsigned long long *stamps;
  int nctx;
};
KernelCall is_min_call(const NodeDesc *nodes, int32_t nnodes, const SlotDesc *slots, const DevDB *dbs,
                       const uint2 *codes, int4 *sel, int32_t sel_cap, unsigned long long *head, bool check,
                       const ResultsOut &out);
// Children to materialise: their tables (n16 16-byte pieces, in pinned host
// memory) copied to dst, childmap[pairs[i].x] = pairs[i].y, cursor[0..ncursor)
// = 0, bit pairs[i].x of chosen (may be null) set, and the context's
// materialise stamps started.
void launch_children(void *dst, const void *src, long long n16, const int2 *pairs, int32_t n, int32_t *childmap,
                     uint32_t *chosen, int32_t *cursor, int32_t ncursor, unsigned long long *stamps, cudaStream_t s);

// Lists strategy: the per-row lists of a wave's nodes' frequent forward
// extensions, built from the count pass's records (ListBuild, gs_lists.cuh):
// the records materialise pass adds each list row's entry count at off[r + 1]
// (off zeroed before), then launch_fill_lists turns the counts into offsets
// off[0..nrows_total] and writes ent[off[r] ..], the entries {neighbour, the
// node's forward key} of list row r; entries past ent_cap set err bit 4 and
// are dropped.  scratch holds list_scan_scratch(nrows_total) ints.
// The lists of one wave: lnode[wave key] = the node of a frequent forward key
// (else -1); node n's rows are list rows rowbase[n] .. (rowbase[n] < 0: the
// node keeps no lists).
struct ListBuild {
  const int32_t *lnode;
  const NodeDesc *nodes;
  const int32_t *rowbase;
};
int64_t list_scan_scratch(int64_t n);

// The reference's packed segmented scan (cuda_segmented_scan::scan,
// src/reduction/cuda_segmented_scan.hpp): bit 31 of an element starts a new
// segment, bits 0-30 are its value; out[i] = the sum of the values of i's
// segment up to i (inclusive) or before i (exclusive), modulo 2^32.
// scratch: segmented_scan_scratch(n) ints.  out may alias x.
int64_t segmented_scan_scratch(int64_t n);
void launch_segmented_scan(const uint32_t *x, int64_t n, int exclusive, int32_t *scratch, uint32_t *out,
                           cudaStream_t s);
// res[j] = scanned[ends[j]]; an index outside [0, n) sets bit 0 of *err.
void launch_gather_ends(const uint32_t *scanned, int64_t n, const long long *ends, int64_t m, uint32_t *res,
                        unsigned int *err, cudaStream_t s);

// Backward child column on its own (gs_filter_backward; the reference's
// filter_backward_embeddings, src/gspan_cuda/filter_backward.cpp:288-352):
// out = the elements of col at the rows named by the records (8 ints each,
// {from, to, fromlabel, elabel, tolabel, from_grph, to_grph, row}) equal to
// the edge e[0..5), in row order; pos[nrows + 1] (zeroed by the caller) ends
// holding the exclusive scan of the row flags (pos[nrows] = the count).  scratch holds
// filter_backward_scratch(nrows) ints.
int64_t filter_backward_scratch(int64_t nrows);
void launch_filter_backward(const int2 *col, int64_t nrows, const int32_t *rec, int64_t nrec, const int32_t *e,
                            int32_t *pos, int32_t *scratch, int2 *out, cudaStream_t s);
void launch_fill_lists(const int4 *rec, const uint32_t *reg, long long rec_cap, long long most, const ListBuild &lb,
                       int32_t *off, int64_t nrows_total,
                       int2 *ent, int64_t ent_cap, int32_t *scratch, unsigned int *err, cudaStream_t s);

}  // namespace gsgb
