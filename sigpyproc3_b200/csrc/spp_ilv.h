// Host interface of the interleaved bit-plane DM-time kernels (spp_ilv.cu),
// used by the DM plans in spp_core.cu.
#pragma once

#include <vector>

#include "spp_common.cuh"

namespace spp {

// One kernel shape: rows of `G` summed channels (NP bit planes), DW trials x
// W words per CTA.
struct IlvCfg {
  int nb;       // sample width, bits
  int G;        // channels summed per row
  int np;       // bit planes per row
  int P;        // words per thread
  int DW, TW;   // trials per CTA, warps per trial
  int nq;       // quads of groups per slab
  int levels;   // counter levels
  int threads;
  int64_t hi_bytes;  // counter levels kept in shared memory
  const void* fn;
  double us_wave, ns_group;  // measured time of one wave of CTAs: us_wave + groups x ns_group
  int words() const { return TW * 32 * P; }  // words per CTA tile
};
const std::vector<IlvCfg>& ilv_cfgs();

// Rows of one grouping (G channels) of a delay table: row e of group g covers
// the words [lo, lo + words + ext) of its first channel's grid.
struct IlvRows {
  int G = 0;
  int64_t nrows = 0;       // rows over all groups
  int64_t ext_total = 0;   // words beyond the common row length, all rows
  int64_t max_ext = 0;     // the same, widest row
  int64_t max_group = 0;   // G = 1: words beside M that the rows a turning CTA owns span, most
  int32_t* d_lo = nullptr;     // device, nrows: first word of the row (multiple of 8)
  int32_t* d_ext = nullptr;    // device, nrows + 1: prefix sums of the extra words
  int max_offsets = 0;         // G = 2: relative offsets of one pair, most
  int32_t* d_rbase = nullptr;  // device, G = 2, pairs + 1: first row of each pair
  int32_t* d_rlo = nullptr;    // device, G = 2: smallest relative offset of each pair
};

// Staging tables of one kernel shape for one delay table.
struct IlvTables {
  int emax = 0;          // staged rows per slab, most
  int64_t stage_bytes = 0;
  int stages = 0;
  int64_t smem = 0;
  int32_t* d_off = nullptr;  // (tile, slab, trial, group): byte offset in the stage
  int4* d_ent = nullptr;     // (tile, slab, entry): row, word offset, words, stage position
  bool own = false;          // d_off is an allocation (of both), not a plan's room
  int64_t bytes = 0;         // of both
  bool no_memory = false;    // the last attempt found no memory for them
};

// A delay table on the device.
struct IlvDelays {
  const int32_t* d_delays;  // ndm x nchans
  int64_t ndm, nchans;
  int sign;
  int nb;  // sample width, bits
};

// Device words that ilv_find needs for at most `max_rows` pair rows.
int64_t ilv_plan_words(int64_t nchans, int64_t max_rows);
// Bytes that the tables of any shape of this width may take.
int64_t ilv_table_room(int nb, int64_t nchans, int64_t ndm);

void ilv_free_tables(IlvTables* t);
// Range of a table's offsets, and the widest spread over tiles of four and of
// eight trials.
struct IlvRange {
  int32_t omin, omax, span4, span8;
};
// One pass over a delay table: its range, the rows of both groupings (nrows = 0:
// none, as more than `max_rows` pair rows) and the staging sizes of the shapes
// `which` (stages = 0: the spreads do not fit).  `words`: device words that the
// rows live in, on an 8-byte boundary.
int ilv_find(const std::vector<int>& which, const IlvDelays& d, int64_t max_rows, int32_t* words,
             IlvRange* range, IlvRows* rows, std::vector<IlvTables>* tabs);
// Device bytes that the tables of a sized shape take.
int64_t ilv_table_bytes(const IlvCfg& c, const IlvDelays& d, const IlvTables& t);
// Builds them in `room` where it is large enough, else in memory of their own.
int ilv_build_tables(const IlvCfg& c, const IlvDelays& d, const IlvRows& r, void* room, int64_t room_bytes,
                     IlvTables* t);

struct IlvGeom {
  int64_t M;        // words per row that carry outputs (32 * M >= nvalid)
  int64_t mp;       // words of a row without its extra words
  int64_t chan_bytes, row_bytes;  // channel rows, pair rows (0 for G = 1)
};
IlvGeom ilv_geometry(const IlvCfg& c, const IlvRows& chan, const IlvRows& rows, int64_t nchans,
                     int64_t nvalid);
// Raw block -> channel rows (and pair rows) in `ws`.
int ilv_corner_turn(const IlvCfg& c, const IlvRows& chan, const IlvGeom& g, const void* in,
                    int bitorder, int64_t nchans, int64_t nsamps, void* ws, cudaStream_t st);
int ilv_group_rows(const IlvCfg& c, const IlvRows& chan, const IlvRows& rows, const IlvGeom& g,
                   int64_t nchans, void* ws, cudaStream_t st);
int ilv_launch(const IlvCfg& c, const IlvTables& t, const IlvRows& rows, const IlvGeom& g,
               int64_t ngroups, int64_t ndm, const void* ws, void* out, int out_kind,
               int64_t out_stride, int64_t out_start, int64_t nvalid, uint32_t* status,
               cudaStream_t st);

}  // namespace spp
