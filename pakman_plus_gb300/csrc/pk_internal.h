// Internal launcher interface between the C-ABI host runtime (pk_capi.cpp) and the
// sm_103a kernels (pk_kernels.cu).  Not part of the public ABI.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/pakman_gb300.h"

namespace pk {

// Records the calling thread's last-error text (pk_last_error) and returns s.
pk_status set_error(pk_status s, const std::string& msg);

// Counts one kernel launch made by this library (read by pk_kernel_launches); every
// launch site calls it as `note_launch(), kernel<<<...>>>(...)`.
void note_launch();

// Device error word bits (pk_job error flag).
enum : uint32_t {
  ERR_FORMAT = 1u,        // a record start is not '>' (reference asserts)
  ERR_LOOKBACK = 2u,      // a bounded look-back wait ran out
  ERR_BUCKET = 4u,        // a bucket could not be split small enough for on-chip counting
  ERR_MN_CAPACITY = 8u,   // a macro-node segment exceeded on-chip capacity
  ERR_BOUNDS = 32u,       // a computed index fell outside its buffer (write skipped)
};

constexpr int kTileBytes = 65536;   // line-scan tile; chunk boundaries are multiples of it
constexpr int kSegBytes = 64;       // bytes per thread per extraction step
constexpr int kMnThreads = 256;
constexpr int kMnCap = 1568;        // items per segment of a sorted unit
constexpr int kMnFit = kMnCap - 16; // rows per segment before ties; both sides of a joined unit
constexpr int kMnJoin = 768;        // items a side of a joined macro-node unit
constexpr int kSmallCounts = 16;    // per-bucket histogram of the table kernel: counts 0..15
constexpr int kMnBinBits = 9;       // counting-sort bins of a macro-node segment
constexpr int kMnBins = 1 << kMnBinBits;
constexpr int kMnBinMax = 32;       // largest bin ranked within itself (else merge ranks)
constexpr int kHistSmem = 1024;     // count-histogram bins kept in shared memory
constexpr int kBucketStack = 256;   // pending sub-ranges of one bucket
constexpr int kSplitWays = 4;      // pieces an overflowing sub-range is cut into
constexpr int kSplitSamples = 256; // distinct keys sampled for the cut
constexpr int kTableHist = 512;    // count-histogram bins the table kernel keeps on chip
constexpr int kMaxBucketAttempts = 1 << 16;  // sub-range attempts per bucket before giving up
constexpr int kCoarseBits = 7;     // pass-1 partition digits (coarse regions)
constexpr int kMaxPartBits = 18;   // partition digits (table buckets) at most
constexpr int kHistBits = 15;      // digits the counting pass histograms in shared memory
constexpr int kSortBinBits = 10;    // top remainder bits of the per-bucket counting sort
constexpr int kBinMax = 128;        // largest bin sorted by ranking (else bitonic sort)
// Giant buckets (skewed input: a homopolymer or tandem repeat and its error variants)
// are first reduced chunk by chunk, by many CTAs, to (key, count) pairs.
constexpr uint32_t kGiantKeys = 1u << 19;           // a bucket this large is giant
constexpr int kGiantParts = 16;                     // work items that count one giant bucket
constexpr uint32_t kChunkRaw = 0xffffffffu;         // chunk left as keys (too many distinct)

struct Scalars {                    // device-side scalars of one job
  unsigned long long s0;            // index of the first '>' (F if none)
  unsigned long long n_windows;     // number of k-mer instances
  unsigned long long n_reads;       // number of '>' bytes from s0 on
  uint32_t nl_before_s0;            // newlines in [0, s0)
  uint32_t err;                     // ERR_* bits
  uint32_t ticket_bucket;           // work tickets
  uint32_t cutoff;                  // histogram cutoff
  uint32_t ticket_fine;
  uint32_t ticket_fcount;
  uint32_t n_chunk_items;           // chunk items of giant buckets (table kernel)
  uint32_t n_giants;                // giant buckets
  uint32_t part_beats;              // passes of giant buckets' parts so far
  unsigned long long n_unique;      // U
  unsigned long long n_kept;        // V
  // zeroed together before macro-nodes are built
  unsigned long long mn_begin[0];
  unsigned long long n_nodes;       // M
  uint32_t ticket_mn;
  uint32_t ticket_filter;
  uint32_t n_big;                   // macro-node units of more than one segment
  uint32_t mn_end[0];
};

struct CountArgs {
  const uint8_t* fasta;
  unsigned long long F;
  int k;
  int lmer_m;        // min(k, LMER_LENGTH): record-start checks follow the l-mer pass
  int drop_n;
  int bbits;         // bucket bits (top bits of the 2k-bit key)
  int cbits;         // coarse bits of the pass-1 partition (<= bbits, <= kCoarseBits)
  int grid;          // extraction CTAs (chunks)
  unsigned long long chunk;  // bytes per chunk (multiple of kTileBytes)
  uint32_t* tile_nl;         // ceil(F / kTileBytes) + 1, exclusive newline prefix
  uint32_t* counts;          // grid x 2^bbits  (per-chunk bucket counts, then prefixes)
  uint32_t* bstart;          // 2^bbits + 1 bucket starts
  unsigned long long n_keys; // capacity of the bucketed key buffer (scatter pass)
  Scalars* sc;
  // Packed units written by the counting pass and rolled again by the coarse scatter.
  // Unit u (0..3) of kSegBytes-byte segment g (its bytes 16u..16u+15) sits at
  // [u * nseg + g] of the code and bit-2 planes; windows[g] has bit 16u + j set iff the
  // window whose newest byte is byte j of that unit was counted.  The bit-2 plane holds the
  // segment's sequence bytes; unit 3's word is always written, with bit 1 set when the
  // segment has any such byte, the other three only then.
  uint32_t* unit_codes;      // 4 x nseg
  uint32_t* unit_nbits;      // 4 x nseg
  unsigned long long* unit_windows;  // nseg
  unsigned long long nseg;   // ceil(F / kSegBytes)
};

// The table is kept "sparse": the u rows of bucket b sit at [bstart[b], bstart[b] + u),
// inside the bucket's own key range, ascending.
struct BucketArgs {
  void* keys;                // bucketed keys (uint64 or u128), N entries; chunks of giant
                             // buckets are rewritten in place as (key, count) pairs
  const uint32_t* bstart;    // 2^bbits + 1
  void* tkeys;               // table keys out (N capacity)
  uint32_t* tcounts;         // table counts out (N capacity)
  uint32_t* tu;              // 2^bbits: rows per bucket
  unsigned long long* hist;  // t bins (zeroed)
  int t;
  int k;
  int bbits;
  unsigned long long cap;    // table capacity (rows)
  const uint32_t* gfirst;    // 2^bbits: first chunk item of each giant bucket (null: none)
  const uint32_t* gcount;    // 2^bbits: its chunk items (0: not giant)
  const uint32_t* chunk_bucket;  // per chunk item: its bucket
  uint32_t* gdone;           // 2^bbits: chunk items of the bucket finished
  uint32_t* chunk_u;         // per chunk item: pairs it left, or kChunkRaw
  // per giant bucket kGiantParts look-back words (rows up to the part's end), and its bucket
  unsigned long long* gpart;
  const uint32_t* glist;
  uint32_t* bsmall;          // kSmallCounts x 2^bbits: rows of each bucket by count < kSmallCounts
  int spin_limit;            // polls of a bounded wait before it gives up (0: default)
  Scalars* sc;
};

// Kept rows (count >= cutoff), dense and ascending, with per-bucket extents.
struct FilterArgs {
  const void* tkeys;
  const uint32_t* tcounts;
  const uint32_t* bstart;
  const uint32_t* tu;
  unsigned long long* flags; // look-back words of the offsets, one per 256 buckets (zeroed)
  void* kkeys;               // kept keys out
  uint32_t* kcounts;         // kept counts out
  uint32_t* kstart;          // 2^bbits
  uint32_t* kcount;          // 2^bbits
  uint32_t* ksub;            // 3 * 2^bbits
  unsigned long long cap;    // kept-row capacity
  unsigned long long trows;  // rows the table count buffer holds (reads stay below)
  // the table kernel's rows per bucket by count below kSmallCounts (null: not known);
  // with a cutoff <= kSmallCounts a bucket's kept rows follow from them and its row count
  const uint32_t* bsmall;
  int k;
  int bbits;
  int spin_limit;            // polls of a bounded wait before it gives up (0: default)
  Scalars* sc;
};

struct MnArgs {
  const void* kkeys;
  const uint32_t* kcounts;
  const uint32_t* kstart;
  const uint32_t* kcount;
  const uint32_t* ksub;
  unsigned long long* flags; // mn_flag_words(bbits) look-back words (zeroed)
  uint32_t* big;             // 2^bbits: the units of more than one segment
  void* nkeys;               // node keys out (capacity cap)
  uint32_t* nsuf;            // 4 * cap
  uint32_t* npre;            // 4 * cap
  unsigned long long cap;
  unsigned long long kcap;   // kept rows the kept buffers hold
  int k;
  int bbits;
  int xbits;                 // node units cover 2^xbits table buckets' node keys
  int spin_limit;            // polls of a bounded wait before it gives up (0: default)
  int withhold_unit;         // a unit that publishes no look-back word (-1: none; tests of
                             // the bounded waits)
  Scalars* sc;
};

// One macro-node's initial wiring (the pk_wiring layout of the C ABI).
struct WireRow {
  int32_t ns, np, term_suf, term_pre, nw;
  int32_t wire[9][3];
  int32_t begin[5][2];
};

// Launchers (all stream-ordered, no host synchronisation).
// SM count the calling thread's launches are sized for (a serving worker on an SM
// partition sets its partition's count; 0 restores the whole device)
void set_thread_sms(int n);
int thread_sms(int device_sms);

cudaError_t launch_line_scan(const CountArgs& a, cudaStream_t st);
// chunk items of the giant buckets (n_b >= kGiantKeys): floor(n_b / chunk_keys)
// consecutive items each, from gfirst[b], gcount[b] of them; chunk_bucket maps an item
// to its bucket; sc->n_chunk_items = all items; sc->n_giants and glist: the buckets; gdone,
// gpart and the giants' rows of bsmall = 0
int chunk_keys(int wide);
cudaError_t launch_giant_chunks(const BucketArgs& a, int wide, uint32_t* gfirst, uint32_t* gcount,
                                uint32_t* chunk_bucket, uint32_t* glist, cudaStream_t st);
size_t giant_part_bytes(unsigned long long keys);  // gpart, then glist
// the line scan in two halves: per-tile newline counts for tiles [tile0, tile0 + ntiles)
// (any order, any number of launches), then the prefix over all tiles
cudaError_t launch_line_tiles(const uint8_t* buf, unsigned long long F, uint32_t* tile_nl, Scalars* sc,
                              unsigned long long tile0, unsigned long long ntiles, cudaStream_t st);
cudaError_t launch_tile_prefix(const CountArgs& a, cudaStream_t st);
cudaError_t launch_bucket_count(const CountArgs& a, int wide, cudaStream_t st);
cudaError_t launch_fine_count(const void* in, const uint32_t* cstart, const uint32_t* slice_start,
                              uint32_t* bcount, int k, int bbits, int cbits, int wide, uint32_t* ticket,
                              cudaStream_t st);
cudaError_t launch_prefix(uint32_t* counts, int B, cudaStream_t st);
cudaError_t launch_wire(const void* nsuf, const void* npre, unsigned long long m, int coverage, WireRow* out,
                        cudaStream_t st);
// batch: reserve a set's rows in the batch macro-node table and copy them there
cudaError_t launch_batch_emit(const Scalars* sc, unsigned long long* counter, unsigned long long cap,
                              unsigned long long* res, const void* nkeys, const void* nsuf, const void* npre,
                              int wide, void* okeys, void* osuf, void* opre, cudaStream_t st);
cudaError_t launch_bucket_offsets(const CountArgs& a, cudaStream_t st);
// Two-pass partition: coarse regions (pass 1) then fine buckets inside each region.
// keys per pass-2 slice for a fan-out of 2^fb fine buckets per coarse region
int fine_slice_keys(int wide, int fb);
// also, when the histogram has the partition's pbits digits, its bucket starts (bstart) and
// the fine scatter's cursors (fcur); zeroes the fine scatter's ticket
cudaError_t launch_coarse_offsets(const CountArgs& a, int pbits, uint32_t* coff, uint32_t* cstart,
                                  uint32_t* slice_start, int slice_keys, uint32_t* bstart, uint32_t* fcur,
                                  cudaStream_t st);
cudaError_t launch_scatter_coarse(const CountArgs& a, const uint32_t* coff, void* out, int wide,
                                  cudaStream_t st);
cudaError_t launch_scatter_fine(const void* in, const uint32_t* cstart, const uint32_t* slice_start,
                                uint32_t* fcur, void* out, int k, int bbits, int cbits, int wide,
                                uint32_t* ticket, unsigned long long cap, uint32_t* err, cudaStream_t st);
cudaError_t launch_bucket_table(const BucketArgs& a, int wide, int grid, cudaStream_t st);
// checks the rows of a loaded table and histograms their counts below t (hist null: not
// wanted); chk = {all ones, 0} beforehand, {4 * first bad row + rule, sum of counts} after
// (rule 0: not a k-mer, 1: not above the row before, 2: count 0)
cudaError_t launch_table_check(const void* keys, const uint32_t* counts, unsigned long long n, int k, int wide,
                               unsigned long long* chk, int t, unsigned long long* hist, cudaStream_t st);
// bstart / tu of a dense ascending table (pk_table_load)
cudaError_t launch_table_bounds(const void* keys, unsigned long long n, int bbits, int k, uint32_t* bstart,
                                uint32_t* tu, int wide, cudaStream_t st);
// rows by count below t of the table in its buckets (hist zeroed beforehand)
cudaError_t launch_histogram(const uint32_t* tcounts, const uint32_t* bstart, const uint32_t* tu, int B, int t,
                             unsigned long long* hist, cudaStream_t st);
cudaError_t launch_cutoff(const unsigned long long* hist, int t, Scalars* sc, cudaStream_t st);
// count_rows: the cutoff may be above what the small-count histograms tell, or there are none
cudaError_t launch_filter_kept(const FilterArgs& a, int wide, bool count_rows, cudaStream_t st);
size_t mn_flag_words(int bbits);  // look-back words of the macro-node kernel
cudaError_t launch_macro_nodes(const MnArgs& a, int wide, int grid, cudaStream_t st);
// Dense copy of the sparse table (doff: exclusive prefix of tu, computed by
// launch_row_offsets).  packed != null writes KmerPairs records instead of arrays.
cudaError_t launch_row_offsets(const uint32_t* tu, uint32_t* doff, int B, cudaStream_t st);
cudaError_t launch_compact_rows(const void* tkeys, const uint32_t* tcounts, const uint32_t* bstart,
                                const uint32_t* tu, const uint32_t* doff, int B, int wide,
                                void* dkeys, uint32_t* dcounts, void* packed, cudaStream_t st);

size_t bucket_smem_bytes(int wide);
size_t mn_smem_bytes(int wide);
int bucket_ctas_per_sm(int wide);
int mn_ctas_per_sm(int wide);

}  // namespace pk
