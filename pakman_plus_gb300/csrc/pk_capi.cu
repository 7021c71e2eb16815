// Host runtime behind the C ABI (include/pakman_gb300.h): contexts with an HBM
// budget, jobs that own their device buffers, and the stream-ordered launch
// sequence of the counting -> cutoff -> macro-node path.  No CPU fallback: every
// result comes from the kernels in pk_kernels.cu.
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <iterator>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/pakman_gb300.h"
#include "pk_internal.h"
#include "pk_runtime.h"

using namespace pk;

static const int kMaxPartitionBits = kMaxPartBits;

// ------------------------------------------------------------------ errors ------
static thread_local std::string t_last_error;

static pk_status fail(pk_status s, const std::string& msg) {
  t_last_error = msg;
  return s;
}

pk_status pk::set_error(pk_status s, const std::string& msg) { return fail(s, msg); }


pk_status pk::set_device(pk_ctx* c) {
  PK_CUDA(cudaSetDevice(c->device));
  return PK_OK;
}

// ------------------------------------------------------------ device blocks -----
// A cached block of at least `bytes`: up to an eighth (or 64 KB) larger, but with a budget of
// just that size, as every byte of it counts there.
static void* cache_take(pk_ctx* c, size_t bytes, size_t* block) {
  const size_t most = c->budget ? bytes : std::max(bytes + bytes / 8, bytes + 65536);
  std::lock_guard<std::mutex> lk(c->cache_mu);
  auto it = c->cache.lower_bound(bytes);
  if (it == c->cache.end() || it->first > most) return nullptr;
  void* p = it->second;
  *block = it->first;
  c->cached -= it->first;
  c->cache.erase(it);
  return p;
}

// Gives the cached blocks back to the pool when they are more than `keep` bytes: all of them,
// as the pool joins what is free and a block here and there leaves it pieces that nothing fits.
static void cache_trim(pk_ctx* c, uint64_t keep) {
  std::lock_guard<std::mutex> lk(c->cache_mu);
  if (c->cached <= keep) return;
  for (auto& b : c->cache) cudaFree(b.second);  // idle: nothing to wait for
  c->cache.clear();
  c->cached = 0;
}

static void cache_put(pk_ctx* c, DevBuf& b) {
  if (b.p) {
    c->used -= b.bytes;
    bool room;
    {
      // what is in use is read under the lock: an allocation that is not in it yet trims later
      std::lock_guard<std::mutex> lk(c->cache_mu);
      uint64_t keep = c->cache_limit;
      if (c->budget) keep = std::min<uint64_t>(keep, c->budget - std::min<uint64_t>(c->budget, c->used.load()));
      // the largest blocks make room: a job of few bytes is the one that feels an allocation
      while (c->cached + b.bytes > keep && !c->cache.empty()) {
        auto it = std::prev(c->cache.end());
        if (it->first <= b.bytes) break;
        cudaFree(it->second);  // idle: nothing to wait for
        c->cached -= it->first;
        c->cache.erase(it);
      }
      room = c->cached + b.bytes <= keep;
      if (room) {
        c->cache.emplace(b.bytes, b.p);
        c->cached += b.bytes;
      }
    }
    if (!room) cudaFree(b.p);
  }
  b = DevBuf{};
}

// Every device buffer of the context comes from here: charged whole to the budget, which
// blocks in use and cached blocks share.
pk_status pk::ctx_alloc(pk_ctx* c, cudaStream_t st, DevBuf& b, size_t bytes) {
  bytes = std::max<size_t>(256, (bytes + 255) & ~(size_t)255);
  uint64_t now = c->used.fetch_add(bytes) + bytes;
  if (c->budget && now > c->budget) {
    c->used -= bytes;
    return fail(PK_ERR_NOMEM, "HBM budget exceeded: need " + std::to_string(bytes) + " more bytes, " +
                                  std::to_string(now - bytes) + " of " + std::to_string(c->budget) +
                                  " in use");
  }
  size_t block = bytes;
  void* p = cache_take(c, bytes, &block);
  if (!p) {
    if (c->budget) cache_trim(c, c->budget - now);  // what is in use and what is kept stay within it
    cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, c->pool, st);
    if (e != cudaSuccess) {
      cudaGetLastError();
      cache_trim(c, 0);
      e = cudaMallocFromPoolAsync(&p, bytes, c->pool, st);
    }
    if (e != cudaSuccess) {
      c->used -= bytes;
      return fail(PK_ERR_NOMEM, std::string("device allocation failed: ") + cudaGetErrorString(e));
    }
  }
  c->used += block - bytes;
  b.p = p;
  b.bytes = block;
  return PK_OK;
}

pk_status pk::job_alloc(pk_job* j, DevBuf& b, size_t bytes) {
  if (b.p && b.bytes >= bytes) return PK_OK;
  if (j->graph_mode) return fail(PK_ERR_STATE, "batch buffers are smaller than a set needs");
  job_free(j, b);
  return ctx_alloc(j->ctx, j->stream, b, bytes);
}

void pk::job_free(pk_job* j, DevBuf& b) {
  if (b.p) {
    cudaFreeAsync(b.p, j->stream);
    j->ctx->used -= b.bytes;
  }
  b = DevBuf{};
}

void pk::job_free_idle(pk_job* j, DevBuf& b) { cache_put(j->ctx, b); }

int pk::job_buffers(pk_job* j, DevBuf** out, int cap) {
  DevBuf* all[] = {&j->fasta, &j->tile_nl, &j->counts, &j->bstart, &j->hstart, &j->keys,  &j->tkeys,
                   &j->tcounts, &j->tu,    &j->flags_m, &j->hist,  &j->hist2,
                   &j->nkeys,  &j->nsuf,   &j->npre,    &j->packed,  &j->doff,  &j->dkeys,
                   &j->dcounts, &j->kkeys, &j->kcounts, &j->kstart, &j->kcount,
                   &j->ksub,  &j->coff,    &j->cstart,  &j->slice_start, &j->fcur, &j->wiring,
                   &j->gfirst, &j->gcount, &j->chunk_bucket, &j->gdone,
                   &j->chunk_u, &j->gpart, &j->acc_keys[0], &j->acc_keys[1], &j->acc_counts[0], &j->acc_counts[1],
                   &j->merge_keys, &j->merge_counts, &j->merge_part, &j->units, &j->bsmall};
  const int n = (int)(sizeof(all) / sizeof(all[0]));
  for (int i = 0; i < n && i < cap; i++) out[i] = all[i];
  return n;
}

void pk::job_free_all(pk_job* j) {
  DevBuf* all[64];
  const int n = job_buffers(j, all, 64);
  const bool idle = cudaStreamSynchronize(j->stream) == cudaSuccess;
  for (int i = 0; i < n; i++) {
    if (idle) job_free_idle(j, *all[i]);
    else job_free(j, *all[i]);
  }
  j->bsmall_valid = false;
  cp_free(j);
  j->compacted = false;
  j->dense_valid = false;
}

void pk::release_piece_buffers(pk_job* j) {
  DevBuf* all[64];
  const int n = job_buffers(j, all, 64);
  for (int i = 0; i < n; i++)
    if (all[i] != &j->tkeys && all[i] != &j->tcounts) job_free(j, *all[i]);
  j->dense_valid = false;
}

// per-stage CUDA events on the job's stream (begin/end pairs, so host-side gaps
// between stages are not charged to a kernel)
void pk::mark_begin(pk_job* j, int st) {
  if (j->timing) cudaEventRecord(j->ev0[st], j->stream);
}
void pk::mark_end(pk_job* j, int st) {
  if (j->timing) {
    cudaEventRecord(j->ev1[st], j->stream);
    j->ev_rec[st] = true;
  }
}

// ---------------------------------------------------------------- C ABI ---------
void pk_params_default(pk_params* p) {
  if (!p) return;
  memset(p, 0, sizeof(*p));
  p->k = 32;
  p->lmer_length = 8;
  p->num_buckets = 21;
  p->coverage = 1;
  p->read_length = 100;
  p->drop_n = 0;
  p->batch_kmers = 100000000ull;
  p->bucket_bits = 0;
}

const char* pk_status_string(pk_status s) {
  switch (s) {
    case PK_OK: return "ok";
    case PK_ERR_INVALID: return "invalid argument";
    case PK_ERR_FORMAT: return "FASTA record does not start with '>'";
    case PK_ERR_EMPTY: return "no k-mer reaches the histogram cutoff";
    case PK_ERR_NOMEM: return "out of device memory or HBM budget";
    case PK_ERR_CUDA: return "CUDA error";
    case PK_ERR_STATE: return "call out of order";
    case PK_ERR_LIMIT: return "input beyond supported size";
    case PK_ERR_DEVICE: return "device-side failure";
    case PK_ERR_BUSY: return "busy";
    case PK_ERR_NO_DEVICE: return "no CUDA device";
    case PK_ERR_IO: return "input file cannot be read";
    case PK_ERR_CANCELLED: return "cancelled";
  }
  return "unknown status";
}

const char* pk_last_error(void) { return t_last_error.c_str(); }

const char* pk_version(void) { return "pakman-gb300 0.1 (sm_103a)"; }

pk_status pk_ctx_create(int device, uint64_t budget, pk_ctx** out) {
  if (!out) return fail(PK_ERR_INVALID, "out is null");
  *out = nullptr;
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n <= 0)
    return fail(PK_ERR_NO_DEVICE, std::string("no CUDA device: ") + cudaGetErrorString(e));
  if (device < 0 || device >= n) return fail(PK_ERR_INVALID, "device index out of range");
  PK_CUDA(cudaSetDevice(device));
  pk_ctx* c = new pk_ctx();
  c->device = device;
  c->budget = budget;
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  e = cudaMemPoolCreate(&c->pool, &props);
  if (e != cudaSuccess) {
    delete c;
    return fail(PK_ERR_CUDA, std::string("cudaMemPoolCreate: ") + cudaGetErrorString(e));
  }
  uint64_t thr = ~0ull;
  cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &thr);
  cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device);
  size_t mem_free = 0, mem_total = 0;
  if (cudaMemGetInfo(&mem_free, &mem_total) != cudaSuccess) cudaGetLastError();
  c->cache_limit = mem_total / 8;
  *out = c;
  return PK_OK;
}

void pk_ctx_destroy(pk_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  cudaDeviceSynchronize();
  cache_trim(c, 0);
  if (c->pool) cudaMemPoolDestroy(c->pool);
  delete c;
}

pk_status pk_ctx_memory(pk_ctx* c, uint64_t* used, uint64_t* budget) {
  if (!c) return fail(PK_ERR_INVALID, "ctx is null");
  if (used) *used = c->used.load();
  if (budget) *budget = c->budget;
  return PK_OK;
}

pk_status pk_job_create(pk_ctx* c, void* stream, pk_job** out) {
  if (!c || !out) return fail(PK_ERR_INVALID, "null argument");
  PK_TRY(set_device(c));
  pk_job* j = new pk_job();
  j->ctx = c;
  if (stream) {
    j->stream = (cudaStream_t)stream;
  } else {
    cudaError_t e = cudaStreamCreateWithFlags(&j->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
      delete j;
      return fail(PK_ERR_CUDA, std::string("cudaStreamCreate: ") + cudaGetErrorString(e));
    }
    j->own_stream = true;
  }
  cudaError_t e = cudaMalloc(&j->d_sc, sizeof(Scalars));
  if (e == cudaSuccess) e = cudaHostAlloc(&j->h_sc, sizeof(Scalars), cudaHostAllocDefault);
  if (e != cudaSuccess) {
    if (j->d_sc) cudaFree(j->d_sc);
    if (j->own_stream) cudaStreamDestroy(j->stream);
    delete j;
    return fail(PK_ERR_NOMEM, std::string("job scalars: ") + cudaGetErrorString(e));
  }
  memset(j->h_sc, 0, sizeof(Scalars));
  for (int i = 0; i < ST_COUNT_; i++) {
    cudaEventCreate(&j->ev0[i]);
    cudaEventCreate(&j->ev1[i]);
  }
  *out = j;
  return PK_OK;
}

void pk_job_destroy(pk_job* j) {
  if (!j) return;
  cudaSetDevice(j->ctx->device);
  job_free_all(j);
  cudaStreamSynchronize(j->stream);
  for (int i = 0; i < ST_COUNT_; i++) {
    if (j->ev0[i]) cudaEventDestroy(j->ev0[i]);
    if (j->ev1[i]) cudaEventDestroy(j->ev1[i]);
  }
  if (j->d_sc) cudaFree(j->d_sc);
  if (j->h_sc) cudaFreeHost(j->h_sc);
  if (j->cp_dev) cudaFree(j->cp_dev);
  if (j->cp_host) cudaFreeHost(j->cp_host);
  for (int i = 0; i < pk_job::kIngestBufs; i++) {
    if (j->ing_host[i]) cudaFreeHost(j->ing_host[i]);
    if (j->ing_ev[i]) cudaEventDestroy(j->ing_ev[i]);
  }
  if (j->own_stream) cudaStreamDestroy(j->stream);
  delete j;
}

pk_status pk_job_reset(pk_job* j) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  PK_TRY(set_device(j->ctx));
  job_free_all(j);
  j->stage = 0;
  j->wired = false;
  PK_CUDA(cudaStreamSynchronize(j->stream));
  return PK_OK;
}

pk_status pk_job_sync(pk_job* j) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  PK_TRY(set_device(j->ctx));
  PK_CUDA(cudaStreamSynchronize(j->stream));
  return PK_OK;
}

pk_status pk_job_memory(pk_job* j, uint64_t* bytes) {
  if (!j || !bytes) return fail(PK_ERR_INVALID, "null argument");
  DevBuf* all[64];
  const int n = job_buffers(j, all, 64);
  uint64_t s = 0;
  for (int i = 0; i < n; i++) s += all[i]->bytes;
  *bytes = s;
  return PK_OK;
}

pk_status pk_job_set_wait_limit(pk_job* j, uint32_t spins, int32_t withhold_unit) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (spins > (1u << 30)) return fail(PK_ERR_INVALID, "spins must be at most 2^30");
  j->wait_limit = spins;
  j->withhold_unit = withhold_unit < 0 ? -1 : withhold_unit;
  return PK_OK;
}

pk_status pk_job_enable_timing(pk_job* j, int on) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  j->timing = on != 0;
  return PK_OK;
}

pk_status pk_job_stage_times(pk_job* j, float* ms, int cap, int* n) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  PK_TRY(set_device(j->ctx));
  PK_CUDA(cudaStreamSynchronize(j->stream));
  if (n) *n = ST_COUNT_;
  for (int s = 0; s < ST_COUNT_ && s < cap; s++) {
    float v = 0.f;
    if (j->ev_rec[s]) cudaEventElapsedTime(&v, j->ev0[s], j->ev1[s]);
    ms[s] = v;
  }
  return PK_OK;
}

const char* pk_stage_name(int s) { return (s >= 0 && s < ST_COUNT_) ? kStageNames[s] : ""; }

pk_status pk_host_alloc(uint64_t bytes, void** out) {
  if (!out) return fail(PK_ERR_INVALID, "out is null");
  PK_CUDA(cudaHostAlloc(out, bytes ? bytes : 1, cudaHostAllocDefault));
  return PK_OK;
}

void pk_host_free(void* p) {
  if (p) cudaFreeHost(p);
}

pk_status pk::check_params(const pk_params* p) {
  if (!p) return fail(PK_ERR_INVALID, "params is null");
  if (p->k < 2 || p->k > 64) return fail(PK_ERR_INVALID, "k must be in 2..64");
  if (p->lmer_length < 1 || p->lmer_length > 32) return fail(PK_ERR_INVALID, "lmer_length must be in 1..32");
  if (p->num_buckets < 1) return fail(PK_ERR_INVALID, "num_buckets (-t) must be >= 1");
  if (p->mn_units < 0 || p->mn_units > 16) return fail(PK_ERR_INVALID, "mn_units must be in 0..16");
  if (p->chunking < 0 || p->chunking > 2) return fail(PK_ERR_INVALID, "chunking must be 0, 1 or 2");
  if (p->bucket_bits < 0 || p->bucket_bits > kMaxPartitionBits)
    return fail(PK_ERR_INVALID, "bucket_bits must be in 0.." + std::to_string(kMaxPartitionBits));
  return PK_OK;
}

// Partition digits: the leading key bits that pick a bucket.  The keys reach their buckets
// in two passes (kCoarseBits coarse regions, then fine buckets inside each region), so the
// digit count is not tied to L2 capacity.
//
// Keys per bucket aimed at, by how many buckets that makes.  Many: large enough to amortise
// the per-bucket work of the table and macro-node kernels, small enough that a bucket's
// distinct keys fit half an on-chip hash table (8192 64-bit or 4096 128-bit slots).  Fewer
// than about a thousand: smaller, so that every SM has buckets; a handful: a few hundred.
// Stage sums measured at the neighbours of each choice (us; digits): 20.7k windows 4: 132,
// 6: 130, 8: 151 (two digits, one bucket per 5200 keys: 266 before); 1.7M 8: 203, 9: 195, 10:
// 204; 3.5M 9: 249, 10: 241, 11: 247; 13.8M 10: 504, 11: 464, 12: 488; 83M 12: 2036, 13: 1683,
// 14: 1874; 254M 13: 6450, 14: 5310, 15: 5870; 128-bit keys, 1.9M 9: 273, 10: 264, 12: 295;
// 15M 11: 1285, 12: 895, 13: 959; 70M 13: 3744, 14: 2937, 15: 3356; 568M 17: 28900, 18: 32400.
static int partition_bits(double n, int k, int wide) {
  int b = 2;
  while (b < kMaxPartitionBits) {
    const double most = b < 6 ? 350.0 : wide ? (b < 10 ? 2000.0 : 4500.0)
                                             : (b < 10 ? 3500.0 : b < 12 ? 9000.0 : b < 14 ? 10500.0 : 16000.0);
    if (n / (double)(1u << b) <= most) break;
    b++;
  }
  return std::max(2, std::min(b, 2 * k - 2));
}

// The digits for an input whose windows are not counted yet: windows per byte of 100 bp
// reads at k = 32 and of 100-150 bp reads at k = 63.
int pk::auto_bucket_bits(uint64_t F, int k, int wide) {
  return partition_bits((wide ? 0.45 : 0.62) * (double)F, k, wide);
}

// The digits of a table that is there already (loaded, or merged from pieces): up to 1000 rows
// per bucket, 768 of which a joined macro-node unit takes.  With 4000, units were sorted in
// segments: 5.0M rows, load to macro-nodes, 0.81 ms at 4000, 0.70 at 2000, 0.68 at 1000, 0.69
// at 400.
int pk::row_bits(uint64_t rows, const pk_params* p) {
  int b = p->bucket_bits;
  if (!b) {
    b = 2;
    while (b < kMaxPartitionBits && (double)rows / (double)(1u << b) > 1000.0) b++;
  }
  return std::max(2, std::min(b, std::min(kMaxPartitionBits, 2 * p->k - 2)));
}

// The digits the counting pass histograms when the partition's own follow from its window
// count: enough for long reads (0.85 windows per byte) where a digit more is cheap, as many
// as the histogram holds at most.
static int hist_bits(uint64_t F, int k, int wide) {
  int b = partition_bits(0.62 * (double)F, k, wide);
  if (b < 14) b = std::max(b, std::min(14, partition_bits(0.85 * (double)F, k, wide)));
  return std::min(b, kHistBits);
}

static const char* kFormatError =
    "a FASTA record start is not '>' (one '>' header line and one sequence line per record expected)";

static pk_status table_impl(pk_job* j, uint64_t N, int t);

// Stages 1-5: device FASTA -> sorted (k-mer, count) table, resident.
pk_status pk::count_impl(pk_job* j, const void* d_fasta, uint64_t n, const pk_params* p) {
  const int k = p->k;
  j->params = *p;
  j->wide = k > 32;
  j->F = n;
  j->stage = 0;
  j->sc_fresh = false;
  j->wired = false;
  j->compacted = false;
  const int W = j->wide ? 16 : 8;
  // automatic digits follow from the window count, which the counting pass takes with hb
  // digits first (graph mode and small runs know no counts)
  const bool waits = !j->graph_mode && !j->no_wait;
  const bool by_count = !p->bucket_bits && waits;
  const int bb = p->bucket_bits ? std::min(p->bucket_bits, std::min(kMaxPartitionBits, 2 * k - 2))
                                : auto_bucket_bits(n, k, j->wide);
  j->bbits = std::max(2, bb);
  // the counting pass histograms at most kHistBits digits; deeper partitions get their
  // fine bucket sizes from a count over the coarse regions (k_fine_count)
  const int hb = by_count ? hist_bits(n, k, j->wide) : std::min(j->bbits, kHistBits);
  const int HB = 1 << hb;
  const uint64_t ntiles = (n + kTileBytes - 1) / kTileBytes;
  int grid = (int)std::min<uint64_t>((uint64_t)thread_sms(j->ctx->sms), std::max<uint64_t>(ntiles, 1));
  unsigned long long chunk = (ntiles + grid - 1) / grid * (unsigned long long)kTileBytes;
  if (chunk == 0) chunk = kTileBytes;
  if (j->chunk_mult > 1) chunk *= (unsigned long long)j->chunk_mult;  // fewer, longer chunks
  grid = (int)std::max<uint64_t>(1, (n + chunk - 1) / chunk);
  j->grid = grid;
  j->chunk = chunk;

  PK_TRY(job_alloc(j, j->tile_nl, sizeof(uint32_t) * (ntiles + 1)));
  PK_TRY(job_alloc(j, j->counts, sizeof(uint32_t) * (size_t)grid * HB));
  // packed units: 4 x nseg codes, 4 x nseg bit-2 planes, nseg window masks (10 bytes per
  // 16 input bytes)
  const uint64_t nseg = (n + kSegBytes - 1) / kSegBytes;
  PK_TRY(job_alloc(j, j->units, (size_t)40 * nseg));
  PK_TRY(job_alloc(j, j->hstart, sizeof(uint32_t) * (HB + 1)));
  uint32_t* hstart = (uint32_t*)j->hstart.p;
  if (!j->graph_mode && !j->lines_ready) {
    Scalars init{};
    memset(&init, 0, sizeof(init));
    init.s0 = ~0ull;
    *j->h_sc = init;
    PK_CUDA(cudaMemcpyAsync(j->d_sc, j->h_sc, sizeof(Scalars), cudaMemcpyHostToDevice, j->stream));
  }

  CountArgs a{};
  a.fasta = (const uint8_t*)d_fasta;
  a.F = n;
  a.k = k;
  a.lmer_m = std::min(k, p->lmer_length);
  a.drop_n = p->drop_n ? 1 : 0;
  a.bbits = hb;
  a.grid = grid;
  a.chunk = chunk;
  a.tile_nl = (uint32_t*)j->tile_nl.p;
  a.counts = (uint32_t*)j->counts.p;
  a.bstart = hstart;
  a.sc = j->d_sc;
  a.nseg = nseg;
  a.unit_codes = (uint32_t*)j->units.p;
  a.unit_nbits = a.unit_codes + 4 * nseg;
  a.unit_windows = (unsigned long long*)(a.unit_nbits + 4 * nseg);

  mark_begin(j, ST_LINES);
  if (j->lines_ready) PK_CUDA(launch_tile_prefix(a, j->stream));
  else PK_CUDA(launch_line_scan(a, j->stream));
  mark_end(j, ST_LINES);
  mark_begin(j, ST_BUCKET_COUNT);
  PK_CUDA(launch_bucket_count(a, j->wide, j->stream));
  mark_end(j, ST_BUCKET_COUNT);
  mark_begin(j, ST_OFFSETS);
  PK_CUDA(launch_bucket_offsets(a, j->stream));
  mark_end(j, ST_OFFSETS);
  // the key buffer is sized by the exact window count (graph mode: by the bound the
  // caller sized its buffers for; small runs: no more windows than bytes)
  uint64_t N = j->graph_mode ? j->ncap : n;
  if (waits) {
    PK_CUDA(cudaMemcpyAsync(j->h_sc, j->d_sc, sizeof(Scalars), cudaMemcpyDeviceToHost, j->stream));
    PK_CUDA(cudaStreamSynchronize(j->stream));
    if (j->h_sc->err & ERR_FORMAT) return fail(PK_ERR_FORMAT, kFormatError);
    N = j->h_sc->n_windows;
  }
  if (N >= (1ull << 32) - 1)
    return fail(PK_ERR_LIMIT, "more than 2^32-2 k-mer windows in one job; split the input");
  j->N = N;
  if (by_count) {
    j->bbits = partition_bits((double)N, k, j->wide);
    // a digit or two short of the target costs less than a count over the coarse regions
    if (hb < kHistBits) j->bbits = std::min(j->bbits, hb);
  }
  const int B = 1 << j->bbits;
  a.cbits = std::min(j->bbits, kCoarseBits);
  PK_TRY(job_alloc(j, j->bstart, sizeof(uint32_t) * (B + 1)));
  PK_TRY(job_alloc(j, j->keys, (size_t)W * N));
  a.n_keys = N;
  PK_TRY(job_alloc(j, j->tkeys, (size_t)W * N));
  PK_TRY(job_alloc(j, j->tcounts, sizeof(uint32_t) * N));
  PK_TRY(job_alloc(j, j->tu, sizeof(uint32_t) * (size_t)B));
  const int t = p->num_buckets;
  PK_TRY(job_alloc(j, j->hist, sizeof(unsigned long long) * (size_t)t));
  PK_CUDA(cudaMemsetAsync(j->hist.p, 0, sizeof(unsigned long long) * (size_t)t, j->stream));
  j->t_hist = t;
  j->dense_valid = false;

  // two-pass partition: coarse regions (pass 1), then fine buckets (pass 2).  The
  // coarse copy lives in the table buffer, which is written only after pass 2.
  const int Cn = 1 << a.cbits;
  PK_TRY(job_alloc(j, j->coff, sizeof(uint32_t) * (size_t)grid * Cn));
  PK_TRY(job_alloc(j, j->cstart, sizeof(uint32_t) * (Cn + 1)));
  PK_TRY(job_alloc(j, j->slice_start, sizeof(uint32_t) * (Cn + 1)));
  PK_TRY(job_alloc(j, j->fcur, sizeof(uint32_t) * (size_t)B));
  const bool two_pass = a.cbits < j->bbits;
  mark_begin(j, ST_SCATTER);
  PK_CUDA(launch_coarse_offsets(a, j->bbits, (uint32_t*)j->coff.p, (uint32_t*)j->cstart.p,
                                (uint32_t*)j->slice_start.p, fine_slice_keys(j->wide, j->bbits - a.cbits),
                                (uint32_t*)j->bstart.p, (uint32_t*)j->fcur.p, j->stream));
  PK_CUDA(launch_scatter_coarse(a, (const uint32_t*)j->coff.p, two_pass ? j->tkeys.p : j->keys.p,
                                j->wide, j->stream));
  mark_end(j, ST_SCATTER);
  mark_begin(j, ST_SCATTER_FINE);
  if (two_pass) {
    if (hb < j->bbits) {
      PK_CUDA(cudaMemsetAsync(j->bstart.p, 0, sizeof(uint32_t) * (size_t)(B + 1), j->stream));
      PK_CUDA(cudaMemsetAsync(&j->d_sc->ticket_fcount, 0, sizeof(uint32_t), j->stream));
      PK_CUDA(launch_fine_count(j->tkeys.p, (const uint32_t*)j->cstart.p, (const uint32_t*)j->slice_start.p,
                                (uint32_t*)j->bstart.p, k, j->bbits, a.cbits, j->wide, &j->d_sc->ticket_fcount,
                                j->stream));
      PK_CUDA(launch_prefix((uint32_t*)j->bstart.p, B, j->stream));
      PK_CUDA(cudaMemcpyAsync(j->fcur.p, j->bstart.p, sizeof(uint32_t) * (size_t)B, cudaMemcpyDeviceToDevice,
                              j->stream));
    }
    PK_CUDA(launch_scatter_fine(j->tkeys.p, (const uint32_t*)j->cstart.p, (const uint32_t*)j->slice_start.p,
                                (uint32_t*)j->fcur.p, j->keys.p, k, j->bbits, a.cbits, j->wide,
                                &j->d_sc->ticket_fine, N, &j->d_sc->err, j->stream));
  }
  mark_end(j, ST_SCATTER_FINE);
  return table_impl(j, N, t);
}

// Stage 5: bucketed keys -> (k-mer, count) table, resident.
static pk_status table_impl(pk_job* j, uint64_t N, int t) {
  const int k = j->params.k;
  const int B = 1 << j->bbits;
  mark_begin(j, ST_TABLE);
  // giant buckets are reduced chunk by chunk first (chunk items ahead of the buckets);
  // fewer windows than a giant bucket's keys hold none
  const bool giants = N >= kGiantKeys;
  if (giants) {
    PK_TRY(job_alloc(j, j->gfirst, sizeof(uint32_t) * (size_t)B));
    PK_TRY(job_alloc(j, j->gcount, sizeof(uint32_t) * (size_t)B));
    PK_TRY(job_alloc(j, j->gdone, sizeof(uint32_t) * (size_t)B));
    const uint64_t chunks = N / chunk_keys(j->wide) + 1;
    PK_TRY(job_alloc(j, j->chunk_bucket, sizeof(uint32_t) * chunks));
    PK_TRY(job_alloc(j, j->chunk_u, sizeof(uint32_t) * chunks));
    PK_TRY(job_alloc(j, j->gpart, giant_part_bytes(N)));
  }
  PK_TRY(job_alloc(j, j->bsmall, sizeof(uint32_t) * kSmallCounts * (size_t)B));
  BucketArgs b{};
  b.keys = j->keys.p;
  b.bsmall = (uint32_t*)j->bsmall.p;
  b.gfirst = giants ? (const uint32_t*)j->gfirst.p : nullptr;
  b.gcount = (const uint32_t*)j->gcount.p;
  b.chunk_bucket = (const uint32_t*)j->chunk_bucket.p;
  b.gdone = (uint32_t*)j->gdone.p;
  b.chunk_u = (uint32_t*)j->chunk_u.p;
  uint32_t* glist = nullptr;
  if (giants) {
    b.gpart = (unsigned long long*)j->gpart.p;
    glist = (uint32_t*)(b.gpart + (size_t)kGiantParts * (N / kGiantKeys + 1));
  }
  b.glist = glist;
  b.bstart = (const uint32_t*)j->bstart.p;
  b.tkeys = j->tkeys.p;
  b.tcounts = (uint32_t*)j->tcounts.p;
  b.tu = (uint32_t*)j->tu.p;
  b.hist = (unsigned long long*)j->hist.p;
  b.t = t;
  b.k = k;
  b.bbits = j->bbits;
  b.cap = N;
  b.spin_limit = (int)j->wait_limit;
  b.sc = j->d_sc;
  if (giants)
    PK_CUDA(launch_giant_chunks(b, j->wide, (uint32_t*)j->gfirst.p, (uint32_t*)j->gcount.p, (uint32_t*)j->chunk_bucket.p,
                                glist, j->stream));
  PK_CUDA(launch_bucket_table(b, j->wide, j->table_ctas > 0 ? j->table_ctas * thread_sms(j->ctx->sms) : 0, j->stream));
  mark_end(j, ST_TABLE);
  j->bsmall_valid = true;
  j->pieces = 1;
  j->stage = 1;
  return PK_OK;
}

pk_status pk_count_device(pk_job* j, const void* d_fasta, uint64_t n, const pk_params* p) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  PK_TRY(check_params(p));
  if (n && !d_fasta) return fail(PK_ERR_INVALID, "d_fasta is null");
  if (((uintptr_t)d_fasta & 15) != 0) return fail(PK_ERR_INVALID, "d_fasta must be 16-byte aligned");
  PK_TRY(set_device(j->ctx));
  for (int i = 0; i < ST_COUNT_; i++) j->ev_rec[i] = false;
  return count_impl(j, d_fasta, n, p);
}

pk_status pk::count_host(pk_job* j, const char* fasta, uint64_t n, const pk_params* p) {
  for (int i = 0; i < ST_COUNT_; i++) j->ev_rec[i] = false;
  // -b pieces: always (chunking 1), or when the whole input at once does not fit the
  // HBM budget or the 2^32-window limit (chunking 0)
  if (p->chunking == 1) return count_pieces(j, fasta, n, p, p->batch_kmers);
  pk_status s = job_alloc(j, j->fasta, (size_t)n + 16);
  if (s == PK_OK) {
    mark_begin(j, ST_H2D);
    if (n) PK_CUDA(cudaMemcpyAsync(j->fasta.p, fasta, n, cudaMemcpyHostToDevice, j->stream));
    mark_end(j, ST_H2D);
    s = count_impl(j, j->fasta.p, n, p);
  }
  if ((s == PK_ERR_NOMEM || s == PK_ERR_LIMIT) && p->chunking == 0 && n > 1) {
    PK_CUDA(cudaStreamSynchronize(j->stream));
    job_free_all(j);
    const uint64_t b = p->batch_kmers ? p->batch_kmers : 100000000ull;
    return count_pieces(j, fasta, n, p, std::min<uint64_t>(b, (n + 1) / 2));
  }
  return s;
}

pk_status pk_count(pk_job* j, const char* fasta, uint64_t n, const pk_params* p) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  PK_TRY(check_params(p));
  if (n && !fasta) return fail(PK_ERR_INVALID, "fasta is null");
  PK_TRY(set_device(j->ctx));
  return count_host(j, fasta, n, p);
}

// Row check of a loaded table on the host, for a budget with no room to check it on the
// device beside the job's current table.
static pk_status check_rows_host(const uint64_t* kw, const uint32_t* counts, uint64_t n, int k,
                                 unsigned long long* chk) {
  const bool wide = k > 32;
  unsigned __int128 y = 0;
  for (uint64_t i = 0; i < n; i++) {
    const unsigned __int128 x = wide ? ((unsigned __int128)kw[2 * i + 1] << 64) | kw[2 * i]
                                     : (unsigned __int128)kw[i];
    const bool big = k < 64 && (x >> (2 * k)) != 0;
    if (big || (i && !(y < x)) || counts[i] == 0) {
      chk[0] = 4 * i + (big ? 0 : (i && !(y < x)) ? 1 : 2);
      return PK_OK;
    }
    chk[1] += counts[i];
    y = x;
  }
  return PK_OK;
}

static pk_status load_rule(unsigned long long bad) {
  if (bad == ~0ull) return PK_OK;
  const std::string row = std::to_string(bad >> 2);
  switch (bad & 3) {
    case 0: return fail(PK_ERR_INVALID, "row " + row + " is not a k-mer");
    case 1: return fail(PK_ERR_INVALID, "rows must be ascending and unique (row " + row + ")");
    default: return fail(PK_ERR_INVALID, "row " + row + " has count 0");
  }
}

// An existing (k-mer, count) table in place of counting: host rows ascending and
// unique, k-mers below 4^k.  The rows are laid out as the counting stages leave them
// (every bucket's rows contiguous), so cutoff and macro-nodes run unchanged.  The rows go
// to new buffers and are checked there, so a refused table leaves the job's current one.
pk_status pk_table_load(pk_job* j, const void* keys, const uint32_t* counts, uint64_t n, const pk_params* p) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  PK_TRY(check_params(p));
  if (n && (!keys || !counts)) return fail(PK_ERR_INVALID, "keys and counts must not be null");
  if (n >= 0xffffffffull) return fail(PK_ERR_LIMIT, "tables of 2^32-1 rows or more are not supported");
  const int k = p->k;
  const bool wide = k > 32;
  const size_t W = wide ? 16 : 8;
  // the count histogram is taken while the rows are checked, for the usual -t
  const int t = p->num_buckets <= 4096 ? p->num_buckets : 0;
  PK_TRY(set_device(j->ctx));
  unsigned long long chk[2] = {~0ull, 0};
  DevBuf nk, nc, nh, nx;
  pk_status s = job_alloc(j, nk, W * (n ? n : 1));
  if (s == PK_OK) s = job_alloc(j, nc, 4 * (n ? n : 1));
  if (s == PK_OK) s = job_alloc(j, nh, sizeof(unsigned long long) * (size_t)(t ? t : 1));
  if (s == PK_OK) s = job_alloc(j, nx, sizeof(chk));
  const bool on_device = s == PK_OK;
  auto drop = [&](bool idle) {
    for (DevBuf* b : {&nk, &nc, &nh, &nx}) {
      if (idle) job_free_idle(j, *b);
      else job_free(j, *b);
    }
  };
  if (on_device) {
    auto check = [&]() -> pk_status {
      PK_CUDA(cudaMemsetAsync(nx.p, 0xff, 8, j->stream));
      PK_CUDA(cudaMemsetAsync((char*)nx.p + 8, 0, 8, j->stream));
      if (t) PK_CUDA(cudaMemsetAsync(nh.p, 0, sizeof(unsigned long long) * (size_t)t, j->stream));
      if (n) {
        PK_CUDA(cudaMemcpyAsync(nk.p, keys, W * n, cudaMemcpyHostToDevice, j->stream));
        PK_CUDA(cudaMemcpyAsync(nc.p, counts, 4 * n, cudaMemcpyHostToDevice, j->stream));
      }
      PK_CUDA(launch_table_check(nk.p, (const uint32_t*)nc.p, n, k, wide, (unsigned long long*)nx.p, t,
                                 t ? (unsigned long long*)nh.p : nullptr, j->stream));
      PK_CUDA(cudaMemcpyAsync(chk, nx.p, sizeof(chk), cudaMemcpyDeviceToHost, j->stream));
      PK_CUDA(cudaStreamSynchronize(j->stream));
      return load_rule(chk[0]);
    };
    s = check();
    if (s != PK_OK) {
      drop(false);
      return s;
    }
  } else {
    drop(false);
    if (s != PK_ERR_NOMEM) return s;
    PK_TRY(check_rows_host((const uint64_t*)keys, counts, n, k, chk));
    PK_TRY(load_rule(chk[0]));
  }
  for (int i = 0; i < ST_COUNT_; i++) j->ev_rec[i] = false;
  j->bsmall_valid = false;  // the loaded table did not come from the table kernel
  j->params = *p;
  j->wide = wide;
  j->F = 0;
  j->N = n;
  j->stage = 0;
  j->bbits = row_bits(n, p);
  const int B = 1 << j->bbits;
  if (on_device) {
    std::swap(j->tkeys, nk);
    std::swap(j->tcounts, nc);
    if (t) std::swap(j->hist, nh);
    drop(true);  // check() waited for the stream
    j->t_hist = t;  // 0: no histogram of this table yet
  } else {
    j->t_hist = 0;
    PK_TRY(job_alloc(j, j->tkeys, W * (n ? n : 1)));
    PK_TRY(job_alloc(j, j->tcounts, 4 * (n ? n : 1)));
    if (n) {
      PK_CUDA(cudaMemcpyAsync(j->tkeys.p, keys, W * n, cudaMemcpyHostToDevice, j->stream));
      PK_CUDA(cudaMemcpyAsync(j->tcounts.p, counts, 4 * n, cudaMemcpyHostToDevice, j->stream));
    }
  }
  PK_TRY(job_alloc(j, j->bstart, sizeof(uint32_t) * (B + 1)));
  PK_TRY(job_alloc(j, j->tu, sizeof(uint32_t) * (size_t)B));
  PK_CUDA(launch_table_bounds(j->tkeys.p, n, j->bbits, k, (uint32_t*)j->bstart.p, (uint32_t*)j->tu.p,
                              wide, j->stream));
  Scalars init{};
  memset(&init, 0, sizeof(init));
  init.n_unique = n;
  init.n_windows = chk[1];
  *j->h_sc = init;
  PK_CUDA(cudaMemcpyAsync(j->d_sc, j->h_sc, sizeof(Scalars), cudaMemcpyHostToDevice, j->stream));
  PK_CUDA(cudaStreamSynchronize(j->stream));
  j->sc_fresh = true;
  j->dense_valid = false;
  j->stage = 1;
  return PK_OK;
}

// The scalars as the enqueued work leaves them (the stream is idle afterwards unless more
// was enqueued that does not touch them).
pk_status pk::sync_scalars(pk_job* j) {
  if (!j->sc_fresh) {
    PK_CUDA(cudaMemcpyAsync(j->h_sc, j->d_sc, sizeof(Scalars), cudaMemcpyDeviceToHost, j->stream));
    PK_CUDA(cudaStreamSynchronize(j->stream));
    j->sc_fresh = true;
  }
  const uint32_t err = j->h_sc->err;
  if (err & ERR_FORMAT) return fail(PK_ERR_FORMAT, kFormatError);
  if (err & ERR_LOOKBACK) return fail(PK_ERR_DEVICE, "a bounded look-back wait expired");
  if (err & ERR_BUCKET) return fail(PK_ERR_DEVICE, "a bucket could not be split to fit on chip");
  if (err & ERR_MN_CAPACITY) return fail(PK_ERR_DEVICE, "a macro-node segment exceeded on-chip capacity");
  if (err & ERR_BOUNDS) return fail(PK_ERR_DEVICE, "an index fell outside its buffer (write skipped)");
  return PK_OK;
}

pk_status pk_table_info(pk_job* j, uint64_t* u, uint64_t* w, uint64_t* r) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (j->stage < 1) return fail(PK_ERR_STATE, "no table: call pk_count first");
  PK_TRY(set_device(j->ctx));
  PK_TRY(sync_scalars(j));
  if (u) *u = j->h_sc->n_unique;
  if (w) *w = j->h_sc->n_windows;
  if (r) *r = j->h_sc->n_reads;
  return PK_OK;
}

// Dense (contiguous, ascending) copy of the resident sparse table, built on demand.
pk_status pk::dense_table(pk_job* j) {
  if (j->dense_valid) return PK_OK;
  const uint64_t u = j->h_sc->n_unique;
  const int B = 1 << j->bbits;
  const size_t W = j->wide ? 16 : 8;
  PK_TRY(job_alloc(j, j->doff, sizeof(uint32_t) * (B + 1)));
  PK_TRY(job_alloc(j, j->dkeys, W * (u ? u : 1)));
  PK_TRY(job_alloc(j, j->dcounts, 4 * (u ? u : 1)));
  PK_CUDA(launch_row_offsets((const uint32_t*)j->tu.p, (uint32_t*)j->doff.p, B, j->stream));
  PK_CUDA(launch_compact_rows(j->tkeys.p, (const uint32_t*)j->tcounts.p, (const uint32_t*)j->bstart.p,
                              (const uint32_t*)j->tu.p, (const uint32_t*)j->doff.p, B, j->wide,
                              j->dkeys.p, (uint32_t*)j->dcounts.p, nullptr, j->stream));
  j->dense_valid = true;
  return PK_OK;
}

pk_status pk_copy_table(pk_job* j, void* keys, uint32_t* counts, uint64_t cap) {
  uint64_t u = 0;
  PK_TRY(pk_table_info(j, &u, nullptr, nullptr));
  if (cap < u) return fail(PK_ERR_INVALID, "capacity smaller than the table");
  const size_t W = j->wide ? 16 : 8;
  PK_TRY(dense_table(j));
  if (u && keys) PK_CUDA(cudaMemcpyAsync(keys, j->dkeys.p, W * u, cudaMemcpyDeviceToHost, j->stream));
  if (u && counts)
    PK_CUDA(cudaMemcpyAsync(counts, j->dcounts.p, 4 * u, cudaMemcpyDeviceToHost, j->stream));
  PK_CUDA(cudaStreamSynchronize(j->stream));
  return PK_OK;
}

pk_status pk_copy_table_packed(pk_job* j, void* pairs, uint64_t cap) {
  uint64_t u = 0;
  PK_TRY(pk_table_info(j, &u, nullptr, nullptr));
  if (cap < u) return fail(PK_ERR_INVALID, "capacity smaller than the table");
  if (!u) return PK_OK;
  const size_t rec = j->wide ? 20 : 12;
  const int B = 1 << j->bbits;
  PK_TRY(job_alloc(j, j->doff, sizeof(uint32_t) * (B + 1)));
  PK_TRY(job_alloc(j, j->packed, rec * u));
  PK_CUDA(launch_row_offsets((const uint32_t*)j->tu.p, (uint32_t*)j->doff.p, B, j->stream));
  PK_CUDA(launch_compact_rows(j->tkeys.p, (const uint32_t*)j->tcounts.p, (const uint32_t*)j->bstart.p,
                              (const uint32_t*)j->tu.p, (const uint32_t*)j->doff.p, B, j->wide, nullptr,
                              nullptr, j->packed.p, j->stream));
  PK_CUDA(cudaMemcpyAsync(pairs, j->packed.p, rec * u, cudaMemcpyDeviceToHost, j->stream));
  PK_CUDA(cudaStreamSynchronize(j->stream));
  job_free_idle(j, j->packed);
  return PK_OK;
}

pk_status pk_table_device(pk_job* j, const void** k, const uint32_t** c) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (j->stage < 1) return fail(PK_ERR_STATE, "no table: call pk_count first");
  PK_TRY(set_device(j->ctx));
  PK_TRY(sync_scalars(j));
  PK_TRY(dense_table(j));
  PK_CUDA(cudaStreamSynchronize(j->stream));
  if (k) *k = j->dkeys.p;
  if (c) *c = (const uint32_t*)j->dcounts.p;
  return PK_OK;
}

// cutoff on the device; no host synchronisation
pk_status pk::cutoff_enqueue(pk_job* j, int t) {
  const unsigned long long* hist = (const unsigned long long*)j->hist.p;
  if (t != j->t_hist) {
    // histogram for a different -t than the one fused into counting
    PK_TRY(sync_scalars(j));
    PK_TRY(job_alloc(j, j->hist2, sizeof(unsigned long long) * (size_t)t));
    PK_CUDA(cudaMemsetAsync(j->hist2.p, 0, sizeof(unsigned long long) * (size_t)t, j->stream));
    PK_CUDA(launch_histogram((const uint32_t*)j->tcounts.p, (const uint32_t*)j->bstart.p,
                             (const uint32_t*)j->tu.p, 1 << j->bbits, t, (unsigned long long*)j->hist2.p,
                             j->stream));
    hist = (const unsigned long long*)j->hist2.p;
  }
  j->cut_max = (uint32_t)std::max(1, t - 1);
  j->sc_fresh = false;
  mark_begin(j, ST_CUTOFF);
  PK_CUDA(launch_cutoff(hist, t, j->d_sc, j->stream));
  mark_end(j, ST_CUTOFF);
  j->stage = 2;
  return PK_OK;
}

pk_status pk_cutoff(pk_job* j, int32_t t, uint32_t* cutoff, uint64_t* hist, uint64_t* kept) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (t < 1) return fail(PK_ERR_INVALID, "num_buckets must be >= 1");
  if (j->stage < 1) return fail(PK_ERR_STATE, "no table: call pk_count first");
  PK_TRY(set_device(j->ctx));
  PK_TRY(cutoff_enqueue(j, t));
  const void* hsrc = t == j->t_hist ? j->hist.p : j->hist2.p;
  if (hist) PK_CUDA(cudaMemcpyAsync(hist, hsrc, sizeof(uint64_t) * (size_t)t, cudaMemcpyDeviceToHost, j->stream));
  PK_TRY(sync_scalars(j));
  if (cutoff) *cutoff = j->h_sc->cutoff;
  if (kept) *kept = j->h_sc->n_kept;
  if (j->h_sc->n_kept == 0)
    return fail(PK_ERR_EMPTY, "no k-mer reaches the cutoff " + std::to_string(j->h_sc->cutoff) +
                                  "; macro-node construction cannot proceed");
  return PK_OK;
}

pk_status pk::mn_enqueue(pk_job* j, uint32_t min_count, uint64_t kept_bound) {
  const int B = 1 << j->bbits;
  const size_t W = j->wide ? 16 : 8;
  const uint64_t kcap = kept_bound ? kept_bound : 1;
  uint64_t cap = 2 * kept_bound;
  if (cap == 0) cap = 1;
  PK_TRY(job_alloc(j, j->kkeys, W * kcap));
  PK_TRY(job_alloc(j, j->kcounts, 4 * kcap));
  PK_TRY(job_alloc(j, j->kstart, sizeof(uint32_t) * B));
  PK_TRY(job_alloc(j, j->kcount, sizeof(uint32_t) * B));
  PK_TRY(job_alloc(j, j->ksub, sizeof(uint32_t) * 3 * (size_t)B));
  PK_TRY(job_alloc(j, j->nkeys, W * cap));
  PK_TRY(job_alloc(j, j->nsuf, 16 * cap));
  PK_TRY(job_alloc(j, j->npre, 16 * cap));
  // look-back words of the kept offsets and of the macro-node kernel, zeroed together, and
  // that kernel's list of big units behind them
  const size_t fflags = sizeof(unsigned long long) * (((size_t)B + 255) / 256);
  const size_t mflags = sizeof(unsigned long long) * mn_flag_words(j->bbits);
  PK_TRY(job_alloc(j, j->flags_m, fflags + mflags + sizeof(uint32_t) * (size_t)B));
  PK_CUDA(cudaMemsetAsync(j->flags_m.p, 0, fflags + mflags, j->stream));
  j->sc_fresh = false;
  PK_CUDA(cudaMemsetAsync(&j->d_sc->mn_begin, 0, offsetof(Scalars, mn_end) - offsetof(Scalars, mn_begin), j->stream));
  if (min_count) PK_CUDA(cudaMemcpyAsync(&j->d_sc->cutoff, &min_count, sizeof(uint32_t), cudaMemcpyHostToDevice, j->stream));
  j->mn_cap = cap;
  FilterArgs f{};
  f.tkeys = j->tkeys.p;
  f.tcounts = (const uint32_t*)j->tcounts.p;
  f.bstart = (const uint32_t*)j->bstart.p;
  f.tu = (const uint32_t*)j->tu.p;
  f.flags = (unsigned long long*)j->flags_m.p;
  f.kkeys = j->kkeys.p;
  f.kcounts = (uint32_t*)j->kcounts.p;
  f.kstart = (uint32_t*)j->kstart.p;
  f.kcount = (uint32_t*)j->kcount.p;
  f.ksub = (uint32_t*)j->ksub.p;
  f.cap = kcap;
  f.trows = j->tcounts.bytes / sizeof(uint32_t);
  f.bsmall = j->bsmall_valid ? (const uint32_t*)j->bsmall.p : nullptr;
  f.k = j->params.k;
  f.bbits = j->bbits;
  f.spin_limit = (int)j->wait_limit;
  f.sc = j->d_sc;
  mark_begin(j, ST_FILTER);
  const uint32_t cut_max = min_count ? min_count : j->cut_max;
  PK_CUDA(launch_filter_kept(f, j->wide, !f.bsmall || cut_max > (uint32_t)kSmallCounts, j->stream));
  mark_end(j, ST_FILTER);
  MnArgs m{};
  m.kkeys = j->kkeys.p;
  m.kcounts = (const uint32_t*)j->kcounts.p;
  m.kstart = (const uint32_t*)j->kstart.p;
  m.kcount = (const uint32_t*)j->kcount.p;
  m.ksub = (const uint32_t*)j->ksub.p;
  m.flags = (unsigned long long*)((char*)j->flags_m.p + fflags);
  m.big = (uint32_t*)((char*)j->flags_m.p + fflags + mflags);
  m.nkeys = j->nkeys.p;
  m.nsuf = (uint32_t*)j->nsuf.p;
  m.npre = (uint32_t*)j->npre.p;
  m.cap = cap;
  m.kcap = kcap;
  m.k = j->params.k;
  m.bbits = j->bbits;
  // node units of up to 1000 rows where the partition is that fine (each merges 2V / units
  // of them on average, half from each side; a joined unit holds kMnJoin a side)
  {
    int x = 0;
    while (x < j->bbits && 2.0 * (double)kept_bound / (double)(1u << (j->bbits - x - 1)) <= 1000.0) x++;
    if (j->params.mn_units > 0) x = std::min(2 * (j->params.mn_units - 1), j->bbits & ~1);
    m.xbits = x;
  }
  m.spin_limit = (int)j->wait_limit;
  m.withhold_unit = j->withhold_unit;
  m.sc = j->d_sc;
  mark_begin(j, ST_MN);
  PK_CUDA(launch_macro_nodes(m, j->wide, 0, j->stream));
  mark_end(j, ST_MN);
  j->stage = 3;
  j->wired = false;
  j->compacted = false;
  return PK_OK;
}

pk_status pk_build_macro_nodes(pk_job* j, uint32_t min_count, uint64_t* n_nodes) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (j->stage < 1 || (min_count == 0 && j->stage < 2))
    return fail(PK_ERR_STATE, "call pk_count and pk_cutoff (or pass min_count) first");
  PK_TRY(set_device(j->ctx));
  PK_TRY(sync_scalars(j));
  uint64_t bound = min_count ? j->h_sc->n_unique : j->h_sc->n_kept;
  if (bound == 0)
    return fail(PK_ERR_EMPTY, "no k-mer reaches the cutoff; macro-node construction cannot proceed");
  PK_TRY(mn_enqueue(j, min_count, bound));
  PK_TRY(sync_scalars(j));
  if (n_nodes) *n_nodes = j->h_sc->n_nodes;
  return PK_OK;
}

pk_status pk_copy_macro_nodes(pk_job* j, void* keys, uint32_t* suf, uint32_t* pre, uint64_t cap) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (j->stage < 3) return fail(PK_ERR_STATE, "no macro-nodes: call pk_build_macro_nodes first");
  PK_TRY(set_device(j->ctx));
  PK_TRY(sync_scalars(j));
  const uint64_t m = j->h_sc->n_nodes;
  if (cap < m) return fail(PK_ERR_INVALID, "capacity smaller than the node count");
  const size_t W = j->wide ? 16 : 8;
  if (m && keys) PK_CUDA(cudaMemcpyAsync(keys, j->nkeys.p, W * m, cudaMemcpyDeviceToHost, j->stream));
  if (m && suf) PK_CUDA(cudaMemcpyAsync(suf, j->nsuf.p, 16 * m, cudaMemcpyDeviceToHost, j->stream));
  if (m && pre) PK_CUDA(cudaMemcpyAsync(pre, j->npre.p, 16 * m, cudaMemcpyDeviceToHost, j->stream));
  PK_CUDA(cudaStreamSynchronize(j->stream));
  return PK_OK;
}

pk_status pk_macro_nodes_device(pk_job* j, const void** k, const uint32_t** s, const uint32_t** p) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (j->stage < 3) return fail(PK_ERR_STATE, "no macro-nodes: call pk_build_macro_nodes first");
  if (k) *k = j->nkeys.p;
  if (s) *s = (const uint32_t*)j->nsuf.p;
  if (p) *p = (const uint32_t*)j->npre.p;
  return PK_OK;
}

pk_status pk_wire_macro_nodes(pk_job* j, int32_t coverage) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (j->stage < 3) return fail(PK_ERR_STATE, "no macro-nodes: call pk_build_macro_nodes first");
  const int cov = coverage ? coverage : j->params.coverage;
  if (cov <= 0) return fail(PK_ERR_INVALID, "coverage must be >= 1");
  PK_TRY(set_device(j->ctx));
  PK_TRY(sync_scalars(j));
  const uint64_t m = j->h_sc->n_nodes;
  PK_TRY(job_alloc(j, j->wiring, sizeof(WireRow) * (m ? m : 1)));
  PK_CUDA(launch_wire(j->nsuf.p, j->npre.p, m, cov, (WireRow*)j->wiring.p, j->stream));
  j->wired = true;
  return PK_OK;
}

pk_status pk_copy_wiring(pk_job* j, pk_wiring* out, uint64_t cap) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  if (!j->wired) return fail(PK_ERR_STATE, "no wiring: call pk_wire_macro_nodes first");
  PK_TRY(set_device(j->ctx));
  PK_TRY(sync_scalars(j));
  const uint64_t m = j->h_sc->n_nodes;
  if (cap < m) return fail(PK_ERR_INVALID, "capacity smaller than the node count");
  if (m && out) PK_CUDA(cudaMemcpyAsync(out, j->wiring.p, sizeof(pk_wiring) * m, cudaMemcpyDeviceToHost, j->stream));
  PK_CUDA(cudaStreamSynchronize(j->stream));
  return PK_OK;
}

pk_status pk_wiring_device(pk_job* j, const pk_wiring** d) {
  if (!j || !d) return fail(PK_ERR_INVALID, "null argument");
  if (!j->wired) return fail(PK_ERR_STATE, "no wiring: call pk_wire_macro_nodes first");
  *d = (const pk_wiring*)j->wiring.p;
  return PK_OK;
}

pk_status pk_summary_get(pk_job* j, pk_summary* o) {
  if (!j || !o) return fail(PK_ERR_INVALID, "null argument");
  PK_TRY(set_device(j->ctx));
  PK_TRY(sync_scalars(j));
  o->n_reads = j->h_sc->n_reads;
  o->n_windows = j->h_sc->n_windows;
  o->n_unique = j->stage >= 1 ? j->h_sc->n_unique : 0;
  o->n_kept = j->stage >= 2 ? j->h_sc->n_kept : 0;
  o->n_nodes = j->stage >= 3 ? j->h_sc->n_nodes : 0;
  o->cutoff = j->stage >= 2 ? j->h_sc->cutoff : 0;
  o->key_bytes = j->wide ? 16 : 8;
  return PK_OK;
}

static pk_status empty_after_cutoff(pk_job* j) {
  return fail(PK_ERR_EMPTY, "no k-mer reaches the cutoff " + std::to_string(j->h_sc->cutoff) +
                                "; macro-node construction cannot proceed");
}

static pk_status run_rest(pk_job* j, const pk_params* p, pk_summary* out) {
  PK_TRY(cutoff_enqueue(j, p->num_buckets));
  uint64_t kept = j->N;  // small runs: no more kept k-mers than windows
  if (!j->no_wait) {
    PK_TRY(sync_scalars(j));
    kept = j->h_sc->n_kept;
    if (kept == 0) {
      if (out) pk_summary_get(j, out);
      return empty_after_cutoff(j);
    }
  }
  PK_TRY(mn_enqueue(j, 0, kept));
  const pk_status s = sync_scalars(j);
  if (s == PK_ERR_FORMAT && j->no_wait) j->stage = 0;  // as when the count is waited for
  PK_TRY(s);
  if (j->no_wait && j->h_sc->n_kept == 0) {
    j->stage = 2;
    if (out) pk_summary_get(j, out);
    return empty_after_cutoff(j);
  }
  return out ? pk_summary_get(j, out) : PK_OK;
}

// The whole path.  Small inputs (whose buffers are small at their bounds too) run without
// waiting for the window count and the kept count in between: a wait is 10 us of the 150 or
// so that they take.  Not with a budget, which counts exact sizes.
constexpr uint64_t kSmallRun = 1ull << 20;
static pk_status run_all(pk_job* j, const void* fasta, uint64_t n, const pk_params* p, pk_summary* out, bool host) {
  if (!j) return fail(PK_ERR_INVALID, "job is null");
  j->no_wait = p && n <= kSmallRun && p->chunking != 1 && j->ctx->budget == 0;
  pk_status s = host ? pk_count(j, (const char*)fasta, n, p) : pk_count_device(j, fasta, n, p);
  if (s == PK_OK) s = run_rest(j, p, out);
  // an allocation that failed on the way: the caller's buffer may still be read
  if (s != PK_OK && j->no_wait) cudaStreamSynchronize(j->stream);
  j->no_wait = false;
  return s;
}

pk_status pk_run(pk_job* j, const char* fasta, uint64_t n, const pk_params* p, pk_summary* out) {
  return run_all(j, fasta, n, p, out, true);
}

pk_status pk_run_device(pk_job* j, const void* d_fasta, uint64_t n, const pk_params* p, pk_summary* out) {
  return run_all(j, d_fasta, n, p, out, false);
}
