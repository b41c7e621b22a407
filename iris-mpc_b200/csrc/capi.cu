// C ABI of the B200 iris hot path (declarations and reference citations in
// include/irisb200.h).  Host-side object management: per-party streams and
// memory pools, device-resident share databases, query staging, and the
// launches of the limb GEMM, the fused threshold kernels and the result
// kernels.  No entry point aborts: every failure returns a status and sets
// the thread's last-error string.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <map>
#include <mutex>
#include <shared_mutex>
#include <string>
#include <vector>

#include "../../include/irisb200.h"
#include "or_tree.h"
#include "common.cuh"
#include "fused_scan.h"
#include "gemm_limb.h"
#include "internal.h"
#include "prep.h"
#include "quad_gemm.h"
#include "results.h"
#include "threshold.h"

using namespace irs;

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
  return code;
}

#define CU(call)                                                                                     \
  do {                                                                                               \
    cudaError_t e_ = (call);                                                                         \
    if (e_ != cudaSuccess) return fail(IRS_ERR_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), \
                                       __FILE__, __LINE__);                                          \
  } while (0)

#define CHECK(cond, code, ...) \
  do {                         \
    if (!(cond)) return fail((code), __VA_ARGS__); \
  } while (0)

size_t round_up(size_t x, size_t m) { return (x + m - 1) / m * m; }

}  // namespace

struct irs_device_manager {
  int device = 0;
  int n_sms = 148;
  cudaStream_t streams[3] = {nullptr, nullptr, nullptr};
  cudaMemPool_t pools[3] = {nullptr, nullptr, nullptr};
  int* d_err = nullptr;
  uint64_t* d_batch = nullptr;  // device batch counter (irs_device_manager_set_batch_counter)
  bool capturing = false;  // a graph capture on streams[0] is open
  cudaEvent_t graph_done = nullptr;  // complete when every graph launched so far has run
  cudaStream_t graph_join = nullptr;  // the graphs' streams meet here, and graph_done follows them
  cudaEvent_t graph_ran = nullptr;    // recorded after each graph launch, on its stream
  // recorded on the parties' streams before a graph launch or a capture
  cudaEvent_t uploads[3] = {nullptr, nullptr, nullptr};
  bool host_sync = true;  // false: host-buffer calls return once enqueued (irs_device_manager_set_host_sync)
  // stage timers (irs_device_manager_set_timing): event pairs per label, resolved on read
  bool timing = false;
  struct Timer {
    const char* label;
    cudaEvent_t start, stop;
  };
  std::vector<Timer> timers;
  std::map<std::string, std::pair<double, long>> timer_totals;  // label -> (ms, launches)
  uint64_t stall_limit_ns = 0;  // armed by irs_device_manager_test_stall_next_dot (one shot)
};

// Brackets one stage launch on stream s with a pair of timing events when the
// device manager's stage timers are on (outside graph capture).
struct StageTimer {
  irs_device_manager* dm;
  cudaStream_t s;
  cudaEvent_t a = nullptr, b = nullptr;
  const char* label;
  StageTimer(irs_device_manager* d, cudaStream_t st, const char* l) : dm(d), s(st), label(l) {
    if (!dm->timing || dm->capturing) return;
    if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) {
      cudaGetLastError();
      a = b = nullptr;
      return;
    }
    cudaEventRecord(a, s);
  }
  ~StageTimer() {
    if (!a) return;
    cudaEventRecord(b, s);
    dm->timers.push_back({label, a, b});
  }
};

struct irs_graph {
  irs_device_manager* dm = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

struct irs_sharedb {
  irs_device_manager* dm = nullptr;
  int peer = 0;
  size_t max_db = 0, query_length = 0, code_length = 0;
  ChaChaKey seed0{}, seed1{};
  bool remote = false;
  // device-resident DB limb planes [db_cap][K]
  uint8_t* db_lo = nullptr;
  uint8_t* db_hi = nullptr;
  size_t db_cap = 0, db_len = 0;
  // query limb planes [n_pad][K]
  uint8_t* q_lo = nullptr;
  uint8_t* q_hi = nullptr;
  uint16_t* q_stage = nullptr;  // u16 staging [n_pad][K]
  QuerySlot* d_slots = nullptr;
  size_t n_pad = 0;          // active padded query rows (result row stride)
  size_t n_cap = 0;          // query row capacity
  size_t rows_uploaded = 0;  // rows of the last upload
  int tile_override = 0;     // tile width requested by irs_sharedb_set_tile (0 = auto)
  bool pair = false;         // two-SM GEMM for the 256-row tile (irs_sharedb_set_pair)
  bool batch_from_device = false;
  bool have_query = false;
  // results [max_db][n_pad] u16 (entry-major)
  uint16_t* results = nullptr;
  size_t res_offset = 0, res_len = 0;
  int last_gemm = IRS_GEMM_NONE;
  uint64_t batch = 0;
  // rotation-structured GEMM (quad_gemm.cu): the records' derived sums, one
  // allocation (outer lo, hi [db_cap][K/2], inner lo, hi [db_cap][3K/4]), and
  // the query forms (lo, hi [9][n_pad/4][K/4]) with the slots' row masks
  uint8_t* sums = nullptr;
  uint8_t* forms = nullptr;
  uint32_t* row_valid = nullptr;
  uint32_t* quad_flag = nullptr;  // QuadFlags word, for captured launches
  std::vector<uint32_t*> old_flags;  // words of graphs over sums that are gone: zero, kept until destroy
  uint32_t flag_rows = 0;     // what the last upload left in it
  bool quad_rows = false;     // the uploaded rows are quads of rotations and the forms hold them
  size_t stale_end = 0;       // records below it may have sums that a gather left behind
  size_t forms_pad = 0;       // padded rows that the form maps are for (0: none)
  bool dot_captured = false;  // a graph of this library reads the sums where quad_flag says so
  bool sums_pinned = false;   // another capture uses the sums: they stay until alloc_db or destroy
  bool rows_captured = false; // a captured upload rewrites the rows when it is replayed: no forms
  CUtensorMap tm_sum_lo[2]{}, tm_sum_hi[2]{}, tm_form_lo[kQuadWidths]{},
      tm_form_hi[kQuadWidths]{};
  CUtensorMap tm_db_lo{}, tm_db_hi{}, tm_q_lo{}, tm_q_hi{};
  CUtensorMap tm_qp_lo{}, tm_qp_hi{};    // half a tile of the two-SM GEMM
  CUtensorMap tm_qf_lo[2]{}, tm_qf_hi[2]{};  // 64 and 128 rows, for launches of few rounds
  int block_n = 0;
  cudaEvent_t done = nullptr;  // recorded after the engine's last dot launch
  cudaEvent_t copied = nullptr;  // recorded after an upload's last read of host memory
};

struct irs_circuits {
  irs_device_manager* dm = nullptr;
  ChaChaKey keys[3]{};
  uint64_t batch = 0;
  bool batch_from_device = false;
};

struct irs_distance_comparator {
  irs_device_manager* dm = nullptr;
  size_t max_queries = 0, max_db = 0, stride_bits = 0, self_stride_bits = 0, match_cap = 0;
  uint32_t* bitmap = nullptr;       // [max_queries][stride_bits/32]
  uint32_t* self_bitmap = nullptr;  // [max_queries][self_stride_bits/32]
  uint32_t* match_list = nullptr;   // pairs
  uint32_t* counters = nullptr;     // [0] match count, [1] partial count
  uint32_t* partial = nullptr;      // [max_db] compaction output
  // one allocation, so that one copy fetches them:
  uint32_t* results_err = nullptr;    // [4]: word 0 takes the device error word
  uint32_t* final_results = nullptr;  // [max_queries]
  uint32_t* match_counters = nullptr; // [max_queries]
  uint32_t* all_matches = nullptr;    // [max_queries][256]
  uint32_t* d_slot_valid = nullptr;
  uint32_t* d_slot_query = nullptr;
  // irs_dc_take_rows: row list [max_queries], error word [4], counts [max_queries], ids [max_queries][256]
  uint32_t* d_take = nullptr;
  // distance capture (irs_dc_enable_distance_capture): count, entry, row, code [3], mask [3]
  uint32_t* d_dist = nullptr;
  size_t dist_cap = 0;
  uint32_t* d_forced = nullptr;  // forced records: query [256], entry [256]
  uint32_t n_forced = 0;
  size_t slot_cap = 0;
  // segment table (irs_dc_set_segments)
  uint32_t* d_seg_start = nullptr;  // [slot_cap + 1]
  uint32_t* d_seg_query = nullptr;  // [seg_cap]
  uint32_t* d_seg_mask = nullptr;   // [seg_cap]
  size_t seg_cap = 0, n_seg_slots = 0;
  bool have_segments = false;
  // dot-share ring of the fused scan (irs_dc_scan_fused), allocated on first use
  uint16_t* ring = nullptr;
  size_t ring_bytes = 0;
};

namespace {

cudaStream_t party_stream(irs_device_manager* dm, int party, void* s) {
  return s ? static_cast<cudaStream_t>(s) : dm->streams[party];
}

// Engines of a device that hold derived sums, over all device managers of the
// process.  The sums are an extra layout of records that are resident anyway, so
// they give way when an allocation of the library fails.  A launch that may read
// an engine's sums holds the lock shared from the look at them until it is
// enqueued, so that launches do not wait for one another; whoever takes sums away
// holds it alone.  Each device has its own: a thread that waits for a full launch
// queue, or frees memory, does not hold up those that drive other devices.
struct SumHolders {
  std::shared_mutex mu;
  std::vector<irs_sharedb*> engines;
  std::vector<irs_device_manager*> managers;  // all of the device
};
using SumReader = std::shared_lock<std::shared_mutex>;
using SumWriter = std::lock_guard<std::shared_mutex>;
SumHolders& sum_holders(int device) {
  static SumHolders h[64];
  return h[device & 63];
}
SumHolders& sum_holders(const irs_sharedb* db) { return sum_holders(db->dm->device); }

// Memory of an engine's sums and forms that nothing new can reach.
struct DroppedSums {
  uint8_t* sums = nullptr;
  uint8_t* forms = nullptr;
};

// Takes an engine's sums and forms away from it (its device's lock is held
// alone); the caller frees them once it has released the lock: cudaFree waits
// for the launches that read them.
// A graph that holds the quad GEMM is told by the flag to run the plain one, for
// good: the word is its own from here on, and whatever sums the engine gets next
// have another.  Replays start under the lock, so that none reads it half-way.
DroppedSums take_sums(irs_sharedb* db) {
  if (db->quad_flag && (db->dot_captured || db->sums_pinned)) {
    if (cudaEventSynchronize(db->dm->graph_done) != cudaSuccess) {
      cudaGetLastError();
      cudaDeviceSynchronize();
    }
    cudaMemsetAsync(db->quad_flag, 0, 4, db->dm->streams[db->peer]);
    cudaStreamSynchronize(db->dm->streams[db->peer]);
    try {
      db->old_flags.push_back(db->quad_flag);
    } catch (const std::bad_alloc&) {  // four bytes of the pool stay with the device manager
    }
    db->quad_flag = nullptr;
    db->flag_rows = 0;
  }
  auto& v = sum_holders(db).engines;
  v.erase(std::remove(v.begin(), v.end(), db), v.end());
  const DroppedSums d{db->sums, db->forms};
  db->sums = db->forms = nullptr;
  db->row_valid = nullptr;
  db->quad_rows = false;
  db->stale_end = 0;
  db->forms_pad = 0;
  db->dot_captured = db->sums_pinned = false;
  return d;
}

void free_sums(const DroppedSums& d) {
  if (d.sums) cudaFree(d.sums);
  if (d.forms) cudaFree(d.forms);
}

void drop_sums(irs_sharedb* db) {
  {
    SumReader lock(sum_holders(db).mu);
    if (!db->sums) return;
  }
  DroppedSums d;
  {
    SumWriter lock(sum_holders(db).mu);
    d = take_sums(db);
  }
  free_sums(d);
}

size_t sums_bytes(size_t cap, size_t K) { return 2 * cap * (K / 2 + 3 * K / 4); }
size_t forms_bytes(size_t n_cap, size_t K) { return 2 * (kQuadProducts * (n_cap / 4) * (K / 4)); }

// Whether reclaim_sums may take an engine's sums (the lock is held): not those
// that a capture other than of this library's own dots uses.
bool sums_reclaimable(const irs_sharedb* db, int device) {
  return db->dm->device == device && !db->sums_pinned && !db->dm->capturing;
}

// Bytes that reclaim_sums would give back on a device.
size_t reclaimable_sums(int device) {
  SumReader lock(sum_holders(device).mu);
  size_t bytes = 0;
  for (const irs_sharedb* db : sum_holders(device).engines)
    if (sums_reclaimable(db, device))
      bytes += sums_bytes(db->db_cap, db->code_length) + forms_bytes(db->n_cap, db->code_length);
  return bytes;
}

// Gives back the sums of one engine on `device` that may lose them, the last
// to have got them; whether there was one.
bool reclaim_sums(int device) {
  DroppedSums d;
  {
    SumWriter lock(sum_holders(device).mu);
    const auto& held = sum_holders(device).engines;
    const auto it = std::find_if(held.rbegin(), held.rend(),
                                 [&](const irs_sharedb* db) { return sums_reclaimable(db, device); });
    if (it == held.rend()) return false;
    d = take_sums(*it);
  }
  free_sums(d);
  return true;
}

// Whether `bytes` can be had on a device once all sums are given back: with
// what is free and what the managers' pools hold unused.
bool fits_without_sums(int device, size_t bytes) {
  size_t room = reclaimable_sums(device), free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) room += free_b;
  SumReader lock(sum_holders(device).mu);
  for (const irs_device_manager* dm : sum_holders(device).managers)
    for (cudaMemPool_t pool : dm->pools) {
      uint64_t reserved = 0, used = 0;
      if (pool && cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
          cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess)
        room += reserved - used;
    }
  cudaGetLastError();
  return bytes <= room;
}

// An allocation (`take`) that gives derived sums back, an engine's at a time,
// before it fails; none where that cannot help.
template <class Take>
cudaError_t alloc_or_reclaim(irs_device_manager* dm, size_t bytes, Take take) {
  cudaError_t e = take();
  for (bool asked = false; e == cudaErrorMemoryAllocation && !dm->capturing; e = take()) {
    cudaGetLastError();
    if (!asked && !fits_without_sums(dm->device, bytes)) return e;
    asked = true;
    if (!reclaim_sums(dm->device)) return e;
  }
  return e;
}

cudaError_t device_malloc(irs_device_manager* dm, void** p, size_t bytes) {
  return alloc_or_reclaim(dm, bytes, [&] { return cudaMalloc(p, bytes); });
}

int pool_alloc(irs_device_manager* dm, int party, size_t bytes, void** out) {
  *out = nullptr;
  if (!bytes) return IRS_OK;
  cudaError_t e = alloc_or_reclaim(
      dm, bytes, [&] { return cudaMallocFromPoolAsync(out, bytes, dm->pools[party], dm->streams[party]); });
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(IRS_ERR_NOMEM, "device allocation of %zu bytes for party %d failed: %s", bytes, party,
                cudaGetErrorString(e));
  }
  e = cudaStreamSynchronize(dm->streams[party]);
  if (e != cudaSuccess) return fail(IRS_ERR_CUDA, "allocation sync: %s", cudaGetErrorString(e));
  return IRS_OK;
}

void pool_free(irs_device_manager* dm, int party, void* p) {
  if (p) cudaFreeAsync(p, dm->streams[party]);
}

// Scratch of one call, ordered on the call's own stream (freed there with
// cudaFreeAsync): unlike pool_alloc it does not wait for the stream.
int scratch_alloc(irs_device_manager* dm, cudaStream_t s, size_t bytes, void** out) {
  *out = nullptr;
  if (!bytes) return IRS_OK;
  const cudaError_t e =
      alloc_or_reclaim(dm, bytes, [&] { return cudaMallocFromPoolAsync(out, bytes, dm->pools[0], s); });
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(IRS_ERR_NOMEM, "device scratch of %zu bytes: %s", bytes, cudaGetErrorString(e));
  }
  return IRS_OK;
}

int device_error(int code) {
  if (code) return fail(IRS_ERR_DEVICE, "kernel reported error code %d (bounded wait expired)", code);
  return IRS_OK;
}

int check_device_error(irs_device_manager* dm) {
  int code = 0;
  CU(cudaMemcpy(&code, dm->d_err, sizeof(int), cudaMemcpyDeviceToHost));
  return device_error(code);
}

ChaChaKey key_of(const uint32_t k[8]) {
  ChaChaKey r;
  for (int i = 0; i < 8; i++) r.k[i] = k[i];
  return r;
}

// Query tensor maps for the current tile width (the two-SM GEMM loads half of
// a query tile per CTA).
int rebuild_query_maps(irs_sharedb* db) {
  if (db->block_n <= 0) return IRS_OK;  // no valid tile width: dot reports it
  const uint32_t box = (uint32_t)db->block_n;
  const uint32_t half = (uint32_t)gemm_pair_n((uint32_t)db->n_pad) / 2;
  if (make_tmap_u8(&db->tm_q_lo, db->q_lo, db->n_cap, db->code_length, box) ||
      make_tmap_u8(&db->tm_q_hi, db->q_hi, db->n_cap, db->code_length, box) ||
      make_tmap_u8(&db->tm_qp_lo, db->q_lo, db->n_cap, db->code_length, half) ||
      make_tmap_u8(&db->tm_qp_hi, db->q_hi, db->n_cap, db->code_length, half) ||
      make_tmap_u8(&db->tm_qf_lo[0], db->q_lo, db->n_cap, db->code_length, 64) ||
      make_tmap_u8(&db->tm_qf_hi[0], db->q_hi, db->n_cap, db->code_length, 64) ||
      make_tmap_u8(&db->tm_qf_lo[1], db->q_lo, db->n_cap, db->code_length, 128) ||
      make_tmap_u8(&db->tm_qf_hi[1], db->q_hi, db->n_cap, db->code_length, 128))
    return fail(IRS_ERR_CUDA, "tensor map for the query planes failed");
  return IRS_OK;
}

// Sets the active padded row count and tile width for `rows` query rows.
// Padded query rows for `rows` real rows: a multiple of 64, raised to a
// multiple of 128 (up to 768 rows) or 256 (above) when the query capacity
// allows, so that the GEMM runs the tile gemm_block_n_for picks for that row
// count instead of falling back to the 64-row tile (1600 rows on the 64-row
// tile take about twice as long as 1792 rows on the 256-row tile).  The extra
// rows are zero and no comparison reads them.
static size_t padded_query_rows(size_t rows, size_t n_cap) {
  const size_t n64 = round_up(rows ? rows : 1, 64);
  const size_t wide = n64 <= 64 ? n64 : (n64 <= 768 ? round_up(n64, 128) : round_up(n64, 256));
  return wide <= n_cap ? wide : n64;
}

// ---- rotation-structured GEMM (quad_gemm.cu) ----

// Fewest padded query rows for which the quad GEMM runs: it reads 2.25x the DB
// bytes of the plain one.  Six engines over 32,768 entries, quad against the
// better plain GEMM: 256 rows 1.73 / 1.05 ms, 384 1.93 / 1.83, 512 2.02 / 2.04,
// 640 2.20 / 2.58, 768 2.40 / 2.78, 2048 5.3 / 7.3.
constexpr size_t kQuadMinRows = 576;
// Fewest records for which an engine keeps (or a gather brings along) the sums:
// under that a launch has too few tiles for the nine products to pay (700
// entries x 2048 rows: 0.19 ms either way; 2,048 entries: 0.35 / 0.52 ms).
constexpr size_t kQuadMinRecords = 1024;

// Allocates the derived sums and query forms of an engine whose DB planes have
// just been allocated (and zeroed, so the sums start at zero too).  Optional:
// without them the engine runs the plain GEMM.  They are kept out of the way
// of the program's other allocations: a twelfth of the device's memory (16 GB)
// stays free, and reclaim_sums gives them back when the library needs the room.
// (A sixth left one of six engines of 524,288 records with 5,632 query rows
// without them: 152 ms for 64 queries instead of 110.)
void alloc_sums(irs_sharedb* db) {
  irs_device_manager* dm = db->dm;
  const size_t K = db->code_length, cap = db->db_cap;
  if (K % kRowLen || !forms_fit(K) || db->n_cap < kQuadMinRows || cap < kQuadMinRecords || dm->capturing) return;
  const size_t forms = forms_bytes(db->n_cap, K), masks = db->n_cap / kSlotRows * 4;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || free_b < sums_bytes(cap, K) + forms + total_b / 12) {
    cudaGetLastError();
    return;
  }
  void *s = nullptr, *f = nullptr, *w = nullptr;
  if (!db->quad_flag) {
    if (pool_alloc(dm, db->peer, 4, &w)) return;
    db->quad_flag = static_cast<uint32_t*>(w);
  }
  if (cudaMalloc(&s, sums_bytes(cap, K)) != cudaSuccess || cudaMalloc(&f, forms + masks) != cudaSuccess) {
    cudaGetLastError();
    if (s) cudaFree(s);
    return;
  }
  db->sums = static_cast<uint8_t*>(s);
  db->forms = static_cast<uint8_t*>(f);
  db->row_valid = reinterpret_cast<uint32_t*>(db->forms + forms);
  db->flag_rows = 0;
  db->stale_end = 0;
  cudaStream_t st = dm->streams[db->peer];
  uint8_t* inner = db->sums + 2 * cap * (K / 2);
  if (make_tmap_plane(&db->tm_sum_lo[0], db->sums, cap, K / 2, 128) ||
      make_tmap_plane(&db->tm_sum_hi[0], db->sums + cap * (K / 2), cap, K / 2, 128) ||
      make_tmap_plane(&db->tm_sum_lo[1], inner, cap, 3 * K / 4, 128) ||
      make_tmap_plane(&db->tm_sum_hi[1], inner + cap * (3 * K / 4), cap, 3 * K / 4, 128) ||
      cudaMemsetAsync(db->sums, 0, sums_bytes(cap, K), st) != cudaSuccess ||
      cudaMemsetAsync(db->quad_flag, 0, 4, st) != cudaSuccess) {
    cudaGetLastError();
    drop_sums(db);
    return;
  }
  bool held = true;
  try {
    SumWriter lock(sum_holders(db).mu);
    sum_holders(db).engines.push_back(db);
  } catch (const std::bad_alloc&) {
    held = false;
  }
  if (!held) drop_sums(db);
}

bool stream_captures(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) == cudaSuccess) return st != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return false;
}

// Whether a gather of n records leaves the sums behind, for the first dot that
// wants them (fresh_sums): unless the rows uploaded so far are enough for the quad
// GEMM, that dot may never come, and the sums would be a third of the gather
// (4,000 records of 12,800, waited for: 110 us instead of 71).  A captured launch
// runs the GEMM that it was captured with, and a captured gather runs whenever it
// is replayed: those keep the sums up.
bool gather_skips_sums(const irs_sharedb* db, size_t n, cudaStream_t s) {
  const bool wanted = n >= kQuadMinRecords && db->have_query && db->n_pad >= kQuadMinRows;
  return !wanted && !db->dot_captured && !db->sums_pinned && !stream_captures(s);
}

// The sums of records [first, first + n) from the planes (the lock is held).
cudaError_t derive_sums(irs_sharedb* db, size_t first, size_t n, cudaStream_t s) {
  const size_t K = db->code_length, cap = db->db_cap, o = K / 2, i = 3 * K / 4;
  uint8_t* inner = db->sums + 2 * cap * o;
  return launch_derive_sums(db->db_lo + first * K, db->db_hi + first * K, (uint32_t)K, n, db->sums + first * o,
                            db->sums + cap * o + first * o, inner + first * i, inner + cap * i + first * i, s);
}

// Brings the sums of records [first, first + n) in line with the planes, on
// the stream that wrote them.
cudaError_t update_sums(irs_sharedb* db, size_t first, size_t n, cudaStream_t s) {
  SumReader lock(sum_holders(db).mu);
  if (!db->sums || !n) return cudaSuccess;
  if (stream_captures(s)) db->sums_pinned = true;
  return derive_sums(db, first, n, s);
}

// Brings the sums that gathers left behind in line, on the party's stream, which
// every dot waits for (the lock is held; no capture on that stream).
cudaError_t fresh_sums(irs_sharedb* db) {
  const cudaError_t e = derive_sums(db, 0, db->stale_end, db->dm->streams[db->peer]);
  if (e == cudaSuccess) db->stale_end = 0;
  return e;
}

// Prepares the query forms' tensor maps for the active row count; false where
// the quad GEMM does not run.
bool quad_forms_ready(irs_sharedb* db) {
  if (!db->sums || db->n_pad < kQuadMinRows || db->rows_captured) return false;
  if (db->forms_pad == db->n_pad) return true;
  const size_t K = db->code_length, rows = kQuadProducts * (db->n_pad / 4);
  db->forms_pad = 0;
  for (int w = 0; w < kQuadWidths; w++) {
    const uint32_t box = (uint32_t)quad_tile_n((uint32_t)db->n_pad, w) / 2;
    if (make_tmap_plane(&db->tm_form_lo[w], db->forms, rows, K / 4, box) ||
        make_tmap_plane(&db->tm_form_hi[w], db->forms + rows * (K / 4), rows, K / 4, box))
      return false;
  }
  db->forms_pad = db->n_pad;
  return true;
}

// Whether the live rows of every quad (rows i, i + 2, i + 4, i + 6 of a slot,
// i in 0, 1, 8, 9, ...) are rotations of one base that keep their distance:
// the rows the quad GEMM can run.  Empty rows fit anywhere.
bool rows_are_quads(const uint32_t* desc, size_t n_rows) {
  for (size_t b = 0; b < n_rows; b += 8)
    for (size_t i = b; i < b + 2; i++) {
      uint32_t want = 0xFFFFFFFFu;  // descriptor of row i, rotation counted back to it (mod 2^32)
      for (size_t m = 0; m < 4; m++) {
        const size_t r = i + 2 * m;
        if (r >= n_rows || desc[r] == 0xFFFFFFFFu) continue;
        // the rotation field has 7 bits and holds at most 30: + 64 keeps the
        // subtraction inside it
        const uint32_t back = desc[r] + 64 - (uint32_t)(2 * m);
        if (want == 0xFFFFFFFFu) want = back;
        else if (want != back) return false;
      }
    }
  return true;
}

uint8_t* forms_hi(irs_sharedb* db) { return db->forms + kQuadProducts * (db->n_pad / 4) * (db->code_length / 4); }

// Notes whether the rows about to be expanded are quads, and where the
// expansion puts their forms and (if it changes) the device flag.  The sums'
// lock is held until the expansion is enqueued.  An upload that is captured
// (on `s`) writes planes alone, and so do the engine's later ones: what the
// rows are after a replay is not known here.
QuadForms begin_forms(irs_sharedb* db, bool quads, cudaStream_t s) {
  if (stream_captures(s)) db->rows_captured = true;
  quads = quads && !db->rows_captured;
  db->quad_rows = quads;
  QuadForms f{nullptr, nullptr, nullptr, nullptr};
  if (quads) f = {db->forms, forms_hi(db), db->row_valid, nullptr};
  const uint32_t rows = quads ? (uint32_t)db->n_pad : 0u;
  if (db->quad_flag && (db->flag_rows != rows || db->rows_captured)) {
    f.flag = db->quad_flag;
    db->flag_rows = rows;
  }
  return f;
}

// Planes and forms of a row table whose bases and table are in the staging.
int expand_row_table(irs_sharedb* db, const uint32_t* desc, size_t n_rows, const uint32_t* d_desc, cudaStream_t s) {
  SumReader lock(sum_holders(db).mu);
  const QuadForms f = begin_forms(db, quad_forms_ready(db) && rows_are_quads(desc, n_rows), s);
  CU(launch_expand_rows(db->q_stage, (uint32_t)db->code_length, d_desc, (uint32_t)n_rows, (uint32_t)db->n_pad, db->q_lo,
                        db->q_hi, f, s));
  return IRS_OK;
}

int set_active_rows(irs_sharedb* db, size_t rows) {
  const size_t n = padded_query_rows(rows, db->n_cap);
  if (n > db->n_cap) return fail(IRS_ERR_INVALID, "%zu rows exceed the query capacity %zu", rows, db->n_cap);
  if (n != db->n_pad) db->quad_rows = false;  // the forms are for another row count; the upload decides
  int bn = gemm_block_n_for((uint32_t)n);
  if (db->tile_override && n % (size_t)db->tile_override == 0) bn = db->tile_override;
  const bool rebuild = bn != db->block_n || n != db->n_pad;
  db->n_pad = n;
  db->block_n = bn;
  db->rows_uploaded = rows;
  return rebuild ? rebuild_query_maps(db) : IRS_OK;
}

}  // namespace

extern "C" {

const char* irs_last_error(void) { return g_err; }

const char* irs_version(void) { return "irisb200 0.1 (sm_100a, tcgen05 i8 limb GEMM, fused 3-party threshold)"; }

// ---------------------------------------------------------------------------
// Device manager
// ---------------------------------------------------------------------------
int irs_device_manager_init(int device, irs_device_manager** out) {
  CHECK(out, IRS_ERR_INVALID, "out is NULL");
  *out = nullptr;
  int n = 0;
  CU(cudaGetDeviceCount(&n));
  CHECK(device >= 0 && device < n, IRS_ERR_INVALID, "device %d out of range (%d devices)", device, n);
  CU(cudaSetDevice(device));
  cudaDeviceProp prop;
  CU(cudaGetDeviceProperties(&prop, device));
  CHECK(prop.major == 10 && prop.minor == 0, IRS_ERR_INVALID,
        "device %d is sm_%d%d; this library is built for sm_100a (B200)", device, prop.major, prop.minor);
  auto* dm = new (std::nothrow) irs_device_manager();
  CHECK(dm, IRS_ERR_NOMEM, "host allocation failed");
  dm->device = device;
  dm->n_sms = prop.multiProcessorCount;
  for (int p = 0; p < 3; p++) {
    CU(cudaStreamCreateWithFlags(&dm->streams[p], cudaStreamNonBlocking));
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    CU(cudaMemPoolCreate(&dm->pools[p], &props));
    uint64_t threshold = UINT64_MAX;
    CU(cudaMemPoolSetAttribute(dm->pools[p], cudaMemPoolAttrReleaseThreshold, &threshold));
  }
  CU(cudaMalloc(&dm->d_err, sizeof(int)));
  CU(cudaMemset(dm->d_err, 0, sizeof(int)));
  CU(cudaMalloc(&dm->d_batch, sizeof(uint64_t)));
  CU(cudaMemset(dm->d_batch, 0, sizeof(uint64_t)));
  CU(cudaEventCreateWithFlags(&dm->graph_done, cudaEventDisableTiming));
  for (cudaEvent_t& e : dm->uploads) CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  try {
    SumWriter lock(sum_holders(device).mu);
    sum_holders(device).managers.push_back(dm);
  } catch (const std::bad_alloc&) {
    irs_device_manager_destroy(dm);
    return fail(IRS_ERR_NOMEM, "host allocation failed");
  }
  *out = dm;
  return IRS_OK;
}

int irs_device_manager_destroy(irs_device_manager* dm) {
  if (!dm) return IRS_OK;
  cudaSetDevice(dm->device);
  {
    SumWriter lock(sum_holders(dm->device).mu);
    auto& v = sum_holders(dm->device).managers;
    v.erase(std::remove(v.begin(), v.end(), dm), v.end());
  }
  for (int p = 0; p < 3; p++) if (dm->streams[p]) cudaStreamSynchronize(dm->streams[p]);
  cudaFree(dm->d_err);
  cudaFree(dm->d_batch);
  if (dm->graph_done) cudaEventDestroy(dm->graph_done);
  if (dm->graph_ran) cudaEventDestroy(dm->graph_ran);
  if (dm->graph_join) cudaStreamDestroy(dm->graph_join);
  for (cudaEvent_t e : dm->uploads)
    if (e) cudaEventDestroy(e);
  for (auto& t : dm->timers) {
    cudaEventDestroy(t.start);
    cudaEventDestroy(t.stop);
  }
  for (int p = 0; p < 3; p++) {
    if (dm->streams[p]) cudaStreamDestroy(dm->streams[p]);
    if (dm->pools[p]) cudaMemPoolDestroy(dm->pools[p]);
  }
  delete dm;
  return IRS_OK;
}

int irs_device_manager_stream(irs_device_manager* dm, int party, void** stream) {
  CHECK(dm && stream && party >= 0 && party < 3, IRS_ERR_INVALID, "bad arguments");
  *stream = dm->streams[party];
  return IRS_OK;
}

int irs_device_manager_synchronize(irs_device_manager* dm) {
  CHECK(dm, IRS_ERR_INVALID, "dm is NULL");
  for (int p = 0; p < 3; p++) CU(cudaStreamSynchronize(dm->streams[p]));
  return check_device_error(dm);
}

int irs_device_manager_error(irs_device_manager* dm, int* code) {
  CHECK(dm && code, IRS_ERR_INVALID, "bad arguments");
  CU(cudaMemcpy(code, dm->d_err, sizeof(int), cudaMemcpyDeviceToHost));
  return IRS_OK;
}

int irs_device_manager_clear_error(irs_device_manager* dm) {
  CHECK(dm, IRS_ERR_INVALID, "dm is NULL");
  CU(cudaMemset(dm->d_err, 0, sizeof(int)));
  return IRS_OK;
}

int irs_device_manager_test_stall_next_dot(irs_device_manager* dm, uint64_t wait_limit_ns) {
  CHECK(dm, IRS_ERR_INVALID, "dm is NULL");
  CHECK(wait_limit_ns >= 1000 && wait_limit_ns <= 10000000000ull, IRS_ERR_INVALID,
        "wait limit %llu ns outside 1 us .. 10 s", (unsigned long long)wait_limit_ns);
  CHECK(!dm->capturing, IRS_ERR_STATE, "arm the stall outside a graph capture");
  dm->stall_limit_ns = wait_limit_ns;
  return IRS_OK;
}

int irs_device_manager_set_batch_counter(irs_device_manager* dm, uint64_t batch_id, void* stream) {
  CHECK(dm, IRS_ERR_INVALID, "dm is NULL");
  CHECK(batch_id < (1ull << 24), IRS_ERR_INVALID, "batch id must be below 2^24");
  CHECK(!dm->capturing, IRS_ERR_STATE, "set the batch counter outside a graph capture");
  static thread_local uint64_t staged;  // pageable source; the copy is synchronised below
  staged = batch_id;
  cudaStream_t s = party_stream(dm, 0, stream);
  CU(cudaMemcpyAsync(dm->d_batch, &staged, sizeof(uint64_t), cudaMemcpyHostToDevice, s));
  CU(cudaStreamSynchronize(s));
  return IRS_OK;
}

__global__ void advance_batch_counter_kernel(uint64_t* b) { *b = *b % ((1ull << 24) - 1) + 1; }

int irs_device_manager_set_timing(irs_device_manager* dm, int on) {
  CHECK(dm, IRS_ERR_INVALID, "dm is NULL");
  dm->timing = on != 0;
  return IRS_OK;
}

int irs_device_manager_timings(irs_device_manager* dm, char* buf, size_t cap, int reset) {
  CHECK(dm && buf && cap > 0, IRS_ERR_INVALID, "bad arguments");
  CU(cudaSetDevice(dm->device));
  for (auto& t : dm->timers) {
    float ms = 0.f;
    CU(cudaEventSynchronize(t.stop));
    CU(cudaEventElapsedTime(&ms, t.start, t.stop));
    auto& tot = dm->timer_totals[t.label];
    tot.first += ms;
    tot.second += 1;
    cudaEventDestroy(t.start);
    cudaEventDestroy(t.stop);
  }
  dm->timers.clear();
  std::string out;
  char line[160];
  for (auto& kv : dm->timer_totals) {
    snprintf(line, sizeof line, "%s%s=%.6f/%ld", out.empty() ? "" : ";", kv.first.c_str(), kv.second.first,
             kv.second.second);
    out += line;
  }
  CHECK(out.size() + 1 <= cap, IRS_ERR_OVERFLOW, "timings need %zu bytes", out.size() + 1);
  memcpy(buf, out.c_str(), out.size() + 1);
  if (reset) dm->timer_totals.clear();
  return IRS_OK;
}

int irs_device_manager_get_batch_counter(irs_device_manager* dm, uint64_t* batch_id) {
  CHECK(dm && batch_id, IRS_ERR_INVALID, "bad arguments");
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  CU(cudaMemcpyAsync(batch_id, dm->d_batch, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  return IRS_OK;
}

int irs_device_manager_advance_batch_counter(irs_device_manager* dm, void* stream) {
  CHECK(dm, IRS_ERR_INVALID, "dm is NULL");
  CU(cudaSetDevice(dm->device));
  advance_batch_counter_kernel<<<1, 1, 0, party_stream(dm, 0, stream)>>>(dm->d_batch);
  CU(cudaGetLastError());
  return IRS_OK;
}

int irs_sharedb_use_batch_counter(irs_sharedb* db, int on) {
  CHECK(db, IRS_ERR_INVALID, "db is NULL");
  db->batch_from_device = on != 0;
  return IRS_OK;
}

int irs_circuits_use_batch_counter(irs_circuits* c, int on) {
  CHECK(c, IRS_ERR_INVALID, "c is NULL");
  c->batch_from_device = on != 0;
  return IRS_OK;
}

int irs_device_manager_set_host_sync(irs_device_manager* dm, int on) {
  CHECK(dm, IRS_ERR_INVALID, "dm is NULL");
  dm->host_sync = on != 0;
  return IRS_OK;
}

int irs_event_create(void** ev) {
  CHECK(ev, IRS_ERR_INVALID, "ev is NULL");
  cudaEvent_t e = nullptr;
  CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  *ev = e;
  return IRS_OK;
}

int irs_event_record(void* ev, void* stream) {
  CHECK(ev, IRS_ERR_INVALID, "ev is NULL");
  CU(cudaEventRecord(static_cast<cudaEvent_t>(ev), static_cast<cudaStream_t>(stream)));
  return IRS_OK;
}

int irs_event_synchronize(void* ev) {
  CHECK(ev, IRS_ERR_INVALID, "ev is NULL");
  CU(cudaEventSynchronize(static_cast<cudaEvent_t>(ev)));
  return IRS_OK;
}

int irs_event_query(void* ev, int* done) {
  CHECK(ev && done, IRS_ERR_INVALID, "bad arguments");
  const cudaError_t e = cudaEventQuery(static_cast<cudaEvent_t>(ev));
  if (e == cudaErrorNotReady) {
    *done = 0;
    return IRS_OK;
  }
  CU(e);
  *done = 1;
  return IRS_OK;
}

int irs_event_destroy(void* ev) {
  if (ev) cudaEventDestroy(static_cast<cudaEvent_t>(ev));
  return IRS_OK;
}

int irs_device_manager_mem_info(irs_device_manager* dm, size_t* free_bytes, size_t* total_bytes) {
  CHECK(dm && free_bytes && total_bytes, IRS_ERR_INVALID, "bad arguments");
  CU(cudaSetDevice(dm->device));
  CU(cudaMemGetInfo(free_bytes, total_bytes));
  return IRS_OK;
}

int irs_device_manager_derived(irs_device_manager* dm, int give_back, size_t* bytes) {
  CHECK(dm && bytes, IRS_ERR_INVALID, "bad arguments");
  CU(cudaSetDevice(dm->device));
  while (give_back && reclaim_sums(dm->device)) {}
  *bytes = reclaimable_sums(dm->device);
  return IRS_OK;
}

int irs_device_manager_sm_count(irs_device_manager* dm, int* n) {
  CHECK(dm && n, IRS_ERR_INVALID, "bad arguments");
  *n = dm->n_sms;
  return IRS_OK;
}

int irs_device_alloc(irs_device_manager* dm, size_t bytes, void** ptr) {
  CHECK(dm && ptr, IRS_ERR_INVALID, "bad arguments");
  cudaError_t e = device_malloc(dm, ptr, bytes ? bytes : 16);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(IRS_ERR_NOMEM, "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
  }
  return IRS_OK;
}

int irs_host_alloc_pinned(size_t bytes, void** ptr) {
  CHECK(ptr, IRS_ERR_INVALID, "ptr is NULL");
  cudaError_t e = cudaMallocHost(ptr, bytes ? bytes : 16);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(IRS_ERR_NOMEM, "cudaMallocHost(%zu): %s", bytes, cudaGetErrorString(e));
  }
  return IRS_OK;
}

int irs_host_free_pinned(void* ptr) {
  if (ptr) CU(cudaFreeHost(ptr));
  return IRS_OK;
}

int irs_device_free(irs_device_manager* dm, void* ptr) {
  (void)dm;
  if (ptr) CU(cudaFree(ptr));
  return IRS_OK;
}

int irs_copy_h2d(void* dst, const void* src, size_t bytes, void* stream) {
  CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, static_cast<cudaStream_t>(stream)));
  return IRS_OK;
}

int irs_copy_d2h(void* dst, const void* src, size_t bytes, void* stream) {
  CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, static_cast<cudaStream_t>(stream)));
  return IRS_OK;
}

int irs_stream_synchronize(void* stream) {
  CU(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  return IRS_OK;
}

// ---------------------------------------------------------------------------
// ShareDB
// ---------------------------------------------------------------------------
int irs_sharedb_init(irs_device_manager* dm, int peer_id, size_t max_db_length, size_t query_length,
                     size_t code_length, const uint32_t seed0[8], const uint32_t seed1[8], int is_remote,
                     irs_sharedb** out) {
  CHECK(dm && out && seed0 && seed1, IRS_ERR_INVALID, "bad arguments");
  *out = nullptr;
  CHECK(peer_id >= 0 && peer_id < 3, IRS_ERR_INVALID, "peer_id %d not in 0..2", peer_id);
  CHECK(code_length > 0 && code_length % 128 == 0, IRS_ERR_INVALID, "code_length %zu must be a multiple of 128",
        code_length);
  CHECK(query_length > 0 && query_length <= 65536, IRS_ERR_INVALID, "query_length %zu out of range", query_length);
  CHECK(max_db_length > 0 && max_db_length < (1ull << 31), IRS_ERR_INVALID, "max_db_length %zu out of range",
        max_db_length);
  CU(cudaSetDevice(dm->device));
  auto* db = new (std::nothrow) irs_sharedb();
  CHECK(db, IRS_ERR_NOMEM, "host allocation failed");
  db->dm = dm;
  db->peer = peer_id;
  db->max_db = max_db_length;
  db->query_length = query_length;
  db->code_length = code_length;
  db->seed0 = key_of(seed0);
  db->seed1 = key_of(seed1);
  db->remote = is_remote != 0;
  db->n_cap = round_up(query_length, 64);
  db->n_pad = db->n_cap;
  db->block_n = gemm_block_n_for((uint32_t)db->n_pad);
  if (cudaEventCreateWithFlags(&db->done, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&db->copied, cudaEventDisableTiming) != cudaSuccess) {
    if (db->done) cudaEventDestroy(db->done);
    delete db;
    return fail(IRS_ERR_CUDA, "event creation failed");
  }
  int rc;
  void* p;
  if ((rc = pool_alloc(dm, peer_id, db->n_cap * code_length, &p))) { irs_sharedb_destroy(db); return rc; }
  db->q_lo = (uint8_t*)p;
  if ((rc = pool_alloc(dm, peer_id, db->n_cap * code_length, &p))) { irs_sharedb_destroy(db); return rc; }
  db->q_hi = (uint8_t*)p;
  if ((rc = pool_alloc(dm, peer_id, db->n_cap * code_length * 2, &p))) { irs_sharedb_destroy(db); return rc; }
  db->q_stage = (uint16_t*)p;
  if ((rc = pool_alloc(dm, peer_id, (db->n_cap / kSlotRows) * sizeof(QuerySlot), &p))) { irs_sharedb_destroy(db); return rc; }
  db->d_slots = (QuerySlot*)p;
  if ((rc = pool_alloc(dm, peer_id, max_db_length * db->n_cap * 2, &p))) { irs_sharedb_destroy(db); return rc; }
  db->results = (uint16_t*)p;
  if ((rc = rebuild_query_maps(db))) {
    irs_sharedb_destroy(db);
    return rc;
  }
  *out = db;
  return IRS_OK;
}

int irs_sharedb_destroy(irs_sharedb* db) {
  if (!db) return IRS_OK;
  irs_device_manager* dm = db->dm;
  cudaSetDevice(dm->device);
  db->dot_captured = false;  // no graph over the engine is launched any more
  drop_sums(db);
  pool_free(dm, db->peer, db->db_lo);
  pool_free(dm, db->peer, db->db_hi);
  pool_free(dm, db->peer, db->q_lo);
  pool_free(dm, db->peer, db->q_hi);
  pool_free(dm, db->peer, db->q_stage);
  pool_free(dm, db->peer, db->d_slots);
  pool_free(dm, db->peer, db->results);
  pool_free(dm, db->peer, db->quad_flag);
  for (uint32_t* w : db->old_flags) pool_free(dm, db->peer, w);
  cudaStreamSynchronize(dm->streams[db->peer]);
  if (db->done) cudaEventDestroy(db->done);
  if (db->copied) cudaEventDestroy(db->copied);
  delete db;
  return IRS_OK;
}

int irs_sharedb_alloc_db(irs_sharedb* db, size_t max_db_length) {
  CHECK(db, IRS_ERR_INVALID, "db is NULL");
  CHECK(max_db_length > 0 && max_db_length < (1ull << 31), IRS_ERR_INVALID, "max_db_length %zu out of range",
        max_db_length);
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  drop_sums(db);
  pool_free(dm, db->peer, db->db_lo);
  pool_free(dm, db->peer, db->db_hi);
  db->db_lo = db->db_hi = nullptr;
  const size_t cap = round_up(max_db_length, 128);
  void* p;
  int rc;
  if ((rc = pool_alloc(dm, db->peer, cap * db->code_length, &p))) return rc;
  db->db_lo = (uint8_t*)p;
  if ((rc = pool_alloc(dm, db->peer, cap * db->code_length, &p))) return rc;
  db->db_hi = (uint8_t*)p;
  CU(cudaMemsetAsync(db->db_lo, 0, cap * db->code_length, dm->streams[db->peer]));
  CU(cudaMemsetAsync(db->db_hi, 0, cap * db->code_length, dm->streams[db->peer]));
  db->db_cap = cap;
  db->db_len = 0;
  if (make_tmap_u8(&db->tm_db_lo, db->db_lo, cap, db->code_length, 128) ||
      make_tmap_u8(&db->tm_db_hi, db->db_hi, cap, db->code_length, 128))
    return fail(IRS_ERR_CUDA, "tensor map for the DB planes failed");
  alloc_sums(db);
  CU(cudaStreamSynchronize(dm->streams[db->peer]));
  return IRS_OK;
}

int irs_sharedb_load_records(irs_sharedb* db, size_t first, size_t n, const uint16_t* records) {
  CHECK(db && (records || !n), IRS_ERR_INVALID, "bad arguments");
  CHECK(db->db_lo, IRS_ERR_STATE, "alloc_db not called");
  CHECK(first + n <= db->db_cap, IRS_ERR_INVALID, "records %zu..%zu exceed the DB capacity %zu", first, first + n,
        db->db_cap);
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  const size_t K = db->code_length;
  const size_t per = std::max<size_t>(1, db->n_cap);  // records per pass through the query staging buffer
  for (size_t done = 0; done < n;) {
    const size_t c = std::min(per, n - done);
    CU(cudaMemcpyAsync(db->q_stage, records + done * K, c * K * 2, cudaMemcpyHostToDevice, s));
    CU(launch_split_limbs(db->q_stage, (uint32_t)K, db->db_lo + (first + done) * K, db->db_hi + (first + done) * K,
                          c * K, s));
    CU(update_sums(db, first + done, c, s));
    CU(cudaStreamSynchronize(s));
    done += c;
  }
  db->db_len = std::max(db->db_len, first + n);
  return IRS_OK;
}

int irs_sharedb_load_records_i8(irs_sharedb* db, size_t first, size_t n, const uint8_t* limb0, const uint8_t* limb1) {
  CHECK(db && ((limb0 && limb1) || !n), IRS_ERR_INVALID, "bad arguments");
  CHECK(db->db_lo, IRS_ERR_STATE, "alloc_db not called");
  CHECK(first + n <= db->db_cap, IRS_ERR_INVALID, "records exceed the DB capacity");
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  const size_t K = db->code_length;
  uint8_t* planes[2] = {db->db_lo + first * K, db->db_hi + first * K};
  const uint8_t* limbs[2] = {limb0, limb1};
  if (i8_plane_in_place(K)) {
    for (int l = 0; l < 2; l++) {
      CU(cudaMemcpyAsync(planes[l], limbs[l], n * K, cudaMemcpyHostToDevice, s));
      CU(launch_i8_plane(planes[l], (uint32_t)K, planes[l], n, s));
    }
  } else {  // a row at a time (the query staging may hold a server's resident bases)
    void* stage = nullptr;
    int rc = n ? pool_alloc(dm, db->peer, K, &stage) : IRS_OK;
    if (rc) return rc;
    cudaError_t e = cudaSuccess;
    for (size_t r = 0; r < 2 * n && e == cudaSuccess; r++) {
      e = cudaMemcpyAsync(stage, limbs[r & 1] + r / 2 * K, K, cudaMemcpyHostToDevice, s);
      if (e == cudaSuccess)
        e = launch_i8_plane(static_cast<uint8_t*>(stage), (uint32_t)K, planes[r & 1] + r / 2 * K, 1, s);
    }
    pool_free(dm, db->peer, stage);
    CU(e);
  }
  CU(update_sums(db, first, n, s));
  CU(cudaStreamSynchronize(s));
  db->db_len = std::max(db->db_len, first + n);
  return IRS_OK;
}

int irs_sharedb_fetch_records(irs_sharedb* db, size_t first, size_t n, uint16_t* records) {
  CHECK(db && (records || !n), IRS_ERR_INVALID, "bad arguments");
  CHECK(db->db_lo, IRS_ERR_STATE, "alloc_db not called");
  CHECK(first + n <= db->db_cap, IRS_ERR_INVALID, "records exceed the DB capacity");
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  const size_t K = db->code_length;
  std::vector<uint8_t> lo(n * K), hi(n * K);
  CU(cudaMemcpyAsync(lo.data(), db->db_lo + first * K, n * K, cudaMemcpyDeviceToHost, s));
  CU(cudaMemcpyAsync(hi.data(), db->db_hi + first * K, n * K, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  // planes are in quarter order (prep.cu): octet o of a row sits in quarter o % 4
  for (size_t r = 0; r < n; r++)
    for (size_t q = 0; q < 4; q++) {
      const uint8_t *l = &lo[r * K + q * (K / 4)], *h = &hi[r * K + q * (K / 4)];
      uint16_t* out = records + r * K + 8 * q;
      for (size_t o = 0; o < K / 32; o++, l += 8, h += 8, out += 32)
        for (int k = 0; k < 8; k++) out[k] = (uint16_t)(l[k] | (h[k] << 8));
    }
  return IRS_OK;
}

int irs_sharedb_set_db_len(irs_sharedb* db, size_t len) {
  CHECK(db, IRS_ERR_INVALID, "db is NULL");
  CHECK(len <= db->db_cap, IRS_ERR_INVALID, "len %zu exceeds capacity %zu", len, db->db_cap);
  db->db_len = len;
  return IRS_OK;
}

int irs_sharedb_db_len(irs_sharedb* db, size_t* len) {
  CHECK(db && len, IRS_ERR_INVALID, "bad arguments");
  *len = db->db_len;
  return IRS_OK;
}

int irs_sharedb_synth_db(irs_sharedb* const code_engines[3], irs_sharedb* const mask_engines[3], uint64_t seed,
                         size_t first, size_t n) {
  SynthOut o;
  for (int p = 0; p < 3; p++) {
    irs_sharedb* c = code_engines[p];
    irs_sharedb* m = mask_engines[p];
    CHECK(c && m && c->db_lo && m->db_lo, IRS_ERR_STATE, "engines of party %d need alloc_db", p);
    CHECK(c->code_length == (size_t)kIrisCodeLength && m->code_length == (size_t)kMaskCodeLength, IRS_ERR_INVALID,
          "synthetic DB needs code_length 12800 / 6400 engines");
    CHECK(first + n <= c->db_cap && first + n <= m->db_cap, IRS_ERR_INVALID, "records exceed the DB capacity");
    o.code_lo[p] = c->db_lo; o.code_hi[p] = c->db_hi;
    o.mask_lo[p] = m->db_lo; o.mask_hi[p] = m->db_hi;
  }
  irs_device_manager* dm = code_engines[0]->dm;
  CU(cudaSetDevice(dm->device));
  for (int p = 0; p < 3; p++) {
    CU(cudaStreamSynchronize(dm->streams[p]));
  }
  const size_t step = 1u << 20;
  for (size_t done = 0; done < n; done += step) {
    const uint32_t c = (uint32_t)std::min(step, n - done);
    CU(launch_synth_db(seed, (uint32_t)(first + done), c, o, dm->streams[0]));
  }
  for (int p = 0; p < 3; p++) {
    CU(update_sums(code_engines[p], first, n, dm->streams[0]));
    CU(update_sums(mask_engines[p], first, n, dm->streams[0]));
  }
  CU(cudaStreamSynchronize(dm->streams[0]));
  for (int p = 0; p < 3; p++) {
    code_engines[p]->db_len = std::max(code_engines[p]->db_len, first + n);
    mask_engines[p]->db_len = std::max(mask_engines[p]->db_len, first + n);
  }
  return IRS_OK;
}

// Orders a write to an engine's query rows or records on stream s after the
// last GEMMs that read them (a direct launch, and every graph launch).
static cudaError_t wait_last_dot(irs_sharedb* db, cudaStream_t s) {
  cudaError_t e = cudaStreamWaitEvent(s, db->done, 0);
  if (e != cudaSuccess) return e;
  return cudaStreamWaitEvent(s, db->dm->graph_done, 0);
}

int irs_sharedb_fill_random(irs_sharedb* db, uint64_t seed, size_t n) {
  CHECK(db && db->db_lo, IRS_ERR_STATE, "alloc_db not called");
  CHECK(n <= db->db_cap, IRS_ERR_INVALID, "%zu records exceed the DB capacity %zu", n, db->db_cap);
  CHECK((n * db->code_length) % 8 == 0, IRS_ERR_INVALID, "records x code_length must be a multiple of 8");
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  CU(wait_last_dot(db, s));
  const uint32_t K = (uint32_t)db->code_length;
  CU(launch_fill_random(db->db_lo, n * db->code_length, seed, K, s));
  CU(launch_fill_random(db->db_hi, n * db->code_length, seed ^ 0x5A5A5A5A5A5A5A5Aull, K, s));
  CU(update_sums(db, 0, n, s));
  CU(cudaStreamSynchronize(s));
  db->db_len = std::max(db->db_len, n);
  return IRS_OK;
}

int irs_device_fill_random(void* ptr, size_t bytes, uint64_t seed, void* stream) {
  CHECK(ptr && bytes % 8 == 0 && reinterpret_cast<uintptr_t>(ptr) % 8 == 0, IRS_ERR_INVALID,
        "8-byte aligned pointer and a multiple of 8 bytes needed");
  CU(launch_fill_random(ptr, bytes, seed, 0, static_cast<cudaStream_t>(stream)));
  return IRS_OK;
}

int irs_sharedb_query_upload(irs_sharedb* db, const uint16_t* rows, size_t n_rows) {
  CHECK(db && (rows || !n_rows), IRS_ERR_INVALID, "bad arguments");
  int rc = set_active_rows(db, n_rows);
  if (rc) return rc;
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  CU(wait_last_dot(db, s));  // the last GEMM has read the old limb planes
  const size_t K = db->code_length;
  CU(cudaMemsetAsync(db->q_stage, 0, db->n_pad * K * 2, s));
  if (n_rows) CU(cudaMemcpyAsync(db->q_stage, rows, n_rows * K * 2, cudaMemcpyHostToDevice, s));
  CU(launch_split_limbs(db->q_stage, (uint32_t)K, db->q_lo, db->q_hi, db->n_pad * K, s));
  {
    SumReader lock(sum_holders(db).mu);
    if (begin_forms(db, false, s).flag) CU(cudaMemsetAsync(db->quad_flag, 0, 4, s));  // rows of no known structure
  }
  db->have_query = true;
  return IRS_OK;
}

int irs_sharedb_query_upload_slots(irs_sharedb* db, const uint16_t* base, size_t n_base, const irs_query_slot* slots,
                                   size_t n_slots) {
  CHECK(db && base && slots && n_base > 0, IRS_ERR_INVALID, "bad arguments");
  CHECK(n_slots * kSlotRows <= db->n_cap, IRS_ERR_INVALID, "%zu slots exceed the query capacity %zu", n_slots,
        db->n_cap);
  CHECK(n_base <= db->n_cap, IRS_ERR_INVALID, "too many base queries");
  CHECK(db->code_length % kRowLen == 0, IRS_ERR_INVALID, "rotations need code_length a multiple of 800");
  for (size_t i = 0; i < n_slots; i++) {
    CHECK(slots[i].src < n_base && slots[i].n_rot <= (uint32_t)kRotations &&
              slots[i].rot_lo + slots[i].n_rot <= (uint32_t)kRotations,
          IRS_ERR_INVALID, "slot %zu is invalid", i);
  }
  int rc = set_active_rows(db, n_slots * kSlotRows);
  if (rc) return rc;
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  CU(wait_last_dot(db, s));
  const size_t K = db->code_length;
  CU(cudaMemcpyAsync(db->q_stage, base, n_base * K * 2, cudaMemcpyHostToDevice, s));
  static_assert(sizeof(QuerySlot) == sizeof(irs_query_slot), "slot layout");
  CU(cudaMemcpyAsync(db->d_slots, slots, n_slots * sizeof(QuerySlot), cudaMemcpyHostToDevice, s));
  CU(cudaEventRecord(db->copied, s));
  {
    SumReader lock(sum_holders(db).mu);
    const QuadForms f = begin_forms(db, quad_forms_ready(db), s);  // a slot's rows are consecutive rotations
    CU(launch_expand_slots(db->q_stage, (uint32_t)K, db->d_slots, (uint32_t)n_slots, (uint32_t)db->n_pad, db->q_lo,
                           db->q_hi, f, s));
  }
  CU(cudaEventSynchronize(db->copied));  // slots / base are caller-owned host memory
  db->have_query = true;
  return IRS_OK;
}

int irs_sharedb_query_upload_rows(irs_sharedb* db, const uint16_t* base, size_t n_base, const uint32_t* row_desc,
                                  size_t n_rows) {
  CHECK(db && base && row_desc && n_base > 0, IRS_ERR_INVALID, "bad arguments");
  CHECK(db->code_length % kRowLen == 0, IRS_ERR_INVALID, "rotations need code_length a multiple of 800");
  const size_t K = db->code_length;
  // staging: base queries, then the row table after them
  const size_t base_bytes = n_base * K * 2, table_bytes = n_rows * 4;
  CHECK(base_bytes + table_bytes + 16 <= db->n_cap * K * 2, IRS_ERR_INVALID, "too many base queries for the staging");
  for (size_t r = 0; r < n_rows; r++)
    CHECK(row_desc[r] == 0xFFFFFFFFu || ((row_desc[r] >> 8) < n_base && (row_desc[r] & 0x7Fu) < (uint32_t)kRotations),
          IRS_ERR_INVALID, "row %zu descriptor 0x%x is invalid", r, row_desc[r]);
  int rc = set_active_rows(db, n_rows);
  if (rc) return rc;
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  CU(wait_last_dot(db, s));
  uint8_t* stage = reinterpret_cast<uint8_t*>(db->q_stage);
  const size_t table_off = (base_bytes + 15) / 16 * 16;
  CU(cudaMemcpyAsync(stage, base, base_bytes, cudaMemcpyHostToDevice, s));
  CU(cudaMemcpyAsync(stage + table_off, row_desc, table_bytes, cudaMemcpyHostToDevice, s));
  if (dm->host_sync) CU(cudaEventRecord(db->copied, s));
  if ((rc = expand_row_table(db, row_desc, n_rows, reinterpret_cast<const uint32_t*>(stage + table_off), s))) return rc;
  if (dm->host_sync) CU(cudaEventSynchronize(db->copied));  // base / row_desc are caller-owned host memory
  db->have_query = true;
  return IRS_OK;
}

int irs_sharedb_query_put_base(irs_sharedb* db, size_t first, size_t n, const uint16_t* base) {
  CHECK(db && (base || !n), IRS_ERR_INVALID, "bad arguments");
  const size_t K = db->code_length;
  CHECK((first + n) * K * 2 + db->n_cap * 4 + 16 <= db->n_cap * K * 2, IRS_ERR_INVALID,
        "base queries [%zu, %zu) exceed the resident pool", first, first + n);
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  if (n) {
    CU(cudaMemcpyAsync(db->q_stage + first * K, base, n * K * 2, cudaMemcpyHostToDevice, s));
    if (dm->host_sync) CU(cudaStreamSynchronize(s));  // caller-owned host memory
  }
  return IRS_OK;
}

int irs_sharedb_query_expand_rows(irs_sharedb* db, size_t n_base, const uint32_t* row_desc, size_t n_rows) {
  CHECK(db && row_desc && n_base > 0, IRS_ERR_INVALID, "bad arguments");
  CHECK(db->code_length % kRowLen == 0, IRS_ERR_INVALID, "rotations need code_length a multiple of 800");
  const size_t K = db->code_length;
  const size_t base_bytes = n_base * K * 2, table_bytes = n_rows * 4;
  CHECK(base_bytes + table_bytes + 16 <= db->n_cap * K * 2, IRS_ERR_INVALID, "pool and row table exceed the staging");
  for (size_t r = 0; r < n_rows; r++)
    CHECK(row_desc[r] == 0xFFFFFFFFu || ((row_desc[r] >> 8) < n_base && (row_desc[r] & 0x7Fu) < (uint32_t)kRotations),
          IRS_ERR_INVALID, "row %zu descriptor 0x%x is invalid", r, row_desc[r]);
  int rc = set_active_rows(db, n_rows);
  if (rc) return rc;
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  CU(wait_last_dot(db, s));
  uint8_t* stage = reinterpret_cast<uint8_t*>(db->q_stage);
  const size_t table_off = (base_bytes + 15) / 16 * 16;
  CU(cudaMemcpyAsync(stage + table_off, row_desc, table_bytes, cudaMemcpyHostToDevice, s));
  if (dm->host_sync) CU(cudaEventRecord(db->copied, s));
  if ((rc = expand_row_table(db, row_desc, n_rows, reinterpret_cast<const uint32_t*>(stage + table_off), s))) return rc;
  if (dm->host_sync) CU(cudaEventSynchronize(db->copied));  // row_desc is caller-owned host memory
  db->have_query = true;
  return IRS_OK;
}

int irs_sharedb_gather_records(irs_sharedb* dst, irs_sharedb* src, const uint32_t* ids, size_t n) {
  CHECK(dst && src && (ids || !n), IRS_ERR_INVALID, "bad arguments");
  CHECK(dst->dm == src->dm && dst->peer == src->peer && dst->code_length == src->code_length, IRS_ERR_INVALID,
        "gather needs engines of the same party and code length");
  CHECK(dst->db_lo && src->db_lo, IRS_ERR_STATE, "alloc_db not called");
  CHECK(n <= dst->db_cap, IRS_ERR_INVALID, "%zu records exceed the destination capacity %zu", n, dst->db_cap);
  for (size_t k = 0; k < n; k++)
    CHECK(ids[k] < src->db_cap, IRS_ERR_INVALID, "record id %u out of range", ids[k]);
  irs_device_manager* dm = dst->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[dst->peer];
  CU(wait_last_dot(dst, s));  // the last GEMM over dst's records has finished
  const size_t K = dst->code_length;
  CHECK(n * 4 <= dst->n_cap * K * 2, IRS_ERR_INVALID, "too many records for one gather");
  // Staging reuse: the gather runs before the next query upload of `dst`.
  CU(cudaMemcpyAsync(dst->q_stage, ids, n * 4, cudaMemcpyHostToDevice, s));
  if (dm->host_sync) CU(cudaEventRecord(dst->copied, s));
  CU(launch_gather_rows(src->db_lo, src->db_hi, reinterpret_cast<const uint32_t*>(dst->q_stage), (uint32_t)n,
                        (uint32_t)K, dst->db_lo, dst->db_hi, s));
  if (dst->sums && gather_skips_sums(dst, n, s)) {
    dst->stale_end = std::max(dst->stale_end, n);
  } else {
    CU(update_sums(dst, 0, n, s));
    if (n >= dst->stale_end) dst->stale_end = 0;
  }
  if (dm->host_sync) CU(cudaEventSynchronize(dst->copied));  // ids is caller-owned host memory
  dst->db_len = n;
  return IRS_OK;
}

int irs_sharedb_set_tile(irs_sharedb* db, int block_n) {
  CHECK(db, IRS_ERR_INVALID, "db is NULL");
  CHECK(block_n == 0 || block_n == 64 || block_n == 128 || block_n == 256, IRS_ERR_INVALID,
        "tile width %d is not 0, 64, 128 or 256", block_n);
  db->tile_override = block_n;
  if (db->have_query) return set_active_rows(db, db->rows_uploaded);
  return IRS_OK;
}

int irs_sharedb_set_pair(irs_sharedb* db, int on) {
  CHECK(db, IRS_ERR_INVALID, "db is NULL");
  db->pair = on != 0;
  return IRS_OK;
}

int irs_sharedb_has_sums(irs_sharedb* db, int* on) {
  CHECK(db && on, IRS_ERR_INVALID, "bad arguments");
  SumReader lock(sum_holders(db).mu);
  *on = db->sums != nullptr;
  return IRS_OK;
}

int irs_sharedb_last_gemm(irs_sharedb* db, int* gemm, size_t* quad_rows) {
  CHECK(db && gemm && quad_rows, IRS_ERR_INVALID, "bad arguments");
  SumReader lock(sum_holders(db).mu);
  *gemm = db->last_gemm;
  *quad_rows = db->sums ? db->flag_rows : 0;
  return IRS_OK;
}

int irs_sharedb_set_batch(irs_sharedb* db, uint64_t batch_id) {
  CHECK(db, IRS_ERR_INVALID, "db is NULL");
  CHECK(batch_id < (1ull << 24), IRS_ERR_INVALID, "batch id must be below 2^24");
  db->batch = batch_id;
  return IRS_OK;
}

// The GEMM that a launch's query maps are for: the one-SM kernel on the engine's
// own tiles, the two-SM one, or the one-SM kernel on 64- or 128-row tiles.
enum class Gemm { kOneSm, kPair, k64, k128 };

static int fill_problem(irs_sharedb* db, uint16_t mult, size_t offset, size_t len, Gemm gemm, GemmProblem& pr) {
  CHECK(db->db_lo, IRS_ERR_STATE, "alloc_db not called");
  CHECK(db->have_query, IRS_ERR_STATE, "no query uploaded");
  CHECK(offset % 32 == 0, IRS_ERR_INVALID, "offset %zu must be a multiple of 32", offset);
  CHECK(offset + len <= db->db_cap && len <= db->max_db, IRS_ERR_INVALID, "entries %zu..%zu out of range", offset,
        offset + len);
  CHECK(db->block_n > 0, IRS_ERR_INVALID, "padded query length %zu has no valid tile width", db->n_pad);
  memset(&pr, 0, sizeof pr);
  pr.tm_a_lo = db->tm_db_lo;
  pr.tm_a_hi = db->tm_db_hi;
  const int f = gemm == Gemm::k128;
  pr.tm_b_lo = gemm == Gemm::kPair ? db->tm_qp_lo : gemm == Gemm::kOneSm ? db->tm_q_lo : db->tm_qf_lo[f];
  pr.tm_b_hi = gemm == Gemm::kPair ? db->tm_qp_hi : gemm == Gemm::kOneSm ? db->tm_q_hi : db->tm_qf_hi[f];
  pr.out = db->results;
  pr.m0 = (uint32_t)offset;
  pr.m_len = (uint32_t)len;
  pr.n_pad = (uint32_t)db->n_pad;
  pr.k_iters = (uint32_t)(db->code_length / 128);
  pr.mult = mult;
  pr.mask_on = db->remote ? 1u : 0u;
  pr.key_own = db->seed0;
  pr.key_prev = db->seed1;
  pr.nonce = nonce_of(db->code_length == (size_t)kIrisCodeLength ? kDomCodeDot : kDomMaskDot,
                      (uint32_t)db->dm->device);
  pr.batch = db->batch;
  pr.batch_dev = db->batch_from_device ? db->dm->d_batch : nullptr;
  return IRS_OK;
}

// Whether a launch takes less than about 2 ms.
static bool short_launch(irs_sharedb* const* engines, int n, size_t len, size_t n_pad) {
  double macs = 0;
  for (int i = 0; i < n; i++) macs += 3.0 * (double)engines[i]->code_length * (double)n_pad * (double)len;
  return macs < 3e12;
}

// Whether the plain GEMM of a launch runs on SM pairs.  Six engines x 32,768
// entries, one-SM against pair: 128 rows 0.86 / 0.87 ms (over 131,072 entries
// with the threshold between the chunks 3.03 / 2.89), 192 1.32 / 1.01, 256
// 1.37 / 1.18, 384 1.93 / 1.74, 512 2.46 / 2.10, 768 3.58 / 3.03, 960 4.18 /
// 4.25, 1024 4.24 / 3.94; at 65,536 entries the last two are 8.6 / 9.0 and 8.4 /
// 8.0.  So from 128 to 768 rows it is the default; above, where the caller chose
// it or the launch is short enough that the clock has not dropped to the power
// limit (one engine x 32,768 entries, 960 rows 0.94 / 0.89, 1984 rows 1.60 /
// 1.51); and in launches of a few rounds where it fills them as well as smaller
// tiles would (few_rounds_tile), unless the caller chose it for whole 256-row
// tiles.  Those run also where the engine's own tiles are wider (64 entries x 2048
// rows, six engines, 128-row tiles 81 us, 256-row ones 112).
struct PlainGemm {
  bool pair;
  int block_n;
};
static PlainGemm plain_gemm_for(irs_sharedb* const* engines, int n, size_t len, size_t n_pad, bool pair,
                                bool narrow_tile = false) {
  const int bn = gemm_block_n_for((uint32_t)n_pad);
  const bool applies = gemm_pair_applies(true, (uint32_t)n_pad);
  if (applies && pair && !narrow_tile && n_pad > 768 && n_pad % 256 == 0) return {true, bn};
  uint32_t K[kMaxGemmProblems];
  for (int i = 0; i < n; i++) K[i] = (uint32_t)engines[i]->code_length;
  const int few = few_rounds_tile(K, n, (uint32_t)len, (uint32_t)n_pad, engines[0]->dm->n_sms);
  if (few) return {false, std::min(bn, few)};
  return {applies && (pair || n_pad <= 768 || short_launch(engines, n, len, n_pad)), bn};
}

// Whether the engine runs one-SM tiles of a width that the caller gave (one that
// divides the rows) rather than two-SM ones.
static bool own_tiles(const irs_sharedb* e) {
  return e->tile_override && e->n_pad % (size_t)e->tile_override == 0 && !e->pair;
}

static PlainGemm plain_gemm(irs_sharedb* const* engines, int n, size_t len) {
  const irs_sharedb* e = engines[0];
  const PlainGemm own{false, e->block_n};
  if (!len || own_tiles(e)) return own;
  for (int i = 1; i < n; i++)
    if (engines[i]->n_pad != e->n_pad) return own;  // one tile width for the launch
  return plain_gemm_for(engines, n, len, e->n_pad, e->pair, e->tile_override && e->tile_override < 256);
}

// The tile width with which a launch over `len` entries can run as the
// rotation-structured GEMM, or -1: every engine holds sums and form maps, the
// caller left the GEMM open (no tile width asked for) or chose the two-SM one,
// and the quad GEMM is expected to take less.  Whether it does run depends on
// the uploaded rows.
static int quad_width(irs_sharedb* const* engines, int n, size_t offset, size_t len, const PlainGemm& plain,
                      bool captured) {
  uint32_t K[kMaxGemmProblems];
  for (int i = 0; i < n; i++) {
    const irs_sharedb* e = engines[i];
    if (!e->sums || e->n_pad != engines[0]->n_pad || e->forms_pad != e->n_pad) return -1;
    // (sums that a gather left behind are derived on the party's stream: not in a capture)
    if (offset < e->stale_end && (captured || e->dm->capturing || stream_captures(e->dm->streams[e->peer]))) return -1;
    if (own_tiles(e)) return -1;
    K[i] = (uint32_t)e->code_length;
  }
  const irs_sharedb* e = engines[0];
  return quad_width_for(K, n, (uint32_t)len, (uint32_t)e->n_pad, plain.block_n, plain.pair, e->dm->n_sms);
}

static void fill_quad_problem(const irs_sharedb* db, const GemmProblem& g, int width, QuadProblem& pr) {
  pr.tm_a_lo[0] = db->tm_db_lo;
  pr.tm_a_hi[0] = db->tm_db_hi;
  for (int k = 0; k < 2; k++) {
    pr.tm_a_lo[1 + k] = db->tm_sum_lo[k];
    pr.tm_a_hi[1 + k] = db->tm_sum_hi[k];
  }
  pr.tm_b_lo = db->tm_form_lo[width];
  pr.tm_b_hi = db->tm_form_hi[width];
  pr.out = g.out;
  pr.row_valid = db->row_valid;
  pr.m0 = g.m0;
  pr.m_len = g.m_len;
  pr.n_pad = g.n_pad;
  pr.quarter = (uint32_t)(db->code_length / 4);
  pr.mult = g.mult;
  pr.mask_on = g.mask_on;
  pr.key_own = g.key_own;
  pr.key_prev = g.key_prev;
  pr.nonce = g.nonce;
  pr.batch = g.batch;
  pr.batch_dev = g.batch_dev;
}

int irs_sharedb_runs_quads(irs_sharedb* const* engines, int n, size_t rows, size_t len, int pair, int* on) {
  CHECK(engines && on && n > 0 && n <= kMaxGemmProblems, IRS_ERR_INVALID, "1..6 engines per launch");
  *on = 0;
  uint32_t K[kMaxGemmProblems];
  for (int i = 0; i < n; i++) {
    CHECK(engines[i] && engines[i]->dm == engines[0]->dm, IRS_ERR_INVALID, "engine %d missing or on another device", i);
    K[i] = (uint32_t)engines[i]->code_length;
  }
  const size_t n_pad = padded_query_rows(rows, engines[0]->n_cap);
  SumReader lock(sum_holders(engines[0]).mu);
  for (int i = 0; i < n; i++)
    if (!engines[i]->sums || padded_query_rows(rows, engines[i]->n_cap) != n_pad || n_pad > engines[i]->n_cap)
      return IRS_OK;
  if (n_pad < kQuadMinRows || !len) return IRS_OK;
  const PlainGemm g = plain_gemm_for(engines, n, len, n_pad, pair != 0);
  *on = quad_width_for(K, n, (uint32_t)len, (uint32_t)n_pad, g.block_n, g.pair, engines[0]->dm->n_sms) >= 0;
  return IRS_OK;
}

int irs_sharedb_dot_many(irs_sharedb* const* engines, const uint16_t* multipliers, int n, size_t offset, size_t len,
                         void* stream) {
  CHECK(engines && multipliers && n > 0 && n <= kMaxGemmProblems, IRS_ERR_INVALID, "1..6 engines per launch");
  irs_device_manager* dm = engines[0]->dm;
  CU(cudaSetDevice(dm->device));
  GemmParams P;
  memset(&P, 0, sizeof P);
  P.n_prob = n;
  P.err = dm->d_err;
  for (int i = 0; i < n; i++) {
    CHECK(engines[i] && engines[i]->dm == dm, IRS_ERR_INVALID, "engine %d missing or on another device", i);
    CHECK(engines[i]->block_n == engines[0]->block_n, IRS_ERR_INVALID, "engines need the same padded query length");
    CHECK(engines[i]->pair == engines[0]->pair, IRS_ERR_INVALID, "engines need the same GEMM variant (set_pair)");
  }
  // the stall hook is the one-SM kernel's
  const bool stall = len && dm->stall_limit_ns && !dm->capturing;
  const PlainGemm plain = stall ? PlainGemm{false, engines[0]->block_n} : plain_gemm(engines, n, len);
  const Gemm kind = plain.pair                               ? Gemm::kPair
                    : plain.block_n == engines[0]->block_n ? Gemm::kOneSm
                    : plain.block_n == 64                  ? Gemm::k64
                                                           : Gemm::k128;
  for (int i = 0; i < n; i++) {
    int rc = fill_problem(engines[i], multipliers[i], offset, len, kind, P.prob[i]);
    if (rc) return rc;
  }
  cudaStream_t s = party_stream(dm, engines[0]->peer, stream);
  SumReader lock(sum_holders(dm->device).mu);
  const bool captured = stream_captures(s);
  const int width = stall || !len ? -1 : quad_width(engines, n, offset, len, plain, captured);
  bool quads = width >= 0;
  for (int i = 0; i < n && !captured; i++) quads = quads && engines[i]->quad_rows;
  for (int i = 0; i < n && quads; i++)
    if (offset < engines[i]->stale_end) CU(fresh_sums(engines[i]));
  // The engines' inputs may have been written on their own party streams
  // (not while a graph is being captured: then all work is on the capture
  // stream and the uploads happened before the capture began).
  for (int i = 0; i < n; i++)
    if (!dm->capturing && dm->streams[engines[i]->peer] != s) {
      CU(cudaEventRecord(engines[i]->done, dm->streams[engines[i]->peer]));
      CU(cudaStreamWaitEvent(s, engines[i]->done, 0));
    }
  if (len) {
    if (stall) {  // one-shot test hook
      P.test_stall = 1;
      P.wait_timeout_ns = dm->stall_limit_ns;
      dm->stall_limit_ns = 0;
    }
    StageTimer timer(dm, s, "dot");
    if (quads) {
      QuadParams Q;
      memset(&Q, 0, sizeof Q);
      Q.n_prob = n;
      Q.err = dm->d_err;
      Q.tile_n = quad_tile_n((uint32_t)engines[0]->n_pad, width);
      for (int i = 0; i < n; i++) {
        fill_quad_problem(engines[i], P.prob[i], width, Q.prob[i]);
        if (!captured) continue;
        (dm->capturing ? engines[i]->dot_captured : engines[i]->sums_pinned) = true;
        Q.run.word[i] = engines[i]->quad_flag;
        Q.run.n = n;
        Q.run.rows = (uint32_t)engines[i]->n_pad;
      }
      P.skip = Q.run;
      CU(launch_quad_gemm(Q, dm->n_sms, s));
    }
    if (!quads || captured) CU(launch_limb_gemm(P, plain.block_n, plain.pair, dm->n_sms, s));
    for (int i = 0; i < n; i++)
      engines[i]->last_gemm =
          quads ? (captured ? IRS_GEMM_CAPTURED : IRS_GEMM_QUAD) : plain.pair ? IRS_GEMM_PAIR : IRS_GEMM_ONE_SM;
  }
  for (int i = 0; i < n; i++) {
    engines[i]->res_offset = offset;
    engines[i]->res_len = len;
    if (!dm->capturing) CU(cudaEventRecord(engines[i]->done, s));  // a graph launch records graph_done instead
  }
  return IRS_OK;
}

int irs_sharedb_dot(irs_sharedb* db, size_t offset, size_t len, uint16_t multiplier, void* stream) {
  CHECK(db, IRS_ERR_INVALID, "db is NULL");
  irs_sharedb* e[1] = {db};
  uint16_t m[1] = {multiplier};
  return irs_sharedb_dot_many(e, m, 1, offset, len, stream ? stream : db->dm->streams[db->peer]);
}

int irs_sharedb_fetch_results(irs_sharedb* db, uint16_t* host, size_t len) {
  CHECK(db && host, IRS_ERR_INVALID, "bad arguments");
  CHECK(len <= db->res_len, IRS_ERR_STATE, "only %zu results available", db->res_len);
  irs_device_manager* dm = db->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[db->peer];
  std::vector<uint16_t> tmp(len * db->n_pad);
  CU(cudaMemcpyAsync(tmp.data(), db->results, tmp.size() * 2, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  int rc = check_device_error(dm);
  if (rc) return rc;
  for (size_t m = 0; m < len; m++)
    for (size_t q = 0; q < db->query_length; q++)
      host[q * len + m] = q < db->n_pad ? tmp[m * db->n_pad + q] : (uint16_t)0;
  return IRS_OK;
}

int irs_sharedb_result_view(irs_sharedb* db, const uint16_t** dev, size_t* row_stride) {
  CHECK(db && dev && row_stride, IRS_ERR_INVALID, "bad arguments");
  *dev = db->results;
  *row_stride = db->n_pad;
  return IRS_OK;
}

// ---------------------------------------------------------------------------
// Circuits
// ---------------------------------------------------------------------------
int irs_circuits_new(irs_device_manager* dm, const uint32_t seeds[3][2][8], irs_circuits** out) {
  CHECK(dm && seeds && out, IRS_ERR_INVALID, "bad arguments");
  *out = nullptr;
  for (int p = 0; p < 3; p++)
    CHECK(memcmp(seeds[p][1], seeds[(p + 2) % 3][0], 32) == 0, IRS_ERR_INVALID,
          "seed1 of party %d must equal seed0 of party %d", p, (p + 2) % 3);
  auto* c = new (std::nothrow) irs_circuits();
  CHECK(c, IRS_ERR_NOMEM, "host allocation failed");
  c->dm = dm;
  for (int p = 0; p < 3; p++) c->keys[p] = key_of(seeds[p][0]);
  *out = c;
  return IRS_OK;
}

int irs_circuits_destroy(irs_circuits* c) {
  delete c;
  return IRS_OK;
}

int irs_circuits_set_batch(irs_circuits* c, uint64_t batch_id) {
  CHECK(c, IRS_ERR_INVALID, "c is NULL");
  CHECK(batch_id < (1ull << 24), IRS_ERR_INVALID, "batch id must be below 2^24");
  c->batch = batch_id;
  return IRS_OK;
}

static void base_params(irs_circuits* c, ThresholdParams& P) {
  memset(&P, 0, sizeof P);
  for (int p = 0; p < 3; p++) P.key[p] = c->keys[p];
  P.nonce = nonce_of(kDomCircuit, (uint32_t)c->dm->device);
  P.batch = c->batch;
  P.batch_dev = c->batch_from_device ? c->dm->d_batch : nullptr;
}

// Splits [3][n/32] result components into each party's (a, b) u64 words.
__global__ void scatter_views_kernel(const uint32_t* comp, size_t n_words32, uint64_t* a0, uint64_t* a1, uint64_t* a2,
                                     uint64_t* b0, uint64_t* b1, uint64_t* b2, uint64_t* opened) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;  // u64 word
  if (2 * i >= n_words32) return;
  auto w64 = [&](int p) {
    const uint32_t* c = comp + (size_t)p * n_words32;
    return (uint64_t)c[2 * i] | ((uint64_t)c[2 * i + 1] << 32);
  };
  const uint64_t c0 = w64(0), c1 = w64(1), c2 = w64(2);
  if (a0) a0[i] = c0;
  if (a1) a1[i] = c1;
  if (a2) a2[i] = c2;
  if (b0) b0[i] = c2;
  if (b1) b1[i] = c0;
  if (b2) b2[i] = c1;
  if (opened) opened[i] = c0 ^ c1 ^ c2;
}

// Begins a call over flat share vectors on stream s.  Work of party 0's stream
// comes first, whichever stream the caller chose: the shares may be dot results
// that it is still writing.  Such calls take scratch memory and may wait, so
// they are not captured (irs_circuits_compare_threshold_masked_many_noalloc is).
static int begin_flat(irs_device_manager* dm, cudaStream_t s) {
  CU(cudaSetDevice(dm->device));
  CHECK(!dm->capturing && !stream_captures(s), IRS_ERR_CUDA,
        "a call over flat shares cannot be captured; the no-allocation entry point can");
  if (s == dm->streams[0] || stream_captures(dm->streams[0])) return IRS_OK;
  CU(cudaEventRecord(dm->uploads[0], dm->streams[0]));
  CU(cudaStreamWaitEvent(s, dm->uploads[0], 0));
  return IRS_OK;
}

// Whether a result array of a flat call shares memory with an input: the kernel
// then may not write results while other words' shares are still to be read.
static bool results_overlap_shares(const ThresholdParams& P, int stage, uint64_t* const res_a[3],
                                   uint64_t* const res_b[3], const uint64_t* opened) {
  const uintptr_t in = P.n_words * 64, out = P.n_words * 4;
  for (int k = 0; k < 7; k++) {
    const void* r = k == 6 ? opened : k < 3 ? (res_a ? res_a[k] : nullptr) : (res_b ? res_b[k - 3] : nullptr);
    if (!r) continue;
    const uintptr_t a = reinterpret_cast<uintptr_t>(r);
    for (int p = 0; p < 3; p++) {
      const uintptr_t c = reinterpret_cast<uintptr_t>(P.code[p]), m = reinterpret_cast<uintptr_t>(P.mask[p]);
      if ((a < c + in && c < a + out) || (stage == kStageFull && a < m + in && m < a + out)) return true;
    }
  }
  return false;
}

static int run_flat(irs_circuits* c, const uint16_t* const code_a[3], const uint16_t* const mask_a[3], size_t n,
                    uint32_t threshold_a, uint64_t* const res_a[3], uint64_t* const res_b[3], uint64_t* opened,
                    int stage, void* stream) {
  CHECK(c && code_a, IRS_ERR_INVALID, "bad arguments");
  CHECK(n % 64 == 0, IRS_ERR_INVALID, "n = %zu must be a multiple of 64", n);
  for (int p = 0; p < 3; p++) {
    CHECK(code_a[p] && (stage != kStageFull || (mask_a && mask_a[p])), IRS_ERR_INVALID, "share pointer missing");
    CHECK(((uintptr_t)code_a[p] & 15) == 0 && (stage != kStageFull || ((uintptr_t)mask_a[p] & 15) == 0),
          IRS_ERR_INVALID, "share pointers must be 16-byte aligned");
  }
  irs_device_manager* dm = c->dm;
  cudaStream_t s = party_stream(dm, 0, stream);
  int rc = begin_flat(dm, s);
  if (rc) return rc;
  ThresholdParams P;
  base_params(c, P);
  for (int p = 0; p < 3; p++) {
    P.code[p] = code_a[p];
    P.mask[p] = stage == kStageFull ? mask_a[p] : code_a[p];
  }
  P.threshold_a = threshold_a;
  P.n_words = n / 32;
  P.word_base = 0;
  if (threshold_writes_shares(P.n_words) && !results_overlap_shares(P, stage, res_a, res_b, opened)) {
    for (int p = 0; p < 3; p++) {
      P.res_a[p] = res_a ? reinterpret_cast<uint32_t*>(res_a[p]) : nullptr;
      P.res_b[p] = res_b ? reinterpret_cast<uint32_t*>(res_b[p]) : nullptr;
    }
    P.revealed = reinterpret_cast<uint32_t*>(opened);
    CU(launch_threshold_flat(P, stage, s));
    return IRS_OK;
  }
  // (or results over the shares: every share is read before the first is written)
  uint32_t* comp = nullptr;
  void* p;
  rc = scratch_alloc(dm, s, 3 * P.n_words * 4, &p);
  if (rc) return rc;
  comp = (uint32_t*)p;
  P.res_comp = comp;
  cudaError_t e = launch_threshold_flat(P, stage, s);
  if (e == cudaSuccess) {
    const size_t w64 = n / 64;
    scatter_views_kernel<<<(unsigned)((w64 + 255) / 256), 256, 0, s>>>(
        comp, P.n_words, res_a ? res_a[0] : nullptr, res_a ? res_a[1] : nullptr, res_a ? res_a[2] : nullptr,
        res_b ? res_b[0] : nullptr, res_b ? res_b[1] : nullptr, res_b ? res_b[2] : nullptr, opened);
    e = cudaGetLastError();
  }
  cudaFreeAsync(comp, s);
  if (e != cudaSuccess) return fail(IRS_ERR_CUDA, "threshold launch: %s", cudaGetErrorString(e));
  return IRS_OK;
}

int irs_circuits_compare_threshold_masked_many(irs_circuits* c, const uint16_t* const code_a[3],
                                               const uint16_t* const mask_a[3], size_t n, uint32_t threshold_a,
                                               uint64_t* const res_a[3], uint64_t* const res_b[3], uint64_t* opened,
                                               void* stream) {
  return run_flat(c, code_a, mask_a, n, threshold_a, res_a, res_b, opened, kStageFull, stream);
}

// The shared OR of the bit vector whose components are comp[p * n_words + w]
// (party p's a-share), into host out[4]: the three components and the opened
// bit.  Synchronous.
static int run_or_tree(irs_circuits* c, const uint32_t* comp, size_t n_words, uint32_t* out, cudaStream_t s) {
  irs_device_manager* dm = c->dm;
  OrTreeParams P;
  memset(&P, 0, sizeof P);
  for (int p = 0; p < 3; p++) P.key[p] = c->keys[p];
  P.nonce = nonce_of(kDomOrTree, (uint32_t)dm->device);
  P.batch = c->batch;
  P.batch_dev = c->batch_from_device ? dm->d_batch : nullptr;
  P.err = dm->d_err;
  void* p;
  int rc = scratch_alloc(dm, s, (6 * n_words + 5) * 4, &p);
  if (rc) return rc;
  uint32_t* scratch = static_cast<uint32_t*>(p);
  uint32_t* out5 = scratch + 6 * n_words;
  uint32_t got[5] = {};
  cudaError_t e = launch_or_tree(P, comp, n_words, scratch, out5, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(got, out5, sizeof got, cudaMemcpyDeviceToHost, s);
  cudaFreeAsync(scratch, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(IRS_ERR_CUDA, "or tree: %s", cudaGetErrorString(e));
  memcpy(out, got, 16);
  return device_error((int)got[4]);
}

int irs_circuits_or_reduce(irs_circuits* c, const uint64_t* const res_a[3], size_t n, uint32_t out[4], void* stream) {
  CHECK(c && res_a && out, IRS_ERR_INVALID, "bad arguments");
  CHECK(n > 0 && n % 64 == 0, IRS_ERR_INVALID, "n = %zu must be a positive multiple of 64", n);
  for (int p = 0; p < 3; p++) CHECK(res_a[p], IRS_ERR_INVALID, "share pointer missing");
  irs_device_manager* dm = c->dm;
  cudaStream_t s = party_stream(dm, 0, stream);
  int rc = begin_flat(dm, s);
  if (rc) return rc;
  const size_t n_words = n / 32;
  // gather the three a-shares (u64 words = pairs of u32 words) into one [3][n_words] vector
  void* p;
  rc = scratch_alloc(dm, s, 3 * n_words * 4, &p);
  if (rc) return rc;
  uint32_t* comp = static_cast<uint32_t*>(p);
  cudaError_t e = cudaSuccess;
  for (int q = 0; q < 3 && e == cudaSuccess; q++)
    e = cudaMemcpyAsync(comp + q * n_words, res_a[q], n_words * 4, cudaMemcpyDeviceToDevice, s);
  rc = e == cudaSuccess ? run_or_tree(c, comp, n_words, out, s) : fail(IRS_ERR_CUDA, "copy: %s", cudaGetErrorString(e));
  cudaFreeAsync(comp, s);
  return rc;
}

int irs_circuits_compare_threshold_masked_many_with_or_tree(irs_circuits* c, const uint16_t* const code_a[3],
                                                            const uint16_t* const mask_a[3], size_t n,
                                                            uint32_t threshold_a, uint32_t out[4], void* stream) {
  CHECK(c && code_a && mask_a && out, IRS_ERR_INVALID, "bad arguments");
  CHECK(n > 0 && n % 64 == 0, IRS_ERR_INVALID, "n = %zu must be a positive multiple of 64", n);
  for (int p = 0; p < 3; p++) {
    CHECK(code_a[p] && mask_a[p], IRS_ERR_INVALID, "share pointer missing");
    CHECK(((uintptr_t)code_a[p] & 15) == 0 && ((uintptr_t)mask_a[p] & 15) == 0, IRS_ERR_INVALID,
          "share pointers must be 16-byte aligned");
  }
  irs_device_manager* dm = c->dm;
  cudaStream_t s = party_stream(dm, 0, stream);
  int rc = begin_flat(dm, s);
  if (rc) return rc;
  ThresholdParams P;
  base_params(c, P);
  for (int p = 0; p < 3; p++) {
    P.code[p] = code_a[p];
    P.mask[p] = mask_a[p];
  }
  P.threshold_a = threshold_a;
  P.n_words = n / 32;
  void* p;
  rc = scratch_alloc(dm, s, 3 * P.n_words * 4, &p);
  if (rc) return rc;
  P.res_comp = static_cast<uint32_t*>(p);
  cudaError_t e = launch_threshold_flat(P, kStageFull, s);
  rc = e == cudaSuccess ? run_or_tree(c, P.res_comp, P.n_words, out, s)
                        : fail(IRS_ERR_CUDA, "threshold launch: %s", cudaGetErrorString(e));
  cudaFreeAsync(P.res_comp, s);
  return rc;
}

int irs_circuits_extract_msb_of_code(irs_circuits* c, const uint16_t* const code_a[3], size_t n,
                                     uint64_t* const res_a[3], uint64_t* const res_b[3], uint64_t* opened,
                                     void* stream) {
  return run_flat(c, code_a, nullptr, n, 0, res_a, res_b, opened, kStageMsbOnly, stream);
}

int irs_circuits_lift_mpc(irs_circuits* c, const uint16_t* const mask_a[3], size_t n, uint16_t* const corr[3],
                          void* stream) {
  CHECK(c && mask_a && corr, IRS_ERR_INVALID, "bad arguments");
  CHECK(n % 64 == 0, IRS_ERR_INVALID, "n = %zu must be a multiple of 64", n);
  irs_device_manager* dm = c->dm;
  cudaStream_t s = party_stream(dm, 0, stream);
  int rc = begin_flat(dm, s);
  if (rc) return rc;
  ThresholdParams P;
  base_params(c, P);
  for (int p = 0; p < 3; p++) {
    CHECK(mask_a[p] && corr[p] && ((uintptr_t)mask_a[p] & 15) == 0, IRS_ERR_INVALID, "bad share pointer");
    P.mask[p] = mask_a[p];
    P.code[p] = mask_a[p];
  }
  P.n_words = n / 32;
  void* p;
  rc = scratch_alloc(dm, s, 6 * n * 2, &p);
  if (rc) return rc;
  uint16_t* tmp = (uint16_t*)p;
  cudaError_t e = launch_lift_flat(P, tmp, s);
  for (int q = 0; q < 3 && e == cudaSuccess; q++)
    e = cudaMemcpyAsync(corr[q], tmp + (size_t)2 * q * n, 2 * n * 2, cudaMemcpyDeviceToDevice, s);
  cudaFreeAsync(tmp, s);
  if (e != cudaSuccess) return fail(IRS_ERR_CUDA, "lift launch: %s", cudaGetErrorString(e));
  return IRS_OK;
}

// ---------------------------------------------------------------------------
// DistanceComparator
// ---------------------------------------------------------------------------
constexpr uint32_t kMaxForced = 256;

// Buffer layout of the distance capture: [0] count, then entry [cap], row
// [cap], code [3][cap] u16, mask [3][cap] u16.
static void set_distance_capture(irs_distance_comparator* dc, ThresholdParams& P) {
  if (!dc->d_dist) return;
  const size_t cap = dc->dist_cap;
  P.dist_count = dc->d_dist;
  P.dist_entry = dc->d_dist + 1;
  P.dist_row = dc->d_dist + 1 + cap;
  P.dist_code = reinterpret_cast<uint16_t*>(dc->d_dist + 1 + 2 * cap);
  P.dist_mask = P.dist_code + 3 * cap;
  P.dist_cap = (uint32_t)cap;
  if (dc->d_forced && dc->n_forced) {
    P.forced_query = dc->d_forced;
    P.forced_entry = dc->d_forced + kMaxForced;
    P.n_forced = dc->n_forced;
  }
}

int irs_dc_init(irs_device_manager* dm, size_t max_queries, size_t max_db_length, size_t match_list_cap,
                irs_distance_comparator** out) {
  CHECK(dm && out && max_queries > 0 && max_db_length > 0, IRS_ERR_INVALID, "bad arguments");
  *out = nullptr;
  CU(cudaSetDevice(dm->device));
  auto* dc = new (std::nothrow) irs_distance_comparator();
  CHECK(dc, IRS_ERR_NOMEM, "host allocation failed");
  dc->dm = dm;
  dc->max_queries = max_queries;
  dc->max_db = max_db_length;
  dc->stride_bits = round_up(max_db_length, 64);
  dc->self_stride_bits = round_up(max_queries, 64);
  dc->match_cap = match_list_cap ? match_list_cap : 1;
  dc->slot_cap = 65536 / kSlotRows;
  dc->seg_cap = dc->slot_cap * 32;
  struct { void** p; size_t bytes; } allocs[] = {
      {(void**)&dc->bitmap, max_queries * dc->stride_bits / 8},
      {(void**)&dc->self_bitmap, max_queries * dc->self_stride_bits / 8},
      {(void**)&dc->match_list, dc->match_cap * 8},
      {(void**)&dc->counters, 16},
      {(void**)&dc->partial, max_db_length * 4},
      {(void**)&dc->results_err, (4 + max_queries * (2 + kMaxMatchesLen)) * 4},
      {(void**)&dc->d_slot_valid, dc->slot_cap * 4},
      {(void**)&dc->d_slot_query, dc->slot_cap * 4},
      {(void**)&dc->d_seg_start, (dc->slot_cap + 1) * 4},
      {(void**)&dc->d_seg_query, dc->slot_cap * 32 * 4},
      {(void**)&dc->d_seg_mask, dc->slot_cap * 32 * 4},
      {(void**)&dc->d_take, (4 + max_queries * (2 + kMaxMatchesLen)) * 4},
  };
  for (auto& a : allocs) {
    cudaError_t e = device_malloc(dm, a.p, a.bytes);
    if (e != cudaSuccess) {
      cudaGetLastError();
      irs_dc_destroy(dc);
      return fail(IRS_ERR_NOMEM, "distance comparator allocation of %zu bytes failed", a.bytes);
    }
  }
  dc->final_results = dc->results_err + 4;
  dc->match_counters = dc->final_results + max_queries;
  dc->all_matches = dc->match_counters + max_queries;
  CU(cudaMemsetAsync(dc->all_matches, 0, max_queries * kMaxMatchesLen * 4, dm->streams[0]));
  int rc = irs_dc_reset(dc, nullptr);
  if (rc) { irs_dc_destroy(dc); return rc; }
  CU(cudaStreamSynchronize(dm->streams[0]));
  *out = dc;
  return IRS_OK;
}

int irs_dc_destroy(irs_distance_comparator* dc) {
  if (!dc) return IRS_OK;
  cudaSetDevice(dc->dm->device);
  void* ps[] = {dc->bitmap, dc->self_bitmap, dc->match_list, dc->counters, dc->partial, dc->results_err,
                dc->d_slot_valid, dc->d_slot_query,
                dc->d_seg_start, dc->d_seg_query, dc->d_seg_mask, dc->d_take, dc->d_dist, dc->d_forced,
                dc->ring};
  for (void* p : ps) if (p) cudaFree(p);
  delete dc;
  return IRS_OK;
}

int irs_dc_reset(irs_distance_comparator* dc, void* stream) {
  CHECK(dc, IRS_ERR_INVALID, "dc is NULL");
  cudaStream_t s = party_stream(dc->dm, 0, stream);
  CU(launch_reset(dc->bitmap, dc->max_queries * dc->stride_bits / 32, dc->self_bitmap,
                  dc->max_queries * dc->self_stride_bits / 32, dc->counters, dc->final_results, dc->match_counters,
                  (uint32_t)dc->max_queries, s));
  return IRS_OK;
}

// Fetches a block of `words` result words behind its four error words in one
// copy: the device error word joins it on the device.  out[0..words) follows the
// four; returns the error word's status.
static int fetch_block(irs_distance_comparator* dc, uint32_t* block, size_t words, std::vector<uint32_t>& out,
                       cudaStream_t s) {
  try {
    out.resize(4 + words);
  } catch (const std::bad_alloc&) {
    out.clear();
    return fail(IRS_ERR_NOMEM, "host buffer of %zu result words failed", words);
  }
  CU(cudaMemcpyAsync(block, dc->dm->d_err, 4, cudaMemcpyDeviceToDevice, s));
  CU(cudaMemcpyAsync(out.data(), block, out.size() * 4, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  return device_error((int)out[0]);
}

int irs_dc_compare_threshold_open(irs_distance_comparator* dc, irs_circuits* c, irs_sharedb* const code_engines[3],
                                  irs_sharedb* const mask_engines[3], size_t offset, size_t len, size_t n_slots,
                                  const uint32_t* slot_valid, const uint32_t* slot_query, uint32_t threshold_a,
                                  int self_check, void* stream) {
  CHECK(dc && c && code_engines && mask_engines, IRS_ERR_INVALID, "bad arguments");
  CHECK(offset % 32 == 0, IRS_ERR_INVALID, "offset must be a multiple of 32");
  CHECK(n_slots <= dc->slot_cap, IRS_ERR_INVALID, "too many slots");
  const size_t n_pad = code_engines[0]->n_pad;
  CHECK(n_slots * kSlotRows <= n_pad, IRS_ERR_INVALID, "slots exceed the padded query rows");
  for (int p = 0; p < 3; p++) {
    CHECK(code_engines[p] && mask_engines[p], IRS_ERR_INVALID, "engine missing");
    CHECK(code_engines[p]->n_pad == n_pad && mask_engines[p]->n_pad == n_pad, IRS_ERR_INVALID,
          "engines need the same query padding");
    CHECK(code_engines[p]->res_offset == offset && mask_engines[p]->res_offset == offset &&
              code_engines[p]->res_len >= len && mask_engines[p]->res_len >= len,
          IRS_ERR_STATE, "engine results do not cover entries %zu..%zu", offset, offset + len);
  }
  const size_t stride_bits = self_check ? dc->self_stride_bits : dc->stride_bits;
  CHECK(offset + len <= stride_bits, IRS_ERR_INVALID, "entries exceed the bitmap width");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = party_stream(dm, 0, stream);
  // Receive: wait until every party's shares have been produced.
  // The GEMMs ran on another stream: wait for them (inside a graph capture
  // they are earlier nodes of the same capture stream).
  for (int p = 0; !dm->capturing && p < 3; p++) {
    CU(cudaStreamWaitEvent(s, code_engines[p]->done, 0));
    CU(cudaStreamWaitEvent(s, mask_engines[p]->done, 0));
  }
  ThresholdParams P;
  base_params(c, P);
  for (int p = 0; p < 3; p++) {
    P.code[p] = code_engines[p]->results;
    P.mask[p] = mask_engines[p]->results;
  }
  P.threshold_a = threshold_a;
  P.n_entries = (uint32_t)len;
  P.m0 = (uint32_t)offset;
  P.n_pad = (uint32_t)n_pad;
  P.n_slots = (uint32_t)n_slots;
  if (slot_valid) {
    CU(cudaMemcpyAsync(dc->d_slot_valid, slot_valid, n_slots * 4, cudaMemcpyHostToDevice, s));
    P.slot_valid = dc->d_slot_valid;
  }
  if (slot_query) {
    for (size_t i = 0; i < n_slots; i++)
      CHECK(slot_query[i] < dc->max_queries, IRS_ERR_INVALID, "slot %zu reports to query %u >= max", i, slot_query[i]);
    CU(cudaMemcpyAsync(dc->d_slot_query, slot_query, n_slots * 4, cudaMemcpyHostToDevice, s));
    P.slot_query = dc->d_slot_query;
  } else {
    CHECK(n_slots <= dc->max_queries, IRS_ERR_INVALID, "more slots than queries");
  }
  P.bitmap = self_check ? dc->self_bitmap : dc->bitmap;
  P.bitmap_stride = (uint32_t)stride_bits;
  P.match_count = dc->counters;
  P.match_list = self_check ? nullptr : dc->match_list;
  P.match_cap = (uint32_t)dc->match_cap;
  if (!self_check) set_distance_capture(dc, P);
  {
    StageTimer timer(dm, s, "threshold_open");
    CU(launch_threshold_bitmap(P, s));
  }
  if (slot_valid || slot_query) CU(cudaStreamSynchronize(s));  // host arrays are caller-owned
  return IRS_OK;
}

int irs_dc_set_segments(irs_distance_comparator* dc, size_t n_slots, const uint32_t* seg_start,
                        const uint32_t* seg_query, const uint32_t* seg_mask) {
  CHECK(dc && seg_start && n_slots > 0 && n_slots <= dc->slot_cap, IRS_ERR_INVALID, "bad arguments");
  CHECK(seg_start[0] == 0, IRS_ERR_INVALID, "seg_start[0] must be 0");
  for (size_t i = 0; i < n_slots; i++)
    CHECK(seg_start[i + 1] >= seg_start[i], IRS_ERR_INVALID, "seg_start must be non-decreasing");
  const size_t n_seg = seg_start[n_slots];
  CHECK(n_seg <= dc->seg_cap && (n_seg == 0 || (seg_query && seg_mask)), IRS_ERR_INVALID, "too many segments");
  for (size_t k = 0; k < n_seg; k++)
    CHECK(seg_query[k] < dc->max_queries, IRS_ERR_INVALID, "segment %zu reports to query %u >= max", k, seg_query[k]);
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  CU(cudaMemcpyAsync(dc->d_seg_start, seg_start, (n_slots + 1) * 4, cudaMemcpyHostToDevice, s));
  if (n_seg) {
    CU(cudaMemcpyAsync(dc->d_seg_query, seg_query, n_seg * 4, cudaMemcpyHostToDevice, s));
    CU(cudaMemcpyAsync(dc->d_seg_mask, seg_mask, n_seg * 4, cudaMemcpyHostToDevice, s));
  }
  if (dm->host_sync) CU(cudaStreamSynchronize(s));  // the tables are caller-owned host memory
  dc->n_seg_slots = n_slots;
  dc->have_segments = true;
  return IRS_OK;
}

int irs_dc_compare_threshold_open_prepared(irs_distance_comparator* dc, irs_circuits* c,
                                           irs_sharedb* const code_engines[3], irs_sharedb* const mask_engines[3],
                                           size_t offset, size_t len, uint32_t threshold_a, int self_check,
                                           void* stream) {
  CHECK(dc && c && code_engines && mask_engines, IRS_ERR_INVALID, "bad arguments");
  CHECK(dc->have_segments, IRS_ERR_STATE, "irs_dc_set_segments not called");
  CHECK(offset % 32 == 0, IRS_ERR_INVALID, "offset must be a multiple of 32");
  const size_t n_pad = code_engines[0]->n_pad;
  CHECK(dc->n_seg_slots * kSlotRows <= n_pad, IRS_ERR_INVALID, "segment slots exceed the padded query rows");
  for (int p = 0; p < 3; p++) {
    CHECK(code_engines[p] && mask_engines[p], IRS_ERR_INVALID, "engine missing");
    CHECK(code_engines[p]->n_pad == n_pad && mask_engines[p]->n_pad == n_pad, IRS_ERR_INVALID,
          "engines need the same query padding");
    CHECK(code_engines[p]->res_offset == offset && mask_engines[p]->res_offset == offset &&
              code_engines[p]->res_len >= len && mask_engines[p]->res_len >= len,
          IRS_ERR_STATE, "engine results do not cover entries %zu..%zu", offset, offset + len);
  }
  const size_t stride_bits = self_check ? dc->self_stride_bits : dc->stride_bits;
  CHECK(offset + len <= stride_bits, IRS_ERR_INVALID, "entries exceed the bitmap width");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = party_stream(dm, 0, stream);
  // The GEMMs ran on another stream: wait for them (inside a graph capture
  // they are earlier nodes of the same capture stream).
  for (int p = 0; !dm->capturing && p < 3; p++) {
    CU(cudaStreamWaitEvent(s, code_engines[p]->done, 0));
    CU(cudaStreamWaitEvent(s, mask_engines[p]->done, 0));
  }
  ThresholdParams P;
  base_params(c, P);
  for (int p = 0; p < 3; p++) {
    P.code[p] = code_engines[p]->results;
    P.mask[p] = mask_engines[p]->results;
  }
  P.threshold_a = threshold_a;
  P.n_entries = (uint32_t)len;
  P.m0 = (uint32_t)offset;
  P.n_pad = (uint32_t)n_pad;
  P.n_slots = (uint32_t)dc->n_seg_slots;
  P.seg_start = dc->d_seg_start;
  P.seg_query = dc->d_seg_query;
  P.seg_mask = dc->d_seg_mask;
  P.bitmap = self_check ? dc->self_bitmap : dc->bitmap;
  P.bitmap_stride = (uint32_t)stride_bits;
  P.match_count = dc->counters;
  P.match_list = self_check ? nullptr : dc->match_list;
  P.match_cap = (uint32_t)dc->match_cap;
  if (!self_check) set_distance_capture(dc, P);
  {
    StageTimer timer(dm, s, "threshold_open");
    CU(launch_threshold_bitmap(P, s));
  }
  return IRS_OK;
}

int irs_dc_scan_fused(irs_distance_comparator* dc, irs_circuits* c, irs_sharedb* const code_engines[3],
                      irs_sharedb* const mask_engines[3], size_t offset, size_t len, size_t n_slots,
                      uint32_t threshold_a, int use_segments, void* stream) {
  CHECK(dc && c && code_engines && mask_engines, IRS_ERR_INVALID, "bad arguments");
  CHECK(offset % 32 == 0, IRS_ERR_INVALID, "offset must be a multiple of 32");
  irs_sharedb* eng[kFusedEngines] = {code_engines[0], code_engines[1], code_engines[2],
                                      mask_engines[0], mask_engines[1], mask_engines[2]};
  for (int e = 0; e < kFusedEngines; e++) {
    CHECK(eng[e] && eng[e]->dm == dc->dm, IRS_ERR_INVALID, "engine %d missing or on another device", e);
    CHECK(eng[e]->peer == e % 3, IRS_ERR_INVALID, "engine %d must belong to party %d", e, e % 3);
    CHECK(eng[e]->code_length == (size_t)(e < 3 ? kIrisCodeLength : kMaskCodeLength), IRS_ERR_INVALID,
          "engine %d has code length %zu", e, eng[e]->code_length);
  }
  const size_t n_pad = eng[0]->n_pad;
  for (int e = 1; e < kFusedEngines; e++)
    CHECK(eng[e]->n_pad == n_pad, IRS_ERR_INVALID, "engines need the same query padding");
  CHECK(n_pad % kFusedBlockN == 0, IRS_ERR_INVALID,
        "the fused scan needs padded query rows in multiples of %d (got %zu)", kFusedBlockN, n_pad);
  if (use_segments) {
    CHECK(dc->have_segments, IRS_ERR_STATE, "irs_dc_set_segments not called");
    n_slots = dc->n_seg_slots;
  } else {
    CHECK(n_slots <= dc->max_queries && n_slots <= dc->slot_cap, IRS_ERR_INVALID, "too many slots");
  }
  CHECK(n_slots * kSlotRows <= n_pad, IRS_ERR_INVALID, "slots exceed the padded query rows");
  CHECK(offset + len <= dc->stride_bits, IRS_ERR_INVALID, "entries exceed the bitmap width");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = party_stream(dm, 0, stream);
  FusedParams F;
  memset(&F, 0, sizeof F);
  const uint16_t mults[kFusedEngines] = {1, 1, 1, 2, 2, 2};
  for (int e = 0; e < kFusedEngines; e++) {
    int rc = fill_problem(eng[e], mults[e], offset, len, Gemm::kOneSm, F.prob[e]);
    if (rc) return rc;
    // the fused kernel's query tile is 128 rows whatever the engine's own tile width
    if (make_tmap_u8(&F.prob[e].tm_b_lo, eng[e]->q_lo, eng[e]->n_cap, eng[e]->code_length, kFusedBlockN) ||
        make_tmap_u8(&F.prob[e].tm_b_hi, eng[e]->q_hi, eng[e]->n_cap, eng[e]->code_length, kFusedBlockN))
      return fail(IRS_ERR_CUDA, "tensor map for the query planes failed");
  }
  F.tiles_m = (int)((len + 127) / 128);
  F.tiles_n = (int)(n_pad / kFusedBlockN);
  F.total_work = F.tiles_m * F.tiles_n;
  F.err = dm->d_err;
  const size_t need = (size_t)dm->n_sms * kFusedRingBytesPerCta;  // the grid never exceeds one CTA per SM
  if (need > dc->ring_bytes) {
    // scratch for the dot shares of the CTAs' current tiles; allocated outside any capture
    CHECK(!dm->capturing, IRS_ERR_STATE,
          "the first fused scan of a comparator (which allocates its %zu-byte ring) must come before a graph capture",
          need);
    if (dc->ring) CU(cudaFree(dc->ring));
    dc->ring = nullptr;
    dc->ring_bytes = 0;
    void* p = nullptr;
    cudaError_t e = device_malloc(dm, &p, need);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(IRS_ERR_NOMEM, "fused scan ring of %zu bytes: %s", need, cudaGetErrorString(e));
    }
    dc->ring = static_cast<uint16_t*>(p);
    dc->ring_bytes = need;
  }
  F.ring = dc->ring;
  ThresholdParams& T = F.T;
  base_params(c, T);
  T.threshold_a = threshold_a;
  T.n_entries = (uint32_t)len;
  T.m0 = (uint32_t)offset;
  T.n_pad = (uint32_t)n_pad;
  T.n_slots = (uint32_t)n_slots;
  if (use_segments) {
    T.seg_start = dc->d_seg_start;
    T.seg_query = dc->d_seg_query;
    T.seg_mask = dc->d_seg_mask;
  } else {
    CHECK(n_slots <= dc->max_queries, IRS_ERR_INVALID, "more slots than queries");
  }
  T.bitmap = dc->bitmap;
  T.bitmap_stride = (uint32_t)dc->stride_bits;
  T.match_count = dc->counters;
  T.match_list = dc->match_list;
  T.match_cap = (uint32_t)dc->match_cap;
  set_distance_capture(dc, T);
  // The engines' inputs may have been written on their own party streams.
  for (int e = 0; e < kFusedEngines; e++)
    if (!dm->capturing && dm->streams[eng[e]->peer] != s) {
      CU(cudaEventRecord(eng[e]->done, dm->streams[eng[e]->peer]));
      CU(cudaStreamWaitEvent(s, eng[e]->done, 0));
    }
  if (len && n_slots) {
    StageTimer timer(dm, s, "scan_fused");
    CU(launch_fused_scan(F, dm->n_sms, s));
  }
  for (int e = 0; e < kFusedEngines; e++) {
    eng[e]->res_offset = offset;
    eng[e]->res_len = 0;  // the dot shares stayed in the ring: no buffered results
    if (!dm->capturing) CU(cudaEventRecord(eng[e]->done, s));
  }
  return IRS_OK;
}

// ---------------------------------------------------------------------------
// CUDA graphs
// ---------------------------------------------------------------------------
int irs_graph_begin_capture(irs_device_manager* dm) {
  CHECK(dm, IRS_ERR_INVALID, "dm is NULL");
  CHECK(!dm->capturing, IRS_ERR_STATE, "a capture is already open");
  CU(cudaSetDevice(dm->device));
  CU(cudaEventRecord(dm->uploads[0], dm->streams[0]));  // for graph launches beside the capture
  CU(cudaStreamBeginCapture(dm->streams[0], cudaStreamCaptureModeThreadLocal));
  dm->capturing = true;
  return IRS_OK;
}

int irs_graph_end_capture(irs_device_manager* dm, irs_graph** out) {
  CHECK(dm && out, IRS_ERR_INVALID, "bad arguments");
  CHECK(dm->capturing, IRS_ERR_STATE, "no capture is open");
  *out = nullptr;
  dm->capturing = false;
  cudaGraph_t g = nullptr;
  CU(cudaStreamEndCapture(dm->streams[0], &g));
  cudaError_t made = cudaSuccess;  // with the first graph: most managers have none
  if (!dm->graph_ran) made = cudaEventCreateWithFlags(&dm->graph_ran, cudaEventDisableTiming);
  if (made == cudaSuccess && !dm->graph_join) made = cudaStreamCreateWithFlags(&dm->graph_join, cudaStreamNonBlocking);
  if (made != cudaSuccess) {
    cudaGraphDestroy(g);
    return fail(IRS_ERR_CUDA, "stream or event of the graphs: %s", cudaGetErrorString(made));
  }
  auto* gr = new (std::nothrow) irs_graph();
  if (!gr) {
    cudaGraphDestroy(g);
    return fail(IRS_ERR_NOMEM, "host allocation failed");
  }
  gr->graph = g;
  gr->dm = dm;
  cudaError_t e = cudaGraphInstantiate(&gr->exec, g, 0);
  if (e != cudaSuccess) {
    cudaGraphDestroy(g);
    delete gr;
    return fail(IRS_ERR_CUDA, "cudaGraphInstantiate: %s", cudaGetErrorString(e));
  }
  *out = gr;
  return IRS_OK;
}

int irs_graph_launch(irs_graph* g, void* stream) {
  CHECK(g && g->exec, IRS_ERR_INVALID, "graph is NULL");
  // the graph's GEMMs read what the parties' streams have uploaded (a launch
  // that is captured itself cannot wait for work outside its capture)
  const bool captured = stream_captures(static_cast<cudaStream_t>(stream));
  for (int p = 0; p < 3 && !captured; p++)
    if (g->dm->streams[p] != static_cast<cudaStream_t>(stream)) {
      // (a party's stream that is being captured: its uploads ended with the
      // event that irs_graph_begin_capture recorded)
      if (!stream_captures(g->dm->streams[p])) CU(cudaEventRecord(g->dm->uploads[p], g->dm->streams[p]));
      CU(cudaStreamWaitEvent(static_cast<cudaStream_t>(stream), g->dm->uploads[p], 0));
    }
  if (captured) {  // replays start outside the lock
    SumWriter lock(sum_holders(g->dm->device).mu);
    for (irs_sharedb* db : sum_holders(g->dm->device).engines)
      if (db->dm == g->dm && db->dot_captured) db->sums_pinned = true;
  }
  {
    SumReader lock(sum_holders(g->dm->device).mu);
    CU(cudaGraphLaunch(g->exec, static_cast<cudaStream_t>(stream)));
  }
  // Later query uploads on other party streams wait for the graph's GEMMs, and
  // for those of every graph before it: graphs over different engines may run
  // on different streams, and an upload knows only the engine it writes.
  if (captured) {  // part of another capture: the event belongs to it
    CU(cudaEventRecord(g->dm->graph_done, static_cast<cudaStream_t>(stream)));
    return IRS_OK;
  }
  CU(cudaEventRecord(g->dm->graph_ran, static_cast<cudaStream_t>(stream)));
  CU(cudaStreamWaitEvent(g->dm->graph_join, g->dm->graph_ran, 0));
  CU(cudaEventRecord(g->dm->graph_done, g->dm->graph_join));
  return IRS_OK;
}

int irs_graph_destroy(irs_graph* g) {
  if (!g) return IRS_OK;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  delete g;
  return IRS_OK;
}

int irs_dc_take_rows(irs_distance_comparator* dc, const uint32_t* rows, size_t n, size_t db_len, int clear,
                     uint32_t* counts, uint32_t* ids) {
  CHECK(dc && (n == 0 || (rows && counts && ids)), IRS_ERR_INVALID, "bad arguments");
  CHECK(n <= dc->max_queries, IRS_ERR_INVALID, "%zu rows exceed the comparator's %zu", n, dc->max_queries);
  CHECK(db_len <= dc->stride_bits, IRS_ERR_INVALID, "db_len %zu exceeds the bitmap width", db_len);
  for (size_t i = 0; i < n; i++)
    CHECK(rows[i] < dc->max_queries, IRS_ERR_INVALID, "row %u out of range", rows[i]);
  if (!n) return IRS_OK;
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  uint32_t* d_rows = dc->d_take;
  uint32_t* d_counts = d_rows + dc->max_queries + 4;
  uint32_t* d_ids = d_counts + dc->max_queries;
  CU(cudaMemcpyAsync(d_rows, rows, n * 4, cudaMemcpyHostToDevice, s));
  CU(launch_take_rows(dc->bitmap, (uint32_t)(dc->stride_bits / 32), d_rows, (uint32_t)n, (uint32_t)db_len, clear,
                      d_counts, d_ids, kMaxMatchesLen, s));
  if (!dm->host_sync) {  // outputs valid once the stream passes the copies
    CU(cudaMemcpyAsync(counts, d_counts, n * 4, cudaMemcpyDeviceToHost, s));
    CU(cudaMemcpyAsync(ids, d_ids, n * kMaxMatchesLen * 4, cudaMemcpyDeviceToHost, s));
    return IRS_OK;
  }
  std::vector<uint32_t> got;
  const int rc = fetch_block(dc, d_counts - 4, dc->max_queries + n * kMaxMatchesLen, got, s);
  if (got.empty()) return rc;
  memcpy(counts, got.data() + 4, n * 4);
  memcpy(ids, got.data() + 4 + dc->max_queries, n * kMaxMatchesLen * 4);
  return rc;
}

static size_t dist_bytes(size_t cap) { return (1 + 2 * cap) * 4 + 6 * cap * 2 + 16; }

int irs_dc_enable_distance_capture(irs_distance_comparator* dc, size_t cap) {
  CHECK(dc && cap > 0 && cap < (1u << 30), IRS_ERR_INVALID, "bad arguments");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  CU(cudaStreamSynchronize(dm->streams[0]));
  if (dc->d_dist) {
    cudaFree(dc->d_dist);
    dc->d_dist = nullptr;
  }
  void* p = nullptr;
  if (device_malloc(dm, &p, dist_bytes(cap)) != cudaSuccess) {
    cudaGetLastError();
    return fail(IRS_ERR_NOMEM, "distance capture allocation of %zu bytes failed", dist_bytes(cap));
  }
  dc->d_dist = static_cast<uint32_t*>(p);
  dc->dist_cap = cap;
  CU(cudaMemset(dc->d_dist, 0, 4));
  return IRS_OK;
}

int irs_dc_set_forced_distances(irs_distance_comparator* dc, const uint32_t* query, const uint32_t* entry, size_t n) {
  CHECK(dc && (n == 0 || (query && entry)), IRS_ERR_INVALID, "bad arguments");
  CHECK(dc->d_dist, IRS_ERR_STATE, "distance capture not enabled");
  CHECK(n <= kMaxForced, IRS_ERR_INVALID, "%zu forced pairs exceed %u", n, kMaxForced);
  for (size_t i = 0; i < n; i++)
    CHECK(query[i] < dc->max_queries && entry[i] < dc->max_db, IRS_ERR_INVALID, "forced pair %zu out of range", i);
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  if (!dc->d_forced) {
    void* p = nullptr;
    if (device_malloc(dm, &p, 2 * kMaxForced * 4) != cudaSuccess) {
      cudaGetLastError();
      return fail(IRS_ERR_NOMEM, "forced-pair table allocation failed");
    }
    dc->d_forced = static_cast<uint32_t*>(p);
  }
  if (n) {
    CU(cudaMemcpyAsync(dc->d_forced, query, n * 4, cudaMemcpyHostToDevice, s));
    CU(cudaMemcpyAsync(dc->d_forced + kMaxForced, entry, n * 4, cudaMemcpyHostToDevice, s));
    CU(cudaStreamSynchronize(s));  // caller-owned host memory
  }
  dc->n_forced = (uint32_t)n;
  return IRS_OK;
}

int irs_dc_fetch_distances(irs_distance_comparator* dc, size_t cap, uint32_t* entry, uint32_t* row, uint16_t* code,
                           uint16_t* mask, size_t* n, int reset) {
  CHECK(dc && n, IRS_ERR_INVALID, "bad arguments");
  CHECK(dc->d_dist, IRS_ERR_STATE, "distance capture not enabled");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  uint32_t count = 0;
  CU(cudaMemcpyAsync(&count, dc->d_dist, 4, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  *n = count;  // may exceed the capture capacity: records beyond it were dropped
  const size_t k = std::min<size_t>(std::min<size_t>(count, dc->dist_cap), cap);
  const size_t dcap = dc->dist_cap;
  if (k) {
    CHECK(entry && row && code && mask, IRS_ERR_INVALID, "output arrays missing");
    CU(cudaMemcpyAsync(entry, dc->d_dist + 1, k * 4, cudaMemcpyDeviceToHost, s));
    CU(cudaMemcpyAsync(row, dc->d_dist + 1 + dcap, k * 4, cudaMemcpyDeviceToHost, s));
    const uint16_t* dcode = reinterpret_cast<const uint16_t*>(dc->d_dist + 1 + 2 * dcap);
    for (int p = 0; p < 3; p++) {
      CU(cudaMemcpyAsync(code + p * cap, dcode + p * dcap, k * 2, cudaMemcpyDeviceToHost, s));
      CU(cudaMemcpyAsync(mask + p * cap, dcode + (3 + p) * dcap, k * 2, cudaMemcpyDeviceToHost, s));
    }
  }
  if (reset) CU(cudaMemsetAsync(dc->d_dist, 0, 4, s));
  CU(cudaStreamSynchronize(s));
  return check_device_error(dm);
}

int irs_dc_clear_rows(irs_distance_comparator* dc, size_t first, size_t n, void* stream) {
  CHECK(dc && first + n <= dc->max_queries, IRS_ERR_INVALID, "rows out of range");
  cudaStream_t s = party_stream(dc->dm, 0, stream);
  const size_t words = dc->stride_bits / 32;
  CU(cudaMemsetAsync(dc->bitmap + first * words, 0, n * words * 4, s));
  return IRS_OK;
}

int irs_dc_fetch_rows(irs_distance_comparator* dc, size_t first, size_t n, uint32_t* host, size_t cap_words,
                      size_t* row_words) {
  CHECK(dc && host && row_words && first + n <= dc->max_queries, IRS_ERR_INVALID, "bad arguments");
  const size_t words = dc->stride_bits / 32;
  *row_words = words;
  CHECK(n * words <= cap_words, IRS_ERR_INVALID, "host buffer holds %zu words, %zu needed", cap_words, n * words);
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  if (n) {
    CU(cudaMemcpyAsync(host, dc->bitmap + first * words, n * words * 4, cudaMemcpyDeviceToHost, s));
    if (!dm->host_sync) return IRS_OK;  // rows valid once the stream passes the copy
    uint32_t err = 0;
    CU(cudaMemcpyAsync(&err, dm->d_err, 4, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    return device_error((int)err);
  }
  return check_device_error(dm);
}

int irs_dc_fetch_bitmap(irs_distance_comparator* dc, size_t n_queries, size_t db_len, uint64_t* host) {
  CHECK(dc && host && n_queries <= dc->max_queries && db_len <= dc->stride_bits, IRS_ERR_INVALID, "bad arguments");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  std::vector<uint32_t> tmp(n_queries * dc->stride_bits / 32);
  CU(cudaMemcpyAsync(tmp.data(), dc->bitmap, tmp.size() * 4, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  int rc = check_device_error(dm);
  if (rc) return rc;
  const size_t words = (n_queries * db_len + 63) / 64;
  memset(host, 0, words * 8);
  for (size_t q = 0; q < n_queries; q++)
    for (size_t e = 0; e < db_len; e++) {
      const uint32_t bit = (tmp[q * (dc->stride_bits / 32) + e / 32] >> (e % 32)) & 1u;
      if (bit) {
        const size_t o = q * db_len + e;
        host[o / 64] |= 1ull << (o % 64);
      }
    }
  return IRS_OK;
}

int irs_dc_fetch_matches(irs_distance_comparator* dc, uint32_t* pairs, size_t cap, size_t* n) {
  CHECK(dc && n && (pairs || !cap), IRS_ERR_INVALID, "bad arguments");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  uint32_t count = 0;
  CU(cudaMemcpyAsync(&count, dc->counters, 4, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  *n = count;
  const size_t avail = std::min<size_t>(std::min<size_t>(count, dc->match_cap), cap);
  if (avail) {
    CU(cudaMemcpyAsync(pairs, dc->match_list, avail * 8, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
  }
  int rc = check_device_error(dm);
  if (rc) return rc;
  if (count > dc->match_cap) return fail(IRS_ERR_OVERFLOW, "%u matches exceed the list capacity %zu", count, dc->match_cap);
  return IRS_OK;
}

int irs_dc_get_partial_results(irs_distance_comparator* dc, size_t n_queries, size_t db_len, uint32_t* ids, size_t cap,
                               size_t* n) {
  CHECK(dc && n && (ids || !cap) && n_queries <= dc->max_queries && db_len <= dc->max_db, IRS_ERR_INVALID,
        "bad arguments");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  CU(cudaMemsetAsync(dc->counters + 1, 0, 4, s));
  CU(launch_compact(dc->bitmap, (uint32_t)n_queries, (uint32_t)db_len, (uint32_t)(dc->stride_bits / 32), dc->partial,
                    dc->counters + 1, (uint32_t)dc->max_db, s));
  uint32_t count = 0;
  CU(cudaMemcpyAsync(&count, dc->counters + 1, 4, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  std::vector<uint32_t> tmp(std::min<size_t>(count, dc->max_db));
  if (!tmp.empty()) {
    CU(cudaMemcpyAsync(tmp.data(), dc->partial, tmp.size() * 4, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
  }
  std::sort(tmp.begin(), tmp.end());
  tmp.erase(std::unique(tmp.begin(), tmp.end()), tmp.end());
  *n = tmp.size();
  const size_t k = std::min(cap, tmp.size());
  if (k) memcpy(ids, tmp.data(), k * 4);
  if (tmp.size() > cap) return fail(IRS_ERR_OVERFLOW, "%zu ids exceed cap %zu", tmp.size(), cap);
  return IRS_OK;
}

int irs_dc_join_db_matches(irs_distance_comparator* dc, irs_distance_comparator* right, const uint32_t* or_policy,
                           size_t n_queries, size_t db_len, void* stream) {
  CHECK(dc && n_queries <= dc->max_queries && db_len <= dc->max_db, IRS_ERR_INVALID, "bad arguments");
  CHECK(!right || right->stride_bits == dc->stride_bits, IRS_ERR_INVALID, "comparators differ in bitmap width");
  cudaStream_t s = party_stream(dc->dm, 0, stream);
  CU(launch_merge_db(dc->bitmap, right ? right->bitmap : nullptr, or_policy, (uint32_t)n_queries, (uint32_t)db_len,
                     (uint32_t)(dc->stride_bits / 32), dc->final_results, dc->match_counters, dc->all_matches, s));
  return IRS_OK;
}

int irs_dc_join_batch_matches(irs_distance_comparator* dc, irs_distance_comparator* right, size_t n_queries,
                              void* stream) {
  CHECK(dc && n_queries <= dc->max_queries, IRS_ERR_INVALID, "bad arguments");
  CHECK(!right || right->self_stride_bits == dc->self_stride_bits, IRS_ERR_INVALID, "comparators differ");
  cudaStream_t s = party_stream(dc->dm, 0, stream);
  CU(launch_merge_batch(dc->self_bitmap, right ? right->self_bitmap : nullptr, (uint32_t)n_queries,
                        (uint32_t)(dc->self_stride_bits / 32), dc->final_results, dc->match_counters,
                        dc->all_matches, s));
  return IRS_OK;
}

int irs_dc_fetch_final_results(irs_distance_comparator* dc, size_t n_queries, uint32_t* final_results,
                               uint32_t* match_counters, uint32_t* all_matches) {
  CHECK(dc && n_queries <= dc->max_queries, IRS_ERR_INVALID, "bad arguments");
  irs_device_manager* dm = dc->dm;
  CU(cudaSetDevice(dm->device));
  cudaStream_t s = dm->streams[0];
  if (dm->host_sync) {
    const size_t mq = dc->max_queries, words = all_matches ? 2 * mq + n_queries * kMaxMatchesLen : mq + n_queries;
    std::vector<uint32_t> got;
    const int rc = fetch_block(dc, dc->results_err, words, got, s);
    if (got.empty()) return rc;
    if (final_results) memcpy(final_results, got.data() + 4, n_queries * 4);
    if (match_counters) memcpy(match_counters, got.data() + 4 + mq, n_queries * 4);
    if (all_matches) memcpy(all_matches, got.data() + 4 + 2 * mq, n_queries * kMaxMatchesLen * 4);
    return rc;
  }
  // outputs valid once the stream passes the copies
  if (final_results) CU(cudaMemcpyAsync(final_results, dc->final_results, n_queries * 4, cudaMemcpyDeviceToHost, s));
  if (match_counters) CU(cudaMemcpyAsync(match_counters, dc->match_counters, n_queries * 4, cudaMemcpyDeviceToHost, s));
  if (all_matches)
    CU(cudaMemcpyAsync(all_matches, dc->all_matches, n_queries * kMaxMatchesLen * 4, cudaMemcpyDeviceToHost, s));
  return IRS_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Internal accessors (internal.h)
// ---------------------------------------------------------------------------
namespace irs {

int set_error(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
  return code;
}

int circuit_view(irs_circuits* c, CircuitView* v) {
  if (!c || !v) return set_error(IRS_ERR_INVALID, "circuits handle is NULL");
  for (int p = 0; p < 3; p++) v->keys[p] = c->keys[p];
  v->nonce = nonce_of(kDomCircuit, (uint32_t)c->dm->device);
  v->batch = c->batch;
  v->batch_dev = c->batch_from_device ? c->dm->d_batch : nullptr;
  v->device = c->dm->device;
  v->stream0 = c->dm->streams[0];
  return IRS_OK;
}

}  // namespace irs
