// mgcd_plan.h -- host-side state of the library: the context (device, moduli table,
// inverse table, launch configuration) and plans (one batch's buffers, streams and
// schedule).  A context owns one plan for its own calls; the request server owns one plan
// per in-flight wave, all sharing the context's resident tables.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "../../include/modgcd.h"
#include "mgcd_internal.h"

namespace mgcd {

// Device buffer from the context's stream-ordered memory pool: growing it neither blocks
// the host nor serialises the other streams (plain cudaMalloc/cudaFree would).
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaError_t grow(size_t want, cudaMemPool_t pool, cudaStream_t s);
  void release(cudaStream_t s);
  template <class T> T* as() const { return static_cast<T*>(p); }
};

// Pinned host buffer (grow-only, doubling).  A buffer it outgrows is kept until release():
// cudaFreeHost waits for all work on the device, which would stall a server behind every
// kernel in flight.
struct HostBuf {
  void* p = nullptr;
  size_t bytes = 0;
  std::vector<void*> retired;
  cudaError_t grow(size_t want);
  void release();
  template <class T> T* as() const { return static_cast<T*>(p); }
};

struct Bucket {
  int threads, k;      // CTA size, pairs per CTA in lockstep
  int csize;           // CTAs per thread-block cluster (0: one CTA per pair)
  int cls;             // size class
  uint32_t first, n, nq_max;
  int grid;            // CTAs (csize = 0) or clusters
  size_t smem;
  size_t scratch_off;  // words
};

// Size classes of the batched path, one persistent kernel each: pairs with at
// most 1,024 / 4,096 / 16,384 moduli run K per CTA (or K per small cluster, when the class
// or a serving lane asks for one); larger pairs K per thread-block cluster.
constexpr int NSTREAMS = MGCD_NUM_SIZE_CLASSES;
constexpr int CLUSTER_CLASS = 3;
constexpr size_t GSYNC_PLACES = 16, GSYNC_STRIDE = 36864;   // bytes between the places
constexpr size_t INVTAB_N = 16384;        // moduli covered by the pairwise inverse table

inline int size_class(uint32_t nq) { return nq <= 1024 ? 0 : nq <= 4096 ? 1 : nq <= CTA_MAX_NQ ? 2 : CLUSTER_CLASS; }

// Moduli a batched pair may grow to (mgcd_set_growth): a sixteenth more than the reference's
// count, so that a pair whose smaller sets took more iterations still ends in its own loop
// (with the growth policy's defaults no pair of the mixed 1k-64k-bit batches went past the
// reference's count in the oracle's runs), rounded up to a warp.  The cap sizes a bucket's
// shared memory and scratch: the mixed batch ran 73.9 ms with an eighth, 72.8 with this.
inline uint32_t grow_cap(uint32_t ref) { return std::min<uint32_t>(CTA_MAX_NQ, (ref + ref / 16 + 31u) / 32u * 32u); }

struct Plan {
  cudaStream_t stream = nullptr;       // every launch of the plan
  cudaEvent_t t_run0 = nullptr, t_run1 = nullptr;   // timing of the whole run

  size_t np = 0;                       // pairs in the plan
  std::vector<int32_t> status;         // per pair: MGCD_OK / error code / -1 = computed on the GPU
  std::vector<int> slot;               // per pair: index into GPU arrays, or -1
  std::vector<std::vector<uint32_t>> trivial;  // per pair: host-decided result (zero operand)
  std::vector<PairDesc> descs;         // GPU pairs
  std::vector<uint32_t> order;
  std::vector<Bucket> buckets;
  std::vector<uint32_t> grid_pairs;    // GPU indices run as single-pair launches
  std::vector<uint32_t> ref_nq, eff_nq; // per GPU pair: reference count, count of the final run
  size_t ndig = 0, scratch_words = 0, grid_scratch_off = 0;
  size_t nglimbs = 0;                  // result limbs reserved (sum of g_cap)
  // results planned in the caller's layout (mgcd_gcd_batch, slots contiguous): the device's limb x
  // is the caller's g[direct_base + x], copied there in one piece; in_place: fetch did so
  bool direct = false, in_place = false;
  uint64_t direct_base = 0;
  bool plain = false;                  // single-pair latency policy
  bool graphable = true;               // may be recorded into a CUDA graph (context setting)
  bool spread = false;                 // small batches spread their pairs over clusters (schedule)
  int cluster_ctas = 0;                // CTAs per cluster of size class 3 (0: the context's setting)
  int small_cluster_ctas = 0;          // CTAs per cluster for pairs of size classes 1-2 (0: the
                                       // context's setting); serving waves favour latency
  int cluster_k = 0;                   // pairs per cluster of size class 3 (0: the context's setting)

  // One block for what goes up and one for what comes back, so that a small call costs one
  // copy each way and two fills: a copy or a fill takes about 2 us of the stream and as much of
  // the host, and the separate buffers had 3 copies up, 8 back and 5 fills (a 512-bit pair
  // 125 us with them, 106 with the blocks).
  DevBuf d_in;                         // operand limbs, then `in`'s parts
  DevBuf d_res;                        // `res`'s parts
  struct In { size_t pairs = 0, order = 0, end = 0; } in;      // byte offsets; order has room for a rerun's
  struct Res {                         // byte offsets
    size_t span = 0, status = 0;       // filled with ones: span (per bucket kernel: earliest CTA
                                       // start, ~(latest CTA end), ns), status per pair
    size_t upd = 0, nqf = 0, queue = 0;   // zeroed: per pair (K-slot kernels) loop updates and final
                                       // moduli count; the buckets' work counters, a rerun's after them
    size_t count = 0, iters = 0, glen = 0;   // per pair
    size_t glimbs = 0;                 // binary gcds converted on the device
    size_t digits = 0, end = 0;
  } res;
  std::vector<unsigned char> in_host;  // a small plan's d_in, put together for one copy
  DevBuf d_scratch, d_retry;
  DevBuf d_trace;                      // per-CTA occupancy trace of the bucket kernels (4 words each)
  DevBuf d_phases;                     // per-CTA phase accounting of the K-slot kernels (8 words each)
  std::vector<int> trace_cls;          // size class of each traced CTA (launch order)
  HostBuf h_res;                       // d_res's start, up to what fetch copies
  HostBuf h_digits;                    // digits the host converts (batches)
  bool fetched = false;                // h_res holds a run of this plan
  int launches = 0, retried = 0;
  bool ran = false, synced = false, bucket_timed = false;
  double work[4] = {0, 0, 0, 0};       // residue steps, loop updates, recovery updates, operand bytes
  double alg_bytes = 0;                // algorithmic bytes: operands + (prime, constant) per modulus + digits
  std::vector<double> bucket_work;     // the same per bucket kernel (4 per bucket)
  uint64_t h2d_bytes = 0, d2h_bytes = 0;

  // CUDA graph of the plan's GPU work; dropped whenever a buffer it uses moves
  cudaGraphExec_t graph = nullptr;
  int graph_kernels = 0;

  cudaError_t create(int priority = 0);   // the stream at this priority (lower = more urgent)
  void destroy(cudaMemPool_t pool);
  void drop_graph();
  size_t device_bytes() const;
  void layout(size_t ng, uint64_t limb_words);
  size_t fetch_bytes() const { return plain ? res.end : res.digits; }   // d_res's part for the host
  template <class T> T* din(size_t off) const { return reinterpret_cast<T*>(d_in.as<unsigned char>() + off); }
  template <class T> T* dres(size_t off) const { return reinterpret_cast<T*>(d_res.as<unsigned char>() + off); }
  template <class T> T* hres(size_t off) const { return reinterpret_cast<T*>(h_res.as<unsigned char>() + off); }
};

}  // namespace mgcd

struct mgcd_context {
  int device = 0, L = 32, sms = 0;
  size_t smem_optin = 0;               // largest dynamic shared memory per CTA
  cudaMemPool_t pool = nullptr;
  std::vector<uint32_t> moduli;
  mgcd::DevBuf mods;
  mgcd::DevBuf d_invtab;               // pairwise inverse table (InvTab)
  uint32_t invtab_n = 0;
  mgcd::DevBuf d_xchg;                 // GSYNC_PLACES places for the grid exchange's lines
  mgcd::GridSync* gsync = nullptr;     // the fastest of them (calibrate_exchange), from the first grid pair on
  mgcd::Plan main;                     // the plan of the context's own calls
  bool serving = false;                // a request server runs on this context

  // Per size class of the batched path: CTA size, pairs per CTA in lockstep, fraction of
  // the reference moduli count, CTAs per cluster (cluster class only).
  struct ClassCfg { int threads, k; float nq_scale; int csize; };
  ClassCfg cfg[mgcd::NSTREAMS] = {{256, 2, 1.0f, 0}, {512, 2, 1.0f, 0}, {1024, 2, 1.0f, 0}, {1024, 1, 1.0f, 8}};
  bool spread = true;                  // small batches spread their pairs over clusters; off once the
                                       // caller sets a shape, fraction or growth (mgcd_set_spread)
  bool shaped[mgcd::NSTREAMS] = {};    // classes whose shape the caller has set (mgcd_set_size_class)
  bool use_graph = false;
  // How many clusters of a shape fit at once, as the runtime answered (it takes ~1 us a shape
  // and a small batch asks for up to twelve per class); at most FITS of them.
  static constexpr size_t FITS = 256;
  struct Fit { int threads, k, csize; size_t smem; int clusters; };
  std::vector<Fit> fits;
  int single_policy = MGCD_SINGLE_AUTO;  // launch shape of pairs that span several CTAs
  unsigned long long wait_timeout_ns = 2000000000ull;   // bound of every cross-CTA wait
  uint32_t withhold_cta = 0xFFFFFFFFu;                  // test hook (mgcd_test_withhold_cta)
  uint32_t stage_fail_cta = 0xFFFFFFFFu;                // test hook (mgcd_test_fail_staging)
  uint32_t force_nq = 0;                                // test hook (mgcd_test_force_moduli)
  bool trace = false;                                   // record per-CTA occupancy (mgcd_set_cta_trace)
  // Moduli grown on demand in the K-slot kernels (mgcd_set_growth): batched pairs start with
  // this fraction of the reference count (0: off) and grow by grow_permille thousandths of it
  // at a time, up to the reference count.
  float grow_start = 0.4f;
  uint32_t grow_permille = 50;
};

namespace mgcd {

// Plan operations (mgcd_capi.cpp).  All return MGCD_* codes.
//   plan_batch   validate, order and size the pairs on the host, copy the batch to the
//                device on P.stream (asynchronous when `limbs` is pinned); given the
//                caller's result layout (g_off, g_cap), results are planned in it when its
//                slots are contiguous (Plan::direct);
//   run_plan     launch the GPU work (asynchronous);
//   sync_plan    wait; rerun uncertified pairs of a scaled run with the reference count;
//   fetch        copy the results back (pinned; a direct plan's binary results straight
//                into `direct_g`, the caller's array) and account the work;
//   convert_all  digits -> binary gcds for every pair of the plan.
int plan_batch(mgcd_context* c, Plan& P, size_t np, const uint32_t* limbs, const uint64_t* u_off,
               const uint32_t* u_len, const uint64_t* v_off, const uint32_t* v_len, bool plain,
               const uint64_t* g_off = nullptr, const uint32_t* g_cap = nullptr);
int run_plan(mgcd_context* c, Plan& P);
int sync_plan(mgcd_context* c, Plan& P, bool fetch_next = false);
int fetch(mgcd_context* c, Plan& P, uint32_t* direct_g = nullptr);
int convert_all(mgcd_context* c, Plan& P, uint32_t* g, const uint64_t* g_off, const uint32_t* g_cap,
                uint32_t* g_len, int32_t* status, bool threaded);
int to_status(int32_t st);

}  // namespace mgcd
