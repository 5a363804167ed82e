// hg_host.h -- host-side pieces of the library shared between hg_api.cu
// (the C ABI, the context, single and batched products) and hg_service.cu
// (the device-resident multiply service).
#pragma once

#include <cstdint>
#include <mutex>
#include <vector>

#include "hg_epoch.h"
#include "hg_internal.h"

namespace hg {

// One pass of a transform plan: logR row bits, stride 2^logS, 2^logT-word tiles.
struct PassPlan {
  int logR, logS, logT;
};

// Products of one transform length and kind, run as one launch per pass.
struct BatchGroup {
  int L = 0;
  int k16 = 16;                    // sixteenths of the 2^L points that are kept (16: a whole transform)
  bool dig80 = false;              // coefficients are 80-bit digits
  bool square = false;
  bool tails = false;              // some product has nout > N
  std::vector<PassPlan> plan;
  uint64_t first = 0, nprod = 0;   // descriptors [first, first + nprod)
  uint64_t flags_off = 0;          // first carry-scan flag word
  uint64_t ws_off = 0;             // first workspace word
};

// Streams beside a batch's own, for groups that run at the same time.  Each
// batch (and service slot) has its own: a captured batch captures them too.
struct SideStreams {
  static constexpr int kMax = 3;
  int n = 0;
  cudaStream_t st[kMax] = {};
  cudaEvent_t fork = nullptr, join[kMax] = {};
  cudaError_t create();
  void destroy();
};

// A planned batch: groups contiguous in desc, then the products with an empty
// operand (zeroed, no transform).  Where the workspace of all groups fits the
// cap (parallel), each has its own part of it and groups may run at the same
// time; else they run one after another and share it.
struct BatchPlan {
  std::vector<BatchGroup> groups;
  bool parallel = false;
  std::vector<ProductDesc> desc;
  uint64_t zero_first = 0, nzero = 0;
  uint64_t ws_words = 0, flag_words = 0;
  uint64_t in_turn_words = 0;  // ws_words of groups that run one after another
  void run_in_turn() {
    parallel = false;
    ws_words = in_turn_words;
    for (BatchGroup &g : groups) g.ws_off = 0;
  }
};

// Device buffers a planned batch runs in.
struct BatchBufs {
  const ProductDesc *desc;    // device copy of BatchPlan::desc
  uint64_t *ws;               // ws_words words
  unsigned long long *flags;  // flag_words words
  unsigned long long *tickets;  // one per group (the carry's finished-tile count), zero between runs
  int *err;                   // device error word
  const SideStreams *side;    // or null: groups one after another
  uint32_t epoch;             // this run's (ScanEpoch)
};

// Workspace bytes one product occupies while its group runs.
uint64_t product_workspace_bytes(uint64_t nx, uint64_t ny, bool square);

// Group validated descriptors by (transform length, square) and split groups
// so that none needs more than ws_cap_bytes of workspace.  whole: every product
// by the whole transform of its limbs.
int plan_batch(const ProductDesc *items, size_t n, uint64_t ws_cap_bytes, BatchPlan &bp, bool whole = false);

// sa |a| + sb |b| into out[0, nout) over the whole GPU (nout >= the longer
// operand's end + 1; limbs past the sum are zeroed); (sign, size) into result[0, 2)
// on the device.  Uses the library's carry-scan state, ordered like the
// products' workspace.
int large_sum_device(const SumOperand &a, int64_t sa, const SumOperand &b, int64_t sb, uint64_t *out, uint64_t nout,
                     int64_t *result, cudaStream_t st);

// Enqueue a planned batch on st: zero the empty products, run every group.  A
// captured run, whose epoch is the same on every replay, clears its flags.  Takes no lock and allocates nothing.
int enqueue_batch(const BatchPlan &bp, const BatchBufs &bb, cudaStream_t st);

// Fill or upload device memory, done on return.  cudaMemset and cudaMemcpy from
// pageable memory may return before the device is done, and neither the
// library's streams nor a caller's are ordered after the null stream.
inline cudaError_t fill_now(void *p, int byte, size_t bytes) {
  const cudaError_t e = cudaMemset(p, byte, bytes);
  return e == cudaSuccess ? cudaStreamSynchronize(nullptr) : e;
}
inline cudaError_t upload_now(void *dst, const void *src, size_t bytes) {
  const cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  return e == cudaSuccess ? cudaStreamSynchronize(nullptr) : e;
}

// Page-locked words that kernels write and the host reads after a
// synchronisation: one call's from take to give, then kept for the next (64 MB
// of them) until hg_shutdown.  Taking and giving hold no lock that
// any other is taken under.
struct HostWords {
  int64_t *host = nullptr, *dev = nullptr;
  size_t words = 0;
};
int host_words_take(size_t words, HostWords *w);
void host_words_give(const HostWords &w);

// The library's device error word; lib_device_error resets it when `err`,
// read from it, is not 0, and returns the error (in checked builds also a
// fault that a check latched).
int *lib_err_word();
int lib_device_error(int err, cudaStream_t st);

// Give back the descriptor memory that hg_sum.cu keeps (hg_shutdown).
void lib_release_descs();

// The library's state, for code outside hg_api.cu.
std::recursive_mutex &lib_mutex();
bool lib_ready();
int lib_device();
// Record an error message (hg_last_error) and return code.
int lib_fail(int code, const char *fmt, ...);
int lib_cuda_fail(cudaError_t e, const char *what);
// Count of open services; hg_shutdown refuses while it is nonzero.
void lib_service_count(int delta);

// Butterflies per second of a memory-free network of the library's modular
// butterflies (hg_peak.cu), with prime pc and a device table of at least
// 1024 (twiddle, companion) pairs.
int butterfly_peak(double *per_s, const PrimeConst &pc, const ulonglong2 *table);

}  // namespace hg
