// internal.h -- state shared by the library's translation units (not part
// of the C-ABI).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <string>

// one device and one stream; `scratch` is reusable device memory for calls
// that stage host arrays (the geometry sampling), grown on demand and freed
// with the context.  `relax_tune` caches the smoother autotuner's choice
// (colour cells per thread) per precision, h^2 form and level size class, so
// hierarchies uploaded later on the same context are not re-timed.
struct bsam_ctx_s {
  int device = 0;
  cudaStream_t stream = nullptr;
  void *scratch = nullptr;
  size_t scratch_bytes = 0;
  std::mutex tune_mu;
  std::map<uint64_t, int> relax_tune;
  // the context lives while it is open or a hierarchy made on it exists
  std::mutex ref_mu;
  int refs = 1;
};

// records the message of a failed call for bsam_last_error(); returns code
int bsam_internal_set_error(int code, const std::string &msg);

// most dynamic shared memory of a k_relax_tile block
constexpr int kTileMaxBytes = 200 * 1024;

// what a block of an FP64 tile launch asks for, `need` at least: a block's
// passes share its SM's FP64 pipe with any other block there, so the blocks of
// a grid that covers a good part of the SMs ask for as much as spreads them
// evenly (starfish -1.4%; a handful of blocks only pays for the larger request:
// a 1,024-cell solve +2%).  With more blocks per SM than have a share, need.
// Solves/s with the request / without, 1, 2, 4 and 8 hierarchies on streams of
// their own: disc (64^2 base, three levels) 882 / 846, 1646 / 1584, 2866 / 2933,
// 3546 / 4002; starfish 324 / 317, 475 / 473, 648 / 679, 686 / 731 (chained
// passes: 511, 950, 1601, 2370 and 199, 306, 447, 535): a lone solve is the
// common case, and many side by side still pass the chained ones by far.
inline size_t tile_request(size_t need, int ntiles, int sms) {
  if (4 * (int64_t)ntiles < sms) return need;
  const int per_sm = (ntiles + sms - 1) / sms;
  const int share = std::min(kTileMaxBytes, 224 * 1024 / per_sm - 2048);
  return share > 0 ? std::max(need, (size_t)share) : need;
}
