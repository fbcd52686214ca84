// Copies of states and rates between the device and the caller's memory.
//
// The caller's memory is pageable as a rule.  The driver copies it to the host
// through its own staging and waits in every call, about 10 us however small the
// copy.  Up to kStagingMax bytes the copies of a call are queued together instead,
// through pinned staging of the context, with one wait (from kLaneBytes on in four
// lanes, one copied out on the host while the next arrives).  Larger ones, copies
// to the device, and memory that the caller has registered go directly.  One
// B200, all wake rates: N = 512 35 -> 23 us, 16,384 in two wakes 127 -> 107, 20,011
// in three 188 -> 140; the states of N = 2,048 43 -> 23.  (Above 1 MB a ring of
// lanes took as long as the driver or twice as long; four host threads copying
// 6.3 MB to staging for the device 0.9 ms against 0.6.)
#include <algorithm>
#include <cstring>

#include "runtime.h"

namespace pawan {
namespace {

constexpr size_t kLanes = 4;
constexpr size_t kStagingMax = 1u << 20;
constexpr size_t kLaneBytes = 128u << 10;  // fewer bytes go as one lane

bool pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// Joins neighbours and adds up the bytes.
size_t join(std::vector<HostCopy> &v) {
  size_t k = 0, total = 0;
  for (const HostCopy &c : v) {
    if (c.bytes == 0) continue;
    total += c.bytes;
    const size_t d = k > 0 ? v[k - 1].bytes / sizeof(double) : 0;
    if (k > 0 && v[k - 1].dev + d == c.dev && v[k - 1].host + d == c.host)
      v[k - 1].bytes += c.bytes;
    else
      v[k++] = c;
  }
  v.resize(k);
  return total;
}

// Staging for `bytes` bytes; false when there is no memory for it.
bool ensure_staging(pawan_ctx *ctx, size_t bytes) {
  for (cudaEvent_t &e : ctx->staging_events)
    if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      e = nullptr;
      cudaGetLastError();
      return false;
    }
  if (ctx->staging_bytes >= bytes) return true;
  const size_t size = bytes <= kLaneBytes ? kLaneBytes : kStagingMax;
  void *p = nullptr;
  if (cudaHostAlloc(&p, size, cudaHostAllocDefault) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (ctx->staging) cudaFreeHost(ctx->staging);
  ctx->staging = static_cast<char *>(p);
  ctx->staging_bytes = size;
  return true;
}

// Calls f(copy, offset in it, bytes, position) for the bytes [p0, p1) of the
// copies laid end to end.
template <class F>
void each(const std::vector<HostCopy> &v, size_t p0, size_t p1, F f) {
  size_t at = 0;
  for (const HostCopy &c : v) {
    const size_t a = std::max(at, p0), b = std::min(at + c.bytes, p1);
    if (a < b) f(c, a - at, b - a, a);
    at += c.bytes;
  }
}

}  // namespace

int copy_to_host(pawan_ctx *ctx, std::vector<HostCopy> v) {
  const size_t total = join(v);
  bool staged = total > 0 && total <= kStagingMax;
  for (const HostCopy &c : v) staged = staged && pageable(c.host);
  if (!staged || !ensure_staging(ctx, total)) {
    for (const HostCopy &c : v)
      PAWAN_CUDA(ctx, cudaMemcpyAsync(c.host, c.dev, c.bytes, cudaMemcpyDeviceToHost, ctx->stream));
    PAWAN_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return PAWAN_OK;
  }
  char *const pin = ctx->staging;
  const size_t lane = total <= kLaneBytes ? total : (total + kLanes - 1) / kLanes;
  for (size_t l = 0; l * lane < total; ++l) {
    cudaError_t e = cudaSuccess;
    each(v, l * lane, (l + 1) * lane, [&](const HostCopy &c, size_t at, size_t bytes, size_t pos) {
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(pin + pos, reinterpret_cast<const char *>(c.dev) + at, bytes, cudaMemcpyDeviceToHost,
                            ctx->stream);
    });
    PAWAN_CUDA(ctx, e);
    PAWAN_CUDA(ctx, cudaEventRecord(ctx->staging_events[l], ctx->stream));
  }
  for (size_t l = 0; l * lane < total; ++l) {
    PAWAN_CUDA(ctx, cudaEventSynchronize(ctx->staging_events[l]));
    each(v, l * lane, (l + 1) * lane, [&](const HostCopy &c, size_t at, size_t bytes, size_t pos) {
      std::memcpy(reinterpret_cast<char *>(c.host) + at, pin + pos, bytes);
    });
  }
  return PAWAN_OK;
}

int copy_to_device(pawan_ctx *ctx, std::vector<HostCopy> v) {
  join(v);
  for (const HostCopy &c : v)
    PAWAN_CUDA(ctx, cudaMemcpyAsync(c.dev, c.host, c.bytes, cudaMemcpyHostToDevice, ctx->stream));
  return PAWAN_OK;
}

}  // namespace pawan
