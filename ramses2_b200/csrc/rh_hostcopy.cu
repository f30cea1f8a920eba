// rh_hostcopy.cu — device state to pageable host memory.
//
// A plain copy into pageable memory runs at 4-5 GB/s: the driver stages it in
// small pieces, and one thread takes the page faults of a fresh destination.
// Here up to kSlots worker threads each own a pinned slot and a stream: a
// worker brings one piece of the source into its slot (a copy for FP64; for
// FP32-bulk records a kernel that widens them into the reference's FP64 layout
// and stores straight to the pinned slot), waits for it and copies the slot
// to the destination, so the link, the page faults and the copies of the
// other workers overlap.  FP32-bulk results were widened on the host in a
// scalar loop before.  An FP32-bulk ensemble of 24 problems (50 steps, 620 MB
// read back as FP64): 312 -> 98 ms in all, about 50 ms of it the steps.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>

#include "rh_internal.h"

namespace rh {
namespace {

constexpr int kSlots = 12;  // on 16 cores 622 MB took 119 ms with 1, 50 with 4, 36 with 8, 33 with 12, 31 with 16 workers
constexpr long long kSlotOcts = 13056;  // 4.2 MB of FP64 oct records
constexpr long long kPieceOcts = 1632;  // smallest piece, 522 KB
constexpr size_t kSlotBytes = sizeof(double) * 40 * kSlotOcts;
// Below this a copy is done before the workers have started: FP64 a plain one,
// FP32-bulk through a slot of its own, of one smallest piece (1,024 octs 55 us;
// 88 when the host widens the records; all slots pinned for it: 34 ms once).
constexpr long long kMinOcts = kPieceOcts;
constexpr int kSmall = kSlots;  // index of that slot

struct Ring {
  std::mutex mu;  // one transfer at a time
  double* slot[kSlots + 1] = {};
  cudaStream_t stream[kSlots + 1] = {};
  int n = 0;
};
Ring& ring() {
  static Ring r;
  return r;
}

// FP32-bulk records -> the FP64 layout [oct][5][8], one thread per value in
// output order (stores of a warp are 256 consecutive bytes).
__global__ void unpack_linear_kernel(double* __restrict__ dst, const float* __restrict__ uf,
                                     const double* __restrict__ ue, long long nval) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= nval) return;
  const long long oct = i / 40;
  const int k = (int)(i - 40 * oct);
  dst[i] = k < 32 ? (double)uf[oct * kBulkF + k] : ue[oct * kBulkD + (k - 32)];
}

// Brings octs [o, o + n) into slot w (asynchronously on its stream).
cudaError_t to_slot(Ring& r, int w, const OctSource& s, long long o, long long n) {
  if (!s.uf)
    return cudaMemcpyAsync(r.slot[w], s.ud + o * 40, sizeof(double) * 40 * n, cudaMemcpyDeviceToHost, r.stream[w]);
  unpack_linear_kernel<<<(unsigned)((n * 40 + 255) / 256), 256, 0, r.stream[w]>>>(r.slot[w], s.uf + o * kBulkF,
                                                                                  s.ud + o * kBulkD, n * 40);
  return cudaGetLastError();
}

// The calling thread's device, put back at the end of a transfer.
struct DeviceScope {
  int was = -1;
  cudaError_t set(int device) {
    cudaError_t e = cudaGetDevice(&was);
    if (e != cudaSuccess) was = -1;
    return e == cudaSuccess ? cudaSetDevice(device) : e;
  }
  ~DeviceScope() {
    if (was >= 0) cudaSetDevice(was);
  }
};

// Slot w of the given size and its stream, on the current device, kept for the
// next transfers.  False where pinned memory is short.
bool slot_ready(Ring& r, int w, size_t bytes) {
  if (!r.slot[w] && cudaMallocHost(&r.slot[w], bytes) != cudaSuccess) r.slot[w] = nullptr;
  if (r.slot[w] && !r.stream[w] && cudaStreamCreateWithFlags(&r.stream[w], cudaStreamNonBlocking) != cudaSuccess)
    r.stream[w] = nullptr;
  (void)cudaGetLastError();
  return r.slot[w] && r.stream[w];
}

// Slots for up to want workers: pinning one takes 3 to 6 ms, so a transfer gets
// no more than it has pieces.
int ring_ready(Ring& r, int want) {
  while (r.n < want && slot_ready(r, r.n, kSlotBytes)) ++r.n;
  return std::min(r.n, want);
}

// A plain copy, FP32-bulk records widened on the host: few octs in FP64, or no
// pinned memory.
int plain_copy(double* dst, const OctSource& s, long long noct) {
  if (!s.uf) {
    RH_CUDA(cudaMemcpy(dst, s.ud, sizeof(double) * 40 * noct, cudaMemcpyDeviceToHost));
    return RH_OK;
  }
  const long long step = std::min(noct, kMinOcts);
  std::unique_ptr<float[]> rec(new (std::nothrow) float[step * kBulkF]);
  if (!rec) {
    set_error("no host memory to read a state back");
    return RH_ENOMEM;
  }
  for (long long o = 0; o < noct; o += step) {
    const long long n = std::min(step, noct - o);
    RH_CUDA(cudaMemcpy(rec.get(), s.uf + o * kBulkF, (size_t)kBulkBytes * n, cudaMemcpyDeviceToHost));
    for (long long i = 0; i < n; ++i) {
      for (int k = 0; k < 32; ++k) dst[(o + i) * 40 + k] = rec[i * kBulkF + k];
      std::memcpy(dst + (o + i) * 40 + 32, rec.get() + i * kBulkF + 32, 8 * sizeof(double));
    }
  }
  return RH_OK;
}

}  // namespace

bool pageable(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

int octs_to_host(double* dst, const OctSource& s, long long noct, int device) {
  if (noct <= 0) return RH_OK;
  DeviceScope scope;
  RH_CUDA(scope.set(device));
  // pinned already: the link's rate without a slot (FP32-bulk goes through slots:
  // a kernel storing to dst would need all of it pinned, and only its first byte
  // is known to be)
  if (!s.uf && !pageable(dst)) {
    RH_CUDA(cudaMemcpy(dst, s.ud, sizeof(double) * 40 * noct, cudaMemcpyDeviceToHost));
    return RH_OK;
  }
  Ring& r = ring();
  std::lock_guard<std::mutex> lock(r.mu);
  // pieces of a slot's size, smaller where a transfer would leave workers idle
  // (47 MB in 12 problems: 9.0 ms with whole slots, 6.4 so; 620 MB in 24: 39 ms,
  // 48 with pieces of 522 KB throughout)
  const long long piece = std::min(kSlotOcts, std::max(kPieceOcts, noct / 16));
  const long long npiece = (noct + piece - 1) / piece;
  const int hw = std::max(1, (int)std::thread::hardware_concurrency() * 3 / 4);
  const bool few = noct < kMinOcts;
  const int nw = few ? 0 : ring_ready(r, (int)std::min<long long>(std::min(kSlots, hw), npiece));
  if (few && s.uf && slot_ready(r, kSmall, sizeof(double) * 40 * kMinOcts)) {
    RH_CUDA(to_slot(r, kSmall, s, 0, noct));
    RH_CUDA(cudaStreamSynchronize(r.stream[kSmall]));
    std::memcpy(dst, r.slot[kSmall], sizeof(double) * 40 * noct);
    return RH_OK;
  }
  if (nw == 0) return plain_copy(dst, s, noct);
  std::atomic<long long> next{0};
  std::atomic<int> err{cudaSuccess};
  auto work = [&](int w) {
    // a worker without the device leaves its pieces to the caller, worker 0
    if (w > 0 && cudaSetDevice(device) != cudaSuccess) return;
    for (long long i; (i = next.fetch_add(1)) < npiece;) {
      const long long o = i * piece, n = std::min(piece, noct - o);
      cudaError_t e = to_slot(r, w, s, o, n);
      if (e == cudaSuccess) e = cudaStreamSynchronize(r.stream[w]);
      if (e != cudaSuccess) {
        err = e;
        return;
      }
      std::memcpy(dst + o * 40, r.slot[w], sizeof(double) * 40 * n);
    }
  };
  std::thread th[kSlots];
  for (int w = 1; w < nw; ++w) {
    try {
      th[w] = std::thread(work, w);
    } catch (...) {
      break;  // no more threads, or memory for them: the running ones take the pieces
    }
  }
  work(0);
  for (int w = 1; w < nw; ++w)
    if (th[w].joinable()) th[w].join();
  if (err != cudaSuccess) return cuda_fail((cudaError_t)err.load(), "state to the host");
  return RH_OK;
}

void free_host_ring() {
  Ring& r = ring();
  std::lock_guard<std::mutex> lock(r.mu);
  for (int w = 0; w <= kSlots; ++w) {
    if (r.stream[w]) cudaStreamDestroy(r.stream[w]);
    cudaFreeHost(r.slot[w]);
    r.slot[w] = nullptr;
    r.stream[w] = nullptr;
  }
  r.n = 0;
}

}  // namespace rh
