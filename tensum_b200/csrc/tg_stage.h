// tg_stage.h -- copies between pageable caller buffers and the device.
//
// Up to kMaxLanes host threads, each with its own stream and two pinned slots, so that
// the host memcpy of one slot (and the page faults of a buffer that is touched for the first
// time) overlaps the DMA of the other and the other lanes'.  Pinned caller buffers need none
// of it: one cudaMemcpyAsync.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

namespace tg {

inline bool host_pinned(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

struct Stager {
  static constexpr int kMaxLanes = 8;
  static constexpr size_t kPerLane = size_t(1) << 20;   // the least worth a lane
  int device = 0, lanes = 0;
  size_t slot_bytes = 0;
  char* slots = nullptr;   // pinned, lanes * 2 * slot_bytes
  cudaStream_t st[kMaxLanes] = {};
  cudaEvent_t ev[kMaxLanes][2] = {};

  // A lane per MiB, but never two: one helper thread alone often wakes late, and its lane takes
  // as long as the whole copy.  Medians in us of set_state / get_state from pageable buffers
  // with one lane and two: 229^2 224 / 175 and 320 / 265, 257^2 258 / 210 and 370 / 310; of
  // 300^2 with two and three 400 / 320 and 290 / 215.
  static int lanes_for(size_t bytes) {
    const size_t n = bytes / kPerLane;
    return n < 3 ? 1 : (int)std::min<size_t>(kMaxLanes, n);
  }
  // 512 KiB (page-locking memory is most of a small handle's creation), 1 MiB where every lane
  // fills that twice: 513^2 590 / 435 us either way, 700^2 with 512 KiB / 1 MiB 945 / 780 and
  // 805 / 725, 900^2 1480 / 1310 and 1150 / 1080.
  static size_t slot_for(size_t bytes) { return bytes >= 2 * kMaxLanes * kPerLane ? kPerLane : kPerLane / 2; }
  // lanes for transfers of up to `bytes`, with slots of `most` at most; a later call may ask for more
  cudaError_t init(int dev, size_t bytes, size_t most = kPerLane) {
    device = dev;
    const int want = lanes_for(bytes);
    if (want <= lanes) return cudaSuccess;
    release();
    slot_bytes = std::min(most, slot_for(bytes));
    cudaError_t e = cudaMallocHost((void**)&slots, 2 * (size_t)want * slot_bytes);
    for (int t = 0; t < want && e == cudaSuccess; ++t) {
      e = cudaStreamCreateWithFlags(&st[t], cudaStreamNonBlocking);
      for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaEventCreateWithFlags(&ev[t][k], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) lanes = want;
    else release();
    return e;
  }
  void release() {
    for (int t = 0; t < kMaxLanes; ++t) {
      if (st[t]) cudaStreamSynchronize(st[t]);
      for (int k = 0; k < 2; ++k) {
        if (ev[t][k]) cudaEventDestroy(ev[t][k]);
        ev[t][k] = nullptr;
      }
      if (st[t]) cudaStreamDestroy(st[t]);
      st[t] = nullptr;
    }
    if (slots) cudaFreeHost(slots);
    slots = nullptr;
    lanes = 0;
  }
  char* slot(int lane, int k) const { return slots + (2 * (size_t)lane + k) * slot_bytes; }

  // One lane of a host -> device copy of len bytes.
  cudaError_t lane_in(int lane, char* dst, const char* src, size_t len) const {
    cudaError_t e = cudaSetDevice(device);
    for (size_t off = 0, k = 0; e == cudaSuccess && off < len; off += slot_bytes, ++k) {
      const int s = (int)(k & 1);
      const size_t n = std::min(slot_bytes, len - off);
      if (k >= 2 && (e = cudaEventSynchronize(ev[lane][s])) != cudaSuccess) break;
      std::memcpy(slot(lane, s), src + off, n);
      if ((e = cudaMemcpyAsync(dst + off, slot(lane, s), n, cudaMemcpyHostToDevice, st[lane])) != cudaSuccess) break;
      e = cudaEventRecord(ev[lane][s], st[lane]);
    }
    cudaError_t e2 = cudaStreamSynchronize(st[lane]);
    return e != cudaSuccess ? e : e2;
  }

  // One lane of a device -> host copy; the lane's stream first waits for `ready`.
  cudaError_t lane_out(int lane, char* dst, const char* src, size_t len, cudaEvent_t ready) const {
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st[lane], ready, 0);
    const size_t nk = (len + slot_bytes - 1) / slot_bytes;
    auto issue = [&](size_t k) {
      const int s = (int)(k & 1);
      const size_t n = std::min(slot_bytes, len - k * slot_bytes);
      cudaError_t ei = cudaMemcpyAsync(slot(lane, s), src + k * slot_bytes, n, cudaMemcpyDeviceToHost, st[lane]);
      return ei != cudaSuccess ? ei : cudaEventRecord(ev[lane][s], st[lane]);
    };
    for (size_t k = 0; e == cudaSuccess && k < std::min<size_t>(2, nk); ++k) e = issue(k);
    for (size_t k = 0; e == cudaSuccess && k < nk; ++k) {
      const int s = (int)(k & 1);
      if ((e = cudaEventSynchronize(ev[lane][s])) != cudaSuccess) break;
      std::memcpy(dst + k * slot_bytes, slot(lane, s), std::min(slot_bytes, len - k * slot_bytes));
      if (k + 2 < nk) e = issue(k + 2);
    }
    cudaError_t e2 = cudaStreamSynchronize(st[lane]);
    return e != cudaSuccess ? e : e2;
  }

  // Splits a copy over the lanes (lane 0 on the calling thread; where no thread is to be had,
  // the calling one does the rest).
  template <class Lane>
  cudaError_t run(size_t bytes, Lane lane) const {
    const int n = std::min(lanes, lanes_for(bytes));
    const size_t per = ((bytes + n - 1) / n + 255) & ~size_t(255);
    cudaError_t errs[kMaxLanes] = {};
    std::thread th[kMaxLanes];
    auto work = [&](int t) {
      const size_t off = t * per;
      if (off < bytes) errs[t] = lane(t, off, std::min(per, bytes - off));
    };
    int started = 1;
    try {
      for (; started < n; ++started) th[started] = std::thread(work, started);
    } catch (const std::system_error&) {
    }
    work(0);
    for (int t = started; t < n; ++t) work(t);
    for (int t = 1; t < started; ++t) th[t].join();
    for (cudaError_t e : errs)
      if (e != cudaSuccess) return e;
    return cudaSuccess;
  }

  cudaError_t in(void* dst, const void* src, size_t bytes) const {
    return run(bytes, [&](int t, size_t off, size_t len) { return lane_in(t, (char*)dst + off, (const char*)src + off, len); });
  }
  cudaError_t out(void* dst, const void* src, size_t bytes, cudaEvent_t ready) const {
    return run(bytes, [&](int t, size_t off, size_t len) {
      return lane_out(t, (char*)dst + off, (const char*)src + off, len, ready);
    });
  }
};

}  // namespace tg
