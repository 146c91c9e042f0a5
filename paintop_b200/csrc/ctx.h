// ctx.h -- the library context behind the opaque pt_ctx handle.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdlib>
#include <mutex>
#include <string>

struct pt_ctx {
  int device = 0;
  int sms = 0;
  cudaStream_t stream = nullptr;
  std::mutex mu;               // one call at a time per context
  void *arena = nullptr;       // device memory, grown to a high-water mark
  size_t arena_cap = 0;
  std::string last_error;
  double budget_s = 600.0;     // wall budget of one persistent solve
  int last_grid = 0;           // blocks of the last persistent launch
  int last_cfg = -1;           // tile configuration of the last solve
  int forced_cfg = -1;         // configuration override (-1: use the table)
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};  // call start, solve start/end, call end
  double last_solve_ms = 0.0;  // persistent kernel, CUDA events on `stream`
  double last_call_ms = 0.0;   // whole call from first upload to last download
  long long last_launches = 0; // kernels launched by the last call
  unsigned long long last_h2d = 0, last_d2h = 0;  // bytes the last solve moved each way
  void *pin = nullptr;         // staging of plans and results, grown to a high-water mark
  size_t pin_cap = 0;
  bool pin_paged = false;      // page-locked memory was not to be had
  int solve_grid[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // blocks of k_solve that fit the device, by tile configuration
  int cluster_room = -1;       // largest clusters that fit the device at a time (-1: not asked yet)
  static constexpr int kSides = 7;
  cudaStream_t side[kSides] = {};       // for launches beside one another (made when first needed)
  cudaEvent_t forked = nullptr, joined[kSides] = {};
  bool graphs = true;          // capture device-pointer solves into a CUDA graph
  cudaGraphExec_t gexec = nullptr;
  std::string gkey;            // the plan the cached graph was captured for
  cudaGraphExec_t mgexec[3] = {nullptr, nullptr, nullptr};  // multigrid-CG iteration: first / odd / even
  std::string mgkey;           // the problem shape and arena the multigrid graphs were captured for
  long long mgnodes = 0;       // kernels in one of those iterations
  bool mg_prepared = false;    // the multigrid kernels' attributes are set

  void drop_graphs() {
    if (gexec) { cudaGraphExecDestroy(gexec); gexec = nullptr; }  // they point into the arena
    gkey.clear();
    for (auto &g : mgexec)
      if (g) { cudaGraphExecDestroy(g); g = nullptr; }
    mgkey.clear();
  }

  // Until nothing of a call runs any more, on the side streams either: a call
  // that failed between its fork and its join left those unwaited for.
  void wait_all() {
    cudaStreamSynchronize(stream);
    for (cudaStream_t s : side)
      if (s) cudaStreamSynchronize(s);
  }

  bool reserve(size_t bytes) {
    if (bytes <= arena_cap) return true;
    if (arena) {
      wait_all();
      drop_graphs();
      cudaFree(arena);
      arena = nullptr;
      arena_cap = 0;
    }
    size_t want = bytes + bytes / 4;
    if (cudaMalloc(&arena, want) != cudaSuccess) {
      cudaGetLastError();
      arena = nullptr;
      if (cudaMalloc(&arena, bytes) != cudaSuccess) {
        cudaGetLastError();
        arena = nullptr;
        return false;
      }
      want = bytes;
    }
    arena_cap = want;
    return true;
  }

  // The first n side streams and their events.
  cudaError_t make_sides(int n) {
    cudaError_t e = cudaSuccess;
    if (!forked) e = cudaEventCreateWithFlags(&forked, cudaEventDisableTiming);
    for (int k = 0; k < n && e == cudaSuccess; ++k) {
      if (!side[k]) e = cudaStreamCreateWithFlags(&side[k], cudaStreamNonBlocking);
      if (e == cudaSuccess && !joined[k]) e = cudaEventCreateWithFlags(&joined[k], cudaEventDisableTiming);
    }
    return e;
  }

  void drop_sides() {
    for (auto &s : side)
      if (s) { cudaStreamDestroy(s); s = nullptr; }
    for (auto &e : joined)
      if (e) { cudaEventDestroy(e); e = nullptr; }
    if (forked) { cudaEventDestroy(forked); forked = nullptr; }
  }

  void drop_pin() {
    if (pin) {
      if (pin_paged) std::free(pin);
      else cudaFreeHost(pin);
    }
    pin = nullptr;
    pin_cap = 0;
    pin_paged = false;
  }

  // Staging for at least `bytes`; the calls wait for their copies before they
  // return, so what is there is free. Where no more memory can be page-locked,
  // pageable memory does: its copies are slower, and as safe.
  bool reserve_pin(size_t bytes) {
    if (bytes <= pin_cap) return true;
    drop_pin();
    if (cudaMallocHost(&pin, bytes + bytes / 4) != cudaSuccess) {
      cudaGetLastError();
      pin = std::malloc(bytes + bytes / 4);
      if (!pin) return false;
      pin_paged = true;
    }
    pin_cap = bytes + bytes / 4;
    return true;
  }

  void release() {
    drop_graphs();
    drop_pin();
    for (auto &e : ev)
      if (e) { cudaEventDestroy(e); e = nullptr; }
    if (arena) cudaFree(arena);
    arena = nullptr;
    arena_cap = 0;
  }
};
