// host_only.h — what host_only.cu and host_runtime.cpp share.
#pragma once

#include <cstdint>

extern "C" {

// A launch (test_host_launches.py mirrors it).
enum HostKind { kOther, kProject, kDiffuse, kBatchProject, kBatchDiffuse };
struct HostLaunch {
  int32_t kind, tiles, cluster, cooperative, pdl;
  int32_t n, K, D;       // tile kernels of a single grid, as what follows
  int32_t R, warps, halo, tiles_y;
  uint64_t smem, limit;  // dynamic shared memory, and the limit set for the kernel
  const void *fn, *ui, *vi, *uo, *vo;
  int32_t* err;  // the error word of bounded waits
};
// What the runtime does, and what it saw.
struct HostState {
  int64_t fail_malloc_from;  // allocations of so many bytes and more fail (0: none)
  int32_t fail_attribute;    // so many calls that set a function's attribute fail
  int32_t limits_lowered;    // times a kernel's shared-memory limit went down
};

void host_describe(const void* fn, void** args, HostLaunch* l);
// Segment k of a phase of n sweeps (segment_at): its sweeps and the messages that
// they take, and whether a rounding and an exchange come first. 0: there is none.
int32_t host_segment(int32_t projection, int32_t n, int32_t K, int32_t D, int32_t storage,
                     int32_t k, int32_t* messages, int32_t* round, int32_t* exchange);
// The launches since the last call, `cap` at most; returns their number.
int32_t host_launches(HostLaunch* out, int32_t cap);
extern HostState host_state;
}
