// Internal (non-ABI) services of a context, for the runtime translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <mutex>

#include "ig_kernels.cuh"

struct ig_ctx;

namespace igint {
int fail(ig_ctx* c, int code, const char* fmt, ...);
cudaStream_t stream(ig_ctx* c);
int device(ig_ctx* c);
std::mutex& mutex(ig_ctx* c);
int dalloc(ig_ctx* c, void** p, size_t bytes);
void dfree(ig_ctx* c, void* p, size_t bytes);
int scratch(ig_ctx* c, const char* name, size_t bytes, void** out);
int stage_h2d(ig_ctx* c, void* dst, const void* src, size_t bytes);
void add_launches(ig_ctx* c, unsigned n);
// One extension slot per context for the special_modulus objects, freed at destroy.
void*& sm_slot(ig_ctx* c);
void set_sm_destructor(ig_ctx* c, void (*fn)(ig_ctx*, void*));

// One served request resolved against the context's objects (takes the context lock):
// the parameter set's device constants (the seat's own set when it shares the database's
// ring and width), the shard's device pointers, the seat's device words, and the shard's
// store state. Returns an IG_* status; on refusal `err` holds the
// reference's message.
struct RequestView {
  ig::CrsDev crs;
  const ig::CrsDev* crs_dev;  // device copy of crs, for launches that mix parameter sets
  ig::ShardDev shard;
  const uint64_t* seat;
  uint32_t seat_rows;         // key rows of the seat (its bytes: seat_rows x n x 8)
  uint64_t p;
  bool has_store;
  char err[512];
};
int resolve_request(ig_ctx* c, uint64_t db, uint64_t store, uint64_t handle, uint32_t shard, RequestView* out);
// CTAs per query (1, 2 or 4) for a respond launch of `count` queries of width `gamma` on
// ring n with `in_flight` queries expected on the device with it (its own included): the
// forced shape, else the shape the tuned table times fastest at that many queries, else the
// fixed rule: four CTAs while twice the queries fit the pair threshold and the device runs
// that many clusters of four at once, two while they fit the threshold, else one.
int launch_ctas(ig_ctx* c, uint32_t n, uint32_t gamma, uint32_t count, uint32_t in_flight);
// The launch shape set by ig_ctx_set_launch_shape (0 when the context chooses).
int forced_ctas(ig_ctx* c);
// Device-path lanes (ig_ctx_set_lanes), for callers holding the context lock:
// lane_acquire picks the call's stream (the context stream when lanes == 1, lane -1) and
// orders the context stream after the lane's previous batch, so the lane's scratch can be
// rewritten; lane_enter, after the call's staging copies on the context stream, makes the
// lane wait for them; lane_release marks the lane's work for the next acquire and join.
int lanes(ig_ctx* c);
// A host-buffer call over lanes. begin (before the context lock) picks the call's lane and
// holds its mutex until the call ends; under the context lock, pinned() returns the lane's
// pinned landing buffer (grown to `bytes`), stream() the stream to launch on (after the
// call's staging copies: enter()), launched() marks the end of the call's device work; after
// the context lock is released, wait() blocks until that work is done. With one lane the
// call runs on the context stream.
struct HostCall {
  unsigned k = 0;
  std::unique_lock<std::mutex> lane_lock;
  cudaStream_t queued[2] = {};  // streams with copies of this call's host memory in flight
  ~HostCall() {
    for (cudaStream_t s : queued)
      if (s) cudaStreamSynchronize(s);
  }
};
// A host-buffer call's arrays: one device block (scratch of the lane) and its image in the lane's pinned buffer, so the
// small arrays cross in one copy each way (a lone query of gamma 16 131 -> 120 us, where seven copies and a memset
// went around its two launches). Arrays of COPY_DIRECT_BYTES and more are copied straight between the caller's memory
// and the device where the GPU reads pageable memory through the host's page tables (an MB in 16 us, against 50 in and
// 71 out through the pinned image; below 256 KB the image's copy is the shorter). A caller's result memory that no one
// has touched yet costs the direct copy 180 us an MB in faults that the CPU takes in 10: wait() touches it while the
// device works. 64 queries 1.455 -> 1.285 ms, 128 mixed ones 5.00 -> 4.46 ms, 256 special_modulus ones 4.43 -> 4.07 ms.
constexpr size_t COPY_DIRECT_BYTES = 256 << 10;
struct HostIO {
  // Offsets. The arrays below `down` have a place in the image: those up to `up` go to the device, those from the
  // status words on come back.
  size_t table, queries, work, seeds, bs, status, a, b, up, down;
  size_t table_bytes, query_bytes, work_bytes, seed_bytes, bs_bytes, status_bytes, a_bytes, b_bytes;
  uint8_t *dev, *pin;
};
// Lays the block out (byte counts in its order; status words are `count`) and allocates it.
int host_io_open(ig_ctx* c, HostCall& hc, HostIO& io, size_t table, size_t queries, size_t work, size_t seeds, size_t bs,
                 size_t count, size_t a, size_t b);
// Queues the inputs and zeroed status words on the call's stream, after all context-stream work so far.
int host_io_send(ig_ctx* c, HostCall& hc, HostIO& io, const void* table, const void* queries, const void* work,
                 const void* seeds, const void* bs);
// Queues the results' copies after the launches; under the context lock.
int host_io_receive(ig_ctx* c, HostCall& hc, HostIO& io);
// Waits for them (without the context lock). The status words are then at pin + status.
int host_io_wait(ig_ctx* c, HostCall& hc, HostIO& io, void* a_out, void* b_out);
// Hands the results over: called once the status words are found clean, so a refused call writes no results.
int host_io_finish(ig_ctx* c, HostCall& hc, HostIO& io, void* a_out, void* b_out);
// The lane's copy stream, ordered after nothing: copies that wait for the call's own events alone.
cudaStream_t host_call_copy_stream(ig_ctx* c, HostCall& hc);
void host_call_begin(ig_ctx* c, HostCall& hc);
int host_call_pinned(ig_ctx* c, HostCall& hc, size_t bytes, void** pin);
cudaStream_t host_call_stream(ig_ctx* c, HostCall& hc);
int host_call_enter(ig_ctx* c, HostCall& hc);
int host_call_launched(ig_ctx* c, HostCall& hc);
int host_call_wait(ig_ctx* c, HostCall& hc);
int lane_acquire(ig_ctx* c, cudaStream_t* s, int* lane);
int lane_enter(ig_ctx* c, int lane);
int lane_release(ig_ctx* c, int lane);
int sm_count(ig_ctx* c);
}  // namespace igint
