// Scratch of the kernels whose last CTA adds up the parts that the others leave (attention with few query rows, array
// reductions): partial results and arrival counters that two launches must never use at the same time.
//
// A slot belongs to one stream (by cudaStreamGetId, which tells apart the per-thread default streams behind one handle and
// never comes back for another stream), whose launches follow one another.  A launch that is captured gets a slot of its
// capture instead, one per captured stream: a replay runs on any stream, beside other graphs and beside eager work.  The graph
// holds that slot through a user object and gives it back when the graph and its executables are gone and have run; CUDA
// runs one executable once at a time.  (Two executables instantiated from ONE graph share it and must not run at once.)
//
// Slots are allocated when first asked for.  Eager ones are bounded: once kMarkFrom streams have one, an event is recorded
// behind every launch, and the kSlots + 1st stream waits on the device for the launch whose slot it takes over (never on the
// host: a device-wide wait would end a capture in progress).  Where no slot can be had, the caller takes the form of its
// operation that needs none.
#include <atomic>
#include <mutex>
#include <vector>

#include "ctx.h"

namespace ctb_internal {

namespace {

constexpr int kSlots = 96;     // eager slots of a context (1.25 MB each); torch has 32 streams per priority and the default
constexpr int kMarkFrom = 72;

struct GraphHold {  // shared by a slot and the graph that uses it
  std::atomic<int> holders{2};
  std::atomic<bool> gone{false};
};
void drop(GraphHold* h) {
  if (h && h->holders.fetch_sub(1) == 1) delete h;
}
void CUDART_CB graph_gone(void* hold) {  // may run on a thread of the driver; makes no CUDA call
  GraphHold* h = static_cast<GraphHold*>(hold);
  h->gone.store(true);
  drop(h);
}

// For the calls below that a capture in another thread would otherwise refuse (and that would end that capture).
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
struct OnDevice {
  int before = -1;
  explicit OnDevice(int device) {
    if (cudaGetDevice(&before) == cudaSuccess && before != device) cudaSetDevice(device);
    else before = -1;
  }
  ~OnDevice() {
    if (before >= 0) cudaSetDevice(before);
  }
};

}  // namespace

struct ScratchSlot {
  void* memory = nullptr;  // kStreamScratchBytes, then kTickets counters
  bool owned = false;      // by (stream, capture); capture 0: eager launches
  unsigned long long stream = 0, capture = 0;
  int users = 0;           // calls that have it and have not launched yet
  cudaEvent_t event = nullptr;
  bool marked = false;     // the event lies behind the last launch
  unsigned long long last = 0;  // ScratchPool::calls of it
  GraphHold* hold = nullptr;
};
struct ScratchPool {
  int device;
  std::mutex lock;
  std::vector<ScratchSlot*> slots;
  unsigned long long calls = 0;
};

ScratchPool* scratch_pool_create(int device) {
  ScratchPool* p = new ScratchPool();
  p->device = device;
  return p;
}
void scratch_pool_destroy(ScratchPool* p) {
  if (!p) return;
  for (ScratchSlot* s : p->slots) {
    if (s->memory) cudaFree(s->memory);
    if (s->event) cudaEventDestroy(s->event);
    drop(s->hold);
    delete s;
  }
  delete p;
}

namespace {

bool allocate(ScratchPool* p, ScratchSlot* s) {
  OnDevice on(p->device);
  RelaxedCapture relaxed;
  constexpr size_t ticket_bytes = kTickets * sizeof(unsigned);
  cudaStream_t st = nullptr;
  cudaError_t e = cudaMalloc(&s->memory, kStreamScratchBytes + ticket_bytes);
  if (e != cudaSuccess) s->memory = nullptr;
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMemsetAsync(static_cast<char*>(s->memory) + kStreamScratchBytes, 0, ticket_bytes, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->event, cudaEventDisableTiming);
  if (st) cudaStreamDestroy(st);
  if (e == cudaSuccess) return true;
  if (s->memory) cudaFree(s->memory);
  s->memory = nullptr;
  (void)cudaGetLastError();
  return false;
}

// A slot for `stream`, for eager launches or for a capture.
ScratchSlot* free_slot(ScratchPool* p, cudaStream_t stream, bool captured) {
  int held = 0;  // eager slots
  ScratchSlot *found = nullptr, *oldest = nullptr;
  for (ScratchSlot* s : p->slots) {
    if (s->hold && s->hold->gone.load() && !s->users) {  // the graph is gone and so are its runs
      drop(s->hold);
      s->hold = nullptr;
      s->owned = false;
    }
    if (!s->owned) found = s;
    else if (!s->hold) {
      ++held;
      if (s->marked && !s->users && (!oldest || s->last < oldest->last)) oldest = s;
    }
  }
  if (!captured && held >= kSlots) {
    if (!oldest) return nullptr;
    if (cudaStreamWaitEvent(stream, oldest->event, 0) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    return oldest;
  }
  if (!found) {
    ScratchSlot* s = new ScratchSlot();
    if (!allocate(p, s)) {
      delete s;
      return nullptr;
    }
    p->slots.push_back(s);
    found = s;
  }
  return found;
}

}  // namespace

StreamScratch::StreamScratch(ctb_ctx* ctx, cudaStream_t stream) : pool_(ctx->scratch), stream_(stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long capture = 0, id = 0;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo(stream, &status, &capture, &graph) != cudaSuccess) {
    (void)cudaGetLastError();
    return;
  }
  if (status == cudaStreamCaptureStatusInvalidated) return;
  const bool captured = status == cudaStreamCaptureStatusActive;
  if (captured) {  // asking a capturing stream for its id ends the capture; its handle is its own until the capture ends
    static thread_local char mine;
    id = (unsigned long long)(uintptr_t)(stream == cudaStreamPerThread ? static_cast<void*>(&mine) : static_cast<void*>(stream));
  } else {
    capture = 0;
    if (cudaStreamGetId(stream, &id) != cudaSuccess) {
      (void)cudaGetLastError();
      return;
    }
  }
  std::lock_guard<std::mutex> guard(pool_->lock);
  int held = 0;
  for (ScratchSlot* s : pool_->slots) {
    held += s->owned && !s->hold;
    if (s->owned && s->stream == id && s->capture == capture && (s->hold != nullptr) == captured) slot_ = s;
  }
  if (!slot_) {
    ScratchSlot* s = free_slot(pool_, stream, captured);
    if (!s) return;
    if (captured) {
      GraphHold* hold = new GraphHold();
      cudaUserObject_t object = nullptr;
      cudaError_t e = cudaUserObjectCreate(&object, hold, graph_gone, 1, cudaUserObjectNoDestructorSync);
      if (e != cudaSuccess) {
        delete hold;
        (void)cudaGetLastError();
        return;
      }
      s->hold = hold;
      s->capture = capture;
      s->stream = id;
      s->owned = true;
      e = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
      if (e != cudaSuccess) {  // nothing of this slot is in the graph: the destructor below frees it again
        (void)cudaGetLastError();
        cudaUserObjectRelease(object, 1);
        return;
      }
    } else {
      s->capture = 0;
      s->stream = id;
      s->owned = true;
    }
    slot_ = s;
  }
  ++slot_->users;
  slot_->last = ++pool_->calls;
  slot_->marked = false;
  mark_ = !captured && held >= kMarkFrom;
  data = static_cast<float*>(slot_->memory);
  tickets = reinterpret_cast<unsigned*>(static_cast<char*>(slot_->memory) + kStreamScratchBytes);
}

StreamScratch::~StreamScratch() {
  if (!slot_) return;
  std::lock_guard<std::mutex> guard(pool_->lock);
  --slot_->users;
  if (mark_) slot_->marked = cudaEventRecord(slot_->event, stream_) == cudaSuccess;
}

}  // namespace ctb_internal
