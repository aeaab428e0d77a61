// Execution-graph interpreter for devtype "gpu".
//
// Same instruction set and callable ABI as the reference's SequentialInterpreter
// (src/execution.cpp:19-58, 247-292): LoadArgument, Alloc (re-allocates only when the shape changes),
// BuildTup, ReturnByRef, ReturnByVal. What differs is how device work is issued:
//
//   * every device instruction enqueues kernels on the runtime's CUDA stream and returns at once;
//   * cross-device copies (Transport) are asynchronous; a host instruction that reads array data
//     waits for the stream only when a device->host copy is outstanding. The small arrays that a span takes from
//     the host, the call's arguments that already are on the device among them, are brought to their buffers by ONE
//     kernel at the span's start, what it hands to the host (the function's results at the end) leaves by one kernel
//     at its end; both are nodes of the span's graph (host_copy.cu);
//   * the instruction list is cut into spans after device->host copies and at every non-capturable instruction. Once a
//     span has run twice with identical buffer addresses (steady state: no allocation happens any
//     more), its device instructions are captured into a CUDA graph and later runs replay the graph
//     with one launch. The replay is used only while a key over all buffer addresses and small host
//     operands that the span's device instructions see is unchanged, so a shape change, a set_value()
//     on a shared variable or a changed host scalar falls back to eager issue and re-capture;
//   * a run whose arguments have the buffers, shapes and small host values of the run before it, with no
//     shared variable replaced in between and no allocation in the run before, is a steady run: its host
//     bookkeeping instructions (Alloc, BuildTup, views, shape arithmetic) would reproduce what the storage
//     already holds, so they are skipped, and a span's graph is launched without recomputing its key. Host
//     instructions that compute on array data still run; from the first one whose result differs from the run
//     before, the rest of the run takes the full path again. Without this the host walks the whole instruction
//     list before each launch: thousands of instructions for an unrolled recurrent network, more time than
//     the device needs for them.
#include "host_copy.h"
#include "runtime.h"
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

using namespace cgtb;

namespace {

enum Kind { kLoadArgument, kAlloc, kBuildTup, kReturnByRef, kReturnByVal };
enum Klass { kMeta, kHostData, kDevice, kBarrier, kUpload, kDownload };

struct Loc {
  long idx;
  int dev;
};

struct Instr {
  Kind kind;
  std::string repr;
  int flags = 0;
  std::vector<Loc> reads;
  Loc write{0, 0};
  int arg_index = 0;
  cgtDtype dtype = cgt_f4;
  void* fptr = nullptr;
  void* closure = nullptr;
  Klass klass = kMeta;
  bool fired = false;
  bool arg_view = false;  // host bookkeeping on (a view of) an argument: fired in steady runs too
  bool from_argument = false;  // kUpload: the source is (a view of) an argument, which nothing in the call writes
  ScratchOwner scratch;
  void* stage = nullptr;  // kUpload: pinned copy of the host operand, read by the span's copy kernel
  long stage_cap = 0;
  double prof_ms = 0;
  long prof_count = 0;
};

struct Span {
  int begin = 0, end = 0;  // [begin, end)
  bool barrier = false;    // single Transport / non-capturable instruction
  int n_device = 0;        // device instructions, uploads and downloads
  bool has_hostdata = false;
  bool reads_download = false;  // looks at a value that an earlier span copied to the host
  bool collects = false;        // the last span with device work: it also copies the function's results out
  std::vector<int> steady_host;  // instructions of pass 1 that a steady run fires
  CopyJobs uploads;              // this run's uploads, in program order
  CopyJobs captured_uploads;     // what the copy node of `exec` was last told
  cudaGraphNode_t upload_node = nullptr;
  cudaGraph_t graph = nullptr;   // kept: `upload_node` belongs to it
  cudaGraphExec_t exec = nullptr;
  uint64_t exec_key = 0, last_key = 0;
  bool have_last = false, capture_failed = false;
  long graph_kernels = 0;
};

}  // namespace

struct cgtbGraph {
  long n_args, n_locs;
  std::vector<Instr> instrs;
};

struct cgtbInterp {
  cgtbGraph* g;
  std::vector<Loc> outs;
  std::vector<IRC<cgtObject>> storage;
  cgtTuple* args = nullptr;
  int flags = 0;
  std::vector<Span> spans;
  bool host_pending = false;  // a device->host copy has been queued and not yet waited for
  long runs = 0, last_launches = 0, last_graph_launches = 0, captured = 0;
  long mallocs_at_run_start = 0;
  bool prev_run_allocated = true;
  void (*before_sync)(void*) = nullptr;  // called once per run after all device work has been queued
  void* before_sync_ctx = nullptr;
  // steady-run detection
  std::vector<uint64_t> arg_sig;        // signature of the previous run's arguments
  long state_version_seen = -1;
  bool steady = false;                  // this run repeats the previous one as far as host bookkeeping goes
  bool host_dirty = false;              // a host data instruction of this run produced a new value
  bool prev_run_ok = false;
  uint64_t args_read_in_place = ~0ull;  // arguments whose device buffer a captured instruction reads directly
  std::vector<char> downloaded;         // locations that a device->host copy writes
  std::vector<long> memory_of;          // per location: the location whose memory it is or views
  bool by_value_state = false;          // a host value that an instruction takes is overwritten later in the call
  char* out_stage = nullptr;            // pinned block that holds the device results of the last run
  long out_stage_cap = 0;
  std::vector<void*> out_host;          // per result: its bytes in host memory, or null (not an array on the device)
  std::vector<long> out_offset;
  std::vector<char> out_is_argument;    // per result: it is, or views, one of the call's arguments
  std::vector<cgtArray*> out_array;     // the array that was copied to out_host
  long last_host_ns = 0;                // host time of the last run up to the final wait for the stream
  long steady_runs = 0;
};

static std::atomic<long> g_state_version{0};
// Called by the host side whenever a shared variable's array is replaced (a set_value with a new shape).
CGTB_API void cgtb_state_version_bump(void) { g_state_version.fetch_add(1, std::memory_order_relaxed); }

// ------------------------------------------------------------------------------------------------
// graph construction
// ------------------------------------------------------------------------------------------------
CGTB_API cgtbGraph* cgtb_graph_new(long n_args, long n_locs) {
  cgtbGraph* g = new cgtbGraph();
  g->n_args = n_args;
  g->n_locs = n_locs;
  return g;
}
CGTB_API void cgtb_graph_free(cgtbGraph* g) {
  if (!g) return;
  for (auto& in : g->instrs) {
    free_scratch_owner(&in.scratch);
    if (in.stage) cgtb_free(cgtbCPU, in.stage);
  }
  delete g;
}

static int check_loc(cgtbGraph* g, long idx) {
  if (idx < 0 || idx >= g->n_locs) return fail("memory location %ld out of range (n_locs %ld)", idx, g->n_locs);
  return 0;
}

CGTB_API int cgtb_graph_add_load_argument(cgtbGraph* g, const char* repr, int arg_index, long wloc, int wdev) {
  if (check_loc(g, wloc)) return 1;
  if (arg_index < 0 || arg_index >= g->n_args) return fail("LoadArgument: argument index %d out of range", arg_index);
  Instr in;
  in.kind = kLoadArgument;
  in.repr = repr ? repr : "";
  in.arg_index = arg_index;
  in.write = {wloc, wdev};
  g->instrs.push_back(in);
  return 0;
}
CGTB_API int cgtb_graph_add_alloc(cgtbGraph* g, const char* repr, int dtype, int n_shape, const long* shape_locs, long wloc,
                                  int wdev) {
  if (check_loc(g, wloc)) return 1;
  if (n_shape > CGTB_MAX_NDIM) return fail("Alloc: ndim %d too large", n_shape);
  Instr in;
  in.kind = kAlloc;
  in.repr = repr ? repr : "";
  in.dtype = (cgtDtype)dtype;
  for (int i = 0; i < n_shape; ++i) {
    if (check_loc(g, shape_locs[i])) return 1;
    in.reads.push_back({shape_locs[i], cgtbCPU});
  }
  in.write = {wloc, wdev};
  g->instrs.push_back(in);
  return 0;
}
CGTB_API int cgtb_graph_add_build_tup(cgtbGraph* g, const char* repr, int n, const long* read_locs, long wloc, int wdev) {
  if (check_loc(g, wloc)) return 1;
  Instr in;
  in.kind = kBuildTup;
  in.repr = repr ? repr : "";
  for (int i = 0; i < n; ++i) {
    if (check_loc(g, read_locs[i])) return 1;
    in.reads.push_back({read_locs[i], wdev});
  }
  in.write = {wloc, wdev};
  g->instrs.push_back(in);
  return 0;
}
static int add_return(cgtbGraph* g, Kind kind, const char* repr, int n, const long* read_locs, const int* read_devs, long wloc,
                      int wdev, void* fptr, void* closure, int flags) {
  if (check_loc(g, wloc)) return 1;
  if (!fptr) return fail("%s: null function pointer", repr ? repr : "Return");
  Instr in;
  in.kind = kind;
  in.repr = repr ? repr : "";
  in.flags = flags;
  for (int i = 0; i < n; ++i) {
    if (check_loc(g, read_locs[i])) return 1;
    in.reads.push_back({read_locs[i], read_devs ? read_devs[i] : wdev});
  }
  in.write = {wloc, wdev};
  in.fptr = fptr;
  in.closure = closure;
  g->instrs.push_back(in);
  return 0;
}
CGTB_API int cgtb_graph_add_return_byref(cgtbGraph* g, const char* repr, int n, const long* read_locs, const int* read_devs,
                                         long wloc, int wdev, void* fptr, void* closure, int flags) {
  return add_return(g, kReturnByRef, repr, n, read_locs, read_devs, wloc, wdev, fptr, closure, flags);
}
CGTB_API int cgtb_graph_add_return_byval(cgtbGraph* g, const char* repr, int n, const long* read_locs, const int* read_devs,
                                         long wloc, int wdev, void* fptr, void* closure, int flags) {
  return add_return(g, kReturnByVal, repr, n, read_locs, read_devs, wloc, wdev, fptr, closure, flags);
}

// ------------------------------------------------------------------------------------------------
// interpreter
// ------------------------------------------------------------------------------------------------
// Cut the instruction list into spans at every barrier instruction. A fire-once barrier (a constant's
// transport) that has already fired no longer separates its neighbours, so after the first run the
// whole step usually collapses into one span per real transfer.
static void drop_exec(Span& s) {
  if (s.exec) cudaGraphExecDestroy(s.exec);
  if (s.graph) cudaGraphDestroy(s.graph);
  s.exec = nullptr;
  s.graph = nullptr;
  s.upload_node = nullptr;
}
static void build_spans(cgtbInterp* it) {
  for (auto& s : it->spans) drop_exec(s);
  it->spans.clear();
  auto& instrs = it->g->instrs;
  int n = (int)instrs.size();
  auto is_barrier = [&](int k) {
    Instr& in = instrs[(size_t)k];
    return in.klass == kBarrier && !((in.flags & CGTB_INSTR_ONCE) && in.fired);
  };
  auto reads_downloaded = [&](const Instr& in) {
    for (auto& r : in.reads)
      if (it->downloaded[(size_t)r.idx]) return true;
    return false;
  };
  it->downloaded.assign((size_t)it->g->n_locs, 0);
  int i = 0;
  while (i < n) {
    Span s;
    s.begin = i;
    s.uploads.n = s.captured_uploads.n = 0;
    if (is_barrier(i)) {
      s.barrier = true;
      s.end = i + 1;
    } else {
      int j = i, n_uploads = 0, n_downloads = 0;
      std::vector<char> fresh((size_t)it->g->n_locs, 0);  // copied to the host by this span
      std::vector<char> taken((size_t)it->g->n_locs, 0);  // host memory that a device instruction reads when it is issued
      while (j < n && !is_barrier(j)) {
        Instr& in = instrs[(size_t)j];
        if (n_downloads) {
          // only bookkeeping and further downloads may follow a download in its span
          bool cut = in.klass != kMeta && in.klass != kDownload;
          for (auto& r : in.reads) cut = cut || fresh[(size_t)r.idx];
          if (cut || (in.klass == kDownload && n_downloads == kMaxCopyJobs)) break;
        }
        if (in.klass == kUpload && n_uploads == kMaxCopyJobs) break;
        // device instructions are issued after the span's host instructions: one that overwrites what they take by
        // value (the start of a slice that the call moves on) has to wait for the next span
        if (in.klass == kHostData && taken[(size_t)it->memory_of[(size_t)in.write.idx]]) break;
        if (in.klass == kDevice)
          for (auto& r : in.reads)
            if (r.dev == cgtbCPU) taken[(size_t)it->memory_of[(size_t)r.idx]] = 1;
        if (in.klass == kDownload) {
          ++n_downloads;
          fresh[(size_t)in.write.idx] = 1;
        }
        if (in.klass == kUpload) ++n_uploads;
        if (in.klass == kDevice || in.klass == kUpload || in.klass == kDownload) s.n_device++;
        if (in.klass == kHostData) s.has_hostdata = true;
        if (in.klass != kDevice && reads_downloaded(in)) s.reads_download = true;
        if (in.klass == kHostData || in.klass == kUpload || (in.klass == kMeta && in.arg_view)) s.steady_host.push_back(j);
        ++j;
      }
      for (size_t l = 0; l < fresh.size(); ++l) it->downloaded[l] |= fresh[l];
      s.end = j;
    }
    it->spans.push_back(s);
    i = s.end;
  }
  // results are collected by the last span that has device work, unless a non-capturable instruction comes later
  for (size_t k = it->spans.size(); k-- > 0;) {
    if (it->spans[k].barrier) break;
    if (it->spans[k].n_device > 0) { it->spans[k].collects = true; break; }
  }
}

CGTB_API cgtbInterp* cgtb_interp_new(cgtbGraph* g, int n_out, const long* out_locs, int flags) {
  if (!g) { fail("cgtb_interp_new: null graph"); return nullptr; }
  cgtbInterp* it = new cgtbInterp();
  it->g = g;
  it->flags = flags;
  it->storage.resize((size_t)g->n_locs);
  for (int i = 0; i < n_out; ++i) {
    if (check_loc(g, out_locs[i])) { delete it; return nullptr; }
    it->outs.push_back({out_locs[i], 0});
  }
  bool any_device = false;
  for (auto& in : g->instrs) {
    const bool plain_copy = (in.flags & CGTB_INSTR_TRANSPORT) && !(in.flags & (CGTB_INSTR_NOCAPTURE | CGTB_INSTR_ONCE)) &&
                            in.kind == kReturnByRef && in.reads.size() == 1 && !(flags & CGTB_INTERP_PROFILE);
    if (in.kind == kLoadArgument || in.kind == kAlloc || in.kind == kBuildTup) in.klass = kMeta;
    else if (plain_copy && in.reads[0].dev == cgtbCPU && in.write.dev == cgtbGPU) in.klass = kUpload;
    else if (plain_copy && in.reads[0].dev == cgtbGPU && in.write.dev == cgtbCPU) in.klass = kDownload;
    else if (in.flags & (CGTB_INSTR_TRANSPORT | CGTB_INSTR_NOCAPTURE)) in.klass = kBarrier;
    else if (in.flags & CGTB_INSTR_QUICK) in.klass = kMeta;
    else if (in.write.dev == cgtbGPU) in.klass = (in.kind == kReturnByRef) ? kDevice : kBarrier;
    else in.klass = kHostData;
    if (in.write.dev == cgtbGPU) any_device = true;
    for (auto& r : in.reads) if (r.dev == cgtbGPU) any_device = true;
  }
  if (any_device && !require_runtime("cgtb_interp_new")) { delete it; return nullptr; }
  {
    // Bookkeeping instructions that see an argument object directly or through other bookkeeping (views, tuples,
    // sizes, allocations shaped by them) cannot be skipped in steady runs: the caller passes new objects every time.
    // from_arg[loc]: the arguments (bit i = argument i, the last bit stands for all beyond 62) that location loc holds
    // or views. An argument that a device instruction reads in place must keep its buffer for a run to be steady (the
    // captured graphs hold that address); one that only copies (Transport, a barrier) and bookkeeping look at may
    // move: a batch handed over in alternating staging buffers is still a steady run.
    std::vector<uint64_t> from_arg((size_t)g->n_locs, 0);
    uint64_t in_place = 0;
    for (auto& in : g->instrs) {
      if (in.klass == kDevice) {
        for (auto& r : in.reads) in_place |= from_arg[(size_t)r.idx];
        in_place |= from_arg[(size_t)in.write.idx];
        continue;
      }
      if (in.klass == kUpload) in.from_argument = from_arg[(size_t)in.reads[0].idx] != 0;
      if (in.klass != kMeta) continue;
      uint64_t dep = in.kind == kLoadArgument ? (1ull << (in.arg_index < 63 ? in.arg_index : 63)) : 0;
      for (auto& r : in.reads) dep |= from_arg[(size_t)r.idx];
      in.arg_view = dep != 0;
      if (dep) from_arg[(size_t)in.write.idx] |= dep;
    }
    it->args_read_in_place = in_place;
    it->memory_of.resize((size_t)g->n_locs);
    for (long l = 0; l < g->n_locs; ++l) it->memory_of[(size_t)l] = l;
    std::vector<char> taken((size_t)g->n_locs, 0);
    for (auto& in : g->instrs) {
      if (in.kind == kReturnByVal && in.klass == kMeta && !in.reads.empty()) it->memory_of[(size_t)in.write.idx] = it->memory_of[(size_t)in.reads[0].idx];
      if (in.klass == kHostData) it->by_value_state = it->by_value_state || taken[(size_t)it->memory_of[(size_t)in.write.idx]];
      if (in.klass == kDevice || in.kind == kAlloc)
        for (auto& r : in.reads)
          if (r.dev == cgtbCPU) taken[(size_t)it->memory_of[(size_t)r.idx]] = 1;
    }
    for (auto& o : it->outs) it->out_is_argument.push_back(from_arg[(size_t)o.idx] != 0);
  }
  build_spans(it);
  return it;
}

CGTB_API void cgtb_interp_free(cgtbInterp* it) {
  if (!it) return;
  if (rt().ready) cudaStreamSynchronize(rt().stream);
  for (auto& s : it->spans) drop_exec(s);
  if (it->out_stage) cgtb_free(cgtbCPU, it->out_stage);
  delete it;
}

static inline cgtObject* get(cgtbInterp* it, const Loc& l) { return it->storage[(size_t)l.idx].get(); }

static int fire(cgtbInterp* it, Instr& in) {
  switch (in.kind) {
    case kLoadArgument: {
      if (in.arg_index >= it->args->len) return fail("LoadArgument: missing argument %d", in.arg_index);
      it->storage[(size_t)in.write.idx] = it->args->members[in.arg_index].get();
      return 0;
    }
    case kAlloc: {
      int nd = (int)in.reads.size();
      long shape[CGTB_MAX_NDIM];
      for (int i = 0; i < nd; ++i) {
        cgtArray* sv = (cgtArray*)get(it, in.reads[(size_t)i]);
        if (!sv || sv->kind() != cgtObject::ArrayKind || sv->dtype() != cgt_i8 || sv->devtype() != cgtCPU)
          return fail("Alloc (%s): shape component %d is not a host int64 scalar", in.repr.c_str(), i);
        shape[i] = sv->at<long>(0);
        if (shape[i] < 0) return fail("Alloc (%s): negative extent", in.repr.c_str());
      }
      cgtObject* cur0 = get(it, in.write);
      cgtArray* cur = (cur0 && cur0->kind() == cgtObject::ArrayKind) ? (cgtArray*)cur0 : nullptr;
      bool same = cur && cur->ownsdata() && cur->ndim() == nd && cur->dtype() == in.dtype &&
                  (int)cur->devtype() == in.write.dev;
      for (int i = 0; same && i < nd; ++i) same = cur->shape()[i] == shape[i];
      if (!same) {
        cgtArray* a = new cgtArray(nd, shape, in.dtype, (cgtDevtype)in.write.dev);
        if (!a->data()) { a->Retain(); a->Release(); return 1; }
        it->storage[(size_t)in.write.idx] = a;
      }
      return 0;
    }
    case kBuildTup: {
      // rebuilt only when a member object changed, so a steady-state run allocates nothing
      cgtObject* cur0 = get(it, in.write);
      int n = (int)in.reads.size();
      if (cur0 && cur0->kind() == cgtObject::TupleKind && ((cgtTuple*)cur0)->len == n) {
        cgtTuple* t = (cgtTuple*)cur0;
        bool same = true;
        for (int i = 0; same && i < n; ++i) same = t->getitem(i) == get(it, in.reads[(size_t)i]);
        if (same) return 0;
      }
      cgtTuple* t = new cgtTuple(n);
      for (int i = 0; i < n; ++i) t->setitem(i, get(it, in.reads[(size_t)i]));
      it->storage[(size_t)in.write.idx] = t;
      return 0;
    }
    case kReturnByRef:
    case kReturnByVal: {
      int n = (int)in.reads.size();
      cgtObject* reads_small[16];
      std::vector<cgtObject*> reads_big;
      cgtObject** reads = reads_small;
      if (n > 16) { reads_big.resize((size_t)n); reads = reads_big.data(); }
      for (int i = 0; i < n; ++i) {
        reads[i] = get(it, in.reads[(size_t)i]);
        if (!reads[i]) return fail("%s: input %d was never produced", in.repr.c_str(), i);
      }
      set_scratch_owner(&in.scratch);
      if (in.kind == kReturnByRef) {
        cgtObject* w = get(it, in.write);
        if (!w) { set_scratch_owner(nullptr); return fail("%s: output was never allocated", in.repr.c_str()); }
        ((cgtByRefFun)in.fptr)(in.closure, reads, w);
      } else {
        cgtObject* r = ((cgtByValFun)in.fptr)(in.closure, reads);
        if (r) it->storage[(size_t)in.write.idx] = r;
        else if (cgt_get_status() == cgtStatusOK) fail("%s: callable returned NULL", in.repr.c_str());
      }
      set_scratch_owner(nullptr);
      if (cgt_get_status() != cgtStatusOK) {
        std::string msg = cgtb_last_error();
        return fail("%s: %s", in.repr.c_str(), msg.c_str());
      }
      return 0;
    }
  }
  return 0;
}

static inline uint64_t mix(uint64_t h, uint64_t v) {
  h ^= v + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2);
  return h;
}
static uint64_t key_of_object(uint64_t h, cgtObject* o, int dev) {
  if (!o) return mix(h, 0);
  if (o->kind() == cgtObject::ArrayKind) {
    cgtArray* a = (cgtArray*)o;
    // a small host operand counts by its bytes alone: kernels receive its value at launch, and the object that holds it
    // (a Size, a host scalar) may be a new one on every run
    const bool by_value = a->devtype() == cgtCPU && a->nbytes() <= 64 && a->data();
    if (!by_value) h = mix(h, (uint64_t)(uintptr_t)a->data());
    // a captured graph bakes shape-derived launch parameters into its nodes, and the pool can hand the same block
    // to a differently shaped array of equal size: the extents and the dtype are part of the key
    h = mix(h, ((uint64_t)a->ndim() << 8) | (uint64_t)a->dtype());
    for (int d = 0; d < a->ndim(); ++d) h = mix(h, (uint64_t)a->shape()[d]);
    if (by_value) {
      uint64_t buf[8] = {0};
      memcpy(buf, a->data(), (size_t)a->nbytes());
      for (int i = 0; i < 8; ++i) h = mix(h, buf[i]);
    }
  } else {
    cgtTuple* t = (cgtTuple*)o;
    for (int i = 0; i < t->len; ++i) h = key_of_object(h, t->getitem(i), dev);
  }
  return h;
}
static void* array_data(cgtObject* o) { return o && o->kind() == cgtObject::ArrayKind ? ((cgtArray*)o)->data() : nullptr; }
static uint64_t span_key(cgtbInterp* it, const Span& s) {
  uint64_t h = 1469598103934665603ull;
  for (int i = s.begin; i < s.end; ++i) {
    Instr& in = it->g->instrs[(size_t)i];
    // an upload's source is not part of the key: its copy node is told the new address before each launch
    if (in.klass == kUpload) h = key_of_object(h, get(it, in.write), in.write.dev);
    if (in.klass == kDownload) h = mix(key_of_object(h, get(it, in.reads[0]), in.reads[0].dev), (uint64_t)(uintptr_t)array_data(get(it, in.write)));
    if (in.klass != kDevice) continue;
    for (auto& r : in.reads) h = key_of_object(h, get(it, r), r.dev);
    h = key_of_object(h, get(it, in.write), in.write.dev);
  }
  if (s.collects) {
    h = mix(h, (uint64_t)(uintptr_t)it->out_stage);
    for (size_t i = 0; i < it->outs.size(); ++i) {
      cgtObject* obj = get(it, it->outs[i]);
      if (obj && obj->kind() == cgtObject::ArrayKind && ((cgtArray*)obj)->devtype() == cgtGPU && !it->out_is_argument[i])
        h = key_of_object(h, obj, cgtbGPU);
    }
  }
  return h;
}

static int fire_profiled(cgtbInterp* it, Instr& in) {
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, rt().stream);
  int rc = fire(it, in);
  cudaEventRecord(e1, rt().stream);
  cudaEventSynchronize(e1);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  in.prof_ms += ms;
  in.prof_count += 1;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return rc;
}

// ------------------------------------------------------------------------------------------------
// Capture with several streams. Stream capture of a single stream yields a linear chain of kernel nodes; the
// step's data flow is wider than that (filter gradients next to the data-gradient chain, eight parameter updates,
// the operand preparations of a layer). During capture every device instruction is given the address ranges it
// reads and writes (its operands' device buffers, views and in-place results included, since ranges are
// compared, not locations); an instruction depends on the earlier ones whose writes overlap what it touches or
// whose reads overlap what it writes. It is issued on one of a few side streams that join the capture through
// events: the stream of a dependency if that dependency is the stream's last instruction, otherwise the stream
// idle for longest, after waiting for the events of its dependencies. The graph then holds the true edges and
// independent kernels run side by side. Arithmetic is untouched: the same kernels on the same buffers.
// ------------------------------------------------------------------------------------------------
struct AddrRange { uintptr_t lo, hi; };

static void collect_ranges(cgtObject* o, std::vector<AddrRange>& out) {
  if (!o) return;
  if (o->kind() == cgtObject::ArrayKind) {
    cgtArray* a = (cgtArray*)o;
    if (a->devtype() == cgtGPU && a->data() && a->nbytes() > 0) out.push_back({(uintptr_t)a->data(), (uintptr_t)a->data() + (uintptr_t)a->nbytes()});
  } else {
    cgtTuple* t = (cgtTuple*)o;
    for (int i = 0; i < t->len; ++i) collect_ranges(t->getitem(i), out);
  }
}
static bool overlap(const std::vector<AddrRange>& a, const std::vector<AddrRange>& b) {
  for (const AddrRange& x : a)
    for (const AddrRange& y : b)
      if (x.lo < y.hi && y.lo < x.hi) return true;
  return false;
}

constexpr int kMaxGraphStreams = 8;
static cudaStream_t g_side_streams[kMaxGraphStreams];
static int g_n_side_streams = 0;
static std::vector<cudaEvent_t> g_capture_events;

static int graph_streams() {
  static int n = -1;
  if (n < 0) {
    // default 1 (a linear chain): measured on the five benchmark configurations, two to six streams changed the step
    // time by less than the run-to-run spread, because the large kernels fill every SM and the small ones form
    // dependent chains; the option stays for graphs with wide, independent branches
    const char* e = getenv("CGTB_GRAPH_STREAMS");
    n = e ? atoi(e) : 1;
    if (n < 1) n = 1;
    if (n > kMaxGraphStreams) n = kMaxGraphStreams;
  }
  return n;
}
static cudaEvent_t capture_event(size_t i) {
  while (g_capture_events.size() <= i) {
    cudaEvent_t e = nullptr;
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return nullptr;
    g_capture_events.push_back(e);
  }
  return g_capture_events[i];
}

// Fires the device instructions of span s inside the running capture of `origin`, spread over side streams.
static int fire_span_multistream(cgtbInterp* it, Span& s, cudaStream_t origin) {
  auto& instrs = it->g->instrs;
  const int NS = graph_streams();
  while (g_n_side_streams < NS) {
    if (cudaStreamCreateWithFlags(&g_side_streams[g_n_side_streams], cudaStreamNonBlocking) != cudaSuccess) return fail("cudaStreamCreate failed");
    ++g_n_side_streams;
  }
  struct Node { int instr; int stream; std::vector<AddrRange> rd, wr; bool opaque; };
  std::vector<Node> nodes;
  std::vector<int> last_on_stream((size_t)NS, -1);   // node index of the last instruction issued on each stream
  std::vector<long> last_use((size_t)NS, -1);
  std::vector<bool> joined((size_t)NS, false);
  // event 0: the fork point on the origin stream
  cudaEvent_t fork = capture_event(0);
  if (!fork) return fail("cudaEventCreate failed");
  CGTB_CUDA_TRY(cudaEventRecord(fork, origin));
  int rc = 0;
  long tick = 0;
  for (int i = s.begin; i < s.end && !rc; ++i) {
    Instr& in = instrs[(size_t)i];
    if (in.klass != kDevice) continue;
    if ((in.flags & CGTB_INSTR_ONCE) && in.fired) continue;
    Node nd;
    nd.instr = i;
    nd.opaque = (in.kind != kReturnByRef);   // a device instruction that creates its own result: ordered against everything
    for (auto& r : in.reads) collect_ranges(get(it, r), nd.rd);
    if (!nd.opaque) collect_ranges(get(it, in.write), nd.wr);
    // dependencies: the latest conflicting instruction per stream is enough (a stream is ordered)
    std::vector<int> dep_of_stream((size_t)NS, -1);
    for (int j = (int)nodes.size() - 1; j >= 0; --j) {
      const Node& e = nodes[(size_t)j];
      if (dep_of_stream[(size_t)e.stream] >= 0) continue;
      if (nd.opaque || e.opaque || overlap(e.wr, nd.rd) || overlap(e.wr, nd.wr) || overlap(e.rd, nd.wr)) dep_of_stream[(size_t)e.stream] = j;
    }
    // stream choice
    int chosen = -1;
    for (int st = 0; st < NS; ++st)
      if (dep_of_stream[(size_t)st] >= 0 && dep_of_stream[(size_t)st] == last_on_stream[(size_t)st] && (chosen < 0 || dep_of_stream[(size_t)st] > dep_of_stream[(size_t)chosen])) chosen = st;
    if (chosen < 0) {
      for (int st = 0; st < NS; ++st)
        if (chosen < 0 || last_use[(size_t)st] < last_use[(size_t)chosen]) chosen = st;
    }
    cudaStream_t cs = g_side_streams[chosen];
    if (!joined[(size_t)chosen]) {
      CGTB_CUDA_TRY(cudaStreamWaitEvent(cs, fork, 0));
      joined[(size_t)chosen] = true;
    }
    for (int st = 0; st < NS; ++st) {
      const int d = dep_of_stream[(size_t)st];
      if (d < 0 || st == chosen) continue;
      cudaEvent_t ev = capture_event((size_t)d + 1);
      if (!ev) return fail("cudaEventCreate failed");
      CGTB_CUDA_TRY(cudaStreamWaitEvent(cs, ev, 0));
    }
    nd.stream = chosen;
    cudaStream_t saved = rt().stream;
    rt().stream = cs;
    rc = fire(it, in);
    rt().stream = saved;
    if (rc) break;
    cudaEvent_t mine = capture_event(nodes.size() + 1);
    if (!mine) return fail("cudaEventCreate failed");
    CGTB_CUDA_TRY(cudaEventRecord(mine, cs));
    last_on_stream[(size_t)chosen] = (int)nodes.size();
    last_use[(size_t)chosen] = tick++;
    nodes.push_back(std::move(nd));
  }
  // join every side stream back into the origin
  for (int st = 0; st < NS; ++st) {
    if (!joined[(size_t)st]) continue;
    const int l = last_on_stream[(size_t)st];
    if (l >= 0) CGTB_CUDA_TRY(cudaStreamWaitEvent(origin, capture_event((size_t)l + 1), 0));
    else {
      cudaEvent_t ev = capture_event(nodes.size() + 2 + (size_t)st);
      CGTB_CUDA_TRY(cudaEventRecord(ev, g_side_streams[st]));
      CGTB_CUDA_TRY(cudaStreamWaitEvent(origin, ev, 0));
    }
  }
  return rc;
}

// ------------------------------------------------------------------------------------------------
// Copies between host and device: uploads at a span's start, downloads and results at its end
// ------------------------------------------------------------------------------------------------
// Host part of an upload (pass 1, in program order): what the copy kernel will read is put in place, or a large host
// array is sent through the copy engine at once. The kernel runs after all host instructions of the span, so it may read
// only what none of them can write: an argument, or a copy made here. A variable's host memory (a learning rate that the
// call also decays) is copied now, one on the device by a copy that is queued now, ahead of what pass 1 queues after it.
static int stage_upload(cgtbInterp* it, Span& s, Instr& in) {
  cgtObject *src_o = get(it, in.reads[0]), *dst_o = get(it, in.write);
  if (!src_o || !dst_o) return fail("%s: operand was never produced", in.repr.c_str());
  if (src_o->kind() != cgtObject::ArrayKind || dst_o->kind() != cgtObject::ArrayKind) return fire(it, in);  // tuples: member by member
  cgtArray *src = (cgtArray*)src_o, *dst = (cgtArray*)dst_o;
  const long nbytes = src->nbytes();
  if (src->size() != dst->size() || src->dtype() != dst->dtype()) return fail("%s: cgt_copy_array: size or dtype mismatch", in.repr.c_str());
  if (nbytes == 0) return 0;
  const void* from = src->data();
  if (src->devtype() == cgtCPU) {
    const bool pinned = host_block_is_pinned(from), large = nbytes > kKernelCopyBytes;
    if (large && !pinned) return upload_pageable(dst->data(), from, (size_t)nbytes);
    if (!pinned || !in.from_argument) {
      if (in.stage_cap < nbytes) {
        if (in.stage) cgtb_free(cgtbCPU, in.stage);
        in.stage = cgtb_alloc(cgtbCPU, nbytes);
        in.stage_cap = in.stage ? nbytes : 0;
        if (!in.stage) return 1;
      }
      stage_for_kernel(in.stage, from, (size_t)nbytes);
      from = in.stage;
    }
    if (large) {
      CGTB_CUDA_TRY(cudaMemcpyAsync(dst->data(), from, (size_t)nbytes, cudaMemcpyHostToDevice, rt().stream));
      return 0;
    }
  } else if (!in.from_argument) {
    CGTB_CUDA_TRY(cudaMemcpyAsync(dst->data(), from, (size_t)nbytes, cudaMemcpyDeviceToDevice, rt().stream));
    return 0;
  }
  s.uploads.job[s.uploads.n++] = CopyJob{from, dst->data(), nbytes};
  return 0;
}

static void add_copy_out(CopyJobs& jobs, const void* src, void* dst, long nbytes, int* rc) {
  if (nbytes == 0 || *rc) return;
  if (nbytes > kKernelCopyBytes) {
    const cudaError_t e = cudaMemcpyAsync(dst, src, (size_t)nbytes, cudaMemcpyDeviceToHost, rt().stream);
    if (e != cudaSuccess) *rc = fail("copy to the host failed: %s", cudaGetErrorString(e));
    return;
  }
  if (jobs.n == kMaxCopyJobs) {
    *rc = launch_copy_jobs(jobs);
    jobs.n = 0;
  }
  jobs.job[jobs.n++] = CopyJob{src, dst, nbytes};
}
// Place of every device result in the pinned result block (grown here, outside captures). An argument that the function
// hands back is not copied by the graph, which would keep the address that it had when the graph was captured: the
// caller reads it from the object that this call got.
static int place_outputs(cgtbInterp* it) {
  long total = 0;
  it->out_offset.assign(it->outs.size(), -1);
  it->out_array.assign(it->outs.size(), nullptr);
  for (size_t i = 0; i < it->outs.size(); ++i) {
    cgtObject* o = get(it, it->outs[i]);
    if (!o || o->kind() != cgtObject::ArrayKind || ((cgtArray*)o)->devtype() != cgtGPU || it->out_is_argument[i]) continue;
    it->out_offset[i] = total;
    it->out_array[i] = (cgtArray*)o;
    total += (((cgtArray*)o)->nbytes() + 63) & ~63L;
  }
  if (total > it->out_stage_cap) {
    if (it->out_stage) cgtb_free(cgtbCPU, it->out_stage);
    it->out_stage = (char*)cgtb_alloc(cgtbCPU, total);
    it->out_stage_cap = it->out_stage ? total : 0;
    if (!it->out_stage) return 1;
  }
  return 0;
}
static void add_outputs(cgtbInterp* it, CopyJobs& jobs, int* rc) {
  for (size_t i = 0; i < it->outs.size(); ++i) {
    it->out_host[i] = nullptr;
    if (it->out_offset[i] < 0) continue;
    cgtArray* a = it->out_array[i];
    it->out_host[i] = it->out_stage + it->out_offset[i];
    add_copy_out(jobs, a->data(), it->out_host[i], a->nbytes(), rc);
  }
}
// Copies that end the span: its downloads, and the function's results if it is the last one.
static int issue_copies_out(cgtbInterp* it, Span& s) {
  auto& instrs = it->g->instrs;
  CopyJobs jobs;
  jobs.n = 0;
  int rc = 0;
  for (int i = s.begin; i < s.end && !rc; ++i) {
    Instr& in = instrs[(size_t)i];
    if (in.klass != kDownload) continue;
    cgtObject *src = get(it, in.reads[0]), *dst = get(it, in.write);
    if (!src || !dst) return fail("%s: operand was never produced", in.repr.c_str());
    if (src->kind() != cgtObject::ArrayKind || dst->kind() != cgtObject::ArrayKind || ((cgtArray*)src)->devtype() != cgtGPU ||
        !host_block_is_pinned(((cgtArray*)dst)->data())) {
      rc = fire(it, in);
      continue;
    }
    cgtArray *a = (cgtArray*)src, *b = (cgtArray*)dst;
    if (a->size() != b->size() || a->dtype() != b->dtype()) return fail("%s: cgt_copy_array: size or dtype mismatch", in.repr.c_str());
    add_copy_out(jobs, a->data(), b->data(), a->nbytes(), &rc);
  }
  if (s.collects && !rc) add_outputs(it, jobs, &rc);
  return rc ? rc : launch_copy_jobs(jobs);
}
static int issue_device(cgtbInterp* it, Span& s, bool profile, bool multistream) {
  auto& instrs = it->g->instrs;
  if (launch_copy_jobs(s.uploads)) return 1;
  if (multistream) {
    if (fire_span_multistream(it, s, rt().stream)) return 1;
  } else {
    for (int i = s.begin; i < s.end; ++i) {
      Instr& in = instrs[(size_t)i];
      if (in.klass != kDevice) continue;
      if ((in.flags & CGTB_INSTR_ONCE) && in.fired) continue;
      const int rc = profile ? fire_profiled(it, in) : fire(it, in);
      if (rc) return rc;
    }
  }
  return issue_copies_out(it, s);
}
static void mark_device_fired(cgtbInterp* it, Span& s) {
  for (int i = s.begin; i < s.end; ++i)
    if (it->g->instrs[(size_t)i].klass == kDevice) it->g->instrs[(size_t)i].fired = true;
}
// The graph's first node is the copy kernel (if the span uploads anything): remember it for update_uploads.
static void find_upload_node(Span& s) {
  s.upload_node = nullptr;
  if (!s.uploads.n) return;
  size_t n = 0;
  if (cudaGraphGetRootNodes(s.graph, nullptr, &n) != cudaSuccess || n != 1) return;
  cudaGraphNode_t node;
  cudaKernelNodeParams p;
  if (cudaGraphGetRootNodes(s.graph, &node, &n) == cudaSuccess && cudaGraphKernelNodeGetParams(node, &p) == cudaSuccess && p.func == copy_jobs_function())
    s.upload_node = node;
}
// Before a replay: tell the copy node where this run's arguments are, if they moved. false: the graph cannot be used.
static bool update_uploads(Span& s) {
  const CopyJobs &a = s.uploads, &b = s.captured_uploads;
  if (a.n == b.n && memcmp(a.job, b.job, sizeof(CopyJob) * (size_t)a.n) == 0) return true;
  if (a.n != b.n || !s.upload_node) return false;
  unsigned gx, gy, block;
  copy_jobs_launch_dims(s.uploads, &gx, &gy, &block);
  cudaKernelNodeParams p = {};
  void* args[1] = {&s.uploads};
  p.func = const_cast<void*>(copy_jobs_function());
  p.gridDim = dim3(gx, gy);
  p.blockDim = dim3(block);
  p.kernelParams = args;
  if (cudaGraphExecKernelNodeSetParams(s.exec, s.upload_node, &p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  s.captured_uploads = s.uploads;
  return true;
}
// a replay leaves the results where the captured run put them
static void outputs_of_replay(cgtbInterp* it) {
  for (size_t i = 0; i < it->outs.size(); ++i) it->out_host[i] = it->out_offset[i] < 0 ? nullptr : it->out_stage + it->out_offset[i];
}

static int run_span(cgtbInterp* it, Span& s) {
  auto& instrs = it->g->instrs;
  const bool profile = (it->flags & CGTB_INTERP_PROFILE) && rt().ready;
  if (s.barrier) {
    Instr& in = instrs[(size_t)s.begin];
    if ((in.flags & CGTB_INSTR_ONCE) && in.fired) return 0;
    bool is_transport = in.flags & CGTB_INSTR_TRANSPORT;
    if (!is_transport && rt().ready) {  // arbitrary callable: give it a quiet stream
      cudaStreamSynchronize(rt().stream);
      it->host_pending = false;
    }
    int rc = profile ? fire_profiled(it, in) : fire(it, in);
    if (rc) return rc;
    in.fired = true;
    if (is_transport && in.write.dev == cgtbCPU) it->host_pending = true;
    return 0;
  }
  if ((s.has_hostdata || s.reads_download) && it->host_pending) {
    CGTB_CUDA_TRY(cudaStreamSynchronize(rt().stream));
    it->host_pending = false;
  }
  s.uploads.n = 0;
  // pass 1: host bookkeeping and host scalar arithmetic, in program order. A steady run skips bookkeeping whose result
  // the storage already holds.
  const bool steady_list = it->steady && !it->host_dirty;
  const int n_pass1 = steady_list ? (int)s.steady_host.size() : s.end - s.begin;
  for (int q = 0; q < n_pass1; ++q) {
    const int i = steady_list && !it->host_dirty ? s.steady_host[(size_t)q] : (steady_list ? -1 : s.begin + q);
    if (i < 0) break;  // a host value changed within this span: the rest is walked in full below
    Instr& in = instrs[(size_t)i];
    if (in.klass == kDevice || in.klass == kDownload) continue;
    if ((in.flags & CGTB_INSTR_ONCE) && in.fired) continue;
    if (in.klass == kUpload) {
      if (stage_upload(it, s, in)) return 1;
      continue;
    }
    if (steady_list && in.klass == kHostData) {
      // did this instruction produce the value it produced in the run before? (small results only: a large one
      // counts as new)
      unsigned char before[64];
      size_t nb = 0;
      bool small = false;
      cgtObject* w = get(it, in.write);
      if (w && w->kind() == cgtObject::ArrayKind && ((cgtArray*)w)->devtype() == cgtCPU && ((cgtArray*)w)->nbytes() <= 64 &&
          ((cgtArray*)w)->data()) {
        nb = (size_t)((cgtArray*)w)->nbytes();
        memcpy(before, ((cgtArray*)w)->data(), nb);
        small = true;
      }
      if (fire(it, in)) return 1;
      cgtObject* w2 = get(it, in.write);
      if (!small || w2 != w || memcmp(before, ((cgtArray*)w2)->data(), nb) != 0) {
        it->host_dirty = true;
        in.fired = true;
        // everything after this instruction is walked in full
        for (int k = i + 1; k < s.end; ++k) {
          Instr& rest = instrs[(size_t)k];
          if (rest.klass == kDevice || rest.klass == kDownload) continue;
          if ((rest.flags & CGTB_INSTR_ONCE) && rest.fired) continue;
          if (rest.klass == kUpload ? stage_upload(it, s, rest) : fire(it, rest)) return 1;
          rest.fired = true;
        }
      }
      in.fired = true;
      continue;
    }
    if (fire(it, in)) return 1;
    in.fired = true;
  }
  // on every run, steady ones too: bookkeeping on arguments makes a new view object of the same bytes each time
  if (s.collects && place_outputs(it)) return 1;
  if (s.n_device == 0) return 0;
  for (int i = s.begin; i < s.end && !it->host_pending; ++i) it->host_pending = instrs[(size_t)i].klass == kDownload;
  // pass 2: device instructions, replayed from a CUDA graph when the span is in steady state
  bool use_graphs = (it->flags & CGTB_INTERP_CUDA_GRAPHS) && !profile && !s.capture_failed && s.n_device >= 2;
  const bool unchanged = it->steady && !it->host_dirty && s.exec && s.have_last && s.exec_key == s.last_key;
  uint64_t key = use_graphs && !unchanged ? span_key(it, s) : s.last_key;
  // `unchanged`: nothing that the key covers can have changed since the run before, which launched this graph
  if (use_graphs && s.exec && s.exec_key == key && update_uploads(s)) {
    s.last_key = key;
    s.have_last = true;
    CGTB_CUDA_TRY(cudaGraphLaunch(s.exec, rt().stream));
    if (s.collects) outputs_of_replay(it);
    it->last_graph_launches += 1;
    it->last_launches += s.graph_kernels;
    return 0;
  }
  bool capture = use_graphs && s.have_last && s.last_key == key && !it->prev_run_allocated;
  s.last_key = key;
  s.have_last = true;
  if (capture) {
    drop_exec(s);
    long launches0 = g_kernel_launches.load();
    cudaError_t e = cudaStreamBeginCapture(rt().stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      set_capturing(true);
      int rc = issue_device(it, s, false, graph_streams() > 1);
      set_capturing(false);
      cudaGraph_t graph = nullptr;
      e = cudaStreamEndCapture(rt().stream, &graph);
      if (rc == 0 && e == cudaSuccess && graph) {
        e = cudaGraphInstantiate(&s.exec, graph, 0);
        if (e == cudaSuccess) {
          s.graph = graph;
          find_upload_node(s);
          s.captured_uploads = s.uploads;
          s.exec_key = key;   // == s.last_key
          s.graph_kernels = g_kernel_launches.load() - launches0;
          it->captured += 1;
          mark_device_fired(it, s);
          CGTB_CUDA_TRY(cudaGraphLaunch(s.exec, rt().stream));
          it->last_graph_launches += 1;
          it->last_launches += s.graph_kernels;
          return 0;
        }
        cudaGraphDestroy(graph);
        s.exec = nullptr;
      } else if (graph) {
        cudaGraphDestroy(graph);
      }
    }
    // capture did not work for this span: clear the sticky capture error and issue eagerly from now on
    cudaGetLastError();
    cgtb_clear_error();
    s.capture_failed = true;
  }
  long l0 = g_kernel_launches.load();
  if (issue_device(it, s, profile, false)) return 1;
  mark_device_fired(it, s);
  it->last_launches += g_kernel_launches.load() - l0;
  return 0;
}

CGTB_API int cgtb_interp_run(cgtbInterp* it, cgtbObject* args_obj, cgtbObject** out) {
  if (!it || !args_obj || !out) return fail("cgtb_interp_run: null argument");
  cgtTuple* args = (cgtTuple*)args_obj;
  if (((cgtObject*)args_obj)->kind() != cgtObject::TupleKind || args->len != it->g->n_args)
    return fail("cgtb_interp_run: expected a tuple of %ld arguments", it->g->n_args);
  cgtb_clear_error();
  const auto host_t0 = std::chrono::steady_clock::now();
  it->args = args;
  it->last_launches = 0;
  it->last_graph_launches = 0;
  long mallocs0 = device_malloc_count();
  int rc = 0;
  {
    // signature of the arguments: buffers, dtypes and extents; the bytes of small host arrays (they may be read
    // as operands at launch time); for large host arrays only the shape (they are copied by a Transport)
    std::vector<uint64_t> sig;
    sig.reserve(16);
    std::vector<std::pair<cgtObject*, bool>> stack;   // (object, its device address matters)
    for (int i = 0; i < args->len; ++i)
      stack.push_back({args->getitem(i), ((it->args_read_in_place >> (i < 63 ? i : 63)) & 1ull) != 0});
    while (!stack.empty()) {
      cgtObject* o = stack.back().first;
      const bool pinned = stack.back().second;
      stack.pop_back();
      if (!o) { sig.push_back(0); continue; }
      if (o->kind() == cgtObject::TupleKind) {
        cgtTuple* t = (cgtTuple*)o;
        sig.push_back(0x7475706cull + (uint64_t)t->len);
        for (int i = 0; i < t->len; ++i) stack.push_back({t->getitem(i), pinned});
        continue;
      }
      cgtArray* a = (cgtArray*)o;
      sig.push_back(((uint64_t)a->ndim() << 16) | ((uint64_t)a->dtype() << 8) | (uint64_t)a->devtype());
      for (int d = 0; d < a->ndim(); ++d) sig.push_back((uint64_t)a->shape()[d]);
      if (a->devtype() == cgtGPU) { if (pinned) sig.push_back((uint64_t)(uintptr_t)a->data()); }
      else if (a->nbytes() <= 64 && a->data()) {
        uint64_t buf[8] = {0};
        memcpy(buf, a->data(), (size_t)a->nbytes());
        for (int i = 0; i < 8; ++i) sig.push_back(buf[i]);
      }
    }
    const long ver = g_state_version.load(std::memory_order_relaxed);
    static const bool allow = []() { const char* e = getenv("CGTB_STEADY_RUNS"); return !(e && e[0] == '0'); }();
    // a steady run takes host values from the run before: not where the call itself leaves another value for the next one
    it->steady = allow && !it->by_value_state && it->prev_run_ok && !it->prev_run_allocated && it->runs >= 2 && ver == it->state_version_seen &&
                 sig == it->arg_sig && !(it->flags & CGTB_INTERP_PROFILE);
    it->arg_sig.swap(sig);
    it->state_version_seen = ver;
    it->host_dirty = false;
    if (it->steady) it->steady_runs += 1;
  }
  // The before-sync hook (host work that should overlap this run's device work, e.g. queueing the next batch's
  // upload) runs as soon as the last span that queues device work or a copy has been issued: the host-only
  // spans after it (arithmetic on a scalar that was copied back) wait for the stream.
  long last_queueing = -1;
  for (size_t i = 0; i < it->spans.size(); ++i)
    if (it->spans[i].barrier || it->spans[i].n_device > 0) last_queueing = (long)i;
  bool hooked = false, collected = false;
  it->out_host.assign(it->outs.size(), nullptr);
  for (size_t i = 0; i < it->spans.size(); ++i) {
    rc = run_span(it, it->spans[i]);
    if (rc) break;
    collected = collected || it->spans[i].collects;
    if ((long)i == last_queueing && it->before_sync) {
      it->before_sync(it->before_sync_ctx);
      hooked = true;
    }
  }
  if (!rc && !collected && rt().ready) {
    CopyJobs jobs;
    jobs.n = 0;
    rc = place_outputs(it);
    if (!rc) add_outputs(it, jobs, &rc);
    if (!rc) rc = launch_copy_jobs(jobs);
  }
  it->args = nullptr;
  if (!rc && !hooked && it->before_sync) it->before_sync(it->before_sync_ctx);
  it->last_host_ns = (long)std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now() - host_t0).count();
  if (rt().ready) {
    cudaError_t e = cudaStreamSynchronize(rt().stream);
    it->host_pending = false;
    if (e != cudaSuccess && !rc) rc = fail("device work of this run failed: %s", cudaGetErrorString(e));
    if (!rc) rc = sgemm_tc_check();
  }
  it->prev_run_allocated = device_malloc_count() != mallocs0;
  it->prev_run_ok = rc == 0;
  it->runs += 1;
  if (it->runs == 1 && !rc) build_spans(it);  // fire-once barriers are out of the way now
  if (rc) return rc;
  cgtTuple* o = new cgtTuple((int)it->outs.size());
  o->Retain();
  for (size_t i = 0; i < it->outs.size(); ++i) {
    o->setitem((int)i, get(it, it->outs[i]));
    // an object that bookkeeping replaced after the results were copied is read back by the caller
    if (it->out_host[i] && get(it, it->outs[i]) != it->out_array[i]) it->out_host[i] = nullptr;
  }
  *out = (cgtbObject*)o;
  return 0;
}

CGTB_API const void* cgtb_interp_output_host(cgtbInterp* it, int i) {
  return it && i >= 0 && (size_t)i < it->out_host.size() ? it->out_host[(size_t)i] : nullptr;
}

CGTB_API int cgtb_interp_set_before_sync(cgtbInterp* it, void (*fn)(void*), void* ctx) {
  if (!it) return fail("cgtb_interp_set_before_sync: null interpreter");
  it->before_sync = fn;
  it->before_sync_ctx = ctx;
  return 0;
}

CGTB_API int cgtb_interp_stats(cgtbInterp* it, long* c, int n) {
  long graph_kernels = 0, dev = 0;
  for (auto& s : it->spans) { if (s.exec) graph_kernels += s.graph_kernels; dev += s.n_device; }
  long v[8] = {it->runs, it->last_launches, it->last_graph_launches, it->captured, graph_kernels, dev, it->last_host_ns, it->steady_runs};
  for (int i = 0; i < n && i < 8; ++i) c[i] = v[i];
  return 0;
}
CGTB_API int cgtb_interp_profile(cgtbInterp* it, double* ms, long* counts, int cap) {
  int n = (int)it->g->instrs.size();
  for (int i = 0; i < n && i < cap; ++i) { ms[i] = it->g->instrs[(size_t)i].prof_ms; counts[i] = it->g->instrs[(size_t)i].prof_count; }
  return n;
}
CGTB_API const char* cgtb_interp_instr_repr(cgtbInterp* it, int i) {
  if (i < 0 || i >= (int)it->g->instrs.size()) return "";
  return it->g->instrs[(size_t)i].repr.c_str();
}
CGTB_API int cgtb_apply_byref(void* fptr, void* closure, int n, cgtbObject** reads, cgtbObject* write) {
  if (!fptr) return fail("cgtb_apply_byref: null function pointer");
  cgtb_clear_error();
  ((cgtByRefFun)fptr)(closure, (cgtObject**)reads, (cgtObject*)write);
  if (cgt_get_status() != cgtStatusOK) return 1;
  if (rt().ready) CGTB_CUDA_TRY(cudaStreamSynchronize(rt().stream));
  return 0;
}
