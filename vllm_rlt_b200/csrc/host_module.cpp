// vllm_rlt_b200._host: the host side of the Python calls that a serving loop makes per step or per chunk.
//
// A launch of this library takes a GPU a few to a few hundred microseconds, so the time Python needs to look over block
// tables, fill structs and find the current stream decides how many of them a worker can issue. This module does that
// part in C++: it reads tables (tuples, lists, int32 arrays) straight into the records of block_moves.h, reads tensors'
// addresses and shapes without building Python objects, and calls the C ABI. Checks and messages are those of the
// Python callers' documentation.

#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#define NPY_NO_DEPRECATED_API NPY_2_0_API_VERSION
#include <numpy/arrayobject.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstddef>
#include <cstring>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "block_moves.h"
#include "internal.h"
#include "rlt_kv_handoff.h"

namespace {

struct Failure {};  // a Python error is set

[[noreturn]] void fail(PyObject* type, const char* text) {
  PyErr_SetString(type, text);
  throw Failure{};
}
[[noreturn]] void bad_value(const char* text) { fail(PyExc_ValueError, text); }

// Integers that grow without being zeroed first: every one is written before it is read.
template <typename V>
struct Uninitialised : std::allocator<V> {
  template <typename U>
  struct rebind {
    using other = Uninitialised<U>;
  };
  template <typename U>
  void construct(U* p) {
    ::new (static_cast<void*>(p)) U;
  }
  template <typename U, typename... A>
  void construct(U* p, A&&... a) {
    ::new (static_cast<void*>(p)) U(std::forward<A>(a)...);
  }
};
using Ints = std::vector<int32_t, Uninitialised<int32_t>>;

struct Ref {
  PyObject* p;
  explicit Ref(PyObject* q) : p(q) {
    if (q == nullptr) throw Failure{};
  }
  ~Ref() { Py_DECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
};

void check_code(int code) {
  if (code < 0) fail(PyExc_RuntimeError, rlt_error_string(code));
}

// f() without the interpreter's lock: every call into the CUDA runtime, for any of them may wait for the GPU (a launch where the
// launch queue is full, an upload where all staging slots are busy), and the thread that the GPU waits for may be one of this
// interpreter. Nothing in f touches a Python object; what it reads is held by the caller's arguments and changed by nobody.
template <typename F>
auto unlocked(F f) {
  struct Away {
    PyThreadState* state = PyEval_SaveThread();
    ~Away() { PyEval_RestoreThread(state); }
  } away;
  return f();
}

struct Buffer {
  Py_buffer view;
  bool held = false;
  ~Buffer() {
    if (held) PyBuffer_Release(&view);
  }
};

long long integer(PyObject* o) {
  if (PyLong_Check(o)) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Failure{};
    return v;
  }
  const Ref n(PyNumber_Long(o));
  const long long v = PyLong_AsLongLong(n.p);
  if (v == -1 && PyErr_Occurred()) throw Failure{};
  return v;
}

// A position or size: a fraction is refused, not cut off.
long long index_of(PyObject* o) {
  if (PyLong_CheckExact(o)) return integer(o);
  const Ref n(PyNumber_Index(o));
  return integer(n.p);
}

int32_t int32_of(long long v) {
  if (v < INT32_MIN || v > INT32_MAX) fail(PyExc_OverflowError, "block id or exit plane out of bounds for int32");
  return static_cast<int32_t>(v);
}

bool is_int32(const Py_buffer& v) {
  return v.itemsize == 4 && v.format != nullptr && (std::strcmp(v.format, "i") == 0 || std::strcmp(v.format, "l") == 0);
}

// An int32 array of NumPy's, or nullptr. Its fields are read directly: asked for a buffer, NumPy describes the element type in a string each
// time, 0.1 us an array, and a batch has one for every request and plane.
PyArrayObject* int32_array(PyObject* o) {
  if (!PyArray_Check(o)) return nullptr;
  auto* array = reinterpret_cast<PyArrayObject*>(o);
  const int type = PyArray_TYPE(array);
  const bool whole = type == NPY_INT || (sizeof(long) == 4 && type == NPY_LONG);
  return whole && PyArray_ISALIGNED(array) && PyArray_ISNOTSWAPPED(array) ? array : nullptr;
}

// Appends the int32 values of one table (or exit-plane array) to `out`; returns how many.
Py_ssize_t append_ints(PyObject* o, Ints& out, const char* not_flat) {
  if (PyTuple_CheckExact(o) || PyList_CheckExact(o)) {
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
    PyObject** items = PySequence_Fast_ITEMS(o);
    const size_t at = out.size();
    out.resize(at + static_cast<size_t>(n));
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* item = items[i];
      if (PyTuple_Check(item) || PyList_Check(item)) bad_value(not_flat);
      out[at + i] = int32_of(integer(item));
    }
    return n;
  }
  auto copy = [&](const char* from, Py_ssize_t n, Py_ssize_t stride) {
    const size_t at = out.size();
    out.resize(at + static_cast<size_t>(n));
    if (stride == 4) {
      std::memcpy(out.data() + at, from, 4 * static_cast<size_t>(n));
    } else {
      for (Py_ssize_t i = 0; i < n; ++i) std::memcpy(&out[at + i], from + i * stride, 4);
    }
    return n;
  };
  auto take = [&](PyObject* source) -> Py_ssize_t {
    if (PyArrayObject* array = int32_array(source)) {
      if (PyArray_NDIM(array) != 1) bad_value(not_flat);
      return copy(PyArray_BYTES(array), PyArray_DIM(array, 0), PyArray_STRIDE(array, 0));
    }
    Buffer b;
    if (PyObject_GetBuffer(source, &b.view, PyBUF_RECORDS_RO) != 0) {
      PyErr_Clear();
      return -1;
    }
    b.held = true;
    if (b.view.ndim != 1) bad_value(not_flat);
    if (!is_int32(b.view)) return -1;
    return copy(static_cast<const char*>(b.view.buf), b.view.shape[0], b.view.strides[0]);
  };
  Py_ssize_t n = take(o);
  if (n >= 0) return n;
  const Ref numpy(PyImport_ImportModule("numpy"));
  const Ref array(PyObject_CallMethod(numpy.p, "asarray", "OO", o, Ref(PyObject_GetAttrString(numpy.p, "int32")).p));
  n = take(array.p);
  if (n < 0) fail(PyExc_TypeError, "block tables and exit planes must hold integers");
  return n;
}

Py_ssize_t length(PyObject* o) {
  const Py_ssize_t n = PyObject_Length(o);
  if (n < 0) throw Failure{};
  return n;
}

// ------------------------------------------------------------------------------------------------ batch plans

struct Side {
  bool given = false;
  int planes = 0;
  int width = 0;                       // pages of the longest table
  Ints flat;                           // every table, back to back
  std::vector<size_t> at;              // [n * planes] where each starts
  std::vector<Py_ssize_t> pages;       // [n] of each request's tables
  const int32_t* table(int r, int p) const { return flat.data() + at[static_cast<size_t>(r) * planes + p]; }
};

struct Plan {
  int n = 0, block_size = 0, width = 1;
  Side src, dst;
  std::vector<int64_t> begin, end;
  bool has_exit = false;
  Ints exits;
  std::vector<int64_t> exit_at;  // [n] index in exits of each request's token 0
  int blocks = 0, words = 0;
  Ints records;
  // Where the rows of a dedup image lie, by the image's planes: made once each and never changed, because several threads may use
  // the batch at once, for images of different plane counts.
  struct Wire {
    Ints at;
    int64_t tokens = 0;
  };
  std::map<int, Wire> wires;

  void make_records();
  const Wire& wire(int planes);
};

void read_side(PyObject* tables, Side& side, int n, int block_size, const std::vector<int64_t>& end) {
  side.given = true;
  if (length(tables) != n) bad_value("one table set per request is required");
  const Ref requests(PySequence_Fast(tables, "block tables must be a sequence of requests"));
  std::vector<std::unique_ptr<Ref>> sets;
  sets.reserve(n);
  for (int r = 0; r < n; ++r)
    sets.push_back(std::make_unique<Ref>(PySequence_Fast(PySequence_Fast_GET_ITEM(requests.p, r), "a request's tables must be a sequence")));
  side.planes = static_cast<int>(PySequence_Fast_GET_SIZE(sets[0]->p));
  for (int r = 0; r < n; ++r) {
    if (PySequence_Fast_GET_SIZE(sets[r]->p) != side.planes) bad_value("requests of one batch must have the same number of planes");
  }
  side.at.reserve(static_cast<size_t>(n) * side.planes);
  side.pages.resize(n);
  bool ragged = false;
  for (int r = 0; r < n; ++r) {
    Py_ssize_t first = 0, least = 0;
    for (int p = 0; p < side.planes; ++p) {
      side.at.push_back(side.flat.size());
      const Py_ssize_t pages = append_ints(PySequence_Fast_GET_ITEM(sets[r]->p, p), side.flat, "a block table must be a flat sequence of block ids");
      if (p == 0) first = least = pages;
      ragged |= pages != first;
      least = pages < least ? pages : least;
    }
    if (end[r] > static_cast<int64_t>(least) * block_size) bad_value("KV range exceeds allocation");
    side.pages[r] = first;
    if (first > side.width) side.width = static_cast<int>(first);
  }
  if (ragged) bad_value("the planes of one request must have tables of equal length");
}

// A block id outside the pool matters only on pages that the request's range touches.
void check_blocks(const Side& side, const Plan& plan, long long limit) {
  if (!side.given) return;
  for (int r = 0; r < plan.n; ++r) {
    const int64_t lo = plan.begin[r] / plan.block_size, hi = (plan.end[r] - 1) / plan.block_size;
    for (int p = 0; p < side.planes; ++p) {
      const int32_t* t = side.table(r, p);
      bool bad = false;
      if (limit < 0) {
        for (int64_t i = lo; i <= hi; ++i) bad |= t[i] < 0;
      } else {
        for (int64_t i = lo; i <= hi; ++i) bad |= static_cast<long long>(static_cast<uint32_t>(t[i])) >= limit;
      }
      if (bad) bad_value("physical block outside registered pool");
    }
  }
}

void Plan::make_records() {
  words = kRecordHeader + src.planes + dst.planes + (has_exit ? block_size : 0);
  int64_t total = 0;
  for (int r = 0; r < n; ++r) total += (end[r] - 1) / block_size - begin[r] / block_size + 1;
  blocks = static_cast<int>(total);
  records.resize(static_cast<size_t>(total) * words);
  int32_t* w = records.data();
  int64_t before = 0;
  std::vector<const int32_t*> tables;
  for (int r = 0; r < n; ++r) {
    const int64_t b = begin[r], e = end[r];
    tables.clear();
    for (const Side* side : {&src, &dst}) {
      for (int p = 0; p < side->planes; ++p) tables.push_back(side->table(r, p));
    }
    const int32_t* exit = has_exit ? exits.data() + exit_at[r] : nullptr;
    for (int64_t page = b / block_size; page <= (e - 1) / block_size; ++page, w += words) {
      const int64_t base = page * block_size;
      const int64_t lo = b > base ? b - base : 0, hi = e < base + block_size ? e - base : block_size;
      w[0] = r;
      w[1] = static_cast<int32_t>(page);
      w[2] = static_cast<int32_t>(lo | hi << 8);
      w[3] = static_cast<int32_t>(base + lo - b);
      w[4] = static_cast<int32_t>(before);
      w[5] = static_cast<int32_t>(e - b);
      int32_t* id = w + kRecordHeader;
      for (const int32_t* table : tables) *id++ = table[page];
      if (has_exit) {
        if (hi - lo != block_size) std::memset(id, 0, 4 * static_cast<size_t>(block_size));
        std::memcpy(id + lo, exit + base + lo, 4 * static_cast<size_t>(hi - lo));
      }
    }
    before += e - b;
  }
}

// Wire order: request, plane, page; a page's tokens count on every plane up to their exit plane.
const Plan::Wire& Plan::wire(int planes) {
  if (const auto made = wires.find(planes); made != wires.end()) return made->second;
  Ints at(static_cast<size_t>(blocks) * planes);
  std::vector<int32_t> carried(planes + 1);
  const int exit_word = kRecordHeader + src.planes + dst.planes;
  for (int b = 0; b < blocks; ++b) {
    const int32_t* w = records.data() + static_cast<size_t>(b) * words;
    std::fill(carried.begin(), carried.end(), 0);
    for (int t = w[2] & 0xff; t < w[2] >> 8; ++t) {
      const int32_t e = w[exit_word + t];
      if (e >= 0) ++carried[e < planes ? e : planes - 1];
    }
    int32_t sum = 0;
    for (int p = planes - 1; p >= 0; --p) at[static_cast<size_t>(b) * planes + p] = sum += carried[p];
  }
  int64_t run = 0;
  for (int b = 0; b < blocks;) {
    int next = b;
    while (next < blocks && records[static_cast<size_t>(next) * words] == records[static_cast<size_t>(b) * words]) ++next;
    for (int p = 0; p < planes; ++p) {
      for (int k = b; k < next; ++k) {
        int32_t& slot = at[static_cast<size_t>(k) * planes + p];
        const int32_t count = slot;
        slot = static_cast<int32_t>(run);
        run += count;
      }
    }
    b = next;
  }
  Wire& made = wires[planes];
  made.at = std::move(at);
  made.tokens = run;
  return made;
}

// Plans that are no longer used, for their memory: fresh pages for a large batch's records cost more than writing them. A
// few are kept, none above kKeptPlanBytes. The interpreter's lock guards the list.
constexpr size_t kKeptPlans = 4;
constexpr size_t kKeptPlanBytes = size_t{8} << 20;
std::vector<std::unique_ptr<Plan>> g_plans;

std::unique_ptr<Plan> fresh_plan() {
  if (g_plans.empty()) return std::make_unique<Plan>();
  std::unique_ptr<Plan> plan = std::move(g_plans.back());
  g_plans.pop_back();
  return plan;
}

void give_back(std::unique_ptr<Plan> plan) {
  const size_t held = 4 * (plan->src.flat.capacity() + plan->dst.flat.capacity() + plan->exits.capacity() + plan->records.capacity());
  if (g_plans.size() >= kKeptPlans || held > kKeptPlanBytes) return;
  Plan clean;
  for (auto list : {&Plan::exits, &Plan::records}) {
    (clean.*list).swap((*plan).*list);
    (clean.*list).clear();
  }
  for (auto side : {&Plan::src, &Plan::dst}) {
    (clean.*side).flat.swap(((*plan).*side).flat);
    (clean.*side).flat.clear();
  }
  *plan = std::move(clean);
  g_plans.push_back(std::move(plan));
}

constexpr const char* kPlanName = "vllm_rlt_b200.plan";
void free_plan(PyObject* capsule) { give_back(std::unique_ptr<Plan>(static_cast<Plan*>(PyCapsule_GetPointer(capsule, kPlanName)))); }
Plan& plan_of(PyObject* capsule) {
  auto* p = static_cast<Plan*>(PyCapsule_GetPointer(capsule, kPlanName));
  if (p == nullptr) throw Failure{};
  return *p;
}

// plan(src_tables | None, dst_tables | None, ranges, exit_planes | None, block_size, src_blocks | None, dst_blocks | None,
//      most requests) -> (plan, requests, tokens, width, source planes, destination planes, exit entries, ranges, record bytes)
PyObject* make_plan(PyObject* const* a) {
  auto plan = fresh_plan();
  const Py_ssize_t n = length(a[2]);
  const long long most = integer(a[7]);
  if (n < 1) bad_value("a handoff batch needs at least one request");
  if (n > most) bad_value(("a handoff batch holds at most " + std::to_string(most) + " requests").c_str());
  plan->n = static_cast<int>(n);
  plan->block_size = static_cast<int>(integer(a[4]));
  if (plan->block_size < 1) bad_value("block_size must be positive");
  const Ref ranges(PySequence_Fast(a[2], "ranges must be a sequence of (start, end)"));
  int64_t tokens = 0;
  for (int r = 0; r < n; ++r) {
    const Ref pair(PySequence_Fast(PySequence_Fast_GET_ITEM(ranges.p, r), "a range is (start, end)"));
    if (PySequence_Fast_GET_SIZE(pair.p) != 2) bad_value("a range is (start, end)");
    const int64_t b = integer(PySequence_Fast_GET_ITEM(pair.p, 0)), e = integer(PySequence_Fast_GET_ITEM(pair.p, 1));
    plan->begin.push_back(b);
    plan->end.push_back(e);
    tokens += e - b;
  }
  for (int r = 0; r < n; ++r) {
    if (plan->begin[r] < 0 || plan->begin[r] >= plan->end[r]) bad_value("invalid KV range");
  }
  if (a[0] != Py_None) read_side(a[0], plan->src, plan->n, plan->block_size, plan->end);
  if (a[1] != Py_None) read_side(a[1], plan->dst, plan->n, plan->block_size, plan->end);
  for (const Side* side : {&plan->src, &plan->dst}) plan->width = side->width > plan->width ? side->width : plan->width;
  check_blocks(plan->src, *plan, a[5] == Py_None ? -1 : integer(a[5]));
  check_blocks(plan->dst, *plan, a[6] == Py_None ? -1 : integer(a[6]));
  if (a[3] != Py_None) {
    plan->has_exit = true;
    if (length(a[3]) != n) bad_value("one exit-plane array per request is required");
    const Ref parts(PySequence_Fast(a[3], "exit planes must be a sequence of per-request arrays"));
    constexpr const char* kCover = "exit planes must cover every token position up to the range end";
    for (int r = 0; r < n; ++r) {
      plan->exit_at.push_back(static_cast<int64_t>(plan->exits.size()));
      const Py_ssize_t count = append_ints(PySequence_Fast_GET_ITEM(parts.p, r), plan->exits, kCover);
      if (count < plan->end[r]) bad_value(kCover);
    }
  }
  if (plan->src.given || plan->dst.given) plan->make_records();  // no tables, nothing to move: the entry points say so
  const Ref list(PyList_New(n));
  for (int r = 0; r < n; ++r) {
    PyObject* pair = Py_BuildValue("LL", static_cast<long long>(plan->begin[r]), static_cast<long long>(plan->end[r]));
    if (pair == nullptr) throw Failure{};
    PyList_SET_ITEM(list.p, r, pair);
  }
  Plan* raw = plan.release();
  PyObject* capsule = PyCapsule_New(raw, kPlanName, free_plan);
  if (capsule == nullptr) {
    delete raw;
    throw Failure{};
  }
  return Py_BuildValue("NiLiiiLOL", capsule, raw->n, static_cast<long long>(tokens), raw->width, raw->src.planes, raw->dst.planes,
                       static_cast<long long>(raw->exits.size()), list.p, static_cast<long long>(4 * raw->records.size()));
}

// plan_layout(plan) -> (bytes, {name: offset}) of the padded arrays an RltBatch points at.
// plan_arrays(plan, writable buffer): writes them there.
struct Layout {
  size_t offsets = 0, src = 0, dst = 0, begin = 0, end = 0, exits = 0, bytes = 0;
};
Layout layout_of(const Plan& p) {
  Layout l;
  auto put = [&](size_t bytes) {
    l.bytes = (l.bytes + 15) & ~size_t{15};
    const size_t at = l.bytes;
    l.bytes += bytes;
    return at;
  };
  const size_t n = p.n, row = 4 * n * p.width;
  if (p.has_exit) l.offsets = put(8 * n);
  if (p.src.given) l.src = put(row * p.src.planes);
  if (p.dst.given) l.dst = put(row * p.dst.planes);
  l.begin = put(4 * n);
  l.end = put(4 * n);
  if (p.has_exit) l.exits = put(4 * p.exits.size());
  return l;
}

PyObject* plan_layout(PyObject* const* a) {
  const Plan& p = plan_of(a[0]);
  const Layout l = layout_of(p);
  const Ref names(PyDict_New());
  auto name = [&](const char* key, size_t at) {
    const Ref v(PyLong_FromSize_t(at));
    if (PyDict_SetItemString(names.p, key, v.p) != 0) throw Failure{};
  };
  if (p.has_exit) name("exit_offsets", l.offsets);
  if (p.src.given) name("src_tables", l.src);
  if (p.dst.given) name("dst_tables", l.dst);
  name("tok_begin", l.begin);
  name("tok_end", l.end);
  if (p.has_exit) name("exit_planes", l.exits);
  return Py_BuildValue("nO", static_cast<Py_ssize_t>(l.bytes), names.p);
}

void write_arrays(const Plan& p, const Layout& l, char* out) {
  std::memset(out, 0, l.bytes);
  auto tables = [&](const Side& side, size_t at) {
    for (int r = 0; r < p.n; ++r) {
      for (int q = 0; q < side.planes; ++q)
        std::memcpy(out + at + 4 * (static_cast<size_t>(r) * side.planes + q) * p.width, side.table(r, q), 4 * static_cast<size_t>(side.pages[r]));
    }
  };
  if (p.src.given) tables(p.src, l.src);
  if (p.dst.given) tables(p.dst, l.dst);
  for (int r = 0; r < p.n; ++r) {
    const int32_t lo = static_cast<int32_t>(p.begin[r]), hi = static_cast<int32_t>(p.end[r]);
    std::memcpy(out + l.begin + 4 * static_cast<size_t>(r), &lo, 4);
    std::memcpy(out + l.end + 4 * static_cast<size_t>(r), &hi, 4);
  }
  if (p.has_exit) {
    std::memcpy(out + l.offsets, p.exit_at.data(), 8 * static_cast<size_t>(p.n));
    if (!p.exits.empty()) std::memcpy(out + l.exits, p.exits.data(), 4 * p.exits.size());
  }
}

PyObject* plan_arrays(PyObject* const* a) {
  const Plan& p = plan_of(a[0]);
  const Layout l = layout_of(p);
  Buffer b;
  if (PyObject_GetBuffer(a[1], &b.view, PyBUF_WRITABLE) != 0) throw Failure{};
  b.held = true;
  if (static_cast<size_t>(b.view.len) < l.bytes) bad_value("staging buffer too small");
  write_arrays(p, l, static_cast<char*>(b.view.buf));
  Py_RETURN_NONE;
}

// plan_wire(plan, planes) -> bytes of the wire plan, made at the first call. Tells how a dedup image is laid out.
PyObject* plan_wire(PyObject* const* a) {
  Plan& p = plan_of(a[0]);
  const int planes = static_cast<int>(integer(a[1]));
  return PyLong_FromSize_t(p.has_exit && planes > 0 ? 4 * p.wire(planes).at.size() : 0);
}

// plan_fits(plan, bytes of the wire plan that goes along): whether the launch takes the records as kernel parameters.
PyObject* plan_fits(PyObject* const* a) {
  const Plan& p = plan_of(a[0]);
  return PyBool_FromLong(4 * p.records.size() + static_cast<size_t>(integer(a[1])) <= 4 * static_cast<size_t>(kInlineWords));
}

void* address(PyObject* o) { return o == Py_None ? nullptr : PyLong_AsVoidPtr(o); }

// plan_upload(plan, planes, device address, stream) -> code: records (0 planes), the wire plan of that many or the padded arrays (-1) to
// device memory.
PyObject* plan_upload(PyObject* const* a) {
  Plan& p = plan_of(a[0]);
  const int planes = static_cast<int>(integer(a[1]));
  void* to = address(a[2]);
  const auto stream = static_cast<rlt_stream_t>(address(a[3]));
  std::vector<char> arrays;
  if (planes < 0) {
    const Layout l = layout_of(p);
    arrays.resize(l.bytes);
    write_arrays(p, l, arrays.data());
  }
  const Ints* list = planes < 0 ? nullptr : planes == 0 ? &p.records : &p.wire(planes).at;
  return PyLong_FromLong(unlocked([&] {
    return list == nullptr ? rlt_stage_upload(arrays.data(), arrays.size(), to, stream) : rlt_stage_upload(list->data(), 4 * list->size(), to, stream);
  }));
}

rlt_stream_t stream_of(PyObject* o) {  // None: the current stream of the current device
  if (o != Py_None) return static_cast<rlt_stream_t>(PyLong_AsVoidPtr(o));
  return reinterpret_cast<rlt_stream_t>(c10::cuda::getCurrentCUDAStream().stream());
}

const at::Tensor* tensor_of(PyObject* o) {
  if (o == Py_None) return nullptr;
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "expected a tensor");
  return &THPVariable_Unpack(o);
}

void* data_of(PyObject* o) {
  const at::Tensor* t = tensor_of(o);
  return t == nullptr ? nullptr : t->data_ptr();
}

// capture(stream) -> the id of the graph capture that it takes part in, 0 if it does not
PyObject* capture(PyObject* const* a) {
  const rlt_stream_t stream = stream_of(a[0]);
  uint64_t id = 0;
  check_code(unlocked([&] { return rlt_capture_id(stream, &id); }));
  return PyLong_FromUnsignedLongLong(id);
}

// move(direction, source pool, destination pool, plan, records, wire plan, mode, layer_begin, layer_end, wire_planes,
//      plane_begin, plane_end, deep mask, status, grid_limit, variant, workspace, packed address, packed bytes, stream) -> code
PyObject* move(PyObject* const* a) {
  Plan& p = plan_of(a[3]);
  const long direction = PyLong_AsLong(a[0]);
  RltOptions o = {};
  o.mode = static_cast<int32_t>(integer(a[6]));
  o.layer_begin = static_cast<int32_t>(integer(a[7]));
  o.layer_end = static_cast<int32_t>(integer(a[8]));
  o.wire_planes = static_cast<int32_t>(integer(a[9]));
  o.plane_begin = static_cast<int32_t>(integer(a[10]));
  o.plane_end = static_cast<int32_t>(integer(a[11]));
  o.deep_layer_mask = PyLong_AsUnsignedLongLong(a[12]);
  o.status = static_cast<int32_t*>(data_of(a[13]));
  o.grid_limit = static_cast<int32_t>(integer(a[14]));
  o.variant = static_cast<int32_t>(integer(a[15]));
  if (const at::Tensor* w = tensor_of(a[16])) {
    if (w->scalar_type() != at::kByte || !w->is_contiguous() || !w->is_cuda())
      bad_value("workspace must be a contiguous CUDA uint8 tensor");
    o.workspace = w->data_ptr();
    o.workspace_bytes = w->numel();
  }
  if (PyErr_Occurred()) throw Failure{};
  RltBlockMoves m = {};
  m.host_records = p.records.data();
  m.device_records = static_cast<const int32_t*>(address(a[4]));
  m.blocks = p.blocks;
  m.words = p.words;
  m.src_planes = p.src.planes;
  m.dst_planes = p.dst.planes;
  m.block_size = p.block_size;
  m.has_exit = p.has_exit;
  m.num_requests = p.n;
  m.table_width = p.width;
  const auto* src = static_cast<const RltPool*>(address(a[1]));
  const auto* dst = static_cast<const RltPool*>(address(a[2]));
  const RltPool* image = direction == RLT_MOVE_PACK ? src : direction == RLT_MOVE_SCATTER ? dst : nullptr;
  if (image != nullptr && o.mode == RLT_MODE_DEDUP && p.has_exit && image->num_planes > 0) {
    const Plan::Wire& wire = p.wire(image->num_planes);
    m.host_wire = wire.at.data();
    m.device_wire = static_cast<const int32_t*>(address(a[5]));
    m.wire_tokens = wire.tokens;
  }
  void* packed = address(a[17]);
  const int64_t packed_bytes = integer(a[18]);
  const rlt_stream_t stream = stream_of(a[19]);
  return PyLong_FromLong(unlocked([&] { return rlt_move_blocks(static_cast<int>(direction), src, dst, &m, &o, packed, packed_bytes, stream); }));
}

// ------------------------------------------------------------------------------------------------ other ops

// handoff_host(source pool, destination pool, source tables, destination tables, begin, end, layer_begin, layer_end,
//              plane_begin, plane_end, status, stream) -> code
struct HostArray {
  const int32_t* data;
  int dims;
  const Py_ssize_t* shape;
  Buffer buffer;
  explicit HostArray(PyObject* o) {
    if (PyArrayObject* array = int32_array(o); array != nullptr && PyArray_IS_C_CONTIGUOUS(array)) {
      data = static_cast<const int32_t*>(PyArray_DATA(array));
      dims = PyArray_NDIM(array);
      shape = PyArray_DIMS(array);
      return;
    }
    constexpr const char* kWanted = "host tables and ranges must be C-contiguous int32 arrays";
    if (PyObject_GetBuffer(o, &buffer.view, PyBUF_FORMAT | PyBUF_STRIDES) != 0) {
      PyErr_Clear();
      bad_value(kWanted);
    }
    buffer.held = true;
    if (!is_int32(buffer.view) || !PyBuffer_IsContiguous(&buffer.view, 'C')) bad_value(kWanted);
    data = static_cast<const int32_t*>(buffer.view.buf);
    dims = buffer.view.ndim;
    shape = buffer.view.shape;
  }
};

PyObject* handoff_host(PyObject* const* a) {
  const HostArray s(a[2]), d(a[3]), begin(a[4]), end(a[5]);
  if (s.dims != 3) bad_value("host tables must be [requests, planes, width]");
  const Py_ssize_t n = s.shape[0];
  auto one_per_request = [&](const HostArray& v) { return v.dims == 1 && v.shape[0] == n; };
  if (d.dims != 3 || d.shape[0] != n || d.shape[2] != s.shape[2] || !one_per_request(begin) || !one_per_request(end))
    bad_value("source and destination tables must agree in requests and width, one range per request");
  RltHostBatch hb = {};
  hb.num_requests = static_cast<int32_t>(n);
  hb.table_width = static_cast<int32_t>(s.shape[2]);
  hb.src_planes = static_cast<int32_t>(s.shape[1]);
  hb.dst_planes = static_cast<int32_t>(d.shape[1]);
  hb.src_tables = s.data;
  hb.dst_tables = d.data;
  hb.tok_begin = begin.data;
  hb.tok_end = end.data;
  RltOptions o = {};
  o.layer_begin = static_cast<int32_t>(integer(a[6]));
  o.layer_end = static_cast<int32_t>(integer(a[7]));
  o.plane_begin = static_cast<int32_t>(integer(a[8]));
  o.plane_end = static_cast<int32_t>(integer(a[9]));
  o.status = static_cast<int32_t*>(data_of(a[10]));
  const auto* src = static_cast<const RltPool*>(address(a[0]));
  const auto* dst = static_cast<const RltPool*>(address(a[1]));
  const rlt_stream_t stream = stream_of(a[11]);
  return PyLong_FromLong(unlocked([&] { return rlt_kv_handoff_host(src, dst, &hb, &o, stream); }));
}

// finalize(pool, planes, tables, rows, layer mask, status, stream) -> code
PyObject* finalize(PyObject* const* a) {
  const at::Tensor* tables = tensor_of(a[2]);
  const at::Tensor* rows = tensor_of(a[3]);
  if (tables == nullptr || rows == nullptr) fail(PyExc_TypeError, "expected a tensor");
  if (tables->scalar_type() != at::kInt || !tables->is_contiguous() || !tables->is_cuda())
    bad_value("tables must be a contiguous CUDA int32 tensor");
  if (rows->scalar_type() != at::kInt || !rows->is_contiguous() || !rows->is_cuda())
    bad_value("rows must be a contiguous CUDA int32 tensor");
  if (tables->dim() != 3 || tables->size(1) != integer(a[1]))
    bad_value("tables must be [requests, planes, width] with the pool's plane count");
  if (rows->dim() != 2 || rows->size(1) != 3) bad_value("rows must be [n, 3]: request index, exit plane, token position");
  const auto* pool = static_cast<const RltPool*>(address(a[0]));
  const int32_t *table_data = tables->data_ptr<int32_t>(), *row_data = rows->data_ptr<int32_t>();
  const auto requests = static_cast<int32_t>(tables->size(0)), width = static_cast<int32_t>(tables->size(2));
  const auto count = static_cast<int32_t>(rows->size(0));
  const uint64_t mask = PyLong_AsUnsignedLongLongMask(a[4]);  // a layer past the 64th: the library says that the pool has too many
  auto* status = static_cast<int32_t*>(data_of(a[5]));
  const rlt_stream_t stream = stream_of(a[6]);
  return PyLong_FromLong(unlocked([&] { return rlt_kv_finalize(pool, table_data, requests, width, row_data, count, mask, status, stream); }));
}

// ------------------------------------------------------------------------------------------------ tensor transfers

// A 1-D view of `t`, as at::as_strided makes it, without the dispatcher and the bookkeeping of autograd (these slices never take
// part in it): a step makes a few hundred of them. The caller has checked the bounds.
at::Tensor plain_view(const at::Tensor& t, int64_t offset, int64_t n, int64_t stride) {
  at::Tensor out = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(t.storage()), t.key_set(), t.dtype());
  out.unsafeGetTensorImpl()->set_storage_offset(offset);
  out.unsafeGetTensorImpl()->set_sizes_and_strides(c10::IntArrayRef(&n, 1), c10::IntArrayRef(&stride, 1));
  return out;
}
// t[start : start + n] of a flat tensor
at::Tensor plain_slice(const at::Tensor& t, int64_t start, int64_t n) {
  return plain_view(t, t.storage_offset() + start * t.stride(0), n, t.stride(0));
}

// RLT_DTYPE_* of a tensor, -1 for the types that do not transfer.
int transfer_type(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kInt: return RLT_DTYPE_I32;
    case at::kLong: return RLT_DTYPE_I64;
    case at::kHalf: return RLT_DTYPE_F16;
    case at::kBFloat16: return RLT_DTYPE_BF16;
    case at::kFloat: return RLT_DTYPE_F32;
    default: return -1;
  }
}

void check_source(const at::Tensor& source, const at::Device& device) {
  if (source.is_cuda()) {
    if (source.device() != device) bad_value("cross-device transfers require an explicit connector");
  } else if (!source.is_pinned()) {
    bad_value("host sources must be pinned: this transfer has no pageable-memory path");
  }
}

const at::Tensor& some_tensor(PyObject* o) {
  const at::Tensor* t = tensor_of(o);
  if (t == nullptr) fail(PyExc_TypeError, "expected a tensor");
  return *t;
}

// tensor_copy(source, target, secondary | None) -> code, on the current stream of the target's device
PyObject* tensor_copy(PyObject* const* a) {
  const at::Tensor &source = some_tensor(a[0]), &target = some_tensor(a[1]);
  const at::Tensor* secondary = tensor_of(a[2]);
  if (source.numel() != target.numel() || !source.is_contiguous() || !target.is_contiguous())
    bad_value("copy_tensor requires equal-sized contiguous tensors");
  if (secondary != nullptr &&
      (secondary->numel() != source.numel() || !secondary->is_contiguous() || secondary->device() != target.device()))
    bad_value("secondary output must match target size and device");
  const int from = transfer_type(source), to = transfer_type(target), second = secondary ? transfer_type(*secondary) : 0;
  if (from < 0 || to < 0 || second < 0) bad_value("unsupported transfer dtype");
  if (!target.is_cuda()) bad_value("transfer destination must be a CUDA tensor");
  check_source(source, target.device());
  if (source.numel() == 0) return PyLong_FromLong(RLT_OK);
  const c10::cuda::CUDAGuard guard(target.device());
  const void* in = source.data_ptr();
  void *out = target.data_ptr(), *also = secondary ? secondary->data_ptr() : nullptr;
  const int64_t count = source.numel();
  const rlt_stream_t stream = stream_of(Py_None);
  return PyLong_FromLong(unlocked([&] { return rlt_tensor_copy(in, out, also, count, from, to, second, stream); }));
}

// A TensorTransfer's descriptors, collected as copies are appended: the rows of rlt_tensor_transfer's table.
struct Transfer {
  using Rows = std::vector<int64_t>;  // 8 per copy
  std::shared_ptr<Rows> rows = std::make_shared<Rows>();
  int64_t max_rows = 0, max_cols = 0;
  // The rows to change: a copy of them while a launch, in another thread, still reads the ones there are.
  Rows& own_rows() {
    if (rows.use_count() > 1) rows = std::make_shared<Rows>(*rows);
    return *rows;
  }
};

// Base of TensorTransfer: the batch itself. `append` runs once per copy, so it is a method of this type.
struct CopiesObject {
  PyObject_HEAD
  Transfer* batch;
  PyObject* copies;  // [(source, target)]: what a submitted batch borrows
  long long capacity;
  int from, to, device;
};
CopiesObject* copies_of(PyObject* o) { return reinterpret_cast<CopiesObject*>(o); }

// setup(capacity, source type, target type, device index)
PyObject* copies_setup(PyObject* self, PyObject* const* a) {
  CopiesObject* c = copies_of(self);
  c->capacity = integer(a[0]);
  c->from = static_cast<int>(integer(a[1]));
  c->to = static_cast<int>(integer(a[2]));
  c->device = static_cast<int>(integer(a[3]));
  Py_RETURN_NONE;
}

PyObject* copies_reset(PyObject* self, PyObject* const*) {
  CopiesObject* c = copies_of(self);
  PyObject* fresh = PyList_New(0);
  if (fresh == nullptr) throw Failure{};
  PyObject* old = c->copies;
  c->copies = fresh;
  c->batch->own_rows().clear();
  c->batch->max_rows = c->batch->max_cols = 0;
  Py_XDECREF(old);
  Py_RETURN_NONE;
}

// Records source -> target; `keep_source` and `keep_target` are what the batch holds on to.
void append_copy(CopiesObject* c, const at::Tensor& source, const at::Tensor& target, PyObject* keep_source, PyObject* keep_target,
                 bool checked = false) {
  Transfer& t = *c->batch;
  const int64_t dims = source.dim();
  if (source.sizes() != target.sizes() || (dims != 1 && dims != 2)) bad_value("transfer requires matching 1D/2D shapes");
  if (transfer_type(source) != c->from || transfer_type(target) != c->to) bad_value("transfer dtype does not match its batch");
  const at::Device device(at::kCUDA, static_cast<c10::DeviceIndex>(c->device));
  if (target.device() != device) bad_value("transfer destination must be on the configured device");
  if (source.is_cuda() && source.device() != device) bad_value("transfer source must be on the configured device");
  if (!checked) check_source(source, device);
  if (source.numel() == 0) return;
  if (static_cast<long long>(t.rows->size() / 8) >= c->capacity) bad_value("transfer batch is full");
  const bool flat = dims == 1;
  const int64_t rows = flat ? 1 : source.size(0), cols = source.size(dims - 1);
  const int64_t row[8] = {reinterpret_cast<int64_t>(source.data_ptr()), reinterpret_cast<int64_t>(target.data_ptr()), rows, cols,
                          flat ? cols * source.stride(0) : source.stride(0), source.stride(dims - 1),
                          flat ? cols * target.stride(0) : target.stride(0), target.stride(dims - 1)};
  const Ref pair(PyTuple_Pack(2, keep_source, keep_target));
  if (PyList_Append(c->copies, pair.p) != 0) throw Failure{};
  Transfer::Rows& list = t.own_rows();
  list.insert(list.end(), row, row + 8);
  t.max_rows = rows > t.max_rows ? rows : t.max_rows;
  t.max_cols = cols > t.max_cols ? cols : t.max_cols;
}

PyObject* copies_append(PyObject* self, PyObject* const* a) {
  append_copy(copies_of(self), some_tensor(a[0]), some_tensor(a[1]), a[0], a[1]);
  Py_RETURN_NONE;
}

// append_pieces(flat tensor, [targets]): appends the copies of consecutive slices of it, each as long as its target.
PyObject* copies_append_pieces(PyObject* self, PyObject* const* a) {
  const at::Tensor& source = some_tensor(a[0]);
  const Ref targets(PySequence_Fast(a[1], "targets must be a sequence of tensors"));
  int64_t at = 0;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(targets.p); ++i) {
    PyObject* target = PySequence_Fast_GET_ITEM(targets.p, i);
    const int64_t n = some_tensor(target).size(0);
    if (source.dim() != 1 || at + n > source.size(0)) bad_value("transfer requires matching 1D/2D shapes");
    append_copy(copies_of(self), plain_slice(source, at, n), some_tensor(target), a[0], target, i > 0);  // slices of one tensor: looked at once
    at += n;
  }
  Py_RETURN_NONE;
}

// launch(pinned table) -> code. A small batch between tensors of one type travels with its launch; others are written into
// the table, which the kernel reads where it lies.
PyObject* copies_launch(PyObject* self, PyObject* const* a) {
  const CopiesObject* c = copies_of(self);
  const Transfer& t = *c->batch;
  const std::shared_ptr<const Transfer::Rows> list = t.rows;
  const int count = static_cast<int>(list->size() / 8), from = c->from, to = c->to;
  if (count == 0) return PyLong_FromLong(RLT_OK);
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(c->device));
  const rlt_stream_t stream = stream_of(Py_None);
  const int32_t rows = static_cast<int32_t>(t.max_rows), cols = static_cast<int32_t>(t.max_cols);
  if (from == to && count <= RLT_INLINE_TRANSFERS && t.max_cols <= INT32_MAX && t.max_rows <= INT32_MAX) {
    const int rc = unlocked([&] { return rlt_tensor_transfer_inline(list->data(), count, rows, cols, from, stream); });
    if (rc != RLT_E_LIMIT) return PyLong_FromLong(rc);
  }
  const at::Tensor& table = some_tensor(a[0]);
  int64_t* entries = table.data_ptr<int64_t>();
  std::memcpy(entries, list->data(), 8 * list->size());
  return PyLong_FromLong(unlocked([&] { return rlt_tensor_transfer(entries, count, rows, cols, from, to, stream); }));
}

// ------------------------------------------------------------------------------------------------ staging helpers

template <typename V, typename F>
bool fill_from(PyObject** items, Py_ssize_t n, V* out, F convert) {
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (!convert(items[i], &out[i])) return false;
  }
  return true;
}

// fill(flat CPU tensor, start, values) -> the slice that received them, or None where the values are not a list or tuple of plain
// numbers of the tensor's kind, or do not fit: the caller's general path then does it, or says what is wrong.
PyObject* fill(PyObject* const* a) {
  const at::Tensor& t = some_tensor(a[0]);
  PyObject* values = a[2];
  if (!PyList_CheckExact(values) && !PyTuple_CheckExact(values)) Py_RETURN_NONE;
  const int64_t start = integer(a[1]);
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(values);
  if (!t.is_cpu() || t.dim() != 1 || !t.is_contiguous() || start < 0 || start > t.size(0) - n) Py_RETURN_NONE;
  PyObject** items = PySequence_Fast_ITEMS(values);
  auto whole = [](PyObject* o, long long* v) {
    if (!PyLong_CheckExact(o)) return false;
    int overflow = 0;
    *v = PyLong_AsLongLongAndOverflow(o, &overflow);
    return overflow == 0;
  };
  bool ok = false;
  if (t.scalar_type() == at::kLong) {
    ok = fill_from(items, n, t.data_ptr<int64_t>() + start, [&](PyObject* o, int64_t* v) {
      long long x;
      if (!whole(o, &x)) return false;
      *v = x;
      return true;
    });
  } else if (t.scalar_type() == at::kInt) {
    ok = fill_from(items, n, t.data_ptr<int32_t>() + start, [&](PyObject* o, int32_t* v) {
      long long x;
      if (!whole(o, &x) || x < INT32_MIN || x > INT32_MAX) return false;
      *v = static_cast<int32_t>(x);
      return true;
    });
  } else if (t.scalar_type() == at::kFloat) {
    ok = fill_from(items, n, t.data_ptr<float>() + start, [&](PyObject* o, float* v) {
      if (!PyFloat_CheckExact(o)) return false;
      *v = static_cast<float>(PyFloat_AS_DOUBLE(o));
      return true;
    });
  }
  if (!ok) Py_RETURN_NONE;
  return THPVariable_Wrap(plain_slice(t, start, n));
}

// row_slice(tensor, index, start, count) -> tensor[index][start : start + count] for a 2-D tensor and an int in range; None otherwise
PyObject* row_slice(PyObject* const* a) {
  const at::Tensor& t = some_tensor(a[0]);
  if (!PyLong_CheckExact(a[1]) || t.dim() != 2) Py_RETURN_NONE;
  int64_t index = index_of(a[1]);
  const int64_t start = index_of(a[2]), n = integer(a[3]);
  index += index < 0 ? t.size(0) : 0;
  if (index < 0 || index >= t.size(0) || start < 0 || start > t.size(1) - n) Py_RETURN_NONE;
  return THPVariable_Wrap(plain_view(t, t.storage_offset() + index * t.stride(0) + start * t.stride(1), n, t.stride(1)));
}

// Base of StagedInputTensor: `append` of plain numbers that fit; everything else is the subclass's `append_values`.
struct FilledObject {
  PyObject_HEAD
  PyObject* cpu;
  Py_ssize_t count;
};

PyObject* filled_append(PyObject* self, PyObject* const* a) {
  auto* f = reinterpret_cast<FilledObject*>(self);
  if (f->cpu != nullptr && f->cpu != Py_None) {
    const Ref start(PyLong_FromSsize_t(f->count));
    PyObject* args[3] = {f->cpu, start.p, a[0]};
    PyObject* piece = fill(args);
    if (piece != Py_None) {
      if (piece != nullptr) f->count += PySequence_Fast_GET_SIZE(a[0]);
      return piece;
    }
    Py_DECREF(piece);
  }
  return PyObject_CallMethod(self, "append_values", "O", a[0]);
}

// Base of StagedWriteTensor: `stage_write` of a list of numbers into one row of a 2-D tensor; else the subclass's `stage_values`.
struct WritesObject {
  PyObject_HEAD
  PyObject *gpu, *values, *targets;
};

PyObject* writes_stage(PyObject* self, PyObject* const* a) {
  auto* w = reinterpret_cast<WritesObject*>(self);
  if (PyList_CheckExact(a[2]) && PyList_GET_SIZE(a[2]) > 0 && w->gpu != nullptr && w->gpu != Py_None && w->values != nullptr &&
      w->targets != nullptr && PyList_CheckExact(w->values) && PyList_CheckExact(w->targets)) {
    const Py_ssize_t n = PyList_GET_SIZE(a[2]);
    const Ref count(PyLong_FromSsize_t(n));
    PyObject* args[4] = {w->gpu, a[0], a[1], count.p};
    const Ref target(row_slice(args));
    if (target.p != Py_None) {
      const Py_ssize_t end = PyList_GET_SIZE(w->values);
      if (PyList_SetSlice(w->values, end, end, a[2]) != 0 || PyList_Append(w->targets, target.p) != 0) throw Failure{};
      Py_RETURN_NONE;
    }
  }
  return PyObject_CallMethod(self, "stage_values", "OOO", a[0], a[1], a[2]);
}

// upload(flat CPU tensor, pinned tensor, device tensor, count) -> the device tensor's first `count` elements, to which the CPU tensor's are
// on their way through the pinned one; None where the three are not flat, of one type and large enough, on those devices.
PyObject* upload(PyObject* const* a) {
  const at::Tensor &source = some_tensor(a[0]), &pinned = some_tensor(a[1]), &target = some_tensor(a[2]);
  const int64_t n = integer(a[3]);
  const int type = transfer_type(source);
  for (const at::Tensor* t : {&source, &pinned, &target}) {
    if (t->dim() != 1 || !t->is_contiguous() || t->size(0) < n || transfer_type(*t) != type) Py_RETURN_NONE;
  }
  if (type < 0 || n < 1 || !source.is_cpu() || !target.is_cuda() || !pinned.is_pinned()) Py_RETURN_NONE;
  std::memcpy(pinned.data_ptr(), source.data_ptr(), static_cast<size_t>(n) * source.element_size());
  const c10::cuda::CUDAGuard guard(target.device());
  const void* from = pinned.data_ptr();
  void* to = target.data_ptr();
  const rlt_stream_t stream = stream_of(Py_None);
  check_code(unlocked([&] { return rlt_tensor_copy(from, to, nullptr, n, type, type, 0, stream); }));
  return THPVariable_Wrap(plain_slice(target, 0, n));
}

// ------------------------------------------------------------------------------------------------ transport

void put(std::string& out, const void* p, size_t n) { out.append(static_cast<const char*>(p), n); }
template <typename V>
void put(std::string& out, V v) {
  put(out, &v, sizeof(v));
}

// Values [from, to) of a table, as int32.
void append_range(PyObject* o, Py_ssize_t from, Py_ssize_t to, Ints& out) {
  if (PyTuple_CheckExact(o) || PyList_CheckExact(o)) {
    PyObject** items = PySequence_Fast_ITEMS(o);
    for (Py_ssize_t i = from; i < to; ++i) out.push_back(int32_of(integer(items[i])));
    return;
  }
  const size_t at = out.size();
  append_ints(o, out, "a block table must be a flat sequence of block ids");
  out.erase(out.begin() + static_cast<std::ptrdiff_t>(at) + to, out.end());
  out.erase(out.begin() + static_cast<std::ptrdiff_t>(at), out.begin() + static_cast<std::ptrdiff_t>(at) + from);
}

// encode_chunk(requests, extra, mode, layer_begin, layer_end, plane_begin, plane_end, page size | 0) -> bytes. With a page size, each
// request's tables are cut to the pages its range touches and the range is rebased onto them.
PyObject* encode_chunk(PyObject* const* a) {
  const Ref requests(PySequence_Fast(a[0], "requests must be a sequence"));
  const Ref extra(PySequence_Fast(a[1], "extra ranges must be a sequence"));
  const long long page_size = integer(a[7]);
  std::string out;
  put(out, static_cast<uint32_t>(PySequence_Fast_GET_SIZE(requests.p)));
  put(out, static_cast<uint32_t>(PySequence_Fast_GET_SIZE(extra.p)));
  for (int i = 2; i < 7; ++i) put(out, static_cast<uint32_t>(integer(a[i])));
  put(out, uint32_t{0});
  Ints ids;
  for (Py_ssize_t r = 0; r < PySequence_Fast_GET_SIZE(requests.p); ++r) {
    const Ref request(PySequence_Fast(PySequence_Fast_GET_ITEM(requests.p, r), "a request is (source, target, start, end)"));
    if (PySequence_Fast_GET_SIZE(request.p) != 4) bad_value("a request is (source, target, start, end)");
    const Ref source(PySequence_Fast(PySequence_Fast_GET_ITEM(request.p, 0), "block tables must be a sequence"));
    const Ref target(PySequence_Fast(PySequence_Fast_GET_ITEM(request.p, 1), "block tables must be a sequence"));
    const int64_t start = index_of(PySequence_Fast_GET_ITEM(request.p, 2)), end = index_of(PySequence_Fast_GET_ITEM(request.p, 3));
    const Py_ssize_t ns = PySequence_Fast_GET_SIZE(source.p), nt = PySequence_Fast_GET_SIZE(target.p);
    if (ns == 0 || nt == 0 || start < 0 || start >= end) bad_value("invalid KV range");
    const int64_t first = page_size > 0 ? start / page_size : 0;
    int64_t pages = INT64_MAX;  // of the shortest table, counted from the first page that is sent
    for (const Ref* side : {&source, &target}) {
      for (Py_ssize_t p = 0; p < PySequence_Fast_GET_SIZE(side->p); ++p) {
        const int64_t n = length(PySequence_Fast_GET_ITEM(side->p, p)) - first;
        pages = n < pages ? n : pages;
      }
    }
    if (page_size > 0 && pages > (end - 1) / page_size - first + 1) pages = (end - 1) / page_size - first + 1;
    if (pages < 0) pages = 0;
    put(out, static_cast<uint32_t>(ns));
    put(out, static_cast<uint32_t>(nt));
    put(out, static_cast<int64_t>(start - first * page_size));
    put(out, static_cast<int64_t>(end - first * page_size));
    put(out, static_cast<uint32_t>(pages));
    ids.clear();
    for (const Ref* side : {&source, &target}) {
      for (Py_ssize_t p = 0; p < PySequence_Fast_GET_SIZE(side->p); ++p) {
        if (pages > 0) append_range(PySequence_Fast_GET_ITEM(side->p, p), first, first + pages, ids);
      }
    }
    put(out, ids.data(), 4 * ids.size());
  }
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(extra.p); ++i) {
    const Ref triple(PySequence_Fast(PySequence_Fast_GET_ITEM(extra.p, i), "a range is (source, target, bytes)"));
    if (PySequence_Fast_GET_SIZE(triple.p) != 3) bad_value("a range is (source, target, bytes)");
    for (int k = 0; k < 3; ++k) put(out, static_cast<int64_t>(index_of(PySequence_Fast_GET_ITEM(triple.p, k))));
  }
  return PyBytes_FromStringAndSize(out.data(), static_cast<Py_ssize_t>(out.size()));
}

// Records of an all-planes handoff, page by page, and their launch.
struct RequestRecords {
  const RltPool *src, *dst;
  Ints records;
  int words;
  int64_t requests = 0, before = 0, blocks = 0, width = 1;
  RequestRecords(const RltPool* s, const RltPool* d) : src(s), dst(d), words(kRecordHeader + s->num_planes + d->num_planes) {}
  bool fits(int64_t pages) const { return pages <= (1 << 20) && (blocks + pages) * words * 4 <= (1 << 20) && requests < RLT_MAX_REQUESTS; }
  bool valid(const int32_t* ids, int64_t n, const RltPool* pool) const {
    bool ok = true;
    for (int64_t i = 0; i < n; ++i) ok &= static_cast<uint32_t>(ids[i]) < static_cast<uint32_t>(pool->num_blocks);
    return ok;
  }
  // ids: [planes of both sides][stride], the range's first page at column `first_column`
  void add(const int32_t* ids, int64_t stride, int64_t first_column, int64_t first_page, int64_t pages, int64_t start, int64_t end) {
    const int64_t bs = src->block_size;
    const int planes = src->num_planes + dst->num_planes;
    records.reserve(records.size() + static_cast<size_t>(pages * words));
    for (int64_t k = 0; k < pages; ++k) {
      const int64_t base = (first_page + k) * bs;
      const int64_t lo = start > base ? start - base : 0, hi = end < base + bs ? end - base : bs;
      const int32_t head[kRecordHeader] = {static_cast<int32_t>(requests), static_cast<int32_t>(first_page + k), static_cast<int32_t>(lo | hi << 8),
                                           static_cast<int32_t>(base + lo - start), static_cast<int32_t>(before), static_cast<int32_t>(end - start)};
      records.insert(records.end(), head, head + kRecordHeader);
      for (int p = 0; p < planes; ++p) records.push_back(ids[p * stride + first_column + k]);
    }
    ++requests;
    blocks += pages;
    before += end - start;
  }
  int launch(const RltOptions& o, rlt_stream_t stream) const {
    const RltBlockMoves m = moves();
    return rlt_handoff_staged(src, dst, &m, &o, stream);
  }
  RltBlockMoves moves() const {
    RltBlockMoves m = {};
    m.host_records = records.data();
    m.blocks = static_cast<int32_t>(blocks);
    m.words = words;
    m.src_planes = src->num_planes;
    m.dst_planes = dst->num_planes;
    m.block_size = src->block_size;
    m.num_requests = static_cast<int32_t>(requests);
    m.table_width = static_cast<int32_t>(width);
    return m;
  }
};

// A mailbox message: slot address, 56-byte body, stamp.
struct Message {
  void* slot;
  const uint8_t* body;
  uint64_t stamp;
  explicit Message(PyObject* const* a) : slot(address(a[0])) {
    char* bytes = nullptr;
    Py_ssize_t n = 0;
    if (PyBytes_AsStringAndSize(a[1], &bytes, &n) != 0) throw Failure{};
    if (n != 56) bad_value("a message body has 56 bytes");
    body = reinterpret_cast<const uint8_t*>(bytes);
    stamp = PyLong_AsUnsignedLongLong(a[2]);
    if (PyErr_Occurred()) throw Failure{};
  }
  // Posted behind copies of `ranges`, [n](source, destination, bytes): with them where they are few and small.
  int post(const std::vector<int64_t>& ranges, rlt_stream_t stream) const {
    const int rc = rlt_post_behind(ranges.data(), static_cast<int32_t>(ranges.size() / 3), slot, body, stamp, stream);
    return rc == RLT_E_LIMIT ? post_last(ranges, stream) : rc;
  }

 private:
  int post_last(const std::vector<int64_t>& ranges, rlt_stream_t stream) const {
    for (size_t i = 0; i < ranges.size(); i += 3) {
      const int rc = rlt_kv_push(reinterpret_cast<void*>(ranges[i]), reinterpret_cast<void*>(ranges[i + 1]), ranges[i + 2], stream);
      if (rc != RLT_OK) return rc;
    }
    return rlt_kv_post(slot, body, stamp, stream);
  }
};

// The records of [(source tables, target tables, start, end)]; false where something about the requests looks wrong or the library's
// own staging does not hold their records: the general path then does it, or says what is wrong.
bool records_of(PyObject* sequence, RequestRecords& out) {
  const Ref requests(PySequence_Fast(sequence, "requests must be a sequence"));
  const int64_t bs = out.src->block_size;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(requests.p);
  if (n < 1 || bs < 1) return false;
  Ints ids;
  for (Py_ssize_t r = 0; r < n; ++r) {
    const Ref request(PySequence_Fast(PySequence_Fast_GET_ITEM(requests.p, r), "a request is (source, target, start, end)"));
    if (PySequence_Fast_GET_SIZE(request.p) < 4) return false;
    const int64_t start = integer(PySequence_Fast_GET_ITEM(request.p, 2)), end = integer(PySequence_Fast_GET_ITEM(request.p, 3));
    if (start < 0 || start >= end) return false;
    const int64_t first = start / bs, pages = (end - 1) / bs - first + 1;
    if (!out.fits(pages)) return false;
    ids.clear();
    for (int side = 0; side < 2; ++side) {
      const RltPool* pool = side == 0 ? out.src : out.dst;
      const Ref tables(PySequence_Fast(PySequence_Fast_GET_ITEM(request.p, side), "block tables must be a sequence"));
      if (PySequence_Fast_GET_SIZE(tables.p) != pool->num_planes) return false;
      Py_ssize_t of_request = -1;
      const size_t at = ids.size();
      for (int p = 0; p < pool->num_planes; ++p) {
        PyObject* table = PySequence_Fast_GET_ITEM(tables.p, p);
        const Py_ssize_t held = length(table);
        if (held < first + pages || (of_request >= 0 && held != of_request)) return false;
        of_request = held;
        out.width = held > out.width ? held : out.width;
        append_range(table, first, first + pages, ids);
      }
      if (!out.valid(ids.data() + at, static_cast<int64_t>(ids.size() - at), pool)) return false;
    }
    out.add(ids.data(), pages, 0, first, pages, start, end);
  }
  return true;
}

RltOptions slice_of(PyObject* const* a) {  // layer_begin, layer_end, plane_begin, plane_end
  RltOptions o = {};
  o.layer_begin = static_cast<int32_t>(integer(a[0]));
  o.layer_end = static_cast<int32_t>(integer(a[1]));
  o.plane_begin = static_cast<int32_t>(integer(a[2]));
  o.plane_end = static_cast<int32_t>(integer(a[3]));
  return o;
}

// handoff_requests(source pool, destination pool, requests, layer_begin, layer_end, plane_begin, plane_end, device, stream) -> code of an
// all-planes handoff of the requests, or RLT_MOVE_UNSUITED (nothing queued) where records_of leaves them to the general path.
PyObject* handoff_requests(PyObject* const* a) {
  RequestRecords out(static_cast<const RltPool*>(address(a[0])), static_cast<const RltPool*>(address(a[1])));
  if (!records_of(a[2], out)) return PyLong_FromLong(RLT_MOVE_UNSUITED);
  const RltOptions o = slice_of(a + 3);
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[7])));
  const rlt_stream_t stream = stream_of(a[8]);
  return PyLong_FromLong(unlocked([&] { return out.launch(o, stream); }));
}

// push_chunk(source pool, destination pool, requests, [(source address, destination address, bytes)], layer_begin, layer_end, plane_begin,
//            plane_end, slot, body, stamp, device, stream) -> code of handoff_requests, with copies of the ranges and the message behind it
PyObject* push_chunk(PyObject* const* a) {
  RequestRecords out(static_cast<const RltPool*>(address(a[0])), static_cast<const RltPool*>(address(a[1])));
  if (!records_of(a[2], out)) return PyLong_FromLong(RLT_MOVE_UNSUITED);
  std::vector<int64_t> ranges;
  const Ref list(PySequence_Fast(a[3], "ranges must be a sequence"));
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(list.p); ++i) {
    const Ref range(PySequence_Fast(PySequence_Fast_GET_ITEM(list.p, i), "a range is (source, target, bytes)"));
    if (PySequence_Fast_GET_SIZE(range.p) != 3) bad_value("a range is (source, target, bytes)");
    for (int k = 0; k < 3; ++k) ranges.push_back(integer(PySequence_Fast_GET_ITEM(range.p, k)));
  }
  const RltOptions o = slice_of(a + 4);
  const Message message(a + 8);
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[11])));
  const rlt_stream_t stream = stream_of(a[12]);
  return PyLong_FromLong(unlocked([&] {
    const int rc = out.launch(o, stream);
    return rc == RLT_OK ? message.post(ranges, stream) : rc;
  }));
}

// A recorded event of the library's pool.
struct EventObject {
  PyObject_HEAD
  RltEvent* event;
};
PyTypeObject* g_event_type = nullptr;


// An event of the library until a Python object owns it.
struct RecordedEvent {
  RltEvent* event = nullptr;
  ~RecordedEvent() {
    if (event != nullptr) rlt_event_release(event);
  }
  PyObject* object() {
    auto* o = PyObject_New(EventObject, g_event_type);
    if (o == nullptr) throw Failure{};
    o->event = event;
    event = nullptr;
    return reinterpret_cast<PyObject*>(o);
  }
};

// event(timed, device, stream) -> an event recorded there
PyObject* event(PyObject* const* a) {
  const bool timed = PyObject_IsTrue(a[0]) == 1;
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[1])));
  const rlt_stream_t stream = stream_of(a[2]);
  RecordedEvent recorded;
  check_code(unlocked([&] { return rlt_event_record(timed, stream, &recorded.event); }));
  return recorded.object();
}

template <typename V>
bool take(const char*& at, const char* end, V* out) {
  if (end - at < static_cast<ptrdiff_t>(sizeof(V))) return false;
  std::memcpy(out, at, sizeof(V));
  at += sizeof(V);
  return true;
}

// pull_chunk(source pool, destination pool, descriptor, spans, device, stream) -> (begun, done, bytes): the launches that a chunk's
// descriptor (encode_chunk) asks for, between two timing events; None (nothing queued) where handoff_requests would not do.
PyObject* pull_chunk(PyObject* const* a) {
  const auto* src = static_cast<const RltPool*>(address(a[0]));
  const auto* dst = static_cast<const RltPool*>(address(a[1]));
  char* raw = nullptr;
  Py_ssize_t size = 0;
  if (PyBytes_AsStringAndSize(a[2], &raw, &size) != 0) throw Failure{};
  const char *at = raw, *end = raw + size;
  uint32_t head[8];
  if (!take(at, end, &head) || head[2] != RLT_MODE_ALL_PLANES || head[0] == 0) Py_RETURN_NONE;
  const int64_t bs = src->block_size;
  RequestRecords out(src, dst);
  Ints ids;
  for (uint32_t r = 0; r < head[0]; ++r) {
    uint32_t planes[2], columns;
    int64_t range[2];
    if (!take(at, end, &planes) || !take(at, end, &range) || !take(at, end, &columns)) Py_RETURN_NONE;
    if (planes[0] != static_cast<uint32_t>(src->num_planes) || planes[1] != static_cast<uint32_t>(dst->num_planes) || range[0] < 0 ||
        range[0] >= range[1])
      Py_RETURN_NONE;
    const int64_t first = range[0] / bs, pages = (range[1] - 1) / bs - first + 1;
    const size_t count = static_cast<size_t>(planes[0] + planes[1]) * columns;
    if (first + pages > columns || !out.fits(pages) || end - at < static_cast<ptrdiff_t>(4 * count)) Py_RETURN_NONE;
    ids.resize(count);
    std::memcpy(ids.data(), at, 4 * count);
    at += 4 * count;
    const size_t split = static_cast<size_t>(planes[0]) * columns;
    if (!out.valid(ids.data(), static_cast<int64_t>(split), src) || !out.valid(ids.data() + split, static_cast<int64_t>(count - split), dst))
      Py_RETURN_NONE;
    out.width = columns > out.width ? columns : out.width;
    out.add(ids.data(), columns, first, first, pages, range[0], range[1]);
  }
  if (static_cast<size_t>(end - at) / 24 < head[1]) Py_RETURN_NONE;  // the count is another process's word: looked at before it is used
  std::vector<int64_t> extra(3 * static_cast<size_t>(head[1]));
  if (!extra.empty()) std::memcpy(extra.data(), at, 8 * extra.size());
  if (!extra.empty()) {
    const Ref spans(PySequence_Fast(a[3], "spans must be a sequence"));
    for (size_t i = 0; i < extra.size(); i += 3) {
      bool found = false;
      for (Py_ssize_t k = 0; k < PySequence_Fast_GET_SIZE(spans.p) && !found; ++k) {
        const Ref s(PySequence_Fast(PySequence_Fast_GET_ITEM(spans.p, k), "a span is (low, high, base)"));
        const int64_t lo = integer(PySequence_Fast_GET_ITEM(s.p, 0)), hi = integer(PySequence_Fast_GET_ITEM(s.p, 1));
        found = lo <= extra[i] && extra[i] <= hi && extra[i + 2] >= 0 && extra[i + 2] <= hi - extra[i];
        if (found) extra[i] += integer(PySequence_Fast_GET_ITEM(s.p, 2)) - lo;
      }
      if (!found) Py_RETURN_NONE;
    }
  }
  RltOptions o = {};
  o.layer_begin = static_cast<int32_t>(head[3]);
  o.layer_end = static_cast<int32_t>(head[4]);
  o.plane_begin = static_cast<int32_t>(head[5]);
  o.plane_end = static_cast<int32_t>(head[6]);
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[4])));
  const rlt_stream_t stream = stream_of(a[5]);
  RecordedEvent begun, done;
  const int code = unlocked([&] {
    int rc = rlt_event_record(true, stream, &begun.event);
    if (rc == RLT_OK) rc = out.launch(o, stream);
    for (size_t i = 0; rc == RLT_OK && i < extra.size(); i += 3)
      rc = rlt_kv_push(reinterpret_cast<void*>(extra[i]), reinterpret_cast<void*>(extra[i + 1]), extra[i + 2], stream);
    return rc != RLT_OK ? rc : rlt_event_record(true, stream, &done.event);
  });
  if (code == RLT_MOVE_UNSUITED) Py_RETURN_NONE;
  if (code != RLT_OK) return PyLong_FromLong(code);
  const int64_t layers = (head[4] ? head[4] : src->num_layers) - head[3], planes = (head[6] ? head[6] : dst->num_planes) - head[5];
  int64_t bytes = out.before * planes * 2 * layers * (src->codes.token_bytes + (src->scales.key != nullptr ? src->scales.token_bytes : 0));
  for (size_t i = 0; i < extra.size(); i += 3) bytes += extra[i + 2];
  const Ref first(begun.object()), last(done.object());
  return Py_BuildValue("OOL", first.p, last.p, static_cast<long long>(bytes));
}

// pack_segments([(address, bytes, device)], [(address, bytes, device)], [(low, high, base)]) -> the (source, destination, bytes)
// triples as int64, destinations translated by the span that holds them.
PyObject* pack_segments(PyObject* const* a) {
  const Ref local(PySequence_Fast(a[0], "descriptors must be a sequence")), remote(PySequence_Fast(a[1], "descriptors must be a sequence"));
  const Ref spans(PySequence_Fast(a[2], "spans must be a sequence"));
  std::vector<int64_t> span;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(spans.p); ++i) {
    const Ref s(PySequence_Fast(PySequence_Fast_GET_ITEM(spans.p, i), "a span is (low, high, base)"));
    for (int k = 0; k < 3; ++k) span.push_back(integer(PySequence_Fast_GET_ITEM(s.p, k)));
  }
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(local.p);
  if (n != PySequence_Fast_GET_SIZE(remote.p)) bad_value("incompatible source/target KV geometry");
  const Ref out(PyBytes_FromStringAndSize(nullptr, 24 * n));
  auto* triple = reinterpret_cast<int64_t*>(PyBytes_AS_STRING(out.p));
  size_t hit = 0;  // ranges of one tensor follow one another: try the last span first
  for (Py_ssize_t i = 0; i < n; ++i, triple += 3) {
    const Ref s(PySequence_Fast(PySequence_Fast_GET_ITEM(local.p, i), "a descriptor is (address, bytes, device)"));
    const Ref d(PySequence_Fast(PySequence_Fast_GET_ITEM(remote.p, i), "a descriptor is (address, bytes, device)"));
    if (PySequence_Fast_GET_SIZE(s.p) < 2 || PySequence_Fast_GET_SIZE(d.p) < 2) bad_value("a descriptor is (address, bytes, device)");
    const int64_t bytes = integer(PySequence_Fast_GET_ITEM(s.p, 1)), to = integer(PySequence_Fast_GET_ITEM(d.p, 0));
    if (bytes != integer(PySequence_Fast_GET_ITEM(d.p, 1))) bad_value("incompatible source/target KV geometry");
    auto inside = [&](size_t k) { return span[k] <= to && to <= span[k + 1] && bytes <= span[k + 1] - to; };
    if (hit >= span.size() || !inside(hit)) {
      for (hit = 0; hit < span.size() && !inside(hit); hit += 3) {
      }
      if (hit >= span.size()) bad_value("remote descriptor outside the peer's registered memory");
    }
    triple[0] = integer(PySequence_Fast_GET_ITEM(s.p, 0));
    triple[1] = span[hit + 2] + (to - span[hit]);
    triple[2] = bytes;
  }
  Py_INCREF(out.p);
  return out.p;
}

// copy_segments(triples, device, stream) -> code
PyObject* copy_segments(PyObject* const* a) {
  char* data = nullptr;
  Py_ssize_t n = 0;
  if (PyBytes_AsStringAndSize(a[0], &data, &n) != 0) throw Failure{};
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[1])));
  const auto* triples = reinterpret_cast<const int64_t*>(data);
  const rlt_stream_t stream = stream_of(a[2]);
  return PyLong_FromLong(unlocked([&] {
    int rc = RLT_OK;
    for (Py_ssize_t left = n / 24; rc == RLT_OK && left > 0;) {
      const int32_t count = static_cast<int32_t>(left < RLT_INLINE_SEGMENTS ? left : RLT_INLINE_SEGMENTS);
      rc = rlt_copy_segments_inline(triples, count, stream);
      triples += 3 * static_cast<ptrdiff_t>(count);
      left -= count;
    }
    return rc;
  }));
}

// push(source, destination, bytes, device, stream) -> code
PyObject* push(PyObject* const* a) {
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[3])));
  const void* from = address(a[0]);
  void* to = address(a[1]);
  const int64_t bytes = integer(a[2]);
  const rlt_stream_t stream = stream_of(a[4]);
  return PyLong_FromLong(unlocked([&] { return rlt_kv_push(from, to, bytes, stream); }));
}

// post(slot address, 56-byte body, stamp, device, stream) -> code
PyObject* post(PyObject* const* a) {
  char* body = nullptr;
  Py_ssize_t n = 0;
  if (PyBytes_AsStringAndSize(a[1], &body, &n) != 0) throw Failure{};
  if (n != 56) bad_value("a message body has 56 bytes");
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[3])));
  void* slot = address(a[0]);
  const uint64_t stamp = PyLong_AsUnsignedLongLong(a[2]);
  const rlt_stream_t stream = stream_of(a[4]);
  return PyLong_FromLong(unlocked([&] { return rlt_kv_post(slot, reinterpret_cast<const uint8_t*>(body), stamp, stream); }));
}

// load_transport(device, planes) -> code
PyObject* load_transport(PyObject* const* a) {
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[0])));
  const auto planes = static_cast<int32_t>(integer(a[1]));
  return PyLong_FromLong(unlocked([&] { return rlt_load_transport(planes); }));
}

// ------------------------------------------------------------------------------------------------ the module

template <PyObject* (*kFunction)(PyObject* const*), int kArgs>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != kArgs) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", kArgs, n);
    return nullptr;
  }
  try {
    return kFunction(args);
  } catch (const Failure&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

#define RLT_ENTRY(name, function, args) \
  {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&entry<function, args>)), METH_FASTCALL, nullptr}

PyMethodDef kMethods[] = {
    RLT_ENTRY("plan", make_plan, 8),
    RLT_ENTRY("plan_layout", plan_layout, 1),
    RLT_ENTRY("plan_arrays", plan_arrays, 2),
    RLT_ENTRY("plan_wire", plan_wire, 2),
    RLT_ENTRY("plan_fits", plan_fits, 2),
    RLT_ENTRY("plan_upload", plan_upload, 4),
    RLT_ENTRY("capture", capture, 1),
    RLT_ENTRY("move", move, 20),
    RLT_ENTRY("handoff_host", handoff_host, 12),
    RLT_ENTRY("finalize", finalize, 7),
    RLT_ENTRY("encode_chunk", encode_chunk, 8),
    RLT_ENTRY("handoff_requests", handoff_requests, 9),
    RLT_ENTRY("event", event, 3),
    RLT_ENTRY("pull_chunk", pull_chunk, 6),
    RLT_ENTRY("pack_segments", pack_segments, 3),
    RLT_ENTRY("copy_segments", copy_segments, 3),
    RLT_ENTRY("push_chunk", push_chunk, 13),
    RLT_ENTRY("load_transport", load_transport, 2),
    RLT_ENTRY("push", push, 5),
    RLT_ENTRY("post", post, 5),
    RLT_ENTRY("tensor_copy", tensor_copy, 3),
    RLT_ENTRY("fill", fill, 3),
    RLT_ENTRY("upload", upload, 4),
    {nullptr, nullptr, 0, nullptr},
};

// ------------------------------------------------------------------------------------------------ types

template <PyObject* (*kMethod)(PyObject*, PyObject* const*), int kArgs>
PyObject* method(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  if (n != kArgs) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", kArgs, n);
    return nullptr;
  }
  try {
    return kMethod(self, args);
  } catch (const Failure&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}
#define RLT_METHOD(name, function, args) \
  {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&method<function, args>)), METH_FASTCALL, nullptr}

// The same for methods whose arguments may be given by name. kNames: the parameters in order.
template <PyObject* (*kMethod)(PyObject*, PyObject* const*), int kArgs, const char* const* kNames>
PyObject* named_method(PyObject* self, PyObject* const* args, Py_ssize_t n, PyObject* names) {
  const Py_ssize_t named = names == nullptr ? 0 : PyTuple_GET_SIZE(names);
  if (named == 0) return method<kMethod, kArgs>(self, args, n);
  PyObject* all[kArgs] = {};
  for (Py_ssize_t i = 0; i < n && i < kArgs; ++i) all[i] = args[i];
  for (Py_ssize_t k = 0; k < named; ++k) {
    int at = 0;
    while (at < kArgs && PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(names, k), kNames[at]) != 0) ++at;
    if (at == kArgs || all[at] != nullptr) {
      PyErr_Format(PyExc_TypeError, "unexpected argument %R", PyTuple_GET_ITEM(names, k));
      return nullptr;
    }
    all[at] = args[n + k];
  }
  return method<kMethod, kArgs>(self, all, n + named);
}
#define RLT_NAMED_METHOD(name, function, args, names)                                                                    \
  {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&named_method<function, args, names>)),           \
   METH_FASTCALL | METH_KEYWORDS, nullptr}
constexpr const char* kAppendNames[] = {"source", "target"};
constexpr const char* kValuesNames[] = {"values"};
constexpr const char* kWriteNames[] = {"index", "start", "values"};

// The object fields of a type, for the collector: their offsets.
template <size_t... kOffsets>
struct Fields {
  static PyObject*& at(PyObject* self, size_t offset) { return *reinterpret_cast<PyObject**>(reinterpret_cast<char*>(self) + offset); }
  static int traverse(PyObject* self, visitproc visit, void* arg) {
    Py_VISIT(Py_TYPE(self));
    for (size_t offset : {kOffsets...}) Py_VISIT(at(self, offset));
    return 0;
  }
  static int clear(PyObject* self) {
    for (size_t offset : {kOffsets...}) Py_CLEAR(at(self, offset));
    return 0;
  }
  static void dealloc(PyObject* self) {
    PyTypeObject* type = Py_TYPE(self);
    PyObject_GC_UnTrack(self);
    clear(self);
    reinterpret_cast<freefunc>(PyType_GetSlot(type, Py_tp_free))(self);
    Py_DECREF(type);
  }
};

using CopiesFields = Fields<offsetof(CopiesObject, copies)>;
void copies_dealloc(PyObject* self) {
  delete copies_of(self)->batch;
  copies_of(self)->batch = nullptr;
  CopiesFields::dealloc(self);
}
PyObject* copies_new(PyTypeObject* type, PyObject*, PyObject*) {
  PyObject* self = type->tp_alloc(type, 0);
  if (self == nullptr) return nullptr;
  copies_of(self)->batch = new Transfer;
  copies_of(self)->copies = PyList_New(0);
  return self;
}
PyObject* copies_max_rows(PyObject* self, void*) { return PyLong_FromLongLong(copies_of(self)->batch->max_rows); }
PyObject* copies_max_cols(PyObject* self, void*) { return PyLong_FromLongLong(copies_of(self)->batch->max_cols); }

PyMethodDef kCopiesMethods[] = {RLT_METHOD("setup", copies_setup, 4), RLT_METHOD("reset", copies_reset, 0),
                                RLT_NAMED_METHOD("append", copies_append, 2, kAppendNames), RLT_METHOD("append_pieces", copies_append_pieces, 2), RLT_METHOD("launch", copies_launch, 1),
                                {nullptr, nullptr, 0, nullptr}};
PyMemberDef kCopiesMembers[] = {{"copies", Py_T_OBJECT_EX, offsetof(CopiesObject, copies), Py_READONLY, nullptr},
                                {"capacity", Py_T_LONGLONG, offsetof(CopiesObject, capacity), Py_READONLY, nullptr},
                                {nullptr, 0, 0, 0, nullptr}};
PyGetSetDef kCopiesProperties[] = {{"max_rows", copies_max_rows, nullptr, nullptr, nullptr},
                                   {"max_cols", copies_max_cols, nullptr, nullptr, nullptr},
                                   {nullptr, nullptr, nullptr, nullptr, nullptr}};
PyType_Slot kCopiesSlots[] = {{Py_tp_new, reinterpret_cast<void*>(copies_new)},
                              {Py_tp_dealloc, reinterpret_cast<void*>(copies_dealloc)},
                              {Py_tp_traverse, reinterpret_cast<void*>(CopiesFields::traverse)},
                              {Py_tp_clear, reinterpret_cast<void*>(CopiesFields::clear)},
                              {Py_tp_methods, kCopiesMethods},
                              {Py_tp_members, kCopiesMembers},
                              {Py_tp_getset, kCopiesProperties},
                              {0, nullptr}};

using FilledFields = Fields<offsetof(FilledObject, cpu)>;
PyMethodDef kFilledMethods[] = {RLT_NAMED_METHOD("append", filled_append, 1, kValuesNames), {nullptr, nullptr, 0, nullptr}};
PyMemberDef kFilledMembers[] = {{"cpu", Py_T_OBJECT_EX, offsetof(FilledObject, cpu), 0, nullptr},
                                {"count", Py_T_PYSSIZET, offsetof(FilledObject, count), 0, nullptr},
                                {nullptr, 0, 0, 0, nullptr}};
PyType_Slot kFilledSlots[] = {{Py_tp_new, reinterpret_cast<void*>(PyType_GenericNew)},
                              {Py_tp_dealloc, reinterpret_cast<void*>(FilledFields::dealloc)},
                              {Py_tp_traverse, reinterpret_cast<void*>(FilledFields::traverse)},
                              {Py_tp_clear, reinterpret_cast<void*>(FilledFields::clear)},
                              {Py_tp_methods, kFilledMethods},
                              {Py_tp_members, kFilledMembers},
                              {0, nullptr}};

using WritesFields = Fields<offsetof(WritesObject, gpu), offsetof(WritesObject, values), offsetof(WritesObject, targets)>;
PyMethodDef kWritesMethods[] = {RLT_NAMED_METHOD("stage_write", writes_stage, 3, kWriteNames), {nullptr, nullptr, 0, nullptr}};
PyMemberDef kWritesMembers[] = {{"gpu", Py_T_OBJECT_EX, offsetof(WritesObject, gpu), 0, nullptr},
                                {"values", Py_T_OBJECT_EX, offsetof(WritesObject, values), 0, nullptr},
                                {"targets", Py_T_OBJECT_EX, offsetof(WritesObject, targets), 0, nullptr},
                                {nullptr, 0, 0, 0, nullptr}};
PyType_Slot kWritesSlots[] = {{Py_tp_new, reinterpret_cast<void*>(PyType_GenericNew)},
                              {Py_tp_dealloc, reinterpret_cast<void*>(WritesFields::dealloc)},
                              {Py_tp_traverse, reinterpret_cast<void*>(WritesFields::traverse)},
                              {Py_tp_clear, reinterpret_cast<void*>(WritesFields::clear)},
                              {Py_tp_methods, kWritesMethods},
                              {Py_tp_members, kWritesMembers},
                              {0, nullptr}};

PyObject* event_query(PyObject* self, PyObject* const*) {
  RltEvent* event = reinterpret_cast<EventObject*>(self)->event;
  const int fired = unlocked([&] { return rlt_event_query(event); });
  check_code(fired);
  return PyBool_FromLong(fired);
}
PyObject* event_synchronize(PyObject* self, PyObject* const*) {
  RltEvent* event = reinterpret_cast<EventObject*>(self)->event;
  check_code(unlocked([&] { return rlt_event_wait(event); }));
  Py_RETURN_NONE;
}
// order(device, stream): what is queued on that device's stream from now on comes after the event
PyObject* event_order(PyObject* self, PyObject* const* a) {
  RltEvent* event = reinterpret_cast<EventObject*>(self)->event;
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(integer(a[0])));
  const rlt_stream_t stream = stream_of(a[1]);
  check_code(unlocked([&] { return rlt_event_order(event, stream); }));
  Py_RETURN_NONE;
}
PyObject* event_elapsed_time(PyObject* self, PyObject* const* a) {
  if (Py_TYPE(a[0]) != g_event_type) fail(PyExc_TypeError, "expected an event");
  float ms = 0.0f;
  check_code(rlt_event_elapsed(reinterpret_cast<EventObject*>(self)->event, reinterpret_cast<EventObject*>(a[0])->event, &ms));
  return PyFloat_FromDouble(ms);
}
void event_dealloc(PyObject* self) {
  PyTypeObject* type = Py_TYPE(self);
  rlt_event_release(reinterpret_cast<EventObject*>(self)->event);
  PyObject_Free(self);
  Py_DECREF(type);
}
PyMethodDef kEventMethods[] = {RLT_METHOD("query", event_query, 0), RLT_METHOD("synchronize", event_synchronize, 0), RLT_METHOD("order", event_order, 2),
                               RLT_METHOD("elapsed_time", event_elapsed_time, 1), {nullptr, nullptr, 0, nullptr}};
PyType_Slot kEventSlots[] = {{Py_tp_dealloc, reinterpret_cast<void*>(event_dealloc)}, {Py_tp_methods, kEventMethods}, {0, nullptr}};
PyType_Spec kEventType = {"_host.Event", sizeof(EventObject), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_DISALLOW_INSTANTIATION, kEventSlots};

constexpr unsigned kTypeFlags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC;
PyType_Spec kTypes[] = {{"_host.Copies", sizeof(CopiesObject), 0, kTypeFlags, kCopiesSlots},
                        {"_host.Filled", sizeof(FilledObject), 0, kTypeFlags, kFilledSlots},
                        {"_host.Writes", sizeof(WritesObject), 0, kTypeFlags, kWritesSlots}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  if (_import_array() < 0) return nullptr;
  PyObject* module = PyModule_Create(&kModule);
  if (module == nullptr) return nullptr;
  g_event_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&kEventType));
  if (g_event_type == nullptr) return nullptr;
  for (PyType_Spec& spec : kTypes) {
    PyObject* type = PyType_FromSpec(&spec);
    if (type == nullptr || PyModule_AddObject(module, spec.name + sizeof("_host.") - 1, type) != 0) return nullptr;
  }
  return module;
}
