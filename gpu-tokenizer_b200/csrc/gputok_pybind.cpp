// gputok_pybind.cpp -- Python module `gputok_gpu`: the reference's pybind
// surface (PYBIND11_MODULE(gputok_gpu, m), gputok_binding.cu:1015-1065) as a
// thin wrapper over the C ABI of include/gputok_b200.h.  No CUDA code here.
//
//   GpuTokenizer(merges_path, chunk_tokens=2048, max_iters=50, device=0)
//   .tokenize_batch(texts, merge_rule="greedy") -> (list[list[int]], kernel_ms)
//   .tokenize_batch_blockbpe_base(texts) -> (list[list[int]], kernel_ms)
//   .tokenize_batch_cpu(texts, merge_rule="greedy") -> list[list[int]]
// plus array-returning variants that skip the per-token Python objects:
//   .encode_packed(texts, mode="opt")    -> (ids int32[N], text_offsets int64[T+1],
//                                            chunk_offsets int64[C+1], kernel_ms)
//   .decode(ids) -> bytes, .table_info() -> dict, .stage_ms() -> dict
//
// Exceptions follow the reference: chunk_tokens <= 0 -> ValueError
// (std::invalid_argument, :661-663), unreadable/empty merges -> RuntimeError;
// CUDA failures raise RuntimeError instead of terminating the process (:24-30).
#include <pybind11/numpy.h>
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include <cstring>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/gputok_b200.h"

namespace py = pybind11;

namespace {

[[noreturn]] void raise_status(int rc, const std::string& msg)
{
  if (rc == GTK_ERR_INVALID_ARG) throw std::invalid_argument(msg);
  if (rc == GTK_ERR_MEMORY) throw std::bad_alloc();
  throw std::runtime_error(msg);
}

class GpuTokenizer {
 public:
  GpuTokenizer(const std::string& merges_path, int chunk_tokens, int max_iters, int device)
  {
    int rc = gtk_create(merges_path.c_str(), chunk_tokens, max_iters, device, &h_);
    if (rc != GTK_OK) raise_status(rc, gtk_global_error());
  }
  ~GpuTokenizer()
  {
    for (PyObject* o : id_objects_) Py_XDECREF(o);
    gtk_destroy(h_);
  }
  GpuTokenizer(const GpuTokenizer&) = delete;
  GpuTokenizer& operator=(const GpuTokenizer&) = delete;

  // One call at a time from collecting the strings to reading the result.  Waiting happens without the GIL, which the holder needs.
  class Turn {
   public:
    explicit Turn(GpuTokenizer& t) : lock_(t.mu_, std::try_to_lock)
    {
      if (lock_.owns_lock()) return;
      py::gil_scoped_release nogil;
      lock_.lock();
    }

   private:
    std::unique_lock<std::mutex> lock_;
  };

  // Where the strings lie and their offsets, UTF-8 as pybind's str -> std::string caster gives it to the reference; they are
  // gathered inside the call (gtk_encode_strings).  `keep` holds them meanwhile: the caller's list may change while
  // the GIL is released.
  struct Keep {
    py::object items;
    std::vector<std::string> strings;
  };
  void collect(const py::object& texts, Keep& keep)
  {
    PyObject* seq = texts.ptr();
    if (PyList_Check(seq) || PyTuple_Check(seq)) {
      keep.items = PyTuple_Check(seq) ? texts : py::reinterpret_steal<py::object>(PyList_AsTuple(seq));
      if (!keep.items) throw py::error_already_set();
      const Py_ssize_t n = PyTuple_GET_SIZE(keep.items.ptr());
      parts_.resize(size_t(n));
      off_.resize(size_t(n) + 1);
      int64_t total = 0;
      bool plain    = true;
      for (Py_ssize_t i = 0; i < n && plain; ++i) {
        PyObject* o = PyTuple_GET_ITEM(keep.items.ptr(), i);
        if (i + 16 < n) __builtin_prefetch(PyTuple_GET_ITEM(keep.items.ptr(), i + 16));  // strings lie all over the heap
        Py_ssize_t len = 0;
        const char* p  = nullptr;
        if (PyUnicode_Check(o)) {
          if (PyUnicode_IS_COMPACT_ASCII(o)) {
            p   = reinterpret_cast<const char*>(PyUnicode_1BYTE_DATA(o));
            len = PyUnicode_GET_LENGTH(o);
          } else {
            p = PyUnicode_AsUTF8AndSize(o, &len);
          }
        }
        plain             = p != nullptr;
        off_[size_t(i)]   = total;
        parts_[size_t(i)] = reinterpret_cast<const uint8_t*>(p);
        total += len;
      }
      off_[size_t(n)] = total;
      if (plain) return;
      PyErr_Clear();  // something else than str, or a str without a UTF-8 form: the caster below decides
    }
    try {
      keep.strings = texts.cast<std::vector<std::string>>();
    } catch (const py::cast_error&) {
      throw py::type_error("texts must be a sequence of str or bytes");
    }
    parts_.clear();
    off_.assign(1, 0);
    for (auto& t : keep.strings) {
      parts_.push_back(reinterpret_cast<const uint8_t*>(t.data()));
      off_.push_back(off_.back() + int64_t(t.size()));
    }
  }
  size_t n_texts() const { return off_.size() - 1; }

  void check(int rc) const
  {
    if (rc != GTK_OK) raise_status(rc, gtk_last_error(h_));
  }

  // (list[list[int]], kernel_ms); ([], 0.0) for an empty batch or a batch of
  // empty texts, as gputok_binding.cpp:707-709, 734-736.
  py::tuple lists_from_result(size_t n_texts, float kernel_ms)
  {
    int64_t n_ids = 0, n_chunks = 0;
    gtk_result_sizes(h_, &n_ids, &n_chunks, nullptr);
    py::list batch;
    if (n_texts == 0 || n_chunks == 0) return py::make_tuple(batch, 0.0);
    return py::make_tuple(id_lists(n_texts), double(kernel_ms));
  }

  // The last result as list[list[int]].  The int objects of the vocabulary are made once and shared (they are immutable, as
  // Python's own small ints are): a reference count instead of an allocation per id.
  py::list id_lists(size_t n_texts)
  {
    const int32_t* ids;
    const int64_t* toff;
    gtk_result_view(h_, &ids, &toff, nullptr);
    PyObject* batch = PyList_New(Py_ssize_t(n_texts));
    if (!batch) throw py::error_already_set();
    py::list owner = py::reinterpret_steal<py::list>(batch);
    for (size_t t = 0; t < n_texts; ++t) {
      const int64_t lo = toff[t], n = toff[t + 1] - lo;
      PyObject* one    = PyList_New(Py_ssize_t(n));
      if (!one) throw py::error_already_set();
      PyList_SET_ITEM(batch, Py_ssize_t(t), one);
      for (int64_t i = 0; i < n; ++i) {
        const size_t id = size_t(uint32_t(ids[lo + i]));
        if (id >= id_objects_.size()) id_objects_.resize(id + id / 2 + 1024, nullptr);
        PyObject*& o = id_objects_[id];
        if (!o && !(o = PyLong_FromLong(long(id)))) throw py::error_already_set();
        Py_INCREF(o);
        PyList_SET_ITEM(one, Py_ssize_t(i), o);
      }
    }
    return owner;
  }

  py::tuple tokenize(const py::object& texts, int mode)
  {
    Turn turn(*this);
    Keep keep;
    collect(texts, keep);
    float ms = 0.f;
    int rc;
    {
      py::gil_scoped_release nogil;
      rc = gtk_encode_strings(h_, mode, parts_.data(), off_.data(), int64_t(n_texts()), &ms);
    }
    check(rc);
    return lists_from_result(n_texts(), ms);
  }

  py::list tokenize_cpu(const py::object& texts, const std::string& rule)
  {
    int r;
    if (rule == "greedy") r = GTK_RULE_GREEDY;
    else if (rule == "localmin") r = GTK_RULE_LOCALMIN;
    else throw std::invalid_argument("merge_rule must be 'greedy' or 'localmin'");
    Turn turn(*this);
    Keep keep;
    collect(texts, keep);
    std::vector<uint8_t> bytes(size_t(off_.back()));
    for (size_t t = 0; t < n_texts(); ++t)
      if (off_[t + 1] > off_[t]) std::memcpy(bytes.data() + off_[t], parts_[t], size_t(off_[t + 1] - off_[t]));
    int rc;
    {
      py::gil_scoped_release nogil;
      rc = gtk_encode_cpu(h_, r, bytes.data(), off_.data(), int64_t(n_texts()));
    }
    check(rc);
    return id_lists(n_texts());
  }

  py::tuple encode_packed(const py::object& texts, const std::string& mode)
  {
    int m;
    if (mode == "opt") m = GTK_MODE_OPT;
    else if (mode == "base") m = GTK_MODE_BASE;
    else throw std::invalid_argument("mode must be 'opt' or 'base'");
    Turn turn(*this);
    Keep keep;
    collect(texts, keep);
    float ms = 0.f;
    int rc;
    {
      py::gil_scoped_release nogil;
      rc = gtk_encode_strings(h_, m, parts_.data(), off_.data(), int64_t(n_texts()), &ms);
    }
    check(rc);
    int64_t n_ids = 0, n_chunks = 0;
    gtk_result_sizes(h_, &n_ids, &n_chunks, nullptr);
    const int64_t n_text_off = int64_t(n_texts()) + 1, n_chunk_off = n_chunks + 1;
    // large results are taken over, not copied: the arrays look at the page-locked memory that the ids were downloaded to
    constexpr int64_t kTakeBytes = 128 << 10;
    gtk_taken* taken = 4 * n_ids + 8 * (n_text_off + n_chunk_off) >= kTakeBytes ? gtk_result_take(h_) : nullptr;
    if (taken) {
      py::capsule owner(taken, [](void* p) { gtk_result_release(static_cast<gtk_taken*>(p)); });
      const int32_t* ids;
      const int64_t *toff, *coff;
      gtk_result_view(h_, &ids, &toff, &coff);
      return py::make_tuple(py::array_t<int32_t>(n_ids, ids, owner), py::array_t<int64_t>(n_text_off, toff, owner),
                            py::array_t<int64_t>(n_chunk_off, coff, owner), double(ms));
    }
    py::array_t<int32_t> ids(n_ids);
    py::array_t<int64_t> toff(n_text_off), coff(n_chunk_off);
    check(gtk_result_copy(h_, ids.mutable_data(), n_ids, toff.mutable_data(), coff.mutable_data(), n_chunk_off));
    return py::make_tuple(ids, toff, coff, double(ms));
  }

  py::bytes decode(const std::vector<int32_t>& ids) const
  {
    int64_t n = 0;
    check(gtk_decode(h_, ids.data(), int64_t(ids.size()), nullptr, 0, &n));
    std::string out(size_t(n), '\0');
    check(gtk_decode(h_, ids.data(), int64_t(ids.size()), reinterpret_cast<uint8_t*>(&out[0]), n, &n));
    return py::bytes(out);
  }

  py::dict table_info() const
  {
    gtk_table_info ti;
    check(gtk_table_info_get(h_, &ti));
    py::dict d;
    d["vocab_size"] = ti.vocab_size;
    d["num_merges"] = ti.num_merges;
    d["max_rank"] = ti.max_rank;
    d["hash_capacity"] = ti.hash_capacity;
    d["hash_overflow_entries"] = ti.hash_overflow_entries;
    d["hash_bytes"] = ti.hash_bytes;
    d["monotone"] = bool(ti.monotone);
    d["merged_is_256_plus_rank"] = bool(ti.merged_is_256_plus_rank);
    d["byte_ids_identity"] = bool(ti.byte_ids_identity);
    d["adj_bigrams"] = ti.adj_bigrams;
    d["chunk_tokens"] = ti.chunk_tokens;
    d["max_iters"] = ti.max_iters;
    d["device"] = ti.device;
    d["sm_count"] = ti.sm_count;
    d["whole_segment_entries"] = ti.whole_segment_entries;
    d["whole_segment_dropped"] = ti.whole_segment_dropped;
    return d;
  }

  void set_stage_timing(bool per_stage) { check(gtk_set_stage_timing(h_, per_stage ? 1 : 0)); }

  py::dict stage_ms() const
  {
    float ms[5];
    int32_t launches = 0;
    check(gtk_last_stage_ms(h_, ms, &launches));
    py::dict d;
    d["chunker"] = ms[0];
    d["merge"] = ms[1];
    d["scan"] = ms[2];
    d["pack"] = ms[3];
    d["pipeline"] = ms[4];
    d["kernel_launches"] = launches;
    return d;
  }

 private:
  gtk_tokenizer* h_ = nullptr;
  std::mutex mu_;  // see Turn; guards what follows
  std::vector<int64_t> off_;
  std::vector<const uint8_t*> parts_;
  std::vector<PyObject*> id_objects_;
};

}  // namespace

PYBIND11_MODULE(gputok_gpu, m)
{
  m.doc() = "B200-native greedy byte-level BPE tokenizer (drop-in for the reference's gputok_gpu module)";
  m.attr("__version__") = gtk_version();

  py::class_<GpuTokenizer>(m, "GpuTokenizer")
    .def(py::init<const std::string&, int, int, int>(), py::arg("merges_path"), py::arg("chunk_tokens") = 2048,
         py::arg("max_iters") = 50, py::arg("device") = 0)
    .def("tokenize_batch", [](GpuTokenizer& self, const py::object& texts, const std::string& rule) {
           if (rule == "greedy") return self.tokenize(texts, GTK_MODE_OPT);
           if (rule == "localmin") return self.tokenize(texts, GTK_MODE_LOCALMIN);
           throw std::invalid_argument("merge_rule must be 'greedy' or 'localmin'");
         }, py::arg("texts"), py::arg("merge_rule") = "greedy",
         "Tokenize a batch of UTF-8 strings with the segment-parallel kernel (greedy rule).\n"
         "merge_rule='localmin' runs the reference method's own rule (local minimum, max_iters passes,\n"
         "per chunk) on the GPU instead.  Returns (list[list[int]], kernel_time_ms).")
    .def("tokenize_batch_blockbpe_base", [](GpuTokenizer& self, const py::object& texts) {
           return self.tokenize(texts, GTK_MODE_BASE);
         }, py::arg("texts"),
         "Tokenize with the one-CTA-per-chunk Algorithm 1 kernel.\n"
         "Returns (list[list[int]], kernel_time_ms).")
    .def("tokenize_batch_cpu", &GpuTokenizer::tokenize_cpu, py::arg("texts"), py::arg("merge_rule") = "greedy",
         "Host reference tokenizer. merge_rule='greedy' (default) is the rule the GPU paths\n"
         "implement, per chunk; 'localmin' is the reference method's own rule on the whole text.")
    .def("encode_packed", &GpuTokenizer::encode_packed, py::arg("texts"), py::arg("mode") = "opt",
         "Returns (ids int32[N], text_offsets int64[T+1], chunk_offsets int64[C+1], kernel_time_ms).")
    .def("decode", &GpuTokenizer::decode, py::arg("ids"))
    .def("table_info", &GpuTokenizer::table_info)
    .def("stage_ms", &GpuTokenizer::stage_ms)
    .def("set_stage_timing", [](GpuTokenizer& self, bool per_stage) { self.set_stage_timing(per_stage); },
         py::arg("per_stage"),
         "Time every stage of a batch (stage_ms()['chunker'/'merge'/'scan'/'pack']) instead of the pipeline as a\n"
         "whole; off by default.");
}
