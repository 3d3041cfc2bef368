// Host side of attention calls with a single rank, in native code.
//
// A forward is one or two launches, a backward three or four.  Driven from Python small calls waited for the host; most
// of its time went into checks, slices, argument objects and result tensors between the launches.  Here the pieces that
// do not change between calls (tables, arenas, sizes) are laid out once per program, and a call checks its tensors,
// allocates its results and launches.  Host time (8 query heads, 4040 tokens in four sequences): forward 37 -> 8 us,
// backward 105 -> 17, the whole call with autograd 221 -> 100; with 64 fp32 channels 71 -> 9, 110 -> 17 and 302 -> 100.
//
// Only plain calls are taken: tensors on the arenas' device, contiguous, 16-byte aligned, of a type the row kernels
// read.  For anything else the functions return nothing before they launch anything, and the caller goes the general
// way.
#include <ATen/ATen.h>
#include <c10/core/DeviceGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <nvtx3/nvToolsExt.h>
#include <pybind11/stl.h>
#include <torch/csrc/utils/pybind.h>

#include <memory>
#include <optional>
#include <stdexcept>
#include <string>
#include <tuple>
#include <utility>

#include "entries.h"

namespace py = pybind11;
using at::Tensor;

namespace {

constexpr int kHeadDim = 128;   // channels of an arena row

void check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string(what) + " failed with code " + std::to_string(rc));
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }   // of the current device

// The row kernels' number of a type, -1 for one they do not take.
int row_type(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return 0;
    case at::kHalf: return 1;
    case at::kBFloat16: return 2;
    default: return -1;
  }
}

// A call: on the arenas' device, whichever is current, and a range for a profiler.
struct Call {
  c10::DeviceGuard device;
  Call(const char* name, const Tensor& arena) : device(arena.device()) { nvtxRangePushA(name); }
  ~Call() { nvtxRangePop(); }
};

// One program's launches.  Holds its tables and the arenas; nothing in it changes after construction, so threads may
// share it (what they compute shares the arenas all the same).
class SingleRankAttention {
 public:
  Tensor q, kv, dout, lse, dq, dkv, part_out, part_lse, status;      // arenas
  Tensor tiles, kv_entries, fwd_masks, ctas, items, bwd_masks;       // tables
  int n_tiles = 0, n_ctas = 0, max_items = 0, dq_levels = 0;
  long q_local_rows = 0, kv_local_rows = 0, q_rows = 0, kv_rows = 0;
  bool has_bwd = false, all_rows_written = true;
  int channels = kHeadDim;

  // bf16 rows of 128 channels that the attention kernels read or write in place
  bool arena_like(const Tensor& t, long least, long heads) const {
    return plain(t) && t.scalar_type() == at::kBFloat16 && t.dim() >= 3 && t.size(-1) == kHeadDim && t.size(0) >= least &&
           t.numel() == t.size(0) * heads * kHeadDim;
  }
  bool statistics(const Tensor& t) const {
    return t.device() == q.device() && t.layout() == at::kStrided && t.scalar_type() == at::kFloat && t.dim() == 2 &&
           t.size(0) == q.size(1) && t.size(1) >= q_local_rows && t.is_contiguous() && !t.is_neg();
  }
  bool plain(const Tensor& t) const {
    return t.device() == q.device() && t.layout() == at::kStrided && t.is_contiguous() && !t.is_neg() &&
           reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
  }
  bool rows_of(const Tensor& t, long rows, long heads, int d) const {
    return plain(t) && row_type(t) >= 0 && t.numel() == rows * heads * d;
  }

  void launch_forward(const Tensor& q_in, const Tensor& kv_in, const Tensor& o, const Tensor& l, double scale,
                      int out_type = 2, int out_channels = kHeadDim) const {
    void* outs[2] = {part_out.data_ptr(), o.data_ptr()};
    float* lses[2] = {part_lse.data_ptr<float>(), l.data_ptr<float>()};
    check(dcpk_attn_fwd_pair(q_in.const_data_ptr(), q_in.size(0), kv_in.const_data_ptr(), kv_in.size(0), int(q.size(1)),
                             int(kv.size(2)), tiles.const_data_ptr(), n_tiles, kv_entries.const_data_ptr(),
                             int(kv_entries.size(0)), fwd_masks.const_data_ptr(), int(fwd_masks.size(0)), outs, lses, 2,
                             int(part_lse.size(1)), int(l.size(1)), 1, out_type, out_channels, float(scale), channels, nullptr, 0, nullptr,
                             nullptr, 0, status.data_ptr<int>(), stream()),
          "dcpk_attn_fwd_pair");
  }

  // The levels of dQ, in memory of this call's own (null: none).
  std::pair<Tensor, DcpkDqLevels> levels_of_call() const {
    const long bytes = dcpk_attn_bwd_workspace(int(items.size(0)), q_local_rows, int(q.size(1)), channels, dq_levels);
    Tensor memory;
    if (bytes > 0) memory = at::empty({bytes}, q.options().dtype(at::kByte));
    return {memory, {items.const_data_ptr(), int(items.size(0)), dq_levels, int(q_local_rows), int(q.size(1)), channels,
                     bytes > 0 ? memory.data_ptr() : nullptr}};
  }

  // delta and cleared accumulators, then the gradients; `o` and `d_in`: at least the local rows, of `d` channels.
  // Other than rows of 128 in bf16 go to the arena of dO on the way.
  void launch_backward(const Tensor& q_in, const Tensor& d_in, const Tensor& kv_in, const Tensor& o, const Tensor& l, const Tensor& dl,
                       int d, const DcpkDqLevels& levels, bool sum_levels, double scale) const {
    const long hq = q.size(1), hkv = kv.size(2);
    const bool in_place = d == kHeadDim && d_in.scalar_type() == at::kBFloat16;
    const Tensor& d_o = in_place ? d_in : dout;
    if (in_place)
      check(dcpk_attn_bwd_prep(o.const_data_ptr(), d_in.const_data_ptr(), dl.data_ptr<float>(), int(q_local_rows), int(hq),
                               int(dl.size(1)), dq.data_ptr<float>(), q_rows * hq * kHeadDim, dkv.data_ptr<float>(),
                               kv_rows * 2 * hkv * kHeadDim, &levels, stream()),
            "dcpk_attn_bwd_prep");
    else
      check(dcpk_attn_bwd_prep_cast(row_type(d_in), o.const_data_ptr(), d_in.const_data_ptr(), d, dout.data_ptr(), dl.data_ptr<float>(),
                                    int(q_local_rows), int(hq), int(dl.size(1)), dq.data_ptr<float>(), q_rows * hq * kHeadDim,
                                    dkv.data_ptr<float>(), kv_rows * 2 * hkv * kHeadDim, &levels, stream()),
            "dcpk_attn_bwd_prep_cast");
    nvtxMarkA("bwd:dout copy, delta, zero accumulators");
    nvtxMarkA("bwd:wait inputs of peers");
    float* dqs[1] = {dq.data_ptr<float>()};
    float* dkvs[1] = {dkv.data_ptr<float>()};
    check(dcpk_attn_bwd(q_in.const_data_ptr(), d_o.const_data_ptr(), q_local_rows, kv_in.const_data_ptr(), kv_in.size(0), int(hq),
                        int(hkv), ctas.const_data_ptr(), n_ctas, items.const_data_ptr(), int(items.size(0)), max_items,
                        bwd_masks.const_data_ptr(), int(bwd_masks.size(0)), l.const_data_ptr<float>(), dl.const_data_ptr<float>(),
                        int(l.size(1)), dqs, dkvs, 1, float(scale), channels, dq_levels, levels.workspace,
                        sum_levels ? 2 : 0, nullptr, 0, nullptr, nullptr, 0,
                        status.data_ptr<int>(), stream()),
          "dcpk_attn_bwd");
    nvtxMarkA("bwd:kernels (with operand fetch)");
  }

  // ---- operands and results where the caller has them; false: not taken
  bool forward_into(const Tensor& q_in, const Tensor& kv_in, const Tensor& o, const Tensor& l, double scale) const {
    if (!arena_like(q_in, q_local_rows, q.size(1)) || !arena_like(kv_in, kv_local_rows, 2 * kv.size(2)) || kv_in.dim() != 4 ||
        !arena_like(o, q_local_rows, q.size(1)) || !statistics(l))
      return false;
    Call call("dcp.attention.fwd", q);
    nvtxMarkA("fwd:wait inputs of peers");
    launch_forward(q_in, kv_in, o, l, scale);
    nvtxMarkA("fwd:kernels (with operand fetch)");
    nvtxMarkA("fwd:wait partials of peers");
    nvtxMarkA("fwd:merge");
    return true;
  }

  bool backward_from(const Tensor& d_o, const Tensor& q_in, const Tensor& kv_in, const Tensor& o, const Tensor& l,
                     const std::optional<Tensor>& dl, double scale) const {
    if (!has_bwd || !arena_like(q_in, q_local_rows, q.size(1)) || !arena_like(kv_in, kv_local_rows, 2 * kv.size(2)) || kv_in.dim() != 4 ||
        !arena_like(d_o, q_local_rows, q.size(1)) || d_o.size(0) != q_local_rows || !arena_like(o, q_local_rows, q.size(1)) || !statistics(l))
      return false;
    Call call("dcp.attention.bwd", q);
    const auto [memory, levels] = levels_of_call();
    launch_backward(q_in, d_o, kv_in, o, l, dl ? *dl : at::empty_like(l), kHeadDim, levels, true, scale);
    return true;
  }

  // ---- any head dimension and row type; results are the caller's own
  using Forward = std::optional<std::tuple<Tensor, Tensor, int>>;   // output, lse, entries called
  Forward forward(const Tensor& q_in, const Tensor& kv_in, int d, double scale) const {
    const long hq = q.size(1), hkv = kv.size(2);
    if (!rows_of(q_in, q_local_rows, hq, d) || !rows_of(kv_in, kv_local_rows, 2 * hkv, d) || q_in.scalar_type() != kv_in.scalar_type())
      return std::nullopt;
    Call call("dcp.attention.fwd", q);
    const bool in_place = d == kHeadDim && q_in.scalar_type() == at::kBFloat16;
    int entries = 1;
    Tensor o, l;
    const auto form = q.options().dtype(q_in.scalar_type());
    if (all_rows_written) {
      o = at::empty({q_local_rows, hq, d}, form);
      l = at::empty({hq, q_local_rows}, lse.options());
    } else {
      o = at::zeros({q_local_rows, hq, d}, form);
      l = at::zeros({hq, q_local_rows}, lse.options());
    }
    if (!in_place) {
      check(dcpk_pad_cast_rows(row_type(q_in), q_in.const_data_ptr(), q.data_ptr(), q_local_rows * hq, kv_in.const_data_ptr(),
                               kv.data_ptr(), kv_local_rows * 2 * hkv, d, stream()),
            "dcpk_pad_cast_rows");
      ++entries;
    }
    nvtxMarkA("fwd:wait inputs of peers");
    if (in_place) launch_forward(q_in.view({q_local_rows, hq, kHeadDim}), kv_in.view({kv_local_rows, 2, hkv, kHeadDim}), o, l, scale);
    else launch_forward(q, kv, o, l, scale, row_type(q_in), d);
    nvtxMarkA("fwd:kernels (with operand fetch)");
    nvtxMarkA("fwd:wait partials of peers");
    nvtxMarkA("fwd:merge");
    return std::make_tuple(o, l, entries);
  }

  // `reload`: the arenas do not hold q and kv (asked only where they are not read in place)
  using Backward = std::optional<std::tuple<Tensor, Tensor, int>>;   // dq, dkv, entries called
  Backward backward(const Tensor& q_in, const Tensor& kv_in, const Tensor& o_in, const Tensor& do_in, const Tensor& l_in, int d,
                    bool reload, double scale) const {
    const long hq = q.size(1), hkv = kv.size(2);
    if (!has_bwd || !rows_of(q_in, q_local_rows, hq, d) || !rows_of(kv_in, kv_local_rows, 2 * hkv, d) ||
        !rows_of(o_in, q_local_rows, hq, d) || !rows_of(do_in, q_local_rows, hq, d) || q_in.scalar_type() != kv_in.scalar_type() ||
        o_in.scalar_type() != do_in.scalar_type() || l_in.numel() != hq * q_local_rows)
      return std::nullopt;
    if (l_in.device() != q.device() || l_in.scalar_type() != at::kFloat || l_in.layout() != at::kStrided || !l_in.is_contiguous() ||
        l_in.is_neg())
      return std::nullopt;
    const Tensor l = l_in.view({hq, q_local_rows});
    Call call("dcp.attention.bwd", q);
    const bool in_place = d == kHeadDim && q_in.scalar_type() == at::kBFloat16;
    int entries = 3;
    if (!in_place && reload) {
      check(dcpk_pad_cast_rows(row_type(q_in), q_in.const_data_ptr(), q.data_ptr(), q_local_rows * hq, kv_in.const_data_ptr(),
                               kv.data_ptr(), kv_local_rows * 2 * hkv, d, stream()),
            "dcpk_pad_cast_rows");
      ++entries;
    }
    const auto [memory, levels] = levels_of_call();
    launch_backward(in_place ? q_in : q, do_in, in_place ? kv_in.view({kv_local_rows, 2, hkv, kHeadDim}) : kv, o_in, l, at::empty_like(l),
                    d, levels, false, scale);
    Tensor gq = at::empty({q_local_rows, hq, d}, q.options().dtype(q_in.scalar_type()));
    Tensor gkv = at::empty({kv_local_rows, 2, hkv, d}, q.options().dtype(kv_in.scalar_type()));
    if (levels.workspace)
      check(dcpk_cut_cast_gradients(row_type(gq), &levels, dq.const_data_ptr<float>(), gq.data_ptr(), dkv.const_data_ptr<float>(),
                                    gkv.data_ptr(), kv_local_rows * 2 * hkv, d, stream()),
            "dcpk_cut_cast_gradients");
    else
      check(dcpk_cut_cast_rows(1, row_type(gq), dq.const_data_ptr(), gq.data_ptr(), q_local_rows * hq, dkv.const_data_ptr(),
                               gkv.data_ptr(), kv_local_rows * 2 * hkv, d, stream()),
            "dcpk_cut_cast_rows");
    return std::make_tuple(gq, gkv, entries);
  }
};

}  // namespace

PYBIND11_MODULE(_calls, m) {
  using A = SingleRankAttention;
  auto free_gil = py::call_guard<py::gil_scoped_release>();   // a launch may wait for room in the stream's queue
  py::class_<A>(m, "SingleRankAttention")
      .def(py::init([](const py::dict& d) {
        auto a = std::make_unique<A>();
        auto tensor = [&](const char* k) { return d[k].cast<Tensor>(); };
        for (auto [k, t] : {std::pair<const char*, Tensor*>{"q", &a->q}, {"kv", &a->kv}, {"dout", &a->dout}, {"lse", &a->lse},
                            {"dq", &a->dq}, {"dkv", &a->dkv}, {"part_out", &a->part_out},
                            {"part_lse", &a->part_lse}, {"status", &a->status}, {"tiles", &a->tiles},
                            {"kv_entries", &a->kv_entries}, {"fwd_masks", &a->fwd_masks}})
          *t = tensor(k);
        a->has_bwd = d.contains("ctas");
        if (a->has_bwd) {
          a->ctas = tensor("ctas"), a->items = tensor("items"), a->bwd_masks = tensor("bwd_masks");
          a->n_ctas = d["n_ctas"].cast<int>(), a->max_items = d["max_items"].cast<int>();
          a->dq_levels = d["dq_levels"].cast<int>();
        }
        a->n_tiles = d["n_tiles"].cast<int>();
        a->q_local_rows = d["q_local_rows"].cast<long>(), a->kv_local_rows = d["kv_local_rows"].cast<long>();
        a->q_rows = d["q_rows"].cast<long>(), a->kv_rows = d["kv_rows"].cast<long>();
        a->all_rows_written = d["all_rows_written"].cast<bool>(), a->channels = d["channels"].cast<int>();
        const long rq = a->q.size(0), rkv = a->kv.size(0);
        if (a->q_local_rows > rq || a->kv_local_rows > rkv || a->q_rows > a->dq.size(0) || a->kv_rows > a->dkv.size(0))
          throw std::invalid_argument("the program's rows do not fit the arenas");
        return a;
      }))
      .def("forward_into", &A::forward_into, free_gil)
      .def("backward_from", &A::backward_from, free_gil)
      .def("forward", &A::forward, free_gil)
      .def("backward", &A::backward, free_gil);
}
