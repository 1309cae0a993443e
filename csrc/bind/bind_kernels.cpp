// pybind11 bindings of the kernel-level C ABI (csrc/kernels/kvt_kernels.h).
// Everything takes raw addresses (int) so that torch tensors, mapped host memory and
// peer-mapped IPC memory are handled alike:  tensor.data_ptr(), stream.cuda_stream.
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "kernels/kvt_kernels.h"

namespace py = pybind11;

namespace kvx {

static void check_cuda(int err, const char* what) {
  if (err != 0) {
    throw std::runtime_error(std::string(what) + ": " + kvt_error_string(err) + " (" + std::to_string(err) + ")");
  }
}

// Host-side packing of a step's requests into the compact device plan: an array of KvtReqDesc followed by the uint32
// block-id pool, in one buffer, which one copy uploads or a launch carries.
struct HostPlan {
  std::string blob;
  uint32_t n_reqs = 0;
  uint32_t total_tiles = 0;
  uint64_t pool_offset = 0;  // byte offset of the block ids inside blob
};

struct PlanPacker {
  const uint32_t tile_tokens, dst_ntpb;
  std::vector<KvtReqDesc> descs;
  std::vector<uint32_t> pool;
  uint32_t tiles = 0;

  // One request: the callables append its block ids of a side to the pool.
  template <typename Src, typename Dst>
  void add(Src&& src_ids, Dst&& dst_ids, uint32_t seen, uint32_t new_tokens, uint32_t flags) {
    KvtReqDesc d{};
    d.src_blk_off = static_cast<uint32_t>(pool.size());
    src_ids(pool);
    d.dst_blk_off = static_cast<uint32_t>(pool.size());
    dst_ids(pool);
    d.n_src_blocks = d.dst_blk_off - d.src_blk_off;
    d.n_dst_blocks = static_cast<uint32_t>(pool.size()) - d.dst_blk_off;
    d.seen_tokens = seen;
    d.new_tokens = new_tokens;
    d.flags = flags;
    d.first_tile = tiles;
    const uint32_t n = kvt_req_tiles(d.seen_tokens, d.new_tokens, tile_tokens, d.flags, dst_ntpb);
    if (n == 0) return;
    tiles += n;
    descs.push_back(d);
  }
  HostPlan finish() const {
    HostPlan out;
    out.n_reqs = static_cast<uint32_t>(descs.size());
    out.total_tiles = tiles;
    out.pool_offset = descs.size() * sizeof(KvtReqDesc);
    out.blob.resize(out.pool_offset + pool.size() * sizeof(uint32_t));
    if (!descs.empty()) std::memcpy(out.blob.data(), descs.data(), out.pool_offset);
    if (!pool.empty()) std::memcpy(out.blob.data() + out.pool_offset, pool.data(), pool.size() * sizeof(uint32_t));
    return out;
  }
};

// (src_blocks, dst_blocks, seen_tokens, new_tokens, flags)
using ReqTuple = std::tuple<std::vector<uint32_t>, std::vector<uint32_t>, uint32_t, uint32_t, uint32_t>;

static void add_tuple(PlanPacker& pk, const ReqTuple& r) {
  auto ids = [](const std::vector<uint32_t>& v) {
    return [&v](std::vector<uint32_t>& pool) { pool.insert(pool.end(), v.begin(), v.end()); };
  };
  pk.add(ids(std::get<0>(r)), ids(std::get<1>(r)), std::get<2>(r), std::get<3>(r), std::get<4>(r));
}

static py::tuple pack_plan(const std::vector<ReqTuple>& reqs, uint32_t tile_tokens, uint32_t dst_ntpb) {
  PlanPacker pk{tile_tokens, dst_ntpb, {}, {}};
  for (const ReqTuple& r : reqs) add_tuple(pk, r);
  const HostPlan p = pk.finish();
  return py::make_tuple(py::bytes(p.blob), p.n_reqs, p.total_tiles, p.pool_offset);
}

// An unsigned 32-bit number: a plain int is read directly, anything else converted as an argument of that type is.
static uint32_t as_u32(PyObject* o) {
  if (PyLong_CheckExact(o)) {
    int beyond = 0;
    const long long v = PyLong_AsLongLongAndOverflow(o, &beyond);
    if (beyond != 0 || v < 0 || v > 0xffffffffll) throw py::type_error("kvt_pack_chunks: number beyond 32 bits");
    return static_cast<uint32_t>(v);
  }
  py::detail::make_caster<uint32_t> any;
  if (!any.load(o, true)) throw py::type_error("kvt_pack_chunks: not a whole number");
  return py::detail::cast_op<uint32_t>(any);
}

// The same from chunk objects (src_blocks, dst_blocks, seen_tokens, new_tokens, pad_tail) without a Python list per table.
// Objects of another class than `plain` are asked for their tuples: the class may say something else there.
static HostPlan pack_chunks(const py::iterable& chunks, uint32_t tile_tokens, uint32_t dst_ntpb, const py::handle plain) {
  // the attributes' names, interned once: making them for each chunk took a third of the time
  static PyObject* const kSrc = PyUnicode_InternFromString("src_blocks");
  static PyObject* const kDst = PyUnicode_InternFromString("dst_blocks");
  static PyObject* const kSeen = PyUnicode_InternFromString("seen_tokens");
  static PyObject* const kNew = PyUnicode_InternFromString("new_tokens");
  static PyObject* const kPad = PyUnicode_InternFromString("pad_tail");
  PlanPacker pk{tile_tokens, dst_ntpb, {}, {}};
  for (const py::handle c : chunks) {
    if (!plain.is_none() && reinterpret_cast<PyObject*>(Py_TYPE(c.ptr())) != plain.ptr()) {
      const py::object tuple = c.attr("as_tuple")();
      py::detail::make_caster<ReqTuple> req;
      if (!req.load(tuple, true)) throw py::type_error("kvt_pack_chunks: not a request's tuple");
      add_tuple(pk, py::detail::cast_op<ReqTuple>(std::move(req)));
      continue;
    }
    auto attr = [&c](PyObject* name) {
      py::object o = py::reinterpret_steal<py::object>(PyObject_GetAttr(c.ptr(), name));
      if (!o) throw py::error_already_set();
      return o;
    };
    auto ids = [&attr](PyObject* name) {
      return [&attr, name](std::vector<uint32_t>& pool) {
        const py::object table = attr(name);
        const py::object seq = py::reinterpret_steal<py::object>(PySequence_Fast(table.ptr(), "block ids are a sequence"));
        if (!seq) throw py::error_already_set();
        for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq.ptr()); ++i) {
          const py::object id = py::reinterpret_borrow<py::object>(PySequence_Fast_GET_ITEM(seq.ptr(), i));
          pool.push_back(as_u32(id.ptr()));
        }
      };
    };
    auto number = [&attr](PyObject* name) {      // int(...) of it
      const py::object whole = py::reinterpret_steal<py::object>(PyNumber_Long(attr(name).ptr()));
      if (!whole) throw py::error_already_set();
      return as_u32(whole.ptr());
    };
    const py::object pad = attr(kPad);
    const int padded = PyObject_IsTrue(pad.ptr());
    if (padded < 0) throw py::error_already_set();
    const uint32_t seen = number(kSeen), fresh = number(kNew);
    pk.add(ids(kSrc), ids(kDst), seen, fresh, padded != 0 ? KVT_REQ_PAD_TAIL : 0u);
  }
  return pk.finish();
}

void bind_kernels(py::module_& m) {
  py::class_<KvtLayout>(m, "KvtLayout")
      .def(py::init([]() { return KvtLayout{}; }))
      .def_readwrite("block_stride", &KvtLayout::block_stride)
      .def_readwrite("kv_stride", &KvtLayout::kv_stride)
      .def_readwrite("token_stride", &KvtLayout::token_stride)
      .def_readwrite("head_stride", &KvtLayout::head_stride)
      .def_readwrite("scale_base", &KvtLayout::scale_base)
      .def_readwrite("scale_kv_stride", &KvtLayout::scale_kv_stride)
      .def_readwrite("scale_token_stride", &KvtLayout::scale_token_stride)
      .def_readwrite("scale_head_stride", &KvtLayout::scale_head_stride)
      .def_readwrite("ntpb", &KvtLayout::ntpb)
      .def_readwrite("num_heads", &KvtLayout::num_heads)
      .def_readwrite("head_bytes", &KvtLayout::head_bytes)
      .def_readwrite("num_blocks", &KvtLayout::num_blocks)
      .def_readwrite("kv_count", &KvtLayout::kv_count);

  py::class_<KvtSegRule>(m, "KvtSegRule")
      .def(py::init([](int64_t so, int64_t dof, int64_t ss, int64_t ds, uint32_t len, uint32_t count) {
             return KvtSegRule{so, dof, ss, ds, len, count};
           }),
           py::arg("src_off"), py::arg("dst_off"), py::arg("src_stride"), py::arg("dst_stride"), py::arg("len"),
           py::arg("count"))
      .def_readwrite("src_off", &KvtSegRule::src_off)
      .def_readwrite("dst_off", &KvtSegRule::dst_off)
      .def_readwrite("src_stride", &KvtSegRule::src_stride)
      .def_readwrite("dst_stride", &KvtSegRule::dst_stride)
      .def_readwrite("len", &KvtSegRule::len)
      .def_readwrite("count", &KvtSegRule::count)
      .def("pack", [](const KvtSegRule& r) {
        return py::bytes(reinterpret_cast<const char*>(&r), sizeof(KvtSegRule));
      });

  m.attr("KVT_MODE_COPY") = static_cast<int>(KVT_MODE_COPY);
  m.attr("KVT_MODE_BF16_TO_MXFP8") = static_cast<int>(KVT_MODE_BF16_TO_MXFP8);
  m.attr("KVT_MODE_MXFP8_TO_BF16") = static_cast<int>(KVT_MODE_MXFP8_TO_BF16);
  m.attr("KVT_REQ_PAD_TAIL") = static_cast<int>(KVT_REQ_PAD_TAIL);
  m.attr("KVT_REQ_DESC_BYTES") = static_cast<int>(sizeof(KvtReqDesc));
  m.attr("KVT_SEG_RULE_BYTES") = static_cast<int>(sizeof(KvtSegRule));
  m.attr("KVT_TENSOR_MAP_BYTES") = 128;

  m.attr("KVT_PLAN_IN_LAUNCH") = static_cast<int>(KVT_PLAN_IN_LAUNCH);

  py::class_<HostPlan>(m, "HostPlan")
      .def_readonly("n_reqs", &HostPlan::n_reqs)
      .def_readonly("total_tiles", &HostPlan::total_tiles)
      .def_readonly("pool_offset", &HostPlan::pool_offset)
      .def_property_readonly("nbytes", [](const HostPlan& p) { return p.blob.size(); })
      .def_property_readonly("sizes", [](const HostPlan& p) { return py::make_tuple(p.n_reqs, p.total_tiles, p.pool_offset, p.blob.size()); },
                             "(n_reqs, total_tiles, pool_offset, nbytes) in one look: four cost a plan 0.15 us more")
      .def_property_readonly("blob", [](const HostPlan& p) { return py::bytes(p.blob); })
      .def("copy_to_device", [](const HostPlan& p, uint64_t dst, uint64_t after) {
        if (!p.blob.empty()) check_cuda(kvt_copy_now(dst, p.blob.data(), p.blob.size(), reinterpret_cast<void*>(after)), "kvt_copy_now");
      }, py::arg("dst"), py::arg("after"), py::call_guard<py::gil_scoped_release>(),
           "The plan at a device address, behind the event `after`, complete on return and outside of any capture.");
  m.def("kvt_pack_chunks", &pack_chunks, py::arg("chunks"), py::arg("tile_tokens"), py::arg("dst_ntpb"), py::arg("plain") = py::none());
  m.def("kvt_stream_capturing", [](uint64_t stream) { return kvt_stream_capturing(reinterpret_cast<void*>(stream)) != 0; });

  m.def("kvt_req_tiles", &kvt_req_tiles);
  m.def("kvt_pack_plan", &pack_plan, py::arg("reqs"), py::arg("tile_tokens"), py::arg("dst_ntpb"),
        "Pack [(src_blocks, dst_blocks, seen, new, flags)] into (blob, n_reqs, total_tiles, pool_offset).");

  m.def(
      "kvt_encode_tensor_map",
      [](uint64_t base, const KvtLayout& l, uint32_t box_heads, uint32_t box_tokens, uint32_t token_inner) {
        alignas(64) char buf[128];
        const int r = kvt_encode_tensor_map_ordered(buf, base, &l, box_heads, box_tokens, token_inner);
        if (r != 0) throw std::runtime_error("cuTensorMapEncodeTiled failed: " + std::to_string(r));
        return py::bytes(buf, 128);
      },
      py::arg("base"), py::arg("layout"), py::arg("box_heads"), py::arg("box_tokens"), py::arg("token_inner") = 0);
  m.def("kvt_tile_is_flat", [](const KvtLayout& l, uint32_t n_heads, uint32_t tile_tokens, uint32_t token_inner) {
    return kvt_tile_is_flat(&l, n_heads, tile_tokens, token_inner) != 0;
  });

  m.def(
      "kvt_launch_p2d_attn",
      [](uint64_t src_layers, uint64_t dst_layers, uint64_t src_maps, uint64_t dst_maps, const KvtLayout& src,
         const KvtLayout& dst, uint32_t layer_begin, uint32_t layer_end, uint64_t reqs, uint32_t n_reqs,
         uint32_t total_tiles, uint64_t block_ids, uint32_t tile_tokens, uint32_t src_head0, uint32_t dst_head0,
         uint32_t n_heads, uint32_t mode, uint64_t status, uint64_t done_counter, uint64_t flag,
         uint64_t flag_value, int grid, int threads, int use_tma, uint64_t stream, uint32_t simt_tile,
         uint32_t dst_remote, uint32_t tile_order, uint32_t store_form, uint32_t tma_stages, uint32_t cache_hint,
         const HostPlan* plan) {
        KvtAttnLaunch a{};
        if (plan != nullptr) {
          a.plan = plan->blob.data();
          a.plan_bytes = static_cast<uint32_t>(std::min<size_t>(plan->blob.size(), 0xffffffffu));
        }
        a.simt_tile = simt_tile;
        a.dst_remote = dst_remote;
        a.tile_order = tile_order;
        a.store_form = store_form;
        a.tma_stages = tma_stages;
        a.cache_hint = cache_hint;
        a.src_layers = reinterpret_cast<const uint64_t*>(src_layers);
        a.dst_layers = reinterpret_cast<const uint64_t*>(dst_layers);
        a.src_maps = reinterpret_cast<const void*>(src_maps);
        a.dst_maps = reinterpret_cast<const void*>(dst_maps);
        a.src = src;
        a.dst = dst;
        a.layer_begin = layer_begin;
        a.layer_end = layer_end;
        a.reqs = reinterpret_cast<const KvtReqDesc*>(reqs);
        a.n_reqs = n_reqs;
        a.total_tiles = total_tiles;
        a.block_ids = reinterpret_cast<const uint32_t*>(block_ids);
        a.tile_tokens = tile_tokens;
        a.src_head0 = src_head0;
        a.dst_head0 = dst_head0;
        a.n_heads = n_heads;
        a.mode = mode;
        a.status = reinterpret_cast<uint32_t*>(status);
        a.done_counter = reinterpret_cast<uint32_t*>(done_counter);
        a.flag = reinterpret_cast<uint64_t*>(flag);
        a.flag_value = flag_value;
        check_cuda(kvt_launch_p2d_attn(&a, grid, threads, use_tma, reinterpret_cast<void*>(stream)),
                   "kvt_launch_p2d_attn");
      },
      py::arg("src_layers"), py::arg("dst_layers"), py::arg("src_maps"), py::arg("dst_maps"), py::arg("src"),
      py::arg("dst"), py::arg("layer_begin"), py::arg("layer_end"), py::arg("reqs"), py::arg("n_reqs"),
      py::arg("total_tiles"), py::arg("block_ids"), py::arg("tile_tokens"), py::arg("src_head0"),
      py::arg("dst_head0"), py::arg("n_heads"), py::arg("mode"), py::arg("status"), py::arg("done_counter"),
      py::arg("flag"), py::arg("flag_value"), py::arg("grid"), py::arg("threads"), py::arg("use_tma"),
      py::arg("stream"), py::arg("simt_tile") = 0, py::arg("dst_remote") = 0, py::arg("tile_order") = 0,
      py::arg("store_form") = 0, py::arg("tma_stages") = 0, py::arg("cache_hint") = 0, py::arg("plan") = nullptr);

  m.def(
      "kvt_launch_p2d_state",
      [](uint64_t src_layers, uint64_t dst_layers, uint32_t layer_begin, uint32_t layer_end,
         int64_t src_block_stride, int64_t dst_block_stride, uint32_t src_num_blocks, uint32_t dst_num_blocks,
         uint64_t src_blocks, uint64_t dst_blocks, uint32_t n_pages, uint64_t rules, uint32_t n_rules,
         uint64_t status, uint64_t done_counter, uint64_t flag, uint64_t flag_value, int grid, int threads,
         uint64_t stream) {
        KvtStateLaunch a{};
        a.src_layers = reinterpret_cast<const uint64_t*>(src_layers);
        a.dst_layers = reinterpret_cast<const uint64_t*>(dst_layers);
        a.layer_begin = layer_begin;
        a.layer_end = layer_end;
        a.src_block_stride = src_block_stride;
        a.dst_block_stride = dst_block_stride;
        a.src_num_blocks = src_num_blocks;
        a.dst_num_blocks = dst_num_blocks;
        a.src_blocks = reinterpret_cast<const uint32_t*>(src_blocks);
        a.dst_blocks = reinterpret_cast<const uint32_t*>(dst_blocks);
        a.n_pages = n_pages;
        a.rules = reinterpret_cast<const KvtSegRule*>(rules);
        a.n_rules = n_rules;
        a.status = reinterpret_cast<uint32_t*>(status);
        a.done_counter = reinterpret_cast<uint32_t*>(done_counter);
        a.flag = reinterpret_cast<uint64_t*>(flag);
        a.flag_value = flag_value;
        check_cuda(kvt_launch_p2d_state(&a, grid, threads, reinterpret_cast<void*>(stream)), "kvt_launch_p2d_state");
      },
      py::arg("src_layers"), py::arg("dst_layers"), py::arg("layer_begin"), py::arg("layer_end"),
      py::arg("src_block_stride"), py::arg("dst_block_stride"), py::arg("src_num_blocks"),
      py::arg("dst_num_blocks"), py::arg("src_blocks"), py::arg("dst_blocks"), py::arg("n_pages"),
      py::arg("rules"), py::arg("n_rules"), py::arg("status"), py::arg("done_counter"), py::arg("flag"),
      py::arg("flag_value"), py::arg("grid"), py::arg("threads"), py::arg("stream"));

  m.def(
      "kvt_launch_copy_blocks",
      [](uint64_t src_base, uint64_t dst_base, uint64_t triples, uint32_t n, uint64_t src_cap, uint64_t dst_cap,
         uint64_t status, int grid, uint64_t stream) {
        check_cuda(kvt_launch_copy_blocks(src_base, dst_base, reinterpret_cast<const uint64_t*>(triples), n,
                                          src_cap, dst_cap, reinterpret_cast<uint32_t*>(status), grid,
                                          reinterpret_cast<void*>(stream)),
                   "kvt_launch_copy_blocks");
      },
      py::arg("src_base"), py::arg("dst_base"), py::arg("triples"), py::arg("n"), py::arg("src_capacity"),
      py::arg("dst_capacity"), py::arg("status"), py::arg("grid"), py::arg("stream"));

  m.def(
      "kvt_launch_copy_blocks_multi",
      [](const std::vector<uint64_t>& src_bases, const std::vector<uint64_t>& dst_bases,
         const std::vector<uint64_t>& src_caps, const std::vector<uint64_t>& dst_caps, const std::vector<uint32_t>& first,
         const std::vector<uint32_t>& count, uint64_t triples, uint64_t status, int grid, uint64_t stream,
         uint32_t bulk_rounds) {
        const size_t nt = src_bases.size();
        if (nt == 0 || nt > KVT_COPY_MAX_TENSORS || dst_bases.size() != nt || src_caps.size() != nt ||
            dst_caps.size() != nt || first.size() != nt || count.size() != nt)
          throw std::invalid_argument("kvt_launch_copy_blocks_multi: 1..8 entries, every list of that length");
        KvtCopyMulti a{};
        for (size_t t = 0; t < nt; ++t) {
          a.src_base[t] = src_bases[t];
          a.dst_base[t] = dst_bases[t];
          a.src_cap[t] = src_caps[t];
          a.dst_cap[t] = dst_caps[t];
          a.first[t] = first[t];
          a.count[t] = count[t];
        }
        a.n_tensors = static_cast<uint32_t>(nt);
        a.triples = reinterpret_cast<const uint64_t*>(triples);
        a.status = reinterpret_cast<uint32_t*>(status);
        if (bulk_rounds > 0) {
          check_cuda(kvt_launch_copy_blocks_bulk(&a, bulk_rounds, grid, reinterpret_cast<void*>(stream)),
                     "kvt_launch_copy_blocks_bulk");
        } else {
          check_cuda(kvt_launch_copy_blocks_multi(&a, grid, reinterpret_cast<void*>(stream)), "kvt_launch_copy_blocks_multi");
        }
      },
      py::arg("src_bases"), py::arg("dst_bases"), py::arg("src_caps"), py::arg("dst_caps"), py::arg("first"),
      py::arg("count"), py::arg("triples"), py::arg("status"), py::arg("grid"), py::arg("stream"),
      py::arg("bulk_rounds") = 0);
  m.def("kvt_bulk_rounds", &kvt_bulk_rounds, py::arg("first_len"), py::arg("max_len"));

  m.def(
      "kvt_launch_mc_fanout",
      [](uint64_t src_layers, uint64_t mc_layers, uint32_t layer_begin, uint32_t layer_end, int64_t src_block_stride,
         int64_t dst_block_stride, uint32_t src_num_blocks, uint32_t dst_num_blocks, uint64_t src_blocks,
         uint64_t dst_blocks, uint32_t n_blocks, uint32_t block_off, uint32_t block_len, uint64_t status,
         uint64_t done_counter, uint64_t mc_flag, uint64_t flag_value, int grid, uint64_t stream) {
        KvtMcFanout a{};
        a.src_layers = reinterpret_cast<const uint64_t*>(src_layers);
        a.mc_layers = reinterpret_cast<const uint64_t*>(mc_layers);
        a.layer_begin = layer_begin;
        a.layer_end = layer_end;
        a.src_block_stride = src_block_stride;
        a.dst_block_stride = dst_block_stride;
        a.src_num_blocks = src_num_blocks;
        a.dst_num_blocks = dst_num_blocks;
        a.src_blocks = reinterpret_cast<const uint32_t*>(src_blocks);
        a.dst_blocks = reinterpret_cast<const uint32_t*>(dst_blocks);
        a.n_blocks = n_blocks;
        a.block_off = block_off;
        a.block_len = block_len;
        a.status = reinterpret_cast<uint32_t*>(status);
        a.done_counter = reinterpret_cast<uint32_t*>(done_counter);
        a.mc_flag = reinterpret_cast<uint64_t*>(mc_flag);
        a.flag_value = flag_value;
        check_cuda(kvt_launch_mc_fanout(&a, grid, reinterpret_cast<void*>(stream)), "kvt_launch_mc_fanout");
      },
      py::arg("src_layers"), py::arg("mc_layers"), py::arg("layer_begin"), py::arg("layer_end"),
      py::arg("src_block_stride"), py::arg("dst_block_stride"), py::arg("src_num_blocks"), py::arg("dst_num_blocks"),
      py::arg("src_blocks"), py::arg("dst_blocks"), py::arg("n_blocks"), py::arg("block_off"), py::arg("block_len"),
      py::arg("status"), py::arg("done_counter"), py::arg("mc_flag"), py::arg("flag_value"), py::arg("grid"),
      py::arg("stream"));

  m.def("kvt_launch_copy_blocks_cast",
        [](uint64_t src_base, uint64_t dst_base, uint64_t triples, uint32_t n, uint64_t src_cap, uint64_t dst_cap,
           uint64_t status, int grid, uint64_t stream) {
          check_cuda(kvt_launch_copy_blocks_cast(src_base, dst_base, reinterpret_cast<const uint64_t*>(triples), n, src_cap,
                                                 dst_cap, reinterpret_cast<uint32_t*>(status), grid,
                                                 reinterpret_cast<void*>(stream)),
                     "kvt_launch_copy_blocks_cast");
        },
        py::arg("src_base"), py::arg("dst_base"), py::arg("triples"), py::arg("n"), py::arg("src_capacity"),
        py::arg("dst_capacity"), py::arg("status"), py::arg("grid"), py::arg("stream"));
  // end-to-end transfer check: the CPU function, and the kernel over device arrays of {off u64, len u32, index0 u32}
  m.def("kvt_checksum_host", [](py::buffer data, uint32_t index0) {
    const py::buffer_info bi = data.request();
    return kvt_checksum_host(bi.ptr, static_cast<uint64_t>(bi.size) * static_cast<uint64_t>(bi.itemsize), index0);
  }, py::arg("data"), py::arg("index0") = 0);
  m.def("kvt_launch_checksum",
        [](uint64_t bases, uint32_t n_bases, uint64_t capacity, uint64_t chunks, uint32_t n, uint64_t out, uint64_t status,
           int grid, uint64_t stream) {
          check_cuda(kvt_launch_checksum(reinterpret_cast<const uint64_t*>(bases), n_bases, capacity,
                                         reinterpret_cast<const KvtCheckChunk*>(chunks), n, reinterpret_cast<uint64_t*>(out),
                                         reinterpret_cast<uint32_t*>(status), grid, reinterpret_cast<void*>(stream)),
                     "kvt_launch_checksum");
        },
        py::arg("bases"), py::arg("n_bases"), py::arg("capacity"), py::arg("chunks"), py::arg("n"), py::arg("out"),
        py::arg("status"), py::arg("grid"), py::arg("stream"));
  // the row form: device arrays of {blk_off, n_blocks, seen, new_tokens, first, index} (u32 x 6) and of block ids
  m.def("kvt_launch_checksum_attn",
        [](uint64_t bases, uint32_t n_bases, uint64_t capacity, const KvtLayout& layout, uint32_t head0, uint32_t n_heads,
           uint64_t reqs, uint32_t n_reqs, uint32_t total_tokens, uint64_t pool, uint32_t pool_len, uint64_t out, uint64_t status,
           int grid, uint64_t stream) {
          check_cuda(kvt_launch_checksum_attn(reinterpret_cast<const uint64_t*>(bases), n_bases, capacity, &layout, head0, n_heads,
                                              reinterpret_cast<const KvtCheckReq*>(reqs), n_reqs, total_tokens,
                                              reinterpret_cast<const uint32_t*>(pool), pool_len, reinterpret_cast<uint64_t*>(out),
                                              reinterpret_cast<uint32_t*>(status), grid, reinterpret_cast<void*>(stream)),
                     "kvt_launch_checksum_attn");
        },
        py::arg("bases"), py::arg("n_bases"), py::arg("capacity"), py::arg("layout"), py::arg("head0"), py::arg("n_heads"),
        py::arg("reqs"),
        py::arg("n_reqs"), py::arg("total_tokens"), py::arg("pool"), py::arg("pool_len"), py::arg("out"), py::arg("status"),
        py::arg("grid"), py::arg("stream"));
  m.def("kvt_bf16_to_e4m3", [](uint16_t bits) { return static_cast<int>(kvt_bf16_to_e4m3(bits)); });

  m.def("kvt_launch_wait_flag", [](uint64_t flag, uint64_t value, uint64_t timeout_ns, uint64_t status,
                                   uint64_t stream) {
    check_cuda(kvt_launch_wait_flag(reinterpret_cast<const uint64_t*>(flag), value, timeout_ns,
                                    reinterpret_cast<uint32_t*>(status), reinterpret_cast<void*>(stream)),
               "kvt_launch_wait_flag");
  });
  m.def("kvt_launch_set_flag", [](uint64_t flag, uint64_t value, uint64_t stream) {
    check_cuda(kvt_launch_set_flag(reinterpret_cast<uint64_t*>(flag), value, reinterpret_cast<void*>(stream)),
               "kvt_launch_set_flag");
  });

  m.def("kvt_device_count", &kvt_device_count);
  m.def("kvt_can_access_peer", &kvt_can_access_peer);
  m.def("kvt_enable_peer_access",
        [](int dev, int peer) { check_cuda(kvt_enable_peer_access(dev, peer), "cudaDeviceEnablePeerAccess"); });
  m.def("kvt_p2p_attribute", &kvt_p2p_attribute);
  m.def("kvt_sm_count", &kvt_sm_count);
  m.def("kvt_ipc_get_handle", [](uint64_t ptr) {
    char h[64];
    uint64_t base = 0, size = 0;
    check_cuda(kvt_ipc_get_handle(ptr, h, &base, &size), "cudaIpcGetMemHandle");
    return py::make_tuple(py::bytes(h, 64), base, size);
  });
  m.def("kvt_ipc_open_handle", [](const std::string& h) {
    if (h.size() != 64) throw std::runtime_error("IPC handle must be 64 bytes");
    uint64_t p = 0;
    check_cuda(kvt_ipc_open_handle(h.data(), &p), "cudaIpcOpenMemHandle");
    return p;
  });
  m.def("kvt_ipc_close", [](uint64_t p) { check_cuda(kvt_ipc_close(p), "cudaIpcCloseMemHandle"); });
  m.def("kvt_malloc", [](uint64_t bytes) {
    uint64_t p = 0;
    check_cuda(kvt_malloc(bytes, &p), "cudaMalloc");
    return p;
  });
  m.def("kvt_free", [](uint64_t p) { check_cuda(kvt_free(p), "cudaFree"); });
  m.def("kvt_host_alloc_mapped", [](uint64_t bytes) {
    uint64_t h = 0, d = 0;
    check_cuda(kvt_host_alloc_mapped(bytes, &h, &d), "cudaHostAlloc");
    return py::make_tuple(h, d);
  });
  m.def("kvt_host_free", [](uint64_t p) { check_cuda(kvt_host_free(p), "cudaFreeHost"); });
  m.def("kvt_host_register", [](uint64_t p, uint64_t bytes) {
    uint64_t d = 0;
    check_cuda(kvt_host_register(p, bytes, &d), "cudaHostRegister");
    return d;
  });
  m.def("kvt_memcpy_async", [](uint64_t dst, uint64_t src, uint64_t bytes, uint64_t stream) {
    check_cuda(kvt_memcpy_async(dst, src, bytes, reinterpret_cast<void*>(stream)), "cudaMemcpyAsync");
  });
  m.def("kvt_memcpy_triples", [](uint64_t dst_base, uint64_t src_base, py::buffer triples, uint64_t stream) {
    const py::buffer_info bi = triples.request();
    if (bi.itemsize != 8 || bi.size % 3 != 0) throw std::invalid_argument("triples: a contiguous array of u64, 3 per copy");
    py::gil_scoped_release nogil;
    check_cuda(kvt_memcpy_triples(dst_base, src_base, static_cast<const uint64_t*>(bi.ptr),
                                  static_cast<uint32_t>(bi.size / 3), reinterpret_cast<void*>(stream)),
               "cudaMemcpyAsync");
  }, py::arg("dst_base"), py::arg("src_base"), py::arg("triples"), py::arg("stream"));
  m.def("kvt_host_unregister", [](uint64_t p) { check_cuda(kvt_host_unregister(p), "cudaHostUnregister"); });
}

}  // namespace kvx
