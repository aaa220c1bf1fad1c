// Python module functs_b200._C: the pass entry points under the names the reference binds
// (functs/csrc/jit/python/init.cpp:31-76).  Graphs are mutated in place; every function returns None.
#include <torch/csrc/jit/python/pybind_utils.h>
#include <torch/extension.h>

#include <torch/csrc/jit/api/compilation_unit.h>
#include <torch/csrc/jit/api/module.h>
#include <torch/csrc/jit/passes/freeze_module.h>
#include <torch/csrc/jit/passes/shape_analysis.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>

#include "../../../include/functs_b200.h"
#include "detect.h"
#include "fusion.h"
#include "tensorssa.h"

namespace py = pybind11;
using torch::jit::Graph;

namespace {
// What a kernel may be pointed at: float32 on `device`.
void checkInput(const at::Tensor& t, const at::Device& device, const char* name) {
    TORCH_CHECK_VALUE(t.is_cuda(), name, " must be a CUDA tensor (functs_b200 has no CPU path)");
    TORCH_CHECK_VALUE(t.device() == device, name, " must be on ", device, ", not on ", t.device());
    TORCH_CHECK_TYPE(t.scalar_type() == at::kFloat, name, " must be torch.float32");
}
// The same for memory that a kernel writes, or reads as it lies.
void checkBuffer(const at::Tensor& t, const at::Device& device, at::ScalarType dtype, at::IntArrayRef sizes, const char* name) {
    TORCH_CHECK_VALUE(t.device() == device && t.scalar_type() == dtype && t.is_contiguous() && t.sizes() == sizes, name, " must be a contiguous ",
                      dtype, " tensor of sizes ", sizes, " on ", device);
}

// Appends (dets, labels) to a Python list, from code that runs without the interpreter lock.
functs_b200::EmitImage appendTo(py::list& out) {
    return [&out](functs_b200::Detections&& d) {
        py::gil_scoped_acquire gil;
        out.append(py::make_tuple(std::move(d.dets), std::move(d.labels)));
    };
}
}  // namespace

PYBIND11_MODULE(_C, m) {
    m.doc() = "functs_b200: TensorSSA functionalization passes + immut:: operator registrations (loaded as a side effect)";
    py::class_<functs_b200::MutateInfo, std::shared_ptr<functs_b200::MutateInfo>>(m, "TensorSSAMutateInfo")
        .def(py::init<>())
        .def_property_readonly("mutValues", [](functs_b200::MutateInfo& self) { return self.mutValues; })
        .def_property_readonly("mutNodes", [](functs_b200::MutateInfo& self) { return self.mutNodes; });
    m.def("_jit_pass_remove_inplace", [](std::shared_ptr<Graph> g) { functs_b200::RemoveInplace(g); });
    m.def("_jit_pass_dumb_remove_inter_precedure_mutation",
          [](std::shared_ptr<Graph> g) { functs_b200::DumbRemoveInterPrecedureMutation(g); });
    m.def("_jit_pass_convert_to_tensorssa", [](std::shared_ptr<Graph> g) { functs_b200::ConvertToTensorSSA(g); });
    m.def("_jit_pass_tensorssa_remove_update", [](std::shared_ptr<Graph> g) { functs_b200::TensorSSARemoveUpdate(g); });
    m.def("_jit_pass_rewrite_mutation", [](std::shared_ptr<Graph> g, std::shared_ptr<functs_b200::MutateInfo> info) {
        functs_b200::TensorSSARewriteMutation(g, *info);
    });
    m.def("_jit_pass_block_propagation", [](std::shared_ptr<Graph> g, std::shared_ptr<functs_b200::MutateInfo> info) {
        functs_b200::TensorSSAPropagation(g, *info);
    });
    m.def("_jit_pass_rename", [](std::shared_ptr<Graph> g) { functs_b200::TensorSSARename(g); });
    // loop parallelization, grouping, functor lowering (reference: fait passes behind _jit_pass_fait_pipeline)
    m.def("_jit_pass_parallelize_loops", [](std::shared_ptr<Graph> g) { functs_b200::ParallelizeLoops(g); });
    m.def("_jit_pass_fait_fuse_ops", [](std::shared_ptr<Graph> g, py::object /*refined_types*/) { functs_b200::FuseOps(g); },
          py::arg("graph"), py::arg("refined_types") = py::none());
    // the reference's grouper for graphs that did not go through the ParallelMap pipeline (functs.jit.script(backend="jit"),
    // functs/csrc/jit/python/init.cpp:40-42 -> FuncTsFuseTensorExprs): here the same entry point groups the fusable ops of a
    // functionalized graph and lowers the groups to tssa::ParallelFunctor nodes, which run as one launch each
    m.def("_jit_pass_fuse_tensorexpr", [](std::shared_ptr<Graph> g) {
        functs_b200::FuseOps(g);
        functs_b200::LowerToParallelFunctors(g);
    });
    m.def("_jit_pass_match_precompiled_loops", [](std::shared_ptr<Graph> g) { functs_b200::MatchPrecompiledLoops(g); });
    m.def("_jit_pass_unroll_loops_with_deps", [](std::shared_ptr<Graph> g) { functs_b200::UnrollLoopsWithDeps(g); });
    m.def("_jit_pass_split_parallel_maps", [](std::shared_ptr<Graph> g) { functs_b200::SplitParallelMaps(g); });
    m.def("_jit_pass_unroll_simple_maps", [](std::shared_ptr<Graph> g) { functs_b200::UnrollSimpleMaps(g); });
    m.def("_jit_pass_lower_to_parallel_functors", [](std::shared_ptr<Graph> g) { functs_b200::LowerToParallelFunctors(g); });
    m.def("_jit_pass_fait_pipeline",
          [](std::shared_ptr<Graph> g, std::vector<c10::TypePtr> type_hint) {
              // the type hints refine the graph inputs (shapes / dtypes), as the reference's pipeline does first
              for (size_t i = 0; i < type_hint.size() && i < g->inputs().size(); ++i) {
                  // (a tuple hint describes the elements of a list input; the list type itself cannot carry it)
                  if (type_hint[i] && !(type_hint[i]->cast<c10::TupleType>() && g->inputs()[i]->type()->cast<c10::ListType>()))
                      g->inputs()[i]->setType(type_hint[i]);
              }
              functs_b200::FaitPipeline(g);
          },
          py::arg("graph"), py::arg("type_hint") = std::vector<c10::TypePtr>());
    m.def("_jit_pass_fait_shape_infer",
          [](std::shared_ptr<Graph> g, std::vector<c10::TypePtr> type_hint, py::object refined_types) {
              // refined_types (a dict, as in the reference's binding): filled with value -> tuple type of every list of
              // tensors whose elements' types are known; the same pairs are returned keyed by the values' debug names
              auto pairs = functs_b200::InferShapesRefined(g, type_hint);
              py::dict by_name;
              for (auto& kv : pairs) {
                  by_name[py::str(kv.first->debugName())] = kv.second;
                  if (!refined_types.is_none()) refined_types[py::cast(kv.first)] = kv.second;
              }
              return by_name;
          },
          py::arg("graph"), py::arg("type_hint") = std::vector<c10::TypePtr>(), py::arg("refined_types") = py::none());
    // precompiled regions: pattern programs are registered from Python (functs_b200/patterns.py)
    m.def("_jit_pass_prepare_for_matching", [](std::shared_ptr<Graph> g) { functs_b200::PrepareForMatching(g); });
    m.def("_jit_pass_match_precompiled_regions", [](std::shared_ptr<Graph> g) { return functs_b200::MatchPrecompiledRegions(g); });
    m.def("_describe_region",
          [](std::shared_ptr<Graph> g, std::vector<int64_t> fwild, std::vector<int64_t> iwild) {
              auto d = functs_b200::DescribeRegion(g, fwild, iwild);
              py::dict out;
              out["signature"] = d.signature;
              out["num_nodes"] = d.num_nodes;
              out["num_inputs"] = d.num_inputs;
              out["num_outputs"] = d.num_outputs;
              out["num_tensors"] = d.num_tensors;
              out["fconsts"] = d.fconsts;
              out["iconsts"] = d.iconsts;
              return out;
          },
          py::arg("graph"), py::arg("fwild") = std::vector<int64_t>(), py::arg("iwild") = std::vector<int64_t>());
    m.def("_register_region_pattern",
          [](const std::string& name, std::shared_ptr<Graph> g, std::vector<std::pair<std::string, int64_t>> froles,
             std::vector<std::pair<std::string, int64_t>> iroles) { functs_b200::RegisterRegionPattern(name, g, froles, iroles); });
    m.def("_region_pattern_count", []() { return functs_b200::RegionPatternCount(); });
    m.def("_interpreted_functor_runs", []() { return functs_b200::InterpretedFunctorRuns(); });
    m.def("_generic_group_runs", []() { return functs_b200::GenericGroupRuns(); });
    m.def("_last_generic_refusal", []() { return functs_b200::LastGenericRefusal(); });
    m.def("_functor_regions", [](std::shared_ptr<Graph> g) {
        // adapter name of every tssa::ParallelFunctor node ("" = interpreted), in graph order
        std::vector<std::string> out;
        std::function<void(torch::jit::Block*)> visit = [&](torch::jit::Block* b) {
            for (torch::jit::Node* n : b->nodes()) {
                if (n->kind() == c10::Symbol::fromQualString("tssa::ParallelFunctor")) out.push_back(functs_b200::RegionSignature(n));
                for (torch::jit::Block* nb : n->blocks()) visit(nb);
            }
        };
        visit(g->block());
        return out;
    });
    // whole detection calls (functs_b200/workloads.py): one (dets, labels) pair per image
    m.def("_ssd_detect",
          [](const at::Tensor& loc, const at::Tensor& conf, const at::Tensor& priors, double clamp_max, double score_thr, int64_t topk,
             double iou_thr) {
              py::list out;
              {
                  py::gil_scoped_release release;
                  functs_b200::ssdDetect(loc, conf, priors, clamp_max, score_thr, topk, iou_thr, functs_b200::Lists::kOwn, appendTo(out));
              }
              return out;
          });
    m.def("_yolo_detect", [](std::vector<at::Tensor> maps, const std::vector<int64_t>& sizes, at::Device device, double score_thr,
                             int64_t topk, double iou_thr) {
        py::list out;
        {
            py::gil_scoped_release release;
            TORCH_CHECK_VALUE(maps.size() == 3 && sizes.size() == 3, "expected three [B, 255, S, S] maps");
            for (size_t l = 0; l < 3; ++l) {
                at::Tensor& t = maps[l];
                TORCH_CHECK_VALUE(t.dim() == 4 && t.size(1) == 255, "expected three [B, 255, S, S] maps");
                TORCH_CHECK_VALUE(t.size(2) == sizes[l] && t.size(3) == sizes[l], "map ", l, " is not of the configured size ", sizes[l]);
                TORCH_CHECK_TYPE(t.scalar_type() == at::kFloat, "pred map must be float32");
                if (t.device() != device) t = t.to(device, t.scalar_type(), /*non_blocking=*/true);
                t = t.contiguous();
            }
            functs_b200::yoloDetect(maps, score_thr, topk, iou_thr, /*dense=*/false, functs_b200::Lists::kOwn, appendTo(out));
        }
        return out;
    });
    // one LSTM call on prepared weights and buffers: checks, launches and, with `wait`, the wait for the stream.  Returns the
    // library's (negative) error code, else the status word when it has waited.
    m.def("_lstm_forward", [](const at::Tensor& x, const at::Tensor& w_ih, const at::Tensor& w_hh, const at::Tensor& b_ih, const at::Tensor& b_hh,
                              const at::Tensor& hs, const at::Tensor& cs, const at::Tensor& scratch, const at::Tensor& status, int64_t mode,
                              bool wait) -> int64_t {
        py::gil_scoped_release release;
        checkInput(x, x.device(), "x");
        TORCH_CHECK_VALUE(x.dim() == 3 && w_hh.dim() == 3, "x must be [T, B, I], w_hh [4, H, H]");
        const int64_t T = x.size(0), B = x.size(1), I = x.size(2), H = w_hh.size(2);
        TORCH_CHECK_VALUE(w_ih.dim() == 3 && w_ih.size(0) == 4 && w_ih.size(1) == I && w_ih.size(2) == H && w_hh.size(0) == 4 &&
                              w_hh.size(1) == H,
                          "weights must be gate-leading: w_ih [4, I, H], w_hh [4, H, H]");
        TORCH_CHECK_VALUE(b_ih.numel() == 4 * H && b_hh.numel() == 4 * H, "biases must have 4*H elements");
        checkBuffer(w_ih, x.device(), at::kFloat, w_ih.sizes(), "w_ih");
        checkBuffer(w_hh, x.device(), at::kFloat, w_hh.sizes(), "w_hh");
        checkBuffer(b_ih, x.device(), at::kFloat, b_ih.sizes(), "b_ih");
        checkBuffer(b_hh, x.device(), at::kFloat, b_hh.sizes(), "b_hh");
        checkBuffer(hs, x.device(), at::kFloat, {T, B, H}, "hs");
        checkBuffer(cs, x.device(), at::kFloat, {T, B, H}, "cs");
        const int64_t need = functs_b200_lstm_scratch_bytes(static_cast<int32_t>(T), static_cast<int32_t>(B), static_cast<int32_t>(I),
                                                            static_cast<int32_t>(H));
        TORCH_CHECK_VALUE(scratch.device() == x.device() && scratch.is_contiguous() && static_cast<int64_t>(scratch.nbytes()) >= need,
                          "scratch must hold ", need, " bytes on ", x.device());
        TORCH_CHECK_VALUE(status.is_cpu() && status.scalar_type() == at::kInt && status.numel() >= 1 && status.is_pinned(),
                          "status must be an int32 tensor in pinned memory");
        c10::cuda::CUDAGuard guard(x.device());
        const at::Tensor xc = x.contiguous();
        const auto stream = at::cuda::getCurrentCUDAStream();
        const int rc = functs_b200_lstm_forward_mode(xc.data_ptr<float>(), w_ih.data_ptr<float>(), w_hh.data_ptr<float>(), b_ih.data_ptr<float>(),
                                                     b_hh.data_ptr<float>(), static_cast<int32_t>(T), static_cast<int32_t>(B),
                                                     static_cast<int32_t>(I), static_cast<int32_t>(H), hs.data_ptr<float>(), cs.data_ptr<float>(),
                                                     status.data_ptr<int32_t>(), scratch.data_ptr(), stream.stream(), static_cast<int32_t>(mode));
        if (rc != FB_OK || !wait) return rc;
        C10_CUDA_CHECK(cudaStreamSynchronize(stream.stream()));
        return *static_cast<volatile int32_t*>(status.data_ptr<int32_t>());
    });
    // masks into `out` [B, N, H, W]; returns the library's error code
    m.def("_yolact_masks", [](const at::Tensor& proto, const at::Tensor& coef, const at::Tensor& boxes, double thr, const at::Tensor& out) -> int64_t {
        py::gil_scoped_release release;
        checkInput(proto, proto.device(), "proto");
        checkInput(coef, proto.device(), "coef");
        checkInput(boxes, proto.device(), "boxes");
        TORCH_CHECK_VALUE(proto.dim() == 4 && proto.size(3) == 32, "prototype depth must be 32");
        const int64_t B = proto.size(0), H = proto.size(1), W = proto.size(2);
        TORCH_CHECK_VALUE(coef.dim() == 3 && coef.size(0) == B && coef.size(2) == 32 && boxes.dim() == 3 && boxes.size(0) == B &&
                              boxes.size(1) == coef.size(1) && boxes.size(2) == 4,
                          "proto [B, H, W, 32], coef [B, N, 32] and boxes [B, N, 4] do not fit one another");
        checkBuffer(out, proto.device(), at::kByte, {B, coef.size(1), H, W}, "out");
        c10::cuda::CUDAGuard guard(proto.device());
        const at::Tensor p = proto.contiguous(), c = coef.contiguous(), b = boxes.contiguous();
        return functs_b200_yolact_masks(p.data_ptr<float>(), c.data_ptr<float>(), b.data_ptr<float>(), static_cast<int32_t>(B),
                                        static_cast<int32_t>(H), static_cast<int32_t>(W), static_cast<int32_t>(c.size(1)),
                                        static_cast<float>(thr), out.data_ptr<uint8_t>(), nullptr, at::cuda::getCurrentCUDAStream().stream());
    });
    m.def("_count_parallel_functors", [](std::shared_ptr<Graph> g) { return functs_b200::CountParallelFunctors(g); });
    m.def("_jit_pass_freeze", [](torch::jit::Module& module) { return torch::jit::freeze_module(module); });
    m.def("_jit_pass_clone", [](torch::jit::Module& module) { return module.clone(); });
    m.def("_create_function_from_graph", [](const std::string& qualname, std::shared_ptr<Graph> graph) {
        auto cu = std::make_shared<torch::jit::CompilationUnit>();
        auto* fn = cu->create_function(c10::QualifiedName(qualname), graph);
        return torch::jit::StrongFunctionPtr(std::move(cu), fn);
    });
}
