// The operators' autograd functions as C++ graph nodes.
//
// A small call's time is host time: with torch.autograd.Function in Python a forward + backward of 18 us of kernels took
// 91 us (the function's bookkeeping, two launch-hint searches that the kernels ignore, and the GIL for the engine's
// thread in the backward).  As nodes, a call is one binding call in each direction and the backward never enters Python.
//
// Semantics are those of a Python Function with once_differentiable in reverse mode on plain tensors: inputs are saved with
// version checks and saved-tensor hooks, a second backward without retain_graph raises, and differentiating the gradients
// raises (where the Python version raised).  Every other mode takes the Python Function (ops3d_b200/graph.py).
#pragma once

#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <array>
#include <memory>
#include <mutex>
#include <string>

namespace fda_nodes {

using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// What once_differentiable does with a backward's results: while the graph of the gradients is being recorded, they get a
// history that raises when it is differentiated.
inline variable_list once_differentiable(variable_list results, bool recording) {
    if (!recording) return results;
    for (auto &r : results)
        if (r.defined()) {
            r = r.detach();
            r.set_requires_grad(true);
        }
    auto error = std::make_shared<torch::autograd::DelayedError>(
        "trying to differentiate twice a function that was marked with @once_differentiable", (int64_t)results.size());
    return error->apply(std::move(results));
}

inline bool needs_node(std::initializer_list<std::reference_wrapper<const at::Tensor>> inputs) {
    if (!at::GradMode::is_enabled()) return false;
    for (const at::Tensor &t : inputs)
        if (t.requires_grad()) return true;
    return false;
}

// Base: two differentiable inputs saved at most, arguments in the derived class.
struct SavedNode : public torch::autograd::Node {
    std::array<SavedVariable, 4> saved;
    void save(size_t i, const at::Tensor &t) { saved[i] = SavedVariable(t, /*is_output=*/false); }
    // The output's gradient; where nothing has one for it (a later function returned None), zeros, as a Function gets them.
    at::Tensor grad_output(const variable_list &grads) const { return grads[0].defined() ? grads[0] : input_metadata(0).zeros_like(); }
    at::Tensor unpack(size_t i) const { return saved[i].unpack(); }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (auto &s : saved) s.reset_data();
    }
};

// Connects `output` to `node`, whose gradients belong to `inputs` in order.
inline void connect(const std::shared_ptr<SavedNode> &node, at::Tensor &output, torch::autograd::edge_list &&edges) {
    node->set_next_edges(std::move(edges));
    torch::autograd::set_history(output, node);
}

}  // namespace fda_nodes
