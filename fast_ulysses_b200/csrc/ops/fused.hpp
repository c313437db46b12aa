#pragma once
// The fused operators (GEMM, feed-forward, LayerNorm, attention, the sequence-parallel attention
// block, the fp8 exchange) as C++ functions with C++ autograd nodes. The Python modules of
// fast_ulysses_b200.ops and .models are thin: a forward and backward of a DiT block is about thirty
// launches, and building each one's arguments in Python took several times as long as the kernels of
// a small model run.
#include <torch/extension.h>

#include "../runtime/group.hpp"

namespace fu {

// The group as a pybind object (a torch.classes object is slow to pass through torch.ops).
struct GroupRef {
    c10::intrusive_ptr<Group> group;
};

void bind_fused(pybind11::module_& m);

}  // namespace fu
