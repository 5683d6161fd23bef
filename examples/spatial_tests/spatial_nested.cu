// Searches of one message list that are alive at the same time in one agent:
// a loop around every message of a loop, a copied search, and a loop of the
// input list around every message of a loop of a copy of it.
// Registered model:
//   "spatial_nested"  params: dims, min, max, radius, wrap
// Each agent sets outer (messages of its own search), inner (messages of the
// searches around each of those), copied (messages of a copy of its search) and
// list_outer, list_inner (as outer and inner, the outer search from a copy of
// the input list) and list_swapped (as inner, the inner searches from the copy).
#include "flamegpu/flamegpu.h"
#include "flamegpu_gb300/fg_sim.h"

FLAMEGPU_AGENT_FUNCTION(nested_out3, flamegpu::MessageNone, flamegpu::MessageSpatial3D) {
    FLAMEGPU->message_out.setLocation(FLAMEGPU->getVariable<float>("x"), FLAMEGPU->getVariable<float>("y"),
                                      FLAMEGPU->getVariable<float>("z"));
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(nested_out2, flamegpu::MessageNone, flamegpu::MessageSpatial2D) {
    FLAMEGPU->message_out.setLocation(FLAMEGPU->getVariable<float>("x"), FLAMEGPU->getVariable<float>("y"));
    return flamegpu::ALIVE;
}

template <int DIMS, bool WRAP, typename API>
__device__ __forceinline__ flamegpu::AGENT_STATUS nested_count(API* FLAMEGPU) {
    const float x = FLAMEGPU->template getVariable<float>("x"), y = FLAMEGPU->template getVariable<float>("y");
    const float z = DIMS == 3 ? FLAMEGPU->template getVariable<float>("z") : 0.0f;
    auto search_of = [](const auto& in, float px, float py, float pz) {
        if constexpr (DIMS == 3 && WRAP) return in.wrap(px, py, pz);
        else if constexpr (DIMS == 3) return in(px, py, pz);
        else if constexpr (WRAP) return in.wrap(px, py);
        else return in(px, py);
    };
    auto search = [&](float px, float py, float pz) { return search_of(FLAMEGPU->message_in, px, py, pz); };
    auto around = [](const auto& m) {
        if constexpr (DIMS == 3) return m.template getVariable<float>("z");
        else return 0.0f;
    };
    unsigned int list_outer = 0, list_inner = 0, list_swapped = 0;
    const auto in = FLAMEGPU->message_in;
    for (const auto& m : search_of(in, x, y, z)) {
        ++list_outer;
        for (const auto& k : search(m.template getVariable<float>("x"), m.template getVariable<float>("y"), around(m))) {
            (void)k;
            ++list_inner;
        }
    }
    for (const auto& m : search(x, y, z))
        for (const auto& k : search_of(in, m.template getVariable<float>("x"), m.template getVariable<float>("y"), around(m))) {
            (void)k;
            ++list_swapped;
        }
    unsigned int outer = 0, inner = 0, copied = 0;
    for (const auto& m : search(x, y, z)) {
        ++outer;
        float mz = 0.0f;
        if constexpr (DIMS == 3) mz = m.template getVariable<float>("z");
        for (const auto& k : search(m.template getVariable<float>("x"), m.template getVariable<float>("y"), mz)) {
            (void)k;
            ++inner;
        }
    }
    const auto first = search(x, y, z);
    const auto second = first;
    for (const auto& m : second) {
        (void)m;
        ++copied;
    }
    FLAMEGPU->template setVariable<unsigned int>("list_outer", list_outer);
    FLAMEGPU->template setVariable<unsigned int>("list_inner", list_inner);
    FLAMEGPU->template setVariable<unsigned int>("list_swapped", list_swapped);
    FLAMEGPU->template setVariable<unsigned int>("outer", outer);
    FLAMEGPU->template setVariable<unsigned int>("inner", inner);
    FLAMEGPU->template setVariable<unsigned int>("copied", copied);
    return flamegpu::ALIVE;
}

FLAMEGPU_AGENT_FUNCTION(nested_in3, flamegpu::MessageSpatial3D, flamegpu::MessageNone) {
    return nested_count<3, false>(FLAMEGPU);
}
FLAMEGPU_AGENT_FUNCTION(nested_in3_wrapped, flamegpu::MessageSpatial3D, flamegpu::MessageNone) {
    return nested_count<3, true>(FLAMEGPU);
}
FLAMEGPU_AGENT_FUNCTION(nested_in2, flamegpu::MessageSpatial2D, flamegpu::MessageNone) {
    return nested_count<2, false>(FLAMEGPU);
}
FLAMEGPU_AGENT_FUNCTION(nested_in2_wrapped, flamegpu::MessageSpatial2D, flamegpu::MessageNone) {
    return nested_count<2, true>(FLAMEGPU);
}

namespace {

void* make_spatial_nested(const double* p, int32_t np) {
    auto P = [&](int i, double d) { return i < np ? p[i] : d; };
    const int dims = static_cast<int>(P(0, 3));
    const float mn = static_cast<float>(P(1, 0.0)), mx = static_cast<float>(P(2, 8.0)), r = static_cast<float>(P(3, 1.0));
    const bool wrap = P(4, 0.0) != 0.0;
    auto* model = new flamegpu::ModelDescription("SpatialNested");
    flamegpu::AgentDescription a = model->newAgent("agent");
    a.newVariable<float>("x");
    a.newVariable<float>("y");
    if (dims == 3) a.newVariable<float>("z");
    for (const char* n : {"outer", "inner", "copied", "list_outer", "list_inner", "list_swapped"}) a.newVariable<unsigned int>(n);
    if (dims == 3) {
        auto m = model->newMessage<flamegpu::MessageSpatial3D>("location");
        m.setMin(mn, mn, mn);
        m.setMax(mx, mx, mx);
        m.setRadius(r);
        a.newFunction("out", nested_out3).setMessageOutput("location");
        auto in = wrap ? a.newFunction("in", nested_in3_wrapped) : a.newFunction("in", nested_in3);
        in.setMessageInput("location");
        model->newLayer().addAgentFunction(nested_out3);
        model->newLayer().addAgentFunction(in);
    } else {
        auto m = model->newMessage<flamegpu::MessageSpatial2D>("location");
        m.setMin(mn, mn);
        m.setMax(mx, mx);
        m.setRadius(r);
        a.newFunction("out", nested_out2).setMessageOutput("location");
        auto in = wrap ? a.newFunction("in", nested_in2_wrapped) : a.newFunction("in", nested_in2);
        in.setMessageInput("location");
        model->newLayer().addAgentFunction(nested_out2);
        model->newLayer().addAgentFunction(in);
    }
    return model;
}

struct Register {
    Register() { fgs_register_model("spatial_nested", &make_spatial_nested); }
} reg;

}  // namespace
