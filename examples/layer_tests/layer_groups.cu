// Layers whose functions may run side by side and whose functions may not.
// Registered model:
//   "layer_groups"  params: macro (1: two functions of a layer also update one
//                   environment macro property)
// Agents A, B, C (x, y, v, s) and D (states idle, busy). Per step:
//   say    A, B and C output to a list each (spatial, brute force, spatial)
//   hear   B and C read A's spatial list (its build and their sorts, in turn);
//          A and idle D read B's brute-force list
//   work   A gives birth to C; B walks; busy D works; idle D gives birth to C,
//          which joins the first and the third
//   leave  idle D turn busy, some; A die, some; B gives birth to A and die, some;
//          busy D turn idle, some
//   again  C output to their list once more and B read it; A walk
//   macro  A and B add to one macro property (macro = 1; else to their own v)
// Every v folds what it meets in the order it meets it.
#include "flamegpu/flamegpu.h"
#include "flamegpu_gb300/fg_sim.h"

namespace {
constexpr float kEdge = 30.0f;

__device__ __forceinline__ unsigned int fold(unsigned int h, unsigned int v) { return (h ^ v) * 2654435761u + 1u; }

template <typename API>
__device__ __forceinline__ void say(API* FLAMEGPU) {
    FLAMEGPU->message_out.template setVariable<unsigned int>("v", FLAMEGPU->template getVariable<unsigned int>("v"));
}
template <typename API>
__device__ __forceinline__ void place(API* FLAMEGPU) {
    FLAMEGPU->message_out.setLocation(FLAMEGPU->template getVariable<float>("x"), FLAMEGPU->template getVariable<float>("y"));
}
template <typename API>
__device__ __forceinline__ void hear_near(API* FLAMEGPU) {
    unsigned int h = FLAMEGPU->template getVariable<unsigned int>("v");
    float s = 0.0f;
    for (const auto& m : FLAMEGPU->message_in(FLAMEGPU->template getVariable<float>("x"), FLAMEGPU->template getVariable<float>("y"))) {
        h = fold(h, m.template getVariable<unsigned int>("v"));
        s += m.template getVariable<float>("x");
    }
    FLAMEGPU->template setVariable<unsigned int>("v", h);
    FLAMEGPU->template setVariable<float>("s", s);
}
template <typename API>
__device__ __forceinline__ void hear_all(API* FLAMEGPU) {
    unsigned int h = FLAMEGPU->template getVariable<unsigned int>("v");
    for (const auto& m : FLAMEGPU->message_in) h = fold(h, m.template getVariable<unsigned int>("v"));
    FLAMEGPU->template setVariable<unsigned int>("v", h);
}
template <typename API>
__device__ __forceinline__ void walk(API* FLAMEGPU) {
    const float x = FLAMEGPU->template getVariable<float>("x") + FLAMEGPU->random.template uniform<float>() - 0.5f;
    const float y = FLAMEGPU->template getVariable<float>("y") + FLAMEGPU->random.template uniform<float>() - 0.5f;
    FLAMEGPU->template setVariable<float>("x", fminf(fmaxf(x, 0.0f), kEdge));
    FLAMEGPU->template setVariable<float>("y", fminf(fmaxf(y, 0.0f), kEdge));
}
template <typename API>
__device__ __forceinline__ void child(API* FLAMEGPU, unsigned int one_in) {
    const unsigned int v = FLAMEGPU->template getVariable<unsigned int>("v");
    if (v % one_in) return;
    FLAMEGPU->agent_out.template setVariable<float>("x", FLAMEGPU->template getVariable<float>("y"));
    FLAMEGPU->agent_out.template setVariable<float>("y", FLAMEGPU->template getVariable<float>("x"));
    FLAMEGPU->agent_out.template setVariable<unsigned int>("v", fold(v, 7u));
}
}  // namespace

FLAMEGPU_AGENT_FUNCTION(lg_a_say, flamegpu::MessageNone, flamegpu::MessageSpatial2D) {
    place(FLAMEGPU);
    say(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_b_say, flamegpu::MessageNone, flamegpu::MessageBruteForce) {
    say(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_c_say, flamegpu::MessageNone, flamegpu::MessageSpatial2D) {
    place(FLAMEGPU);
    say(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_c_say_again, flamegpu::MessageNone, flamegpu::MessageSpatial2D) {
    place(FLAMEGPU);
    say(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_b_hear, flamegpu::MessageSpatial2D, flamegpu::MessageNone) {
    hear_near(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_c_hear, flamegpu::MessageSpatial2D, flamegpu::MessageNone) {
    hear_near(FLAMEGPU);
    return FLAMEGPU->getVariable<unsigned int>("v") % 11u == 0u ? flamegpu::DEAD : flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_b_hear_again, flamegpu::MessageSpatial2D, flamegpu::MessageNone) {
    hear_near(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_a_all, flamegpu::MessageBruteForce, flamegpu::MessageNone) {
    hear_all(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_d_all, flamegpu::MessageBruteForce, flamegpu::MessageNone) {
    hear_all(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_a_birth, flamegpu::MessageNone, flamegpu::MessageNone) {
    child(FLAMEGPU, 6u);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_b_walk, flamegpu::MessageNone, flamegpu::MessageNone) {
    walk(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_d_work, flamegpu::MessageNone, flamegpu::MessageNone) {
    walk(FLAMEGPU);
    FLAMEGPU->setVariable<unsigned int>("v", fold(FLAMEGPU->getVariable<unsigned int>("v"), FLAMEGPU->getStepCounter()));
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_d_birth, flamegpu::MessageNone, flamegpu::MessageNone) {
    child(FLAMEGPU, 5u);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_a_walk, flamegpu::MessageNone, flamegpu::MessageNone) {
    walk(FLAMEGPU);
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_d_go, flamegpu::MessageNone, flamegpu::MessageNone) { return flamegpu::ALIVE; }
FLAMEGPU_AGENT_FUNCTION(lg_d_back, flamegpu::MessageNone, flamegpu::MessageNone) { return flamegpu::ALIVE; }
FLAMEGPU_AGENT_FUNCTION_CONDITION(lg_third) { return FLAMEGPU->getVariable<unsigned int>("v") % 3u == 0u; }
FLAMEGPU_AGENT_FUNCTION_CONDITION(lg_half) { return FLAMEGPU->getVariable<unsigned int>("v") % 2u == 0u; }
FLAMEGPU_AGENT_FUNCTION(lg_a_die, flamegpu::MessageNone, flamegpu::MessageNone) {
    return FLAMEGPU->getVariable<unsigned int>("v") % 10u == 0u ? flamegpu::DEAD : flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_b_leave, flamegpu::MessageNone, flamegpu::MessageNone) {
    child(FLAMEGPU, 9u);
    return FLAMEGPU->getVariable<unsigned int>("v") % 200u == 0u ? flamegpu::DEAD : flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_a_macro, flamegpu::MessageNone, flamegpu::MessageNone) {
    FLAMEGPU->environment.getMacroProperty<unsigned int, 4>("met")[FLAMEGPU->getID() % 4] += FLAMEGPU->getVariable<unsigned int>("v");
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_b_macro, flamegpu::MessageNone, flamegpu::MessageNone) {
    FLAMEGPU->environment.getMacroProperty<unsigned int, 4>("met")[FLAMEGPU->getID() % 4] += FLAMEGPU->getVariable<unsigned int>("v");
    return flamegpu::ALIVE;
}
FLAMEGPU_AGENT_FUNCTION(lg_d_met, flamegpu::MessageNone, flamegpu::MessageNone) {
    const unsigned int met = FLAMEGPU->environment.getMacroProperty<unsigned int, 4>("met")[FLAMEGPU->getID() % 4];
    FLAMEGPU->setVariable<unsigned int>("v", fold(FLAMEGPU->getVariable<unsigned int>("v"), met));
    return flamegpu::ALIVE;
}

namespace {

void* make_layer_groups(const double* p, int32_t np) {
    const bool macro = np > 0 && p[0] != 0.0;
    auto* model = new flamegpu::ModelDescription("LayerGroups");
    auto agent = [&](const char* name) {
        flamegpu::AgentDescription a = model->newAgent(name);
        a.newVariable<float>("x");
        a.newVariable<float>("y");
        a.newVariable<unsigned int>("v");
        a.newVariable<float>("s", 0.25f);
        return a;
    };
    flamegpu::AgentDescription a = agent("A"), b = agent("B"), c = agent("C"), d = agent("D");
    d.newState("idle");
    d.newState("busy");
    d.setInitialState("idle");
    for (const char* name : {"a_near", "c_near"}) {
        auto m = model->newMessage<flamegpu::MessageSpatial2D>(name);
        m.setMin(0.0f, 0.0f);
        m.setMax(kEdge, kEdge);
        m.setRadius(1.5f);
        m.newVariable<unsigned int>("v");
    }
    model->newMessage<flamegpu::MessageBruteForce>("b_all").newVariable<unsigned int>("v");
    if (macro) model->Environment().newMacroProperty<unsigned int, 4>("met");

    auto a_say = a.newFunction("say", lg_a_say);
    a_say.setMessageOutput("a_near");
    auto b_say = b.newFunction("say", lg_b_say);
    b_say.setMessageOutput("b_all");
    auto c_say = c.newFunction("say", lg_c_say);
    c_say.setMessageOutput("c_near");
    auto b_hear = b.newFunction("hear", lg_b_hear);
    b_hear.setMessageInput("a_near");
    auto c_hear = c.newFunction("hear", lg_c_hear);
    c_hear.setMessageInput("a_near");
    c_hear.setAllowAgentDeath(true);
    auto a_all = a.newFunction("all", lg_a_all);
    a_all.setMessageInput("b_all");
    auto d_all = d.newFunction("all", lg_d_all);
    d_all.setInitialState("idle");
    d_all.setEndState("idle");
    d_all.setMessageInput("b_all");
    auto a_birth = a.newFunction("birth", lg_a_birth);
    a_birth.setAgentOutput(c);
    auto b_walk = b.newFunction("walk", lg_b_walk);
    auto d_work = d.newFunction("work", lg_d_work);
    d_work.setInitialState("busy");
    d_work.setEndState("busy");
    auto d_birth = d.newFunction("birth", lg_d_birth);
    d_birth.setInitialState("idle");
    d_birth.setEndState("idle");
    d_birth.setAgentOutput(c);
    auto d_go = d.newFunction("go", lg_d_go);
    d_go.setInitialState("idle");
    d_go.setEndState("busy");
    d_go.setFunctionCondition(lg_third);
    auto a_die = a.newFunction("die", lg_a_die);
    a_die.setAllowAgentDeath(true);
    auto b_leave = b.newFunction("leave", lg_b_leave);
    b_leave.setAllowAgentDeath(true);
    b_leave.setAgentOutput(a);
    auto c_again = c.newFunction("say_again", lg_c_say_again);
    c_again.setMessageOutput("c_near");
    auto b_again = b.newFunction("hear_again", lg_b_hear_again);
    b_again.setMessageInput("c_near");
    auto a_walk = a.newFunction("walk", lg_a_walk);
    auto d_back = d.newFunction("back", lg_d_back);
    d_back.setInitialState("busy");
    d_back.setEndState("idle");
    d_back.setFunctionCondition(lg_half);

    auto layer = [&](std::initializer_list<flamegpu::AgentFunctionDescription> functions) {
        flamegpu::LayerDescription l = model->newLayer();
        for (const auto& f : functions) l.addAgentFunction(f);
    };
    layer({a_say, b_say, c_say});
    layer({b_hear, a_all, c_hear, d_all});
    layer({a_birth, b_walk, d_work, d_birth});
    layer({d_go, a_die, b_leave, d_back});
    layer({c_again, a_walk, b_again});
    if (macro) {
        layer({a.newFunction("macro", lg_a_macro), b.newFunction("macro", lg_b_macro)});
        auto d_met = d.newFunction("met", lg_d_met);
        d_met.setInitialState("idle");
        d_met.setEndState("idle");
        layer({d_met});
    }
    return model;
}

struct Register {
    Register() { fgs_register_model("layer_groups", &make_layer_groups); }
} reg;

}  // namespace
