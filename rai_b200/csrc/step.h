// A single-token step of few sequences as one kernel (step.cu).
#pragma once

struct rb_model;

namespace rb {

constexpr int kStepLayers = 40;   // (their tensor maps are arguments of the kernel)
struct StepPlan;
int step_reserve(rb_model* m);                  // at the end of a model's creation; leaves no plan where the kernel does not fit
void step_plan_free(StepPlan* plan);
bool step_takes(const rb_model* m, int batch);
// From the embedded rows in m->h to m->logits (want_head), or to the final rows of the stream in m->h alone.  `ran` false: the launch was
// refused, the plan is gone and m->h is as it was.
int step_forward(rb_model* m, int batch, bool want_head, bool* ran);
// Test hooks: the model's next step waits for arrivals that never come, and gives up; its launch is refused.
int step_spoil(rb_model* m);
int step_refuse(rb_model* m);

}  // namespace rb
