// Host side of a rollout's schedule: the later substeps of a table whose first
// entry is filled in. Only the time, the gates and the points that move with
// their velocity differ between the substeps of a call without host callbacks
// (mpm_solver_diff.py:186-291, 795-801 of the reference evaluate them once per
// substep in Python, as this framework did: 20 us a substep with one collider, 60
// with five, more than the substep's kernels take at 20k particles; here 0.3 us,
// the copy of the entry's 2.4 KB).
#include <cstring>

#include "../../include/empm_b200.h"

namespace {

int gate(const EmpmWindow& w, float t) {
    if (w.on && t >= w.start && t < w.end) return EMPM_GATE_APPLY;
    return t < w.zero_until ? EMPM_GATE_ZERO_ALL : EMPM_GATE_OFF;
}

static_assert(sizeof(EmpmWindow) == 64, "mirrored by the ctypes structure");

// point += dt * velocity in double, each kept as float between the substeps.
// The product is rounded before the sum on every host.
void move(EmpmWindow& w, double t, double dt) {
    if (!w.moves || !(t >= w.move_start && t < w.move_end)) return;
    for (int k = 0; k < 3; k++) {
        volatile double step = dt * static_cast<double>(w.velocity[k]);
        w.point[k] = static_cast<float>(static_cast<double>(w.point[k]) + step);
    }
    w.moved = 1;
}

}  // namespace

extern "C" int empm_schedule_fill(EmpmStep* steps, int stride, int n_steps, double t0, double dt,
                                  EmpmWindow* colliders, const EmpmWindow* modifiers, double* t_end) {
    if (!steps || stride < 1 || n_steps < 1 || !t_end) return EMPM_ERR_INVALID;
    const EmpmStep& first = steps[0];
    if (first.n_colliders < 0 || first.n_colliders > EMPM_MAX_COLLIDERS || first.n_modifiers < 0 ||
        first.n_modifiers > EMPM_MAX_MODIFIERS || (first.n_colliders && !colliders) ||
        (first.n_modifiers && !modifiers))
        return EMPM_ERR_INVALID;
    double t = t0;
    for (int s = 0; s < n_steps; s++) {
        EmpmStep& st = steps[static_cast<size_t>(s) * stride];
        if (s) std::memcpy(&st, &first, sizeof(EmpmStep));
        st.time = static_cast<float>(t);
        for (int i = 0; i < first.n_colliders; i++) {
            EmpmWindow& w = colliders[i];
            st.colliders[i].gate = gate(w, st.time);
            if (w.moves) std::memcpy(st.colliders[i].point, w.point, sizeof(w.point));
            move(w, t, dt);
        }
        for (int i = 0; i < first.n_modifiers; i++) st.modifiers[i].gate = gate(modifiers[i], st.time);
        t = t + dt;
    }
    *t_end = t;
    return EMPM_OK;
}
