// Arguments of the one-launch time loops (star7_loop.cuh, star7_cluster.cuh).
#pragma once

#include "node_order.cuh"
#include "star7_border.cuh"

namespace scafes {

template <class T>
struct LoopArgs {
    T* u[2];                 // iterates; u[first] is the old one of the first step
    int first, n_steps;
    const T* fa;
    const T* fb;
    const T* ga;
    const T* gb;
    T gval;
    const T* c0;             // variable coefficients
    const T* ca;
    Layout L;
    NodeOrder o;
    Star7Coeffs c;
    const BorderTable* table;
    const scafes_border_node_rule* nodes;
    const StepTimes* times;  // n_steps entries, or null when nothing reads the time
    uint32_t in_cta, bd_cta; // inner and border nodes per CTA
    unsigned* arrivals;      // barrier counter, 0 at launch
    int* status;
};

}  // namespace scafes
