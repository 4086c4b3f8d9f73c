// Prints whether launch configurations count as a shape of the caller's own
// (cbq_internal.hpp): "volume" and "batch", refill, steps and form per line; then
// the configurations the tuner times: "tuned", form, block, refill, steps, stack.
#include "../cubiquity_gb300/csrc/cbq_internal.hpp"

#include <cstdio>

int main()
{
    for (uint32_t refill : {0u, 1u, 8u, 16u, 32u})
        for (int32_t steps : {0, 1, 8, 16, 32})
            for (int32_t form : {CBQ_FORM_PLAIN, CBQ_FORM_PERSISTENT, CBQ_FORM_SORTED}) {
                cbq_launch_config v{};
                v.refill_min = refill;
                v.steps = steps;
                v.form = form;
                cbq_batch_config b{128, refill, steps, 0, CBQ_STACK_SHARED, form};
                std::printf("volume %u %d %d %d\nbatch %u %d %d %d\n", refill, steps, form, cbq::own_shape(v), refill,
                            steps, form, cbq::own_shape(b));
            }
    cbq_launch_config base{};
    base.chunk = 77;
    cbq::for_each_tuned_config(base, [](const cbq_launch_config& c) {
        std::printf("tuned %d %d %u %d %d\n", c.form, c.block, c.refill_min, c.steps, c.chunk == 77 ? c.stack : -1);
        return true;
    });
    return 0;
}
