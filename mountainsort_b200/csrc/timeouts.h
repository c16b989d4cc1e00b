// Checks that each clear a sticky flag and throw: all of them run, so that no flag stays
// set for the next call, then one error names every one that threw.  Kept free of CUDA
// headers so the rule can be checked on a machine without a GPU.
#pragma once

#include <string>

namespace ms3gpu {

// E: an exception with `code` and a constructor E(code, message).
template <class E, class... Check>
void raise_together(Check&&... checks) {
    int code = 0;
    std::string all;
    auto run = [&](auto&& check) {
        try {
            check();
        } catch (const E& e) {
            if (all.empty())
                code = e.code;
            else
                all += "; ";
            all += e.what();
        }
    };
    (run(checks), ...);
    if (!all.empty()) throw E(code, all);
}

}  // namespace ms3gpu
