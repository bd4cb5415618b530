// Work launched ahead of its results. Plain C++ (no CUDA header), so that it can be checked on the host.
#pragma once
#include <stdint.h>

namespace ak {

// Items 0 .. n - 1 in order, at most `ahead` of them launched and not yet waited for. launch(j) and wait(j, stop) return 0 or an error
// code; wait sets stop where the items after j are not wanted. Whatever ends it, nothing that was launched is still under way
// on return: if an item was launched and not waited for, or anything failed (a launch may have failed half way), drain() waits for all of it.
template <class Launch, class Wait, class Drain>
int run_ahead(uint32_t n, uint32_t ahead, Launch launch, Wait wait, Drain drain) {
    int rc = 0;
    uint32_t launched = 0, done = 0;
    bool stop = false;
    while (done < n && !stop && rc == 0) {
        while (launched < n && launched - done < ahead && (rc = launch(launched)) == 0) launched++;
        if (rc == 0 && (rc = wait(done, stop)) == 0) done++;
    }
    if (rc != 0 || done < launched) {
        const int rd = drain();
        if (rc == 0) rc = rd;
    }
    return rc;
}

}  // namespace ak
