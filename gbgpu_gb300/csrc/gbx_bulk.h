// Order of the copies and reductions of one warp of the row-major fill, written
// apart from the instructions so that it can be run on the host with copies that
// do not arrive.
#pragma once

#include "gbx_index.h"

namespace gbx {

// Every item of `next` goes through one of STAGES buffers: load(stage, item)
// starts its copy in, loaded(stage, parity) waits for the copy (a bounded wait:
// false when it gave up), add(stage, item) starts the reduction that reads the
// buffer, and read() returns once all reductions but the latest have read theirs,
// so that the buffer before it can be filled again.
//
// After a wait that gave up nothing more is started: its buffer, and the phase of
// its barrier, still belong to the copy under way.  The copies already started are
// waited for once more (bounded too), as their shared memory may not be given back
// under them, and the result is false: the remaining bins are missing.
template <int STAGES, typename Item, typename Next, typename Load, typename Loaded, typename Add, typename Read>
GBX_HD bool bulk_pipeline(Next &&next, Load &&load, Loaded &&loaded, Add &&add, Read &&read)
{
    Item items[STAGES];
    int in = 0, done = 0;                // copies started, reductions started
    bool more = true, ok = true;
    // one stage stays free for the reduction that still reads its buffer
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < STAGES - 1; k++) {
        if (more && (more = next(items[k]))) {
            load(k, items[k]);
            in++;
        }
    }
    while (ok && done < in) {
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int k = 0; k < STAGES; k++) {
            if (done >= in) break;
            ok = loaded(k, (unsigned)(done / STAGES) & 1u);
            if (!ok) break;
            add(k, items[k]);
            done++;
            const int kn = k == 0 ? STAGES - 1 : k - 1;
            read();
            if (more && (more = next(items[kn]))) {
                load(kn, items[kn]);
                in++;
            }
        }
    }
    if (!ok)
        for (; done < in; done++) loaded(done % STAGES, (unsigned)(done / STAGES) & 1u);
    return ok;
}

}  // namespace gbx
