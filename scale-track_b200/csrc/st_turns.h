/*
 * st_turns.h -- which of the two control sets of the allocation-free step a call takes, and
 * whether it must reset them first (st_noalloc.cu).  Host code only; the caller holds a lock.
 *
 * A call works in one set, and its last kernel resets the other for the call after it.  That
 * holds from one call to the next only where they do not overlap: of overlapping calls each may
 * reset the set in which another works, or leave one used.  So a call that overlapped another, or
 * that failed before its last kernel had run, leaves the sets to be reset by the next call that
 * starts alone: a race or a failure does not outlive the calls that made it.
 */
#ifndef ST_TURNS_H
#define ST_TURNS_H

namespace st {

struct Turns {
    int next = 0;          /* the set of the next call */
    int running = 0;       /* calls begun and not ended */
    bool overlap = false;  /* of the running calls, some overlapped */
    bool dirty = false;    /* the sets need a reset */

    struct Turn {
        int set;
        bool reset;        /* both sets, before anything else */
    };
    Turn begin()
    {
        const Turn t = {next, dirty && running == 0};
        if (running > 0) overlap = true;
        ++running;
        next ^= 1;
        return t;
    }
    /* complete: every kernel of the call has run */
    void end(bool complete)
    {
        dirty = overlap || !complete;
        if (--running == 0) overlap = false;
    }
};

}  // namespace st

#endif
