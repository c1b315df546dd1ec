// A grid that calls accumulate into and leave zero for the next one (the NUFFT adjoint: gridding,
// then a transform that clears what it has read), without a memset of its own per call. Host logic
// only.
#pragma once

namespace lentils {

// One such call. run: enqueues it; clear: enqueues a memset of the grid; capturing: whether the
// stream is being captured. run and clear return 0 for success. dirty: the grid may not be zero when
// the work enqueued so far is done.
//
// A failed call may have added to the grid without the pass that clears it, so the grid is cleared
// behind it, and if that fails too, ahead of the next call. Work on a capturing stream only joins a
// graph: it changes nothing now, nor may the graph be launched ever, so it leaves `dirty` as it is,
// and a graph captured from a dirty grid clears it itself.
template <class Run, class Clear, class Capturing>
int accumulate_clean(bool &dirty, Run run, Clear clear, Capturing capturing)
{
    if (dirty)
        if (const int st = clear()) return st;
    const int st = run();
    if ((st || dirty) && !capturing()) dirty = st && clear();
    return st;
}

}  // namespace lentils
