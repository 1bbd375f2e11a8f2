// side_work.hpp -- the order of a step that has work on a side stream.
#pragma once

namespace hp {

// begin starts the side work, body runs beside it, end waits for it and goes
// on.  Where one of them fails, join still makes the caller's stream wait for
// what runs on the side, so that nothing started here is left unordered with
// what the caller does next (restoring a state, stepping again, ending a
// capture).  Returns the first failure.
template <class Status, class Begin, class Body, class End, class Join>
Status with_side_work(Status ok, Begin begin, Body body, End end, Join join) {
    Status s = begin();
    if (s == ok) s = body();
    if (s == ok) s = end();
    if (s != ok) join();
    return s;
}

} // namespace hp
