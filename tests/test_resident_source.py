"""The grid-wide wait of the resident step kernel is an acquire of what the other blocks released.

A missing acquire is a data race by the memory model that the hardware rarely shows, so the kernel's text
is checked: every relaxed load of the arrival counter is followed by a GPU-scope fence before the wait
reports success, and every wait is followed by a block barrier before anything else is read."""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "vortexlab_b200", "csrc", "vl_resident.cuh")


def _text():
    with open(SRC) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_the_grid_wait_acquires():
    t = _text()
    assert t.count("ld.relaxed") == 1
    body = t[t.index("bool poll_arrived"):]
    body = body[:body.index("\n}\n")]
    load, fence, done = body.index("ld.relaxed.gpu"), body.find("fence.acq_rel.gpu"), body.index("return true")
    assert load < fence < done
    assert t.index("red.release.gpu") < t.index("bool poll_arrived")


def test_every_wait_is_followed_by_a_block_barrier():
    t = _text()
    waits = [m.end() for m in re.finditer(r"= poll_arrived\(", t)]
    assert len(waits) >= 2
    for at in waits:
        rest = t[at:]
        assert rest.index("__syncthreads();") < re.search(r"if \(!s_go", rest).start()


def test_no_two_blocks_write_one_word_of_the_outlet_sum():
    """The outlet velocities of the start state go to each block's own shared memory, and one block records the
    offset (all blocks used to store the same values to the same global words)."""
    t = _text()
    start = t[t.index("__global__ void"):t.index("for (int s = 0; s < r.steps; ++s)")]
    assert "s_un[k] = outlet_velocity" in start and "r.un" not in start
    assert re.search(r"if \(bid == 0\) __stcg\(r\.drho \+ slot, drho\);", t)
