"""The hand-over of operand buffers in the flash kernels, walked through in every order on the host.

The element-wise warps fill a buffer and arrive at its barrier; the issuing warp waits for the arrival, starts the product that
reads the buffer, and the product's end frees it. A wait names the parity of a phase, so it cannot tell a barrier that is two
phases ahead from one that has not moved: with fewer barriers than buffers there is an order of steps that waits for good."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "idrak_b200" / "csrc"


def _gets_stuck(buffers: int, barriers: int, blocks: int = 7) -> bool:
    """Whether some order of steps ends with work left. State: blocks filled, blocks taken by the issuer, products ended."""
    seen, todo = set(), [(0, 0, 0)]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        filled, taken, ended = state
        steps = []
        if filled < blocks and (filled < buffers or ended > filled - buffers):      # the buffer's last product has ended
            steps.append((filled + 1, taken, ended))
        if taken < blocks:
            phases = sum(1 for j in range(filled) if j % barriers == taken % barriers)      # completed on this block's barrier
            parity = taken // barriers & 1
            if phases & 1 != parity:                         # mbarrier.try_wait.parity: the phase under way has another parity
                assert filled > taken                        # and never lets a wait through early
                steps.append((filled, taken + 1, ended))
        if ended < taken:
            steps.append((filled, taken, ended + 1))
        if not steps and state != (blocks, blocks, blocks):
            return True
        todo += steps
    return False


@pytest.mark.parametrize("buffers,barriers,stuck", [(1, 1, False), (2, 2, False), (3, 3, False), (2, 1, True)])
def test_a_barrier_per_buffer(buffers, barriers, stuck):
    assert _gets_stuck(buffers, barriers) == stuck


@pytest.mark.parametrize("file,barrier,index", [("flash_fwd.cu", "p_ready", "pb"), ("flash_bwd.cu", "ds_ready", "g & 1"),
                                                ("flash_bwd.cu", "ds_ready", "g % DB")])
def test_the_kernels_have_one(file, barrier, index):
    source = (CSRC / file).read_text()
    assert f"mbar_wait(&{barrier}[{index}], " in source and not re.search(rf"mbar_wait\({barrier},", source)
    assert re.search(rf"mbar_init\(&{barrier}\[1\], 8\)", source) and not re.search(rf"warp_arrive\({barrier}\)", source)
