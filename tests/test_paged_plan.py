"""How a step's paged attention is cut up, looked at on the host."""
import pytest

from megatronapp_b200.inference.dynamic import DynamicInferenceContext


def _context(reqs):
    """A context in a step with ``reqs = [(tokens in the cache, new tokens)]``."""
    cx = DynamicInferenceContext(1 << 16, sum(-(-(a + n) // 16) for a, n in reqs) + 1, 16, 1 << 16, len(reqs))
    for i in range(len(reqs)):
        cx.add_request(str(i))
    old = [(str(i), a) for i, (a, _) in enumerate(reqs) if a]
    if old:
        cx.begin_step(old, "cpu")
        cx.end_step()
    cx.begin_step([(str(i), n) for i, (_, n) in enumerate(reqs)], "cpu")
    return cx


def test_a_step_without_portions_plans_no_tiles():
    cx = _context([(99, 1), (5000, 1), (10, 3)])
    cx._wide_plan = None                                           # not asked
    assert cx._kernel_plan(4, 8, 128) == (3, (0, 1, 5001, 1704, False, 0, 1))


@pytest.mark.parametrize("reqs,group,ng,d,want", [
    ([(0, 159)], 4, 8, 128, (0, 1)), ([(0, 160)], 4, 8, 128, (5, 1)),                    # heads of 128: by the longest context
    ([(0, 320)], 1, 4, 64, (0, 1)), ([(0, 321)], 1, 4, 64, (3, 1)),                      # heads of 64: more than five stages
    ([(113, 113)] * 4, 8, 12, 64, (0, 1)), ([(240, 113)] * 4, 8, 12, 64, (0, 1)),        # more than two waves
    ([(600, 113)] * 4, 8, 12, 64, (32, 1)),                                              # ... of more than eleven stages
    ([(0, 214), (214, 214), (428, 214), (0, 214)], 1, 8, 64, (0, 1)),                    # in two ranges five and a half stages
    ([(2159, 122)], 1, 8, 64, (0, 1)),                                                   # in eight ranges five stages
    ([(2584, 22), (223, 219), (304, 22), (48, 22)], 1, 8, 64, (0, 1)),                   # two ranges where the 64-row tiles take four
    ([(4000, 100)], 1, 4, 64, (0, 1)), ([(9000, 100)], 1, 4, 64, (1, 16))])                # in sixteen ranges four stages, nine
def test_tiles_that_have_the_better_kernel(reqs, group, ng, d, want):
    cuts = _context(reqs)._kernel_plan(group, ng, d)[1]
    assert cuts[-2:] == want
