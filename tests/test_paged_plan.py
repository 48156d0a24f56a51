"""How a step's paged attention is cut up, looked at on the host."""
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
