"""Calls on a GPU whose memory is nearly full: what needs much memory to be fast
gives way to what needs little, and the results stay."""

import contextlib

import pytest

from gpuvmem_gb300 import synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def only(mb):
    """All but mb MB of the device's memory held."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - mb * MB, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        torch.cuda.synchronize()
        del held
        torch.cuda.empty_cache()


def _problem(data, engine):
    import gpuvmem_gb300 as gv
    try:
        return gv.Problem(data, [gv.term("Chi2", 1.0)], engine=engine)
    except gv.GvError as e:
        assert "memory" in str(e)
        return None


def test_call_after_a_refused_one():
    """A problem that does not fit is refused, and the next one is created."""
    large = synth.generate(synth.small_config(n=1024, nchan=8, seed=3, n_ant=9, n_times=31))
    small = synth.generate(synth.small_config(n=64, nchan=1, seed=3))
    with only(64):
        for engine in (2, 0):
            assert _problem(large, engine) is None
            prob = _problem(small, engine if engine != 2 else 1)
            assert prob is not None
            prob.close()
