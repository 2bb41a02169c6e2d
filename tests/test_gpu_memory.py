"""Calls on a GPU whose memory is nearly full: what needs much memory to be fast
gives way to what needs little, and the results stay."""

import contextlib

import numpy as np
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


@pytest.mark.parametrize("n,nchan,n_ant,n_times,direct,most,step", [
    (512, 8, 9, 31, 2, 256, 8),       # image-sized buffers: plan, grids, beam table
    (64, 2, 60, 1200, 1, 768, 12),    # visibilities: the plan's scratch among set-up's copies
])
def test_created_wherever_the_direct_sums_are(n, nchan, n_ant, n_times, direct, most, step):
    """From plenty of memory down to where the direct-sum engine is refused: the
    default engine is created as long as the direct one is, as a non-uniform FFT
    first and as direct sums then.  Those take the visibilities in another order
    (by tile) than the engine by itself: 1e-5, as the engines agree elsewhere."""
    import torch
    data = synth.generate(synth.small_config(n=n, nchan=nchan, seed=3, n_ant=n_ant,
                                             n_times=n_times))
    ref, chi2, out = {}, {}, torch.zeros((2, n, n), device="cuda")
    img = None
    for engine in (direct, 0):
        prob = _problem(data, engine)
        if img is None:
            img = prob.initial_image()
            img[0] += (200.0 * torch.rand(img[0].shape, device="cuda") ** 6)
            prob.chi2(img)  # clips it
        chi2[engine] = prob.chi2(img)
        ref[engine] = prob.dchi2(img).clone()
        assert (prob.dchi2_pairs > 0) == (engine == 0)
        prob.close()
    assert chi2[0] == pytest.approx(chi2[direct], rel=1e-12)
    seen, refused = [], None
    for mb in range(most, 0, -step):
        with only(mb):
            prob = _problem(data, direct)
            if prob is None:
                break
            prob.close()
            # one step of slack: a kernel's first launch takes memory of its own
            assert refused is None, f"refused at {refused} MB, the direct engine not at {mb}"
            prob = _problem(data, 0)
            if prob is None:
                refused = mb
                continue
            pairs = prob.dchi2_pairs
            f = prob.chi2(img)
            out.zero_()
            prob.dchi2(img, out=out)
            prob.close()
        seen.append(pairs)
        assert f == pytest.approx(chi2[0], rel=1e-12)
        if pairs:
            assert torch.equal(out, ref[0]), mb
        else:
            assert (out - ref[direct]).abs().max() <= 1e-5 * ref[direct].abs().max(), mb
    assert seen[0] > 0 and seen[-1] == 0, seen


def test_large_plans_leave_room():
    """A plan of 256 MB and more leaves 4 GB, which the optimisers' vectors and
    the images of a call may need."""
    data = synth.generate(synth.small_config(n=1024, nchan=8, seed=3, n_ant=9, n_times=31))
    prob = _problem(data, 0)
    assert prob.dchi2_pairs > 0
    prob.close()
    for mb, runs in ((6000, True), (4200, False)):
        with only(mb):
            prob = _problem(data, 0)
            assert (prob.dchi2_pairs > 0) == runs
            prob.close()


def _under(mb, call):
    """call() with plenty of memory and with mb MB: the results of both, and the
    kernels that each launched."""
    import gpuvmem_gb300 as gv
    call()  # loads the kernels
    n0 = gv.launch_count()
    plenty = call()
    n1 = gv.launch_count()
    with only(mb):
        little = call()
    return plenty, little, n1 - n0, gv.launch_count() - n1


@pytest.mark.parametrize("scheme", ["uniform", "briggs"])
def test_weighting_channel_by_channel(scheme):
    """The sort of all channels (48 MB here) gives way to a sort for each."""
    import gpuvmem_gb300 as gv
    rng = np.random.default_rng(4)
    C, n, M, cell = 24, 30000, 64, 0.05 / 3600.0
    off = np.arange(C + 1, dtype=np.int64) * n
    freqs = np.linspace(220e9, 240e9, C).astype(np.float32)
    uvw = rng.normal(0, 150.0, (C * n, 3))  # some beyond the grid's edge
    w = (rng.random(C * n) + 0.5).astype(np.float32)
    w[::9] = 0.0
    a, b, na, nb = _under(16, lambda: gv.apply_weighting(scheme, 0.5, M, M, -cell, cell, freqs,
                                                         off, uvw, w))
    assert nb > 2 * na
    assert np.array_equal(a, b, equal_nan=True)


def test_gridding_by_taps():
    """The tiles of all channels (90 MB here) give way to a sort of each
    channel's taps."""
    import gpuvmem_gb300 as gv
    rng = np.random.default_rng(5)
    C, n, M, cell = 64, 3000, 128, 0.05 / 3600.0
    off = np.arange(C + 1, dtype=np.int64) * n
    freqs = np.linspace(220e9, 240e9, C).astype(np.float32)
    uvw = rng.normal(0, 0.2 * 1.3e-3 / (cell * np.pi / 180.0), (C * n, 3))
    vo = rng.normal(0, 1, (C * n, 2)).astype(np.float32)
    w = rng.uniform(0.5, 2.0, C * n).astype(np.float32)
    table = rng.uniform(-0.2, 1.0, (3, 3)).astype(np.float32)
    a, b, na, nb = _under(24, lambda: gv.grid_visibilities(table, (1, 1), M, M, -cell, cell, freqs,
                                                           off, uvw, vo, w))
    assert nb > 2 * na
    for x, y in zip(a, b):
        assert x.tobytes() == y.tobytes()


def test_candidates_one_after_another():
    """The grids of all candidates at once (134 MB here) give way to one image
    after another."""
    import gpuvmem_gb300 as gv
    import torch
    data = synth.generate(synth.small_config(n=512, nchan=4, seed=3, n_ant=9, n_times=31))
    prob = gv.Problem(data, [gv.term("Chi2", 1.0), gv.term("Entropy", 0.01, prior_value=0.001,
                                                           eta=-1.0)])
    prob.set_iteration(1)
    imgs = prob.initial_image()[None].repeat(16, 1, 1, 1)
    imgs[:, 0] += torch.rand((16, 512, 512), device="cuda") ** 6
    with only(64):
        little = prob.objective_many(imgs)
        n0 = gv.launch_count()
        assert prob.objective_many(imgs) == little
        n1 = gv.launch_count()
    plenty = prob.objective_many(imgs)
    assert gv.launch_count() - n1 < (n1 - n0) / 4
    assert plenty == little
