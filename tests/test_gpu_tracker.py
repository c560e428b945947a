"""GPU parity: the tracker (reference beam_tracker.cpp:90-146).

mode 0 follows the reference float32 order; its only freedom is the last bit
of the FP64 sin/cos of the phase, so it must match the oracle to 1e-6
relative (and almost everywhere exactly).  mode 1 (tensor-pipe streaming
kernel, fp16 hi+lo weights, fp32 sums) must match within the reference's
CUDA tolerance |gpu - cpu| <= 1e-3 + 1e-5 |cpu| (tests/cuda/
test_cuda_packed.cu:24-25), and its per-window sums within 1e-5 relative of
the FP64 sum.
The fp16 weights are those of windows of up to 16 spectra; longer windows take
int8 digits of the weights and are held to the same bars.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import random_voltage

pytestmark = pytest.mark.gpu
F = 336


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _run(torch, api, mode, v, pos, freq, dirs, T, A, S, want_int=True, want_integ=True):
    W = len(dirs)
    inten = torch.full((T * F,), -1.0, dtype=torch.float32, device="cuda") if want_int else None
    integ = torch.full((W * F,), -1.0, dtype=torch.float32, device="cuda") if want_integ else None
    api.tracker(None, mode, _dev(torch, v), _dev(torch, pos), _dev(torch, api.wave_numbers(freq)),
                _dev(torch, dirs), inten, integ, api.Dimensions(T, F, A, 1), S)
    torch.cuda.synchronize()
    return (None if inten is None else inten.cpu().numpy().reshape(T, F),
            None if integ is None else integ.cpu().numpy().reshape(W, F))


def _case(orc, api, T, A, S, seed, moving=True):
    pos, freq = api.default_positions(A), api.channelized_frequencies(F)
    l0, m0, rl, rm = (0.05, -0.03, 3e-5, -2e-5) if moving else (0.1, 0.0, 0.0, 0.0)
    dirs = api.tracker_window_directions(l0, m0, rl, rm, T, S)
    v = random_voltage(T, F, A, seed)
    ww = orc.tracker_weights(dirs, pos, freq)
    return pos, freq, dirs, v, orc.tracker(v, ww, T, F, A, S)


@pytest.mark.parametrize("A,T,S", [(32, 100, 16), (64, 257, 64), (128, 40, 10), (256, 33, 32)])
def test_mode0_reference_order(cuda, orc, A, T, S):
    from beamform_project_b200 import api
    pos, freq, dirs, v, ref = _case(orc, api, T, A, S, seed=A)
    inten, integ = _run(cuda, api, 0, v, pos, freq, dirs, T, A, S)
    assert np.allclose(inten, ref, rtol=1e-6, atol=1e-6)
    assert np.mean(inten == ref) > 0.99
    # per-window sums in increasing time (src/temporal_integration.cpp:95-109)
    exp = orc.integrate(ref[..., None], T, F, 1, S)[..., 0]
    assert np.allclose(integ, exp, rtol=1e-6, atol=1e-5)


@pytest.mark.parametrize("A,T,S", [(32, 100, 16), (64, 1024, 256), (64, 300, 320),
                                   (128, 50, 10), (256, 48, 32)])
def test_mode1_streaming_within_tolerance(cuda, orc, A, T, S):
    from beamform_project_b200 import api
    pos, freq, dirs, v, ref = _case(orc, api, T, A, S, seed=T)
    inten, integ = _run(cuda, api, 1, v, pos, freq, dirs, T, A, S)
    err = np.abs(inten.astype(np.float64) - ref)
    assert np.all(err <= 1e-3 + 1e-5 * np.abs(ref)), float(np.max(err - 1e-5 * np.abs(ref)))
    exp64 = orc.integrate(ref[..., None], T, F, 1, S)[..., 0].astype(np.float64)
    assert np.all(np.abs(integ - exp64) <= 1e-3 + 1e-5 * np.abs(exp64))


def test_mode1_integrated_only_and_point_source(cuda, orc, ref):
    """A source moving along the tracked trajectory stays in the beam: the
    tracked power is the coherent maximum and equals the oracle."""
    from beamform_project_b200 import api
    T, A, S = 128, 64, 32
    pos, freq = api.default_positions(A), api.channelized_frequencies(F)
    l0, m0, rl, rm = 0.02, 0.01, 1e-4, 0.0
    v = ref.ref_make_moving_point_source(T, F, A, pos, freq, l0, m0, rl, rm, 4.0)
    dirs = api.tracker_window_directions(l0, m0, rl, rm, T, S)
    exp = orc.tracker(v, orc.tracker_weights(dirs, pos, freq), T, F, A, S)
    _, integ = _run(cuda, api, 1, v, pos, freq, dirs, T, A, S, want_int=False)
    exp_w = exp.reshape(T // S, S, F).astype(np.float64).sum(axis=1)
    assert np.allclose(integ, exp_w, rtol=1e-5, atol=1e-3)
    # the tracked beam collects (close to) the full coherent power A^2 * 16
    assert float(np.median(exp)) > 0.5 * A * A * 16


@pytest.mark.parametrize("A,T,S", [(32, 1003, 1), (32, 7005, 7), (32, 950, 16), (64, 530, 17), (64, 200, 64),
                                   (64, 200, 65), (64, 161, 33), (128, 130, 129), (256, 37, 12)])
@pytest.mark.parametrize("outputs", ["both", "integrated"])
def test_mode1_window_edges(cuda, orc, A, T, S, outputs):
    """Both forms of the streaming kernel (windows up to 64 spectra in runs of
    up to 16 per CTA, longer ones one per CTA) at block, run and stage edges,
    with a partial last window; the tolerance is the file's."""
    from beamform_project_b200 import api
    pos, freq, dirs, v, ref = _case(orc, api, T, A, S, seed=T + S)
    inten, integ = _run(cuda, api, 1, v, pos, freq, dirs, T, A, S, want_int=outputs == "both")
    if inten is not None:
        assert np.all(np.abs(inten.astype(np.float64) - ref) <= 1e-3 + 1e-5 * np.abs(ref))
    exp64 = orc.integrate(ref[..., None], T, F, 1, S)[..., 0].astype(np.float64)
    assert np.all(np.abs(integ - exp64) <= 1e-3 + 1e-5 * np.abs(exp64))


@pytest.mark.parametrize("A,S,W", [(64, 17, 530), (32, 33, 243), (64, 64, 119), (32, 64, 119), (64, 65, 119),
                                   (32, 65, 119), (64, 72, 119), (32, 80, 119), (64, 80, 119), (64, 81, 119)])
@pytest.mark.parametrize("outputs", ["both", "integrated"])
def test_mode1_runs_of_windows(cuda, orc, A, S, W, outputs):
    """Launches with so many windows that a CTA keeps several of them where
    the form allows it, around the length at which the one-window form
    begins; the last window is partial and no window keeps the buffers' fill
    value.  The tolerance is the file's."""
    from beamform_project_b200 import api
    T = (W - 1) * S + 7
    pos, freq, dirs, v, ref = _case(orc, api, T, A, S, seed=S)
    inten, integ = _run(cuda, api, 1, v, pos, freq, dirs, T, A, S, want_int=outputs == "both")
    if inten is not None:
        assert np.all(np.abs(inten.astype(np.float64) - ref) <= 1e-3 + 1e-5 * np.abs(ref))
    exp64 = orc.integrate(ref[..., None], T, F, 1, S)[..., 0].astype(np.float64)
    assert np.all(np.abs(integ - exp64) <= 1e-3 + 1e-5 * np.abs(exp64))


@pytest.mark.parametrize("A", [32, 64, 256])
@pytest.mark.parametrize("S", [10, 32, 320])
def test_mode1_not_finite(cuda, orc, A, S):
    """A window direction or wave number that is not finite gives NaN powers
    in its window or channel, in every form of the streaming kernel as in the
    reference order, and changes no other value."""
    from beamform_project_b200 import api
    torch = cuda
    T = 3 * S + 5
    pos, freq, dirs, v, _ = _case(orc, api, T, A, S, seed=S)
    kw = np.asarray(api.wave_numbers(freq))
    bad_dirs, bad_kw = dirs.copy(), kw.copy()
    bad_dirs[1, 0], bad_dirs[3, 1] = np.nan, np.inf
    bad_kw[11], bad_kw[330] = np.nan, np.inf

    def run(mode, kw, dirs):
        inten = torch.full((T * F,), -1.0, dtype=torch.float32, device="cuda")
        integ = torch.full((4 * F,), -1.0, dtype=torch.float32, device="cuda")
        api.tracker(None, mode, _dev(torch, v), _dev(torch, pos), _dev(torch, kw), _dev(torch, dirs), inten, integ,
                    api.Dimensions(T, F, A, 1), S)
        return inten.cpu().numpy().reshape(T, F), integ.cpu().numpy().reshape(4, F)

    good, bad, order = run(1, kw, dirs), run(1, bad_kw, bad_dirs), run(0, bad_kw, bad_dirs)
    win = np.zeros((4, F), bool)
    win[[1, 3]] = True
    win[:, [11, 330]] = True
    expect = win[np.arange(T) // S], win
    for g, b, o, e in zip(good, bad, order, expect):
        assert np.array_equal(np.isnan(b), e) and np.array_equal(np.isnan(o), e)
        assert np.array_equal(b[~e], g[~e])


@pytest.mark.parametrize("S", [2**31, 2**32, 2**32 + 5])
@pytest.mark.parametrize("mode", [0, 1])
def test_window_longer_than_32_bits(cuda, orc, mode, S):
    """An integration length past 32 bits is one window, as any length past
    the run is."""
    from beamform_project_b200 import api
    A, T = 64, 50
    pos, freq, dirs, v, _ = _case(orc, api, T, A, T, seed=3)
    whole, longer = (_run(cuda, api, mode, v, pos, freq, dirs, T, A, s) for s in (T, S))
    for a, b in zip(whole, longer):
        assert np.array_equal(a, b)
