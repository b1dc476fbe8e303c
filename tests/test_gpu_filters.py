"""Receiver filters on the GPU (csrc/filters.cu) against the FP64 oracle (oracle/filters.py):
Pach_SP.ETCToFilter (Pach_SP.cs:1584-1680) and Directional_Histogram.Create_Filter
(Classes_Receivers.cs:1910-1995), through the C ABI.

Both sides are FP64 transforms of the same sums; the GPU's four-step radix-2 transforms and numpy's
pocketfft round differently, so a filter must match within 1e-11 of its largest magnitude."""
import ctypes as C

import numpy as np
import pytest

from oracle import filters as F
from pachydermacoustic_universal_gb300 import _capi, rooms, tracer
from pachydermacoustic_universal_gb300.simulation import (GeodesicSource, Pach_SP, Polygon_Scene, Receiver_Bank,
                                                          SplitRayTracer)

pytestmark = pytest.mark.gpu
RTOL_MAX = 1e-11


def _close(got, ref):
    ref = np.asarray(ref)
    assert got.shape == ref.shape
    scale = max(np.abs(ref).max(), 1e-300)
    err = np.abs(got - ref).max() / scale
    assert err <= RTOL_MAX, err


@pytest.mark.parametrize("T,fs", [(1, 1000), (37, 1000), (3500, 1000), (16385, 1000), (16386, 1000), (2000, 44100),
                                  (40000, 44100)])
def test_etc_to_filter_matches_oracle(T, fs):
    rng = np.random.default_rng(T)
    P = rng.random((8, T)) * (rng.random((8, T)) > 0.2)
    swl = rng.uniform(80, 130, 8)
    _close(tracer.etc_to_filter(P, swl, fs), F.etc_to_filter(P, swl, fs))


@pytest.mark.parametrize("T", [2, 255, 4095, 4096, 4097, 8193, 16384, 49153, 49154])
@pytest.mark.parametrize("fs", [1000, 44100])
def test_integer_transforms_over_lengths(T, fs):
    """The integer transforms' classes (T + 16383 points up to 16384, 32768, 65536; folds of 4096 samples) and the
    first length of the FP64 transforms, with an envelope that falls over 200 dB, a silent band and one outlier.
    Inputs are rounded at 2^-60 of their largest value, so only numpy's transforms round: 1e-14 of the peak."""
    rng = np.random.default_rng(T)
    P = rng.random((8, T)) * 10.0 ** (-10.0 * np.arange(T) / T)
    P[3] = 0.0
    P[5, T // 2] += 40.0
    swl = rng.uniform(80, 130, 8)
    got, ref = tracer.etc_to_filter(P, swl, fs), F.etc_to_filter(P, swl, fs)
    assert np.abs(got - ref).max() <= 1e-14 * np.abs(ref).max()


def test_silent_and_undefined_envelopes():
    """A filter of silence is zero; a value that is not finite makes its whole filter undefined (as every
    output of a transform of it is), and no other filter of the call."""
    P = np.random.default_rng(3).random((4, 8, 600))
    P[1] = 0.0
    P[2, 4, 100] = np.inf
    P[3, 7, 5] = np.nan
    got = tracer.etc_to_filter(P, None, 1000)
    _close(got[0], F.etc_to_filter(P[0], [120] * 8, 1000))
    assert not got[1].any()
    assert np.isnan(got[2]).all() and np.isnan(got[3]).all()


def test_etc_to_filter_batch_and_default_level():
    rng = np.random.default_rng(9)
    P = rng.random((5, 8, 700))
    got = tracer.etc_to_filter(P, None, 1000)
    for i in range(5):
        _close(got[i], F.etc_to_filter(P[i], [120] * 8, 1000))
    _close(Pach_SP.ETCToFilter(list(P[0]), [120] * 8, 1000), got[0])


def _synthetic_histograms(R, T, seed):
    rng = np.random.default_rng(seed)
    E = rng.random((R, 8, T)) * (rng.random((R, 8, T)) > 0.4)
    P = np.sqrt(E * 413.0)
    P[:, :, ::7] += 0.5          # pressure where energy is 0: the directional envelopes stay 0 there
    u = rng.normal(size=(R, 3, 8, T))
    Dp = np.where(u > 0, u, 0.0) * E[:, None]
    Dn = np.where(u < 0, u, 0.0) * E[:, None]
    return E, P, Dp, Dn


def test_receiver_filters_match_oracle():
    E, P, Dp, Dn = _synthetic_histograms(3, 900, 4)
    swl = [100, 105, 110, 115, 120, 125, 118, 112]
    got = tracer.receiver_filters(P, E, Dp, Dn, swl=swl, sample_rate=1000)
    assert got.shape == (3, 7, 900 + 12287)
    for r in range(3):
        ref = F.receiver_filters(E[r], P[r], Dp[r], Dn[r], swl, 1000)
        for k in range(7):
            _close(got[r, k], ref[k])
    omni = tracer.receiver_filters(P, swl=swl, sample_rate=1000)
    assert omni.shape == (3, 1, 900 + 12287)
    np.testing.assert_allclose(omni[:, 0], got[:, 0], rtol=0, atol=1e-12 * np.abs(got[:, 0]).max())


def test_run_filters_equal_filters_of_the_scaled_histograms():
    w = rooms.shoebox_c1()
    w.cutoff_s = 0.5
    ds = tracer.DeviceScene(w.scene)
    run = tracer.Run(ds, w.sources, w.receivers, tracer.make_params(rays=3000, cutoff_length_m=w.cutoff_length_m,
                                                                    hist_cotime_ms=500.0, seed=11))
    run.wait()
    h = run.histograms(scaled=True)
    swl = np.array(w.sources[0].power_db)
    got = run.filters(directional=True, swl=swl)
    ref = tracer.receiver_filters(h["pressure"], h["energy"], h["dir_pos"], h["dir_neg"], swl=swl, sample_rate=1000)
    for r in range(got.shape[0]):
        for k in range(7):
            _close(got[r, k], ref[r, k])
    o = F.receiver_filters(h["energy"][0], h["pressure"][0], h["dir_pos"][0], h["dir_neg"][0], swl, 1000)
    for k in range(7):
        _close(got[0, k], o[k])
    run.close()
    ds.close()


def test_device_form_in_several_passes_equals_one_pass():
    torch = pytest.importorskip("torch")
    E, P, Dp, Dn = _synthetic_histograms(4, 500, 7)
    dev = torch.device("cuda:0")
    t = {k: torch.from_numpy(v).to(dev) for k, v in dict(E=E, P=P, Dp=Dp, Dn=Dn).items()}
    scale = torch.tensor([1.0, 0.5, 2.0, 0.25], dtype=torch.float64, device=dev)
    L = _capi.lib()
    full = L.pach_filters_workspace_bytes(28, 500)
    one = L.pach_filters_workspace_bytes(1, 500)
    outs = []
    for wsb in (full, one + 1000):
        ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
        out = torch.zeros((4, 7, 500 + 12287), dtype=torch.float64, device=dev)
        st = L.pach_filters_device(t["E"].data_ptr(), t["P"].data_ptr(), t["Dp"].data_ptr(), t["Dn"].data_ptr(),
                                   scale.data_ptr(), 4, 500, 7, 1000, None, 4096, out.data_ptr(), ws.data_ptr(), wsb,
                                   C.c_void_p(torch.cuda.current_stream().cuda_stream))
        _capi.check(st)
        torch.cuda.synchronize()
        outs.append(out.cpu().numpy())
    np.testing.assert_array_equal(outs[0], outs[1])
    ref = tracer.receiver_filters(P * np.array([1.0, 0.5, 2.0, 0.25])[:, None, None], E, Dp, Dn, sample_rate=1000)
    _close(outs[0], ref)


@pytest.mark.parametrize("kinds", [1, 7])
@pytest.mark.parametrize("T", [500, 49154])
def test_receiver_factors_of_any_sign(kinds, T):
    """d_scale multiplies a receiver's envelopes as it is, a factor below zero (phase reversal) or of zero too, for the
    integer transforms and (T + 16383 > 65536) the FP64 ones: the filters are the plain ones times the factor."""
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda:0")
    E, P, Dp, Dn = (torch.from_numpy(x).to(dev) for x in _synthetic_histograms(4, T, 9))
    L = _capi.lib()
    wsb = L.pach_filters_workspace_bytes(4 * kinds, T)
    ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
    got = []
    f = [1.0, -1.0, -0.375, 0.0]
    for scale in (None, torch.tensor(f, dtype=torch.float64, device=dev)):
        out = torch.full((4, kinds, T + 12287), np.nan, dtype=torch.float64, device=dev)
        _capi.check(L.pach_filters_device(E.data_ptr(), P.data_ptr(), Dp.data_ptr(), Dn.data_ptr(),
                                          None if scale is None else scale.data_ptr(), 4, T, kinds, 1000, None, 4096,
                                          out.data_ptr(), ws.data_ptr(), wsb, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
        got.append(out.cpu().numpy())
    for r in range(4):
        for k in range(kinds):
            peak = np.abs(got[0][r, k]).max()
            assert peak > 0 and np.abs(got[1][r, k] - f[r] * got[0][r, k]).max() <= 1e-14 * peak, (r, k)


def test_directions_of_energies_at_the_ends_of_the_range():
    """P Dir / E where P / E alone leaves the normal range, upwards or downwards, and the result does not."""
    E, P, Dp, Dn = _synthetic_histograms(3, 300, 4)
    ref = tracer.receiver_filters(P, E, Dp, Dn, sample_rate=1000)
    big, small = 2.0**1000, 2.0**-60  # (P small) / (E big) is subnormal; times (Dir big) it is P Dir / E small again
    got = tracer.receiver_filters(P * small, E * big, Dp * big, Dn * big, sample_rate=1000)
    for r in range(3):
        for k in range(7):
            peak = np.abs(ref[r, k]).max()
            assert np.abs(got[r, k] / small - ref[r, k]).max() <= 1e-14 * peak, (r, k)


def _device_filters(P, wsb):
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda:0")
    n, _, T = P.shape
    p, ws = torch.from_numpy(P).to(dev), torch.empty(wsb, dtype=torch.uint8, device=dev)
    out = torch.full((n, T + 16383), np.nan, dtype=torch.float64, device=dev)
    _capi.check(_capi.lib().pach_filters_device(None, p.data_ptr(), None, None, None, n, T, 1, 1000, None, 0, out.data_ptr(),
                                                ws.data_ptr(), wsb, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    return out


def test_a_workspace_for_thousands_of_filters_equals_the_recommended_one():
    """More single filters than a launch's grid has rows for, with room for all of them at once (2.7 GB)."""
    n = 8200
    P = np.random.default_rng(5).random((n, 8, 1))
    recommended = _capi.lib().pach_filters_workspace_bytes(n, 1)
    one = _capi.lib().pach_filters_workspace_bytes(1, 1)
    a, b = _device_filters(P, recommended), _device_filters(P, one + n * 330_000)
    assert bool((a == b).all())
    _close(b[n - 1].cpu().numpy(), F.etc_to_filter(P[n - 1], [120] * 8, 1000))


@pytest.mark.parametrize("T,least", [(1, 5112064), (500, 9048064), (3500, 9072128), (16386, 17039616), (49153, 17301760)])
def test_workspaces_of_the_fp64_transforms_are_still_taken(T, least):
    """A workspace too small for one filter's integer transforms but large enough for its FP64 ones (`least` bytes, by
    their layout) is taken, a byte less refused; the longest length with integer transforms and the first of each
    transform length."""
    assert _capi.lib().pach_filters_workspace_bytes(1, T) > least
    P = np.random.default_rng(T).random((2, 8, T))
    got = _device_filters(P, least).cpu().numpy()
    for i in range(2):
        _close(got[i], F.etc_to_filter(P[i], [120] * 8, 1000))
    with pytest.raises(_capi.PachError):
        _device_filters(P, least - 1)


def test_receiver_bank_create_filter_after_a_split_ray_tracer_run():
    w = rooms.shoebox_c1()
    room = Polygon_Scene.from_arrays(w.scene)
    room.partition()
    src = GeodesicSource([120.0] * 8, w.sources[0].origin, 0)
    bank = Receiver_Bank([r.origin for r in w.receivers], src, room, 1000, 400.0)
    rt = SplitRayTracer(src, bank, room, 0.4 * room.Sound_speed(0), [0, 7], -1, 2000, seed=3)
    rt.Begin()
    rt.Combine_ThreadLocal_Results()
    bank.Create_Filter()
    rec = bank.Rec_List[1]
    assert rec.HasFilter() and len(bank.Filter_3Axis(1)) == 6
    ref = F.receiver_filters(rec._E, rec._P, rec._Dp, rec._Dn, [120] * 8, 1000)
    _close(rec.F, ref[0])
    for k in range(6):
        _close(rec.Fdir[k], ref[k + 1])
    seven = bank.Create_Filter([110] * 8, 1)
    assert len(seven) == 7
    _close(seven[0], F.receiver_filters(rec._E, rec._P, rec._Dp, rec._Dn, [110] * 8, 1000)[0])
    _close(bank.Create_Filter([110] * 8, 1, 0), seven[0])
    rt.close()
