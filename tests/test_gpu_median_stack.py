"""Median stack on the GPU against the oracle (MedianStackKernels.h:19-55,
CpuComputeBackend.cpp:136-159), bit for bit: the packed two-scalar path
(aligned buffers, even scalar count), the one-scalar path (odd counts,
unaligned buffers), saturated and tied values, and the fused warp + median of
a burst (WarpPerspective of every frame, then MedianStack) including the
burst workload's generator at reduced size."""
import numpy as np
import pytest

from image360_b200 import ComputeResult, synth

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint16)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 12, 16, 17, 24, 32])
def test_median_packed_path_exact(backend, oracle_c, n):
    import torch
    rng = np.random.default_rng(100 + n)
    w, h = 64, 21  # 4032 scalars: even, so two per thread
    ins = [rng.integers(0, 16384, (h, w, 3), dtype=np.uint16) for _ in range(n)]
    for i in range(n):  # saturated values, kept and clipped, and ties
        ins[i][3, :, 0] = 65535
        ins[i][4, 2 * i % w, :] = 65535
        ins[i][6, :, 1] = 7
    if n > 4:
        ins[0][7, :, :] = 60000
    d_in = [_dev(a) for a in ins]
    d_out = torch.zeros((h, w, 3), dtype=torch.int16, device="cuda")
    assert backend.launch_median([t.data_ptr() for t in d_in], w, h, d_out.data_ptr()) == ComputeResult.SUCCESS
    torch.cuda.synchronize()
    assert np.array_equal(_host(d_out), oracle_c.median(ins, 2.0))


@pytest.mark.parametrize("n,sigma", [(6, 2.0), (16, 1.0), (16, 3.5), (32, 0.5)])
def test_median_unaligned_and_sigma(backend, oracle_c, n, sigma):
    """Inputs starting 2 bytes past an alignment boundary take the one-scalar
    path; several clip thresholds."""
    import torch
    rng = np.random.default_rng(7 * n)
    w, h = 30, 10
    ins = [rng.integers(0, 16384, (h, w, 3), dtype=np.uint16) for _ in range(n)]
    for i in range(0, n, 5):
        ins[i][:, ::3, :] = 16383
    bufs = []
    for a in ins:
        b = torch.zeros(a.size + 1, dtype=torch.int16, device="cuda")
        b[1:] = torch.from_numpy(a.reshape(-1).view(np.int16)).cuda()
        bufs.append(b)
    d_out = torch.zeros(h * w * 3 + 1, dtype=torch.int16, device="cuda")
    ptrs = [b.data_ptr() + 2 for b in bufs]
    assert backend.launch_median(ptrs, w, h, d_out.data_ptr() + 2, sigma) == ComputeResult.SUCCESS
    torch.cuda.synchronize()
    got = d_out[1:].cpu().numpy().view(np.uint16).reshape(h, w, 3)
    assert np.array_equal(got, oracle_c.median(ins, sigma))


def _near_identity(rng, w, h, shift, rot_deg):
    th = np.radians(rng.uniform(-rot_deg, rot_deg))
    tx, ty = rng.uniform(-shift, shift, 2)
    c, s = np.cos(th), np.sin(th)
    cx, cy = (w - 1) / 2.0, (h - 1) / 2.0
    return np.array([[c, -s, cx - c * cx + s * cy + tx], [s, c, cy - s * cx - c * cy + ty], [0, 0, 1.0]])


@pytest.mark.parametrize("n,dw,dh,off", [(1, 50, 40, (0, 0)), (3, 61, 33, (2, -1)), (4, 64, 48, (0, 0)),
                                         (9, 77, 31, (-3, 5)), (16, 120, 90, (0, 0)), (32, 45, 21, (1, 1))])
def test_warp_median_matches_warp_then_median(backend, oracle_c, n, dw, dh, off):
    import torch
    rng = np.random.default_rng(n * 1000 + dw)
    sw, sh = 70, 52
    frames = [rng.integers(0, 16384, (sh, sw, 3), dtype=np.uint16) for _ in range(n)]
    for f in frames[: max(1, n // 4)]:
        f[10:20, 5:25, :] = 16383  # transient outliers
    Hs = np.stack([synth.inverse_homography_f32(_near_identity(rng, sw, sh, 3.0, 0.5)) for _ in range(n)])
    d_f = [_dev(f) for f in frames]
    d_out = torch.zeros((dh, dw, 3), dtype=torch.int16, device="cuda")
    rc = backend.launch_warp_median([t.data_ptr() for t in d_f], sw, sh, Hs, d_out.data_ptr(), dw, dh, *off)
    assert rc == ComputeResult.SUCCESS, backend.get_last_error()
    torch.cuda.synchronize()
    warped = [oracle_c.warp(f, dw, dh, H, *off) for f, H in zip(frames, Hs)]
    assert np.array_equal(_host(d_out), oracle_c.median(warped, 2.0))


def test_burst_workload_scaled_exact(backend, oracle_c):
    """The burst generator at 8% size (16 frames of 320x240, 5% outliers):
    demosaic + fused warp/median against the oracle's demosaic, warp of every
    frame and median."""
    import torch
    cfg = synth.scaled_stack(synth.C2, 0.08)
    st = synth.make_stack(cfg)
    assert all(0.05 <= f < 0.15 for f in st.outlier_frac)
    black, cm, rc, filt = synth.demosaic_params(cfg)
    w, h = cfg.frame_w, cfg.frame_h
    d_rgb = []
    host_rgb = []
    for c in st.cfa:
        d_c = _dev(c.numpy())
        d_o = torch.empty((h, w, 3), dtype=torch.int16, device="cuda")
        assert backend.launch_demosaic(d_c.data_ptr(), w, h, black, cm, rc, filt, d_o.data_ptr()) == 0
        d_rgb.append(d_o)
        host_rgb.append(oracle_c.demosaic(c.numpy(), black, cm, rc, filt))
    Hs = np.stack([synth.inverse_homography_f32(H) for H in st.to_ref])
    d_out = torch.zeros((h, w, 3), dtype=torch.int16, device="cuda")
    assert backend.launch_warp_median([t.data_ptr() for t in d_rgb], w, h, Hs, d_out.data_ptr(), w, h) == 0
    torch.cuda.synchronize()
    for d, hr in zip(d_rgb, host_rgb):
        assert np.array_equal(_host(d), hr)
    warped = [oracle_c.warp(f, w, h, H) for f, H in zip(host_rgb, Hs)]
    assert np.array_equal(_host(d_out), oracle_c.median(warped, 2.0))


def test_warp_median_argument_errors(backend):
    assert backend.launch_warp_median([], 10, 10, np.eye(3)[None], 0, 10, 10) == ComputeResult.INVALID_PARAM
    assert backend.launch_warp_median([1] * 33, 10, 10, np.tile(np.eye(3), (33, 1, 1)), 1, 10, 10) == \
        ComputeResult.INVALID_PARAM
    assert backend.launch_warp_median([1], 0, 10, np.eye(3)[None], 1, 10, 10) == ComputeResult.INVALID_PARAM


@pytest.mark.parametrize("n", range(1, 33))
def test_median_every_stack_size_and_threshold(backend, oracle_c, n):
    """Every sorting network, on an odd scalar count (the last scalar alone)
    of full-range values, with thresholds that keep nothing (the reference
    then keeps everything), one value, or all.  Exact."""
    import torch
    rng = np.random.default_rng(5000 + n)
    w, h = 37, 11
    ins = [rng.integers(0, 65536, (h, w, 3), dtype=np.uint16) for _ in range(n)]
    for a in ins:
        a[2] = 65535
        a[3] = 40000 + rng.integers(0, 3)
        a[4, ::2] = 0
    d_in = [_dev(a) for a in ins]
    for sigma in (2.0, 0.3, 0.0, -1.0, float("inf"), float("nan")):
        d_out = torch.zeros((h, w, 3), dtype=torch.int16, device="cuda")
        assert backend.launch_median([t.data_ptr() for t in d_in], w, h, d_out.data_ptr(), sigma) == 0
        torch.cuda.synchronize()
        assert np.array_equal(_host(d_out), oracle_c.median(ins, sigma)), sigma


@pytest.mark.parametrize("sw,sh,dw,dh,shift,proj", [(2, 2, 5, 4, 0, False), (3, 5, 33, 9, 1, True),
                                                    (64, 40, 64, 8, 0, False), (65, 41, 63, 17, 1, False),
                                                    (66, 30, 129, 7, 1, True), (1, 7, 4, 4, 0, False)])
def test_warp_taps_at_every_phase(backend, oracle_c, sw, sh, dw, dh, shift, proj):
    """Taps read as aligned words: odd source widths and a source that starts
    one sample past a word put the rows at both phases; destination widths
    around the 64-pixel segment; affine and projective homographies; gains.
    Full-range values.  Exact, alone and as a stack of two."""
    import torch
    rng = np.random.default_rng(sw * 100 + dw)
    src = rng.integers(0, 65536, (sh, sw, 3), dtype=np.uint16)
    src[0, 0] = 65535
    src[-1, -1] = 65535
    buf = torch.zeros(src.size + 1, dtype=torch.int16, device="cuda")
    buf[shift:shift + src.size] = _dev(src).reshape(-1)
    H = np.array([[0.93, 0.11, -1.25], [-0.08, 0.97, 0.75], [0, 0, 1]], np.float32)
    if proj:
        H[2] = [3e-4, -2e-4, 1.0001]
    for off in ((0, 0), (-3, 2)):
        ref = oracle_c.warp(src, dw, dh, H, *off)
        for gain in (1.0, 1.37, 0.0, -1.0):
            out = torch.full((dh, dw, 3), 9, dtype=torch.int16, device="cuda")
            assert backend.launch_warp(buf.data_ptr() + 2 * shift, sw, sh, out.data_ptr(), dw, dh, H, *off,
                                       gain=gain) == 0
            torch.cuda.synchronize()
            exp = ref if gain == 1.0 else oracle_c.gain(ref.copy(), gain).reshape(ref.shape)
            assert np.array_equal(_host(out), exp), (off, gain)
        out = torch.zeros((dh, dw, 3), dtype=torch.int16, device="cuda")
        p = buf.data_ptr() + 2 * shift
        assert backend.launch_warp_median([p, p], sw, sh, np.stack([H, H]), out.data_ptr(), dw, dh, *off) == 0
        torch.cuda.synchronize()
        assert np.array_equal(_host(out), ref)


@pytest.mark.parametrize("sw,sh,dw,dh,shift,proj", [(301, 200, 502, 501, 0, False), (301, 200, 501, 502, 1, True),
                                                    (700, 511, 1025, 249, 0, True), (700, 511, 63, 4001, 1, False),
                                                    (2, 2, 520, 490, 0, False), (333, 77, 500, 503, 1, True),
                                                    (333, 77, 503, 500, 0, False)])
def test_warp_of_large_tiles_at_every_phase(backend, oracle_c, sw, sh, dw, dh, shift, proj):
    """Tiles around and above the size from which a lane makes two pixels, whose
    taps are words at both phases: widths around the 64-pixel segment, affine
    and projective homographies, gains.  Full-range values.  Exact."""
    import torch
    rng = np.random.default_rng(sw * 100 + dw)
    src = rng.integers(0, 65536, (sh, sw, 3), dtype=np.uint16)
    src[0, 0] = 65535
    src[-1, -1] = 65535
    buf = torch.zeros(src.size + 1, dtype=torch.int16, device="cuda")
    buf[shift:shift + src.size] = _dev(src).reshape(-1)
    H = np.array([[0.93, 0.11, -1.25], [-0.08, 0.97, 0.75], [0, 0, 1]], np.float32)
    if proj:
        H[2] = [3e-4, -2e-4, 1.0001]
    for off in ((0, 0), (-3, 2)):
        ref = oracle_c.warp(src, dw, dh, H, *off)
        for gain in (1.0, 1.37, 0.0, -1.0):
            out = torch.full((dh, dw, 3), 9, dtype=torch.int16, device="cuda")
            assert backend.launch_warp(buf.data_ptr() + 2 * shift, sw, sh, out.data_ptr(), dw, dh, H, *off,
                                       gain=gain) == 0
            torch.cuda.synchronize()
            exp = ref if gain == 1.0 else oracle_c.gain(ref.copy(), gain).reshape(ref.shape)
            assert np.array_equal(_host(out), exp), (off, gain)
