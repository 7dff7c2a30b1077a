"""The size and type ranges at which the kernels change their method, against
the oracle: FFT passes, projection tiles, segments of a back projection, the
adjoint's boxes and the CTF's row blocks.

Tolerances: relative L2 1e-5 against the oracle's FP32 restatement or its FP64
FFT of the same CAS images (FP32 rounding of sums and transforms is about
1e-7 times a few), 1e-3 where the oracle is FP64 (rounding can move a
nearest-index table lookup) or the storage is reduced, 1e-6 absolute for the
CTF (the bounds of the other parity tests).
"""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5


def dptr(t):
    return ctypes.c_void_p(t.data_ptr())


def to_dev(a, dev):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(dev)


# M = 36 (radices 3, 3, 4), 100, 140 and 196 (5 and 7; M no multiple of a
# 16-column tile's rows), 200 through interpolation 2 and 2.5, 400 (the last)
@pytest.mark.parametrize("N,interp", [(18, 2.0), (50, 2.0), (70, 2.0), (98, 2.0), (80, 2.5), (200, 2.0)])
def test_fft_passes(cuda, N, interp):
    import multigpugridder_gb300 as gg

    p = O.Params(N, interp)
    n = 5
    rng = np.random.default_rng(N)
    axes = O.quaternion_axes(n, seed=N).astype(np.float32)
    imgs = rng.standard_normal((n, N, N)).astype(np.float32)
    with gg.MultiGPUGridder(N, n, interpFactor=interp, adjustInterpFactor=False) as g:
        g.setCASVolume(rng.standard_normal((p.V,) * 3).astype(np.float32))
        cas = g.forwardProjectCAS(axes)
        assert cas.shape == (n, p.M, p.M)
        out = np.empty((n, N, N), dtype=np.float32)  # forwardProject would set the volume again
        g._call("gg_forward_project", axes.ctypes.data, n, out.ctypes.data, None)
        assert O.rel_l2(out, O.imgs_from_cas_imgs(cas, N)) < TOL
        g.backProject(imgs, axes)
        got = g.getCASVolume()
        g.backProjectCAS(O.cas_imgs_from_imgs(imgs, p.M).astype(np.float32), axes)
        ref = g.getCASVolume()
    assert np.linalg.norm(ref) > 0
    assert O.rel_l2(got, ref) < TOL


@pytest.mark.parametrize("prec", ["bf16", "f16"])
def test_fft_passes_reduced_storage(cuda, prec):
    import multigpugridder_gb300 as gg

    N = 50
    p = O.Params(N)
    axes = O.quaternion_axes(6, seed=3).astype(np.float32)
    # beyond FP16's range before its storage scale
    imgs = (1e5 * np.random.default_rng(4).standard_normal((6, N, N))).astype(np.float32)
    with gg.MultiGPUGridder(N, 6, precision=prec, adjustInterpFactor=False) as g:
        g.backProject(imgs, axes)
        got = g.getCASVolume()
        g.backProjectCAS(O.cas_imgs_from_imgs(imgs, p.M).astype(np.float32), axes)
        ref = g.getCASVolume()
    # the same storage on both sides: only values on a rounding edge differ
    assert np.linalg.norm(ref) > 0
    assert O.rel_l2(got, ref) < 1e-3


# M = 96 (the smallest), tiles of 16 lines with and without remainders, no
# padding at all (N = M), tiles of 8 lines (M > 400)
@pytest.mark.parametrize("N,interp", [(48, 2.0), (70, 2.0), (80, 2.5), (100, 1.0), (200, 2.0), (210, 2.0)])
def test_volume_passes(cuda, N, interp):
    import multigpugridder_gb300 as gg

    p = O.Params(N, interp)
    rng = np.random.default_rng(N)
    vol = rng.standard_normal((N,) * 3).astype(np.float32)
    with gg.MultiGPUGridder(N, 2, interpFactor=interp, adjustInterpFactor=False) as g:
        g.setCASVolume(np.ones((p.V,) * 3, dtype=np.float32))  # no border may be left over
        g.setVolume(vol)
        got = g.getCASVolume()
        cas = rng.standard_normal((p.V,) * 3).astype(np.float32)
        g.setCASVolume(cas)
        back = g.getVol()
    ref = O.cas_from_vol(vol.astype(np.float64), p.hw, p.interp, p.pad)
    assert O.rel_l2(got, ref) < TOL
    assert np.all(got[ref == 0] == 0)
    assert O.rel_l2(back, O.vol_from_cas(cas, N, p.hw, p.interp)) < TOL


# the division's spectrum through the passes (M = 96, 200, no power of two)
@pytest.mark.parametrize("N", [48, 100])
def test_reconstruction_passes(cuda, N):
    import multigpugridder_gb300 as gg

    p = O.Params(N)
    axes = O.quaternion_axes(8, seed=N).astype(np.float32)
    imgs = np.random.default_rng(N).standard_normal((8, N, N)).astype(np.float32)
    with gg.MultiGPUGridder(N, 8, adjustInterpFactor=False) as g:
        vol = g.reconstructVol(imgs, axes)
        cas = g.getCASVolume()
    assert O.rel_l2(vol, O.vol_from_cas(cas, N, p.hw, p.interp)) < TOL


# few tiles (boxes planned the quick way) and more than four a block of the
# grid; volumes smaller than a box; M no multiple of the tile; axes that are
# not orthonormal (boxes that do not fit, windows that leave the volume)
@pytest.mark.parametrize("prec", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("N,n,scale", [(4, 6, 1.0), (18, 5, 1.0), (26, 700, 1.0), (32, 200, 1.0), (32, 4, 1.7), (50, 6, 0.4)])
def test_forward_tiles(cuda, N, n, scale, prec):
    import torch

    import multigpugridder_gb300 as gg

    p = O.Params(N)
    rng = np.random.default_rng(1000 + N)
    cas = rng.standard_normal((p.V,) * 3).astype(np.float32)
    axes = (scale * O.quaternion_axes(n, seed=N + n)).astype(np.float32)
    stored = cas
    if prec != "f32":  # largest value about 5: FP16 is stored at scale 1
        stored = torch.from_numpy(cas).to(torch.bfloat16 if prec == "bf16" else torch.float16).float().numpy()
    ref = O.fp_ref_f32(stored, axes, p.M, p.mask_radius, p.ker)
    with gg.MultiGPUGridder(N, n, precision=prec, adjustInterpFactor=False) as g:
        g.setCASVolume(cas)
        got = g.forwardProjectCAS(axes)
    assert O.rel_l2(got, ref) < TOL
    assert np.all(got[ref == 0] == 0)


# axes longer than one: some boxes fit and some do not; most windows leave the
# volume; windows far outside it; columns scaled apart
@pytest.mark.parametrize("prec", ["f32", "bf16"])
@pytest.mark.parametrize("N,n,scale", [(50, 30, (1.08, 1.08)), (32, 100, (1.3, 0.9)), (18, 6, (2.5, 2.5)), (16, 4, (40.0, 9.0))])
def test_forward_tiles_long_axes(cuda, N, n, scale, prec):
    import torch

    import multigpugridder_gb300 as gg

    p = O.Params(N)
    cas = np.random.default_rng(6000 + N).standard_normal((p.V,) * 3).astype(np.float32)
    axes = O.quaternion_axes(n, seed=N).astype(np.float32)
    axes = (axes.reshape(n, 3, 3) * np.float32(scale + (1.0,))[None, :, None]).reshape(n, 9)
    stored = cas if prec == "f32" else torch.from_numpy(cas).bfloat16().float().numpy()
    ref = O.fp_ref_f32(stored, axes, p.M, p.mask_radius, p.ker)
    with gg.MultiGPUGridder(N, n, precision=prec, adjustInterpFactor=False) as g:
        g.setCASVolume(cas)
        got = g.forwardProjectCAS(axes)
    assert O.rel_l2(got, ref) < TOL
    assert np.all(got[ref == 0] == 0)


# one handle through every storage type and back (with the 4-tap tiles and with
# five taps), against a handle that has known no other; the volume is replaced on the way
@pytest.mark.parametrize("edge", [0.0, 0.25])
@pytest.mark.parametrize("N", [18, 50])
def test_precision_switches(cuda, N, edge):
    import multigpugridder_gb300 as gg

    p = O.Params(N)
    rng = np.random.default_rng(4000 + N)
    axes = O.quaternion_axes(40, seed=N).astype(np.float32)
    table = p.ker.copy()
    table[0] = edge
    with gg.MultiGPUGridder(N, 40, adjustInterpFactor=False) as g:
        g.setKBTable(table)
        for prec in ("f32", "bf16", "f32", "f16", "bf16", "f16", "f32"):
            cas = rng.standard_normal((p.V,) * 3).astype(np.float32)
            g.set_precision(prec)
            g.setCASVolume(cas)
            got = g.forwardProjectCAS(axes)
            with gg.MultiGPUGridder(N, 40, precision=prec, adjustInterpFactor=False) as f:
                f.setKBTable(table)
                f.setCASVolume(cas)
                assert np.array_equal(got, f.forwardProjectCAS(axes)), prec


# the word that a kernel whose copies did not arrive would set, set from the
# host: the call that finds it reports it, and the next one is as before
def test_copy_fault_is_reported_once(cuda, gglib):
    import multigpugridder_gb300 as gg
    from multigpugridder_gb300._lib import GG_ERR_CUDA

    mark = gglib.gg_mark_copy_fault
    mark.argtypes = [ctypes.c_void_p]
    axes = O.quaternion_axes(5, seed=1).astype(np.float32)
    with gg.MultiGPUGridder(16, 5, adjustInterpFactor=False) as g:
        g.setVolume(O.blob_volume(16, 10, seed=6))
        assert mark(g.handle) != 0  # no projection yet
        good = g.forwardProjectCAS(axes)
        assert mark(g.handle) == 0
        with pytest.raises(gg.GridderError) as e:
            g.forwardProjectCAS(axes)
        assert e.value.code == GG_ERR_CUDA and "did not arrive" in str(e.value)
        assert np.array_equal(g.forwardProjectCAS(axes), good)


# fewer than 32 directions, and each range of the rule's aim, at volumes of few
# bricks; n that the segments do not divide
@pytest.mark.parametrize("N,n", [(64, 9), (16, 33), (18, 101), (32, 210), (16, 600)])
def test_back_projection_segments(cuda, N, n):
    import multigpugridder_gb300 as gg

    p = O.Params(N)
    rng = np.random.default_rng(2000 + n)
    axes = O.quaternion_axes(n, seed=n).astype(np.float32)
    imgs = rng.standard_normal((n, N, N)).astype(np.float32)
    ci = O.cas_imgs_from_imgs(imgs, p.M).astype(np.float32)
    num = O.bp_ref_f32(ci, axes, p.V, p.mask_radius, p.ker)
    den = O.bp_ref_f32(np.ones_like(ci), axes, p.V, p.mask_radius, p.ker)
    with gg.MultiGPUGridder(N, n, adjustInterpFactor=False) as g:
        g.backProjectCAS(ci, axes)
        assert O.rel_l2(g.getCASVolume(), num) < TOL
        g.backProjectCAS(ci, axes, accumulate=True)  # the merge adds to what is there
        assert O.rel_l2(g.getCASVolume(), 2 * num) < TOL
        g.reconstructVol(imgs, axes)
        assert O.rel_l2(g.getCASVolume(), num / (den + np.float32(1e-6))) < TOL


# a small mask in a large volume, where the rule wants the most segments (and
# the 8-deep blocks of M = 512): the scratch holds the mask's box, not the volume
@pytest.mark.parametrize("N,mask,n", [(128, 20, 512), (256, 24, 40), (32, 0, 40), (32, 64, 40)])
def test_back_projection_small_mask(cuda, N, mask, n):
    import torch

    import multigpugridder_gb300 as gg

    p = O.Params(N, mask_radius=mask)
    rng = np.random.default_rng(5000 + N + mask)
    axes = O.quaternion_axes(n, seed=n).astype(np.float32)
    ci = rng.standard_normal((n, p.M, p.M), dtype=np.float32)
    num = O.bp_ref_f32(ci, axes, p.V, mask, p.ker)
    with gg.MultiGPUGridder(N, n, adjustInterpFactor=False) as g:
        g.setMaskRadius(mask)
        g.backProjectCAS(ci[:8], axes[:8])  # the handle's other buffers
        before = torch.cuda.mem_get_info()[0]
        g.backProjectCAS(ci, axes)
        assert before - torch.cuda.mem_get_info()[0] < 140e6
        assert O.rel_l2(g.getCASVolume(), num) < TOL
        imgs = rng.standard_normal((n, N, N), dtype=np.float32)
        g.reconstructVol(imgs, axes)
        got = g.getCASVolume()
    ci = O.cas_imgs_from_imgs(imgs, p.M).astype(np.float32)
    num = O.bp_ref_f32(ci, axes, p.V, mask, p.ker)
    den = O.bp_ref_f32(np.ones_like(ci), axes, p.V, mask, p.ker)
    assert O.rel_l2(got, num / (den + np.float32(1e-6))) < TOL


# under capture the scratch of a split cannot grow: the launch stays unsplit
def test_back_projection_split_under_capture(cuda, gglib):
    import torch

    import multigpugridder_gb300 as gg

    N, n = 32, 300
    p = O.Params(N)
    axes = O.quaternion_axes(n, seed=n).astype(np.float32)
    ci = np.random.default_rng(6).standard_normal((n, p.M, p.M)).astype(np.float32)
    d_axes, d_ci = to_dev(axes, cuda), to_dev(ci, cuda)
    with gg.MultiGPUGridder(N, n, adjustInterpFactor=False) as g:
        g.backProjectCAS(ci[:8], axes[:8])  # the handle's other buffers
        s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            rc = gglib.gg_back_project_dev(g.handle, dptr(d_axes), n, None, dptr(d_ci), 0, ctypes.c_void_p(s.cuda_stream))
        assert rc == 0
        graph.replay()
        torch.cuda.synchronize()
        assert O.rel_l2(g.getCASVolume(), O.bp_ref_f32(ci, axes, p.V, p.mask_radius, p.ker)) < TOL


# the calls that the passes took over run under capture after the calls that
# used to leave their plans and buffers behind: BF16 images after FP32 ones
# (M = 100), setVolume after an adjoint (N = M, where the passes take more room)
@pytest.mark.parametrize("kind", ["bf16_images", "set_volume"])
def test_passes_under_capture(cuda, gglib, kind):
    import torch

    import multigpugridder_gb300 as gg

    N, interp, n = (50, 2.0, 6) if kind == "bf16_images" else (100, 1.0, 2)
    p = O.Params(N, interp)
    rng = np.random.default_rng(7)
    axes = O.quaternion_axes(n, seed=n).astype(np.float32)
    imgs = rng.standard_normal((n, N, N)).astype(np.float32)
    vol = rng.standard_normal((N,) * 3).astype(np.float32)
    d_axes, d_imgs, d_vol = to_dev(axes, cuda), to_dev(imgs, cuda), to_dev(vol, cuda)
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    sp = ctypes.c_void_p(s.cuda_stream)
    with gg.MultiGPUGridder(N, n, interpFactor=interp, adjustInterpFactor=False) as g:
        if kind == "bf16_images":
            g.backProject(imgs, axes)
            g.set_image_precision("bf16")
        else:
            g.resetVolume()
            grad = np.empty((N,) * 3, dtype=np.float32)
            g._call("gg_forward_project_adjoint", axes.ctypes.data, n, imgs.ctypes.data, grad.ctypes.data)
        with torch.cuda.graph(graph, stream=s):
            if kind == "bf16_images":
                rc = gglib.gg_back_project_dev(g.handle, dptr(d_axes), n, dptr(d_imgs), None, 0, sp)
            else:
                rc = gglib.gg_set_volume_dev(g.handle, dptr(d_vol), sp)
        assert rc == 0
        graph.replay()
        torch.cuda.synchronize()
        got = g.getCASVolume()
    if kind == "bf16_images":
        stored = torch.from_numpy(O.cas_imgs_from_imgs(imgs, p.M).astype(np.float32)).bfloat16().float().numpy()
        assert O.rel_l2(got, O.bp_ref_f32(stored, axes, p.V, p.mask_radius, p.ker)) < 1e-3  # values on a rounding edge
    else:
        assert O.rel_l2(got, O.cas_from_vol(vol.astype(np.float64), p.hw, p.interp, p.pad)) < TOL


# CAS images rounded to 2 bytes and read as FP32: M a multiple of 4 and not
@pytest.mark.parametrize("prec", ["bf16", "f16"])
@pytest.mark.parametrize("N,interp", [(32, 2.0), (44, 1.5)])
def test_reduced_cas_images(cuda, N, interp, prec):
    import torch

    import multigpugridder_gb300 as gg

    p = O.Params(N, interp)
    axes = O.quaternion_axes(7, seed=N).astype(np.float32)
    ci = np.random.default_rng(N).standard_normal((7, p.M, p.M)).astype(np.float32)
    # largest value about 5: FP16 is stored at scale 1
    stored = torch.from_numpy(ci).to(torch.bfloat16 if prec == "bf16" else torch.float16).float().numpy()
    ref = O.bp_ref_f32(stored, axes, p.V, p.mask_radius, p.ker)
    with gg.MultiGPUGridder(N, 7, interpFactor=interp, precision=prec, adjustInterpFactor=False) as g:
        g.backProjectCAS(ci, axes)
        assert O.rel_l2(g.getCASVolume(), ref) < TOL


# V = 10, 38, 106 (rows of 2 and of 4 floats), 41 (odd rows); a table too long
# to be kept four times; boxes that do not fit and boxes of few voxels
@pytest.mark.parametrize("N,interp,size,mask,scale",
                         [(2, 2.0, 501, 1, 1.0), (16, 2.0, 1000, 15, 1.0), (50, 2.0, 501, 49, 1.0), (14, 2.5, 501, 16, 1.0),
                          (16, 2.0, 501, 8, 1.7), (16, 2.0, 501, 15, 0.3)])
def test_adjoint_boxes(cuda, gglib, N, interp, size, mask, scale):
    import torch

    p = O.Params(N, interp, table_size=size, mask_radius=mask)
    n = 9
    rng = np.random.default_rng(3000 + N)
    axes = (scale * O.quaternion_axes(n, seed=N)).astype(np.float32)
    y = rng.standard_normal((n, p.M, p.M)).astype(np.float32)
    vol = torch.zeros((p.V,) * 3, device=cuda)
    d_ker, d_axes, d_y = to_dev(p.ker, cuda), to_dev(axes, cuda), to_dev(y, cuda)
    assert gglib.gg_back_project_adjoint_kernel(dptr(vol), dptr(d_y), dptr(d_ker), dptr(d_axes), 2.0, n, p.V, p.M, mask,
                                                size, None) == 0
    torch.cuda.synchronize()
    ref = O.bp_adjoint_f64(y.astype(np.float64), axes, p.V, mask, p.ker)
    assert O.rel_l2(vol.cpu().numpy(), ref) < 1e-3


# radii meant as "no mask": the square fits 31 bits for 46340 and not for the
# others (65536 squared is 0 in 32 bits, 2^31 - 1 squared 1)
@pytest.mark.parametrize("radius", [32, 46340, 46341, 60000, 65536, 2**31 - 1])
def test_adjoint_large_radius(cuda, gglib, radius):
    import torch

    p = O.Params(16)
    n = 5
    axes = O.quaternion_axes(n, seed=7).astype(np.float32)
    y = np.random.default_rng(8).standard_normal((n, p.M, p.M)).astype(np.float32)
    d = np.arange(p.M) - p.M // 2
    y[:, d[:, None]**2 + d**2 > p.mask_radius**2] = 0  # windows that stay in the volume
    vol = torch.zeros((p.V,) * 3, device=cuda)
    d_ker, d_axes, d_y = to_dev(p.ker, cuda), to_dev(axes, cuda), to_dev(y, cuda)
    assert gglib.gg_back_project_adjoint_kernel(dptr(vol), dptr(d_y), dptr(d_ker), dptr(d_axes), 2.0, n, p.V, p.M, radius,
                                                len(p.ker), None) == 0
    torch.cuda.synchronize()
    ref = O.bp_adjoint_f64(y.astype(np.float64), axes, p.V, p.mask_radius, p.ker)
    assert O.rel_l2(vol.cpu().numpy(), ref) < 1e-3


# Repeated calls.  The reference rule: the same bits, split (n = 300) and not.  The
# adjoint adds in any order: a voxel's few hundred terms of either sign, each order
# rounding by 6e-8 a step, spread by some 1e-7 of the sum; 1e-6 bounds it.
def test_repeated_calls(cuda):
    import torch

    import multigpugridder_gb300 as gg
    from multigpugridder_gb300.autograd import ForwardProjector

    N, n = 32, 300
    axes = O.quaternion_axes(n, seed=9).astype(np.float32)
    imgs = np.random.default_rng(9).standard_normal((n, N, N)).astype(np.float32)
    runs = {}
    for mode in ("ref", "adjoint"):
        with gg.MultiGPUGridder(N, n, bp_mode=mode, adjustInterpFactor=False) as g:
            for k in range(4):
                g.backProject(imgs, axes)
                runs[mode, k] = g.getCASVolume()
                g.backProject(imgs[:20], axes[:20])
                runs[mode, k, 20] = g.getCASVolume()
    proj = ForwardProjector(N)
    for k in range(4):
        runs["grad", k] = proj.adjoint(to_dev(imgs, cuda), to_dev(axes, cuda)).cpu().numpy()
    for k in range(1, 4):
        assert np.array_equal(runs["ref", 0], runs["ref", k])
        assert np.array_equal(runs["ref", 0, 20], runs["ref", k, 20])
        for key in (("adjoint",), ("grad",)):
            assert O.rel_l2(runs[key + (k,)], runs[key + (0,)]) < 1e-6
        assert O.rel_l2(runs["adjoint", k, 20], runs["adjoint", 0, 20]) < 1e-6


# a CTF of -1 everywhere gives minus the plain reconstruction, bit for bit: the
# images take the same transform in both, also where they are rounded (M = 100
# through the passes or the library, M = 64 in one kernel)
@pytest.mark.parametrize("prec", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("N", [32, 50])
def test_ctf_of_minus_one(cuda, N, prec):
    import multigpugridder_gb300 as gg

    n = 20
    axes = O.quaternion_axes(n, seed=N).astype(np.float32)
    imgs = np.random.default_rng(N).standard_normal((n, N, N)).astype(np.float32)
    with gg.MultiGPUGridder(N, n, precision=prec, adjustInterpFactor=False) as g:
        plain = g.reconstructVol(imgs, axes).copy()
        ctf = g.reconstructVolCTF(imgs, axes, np.zeros(n, dtype=np.float32), cs_mm=0.0, amp_contrast=1.0)
    assert np.array_equal(ctf, -plain)


# enough images for blocks of 64 rows (1024 of them), also with a remainder, and one too few
@pytest.mark.parametrize("M,n", [(64, 1100), (100, 520), (64, 1000)])
def test_ctf_row_blocks(cuda, gglib, M, n):
    import torch

    kv, cs, amp = (float(np.float32(v)) for v in (300.0, 2.7, 0.1))
    rng = np.random.default_rng(M + n)
    du = rng.uniform(5000.0, 40000.0, n).astype(np.float32)
    dv = (du - rng.uniform(-3000.0, 3000.0, n)).astype(np.float32)
    ang = rng.uniform(-np.pi, np.pi, n).astype(np.float32)
    out = torch.full((n, M, M), float("nan"), device=cuda)
    d_u, d_v, d_a = to_dev(du, cuda), to_dev(dv, cuda), to_dev(ang, cuda)
    for v, a, ref in ((None, None, O.ctf_cas(M, du, kv, cs, amp, 1.5)),
                      (d_v, d_a, O.ctf_cas(M, du, kv, cs, amp, 1.5, dv, ang))):
        assert gglib.gg_filter_apply_ctf(dptr(out), M, n, dptr(d_u), None if v is None else dptr(v),
                                         None if a is None else dptr(a), kv, cs, amp, 1.5, 1, 1, None) == 0
        torch.cuda.synchronize()
        assert np.max(np.abs(out.cpu().numpy() - ref)) < 1e-6
