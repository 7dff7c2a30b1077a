"""The work a user has this library do, as cases whose time can be measured.

A case is one pass of one of eight uses, over the sizes the library is used at
(volume edges 32 to 256, interpFactor 2, 16 to 10,000 directions):

  forward  images of a resident volume (gg_forward_project_dev)
  project  a new volume, then its images (gg_set_volume_dev + gg_forward_project_dev):
           one expectation step of a refinement
  back     images into a zeroed CAS volume, then the volume (gg_back_project_dev + gg_get_volume_dev)
  recon    reconstructVol of images (gg_reconstruct_volume_dev)
  ctf      the same with each image's CTF (gg_reconstruct_volume_ctf_dev)
  train    loss and gradient of a volume against images (ForwardProjector, autograd)
  host     the numpy class: setVolume, forwardProject and reconstructVol on host arrays
  serve    a burst of mixed requests to the serving loop, on two resident volumes

Inputs come from the seed alone: sums of Gaussian blobs (whose projections are
sums of 2-D Gaussians), random or gridded directions, Gaussian noise.
"""
import ctypes
import math

import numpy as np
import torch

import multigpugridder_gb300 as gg
from multigpugridder_gb300 import _lib
from multigpugridder_gb300._lib import check
from multigpugridder_gb300.autograd import ForwardProjector
from multigpugridder_gb300.serve import Server, pinned_empty

PAD = 3          # extraPadding: V = M + 2 * PAD
KV, CS, AMP, PX = 300.0, 2.7, 0.1, 1.1  # microscope of the CTF cases
HEADLINE = 10000 * 256 * 256  # directions x CAS-image pixels of the largest case
SERVE_NS = (64, 128)


def listed():
    return [
        # the smallest request of the serving mix: a few views of a small volume
        {"name": "forward_64_16", "kind": "forward", "N": 64, "n": 16, "precision": "f32"},
        # one default batch (MaxAxesToAllocate = 1000) at the benchmark's size
        {"name": "forward_128_1000", "kind": "forward", "N": 128, "n": 1000, "precision": "f32"},
        # a refinement step on a box that is no power of two (M = 200)
        {"name": "project_100_300", "kind": "project", "N": 100, "n": 300, "precision": "f32"},
        # a large box in BF16 storage, new volume each time
        {"name": "project_256_512_bf16", "kind": "project", "N": 256, "n": 512, "precision": "bf16"},
        # a few images back into a small volume
        {"name": "back_64_16", "kind": "back", "N": 64, "n": 16, "precision": "f32"},
        # the CPU-size workload: 64^3, 1,000 random directions
        {"name": "recon_64_1000", "kind": "recon", "N": 64, "n": 1000, "precision": "f32"},
        # the benchmark's reconstruction: 128^3, the 100 x 100 grid of directions
        {"name": "recon_128_10000", "kind": "recon", "N": 128, "n": 10000, "precision": "f32"},
        # a 192^3 reconstruction (M = 384) in FP16 storage
        {"name": "recon_192_700_f16", "kind": "recon", "N": 192, "n": 700, "precision": "f16"},
        # a CTF-corrected reconstruction
        {"name": "ctf_128_1000", "kind": "ctf", "N": 128, "n": 1000, "precision": "f32"},
        # one gradient step of a mini-batch
        {"name": "train_128_512", "kind": "train", "N": 128, "n": 512, "precision": "f32"},
        # the class as the MATLAB user calls it, host arrays in and out (96 -> M = 256)
        {"name": "host_96_250", "kind": "host", "N": 96, "n": 250, "precision": "f32"},
        # 24 requests at once, 16 to 512 directions each, half of them back projections
        {"name": "serve_24", "kind": "serve", "requests": 24, "most": 512},
    ]


def draw(rng):
    kind = rng.choice(["forward", "forward", "project", "back", "recon", "recon", "ctf", "train", "host", "serve"])
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(4, 32), "most": int(round(math.exp(rng.uniform(math.log(32), math.log(1024)))))}
    if rng.random() < 0.5:
        N = rng.choice([48, 64, 96, 128, 160, 192, 256])
    else:
        N = 2 * int(round(math.exp(rng.uniform(math.log(32), math.log(256))) / 2))
    M = gridder_size(kind, N)
    most = min(4096, int(HEADLINE / (3 * M * M)))
    if kind == "host":
        most = min(most, 1000)
    n = int(round(math.exp(rng.uniform(math.log(16), math.log(most)))))
    precision = "f32" if kind in ("ctf", "train", "host") else rng.choice(["f32", "f32", "bf16", "f16"])
    return {"kind": kind, "N": N, "n": n, "precision": precision}


def interp_of(kind, N):
    # the class rounds interpFactor up so that M is a power of two; the other uses keep 2
    if kind != "host":
        return 2.0
    if N < 64:
        return float(np.float32(128) / np.float32(N))
    return float(np.float32((128 if N <= 64 else 256 if N <= 128 else 512)) / np.float32(N))


def gridder_size(kind, N):
    return int(round(N * interp_of(kind, N)))


# ---- inputs ------------------------------------------------------------------


def make_blobs(N, seed, count=60):
    g = torch.Generator().manual_seed(seed)
    u = torch.rand((count, 5), generator=g, dtype=torch.float64)
    c = N * (0.2 + 0.6 * u[:, :3])              # centres, inner 60% of the box
    s = (2.0 + 4.0 * u[:, 3]) * min(1.0, N / 64)  # widths in voxels
    a = 0.5 + u[:, 4]
    return c.cuda(), s.cuda(), a.cuda()


def make_volume(N, blobs):
    c, s, a = blobs
    x = torch.arange(N, dtype=torch.float64, device="cuda")
    e = [torch.exp(-((x[None] - c[:, d:d + 1]) ** 2) / (2 * s[:, None] ** 2)) for d in range(3)]
    kj = ((a[:, None] * e[2])[:, :, None] * e[1][:, None, :]).reshape(len(a), N * N)
    return (kj.T @ e[0]).reshape(N, N, N).float().contiguous()  # [z, y, x]


def make_axes(n, seed):
    """n directions (n, 9): the x, y, z columns of rotations; a uniform grid for
    square numbers of at least 10,000, random rotations otherwise."""
    side = math.isqrt(n)
    if n >= 10000 and side * side == n:
        az = torch.arange(side, dtype=torch.float64) * (2 * math.pi / side)
        ct = -1.0 + (2 * torch.arange(side, dtype=torch.float64) + 1) / side
        ph, ct = az.repeat(side), ct.repeat_interleave(side)
        st, psi = torch.sqrt(1 - ct * ct), math.radians(30.0 + seed % 30)
        cp, sp, cs, sn = torch.cos(ph), torch.sin(ph), math.cos(psi), math.sin(psi)
        X = torch.stack([cp * ct * cs - sp * sn, sp * ct * cs + cp * sn, -st * cs], 1)
        Y = torch.stack([-cp * ct * sn - sp * cs, -sp * ct * sn + cp * cs, st * sn], 1)
        Z = torch.stack([cp * st, sp * st, ct], 1)
        return torch.cat([X, Y, Z], 1).float().cuda().contiguous()
    q = torch.randn((n, 4), generator=torch.Generator().manual_seed(seed + 7), dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    X = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w)], 1)
    Y = torch.stack([2 * (x * y - z * w), 1 - 2 * (x * x + z * z), 2 * (y * z + x * w)], 1)
    Z = torch.stack([2 * (x * z + y * w), 2 * (y * z - x * w), 1 - 2 * (x * x + y * y)], 1)
    return torch.cat([X, Y, Z], 1).float().cuda().contiguous()


def make_images(N, axes, blobs, seed, noise=0.5):
    """The blobs' projections along axes, plus noise."""
    c, s, a = (t.float() for t in blobs)
    n = axes.shape[0]
    g = torch.Generator(device="cuda").manual_seed(seed + 13)
    x = torch.arange(N, dtype=torch.float32, device="cuda")
    px = axes[:, 0:3] @ (c - N / 2).T + N / 2
    py = axes[:, 3:6] @ (c - N / 2).T + N / 2
    out = torch.empty((n, N, N), dtype=torch.float32, device="cuda")
    for i in range(0, n, 500):
        ex = torch.exp(-((x[None, None] - px[i:i + 500, :, None]) ** 2) / (2 * s[:, None] ** 2))
        ey = torch.exp(-((x[None, None] - py[i:i + 500, :, None]) ** 2) / (2 * s[:, None] ** 2))
        ey *= (a * s * math.sqrt(2 * math.pi))[:, None]
        out[i:i + 500] = ey.transpose(1, 2) @ ex
    level = noise * float(out[: min(n, 64)].std())
    for i in range(0, n, 500):
        out[i:i + 500] += level * torch.randn(out[i:i + 500].shape, generator=g, device="cuda")
    return out


def make_defocus(n, seed):
    u = torch.rand((3, n), generator=torch.Generator().manual_seed(seed + 29))
    du = 10000.0 + 15000.0 * u[0]
    return du.cuda(), (du - 600.0 * u[1]).cuda(), (math.pi * u[2]).cuda()


def make_requests(case):
    """(volume index, operation, directions) of each request of a burst: sizes
    64^3 twice as often as 128^3, directions log-uniform from 16.  The case
    fixes the mix, so that bursts of several seeds are the same work."""
    r = np.random.default_rng(1000 * case["most"] + case["requests"])
    got = []
    for k in range(case["requests"]):
        v = int(r.random() < 1 / 3)
        n = int(round(math.exp(r.uniform(math.log(16), math.log(case["most"])))))
        got.append((v, "back" if k % 2 else "forward", n))
    return got


# ---- the cases ----------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        srv = Server()
        vids, all_blobs = [], []
        for k, N in enumerate(SERVE_NS):
            all_blobs.append(make_blobs(N, seed + k))
            vids.append(srv.add_volume(make_volume(N, all_blobs[k])))
        reqs = []
        for k, (v, op, n) in enumerate(make_requests(case)):
            N = SERVE_NS[v]
            ax = make_axes(n, seed + 100 + k)
            a_h = pinned_empty((n, 9))
            a_h[...] = ax.cpu().numpy()
            im = None
            if op == "back":
                im = pinned_empty((n, N, N))
                im[...] = make_images(N, ax, all_blobs[v], seed + k).cpu().numpy()
            out = pinned_empty((n, N, N) if op == "forward" else (2 * N + 2 * PAD,) * 3)
            reqs.append((vids[v], op, a_h, im, out))
        return {"case": case, "server": srv, "requests": reqs}

    N, n = case["N"], case["n"]
    blobs = make_blobs(N, seed)
    axes = make_axes(n, seed)
    st = {"case": case, "axes": axes, "n": n}
    if kind == "train":
        st["proj"] = ForwardProjector(N)
        st["vol"] = make_volume(N, make_blobs(N, seed + 1)).requires_grad_(True)
        st["target"] = make_images(N, axes, blobs, seed)
        return st
    if kind == "host":
        interp = interp_of(kind, N)
        st["g"] = gg.MultiGPUGridder(N, n, interp)
        st["vol"] = make_volume(N, blobs).cpu().numpy()
        st["axes"] = axes.cpu().numpy()
        return st
    g = gg.MultiGPUGridder(N, n, 2.0, precision=case["precision"], adjustInterpFactor=False)
    st["g"] = g
    if kind in ("forward", "project"):
        st["vol"] = make_volume(N, blobs)
        st["out"] = torch.empty((n, N, N), dtype=torch.float32, device="cuda")
        if kind == "forward":
            check(_lib.lib().gg_set_volume_dev(g.handle, vp(st["vol"]), stream()), g.handle)
    else:
        st["images"] = make_images(N, axes, blobs, seed)
        st["out"] = torch.empty((N, N, N), dtype=torch.float32, device="cuda")
        if kind == "ctf":
            st["defocus"] = make_defocus(n, seed)
    return st


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


def stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def run(st):
    kind = st["case"]["kind"]
    if kind == "serve":
        srv = st["server"]
        sent = [srv.submit(vid, op, ax, im, out=out) for vid, op, ax, im, out in st["requests"]]
        return [srv.wait(r)[0] for r in sent]
    if kind == "train":
        vol = st["vol"]
        vol.grad = None
        images = st["proj"].project(vol, st["axes"])
        loss = 0.5 * (images - st["target"]).square().sum()
        loss.backward()
        return {"images": images.detach(), "grad": vol.grad}
    if kind == "host":
        g = st["g"]
        g.setVolume(st["vol"])
        images = g.forwardProject(st["axes"])
        return {"images": images, "volume": g.reconstructVol(images, st["axes"])}
    L, h, s, n = _lib.lib(), st["g"].handle, stream(), st["n"]
    if kind in ("forward", "project"):
        if kind == "project":
            check(L.gg_set_volume_dev(h, vp(st["vol"]), s), h)
        check(L.gg_forward_project_dev(h, vp(st["axes"]), n, vp(st["out"]), None, s), h)
    elif kind == "back":
        check(L.gg_back_project_dev(h, vp(st["axes"]), n, vp(st["images"]), None, 0, s), h)
        check(L.gg_get_volume_dev(h, vp(st["out"]), s), h)
    elif kind == "recon":
        check(L.gg_reconstruct_volume_dev(h, vp(st["axes"]), n, vp(st["images"]), vp(st["out"]), s), h)
    else:
        du, dv, an = st["defocus"]
        check(L.gg_reconstruct_volume_ctf_dev(h, vp(st["axes"]), n, vp(st["images"]), vp(du), vp(dv), vp(an), KV, CS,
                                              AMP, PX, vp(st["out"]), s), h)
    return st["out"]


def work(case):
    """Bytes: each input read once, each output written once.  Operations: the
    64 taps of each in-mask pixel (forward, adjoint) or the 25 pixels of each
    slab voxel (back), and the FFTs' 2.5 n log2 n of real data."""
    kind = case["kind"]
    if kind == "serve":
        total = {"bytes": 0.0, "flops": 0.0}
        for v, op, n in make_requests(case):
            w = work({"kind": op, "N": SERVE_NS[v], "n": n, "precision": "f32", "resident": True})
            total = {k: total[k] + w[k] for k in total}
        return total
    N, n = case["N"], case["n"]
    M = gridder_size(kind, N)
    R = M / 2 - 1
    disc, vol, imgs = math.pi * R * R * n, 4.0 * N ** 3, 4.0 * n * N * N
    fft2 = n * 2.5 * M * M * math.log2(M * M)
    fft3 = 2.5 * M ** 3 * math.log2(M ** 3)
    fp = 64 * 2 * disc + fft2
    # per pixel of a slab voxel's window: three weights multiplied and one multiply-add
    bp = 25 * 4 * (4.0 * disc) + fft2
    size = 4 if case["precision"] == "f32" else 2
    cas = float((M + 2 * PAD) ** 3)
    if kind == "forward":
        return {"bytes": size * cas + imgs + 36.0 * n, "flops": fp}
    if kind == "project":
        return {"bytes": vol + imgs + 36.0 * n, "flops": fp + fft3}
    if kind == "back":
        return {"bytes": imgs + (4 * cas if case.get("resident") else vol) + 36.0 * n,
                "flops": bp + (0 if case.get("resident") else fft3)}
    if kind == "recon":
        return {"bytes": imgs + vol + 36.0 * n, "flops": bp + 25 * 4.0 * disc + fft3}
    if kind == "ctf":
        return {"bytes": imgs + vol + 48.0 * n, "flops": bp + 25 * 2 * 4.0 * disc + fft3}
    if kind == "train":
        return {"bytes": 2 * vol + 2 * imgs + 36.0 * n, "flops": 2 * fp + 2 * fft3}
    return {"bytes": 2 * vol + 2 * imgs + 36.0 * n, "flops": fp + bp + 25 * 4.0 * disc + 2 * fft3}


# ---- the same in 64 bits --------------------------------------------------------


def window():
    """The Kaiser-Bessel table: 501 entries on [-2, 2], alpha 10, edge value
    subtracted, normalised over the 5^3 integer taps."""
    x = np.linspace(-2.0, 2.0, 501)
    w = np.i0(10.0 * np.sqrt(np.maximum(0.0, 1.0 - (x / 2) ** 2))) / np.i0(10.0)
    w = w / (w.sum() * 4 / 500)
    w = w - w[0]
    w[-1] = 0.0
    return torch.from_numpy(w / w[[0, 125, 250, 375, 500]].sum()).cuda()


def deapodization(M):
    x = np.linspace(-2.0, 2.0, 17)
    w = np.i0(10.0 * np.sqrt(np.maximum(0.0, 1.0 - (x / 2) ** 2)))
    w = w - w[0]
    w[-1] = 0.0
    m = np.arange(M) - M // 2
    pc = (w[None] * np.cos(2 * np.pi * m[:, None] * (np.arange(17) - 8)[None] / (4 * M))).sum(1)
    return torch.from_numpy(w.sum() / pc).cuda()


def inner(N, M):
    return slice(M // 2 - N // 2, M // 2 - N // 2 + N)


def cas_of_volume(vol, M):
    N, p, s = vol.shape[0], deapodization(M), inner(vol.shape[0], M)
    x = torch.zeros((M,) * 3, dtype=torch.float64, device="cuda")
    x[s, s, s] = vol.double() * p[s][:, None, None] * p[s][None, :, None] * p[s]
    F = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(x)))
    out = torch.zeros((M + 2 * PAD,) * 3, dtype=torch.float64, device="cuda")
    out[PAD:-PAD, PAD:-PAD, PAD:-PAD] = F.real + F.imag
    return out


def hermitian(r, dims):
    """The spectrum whose Re + Im is r, its first plane along each of dims zero."""
    f = torch.roll(torch.flip(r, dims), [1] * len(dims), dims)
    c = torch.complex(0.5 * (r + f), 0.5 * (r - f))
    for d in dims:
        c.select(d, 0).zero_()
    return c


def volume_of_cas(cas, N):
    M = cas.shape[0] - 2 * PAD
    c = hermitian(cas[PAD:-PAD, PAD:-PAD, PAD:-PAD], [0, 1, 2])
    y = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(c))).real
    s, p = inner(N, M), deapodization(M)
    return y[s, s, s] * p[s][:, None, None] * p[s][None, :, None] * p[s]


def images_of_cas(ci, N):
    c = hermitian(ci, [1, 2])
    y = torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(c, (1, 2))), (1, 2)).real
    s = inner(N, ci.shape[1])
    return y[:, s, s]


def cas_of_images(img, M):
    s = inner(img.shape[1], M)
    x = torch.zeros((img.shape[0], M, M), dtype=torch.float64, device="cuda")
    x[:, s, s] = img.double()
    F = torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(x, (1, 2))), (1, 2))
    return F.real + F.imag


def taps(axes, M):
    """Of some directions: flat CAS-volume indices and weights of the 4^3 taps
    of each in-mask pixel, and the pixels' flat image indices."""
    V, w = M + 2 * PAD, window()
    d = torch.arange(M, device="cuda") - M // 2
    jj, ii = torch.meshgrid(d, d, indexing="ij")
    keep = ii * ii + jj * jj <= (M // 2 - 1) ** 2
    pix = keep.reshape(-1).nonzero()[:, 0]
    a = axes.double()
    f = a[:, None, 0:3] * ii[keep][None, :, None] + a[:, None, 3:6] * jj[keep][None, :, None] + V // 2
    b = torch.floor(f) - 1
    o = torch.arange(4, device="cuda")
    r = b[..., None] + o - f[..., None]                      # (n, P, 3, 4)
    k = w[torch.floor(r.clamp(-2, 2) * 125 + 250.5).long()]
    b = b.long()[..., None] + o
    lin = (b[:, :, 2, :, None, None] * V + b[:, :, 1, None, :, None]) * V + b[:, :, 0, None, None, :]
    wt = k[:, :, 2, :, None, None] * k[:, :, 1, None, :, None] * k[:, :, 0, None, None, :]
    return lin.reshape(lin.shape[0], -1, 64), wt.reshape(lin.shape[0], -1, 64), pix


def step_of(M):
    return max(1, int(4e7 / (M * M * 50)))


def forward_64(cas, axes, M):
    out = torch.zeros((axes.shape[0], M * M), dtype=torch.float64, device="cuda")
    flat, c = cas.reshape(-1), step_of(M)
    for i in range(0, axes.shape[0], c):
        lin, wt, pix = taps(axes[i:i + c], M)
        out[i:i + c, pix] = (flat[lin] * wt).sum(-1)
    return out.reshape(-1, M, M)


def adjoint_64(ci, axes, M):
    V, c = M + 2 * PAD, step_of(M)
    out = torch.zeros(V ** 3, dtype=torch.float64, device="cuda")
    for i in range(0, axes.shape[0], c):
        lin, wt, pix = taps(axes[i:i + c], M)
        y = ci[i:i + c].reshape(lin.shape[0], -1)[:, pix]
        out.index_add_(0, lin.reshape(-1), (wt * y[..., None]).reshape(-1))
    return out.reshape(V, V, V)


def back_64(stacks, axes, M):
    """The reference's back projection of each stack: every voxel of the mask
    sphere within 2 of a direction's plane sums the 5 x 5 pixels around its
    projection."""
    V, w, n = M + 2 * PAD, window(), axes.shape[0]
    c, R = V // 2, M // 2 - 1
    outs = [torch.zeros(V ** 3, dtype=torch.float64, device="cuda") for _ in stacks]
    flat = [s.reshape(n, -1) for s in stacks]
    g = torch.arange(-R, R + 1, dtype=torch.float64, device="cuda")
    p, q = (t.reshape(-1) for t in torch.meshgrid(g, g, indexing="ij"))
    u = torch.arange(-4, 5, dtype=torch.float64, device="cuda")
    o = torch.arange(-2, 3, dtype=torch.float64, device="cuda")
    oj, oi = (t.reshape(-1) for t in torch.meshgrid(o, o, indexing="ij"))
    lead = axes[:, 6:9].abs().argmax(1).tolist()  # the axis along which a column meets the slab shortest
    for a in range(n):
        X, Y, Z = axes[a].double().reshape(3, 3).unbind(0)
        m = lead[a]
        l0, l1 = [d for d in range(3) if d != m]
        mid = torch.round(-(p * Z[l0] + q * Z[l1]) / Z[m])
        v = [None] * 3
        v[m] = mid[:, None] + u
        v[l0], v[l1] = p[:, None].expand_as(v[m]), q[:, None].expand_as(v[m])
        fk = v[0] * Z[0] + v[1] * Z[1] + v[2] * Z[2]
        at = ((fk.abs() <= 2) & (v[0] ** 2 + v[1] ** 2 + v[2] ** 2 <= R * R)).reshape(-1).nonzero()[:, 0]
        v = [t.reshape(-1)[at] for t in v]
        half = lambda t: torch.sign(t) * torch.floor(t.abs() + 0.5)  # noqa: E731
        pi = half(v[0] * X[0] + v[1] * X[1] + v[2] * X[2] + M // 2) - M // 2 + oi[:, None]
        pj = half(v[0] * Y[0] + v[1] * Y[1] + v[2] * Y[2] + M // 2) - M // 2 + oj[:, None]
        wt = None
        for d in range(3):
            r = (pi * X[d] + pj * Y[d] - v[d]).clamp(-2, 2)
            t = w[torch.floor(r * 125 + 250.5).long()]
            wt = t if wt is None else wt * t
        lin = ((pj + M // 2) * M + pi + M // 2).long()
        wt = torch.where((lin >= 0) & (lin < M * M), wt, 0.0)
        lin = lin.clamp(0, M * M - 1)
        to = (((v[2] + c) * V + v[1] + c) * V + v[0] + c).long()
        for out, s in zip(outs, flat):
            out[to] += (s[a][lin] * wt).sum(0)  # each voxel once per direction
    return [t.reshape(V, V, V) for t in outs]


def ctf_64(n, M, defocus):
    du, dv, an = (t.double()[:, None, None] for t in defocus)
    f32 = lambda x: float(np.float32(x))  # noqa: E731  the parameters as the call receives them
    volts = f32(KV) * 1e3
    lam = 12.2643247 / math.sqrt(volts * (1 + 0.978466e-6 * volts))
    f = (torch.arange(M, dtype=torch.float64, device="cuda") - M // 2) / (M * f32(PX))
    fx, fy = f[None, None, :], f[None, :, None]
    s2 = fx ** 2 + fy ** 2
    df = 0.5 * (du + dv) + 0.5 * (du - dv) * torch.cos(2 * (torch.atan2(fy.expand_as(s2), fx.expand_as(s2)) - an))
    chi = math.pi * lam * df * s2 - 0.5 * math.pi * f32(CS) * 1e7 * lam ** 3 * s2 ** 2
    return -(math.sqrt(1 - f32(AMP) ** 2) * torch.sin(chi) + f32(AMP) * torch.cos(chi))


def recon_64(images, axes, N, M, defocus=None):
    ci = cas_of_images(images, M)
    den = torch.ones_like(ci)
    if defocus is not None:
        k = ctf_64(images.shape[0], M, defocus)
        ci, den = ci * k, k * k
    a, b = back_64([ci, den], axes, M)
    return volume_of_cas(a / (b + 1e-6), N)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        if case["requests"] * case["most"] > 24 * 512:
            return None
        outs = []
        blobs = [make_blobs(N, seed + k) for k, N in enumerate(SERVE_NS)]
        cas = [cas_of_volume(make_volume(N, b), 2 * N) for N, b in zip(SERVE_NS, blobs)]
        for k, (v, op, n) in enumerate(make_requests(case)):
            N = SERVE_NS[v]
            ax = make_axes(n, seed + 100 + k)
            if op == "forward":
                outs.append(images_of_cas(forward_64(cas[v], ax, 2 * N), N))
            else:
                outs.append(back_64([cas_of_images(make_images(N, ax, blobs[v], seed + k), 2 * N)], ax, 2 * N)[0])
        return outs
    N, n = case["N"], case["n"]
    M = gridder_size(kind, N)
    if n * M * M > 1.5e8:
        return None  # over about 20 seconds
    blobs, axes = make_blobs(N, seed), make_axes(n, seed)
    if kind == "train":
        cas = cas_of_volume(make_volume(N, make_blobs(N, seed + 1)), M)
        images = images_of_cas(forward_64(cas, axes, M), N)
        ci = cas_of_images(images - make_images(N, axes, blobs, seed).double(), M) / (M * M)
        ci[:, 0, :] = 0
        ci[:, :, 0] = 0
        g = adjoint_64(ci, axes, M)[PAD:-PAD, PAD:-PAD, PAD:-PAD]
        F = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(g)))
        s, p = inner(N, M), deapodization(M)
        grad = (F.real + F.imag)[s, s, s] * p[s][:, None, None] * p[s][None, :, None] * p[s]
        return {"images": images, "grad": grad}
    if kind in ("forward", "project", "host"):
        images = images_of_cas(forward_64(cas_of_volume(make_volume(N, blobs), M), axes, M), N)
        if kind != "host":
            return images
        return {"images": images, "volume": recon_64(images, axes, N, M)}
    images = make_images(N, axes, blobs, seed)
    if kind == "back":
        return volume_of_cas(back_64([cas_of_images(images, M)], axes, M)[0], N)
    return recon_64(images, axes, N, M, make_defocus(n, seed) if kind == "ctf" else None)
