"""What is timed when a change to the kernels is judged: the calls that users make of this package.

``listed`` names a dozen of them, ``draw`` gives more of the same ranges, ``prepare`` makes a call's inputs
on the GPU, ``run`` makes the call, ``work`` says what it cannot do without and ``exact`` computes it in
64 bits with plain torch.  Ranges: volumes of 48 to 256 voxels per axis and slices of 256 to 768 pixels,
1-4 channels (1-8 in 2-D), orders 1-3, every bound of the sampling functions, float32 and bfloat16 images,
smooth deformations (a few voxels, smoothed over 2-6 voxels) and affine ones.
"""
import math

import torch

import nitorch_b200 as nb
from nitorch_b200 import solve, svf
from nitorch_b200.batch import PullPushBatch

F64 = torch.float64
DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}
# penalties of a displacement grid, nitorch's defaults for registration
PENALTIES = {"absolute": 1e-4, "membrane": 1e-3, "bending": 0.2, "lame": (0.05, 0.2)}


# ------------------------------------------------------------------------------------------------------ #
# the cases                                                                                              #
# ------------------------------------------------------------------------------------------------------ #

def _case(name, op, shape, n=1, c=1, order=1, bound="dct2", dtype="float32", sigma=4.0, std=2.0, **more):
    d = {"name": name, "op": op, "n": n, "c": c, "order": order, "bound": bound, "dtype": dtype,
         "sigma": sigma, "std": std}
    d.update({"s%d" % i: s for i, s in enumerate(shape)})
    d.update(more)
    return {k: v for k, v in d.items() if k != "name" or v}


def listed():
    return [
        # the smallest: a small volume warped and splatted back, linear (interactive use, coarse pyramid level)
        _case("pull_push_64", "pull_push", (64, 64, 64)),
        # one training step of a spatial transformer on a pair of brain-sized volumes: linear, default bound
        _case("warp_linear_train", "warp", (160, 192, 160), n=2, bound="zero", sigma=6.0, std=3.0),
        # the reconstruction chain: prefilter, cubic pull, push, backward to the image and the (rough) grid
        _case("chain_cubic_192", "chain", (192, 192, 192), c=3, order=3, sigma=2.0, std=4.0),
        # cubic warp of a multi-channel volume stored in 16 bits, ragged sizes, forward and backward
        _case("warp_cubic_bf16", "warp", (231, 118, 175), c=4, order=3, dtype="bfloat16"),
        # a batch of slices under affine maps, cubic, many channels, forward and backward
        _case("slices_cubic", "warp", (512, 512), n=4, c=8, order=3, bound="replicate", sigma=0.0, std=0.0),
        # splatting a large image and the splatting weights, linear (template building)
        _case("splat_256", "splat", (256, 256, 256)),
        # an iteration of a stationary-velocity registration: exponential, cubic pull, loss, backward
        _case("svf_iteration", "svf", (160, 192, 160), order=3, sigma=3.0, std=1.0),
        # upsampling a multi-channel volume, cubic with prefilter
        _case("resize_256_320", "resize", (256, 256, 256), c=3, order=3, t0=320, t1=320, t2=320),
        # the regularisation term of a registration, applied to its displacement grid
        _case("regulariser_192", "regulariser", (192, 192, 192), bound="dft", sigma=4.0, std=2.0),
        # image and spatial gradients in one call (Gauss-Newton registration), cubic, ragged sizes
        _case("pull_grad_cubic", "pull_grad", (181, 217, 181), order=3),
        # a quadratic warp of a pair of volumes under antireflecting bounds, forward and backward
        _case("warp_quadratic", "warp", (128, 128, 128), n=2, order=2, bound="dst2"),
        # many uneven volumes in one captured step, orders 1 and 3, 1-4 channels
        _case("batch_6", "batch", (), n=6, lo=64, hi=144, seed=31),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def shape(lo, hi, most):
        s = [size(lo, hi) for _ in range(3)]
        while s[0] * s[1] * s[2] > most:
            s = [max(lo, int(v * 0.95)) for v in s]
        return s

    op = rng.choice(("pull_push", "warp", "warp", "warp2d", "chain", "splat", "svf", "resize", "regulariser",
                     "pull_grad", "batch"))
    sigma, std = rng.choice((2.0, 3.0, 4.0, 6.0)), round(rng.uniform(0.5, 4.0), 2)
    bound = rng.choice(("dct2", "dct2", "zero", "dft", "replicate", "dct1", "dst1", "dst2"))
    order = rng.choice((1, 1, 2, 3, 3))
    more = {"sigma": sigma, "std": std}
    if op == "pull_push":
        return _case(None, op, shape(48, 128, 1 << 20), n=rng.choice((1, 2)), c=rng.choice((1, 2, 3)), order=order,
                     bound=bound, **more)
    if op == "warp":
        return _case(None, op, shape(48, 200, 5 << 20), n=rng.choice((1, 1, 2)), c=rng.choice((1, 2, 3, 4)),
                     order=order, bound=bound, dtype=rng.choice(("float32", "float32", "bfloat16")), **more)
    if op == "warp2d":
        return _case(None, "warp", (size(256, 640), size(256, 640)), n=rng.choice((1, 2, 4)),
                     c=rng.choice((1, 2, 3, 5, 8)), order=order, bound=bound, sigma=0.0, std=0.0)
    if op == "chain":
        return _case(None, op, shape(64, 192, 6 << 20), c=rng.choice((1, 2, 3)), order=rng.choice((2, 3, 3)),
                     bound=rng.choice(("dct2", "dft")), **more)
    if op == "splat":
        return _case(None, op, shape(64, 256, 12 << 20), c=rng.choice((1, 2)), order=rng.choice((1, 1, 3)),
                     bound=bound, **more)
    if op == "svf":
        return _case(None, op, shape(64, 176, 4 << 20), order=rng.choice((1, 3)), sigma=rng.choice((3.0, 4.0)),
                     std=round(rng.uniform(0.5, 2.0), 2))
    if op == "resize":
        s = shape(64, 256, 8 << 20)
        f = rng.uniform(0.5, 1.4)
        t = [max(8, int(v * f * rng.uniform(0.9, 1.1))) for v in s]
        return _case(None, op, s, c=rng.choice((1, 2, 3)), order=order, bound=rng.choice(("dct2", "dft")),
                     t0=t[0], t1=t[1], t2=t[2])
    if op == "regulariser":
        return _case(None, op, shape(64, 224, 7 << 20), n=rng.choice((1, 1, 2)),
                     bound=rng.choice(("dft", "dct2", "dst2")), **more)
    if op == "pull_grad":
        return _case(None, op, shape(64, 224, 7 << 20), c=rng.choice((1, 2)), order=order, bound=bound, **more)
    return _case(None, op, (), n=rng.choice((3, 4, 5, 6)), lo=64, hi=rng.choice((96, 128, 144)),
                 seed=rng.randrange(1 << 20))


def _shape(case):
    return tuple(case["s%d" % i] for i in range(3) if "s%d" % i in case)


def _volumes(case):
    """(shape, channels, order) of the batch's volumes."""
    g = torch.Generator().manual_seed(case["seed"])
    out = []
    for v in range(case["n"]):
        shape = tuple(int(s) for s in torch.randint(case["lo"], case["hi"] + 1, (3,), generator=g))
        out.append((shape, int(torch.randint(1, 5, (1,), generator=g)), 1 if v % 2 == 0 else 3))
    return out


# ------------------------------------------------------------------------------------------------------ #
# inputs                                                                                                 #
# ------------------------------------------------------------------------------------------------------ #

def _smooth_noise(gen, lead, shape, sigma):
    """Unit-variance Gaussian noise smoothed over `sigma` voxels (a spectral, periodic smoothing)."""
    x = torch.randn((*lead, *shape), generator=gen, device="cuda")
    if sigma <= 0:
        return x
    dims = tuple(range(-len(shape), 0))
    f = torch.fft.rfftn(x, dim=dims)
    gain = 1.0
    for d, s in enumerate(shape):
        last = d == len(shape) - 1
        k = torch.fft.rfftfreq(s, device="cuda") if last else torch.fft.fftfreq(s, device="cuda")
        h = torch.exp(-2.0 * (math.pi * sigma * k) ** 2)
        full = torch.exp(-2.0 * (math.pi * sigma * torch.fft.fftfreq(s, dtype=F64)) ** 2)
        gain *= float((full ** 2).mean())
        f = f * h.reshape([-1 if e == d else 1 for e in range(len(shape))])
    return torch.fft.irfftn(f, s=shape, dim=dims) / math.sqrt(gain)


def _grid(case, gen, n, shape):
    """(n, *shape, D) sampling coordinates: identity plus a smooth displacement, or affine maps."""
    ident = nb.identity_grid(shape, device="cuda")
    dim = len(shape)
    if case["sigma"] > 0:
        disp = _smooth_noise(gen, (n, dim), shape, case["sigma"]) * case["std"]
        return (ident + disp.movedim(1, -1)).contiguous()
    # rotation, scaling and shift about the centre of the field of view
    centre = torch.tensor([(s - 1) / 2 for s in shape], device="cuda")
    r = torch.rand((n, 2 * dim + 1), generator=gen, device="cuda") * 2 - 1
    ang = r[:, 0] * math.radians(15)
    rot = torch.stack([torch.stack([ang.cos(), -ang.sin()], -1), torch.stack([ang.sin(), ang.cos()], -1)], -2)
    mat = rot * (1 + 0.1 * r[:, 1:1 + dim])[:, None, :]
    shift = centre + 10 * r[:, 1 + dim:]
    return (torch.einsum("nij,xyj->nxyi", mat, ident - centre) + shift[:, None, None, :]).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    op, n, c = case["op"], case["n"], case["c"]
    if op == "batch":
        vols = _volumes(case)
        b = PullPushBatch([v[0] for v in vols], [v[1] for v in vols], [v[2] for v in vols], form="percall")
        for k, (shape, ch, _) in enumerate(vols):
            b.x[k].copy_(torch.rand((1, ch, *shape), generator=gen, device="cuda"))
            b.grid[k].copy_(_grid(case, gen, 1, shape))
            b.w[k].copy_(torch.randn((1, ch, *shape), generator=gen, device="cuda"))
        return {"case": case, "batch": b.capture()}
    shape, dtype = _shape(case), DTYPES[case["dtype"]]
    s = {"case": case}
    if op == "regulariser":
        disp = _smooth_noise(gen, (n, 3), shape, case["sigma"]) * case["std"]
        s["v"] = disp.movedim(1, -1).contiguous()
    elif op == "svf":
        vel = _smooth_noise(gen, (1, 3), shape, case["sigma"]) * case["std"]
        s["v"] = vel.movedim(1, -1).contiguous().requires_grad_()
        moving = _smooth_noise(gen, (1, 1), shape, 3.0)
        s["x"] = nb.spline_coeff_nd(moving, interpolation=case["order"], bound="dct2", dim=3)
        s["fixed"] = _smooth_noise(gen, (1, 1), shape, 3.0)
    elif op == "resize":
        s["x"] = torch.rand((n, c, *shape), generator=gen, device="cuda")
    else:
        grad = op in ("warp", "chain")
        x = torch.rand((n, c, *shape), generator=gen, device="cuda") + _smooth_noise(gen, (n, c), shape, 2.0)
        s["x"] = x.to(dtype).requires_grad_(grad)
        s["grid"] = _grid(case, gen, n, shape).requires_grad_(grad)
        if grad:
            s["w"] = torch.randn((n, c, *shape), generator=gen, device="cuda").to(dtype)
    return s


# ------------------------------------------------------------------------------------------------------ #
# the calls                                                                                              #
# ------------------------------------------------------------------------------------------------------ #

def run(state):
    case = state["case"]
    op = case["op"]
    if op == "batch":
        b = state["batch"]
        b.step()
        return [b.z, b.dx, b.dgrid]
    opt = {"interpolation": case["order"], "bound": case["bound"]}
    if op == "regulariser":
        return solve.c_regulariser_grid(state["v"], **PENALTIES, bound=case["bound"])
    if op == "resize":
        return nb.resize(state["x"], shape=[case["t0"], case["t1"], case["t2"]], **opt)
    if op == "svf":
        grid = svf.exp(state["v"])
        warped = nb.grid_pull(state["x"], grid, interpolation=case["order"], bound="dct2", extrapolate=True)
        loss = (warped - state["fixed"]).square().mean()
        return [warped.detach(), torch.autograd.grad(loss, state["v"])[0]]
    x, grid = state["x"], state["grid"]
    if op == "pull_push":
        y = nb.grid_pull(x, grid, **opt)
        return [y, nb.grid_push(y, grid, **opt)]
    if op == "splat":
        return [nb.grid_push(x, grid, **opt), nb.grid_count(grid, **opt)]
    if op == "pull_grad":
        return list(nb.grid_pull_grad(x, grid, **opt))
    if op == "warp":
        y = nb.grid_pull(x, grid, **opt)
        return [y.detach(), *torch.autograd.grad(y, (x, grid), state["w"])]
    y = nb.grid_pull(x, grid, prefilter=True, **opt)  # chain
    z = nb.grid_push(y, grid, **opt)
    return [z.detach(), *torch.autograd.grad(z, (x, grid), state["w"])]


def work(case):
    """Bytes: each input read once and each output written once (intermediate results that leave one public
    call and enter the next included).  Operations: the multiplications and additions of the separable sums."""
    op = case["op"]
    if op == "batch":
        parts = [work(_case("", "chain", s, c=c, order=o, prefiltered=True)) for s, c, o in _volumes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    shape, n, c, taps = _shape(case), case["n"], case["c"], case["order"] + 1
    dim, e = len(shape), 2 if case["dtype"] == "bfloat16" else 4
    vox = n * math.prod(shape)
    tap_sum = sum(taps ** (d + 1) for d in range(dim))  # multiply-adds of one separable sum
    img, grd, one = e * c * vox, 4 * dim * vox, 2.0 * tap_sum * c * vox
    if op == "regulariser":
        return {"bytes": 2.0 * grd, "flops": 2.0 * 3 * 33 * vox}
    if op == "resize":
        out = n * c * case["t0"] * case["t1"] * case["t2"]
        return {"bytes": 4.0 * (n * c * math.prod(shape) + out), "flops": 2.0 * 3 * taps * out}
    if op == "svf":  # 8 compositions forward (field in, field out) and backward (field, gradient in, gradient out)
        return {"bytes": float(8 * 5 * grd + 2 * grd + 4 * img), "flops": 2.0 * 14 * 3 * 8 * 3 * vox + 4 * one}
    if op == "pull_push":
        return {"bytes": 2.0 * grd + 4 * img, "flops": 2 * one}
    if op == "splat":
        return {"bytes": 2.0 * grd + 2 * img + 4 * vox, "flops": one + 2.0 * tap_sum * vox}
    if op == "pull_grad":
        return {"bytes": float(grd + 2 * img + dim * img), "flops": (1 + dim) * one}
    if op == "warp":
        return {"bytes": 3.0 * grd + 5 * img, "flops": (2 + dim) * one}
    chain = {"bytes": 6.0 * grd + 10 * img, "flops": (4 + 2 * dim) * one}
    if not case.get("prefiltered"):
        chain["bytes"] += 4 * img
        chain["flops"] += 2 * 2.0 * 2 * dim * c * vox
    return chain


# ------------------------------------------------------------------------------------------------------ #
# the same in 64 bits                                                                                    #
# ------------------------------------------------------------------------------------------------------ #

def _bspline(order, d):
    """Values and derivatives of the centred B-spline of order 1, 2 or 3 at the signed distances d."""
    a, s = d.abs(), torch.sign(d)
    if order == 1:
        return (1 - a).clamp(min=0), -s
    if order == 2:
        near = a < 0.5
        return (torch.where(near, 0.75 - a * a, 0.5 * (1.5 - a).clamp(min=0) ** 2),
                torch.where(near, -2 * d, -s * (1.5 - a).clamp(min=0)))
    near, far = a < 1, (2 - a).clamp(min=0)
    return (torch.where(near, 2 / 3 + a * a * (a / 2 - 1), far ** 3 / 6),
            torch.where(near, s * a * (1.5 * a - 2), -s * far ** 2 / 2))


def _bounded(i, n, bound):
    """Where the bound condition finds node i of an axis of n nodes, and its sign (0: nowhere)."""
    one = torch.ones_like(i, dtype=F64)
    if bound == "zero":
        return i.clamp(0, n - 1), ((i >= 0) & (i < n)).to(F64)
    if bound == "replicate":
        return i.clamp(0, n - 1), one
    if bound == "dft":
        return i % n, one
    if bound == "dct1":
        p = max(1, 2 * (n - 1))
        j = i % p
        return torch.where(j >= n, p - j, j), one
    if bound in ("dct2", "dst2"):
        j = i % (2 * n)
        up = j >= n
        return torch.where(up, 2 * n - 1 - j, j), (one if bound == "dct2" else torch.where(up, -one, one))
    j = i % (2 * (n + 1))  # dst1: odd about the nodes -1 and n, which hold zero
    up = j > n
    sign = torch.where(j % (n + 1) == n, 0 * one, torch.where(up, -one, one))
    return torch.where(up, 2 * n - j, j).clamp(0, n - 1), sign


def _axis(x, n, order, bound):
    """Nodes, weights and derivative weights of the samples x along an axis of n nodes."""
    low = torch.floor(x - (order - 1) / 2)
    taps = []
    for k in range(order + 1):
        w, g = _bspline(order, x - (low + k))
        if order == 1:
            g = torch.full_like(x, 1.0 if k else -1.0)
        idx, sign = _bounded((low + k).long(), n, bound)
        taps.append((idx, w * sign, g * sign))
    return taps


def _taps(grid, shape, order, bound):
    """Every tap of the samples grid (P, D): offset, weight, gradient of the weight per axis."""
    axes = [_axis(grid[:, d], s, order, bound) for d, s in enumerate(shape)]

    def walk(d, off, w, grads):
        if d == len(shape):
            yield off, w, grads
            return
        for idx, wd, gd in axes[d]:
            yield from walk(d + 1, off * shape[d] + idx, w * wd, [g * wd for g in grads] + [w * gd])

    one = torch.ones_like(grid[:, 0])
    yield from walk(0, torch.zeros_like(grid[:, 0], dtype=torch.long), one, [])


def _inside(grid, shape):
    """The samples that the field-of-view test keeps, a comparison in the grid's own precision."""
    ok = torch.ones(grid.shape[:-1], dtype=torch.bool, device=grid.device)
    for d, s in enumerate(shape):
        ok &= (grid[..., d] >= -0.05) & (grid[..., d] < torch.tensor(s - 1, dtype=grid.dtype) + 0.05)
    return ok


def _pull(img, grid, keep, order, bound, grads=False):
    """img (C, *shape), grid (P, D) -> values (C, P) and, if asked, their gradients (C, P, D)."""
    flat = img.reshape(img.shape[0], -1)
    val = torch.zeros((img.shape[0], grid.shape[0]), dtype=F64, device=img.device)
    grad = torch.zeros((*val.shape, grid.shape[1]), dtype=F64, device=img.device) if grads else None
    for off, w, gs in _taps(grid, img.shape[1:], order, bound):
        v = flat[:, off]
        val += v * w
        for d, g in enumerate(gs if grads else ()):
            grad[..., d] += v * g
    return (val * keep, grad * keep[:, None]) if grads else val * keep


def _push(val, grid, keep, shape, order, bound):
    out = torch.zeros((val.shape[0], math.prod(shape)), dtype=F64, device=val.device)
    for off, w, _ in _taps(grid, shape, order, bound):
        out.index_add_(1, off, val * (w * keep))
    return out.reshape(val.shape[0], *shape)


def _axis_matrix(x, n, order, bound):
    m = torch.zeros((x.shape[0], n), dtype=F64, device=x.device)
    rows = torch.arange(x.shape[0], device=x.device)
    for idx, w, _ in _axis(x, n, order, bound):
        m.index_put_((rows, idx), w, accumulate=True)
    return m


def _along(x, mat, axis):
    return torch.movedim(torch.movedim(x, axis, -1) @ mat.T, -1, axis)


def _prefilter(x, dim, order, bound):
    """Spline coefficients along the last `dim` axes: the inverse of sampling the spline at the nodes."""
    if order < 2:
        return x
    for d in range(x.dim() - dim, x.dim()):
        n = x.shape[d]
        nodes = torch.arange(n, dtype=F64, device=x.device)
        x = _along(x, torch.linalg.inv(_axis_matrix(nodes, n, order, bound)), d)
    return x


def _sampled(case, s):
    """The sampling calls, batch item by batch item."""
    order, bound, op = case["order"], case["bound"], case["op"]
    with torch.no_grad():
        outs = []
        for k in range(s["x"].shape[0]):
            x, g32 = s["x"][k].to(F64), s["grid"][k]
            shape, lattice, dim = x.shape[1:], g32.shape[:-1], g32.shape[-1]
            grid, keep = g32.reshape(-1, dim).to(F64), _inside(g32, x.shape[1:]).reshape(-1).to(F64)
            flat = x.reshape(x.shape[0], -1)

            def lat(v):
                return v.reshape(v.shape[0], *lattice, *v.shape[2:])

            if op == "splat":
                outs.append([_push(flat, grid, keep, shape, order, bound),
                             _push(torch.ones_like(flat[:1]), grid, keep, shape, order, bound)])
            elif op == "pull_push":
                y = _pull(x, grid, keep, order, bound)
                outs.append([lat(y), _push(y, grid, keep, shape, order, bound)])
            elif op == "pull_grad":
                y, g = _pull(x, grid, keep, order, bound, True)
                outs.append([lat(y), lat(g)])
            elif op == "warp":
                w = s["w"][k].to(F64).reshape(x.shape[0], -1)
                y, g = _pull(x, grid, keep, order, bound, True)
                outs.append([lat(y), _push(w, grid, keep, shape, order, bound),
                             (w[..., None] * g).sum(0).reshape(g32.shape)])
            else:
                outs.append(_chain(x, grid, keep, s["w"][k].to(F64), order, bound, g32.shape, op == "chain"))
        return [torch.stack(v) for v in zip(*outs)]


def _chain(x, grid, keep, w, order, bound, gshape, prefilter):
    """pull -> push -> <., w>: the pushed image, and the gradients of the image and the grid."""
    dim, shape = x.dim() - 1, x.shape[1:]
    coef = _prefilter(x, dim, order, bound) if prefilter else x
    y, gy = _pull(coef, grid, keep, order, bound, True)
    dy, gw = _pull(w, grid, keep, order, bound, True)
    dx = _push(dy, grid, keep, shape, order, bound)
    return [_push(y, grid, keep, shape, order, bound), _prefilter(dx, dim, order, bound) if prefilter else dx,
            (y[..., None] * gw + dy[..., None] * gy).sum(0).reshape(gshape)]


def _svf(case, s):
    with torch.no_grad():
        shape, order = _shape(case), case["order"]
        ident = torch.stack(torch.meshgrid(*[torch.arange(v, dtype=F64, device="cuda") for v in shape],
                                           indexing="ij"), -1).reshape(-1, 3)
        keep = torch.ones_like(ident[:, 0])

        def image(u):
            return u.T.reshape(3, *shape)

        u, states = s["v"][0].to(F64).reshape(-1, 3) / 256, []
        for _ in range(8):
            states.append(u)
            u = u + _pull(image(u), ident + u, keep, 1, "dft").T
        warped, grad = _pull(s["x"][0].to(F64), ident + u, keep, order, "dct2", True)
        diff = warped - s["fixed"][0].to(F64).reshape(1, -1)
        g = 2 * diff[0][:, None] / diff.numel() * grad[0]
        for u in reversed(states):
            _, gu = _pull(image(u), ident + u, keep, 1, "dft", True)
            back = _push(g.T.contiguous(), ident + u, keep, shape, 1, "dft").reshape(3, -1).T
            g = g + back + torch.einsum("pc,cpd->pd", g, gu)
        return [warped.reshape(1, 1, *shape), (g / 256).reshape(s["v"].shape)]


def _resize(case, s):
    shape, order, bound = _shape(case), case["order"], case["bound"]
    x = _prefilter(s["x"].to(F64), 3, order, bound)
    for d in range(3):
        i, o = shape[d], case["t%d" % d]
        at = torch.arange(o, dtype=F64, device="cuda") * ((i - 1) / (o - 1))
        x = _along(x, _axis_matrix(at, i, order, bound), 2 + d)
    return x


def _regulariser(case, s):
    """The matrix of absolute, membrane, bending and linear-elastic energies of a unit-voxel grid."""
    v, bound = s["v"].to(F64), case["bound"]

    def step(x, axis, k):  # x at the node k steps along the axis
        idx, sign = _bounded(torch.arange(x.shape[axis], device="cuda") + k, x.shape[axis], bound)
        return torch.index_select(x, axis, idx) * sign.reshape([-1 if a == axis else 1 for a in range(x.dim())])

    lam0, lam1, lam2, (mu, lam) = (PENALTIES[k] for k in ("absolute", "membrane", "bending", "lame"))
    out = torch.empty_like(v)
    for d in range(3):
        u = v[..., d]
        acc = lam0 * u
        for a in range(1, 4):
            w1 = -12.0 * lam2 - lam1 - (2 * mu + lam if a == d + 1 else mu)
            acc = acc + w1 * (step(u, a, -1) + step(u, a, 1) - 2 * u)
            acc = acc + lam2 * (step(u, a, -2) + step(u, a, 2) - 2 * u)
            for b in range(a + 1, 4):
                for i in (-1, 1):
                    for j in (-1, 1):
                        acc = acc + 2 * lam2 * (step(step(u, a, i), b, j) - u)
        for e in range(3):
            for i in (-1, 1):
                for j in (-1, 1):
                    if e != d:
                        acc = acc - 0.25 * (mu + lam) * i * j * step(step(v[..., e], d + 1, i), e + 1, j)
        out[..., d] = acc
    return out


def exact(case, seed):
    s = prepare(case, seed)
    if case["op"] == "batch":
        b, outs = s["batch"], []
        with torch.no_grad():
            for k, (shape, _, order) in enumerate(_volumes(case)):
                x, g32 = b.x[k][0].to(F64), b.grid[k][0]
                keep = _inside(g32, shape).reshape(-1).to(F64)
                outs.append(_chain(x, g32.reshape(-1, 3).to(F64), keep, b.w[k][0].to(F64), order, "dct2",
                                   g32.shape, False))
        return [[o[j][None] for o in outs] for j in range(3)]
    if case["op"] == "svf":
        return _svf(case, s)
    if case["op"] == "resize":
        return _resize(case, s)
    if case["op"] == "regulariser":
        return _regulariser(case, s)
    return _sampled(case, s)
