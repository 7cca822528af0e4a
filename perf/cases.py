"""The work that programs have this framework do, as measured cases.

A registration spends its time in the metric's value and derivative, called once per
iteration with host parameters in and value and derivative out; a level of its pyramid
begins with Initialize (smoothing, the moving gradient, the sample list); the filters,
whole registrations and batches of them are called by themselves.  The sizes are those of
the benchmark (64^3, 256x256x200 and its pyramid, 192x192x160) and odd ones among them.

Images are 12 Gaussian blobs with noise (sigma 3 to 10 voxels, amplitude 50 to 200), the
moving image is the fixed one under a small affine (or affine and B-spline) transform with
fresh noise, mapped by a nonlinear intensity function for the mutual informations.

A program keeps its parameters and gradients as float32 (torch's default): that is the
precision of the metric's per-sample arithmetic.  A displacement field's call is on device
buffers, which are float64 by the entry point's own definition.
"""
import ctypes
import math

import numpy as np
import torch

import itk_gb300 as gb

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the smallest call: one iteration of a dense 64^3 MeanSquares registration, where
        # launches and their latency are the time
        dict(name="msq_dense_64", op="eval", metric="msq", transform="affine", nx=64, ny=64, nz=64, fraction=0.0),
        # the coarsest level of a pyramid over 256x256x200 (shrink 4), 20 % random samples, odd sizes
        dict(name="mattes_coarse_61x67x53", op="eval", metric="mattes", transform="affine", nx=61, ny=67, nz=53,
             fraction=0.2, bins=50),
        # the benchmark's evaluation: the finest level of a multimodal affine registration
        dict(name="mattes_256x256x200", op="eval", metric="mattes", transform="affine", nx=256, ny=256, nz=200,
             fraction=0.2, bins=50),
        # the largest call: every voxel of the finest level (no sampling), same-modality images
        dict(name="msq_dense_256x256x200", op="eval", metric="msq", transform="affine", nx=256, ny=256, nz=200,
             fraction=0.0),
        # deformable registration on a coarse control grid: [affine, B-spline of mesh 4], 10 % samples
        dict(name="mattes_bspline4_192", op="eval", metric="mattes", transform="bspline", mesh=4, nx=192, ny=192,
             nz=160, fraction=0.1, bins=50),
        # a finer control grid, same-modality, odd sizes
        dict(name="msq_bspline8_173x181x149", op="eval", metric="msq", transform="bspline", mesh=8, nx=173, ny=181,
             nz=149, fraction=0.2),
        # a dense deformation: displacement field and derivative field stay on the device
        dict(name="mattes_field_192", op="field", metric="mattes", nx=192, ny=192, nz=160, bins=50),
        # the histogram metric with the smoothed joint PDF at its default 20 bins
        dict(name="jhmi_256x256x200", op="eval", metric="jhmi", transform="affine", nx=256, ny=256, nz=200,
             fraction=0.2, bins=20),
        # the start of the middle level of the same pyramid (shrink 2, sigma 1 mm): Initialize
        # and the first evaluation
        dict(name="level_256x256x200", op="level", nx=256, ny=256, nz=200, shrink=2, sigma=1.0, fraction=0.2, bins=50),
        # the moving gradient (or any image's) at full size
        dict(name="gradient_256x256x200", op="gradient", nx=256, ny=256, nz=200, sigma=1.0),
        # a whole small registration from host images to the transform, as a program runs it
        dict(name="register_64", op="register", nx=64, ny=64, nz=64),
        # a batch of small registrations advancing together, half MeanSquares and half Mattes, ten iterations
        dict(name="batch_8", op="batch", count=8, nx=72, ny=72, nz=56, iterations=10, bins=50),
    ]


def draw(rng):
    def axis(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["eval", "eval", "eval", "eval", "field", "level", "gradient", "smooth", "register", "batch"])
    c = dict(op=op, nx=axis(48, 256), ny=axis(48, 256), nz=axis(40, 200))
    if op == "eval":
        c["metric"] = rng.choice(["msq", "mattes", "mattes", "jhmi"])
        c["transform"] = rng.choice(["affine", "affine", "bspline"])
        c["fraction"] = round(math.exp(rng.uniform(math.log(0.02), math.log(0.4))), 3)
        if c["metric"] == "msq" and c["transform"] == "affine" and rng.random() < 0.5:
            c["fraction"] = 0.0
        if c["transform"] == "bspline":
            c["mesh"] = rng.randint(3, 8)
        if c["metric"] != "msq":
            c["bins"] = rng.choice([20, 32, 50, 64])
        c["central"] = rng.random() < 0.2  # CentralDifferenceImageFunction instead of the gradient filter
    elif op == "field":
        c.update(nx=axis(48, 192), ny=axis(48, 192), nz=axis(40, 160), metric=rng.choice(["msq", "mattes"]), bins=50)
    elif op == "level":
        c.update(shrink=rng.choice([1, 2, 4]), sigma=rng.choice([0.0, 1.0, 2.0]), bins=50,
                 fraction=rng.choice([0.1, 0.2]))
    elif op == "gradient" or op == "smooth":
        c["sigma"] = round(rng.uniform(0.7, 4.0), 2)
    elif op == "register":
        c.update(nx=axis(40, 72), ny=axis(40, 72), nz=axis(40, 72))
    else:
        c.update(count=rng.randint(3, 10), nx=axis(40, 80), ny=axis(40, 80), nz=axis(40, 64), iterations=10, bins=50)
    return c


# ---------------------------------------------------------------------------
# inputs: made from the seed alone, with plain torch

def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(1000003 * (int(seed) % 1000003) + 17)


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=DEVICE, dtype=F64)


def _blobs(case, g):
    """The noiseless fixed volume, (nz, ny, nx) float64."""
    n = [case["nx"], case["ny"], case["nz"]]
    k = 12
    c = [_uniform(g, 0.0, 1.0, k) * (n[d] - 1) for d in range(3)]
    s, a = _uniform(g, 3.0, 10.0, k), _uniform(g, 50.0, 200.0, k)
    e = [torch.exp(-(torch.arange(n[d], device=DEVICE, dtype=F64)[None] - c[d][:, None]) ** 2
                   / (2 * s[:, None] ** 2)) for d in range(3)]
    return torch.einsum("k,kz,ky,kx->zyx", a, e[2], e[1], e[0])


def _noise(g, shape, sigma):
    return sigma * torch.randn(*shape, generator=g, device=DEVICE, dtype=torch.float32)


def _affine(g, center, rot_deg, trans, scale):
    """(matrix, translation) of a small affine transform about `center`, float64 numpy."""
    r = np.deg2rad(_uniform(g, -rot_deg, rot_deg, 3).cpu().numpy())
    (cx, cy, cz), (sx, sy, sz) = np.cos(r), np.sin(r)
    m = (np.array([[cz, -sz, 0], [sz, cz, 0], [0, 0, 1]]) @ np.array([[cy, 0, sy], [0, 1, 0], [-sy, 0, cy]])
         @ np.array([[1, 0, 0], [0, cx, -sx], [0, sx, cx]]))
    return m @ np.diag(_uniform(g, 1 - scale, 1 + scale, 3).cpu().numpy()), _uniform(g, -trans, trans, 3).cpu().numpy()


def _voxels(case, lo=0, hi=None):
    """Voxel indices lo..hi of the scan order as (n, 3) xyz, float64."""
    nx, ny = case["nx"], case["ny"]
    i = torch.arange(lo, nx * ny * case["nz"] if hi is None else hi, device=DEVICE)
    return torch.stack([i % nx, i // nx % ny, i // (nx * ny)], 1).to(F64)


def _inputs(case, seed, multimodal):
    """fixed, moving (float32 volumes, 1 mm spacing), an affine's matrix, translation and
    centre near the aligning one, and B-spline coefficients or None."""
    g = _gen(seed)
    f = _blobs(case, g)
    center = (np.array([case["nx"], case["ny"], case["nz"]]) - 1.0) / 2.0
    m, t = _affine(g, center, 4.0, 3.0, 0.03)
    coef = None
    if case.get("transform") == "bspline":
        coef = _uniform(g, -1.0, 1.0, 3, *((case["mesh"] + 3,) * 3)) * (2.0 / math.sqrt(3.0))
    total = f.numel()
    mv = torch.empty(total, device=DEVICE, dtype=torch.float32)
    f32 = f.float()
    for lo in range(0, total, 1 << 22):
        x = _voxels(case, lo, min(total, lo + (1 << 22)))
        y = x if coef is None else x + _spline(case, coef, x)[0]
        y = _map(m, t, center, y)
        v = _trilinear(f32, y)
        mv[lo:lo + len(v)] = torch.where(_inside(f32, y), v, torch.zeros_like(v)).float()
    mv = mv.reshape(f.shape)
    if multimodal:
        mv = 1000.0 * (mv.clamp_min(0.0) / mv.max()) ** 1.7 + _noise(g, f.shape, 5.0)
    else:
        mv = mv + _noise(g, f.shape, 2.0)
    fixed = f32 + _noise(g, f.shape, 2.0)
    # mid-registration: the aligning transform (the generating one's inverse), off by about a voxel
    dm, dt = _affine(g, center, 0.5, 0.8, 0.005)
    m = np.linalg.inv(m)
    return fixed, mv, dm @ m, dt - m @ t, center, None if coef is None else -0.7 * coef


def _points(case, seed, spacing=(1.0, 1.0, 1.0), origin=(0.0, 0.0, 0.0), size=None):
    """RANDOM sampling: voxel picks with replacement and N(0, spacing / 3) jitter, float32."""
    g = _gen(seed + 500009)
    size = size or (case["nx"], case["ny"], case["nz"])
    total = size[0] * size[1] * size[2]
    n = max(64, int(total * case["fraction"]))
    i = (torch.rand(n, generator=g, device=DEVICE, dtype=F64) * total).long().clamp_max(total - 1)
    x = torch.stack([i % size[0], i // size[0] % size[1], i // (size[0] * size[1])], 1).to(F64)
    x = x + torch.randn(n, 3, generator=g, device=DEVICE, dtype=F64) / 3.0
    return (x * torch.tensor(spacing, device=DEVICE, dtype=F64)
            + torch.tensor(origin, device=DEVICE, dtype=F64)).float()


def _field(case, seed):
    """A smooth displacement of every voxel (at most about 2 mm), (nz, ny, nx, 3) float64."""
    g = _gen(seed + 700001)
    a, p = _uniform(g, 0.2, 0.5, 3, 4), _uniform(g, 0.0, 6.28, 3, 4, 3)
    w = [torch.arange(n, device=DEVICE, dtype=F64) / n for n in (case["nx"], case["ny"], case["nz"])]
    u = torch.zeros(case["nz"], case["ny"], case["nx"], 3, device=DEVICE, dtype=F64)
    for d in range(3):
        for k in range(4):
            e = [torch.sin((k + 1) * 3.14 * w[q] + p[d, k, q]) for q in range(3)]
            u[..., d] += a[d, k] * e[2][:, None, None] * e[1][:, None] * e[0]
    return u


def _gradient_image(vol):
    """Central differences of a volume in float64, xyz, (nz, ny, nx, 3)."""
    gz, gy, gx = torch.gradient(vol.to(F64))
    return torch.stack([gx, gy, gz], -1)


# ---------------------------------------------------------------------------
# prepare and run

_METRICS = {"msq": gb.MeanSquaresImageToImageMetricv4, "mattes": gb.MattesMutualInformationImageToImageMetricv4,
            "jhmi": gb.JointHistogramMutualInformationImageToImageMetricv4}


def _affine_transform(m, t, center):
    a = gb.AffineTransform()
    a.SetCenter(center)
    a.SetMatrix(m)
    a.SetTranslation(t)
    return a


def _metric(kind, fixed, moving, transform, bins):
    m = _METRICS[kind]()
    m.SetFixedImage(fixed)
    m.SetMovingImage(moving)
    m.SetMovingTransform(transform)
    if kind != "msq":
        m.SetNumberOfHistogramBins(bins)
    return m


def _host(vol):
    return gb.Image(vol.cpu().numpy())


def _optimizer(size, iterations):
    # scales in the manner of the physical shift: a matrix entry moves points by about the half extent
    r = 0.5 * max(size)
    o = gb.RegularStepGradientDescentOptimizerv4()
    o.SetLearningRate(1.0)
    o.SetMinimumStepLength(1e-3)
    o.SetNumberOfIterations(iterations)
    o.SetScales(np.array([r * r] * 9 + [1.0] * 3))
    return o


def _member(case, k):
    """Registration k of a batch: a smaller volume than the one before it."""
    return dict(case, fraction=0.2, **{n: case[n] - case[n] * k // 20 for n in ("nx", "ny", "nz")})


def prepare(case, seed):
    op = case["op"]
    size = (case["nx"], case["ny"], case["nz"])
    s = dict(op=op, case=case)
    if op in ("gradient", "smooth"):
        vol, _, _, _, _, _ = _inputs(case, seed, False)
        s["in"] = vol
        s["out"] = torch.empty(*vol.shape, *((3,) if op == "gradient" else ()), device=DEVICE)
        s["size"], s["spacing"] = (ctypes.c_int64 * 3)(*size), (ctypes.c_double * 3)(1.0, 1.0, 1.0)
        s["direction"] = (ctypes.c_double * 9)(1, 0, 0, 0, 1, 0, 0, 0, 1)
        s["sigmas"] = (ctypes.c_double * 3)(*[case["sigma"]] * 3)
        s["lib"], s["context"] = gb.lib(), gb.context()
        return s
    if op == "batch":
        s["members"] = []
        for k in range(case["count"]):
            kind = "msq" if k % 2 == 0 else "mattes"
            member = _member(case, k)
            f, mv, _, _, center, _ = _inputs(member, seed + 31 * k, kind == "mattes")
            start = _affine_transform(np.eye(3), np.zeros(3), center)
            m = _metric(kind, _host(f), _host(mv), start, case["bins"])
            if kind == "mattes":
                m.SetVirtualSampledPointSet(_points(member, seed + 31 * k).cpu().numpy())
                m.SetUseSampledPointSet(True)
            m.Initialize()
            o = _optimizer((member["nx"], member["ny"], member["nz"]), case["iterations"])
            o.SetMetric(m)
            s["members"].append((start, o))
        s["begin"] = [t.GetParameters() for t, _ in s["members"]]
        return s
    if op == "register":
        f, mv, _, _, center, _ = _inputs(case, seed, False)
        s["fixed"], s["moving"], s["center"] = _host(f), _host(mv), center
        return s
    kind = case.get("metric", "mattes")
    f, mv, m, t, center, coef = _inputs(case, seed, kind != "msq")
    a = _affine_transform(m, t, center)
    if op == "field":
        u = gb.DisplacementFieldImage(_field(case, seed).cpu().numpy())
        d = gb.DisplacementFieldTransform()
        d.SetDisplacementField(u)
        c = gb.CompositeTransform()
        c.AddTransform(a)
        c.AddTransform(d)
        s["metric"] = _metric(kind, _host(f), _host(mv), c, case.get("bins", 0))
        s["metric"].SetMovingImageGradientImage(gb.GradientImage(_gradient_image(mv).cpu().numpy()))
        s["metric"].Initialize()
        # the field and [value, valid points, derivative] stay on the device
        s["params"] = torch.from_numpy(u.array.reshape(-1)).to(DEVICE)
        s["out"] = torch.zeros(2 + s["params"].numel(), device=DEVICE, dtype=F64)
        return s
    transform = a
    if coef is not None:
        b = gb.BSplineTransform()
        b.SetTransformDomain(np.zeros(3), np.array(size, np.float64) - 1.0, (case["mesh"],) * 3)
        b.SetParameters(coef.cpu().numpy().reshape(-1))
        transform = gb.CompositeTransform()
        transform.AddTransform(a)
        transform.AddTransform(b)
    s["metric"] = _metric(kind, _host(f), _host(mv), transform, case.get("bins", 0))
    if op == "level":
        osize, ospacing, oorigin = _shrunk(case)
        s["metric"].SetLevelShrinkFactors((case["shrink"],) * 3)
        s["metric"].SetLevelSmoothingSigma(case["sigma"])
        s["metric"].SetVirtualSampledPointSet(_points(case, seed, ospacing, oorigin, osize).cpu().numpy())
        s["metric"].SetUseSampledPointSet(True)
    else:
        s["metric"].SetUseMovingImageGradientFilter(not case.get("central", False))
        if case["fraction"] > 0:
            s["metric"].SetVirtualSampledPointSet(_points(case, seed).cpu().numpy())
            s["metric"].SetUseSampledPointSet(True)
        s["metric"].Initialize()
    s["grad"] = np.empty(transform.GetNumberOfParameters(), np.float32)
    return s


def run(s):
    op = s["op"]
    if op == "eval" or op == "level":
        m = s["metric"]
        if op == "level":
            m.Initialize()
        value, derivative = m.GetValueAndDerivative()
        np.copyto(s["grad"], derivative, casting="same_kind")
        return value, s["grad"], m.GetNumberOfValidPoints()
    if op == "field":
        s["metric"].evaluate_device(s["params"].data_ptr(), s["out"].data_ptr(), True)
        _check(s["metric"].synchronize())
        return s["out"]
    if op == "gradient":
        stream = torch.cuda.current_stream().cuda_stream
        _check(s["lib"].gb_gradient_recursive_gaussian(s["context"], stream, s["in"].data_ptr(), s["out"].data_ptr(),
                                                       s["size"], s["spacing"], s["direction"], s["case"]["sigma"],
                                                       1, 1))
        return s["out"]
    if op == "smooth":
        stream = torch.cuda.current_stream().cuda_stream
        _check(s["lib"].gb_smooth_recursive_gaussian(s["context"], stream, s["in"].data_ptr(), s["out"].data_ptr(),
                                                     s["size"], s["spacing"], s["sigmas"]))
        return s["out"]
    if op == "batch":
        b = gb.RegistrationBatch()
        for (t, o), p in zip(s["members"], s["begin"]):
            t.SetParameters(p)
            b.Add(o)
        b.Run()
        return [(t.GetParameters().astype(np.float32), o.GetValue()) for t, o in s["members"]]
    t = _affine_transform(np.eye(3), np.zeros(3), s["center"])
    o = _optimizer(s["fixed"].GetSize(), 100)
    r = gb.ImageRegistrationMethodv4()
    r.SetFixedImage(s["fixed"])
    r.SetMovingImage(s["moving"])
    r.SetMetric(gb.MeanSquaresImageToImageMetricv4())
    r.SetOptimizer(o)
    r.SetInitialTransform(t)
    r.Update()
    return t.GetParameters().astype(np.float32), o.GetValue()


def _check(status):
    if status:
        raise RuntimeError(gb.lib().gb_last_error().decode())


def work(case):
    """Bytes and operations that a pass cannot do without."""
    v = case["nx"] * case["ny"] * case["nz"]
    op = case["op"]
    if op == "gradient":  # per voxel: nine line filters of 16 multiply-adds share five
        return dict(bytes=16.0 * v, flops=8 * 34.0 * v)
    if op == "smooth":
        return dict(bytes=8.0 * v, flops=3 * 34.0 * v)
    if op == "field":  # field in, derivative out, fixed value, moving value and gradient
        return dict(bytes=v * (24.0 + 24 + 4 + 16), flops=250.0 * v)
    if op == "level":
        n = int(v / case["shrink"] ** 3 * case["fraction"])
        return dict(bytes=8.0 * v + 12.0 * n, flops=(2 * 3 * 34.0 if case["sigma"] else 0) * v + 8 * 34.0 * v
                    + 300.0 * n)
    if op == "register":
        return dict(bytes=8.0 * v, flops=200.0 * v)
    if op == "batch":
        return dict(bytes=8.0 * v * case["count"], flops=100.0 * v * case["count"] * case["iterations"])
    # an evaluation: the samples, each voxel under a stencil (fixed, moving, gradient), the parameters
    f = case["fraction"]
    n = v if f == 0 else int(v * f)
    touched = v if f == 0 else v * (1.0 - math.exp(-8.0 * f))
    p = 3 * (case["mesh"] + 3) ** 3 if case["transform"] == "bspline" else 12
    return dict(bytes=12.0 * (0 if f == 0 else n) + 20.0 * touched + 16.0 * p,
                flops=(250.0 if p == 12 else 1000.0) * n)


# ---------------------------------------------------------------------------
# the same results in 64 bits

def _map(m, t, center, x):
    m = torch.as_tensor(m, device=x.device, dtype=F64)
    c = torch.as_tensor(center, device=x.device, dtype=F64)
    return (x - c) @ m.T + (torch.as_tensor(t, device=x.device, dtype=F64) + c)


def _inside(vol, x):
    n = torch.tensor(vol.shape[2::-1], device=x.device, dtype=F64)
    return ((x >= -0.5) & (x < n - 0.5)).all(1)


def _trilinear(vol, x):
    """Trilinear samples of a (nz, ny, nx[, c]) volume at continuous indices x (n, 3),
    neighbours clamped to the buffer."""
    n = torch.tensor(vol.shape[2::-1], device=x.device)
    b = torch.floor(x)
    d = torch.where(b < 0, torch.zeros_like(x), x - b)
    b = b.long()
    lo = torch.minimum(b.clamp_min(0), n - 1)
    hi = torch.minimum((b + 1).clamp_min(0), n - 1)
    out = None
    flat = vol.reshape(-1, *vol.shape[3:])
    for z in (0, 1):
        for y in (0, 1):
            for q in (0, 1):
                i = ((hi if z else lo)[:, 2] * vol.shape[1] + (hi if y else lo)[:, 1]) * vol.shape[2] \
                    + (hi if q else lo)[:, 0]
                w = (d[:, 0] if q else 1 - d[:, 0]) * (d[:, 1] if y else 1 - d[:, 1]) * (d[:, 2] if z else 1 - d[:, 2])
                v = flat[i].to(F64)
                v = v * (w if v.dim() == 1 else w[:, None])
                out = v if out is None else out + v
    return out


def _spline(case, coef, x):
    """Displacement of a cubic B-spline over the volume's extent (1 mm voxels), the 12 axis
    weights, the first node and whether a point is inside the valid region."""
    mesh = case["mesh"]
    extent = torch.tensor([case["nx"], case["ny"], case["nz"]], device=x.device, dtype=F64) - 1.0
    ci = x / (extent / mesh) + 1.0
    top = float(mesh + 1)
    ci = torch.where((ci - top).abs() <= 4 * 2.3e-16 * top, torch.full_like(ci, top * (1 - 6e-16)), ci)
    ok = ((ci >= 1.0) & (ci < top)).all(1)
    start = torch.where(ok[:, None], torch.floor(ci - 1.0), torch.zeros_like(ci)).long()
    t = torch.where(ok[:, None], ci - start - 1.0, torch.zeros_like(ci))
    u = 1.0 - t
    w = torch.stack([u ** 3, 3 * t ** 3 - 6 * t ** 2 + 4, -3 * t ** 3 + 3 * t ** 2 + 3 * t + 1, t ** 3], 2) / 6.0
    g = mesh + 3
    flat = coef.reshape(3, -1).T
    out = torch.zeros_like(x)
    for k in range(64):
        a, b, c = k & 3, (k >> 2) & 3, k >> 4
        node = (start[:, 0] + a) + g * ((start[:, 1] + b) + g * (start[:, 2] + c))
        out += (w[:, 0, a] * w[:, 1, b] * w[:, 2, c])[:, None] * flat[node]
    return torch.where(ok[:, None], out, torch.zeros_like(out)), w, start, ok


def _recursive(vol, axis, sigma, order, across_scale=False):
    """One pass of the recursive Gaussian (Deriche's form with Farneback and Westin's
    parameters, edge values extended) along `axis` (0 = x), 1 mm voxels, float64."""
    a1, b1, w1, l1 = (1.3530, 1.8151, 0.6681, -1.3932) if order == 0 else (-0.6724, -3.4327, 0.6681, -1.3932)
    a2, b2, w2, l2 = (-0.3531, 0.0902, 2.0787, -1.3732) if order == 0 else (0.6724, 0.6100, 2.0787, -1.3732)
    c1, c2, s1, s2 = math.cos(w1 / sigma), math.cos(w2 / sigma), math.sin(w1 / sigma), math.sin(w2 / sigma)
    e1, e2 = math.exp(l1 / sigma), math.exp(l2 / sigma)
    # each pair is (num0 + num1 z) / (1 + den1 z + den2 z^2); their sum is the causal filter
    p1, q1 = np.array([a1, e1 * (b1 * s1 - a1 * c1)]), np.array([1.0, -2 * e1 * c1, e1 * e1])
    p2, q2 = np.array([a2, e2 * (b2 * s2 - a2 * c2)]), np.array([1.0, -2 * e2 * c2, e2 * e2])
    n, d = np.convolve(p1, q2) + np.convolve(p2, q1), np.convolve(q1, q2)
    k = np.arange(4)
    sn, dn, sd, dd = n.sum(), (n * k).sum(), d.sum(), (d * np.arange(5)).sum()
    alpha = 2 * sn / sd - n[0] if order == 0 else 2 * (sn * dd - dn * sd) / sd ** 2
    n = n * ((sigma if order and across_scale else 1.0) / alpha)
    m = (1.0 if order == 0 else -1.0) * (np.append(n[1:], 0.0) - d[1:] * n[0])
    x = vol.to(F64).movedim(2 - axis, 0).contiguous()
    y, z = torch.empty_like(x), torch.empty_like(x)
    last = len(x) - 1
    first = x[0] * (n.sum() / d.sum())
    for i in range(len(x)):
        o = sum(n[j] * x[max(i - j, 0)] for j in range(4))
        y[i] = o - sum(d[j] * (y[i - j] if i >= j else first) for j in range(1, 5))
    first = x[last] * (m.sum() / d.sum())
    for i in range(last, -1, -1):
        o = sum(m[j - 1] * x[min(i + j, last)] for j in range(1, 5))
        z[i] = o - sum(d[j] * (z[i + j] if i + j <= last else first) for j in range(1, 5))
    return (y + z).movedim(0, 2 - axis)


def _smooth(vol, sigma):
    for axis in (2, 0, 1):
        vol = _recursive(vol, axis, sigma, 0)
    return vol


def _gradient(vol, sigma):
    """The normalized gradient (xyz) by first order along one axis and zero order along the others."""
    dx, sx = _recursive(vol, 0, sigma, 1, True), _recursive(vol, 0, sigma, 0)
    sxy = _recursive(sx, 1, sigma, 0)
    return torch.stack([_recursive(_recursive(dx, 1, sigma, 0), 2, sigma, 0),
                        _recursive(_recursive(sx, 1, sigma, 1, True), 2, sigma, 0),
                        _recursive(sxy, 2, sigma, 1, True)], -1)


def _shrunk(case):
    """Size, spacing and origin of the volume's grid shrunk about its centre (1 mm voxels)."""
    f = case["shrink"]
    n = [case["nx"], case["ny"], case["nz"]]
    size = [max(1, k // f) for k in n]
    return size, [float(f)] * 3, [(k - 1) / 2.0 - f * (o - 1) / 2.0 for k, o in zip(n, size)]


def _moving_at(mv, grad, y):
    """Moving value and gradient at continuous indices; `grad` None: central differences of
    half a voxel to each side, zero where one of them is outside."""
    v = _trilinear(mv, y)
    if grad is not None:
        return v, _trilinear(grad, y)
    g = torch.zeros_like(y)
    for k in range(3):
        h = torch.zeros(3, device=y.device, dtype=F64)
        h[k] = 0.5
        ok = _inside(mv, y - h) & _inside(mv, y + h)
        g[:, k] = torch.where(ok, _trilinear(mv, y + h) - _trilinear(mv, y - h), g[:, k])
    return v, g


def _evaluate(case, kind, f, mv, grad, x, params, bins, field=None):
    """value, derivative, valid points of a metric in 64 bits; x: the virtual points;
    params: (matrix, translation, centre, B-spline coefficients or None)."""
    m, t, center, coef = params
    dense = x is None
    total = f.numel() if dense else len(x)
    keep = []  # per chunk: rows, fixed value, moving value, gradient, what the Jacobian needs
    for lo in range(0, total, 1 << 21):
        xs = _voxels(case, lo, min(total, lo + (1 << 21))) if dense else x[lo:lo + (1 << 21)].to(F64)
        ok = _inside(f, xs)
        fv = _trilinear(f, xs).float().to(F64)
        w = start = jac = None
        y = xs
        if coef is not None:
            u, w, start, jac = _spline(case, coef, xs)
            y = xs + u
        elif field is not None:
            y = xs + field.reshape(-1, 3)[lo:lo + len(xs)]
        y = _map(m, t, center, y)
        ok = ok & _inside(mv, y)
        v, g = _moving_at(mv, grad, y[ok])
        keep.append((torch.nonzero(ok)[:, 0] + lo, fv[ok], v, g, xs[ok], *((w[ok], start[ok], jac[ok]) if coef is not None
                                                                           else (None,) * 3)))
    rows, fv, v, g, xs, w, start, jac = [None if c[0] is None else torch.cat(c) for c in zip(*keep)]
    del keep

    def contract(s, sel=slice(None)):
        """sum over the samples of s J^T g, or s M^T g per voxel for a field."""
        mt = torch.as_tensor(m, device=g.device, dtype=F64)
        gs = g[sel] * s[:, None]
        if coef is None and field is None:
            d = gs.T @ (xs[sel] - torch.as_tensor(center, device=g.device, dtype=F64))
            return torch.cat([d.reshape(-1), gs.sum(0)])
        a = gs @ mt
        if field is not None:
            out = torch.zeros(total, 3, device=g.device, dtype=F64)
            out[rows[sel]] = a
            return out.reshape(-1)
        a = torch.where(jac[sel][:, None], a, torch.zeros_like(a))
        gn = case["mesh"] + 3
        out = torch.zeros(gn ** 3, 3, device=g.device, dtype=F64)
        ww, st = w[sel], start[sel]
        for k in range(64):
            p, q, r = k & 3, (k >> 2) & 3, k >> 4
            node = (st[:, 0] + p) + gn * ((st[:, 1] + q) + gn * (st[:, 2] + r))
            out.index_add_(0, node, (ww[:, 0, p] * ww[:, 1, q] * ww[:, 2, r])[:, None] * a)
        return out.T.reshape(-1)

    if kind == "msq":
        n = len(fv)
        d = contract(2.0 * (fv - v))
        return ((fv - v) ** 2).sum() / n, d if field is not None else d / n, n
    mlo, mhi = float(mv.min()), float(mv.max())
    if kind == "mattes":
        if dense:
            flo, fhi = float(f.min()), float(f.max())
        else:
            i = torch.floor(x.to(F64) + 0.5).long()
            n = torch.tensor(f.shape[2::-1], device=i.device)
            i = i[((i >= 0) & (i < n)).all(1)]
            at = f[i[:, 2], i[:, 1], i[:, 0]]
            flo, fhi = float(at.min()), float(at.max())
        fb, mb = (fhi - flo) / (bins - 4), (mhi - mlo) / (bins - 4)
        sel = (v >= mlo) & (v <= mhi)
        row = (fv[sel] / fb - (flo / fb - 2.0)).long().clamp(2, bins - 3)
        term = (v[sel] - mlo) / mb + 2.0
        mid = term.long().clamp(2, bins - 3)
        t1 = term - mid
        u1 = 1 - t1
        wt = torch.stack([u1 ** 3, 3 * t1 ** 3 - 6 * t1 ** 2 + 4, -3 * t1 ** 3 + 3 * t1 ** 2 + 3 * t1 + 1, t1 ** 3], 1) / 6
        dw = torch.stack([0.5 * u1 ** 2, t1 * (2 - 1.5 * t1), u1 * (1.5 * u1 - 2), -0.5 * t1 ** 2], 1)
        cols = mid[:, None] - 1 + torch.arange(4, device=mid.device)
        p = torch.zeros(bins * bins, device=g.device, dtype=F64)
        p.index_add_(0, (row[:, None] * bins + cols).reshape(-1), wt.reshape(-1))
        p = (p / p.sum()).reshape(bins, bins)
        n = len(row)
        pf, pm = torch.bincount(row, minlength=bins).to(F64) / n, p.sum(0)
        eps = 2.220446049250313e-16
        ok = (p > eps) & (pm > eps)[None] & (pf > eps)[:, None]
        ratio = torch.where(ok, torch.log(torch.where(ok, p, 1.0) / torch.where(ok, pm[None], 1.0)), 0.0)
        value = -(p * torch.where(ok, ratio - torch.log(torch.where(ok, pf[:, None], 1.0)), 0.0)).sum()
        s = (ratio[row[:, None], cols] * dw).sum(1)
        return value, contract(s, sel) * (-1.0 / (mb * n)), n
    # joint histogram: counts of nearest bins, smoothed by a discrete Gaussian of variance 1.5
    flo, fhi = float(f.min()), float(f.max())
    h = 1.0 / (bins - 5)
    pa, pb = (fv - flo) / (fhi - flo), (v - mlo) / (mhi - mlo)
    ca, cb = (pa + 2 * h) / h, (pb + 2 * h) / h
    ia, ib = torch.floor(ca + 0.5).long(), torch.floor(cb + 0.5).long()
    ok = (ia >= 0) & (ia < bins) & (ib >= 0) & (ib < bins)
    p = torch.bincount(ia[ok] + bins * ib[ok], minlength=bins * bins).to(F64).reshape(bins, bins) / int(ok.sum())
    kern = _discrete_gaussian(1.5)
    r = len(kern) // 2
    at = (torch.arange(bins)[:, None] + torch.arange(-r, r + 1)).clamp(0, bins - 1).to(g.device)
    kern = torch.tensor(kern, device=g.device, dtype=F64)
    p = torch.einsum("ikj,k->ij", p[at], kern)          # moving axis (rows)
    p = torch.einsum("jik,k->ji", p[:, at], kern)       # fixed axis
    pf, pm = p.sum(0), p.sum(1)
    den = pm[:, None] * pf[None]
    eps = 2.220446049250313e-16
    good = den > eps
    q = torch.where(good, p / torch.where(good, den, 1.0), 0.0)
    good &= q > eps
    value = -(p * torch.log(torch.where(good, q, 1.0))).sum() / math.log(2.0)

    def two(a, b):
        return _trilinear(p[None], torch.stack([a, b, torch.zeros_like(a)], 1))

    def one(b):
        return _trilinear(pm[None, None], torch.stack([b, torch.zeros_like(b), torch.zeros_like(b)], 1))

    sel = (v >= mlo) & (v <= mhi) & (ca >= -0.5) & (ca < bins - 0.5) & (cb >= -0.5) & (cb < bins - 0.5)
    ca, cb, pb = ca[sel], cb[sel], pb[sel]
    lo, hi = (pb - 0.5 * h).clamp(h, 1.0), (pb + 0.5 * h).clamp(h, 1.0)
    cl, cr, step = (lo + 2 * h) / h, (hi + 2 * h) / h, hi - lo
    wide = step > 0
    step = torch.where(wide, step, 1.0)
    dj = torch.where(wide, (two(ca, cr) - two(ca, cl)) / step, 0.0)
    dm = torch.where(wide, (one(cr) - one(cl)) / step, 0.0)
    jv, pv = two(ca, cb), one(cb)
    top = -math.log(1e-16) / h
    good = (jv > 1e-16) & (pv > 1e-16)
    s = (dj / torch.where(good, jv, 1.0)).clamp(-top, top) - (dm / torch.where(good, pv, 1.0)).clamp(-top, top)
    s = torch.where(good, s, 0.0) / (math.log(2.0) * (mhi - mlo))
    n = int(sel.sum())
    return value, contract(s, sel) / n, n


def _discrete_gaussian(variance, max_error=0.01):
    """e^-v I_k(v) until its two-sided sum reaches 1 - max_error, normalized."""
    def bessel(k):
        return sum((variance / 2) ** (2 * j + k) / (math.factorial(j) * math.factorial(j + k)) for j in range(60))

    half = [math.exp(-variance) * bessel(0), math.exp(-variance) * bessel(1)]
    while half[0] + 2 * sum(half[1:]) < 1 - max_error:
        half.append(math.exp(-variance) * bessel(len(half)))
    half = np.array(half) / (half[0] + 2 * sum(half[1:]))
    return np.concatenate([half[:0:-1], half])


def _descend(case, f, mv, kind, x, center, size, iterations, bins):
    """RegularStep gradient descent from the identity: parameters, value."""
    grad = _gradient(mv, 1.0).float()
    r = 0.5 * max(size)
    scales = np.array([r * r] * 9 + [1.0] * 3)
    p = np.concatenate([np.eye(3).reshape(-1), np.zeros(3)])
    prev, relax, value = np.zeros(12), 1.0, 0.0
    for _ in range(iterations):
        value, d, _ = _evaluate(case, kind, f, mv, grad, x, (p[:9].reshape(3, 3), p[9:], center, None), bins)
        d = d.cpu().numpy() / scales
        mag = np.linalg.norm(d)
        if mag < 1e-4:
            break
        relax *= 0.5 if float(d @ (prev / scales)) < 0 else 1.0
        if relax < 1e-3:
            break
        prev = d * relax
        p = p + prev / mag
    return p, float(value)


def exact(case, seed):
    op = case["op"]
    kind = case.get("metric", "mattes")
    size = (case["nx"], case["ny"], case["nz"])
    if op in ("gradient", "smooth"):
        vol = _inputs(case, seed, False)[0]
        return _gradient(vol, case["sigma"]) if op == "gradient" else _smooth(vol, case["sigma"])
    if op == "register":
        f, mv, _, _, center, _ = _inputs(case, seed, False)
        return _descend(case, f, mv, "msq", None, center, size, 100, 0)
    if op == "batch":
        out = []
        for k in range(case["count"]):
            kind = "msq" if k % 2 == 0 else "mattes"
            member = _member(case, k)
            f, mv, _, _, center, _ = _inputs(member, seed + 31 * k, kind == "mattes")
            out.append(_descend(member, f, mv, kind, _points(member, seed + 31 * k) if kind == "mattes" else None,
                                center, (member["nx"], member["ny"], member["nz"]), case["iterations"], case["bins"]))
        return out
    f, mv, m, t, center, coef = _inputs(case, seed, kind != "msq")
    params = (m, t, center, coef)
    if op == "field":
        value, d, n = _evaluate(case, kind, f, mv, _gradient_image(mv).float(), None, params, case["bins"],
                                _field(case, seed))
        return torch.cat([value.reshape(1), torch.tensor([float(n)], device=d.device, dtype=F64), d])
    if op == "level":
        osize, ospacing, oorigin = _shrunk(case)
        x = _points(case, seed, ospacing, oorigin, osize)
        if case["sigma"] > 0:
            f, mv = _smooth(f, case["sigma"]).float(), _smooth(mv, case["sigma"]).float()
        value, d, _ = _evaluate(case, kind, f, mv, _gradient(mv, 1.0).float(), x, params, case["bins"])
        return float(value), d.cpu().numpy(), None
    x = _points(case, seed) if case["fraction"] > 0 else None
    grad = None if case.get("central") else _gradient(mv, 1.0).float()
    value, d, _ = _evaluate(case, kind, f, mv, grad, x, params, case.get("bins", 0))
    return float(value), d.cpu().numpy(), None
