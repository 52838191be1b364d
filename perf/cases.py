"""The work a user of py4dstem_gb300 has it do, as a list of cases.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` builds what a program has in hand before the call (data,
plans, device state), ``run(state)`` makes one pass through the package's entry
points, ``work(case)`` counts the bytes and operations the pass cannot do
without, and ``exact(case, seed)`` evaluates the same pass in 64 bits with plain
torch / NumPy / SciPy operations.

The data are synthetic: a smooth random phase object with a band of atoms'
resolution, an aperture-limited defocused probe, a jittered raster of positions
and Poisson counts. A reconstruction starts from a perturbed copy of the true
object, the state of a run that is under way, and every pass starts from that
state again (the reset of a reconstruction), so that it can be repeated.
"""

import ctypes
import math

import numpy as np
import torch

from py4dstem_gb300 import DataCube, SingleslicePtychography, _native, device_preprocess, engine
from py4dstem_gb300.autograd import PtychoForwardModel
from py4dstem_gb300.tomography import VolumeOps

DEV = "cuda"
SAMPLING = 0.25      # object pixel, Angstrom
WAVELENGTH = 0.0196875  # Angstrom (300 kV)


def listed():
    """The cases; `path` selects the entry points, the rest are sizes and options."""
    return [
        # the CPU-runnable workload of the package through its class: a 32 x 32 scan
        # on a 64^2 detector in batches of 64, four iterations per call; 64 small
        # batches, so launches and host work between them count
        dict(name="gd64_class", path="class", det=64, scan_x=32, scan_y=32, batch=64, iters=4,
             step=2.0, pad=1),
        # the throughput benchmark: one gradient-descent iteration of a 128 x 128
        # scan on a 128^2 detector, 512^2 object, batches of 1024
        dict(name="gd128_scan", path="gd", det=128, scan_x=128, scan_y=128, batch=1024, T=1, M=1,
             potential=False, mask=False, step=3.0, pad=1),
        # a ragged scan on a 96^2 detector with a detector mask and a potential
        # object: the options and odd sizes of everyday data sets
        dict(name="gd96_potential", path="gd", det=96, scan_x=43, scan_y=41, batch=250, T=1, M=1,
             potential=True, mask=True, step=2.7, pad=5),
        # thick samples: 8 slices, 128^2 detector, batches of 256
        dict(name="multislice8_128", path="gd", det=128, scan_x=48, scan_y=48, batch=256, T=8,
             M=1, potential=False, mask=False, step=1.6, pad=3),
        # partial coherence: 4 probe modes, 128^2 detector, the modes
        # orthogonalised on the device in every iteration
        dict(name="mixed4_128", path="gd", det=128, scan_x=48, scan_y=48, batch=256, T=1, M=4,
             potential=False, mask=False, step=2.0, pad=3),
        # difference map (projection sets) on whole-scan batches with persistent
        # exit waves; two iterations, the first seeds the exit waves
        dict(name="difference_map_128", path="projection", det=128, scan_x=64, scan_y=64, a=-1.0,
             b=1.0, c=2.0, step=3.0, pad=2),
        # gradient descent with position correction after every batch
        dict(name="poscorr_128", path="poscorr", det=128, scan_x=64, scan_y=64, batch=1024,
             step=3.0, pad=2),
        # large detectors: 256^2 in batches of 128
        dict(name="gd256", path="gd", det=256, scan_x=32, scan_y=32, batch=128, T=1, M=1,
             potential=False, mask=False, step=3.0, pad=1),
        # the autograd function: loss and both gradients of a 16-slice model, as an
        # optimiser's step calls it
        dict(name="autograd16_128", path="gradient", det=128, scan_x=23, scan_y=21, batch=256,
             T=16, M=1, potential=False, step=1.6, pad=1),
        # tomography: one tilt's volume work (rotate, project onto the slices, spread
        # the slice update, rotate back into the collective update)
        dict(name="volume_tilt", path="volume", n0=96, n1=160, n2=160, slices=8, angle=20.0),
        # preprocessing of a loaded scan: centre of mass, centred amplitudes, overlap
        dict(name="preprocess_128", path="preprocess", det=128, scan_x=64, scan_y=64, step=3.0,
             pad=2),
        # the largest convolution of the learned initializer's training step: forward,
        # input and weight gradients of a 3 x 3 layer on 16 images
        dict(name="unet_conv", path="conv", nb=16, height=128, width=128, cin=96, cout=32),
    ]


# 96 x 128 and 128 x 96 regions are kept out: the detectors of the listed cases
_DETECTORS = (32, 48, 64, 96, 128, 256)
_BUDGET = 128 * 128 * 128 * 128  # pixels x positions (x slices x modes) of the largest case


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["gd"] * 5 + ["class", "projection", "poscorr", "gradient", "volume",
                                    "preprocess", "conv"])
    if path == "volume":
        return dict(path=path, n0=_log_int(rng, 24, 96), n1=_log_int(rng, 40, 160),
                    n2=_log_int(rng, 40, 160), slices=rng.randint(1, 12),
                    angle=round(rng.uniform(-60.0, 60.0), 2))
    if path == "conv":
        level = rng.choice([0, 1, 2, 3])
        return dict(path=path, nb=rng.randint(1, 16), height=rng.randint(64, 128) >> level,
                    width=max(8, (rng.randint(64, 128) >> level) // 8 * 8),
                    cin=32 << rng.choice([level, max(0, level - 1)]), cout=32 << level)
    step = round(rng.uniform(1.2, 3.2), 2)
    pad = rng.randint(1, 9)
    if path == "class":
        n = rng.randint(9, 32)
        return dict(path=path, det=rng.choice([32, 48, 64]), scan_x=n, scan_y=rng.randint(9, 32),
                    batch=_log_int(rng, 16, 256), iters=rng.randint(1, 4), step=step, pad=pad)
    det = rng.choice(_DETECTORS if path == "gd" else _DETECTORS[:-1])
    T, M = 1, 1
    if path == "gd":
        T = rng.choice([1, 1, 1, 2, 4, 8])
        M = rng.choice([1, 1, 1, 2, 4])
    if path == "gradient":
        T = rng.choice([1, 4, 16])
        M = rng.choice([1, 2]) if T < 16 else 1
    most = _BUDGET // (det * det * T * M * (4 if path != "gd" else 2))
    side = max(9, min(128, int(math.sqrt(most))))
    sx = _log_int(rng, 8, side)
    sy = _log_int(rng, 8, side)
    base = dict(path=path, det=det, scan_x=sx, scan_y=sy, step=step, pad=pad)
    if path == "preprocess":
        return base
    if path == "projection":
        return dict(base, **rng.choice([dict(a=-1.0, b=1.0, c=2.0), dict(a=-0.6, b=0.8, c=2.0),
                                        dict(a=0.0, b=1.0, c=2.0)]))
    batch = _log_int(rng, 16, 1024 if T * M == 1 else 256)
    if path == "poscorr":
        return dict(base, batch=batch)
    potential = rng.random() < 0.3
    if path == "gradient":
        return dict(base, batch=batch, T=T, M=M, potential=potential)
    return dict(base, batch=batch, T=T, M=M, potential=potential, mask=rng.random() < 0.3)


# --------------------------------------------------------------------- synthetic data
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) + 7919)
    return g


def _freq(n):
    return torch.fft.fftfreq(n, 1.0, device=DEV, dtype=torch.float64)


def _smooth(gen, px, py, width):
    """A real random field of unit peak with a Gaussian spectrum (width in pixels)."""
    f = torch.randn((px, py), generator=gen, device=DEV, dtype=torch.float64)
    q2 = _freq(px)[:, None] ** 2 + _freq(py)[None] ** 2
    f = torch.fft.ifft2(torch.fft.fft2(f) * torch.exp(-2.0 * (math.pi * width) ** 2 * q2)).real
    return f / f.abs().max()


def _probe(det, modes, gen):
    """(M, det, det) complex128 probes: a 20 mrad aperture with a soft edge, 100 A
    defocus, further modes with other defoci, astigmatism and less intensity."""
    k = _freq(det) / SAMPLING * WAVELENGTH
    kx, ky = k[:, None], k[None]
    alpha = torch.sqrt(kx ** 2 + ky ** 2)
    phi = torch.atan2(ky.expand(det, det), kx.expand(det, det))
    edge = torch.clamp((0.020 - alpha) / 0.002 + 0.5, 0.0, 1.0)
    weights = (0.7, 0.15, 0.1, 0.05)
    out = []
    for m in range(modes):
        z = torch.randn(3, generator=gen, device=DEV, dtype=torch.float64).tolist() if m else (0, 0, 0)
        chi = math.pi / WAVELENGTH * alpha ** 2 * (
            -(100.0 + 25.0 * z[0]) + 15.0 * z[1] * torch.cos(2 * (phi - z[2])))
        p = torch.fft.ifft2(edge * torch.exp(-1j * chi))
        out.append(p / torch.sqrt((p.abs() ** 2).sum()) * (math.sqrt(weights[m]) if modes > 1 else 1.0))
    return torch.stack(out)


def _positions(case, gen):
    """(J, 2) float32 positions in object pixels and the object's shape."""
    det, step = case["det"], case["step"]
    sx, sy = case["scan_x"], case["scan_y"]
    px = int(math.ceil((sx - 1) * step)) + det + 2 * case["pad"]
    py = int(math.ceil((sy - 1) * step)) + det + 2 * case["pad"] + 1
    x = torch.arange(sx, device=DEV, dtype=torch.float64) * step
    y = torch.arange(sy, device=DEV, dtype=torch.float64) * step
    pos = torch.stack(torch.meshgrid(x, y, indexing="ij"), -1).reshape(-1, 2)
    pos = pos + (torch.rand(pos.shape, generator=gen, device=DEV, dtype=torch.float64) - 0.5) * 0.4
    pos = pos + torch.tensor([det / 2 + case["pad"], det / 2 + case["pad"]], device=DEV)
    return pos.float(), (px, py)


def _propagators(det, count):
    k = _freq(det) / SAMPLING
    h = torch.exp(-1j * math.pi * WAVELENGTH * 20.0 * (k[:, None] ** 2 + k[None] ** 2))
    return h.to(torch.complex64).expand(count, det, det).contiguous() if count else None


def _patch_rows(pos, n, size):
    f = torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=torch.float64).round().long()
    return (torch.round(pos).long()[:, None] + f[None]) % size


def _indices(pos, det, shape):
    """Flat (B, det, det) object indices of the patches."""
    r = _patch_rows(pos[:, 0], det, shape[0])
    c = _patch_rows(pos[:, 1], det, shape[1])
    return r[:, :, None] * shape[1] + c[:, None, :]


def _shifted(probe, pos, dtype):
    """(B, M, det, det): the probes shifted by the positions' sub-pixel parts."""
    frac = (pos - torch.round(pos)).double()
    k = _freq(probe.shape[-1])
    rx = torch.exp(-2j * math.pi * k[None] * frac[:, :1]).to(dtype)
    ry = torch.exp(-2j * math.pi * k[None] * frac[:, 1:]).to(dtype)
    return torch.fft.ifft2(torch.fft.fft2(probe)[None] * (rx[:, :, None] * ry[:, None, :])[:, None])


def _data(case, seed):
    """Inputs of a scan: a dict of device tensors (float32 / complex64)."""
    gen = _gen(seed)
    det, T, M = case["det"], case.get("T", 1), case.get("M", 1)
    pos, shape = _positions(case, gen)
    true, start = [], []
    for _ in range(T):
        phase = 0.35 * _smooth(gen, *shape, 1.2) + 0.3 * _smooth(gen, *shape, 4.0)
        if case.get("potential"):
            phase = phase - phase.min()
        amp = torch.exp(-0.1 * phase.abs())
        guess = phase * 0.8 + 0.05 * _smooth(gen, *shape, 6.0)
        if case.get("potential"):
            true.append(torch.exp(1j * phase))
            start.append(guess.abs())
        else:
            true.append(amp * torch.exp(1j * phase))
            start.append((1.0 - 0.05 * phase.abs()) * torch.exp(1j * guess))
    true = torch.stack(true).to(torch.complex64)
    start = torch.stack(start).to(torch.float32 if case.get("potential") else torch.complex64)
    probe = _probe(det, M, gen)
    dose = 1e5
    pr = probe.to(torch.complex64)
    props = _propagators(det, T - 1)
    J = pos.shape[0]
    amps = torch.empty((J, det, det), dtype=torch.float32, device=DEV)
    chunk = max(1, (1 << 24) // (det * det * M))
    for s in range(0, J, chunk):
        p = pos[s:s + chunk]
        idx = _indices(p, det, shape)
        w = _shifted(pr, p, torch.complex64)
        for t in range(T):
            w = w * true[t].reshape(-1)[idx][:, None]
            if t + 1 < T:
                w = torch.fft.ifft2(torch.fft.fft2(w) * props[t])
        inten = (torch.fft.fft2(w).abs() ** 2).sum(1)
        inten = inten * (dose / (det * det))
        amps[s:s + chunk] = torch.sqrt(torch.poisson(inten, generator=gen))
    # the probe carries the dose: sum |FFT2 P|^2 = counts per pattern
    probe = probe * math.sqrt(dose) / det
    order = torch.randperm(J, generator=gen, device=DEV)
    start_probe = probe * torch.exp(0.1j * _smooth(gen, det, det, 6.0))
    mask = None
    if case.get("mask"):
        q = _freq(det)
        mask = ((q[:, None] ** 2 + q[None] ** 2) < 0.2).float()
        mask[det // 3, det // 5] = 0.0
    return dict(pos=pos, shape=shape, object=start[0] if T == 1 else start,
                probe=start_probe.to(torch.complex64), amps=amps, props=props, order=order,
                mask=mask, mean=float((amps.double() ** 2).sum((1, 2)).mean()))


# ------------------------------------------------------------------------ preparation
def prepare(case, seed):
    with torch.no_grad():
        return _PREPARE[case["path"]](case, seed)


def _state(case, d, batch, **kw):
    M = case.get("M", 1)
    probe = d["probe"].cpu().numpy()
    return engine.create_state(
        roi_shape=(case["det"],) * 2, object_array=d["object"].cpu().numpy(),
        probe_array=probe if M > 1 else probe[0], amplitudes=d["amps"],
        positions_px=d["pos"].cpu().numpy(), num_slices=case.get("T", 1), num_probes=M,
        potential=bool(case.get("potential", False)), max_batch=min(batch, d["pos"].shape[0]),
        storage="gpu", propagators=None if d["props"] is None else d["props"].cpu().numpy(),
        detector_mask=None if d["mask"] is None else d["mask"].cpu().numpy(),
        mixed_state=M > 1, **kw)


def _prepare_gd(case, seed):
    d = _data(case, seed)
    st = _state(case, d, case["batch"])
    drv = engine.IterationDriver(
        st, max_batch=st.max_batch, step_size=0.5, normalization_min=1.0,
        orthogonalize_probe=case["M"] > 1, device_orthogonalization=True,
        mean_intensity=d["mean"], graph=True)
    return dict(path="gd", st=st, drv=drv, object=st.object.clone(), probe=st.probe.clone(),
                order=d["order"].cpu().numpy())


def _prepare_projection(case, seed):
    d = _data(case, seed)
    st = _state(case, d, d["pos"].shape[0], projection=True)
    drv = engine.IterationDriver(
        st, max_batch=st.max_batch, projection=True,
        projection_abc=(case["a"], case["b"], case["c"]), normalization_min=1.0,
        mean_intensity=d["mean"])
    return dict(path="projection", st=st, drv=drv, object=st.object.clone(),
                probe=st.probe.clone(), order=np.arange(d["pos"].shape[0]))


def _prepare_poscorr(case, seed):
    d = _data(case, seed)
    st = _state(case, d, case["batch"], positions_initial=d["pos"].cpu().numpy())
    drv = engine.IterationDriver(
        st, max_batch=st.max_batch, step_size=0.5, normalization_min=1.0,
        mean_intensity=d["mean"],
        position_correction=dict(step_size=0.9, max_update_px=0.5, max_total_px=2.0,
                                 center_of_mass=False))
    return dict(path="poscorr", st=st, drv=drv, object=st.object.clone(), probe=st.probe.clone(),
                positions=st.positions.clone(), order=d["order"].cpu().numpy())


def _class_data(case, seed):
    """What the class call takes: detector-centred counts, scan positions (A) and
    start arrays on the host."""
    d = _data(case, seed)
    det = case["det"]
    counts = torch.fft.fftshift(torch.round(d["amps"].double() ** 2).float(), dim=(-2, -1))
    counts = counts.reshape(case["scan_x"], case["scan_y"], det, det).cpu().numpy()
    return d, counts


def _prepare_class(case, seed):
    d, counts = _class_data(case, seed)
    det = case["det"]
    scan = (case["scan_x"], case["scan_y"])
    px, py = d["shape"]
    cube = DataCube(counts, r_pixel_size=case["step"] * SAMPLING, r_pixel_units="A",
                    q_pixel_size=1.0 / (det * SAMPLING), q_pixel_units="A^-1")
    p = SingleslicePtychography(
        energy=300e3, datacube=cube, initial_object_guess=d["object"].cpu().numpy(),
        initial_probe_guess=d["probe"][0].cpu().numpy(),
        initial_scan_positions=d["pos"].double().cpu().numpy() * SAMPLING,
        object_padding_px=(0, 0), verbose=False, device="gpu")
    centre = np.full(scan, det / 2, np.float32)
    p.preprocess(force_com_measured=(centre, centre), force_com_shifts=(centre, centre),
                 force_com_rotation=0.0, force_com_transpose=False, object_fov_mask=True, center_positions_in_fov=False,
                 plot_center_of_mass=False, plot_rotation=False, plot_probe_overlaps=False)
    return dict(path="class", p=p, seed=int(seed) % 1000, iters=case["iters"],
                batch=min(case["batch"], scan[0] * scan[1]))


def _prepare_gradient(case, seed):
    d = _data(case, seed)
    model = PtychoForwardModel(
        d["amps"], d["pos"], d["shape"], num_slices=case["T"], num_probes=case["M"],
        potential=case["potential"],
        propagators=None if d["props"] is None else d["props"].cpu().numpy(),
        max_batch=case["batch"])
    probe = d["probe"] if case["M"] > 1 else d["probe"][0]
    return dict(path="gradient", model=model, object=d["object"].clone().requires_grad_(True),
                probe=probe.clone().requires_grad_(True))


def _volume_data(case, seed):
    gen = _gen(seed)
    shape = (case["n0"], case["n1"], case["n2"])
    f = torch.randn(shape, generator=gen, device=DEV, dtype=torch.float32)
    q = [torch.fft.fftfreq(n, 1.0, device=DEV) for n in shape]
    q2 = q[0][:, None, None] ** 2 + q[1][None, :, None] ** 2 + q[2][None, None] ** 2
    f = torch.fft.ifftn(torch.fft.fftn(f) * torch.exp(-30.0 * q2)).real
    vol = (f.clamp_min(0) / f.max() * 0.2).float().contiguous()
    upd = (0.01 * torch.randn((case["slices"],) + shape[1:], generator=gen, device=DEV)).float()
    t = math.radians(case["angle"])
    rot = np.array([[1.0, 0.0, 0.0], [0.0, math.cos(t), -math.sin(t)],
                    [0.0, math.sin(t), math.cos(t)]])
    return shape, vol, upd, rot


def _prepare_volume(case, seed):
    shape, vol, upd, rot = _volume_data(case, seed)
    ops = VolumeOps(shape, case["slices"], torch.device(DEV, torch.cuda.current_device()))
    return dict(path="volume", ops=ops, vol=vol, new=upd, rot=rot, tilted=torch.empty_like(vol),
                sliced=torch.empty_like(upd), collective=torch.empty_like(vol),
                update=torch.empty(shape, dtype=torch.float64, device=DEV))


def _preprocess_data(case, seed):
    d = _data(case, seed)
    det = case["det"]
    counts = torch.fft.fftshift(d["amps"] ** 2, dim=(-2, -1)).contiguous()
    J = counts.shape[0]
    ramp = np.linspace(-0.4, 0.6, J).reshape(case["scan_x"], case["scan_y"])
    cfx = (det / 2 + ramp).astype(np.float32)
    cfy = (det / 2 + 0.25 - 0.7 * ramp).astype(np.float32)
    return d, counts, cfx, cfy


def _prepare_preprocess(case, seed):
    d, counts, cfx, cfy = _preprocess_data(case, seed)
    return dict(path="preprocess", counts=counts, cfx=cfx, cfy=cfy,
                probe=d["probe"][0].cpu().numpy(), pos=d["pos"].cpu().numpy(), shape=d["shape"])


def _conv_data(case, seed):
    gen = _gen(seed)
    nb, h, w, ci, co = (case[k] for k in ("nb", "height", "width", "cin", "cout"))

    def rand(*s):
        return torch.randn(s, generator=gen, device=DEV)

    x = torch.relu(rand(nb, h, w, ci)).to(torch.bfloat16)
    weight = (rand(co, 9, ci) * math.sqrt(2.0 / (9 * ci))).to(torch.bfloat16)
    return x, weight, 0.1 * rand(co), (1e-3 * rand(nb, h, w, co)).to(torch.bfloat16)


def _prepare_conv(case, seed):
    x, weight, bias, dy = _conv_data(case, seed)
    nb, h, w, ci, co = (case[k] for k in ("nb", "height", "width", "cin", "cout"))
    nbytes = int(_native.lib().ptycho_nn_conv3x3_wgrad_workspace_bytes(nb, h, w, ci, co))
    return dict(path="conv", sizes=(nb, h, w, ci, co), x=x, weight=weight, bias=bias, dy=dy,
                weight_t=weight.permute(2, 1, 0).contiguous(),
                y=torch.empty((nb, h, w, co), dtype=torch.bfloat16, device=DEV),
                dx=torch.empty((nb, h, w, ci), dtype=torch.float32, device=DEV),
                dw=torch.empty((co, 9, ci), dtype=torch.float32, device=DEV),
                db=torch.empty(co, dtype=torch.float32, device=DEV),
                ws=torch.empty(max(nbytes, 1), dtype=torch.uint8, device=DEV), nbytes=nbytes,
                flag=torch.zeros(1, dtype=torch.int32, device=DEV))


_PREPARE = dict(gd=_prepare_gd, projection=_prepare_projection, poscorr=_prepare_poscorr,
                gradient=_prepare_gradient, volume=_prepare_volume,
                preprocess=_prepare_preprocess, conv=_prepare_conv)
_PREPARE["class"] = _prepare_class


# ------------------------------------------------------------------------------- runs
def run(state):
    return _RUN[state["path"]](state)


def _reset(s):
    s["st"].object.copy_(s["object"])
    s["st"].probe.copy_(s["probe"])


def _run_gd(s):
    st = s["st"]
    _reset(s)
    s["drv"].iterate(s["order"])
    return dict(object=st.object, probe=st.probe, error=st.error_accum)


def _run_projection(s):
    st = s["st"]
    _reset(s)
    st.exit_waves_valid = False
    s["drv"].iterate(s["order"])
    s["drv"].iterate(s["order"])
    return dict(object=st.object, probe=st.probe, error=st.error_accum, exit_waves=st.exit_waves)


def _run_poscorr(s):
    st = s["st"]
    _reset(s)
    st.positions.copy_(s["positions"])
    s["drv"].iterate(s["order"])
    return dict(object=st.object, probe=st.probe, error=st.error_accum, positions=st.positions)


def _run_class(s):
    p = s["p"]
    p.reconstruct(num_iter=s["iters"], max_batch_size=s["batch"], seed_random=s["seed"],
                  step_size=0.5, reset=True, progress_bar=False)
    return dict(object=p.object, probe=p.probe, errors=np.array(p.error_iterations))


def _run_gradient(s):
    loss = s["model"].loss(s["object"], s["probe"])
    g_obj, g_probe = torch.autograd.grad(loss, (s["object"], s["probe"]))
    return dict(loss=loss.detach(), object=g_obj, probe=g_probe)


def _run_volume(s):
    ops = s["ops"]
    ops.rotate(s["vol"], s["tilted"], s["rot"], 0)
    ops.project(s["tilted"], s["sliced"])
    ops.expand(s["new"], s["sliced"], s["update"], 1)
    s["collective"].zero_()
    ops.rotate(s["update"], s["collective"], s["rot"].T, 2)
    return dict(tilted=s["tilted"], sliced=s["sliced"], collective=s["collective"])


def _run_preprocess(s):
    cx, cy = device_preprocess.pattern_com(s["counts"])
    amps, mean = device_preprocess.normalize_patterns(s["counts"], s["cfx"], s["cfy"], None, 0)
    overlap = device_preprocess.probe_overlap(s["probe"], s["pos"], s["shape"], 1024)
    return dict(com_x=cx, com_y=cy, amplitudes=amps, mean=float(mean), overlap=overlap)


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _run_conv(s):
    lib = _native.lib()
    nb, h, w, ci, co = s["sizes"]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for status in (
            lib.ptycho_nn_conv3x3_forward(_p(s["x"]), nb, h, w, ci, _p(s["weight"]),
                                          _p(s["bias"]), co, 1, _p(s["y"]), _p(s["flag"]),
                                          stream),
            lib.ptycho_nn_conv3x3_backward_data(_p(s["dy"]), nb, h, w, co, _p(s["weight_t"]), ci,
                                                _p(s["dx"]), _p(s["flag"]), stream),
            lib.ptycho_nn_conv3x3_backward_weight(_p(s["x"]), _p(s["dy"]), nb, h, w, ci, co,
                                                  _p(s["dw"]), _p(s["db"]), _p(s["ws"]),
                                                  s["nbytes"], _p(s["flag"]), stream)):
        if status:
            raise RuntimeError(lib.ptycho_nn_last_error().decode())
    return dict(y=s["y"], dx=s["dx"], dweight=s["dw"], dbias=s["db"])


_RUN = dict(gd=_run_gd, projection=_run_projection, poscorr=_run_poscorr, gradient=_run_gradient,
            volume=_run_volume, preprocess=_run_preprocess, conv=_run_conv)
_RUN["class"] = _run_class


# ------------------------------------------------------------------------------- work
def _object_shape(case):
    return (int(math.ceil((case["scan_x"] - 1) * case["step"])) + case["det"] + 2 * case["pad"],
            int(math.ceil((case["scan_y"] - 1) * case["step"])) + case["det"] + 2 * case["pad"] + 1)


def work(case):
    path = case["path"]
    if path == "volume":
        n = case["n0"] * case["n1"] * case["n2"]
        sl = case["slices"] * case["n1"] * case["n2"]
        # volume read, tilted and collective written, slices read and written; a
        # separable 4-tap sum over 3 axes and the three prefilter recursions, twice
        return dict(bytes=4.0 * (3 * n + 2 * sl), flops=2.0 * n * (2 * 84 + 3 * 6))
    if path == "conv":
        nb, h, w, ci, co = (case[k] for k in ("nb", "height", "width", "cin", "cout"))
        pix = nb * h * w
        return dict(bytes=pix * (2.0 * ci + 4.0 * co + 4.0 * ci) + 9.0 * ci * co * 8.0,
                    flops=3.0 * 2.0 * 9 * ci * co * pix)
    n = case["det"] ** 2
    J = case["scan_x"] * case["scan_y"]
    px, py = _object_shape(case)
    if path == "preprocess":
        # counts read, amplitudes and the overlap written; one transform per position
        return dict(bytes=8.0 * J * n + 4.0 * px * py,
                    flops=J * n * (5.0 * math.log2(n) + 40.0))
    T, M = case.get("T", 1), case.get("M", 1)
    iters = case.get("iters", 2 if path == "projection" else 1)
    obj = T * px * py * (4 if case.get("potential") else 8)
    ffts = 3 + 4 * (T - 1) + (1 if path == "gradient" else 0) + (2 if path == "poscorr" else 0)
    flops = J * M * n * (ffts * 5.0 * math.log2(n) + 50.0 * T) * iters
    nbytes = iters * (4.0 * J * n + 2.0 * obj + 16.0 * M * n)
    if path == "projection":
        nbytes += 3 * 8.0 * J * n  # exit waves: written, then read and written
    return dict(bytes=nbytes, flops=flops)


# -------------------------------------------------------------------- 64-bit evaluation
def exact(case, seed):
    with torch.no_grad():
        return _EXACT[case["path"]](case, seed)


def _batches(n, most):
    nb = -(-n // most)
    base, extra = divmod(n, nb)
    start = 0
    for i in range(nb):
        size = base + (1 if i < extra else 0)
        yield start, start + size
        start += size


def _normaliser(s, m=1.0):
    return 1.0 / torch.sqrt(1e-16 + ((1 - m) * s) ** 2 + (m * s.max()) ** 2)


class _Model64:
    """The reconstruction loop in complex128 (single slice, multislice, mixed state
    and both; gradient descent, projection sets, position correction)."""

    def __init__(self, case, d):
        self.det, self.T, self.M = case["det"], case.get("T", 1), case.get("M", 1)
        self.mixed = self.M > 1
        self.potential = bool(case.get("potential"))
        self.shape = d["shape"]
        obj = d["object"].reshape((self.T,) + tuple(self.shape))
        self.object = obj.double() if self.potential else obj.to(torch.complex128)
        self.probe = d["probe"].to(torch.complex128)
        self.props = None if d["props"] is None else d["props"].to(torch.complex128)
        self.amps, self.pos, self.mask = d["amps"], d["pos"].double(), d["mask"]
        self.pos0 = self.pos.clone()
        self.exit_waves = None
        self.error = 0.0

    def _transmission(self, t):
        return torch.exp(1j * self.object[t]) if self.potential else self.object[t]

    def _forward(self, w, idx):
        """Per-slice probes, patches and the exit waves (B, M, S, S)."""
        probes, patches = [], []
        for t in range(self.T):
            o = self._transmission(t).reshape(-1)[idx][:, None]
            probes.append(w)
            patches.append(o)
            w = w * o
            if t + 1 < self.T:
                w = torch.fft.ifft2(torch.fft.fft2(w) * self.props[t])
        return probes, patches, w

    def _far(self, f):
        return torch.sqrt((f.abs() ** 2).sum(1))

    def _scatter(self, v, idx):
        out = torch.zeros(self.shape[0] * self.shape[1], dtype=v.dtype, device=v.device)
        if v.is_complex():
            flat = torch.view_as_real(out)
            flat.index_add_(0, idx.reshape(-1), torch.view_as_real(v.reshape(-1).contiguous()))
        else:
            out.index_add_(0, idx.reshape(-1), v.reshape(-1))
        return out.reshape(self.shape)

    def batch(self, rows, step=0.5, abc=None, correct=None):
        pos = self.pos[rows]
        idx = _indices(pos, self.det, self.shape)
        amps = self.amps[rows].double()
        shifted = _shifted(self.probe, pos, torch.complex128)
        probes, patches, psi = self._forward(shifted, idx)
        if abc is None:
            f = torch.fft.fft2(psi)
            if self.mask is not None:
                f = f * self.mask.double()
            ff = self._far(f)
            self.error += float(((amps - ff) ** 2).sum())
            r = torch.where(ff > 0, amps / ff, torch.zeros_like(ff))[:, None] * f
            if not self.mixed:
                r = torch.where((ff > 0)[:, None], r, amps[:, None].to(r.dtype))
            r = r - f
            if self.mask is not None:
                r = r * self.mask.double()
            chi = torch.fft.ifft2(r)
        else:
            a, b, c = abc
            ew = psi if self.exit_waves is None else self.exit_waves
            f = torch.fft.fft2(c * psi + (1 - c) * ew)
            ff = self._far(f)
            self.error += float(((amps - ff) ** 2).sum())
            r = torch.where(ff > 0, amps / ff, torch.zeros_like(ff))[:, None] * f
            r = torch.where((ff > 0)[:, None], r, amps[:, None].to(r.dtype))
            chi = (1 - a - b) * ew + a * psi + b * torch.fft.ifft2(r)
            self.exit_waves = chi
        back = chi
        for t in range(self.T - 1, -1, -1):
            o, p = patches[t], probes[t]
            term = torch.conj(p) * back
            if self.potential:
                term = (-1j * torch.conj(o) * term).real
            g = self._scatter(term.sum(1), idx)
            n = _normaliser(self._scatter((p.abs() ** 2).sum(1), idx))
            if abc is None:
                self.object[t] += step * g * n
            else:
                self.object[t] = g * n
            back = back * torch.conj(o)
            if t > 0:
                back = torch.fft.ifft2(torch.fft.fft2(back) * torch.conj(self.props[t - 1]))
            else:
                pn = _normaliser((o[:, 0].abs() ** 2).sum(0))
                g = back.sum(0) * pn
                self.probe = self.probe + step * g if abc is None else g
        if correct is not None:
            fo = torch.fft.fft2(psi)
            diff = (amps ** 2 - self._far(fo) ** 2).reshape(len(rows), -1)
            cols = []
            for dx, dy in ((1, 0), (0, 1)):
                r = (_patch_rows(pos[:, 0], self.det, self.shape[0]) + dx) % self.shape[0]
                q = (_patch_rows(pos[:, 1], self.det, self.shape[1]) + dy) % self.shape[1]
                at = r[:, :, None] * self.shape[1] + q[:, None, :]
                moved = torch.fft.fft2(self._forward(shifted, at)[2])
                cols.append((2 * ((fo - moved) * torch.conj(fo)).real).sum(1).reshape(
                    len(rows), -1))
            A = torch.stack(cols, -1)
            u = torch.linalg.solve(A.mT @ A, A.mT @ diff[..., None])[..., 0] * correct[0]
            norm = u.norm(dim=1, keepdim=True)
            u = torch.where(norm > correct[1], u / (norm / correct[1]), u)
            far = ((pos - self.pos0[rows]) - u).norm(dim=1, keepdim=True) > correct[2]
            self.pos[rows] = pos - torch.where(far, torch.zeros_like(u), u)

    def constraints(self):
        if self.potential:
            self.object = self.object.clamp_min(0.0)
        else:
            a = self.object.abs()
            self.object = self.object / a * a.clamp_max(1.0)
        inten = self.probe[0].abs() ** 2
        k = torch.fft.fftfreq(self.det, 1.0 / self.det, device=DEV, dtype=torch.float64)
        com = torch.stack([(k[:, None] * inten).sum(), (k[None] * inten).sum()]) / inten.sum()
        q = _freq(self.det)
        ramp = torch.exp(2j * math.pi * (q[:, None] * com[0] + q[None] * com[1]))
        self.probe = torch.fft.ifft2(torch.fft.fft2(self.probe) * ramp)
        if self.mixed:
            flat = self.probe.reshape(self.M, -1)
            vals, vecs = torch.linalg.eigh(torch.conj(flat) @ flat.T)
            vecs = vecs[:, vals.argsort(descending=True)]
            big = vecs.gather(0, vecs.abs().argmax(0, keepdim=True))
            vecs = vecs * (torch.conj(big) / big.abs())
            self.probe = (vecs.T @ flat).reshape(self.probe.shape)

    def iteration(self, order, most, **kw):
        self.error = 0.0
        for s, e in _batches(len(order), most):
            self.batch(order[s:e], **kw)
        self.constraints()

    def outputs(self):
        obj = self.object if self.T > 1 else self.object[0]
        return dict(object=obj, probe=self.probe,
                    error=torch.tensor([self.error], dtype=torch.float64))


def _exact_gd(case, seed):
    d = _data(case, seed)
    m = _Model64(case, d)
    m.iteration(d["order"], case["batch"])
    return m.outputs()


def _exact_projection(case, seed):
    d = _data(case, seed)
    m = _Model64(case, d)
    rows = torch.arange(d["pos"].shape[0], device=DEV)
    for _ in range(2):
        m.iteration(rows, len(rows), abc=(case["a"], case["b"], case["c"]))
    return dict(m.outputs(), exit_waves=m.exit_waves)


def _exact_poscorr(case, seed):
    d = _data(case, seed)
    m = _Model64(case, d)
    m.iteration(d["order"], case["batch"], correct=(0.9, 0.5, 2.0))
    return dict(m.outputs(), positions=m.pos)


def _exact_class(case, seed):
    d, counts = _class_data(case, seed)
    counts = torch.as_tensor(counts, device=DEV).double().reshape(d["amps"].shape)
    d["amps"] = torch.fft.ifftshift(torch.sqrt(counts), dim=(-2, -1))
    pos = d["pos"].double()
    pos = pos - torch.clamp(pos.min(0).values, max=0.0)
    d["pos"] = pos.float()
    m = _Model64(case, d)
    rng = np.random.RandomState(int(seed) % 1000)
    order = np.arange(d["pos"].shape[0])
    norm = float(counts.sum())
    errors = []
    for _ in range(case["iters"]):
        rng.shuffle(order)
        m.iteration(torch.from_numpy(order).to(DEV), case["batch"])
        errors.append(m.error / norm)
    out = m.outputs()
    return dict(object=out["object"].cpu().numpy(),
                probe=torch.fft.fftshift(m.probe[0], dim=(-2, -1)).cpu().numpy(),
                errors=np.array(errors))


def _exact_gradient(case, seed):
    d = _data(case, seed)
    m = _Model64(case, d)
    J = d["pos"].shape[0]
    chunk = max(1, (1 << 22) // (case["det"] ** 2 * case["T"] * case["M"]) * 8)
    obj, probe, total = m.object, m.probe, 0.0
    g_obj, g_probe = torch.zeros_like(obj), torch.zeros_like(probe)
    for s in range(0, J, chunk):
        rows = torch.arange(s, min(J, s + chunk), device=DEV)
        with torch.enable_grad():
            m.object = obj.detach().clone().requires_grad_(True)
            m.probe = probe.detach().clone().requires_grad_(True)
            idx = _indices(m.pos[rows], m.det, m.shape)
            w = _shifted(m.probe, m.pos[rows], torch.complex128)
            f = torch.fft.fft2(m._forward(w, idx)[2])
            far = f[:, 0].abs() if m.M == 1 else m._far(f)
            loss = ((m.amps[rows].double() - far) ** 2).sum()
            a, b = torch.autograd.grad(loss, (m.object, m.probe))
        g_obj += a
        g_probe += b
        total += float(loss)
    return dict(loss=torch.tensor(total, dtype=torch.float64),
                object=g_obj if case["T"] > 1 else g_obj[0],
                probe=g_probe if case["M"] > 1 else g_probe[0])


def _exact_volume(case, seed):
    from scipy.ndimage import affine_transform

    shape, vol, new, rot = _volume_data(case, seed)
    swap = np.array([[0, 1, 0], [0, 0, 1], [1, 0, 0]])

    def turned(v, r):
        tf = swap.T @ r.T @ swap
        centre = (np.array(shape) - 1) / 2
        return affine_transform(v, tf, offset=centre - tf @ centre, order=3, mode="constant")

    tilted = turned(vol.double().cpu().numpy(), rot)
    per = -(-case["n0"] // case["slices"])
    padded = np.zeros((per * case["slices"],) + tuple(shape[1:]))
    padded[:case["n0"]] = tilted
    sliced = padded.reshape((case["slices"], per) + tuple(shape[1:])).sum(1)
    upd = (new.double().cpu().numpy() - sliced) / per
    upd = np.repeat(upd, per, axis=0)[:case["n0"]]
    return dict(tilted=tilted, sliced=sliced, collective=turned(upd, rot.T))


def _exact_preprocess(case, seed):
    d, counts, cfx, cfy = _preprocess_data(case, seed)
    det = case["det"]
    c = counts.double()
    k = torch.arange(det, device=DEV, dtype=torch.float64)
    tot = c.sum((1, 2))
    out = dict(com_x=((c * k[:, None]).sum((1, 2)) / tot).cpu().numpy(),
               com_y=((c * k[None]).sum((1, 2)) / tot).cpu().numpy())
    sx = -torch.as_tensor(cfx, device=DEV).double().reshape(-1)
    sy = -torch.as_tensor(cfy, device=DEV).double().reshape(-1)
    fx, fy = torch.floor(sx), torch.floor(sy)
    wx, wy = (sx - fx)[:, None, None], (sy - fy)[:, None, None]
    ints = torch.arange(det, device=DEV)

    def rolled(ax, ay):
        r = (ints[None] - fx.long()[:, None] - ax) % det
        q = (ints[None] - fy.long()[:, None] - ay) % det
        b = torch.arange(c.shape[0], device=DEV)[:, None, None]
        return c[b, r[:, :, None], q[:, None, :]]

    moved = (rolled(0, 0) * ((1 - wx) * (1 - wy)) + rolled(1, 0) * (wx * (1 - wy))
             + rolled(0, 1) * ((1 - wx) * wy) + rolled(1, 1) * (wx * wy))
    out["amplitudes"] = torch.sqrt(moved.clamp_min(0))
    out["mean"] = float(moved.sum() / c.shape[0])
    m = _Model64(dict(case, T=1, M=1), d)
    overlap = torch.zeros(d["shape"], dtype=torch.float64, device=DEV)
    for s, e in _batches(c.shape[0], 1024):
        w = _shifted(m.probe, m.pos[s:e], torch.complex128)[:, 0]
        overlap += m._scatter(w.abs() ** 2, _indices(m.pos[s:e], det, m.shape))
    out["overlap"] = overlap.cpu().numpy()
    return out


def _exact_conv(case, seed):
    x, weight, bias, dy = _conv_data(case, seed)
    ci, co = case["cin"], case["cout"]
    x64 = x.double().permute(0, 3, 1, 2)
    w64 = weight.double().reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
    d64 = dy.double().permute(0, 3, 1, 2)
    xp = torch.nn.functional.pad(x64, (1, 1, 1, 1))
    dp = torch.nn.functional.pad(d64, (1, 1, 1, 1))
    h, w = x64.shape[-2:]
    y = bias.double()[None, :, None, None].expand(x64.shape[0], co, h, w).clone()
    dx = torch.zeros_like(x64)
    dw = torch.zeros((co, 9, ci), dtype=torch.float64, device=DEV)
    for ky in range(3):
        for kx in range(3):
            part = xp[:, :, ky:ky + h, kx:kx + w]
            y += torch.einsum("nchw,oc->nohw", part, w64[:, :, ky, kx])
            dx += torch.einsum("nohw,oc->nchw", dp[:, :, 2 - ky:2 - ky + h, 2 - kx:2 - kx + w],
                               w64[:, :, ky, kx])
            dw[:, ky * 3 + kx] = torch.einsum("nohw,nchw->oc", d64, part)
    return dict(y=torch.relu(y).permute(0, 2, 3, 1), dx=dx.permute(0, 2, 3, 1), dweight=dw,
                dbias=d64.sum((0, 2, 3)))


_EXACT = dict(gd=_exact_gd, projection=_exact_projection, poscorr=_exact_poscorr,
              gradient=_exact_gradient, volume=_exact_volume, preprocess=_exact_preprocess,
              conv=_exact_conv)
_EXACT["class"] = _exact_class
