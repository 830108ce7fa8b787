"""Performance cases: the calls a user of the library makes, over the sizes they are made at.

    listed()            the cases that are timed every time
    draw(rng)           one more case from the same ranges
    prepare(case, seed) inputs, library contexts and networks, as a program holds them before the call
    run(state)          one pass through the public entry points, and its results
    exact(case, seed)   the same results in 64 bits (plain torch)
    work(case)          bytes and operations of one pass that no implementation can leave out

Kinds of case
    probe   one probe position at a time through the reference's flat calls (OffsetIncomingWave,
            GPUMultislice, GetResult / GetAvgResult), as a caller of the reference drives the library
    scan    many positions x frozen-phonon configurations in one call (JMS_ScanGPU, or
            JMS_ScanGPUDevice on device buffers)
    qep     phase gratings with fresh phonon displacements made on the device (JMS_PgrCalculate into the
            grating store), then the scan of those configurations
    mf      multi-fidelity scan: one full-grid and all coarse-grid configurations (JMS_ScanMultiFidelity)
    train   one training step of the control-variate surrogate (SurrogateNet.train_step)

Specimens are perovskite-like cells of Gaussian atoms displaced by phonon noise, strong enough that the
high-angle detector collects a few percent of the beam; everything is made from the seed alone.
"""
import ctypes as C
import math

import numpy as np
import torch

import jmultislicelib_b200 as jb

GPU = 2
CELL, DZ, KV = 0.3905, 0.19525, 300.0           # cell edge and slice thickness [nm], beam energy [keV]
PHONON = 0.008                                  # displacement per axis [nm]
RINGS = ((0.0, 10.0), (20.0, 50.0), (80.0, 200.0))   # annular detectors [mrad]
# atom sites (type, fx, fy) of the two alternating layers of the cell
LAYERS = (((0, 0.0, 0.0), (2, 0.5, 0.5)), ((1, 0.5, 0.5), (2, 0.5, 0.0), (2, 0.0, 0.5)))
ME0, QEL, HPL, C0 = 9.1093837015e-31, 1.602176634e-19, 6.62607015e-34, 299792458.0
E0 = ME0 * C0 ** 2 / QEL / 1000.0               # electron rest energy [keV]
LAMBDA = C0 * HPL / QEL * 1.0e6 / math.sqrt(KV * (KV + 2 * E0))      # wavelength [nm]
SIGMA = 2 * math.pi * ME0 * (1 + KV / E0) * QEL * LAMBDA * 1e-9 / HPL ** 2 * 1e-9   # rad / (V nm)


def _scan(name, nx, ny, nobj, npos, npass, batch, ntype=4, nvar=4, ndetper=20, bin=0, device=False):
    return {"name": name, "kind": "scan", "nx": nx, "ny": ny, "nobj": nobj, "npos": npos, "npass": npass,
            "batch": batch, "ntype": ntype, "nvar": nvar, "ndetper": ndetper, "bin": bin, "device": device}


def _probe(name, nx, ny, nobj, npos, ndetper, pacbed=False):
    return {"name": name, "kind": "probe", "nx": nx, "ny": ny, "nobj": nobj, "npos": npos, "ntype": 2,
            "ndetper": ndetper, "pacbed": pacbed}


def listed():
    return [
        # the smallest call: one probe of a small simulation cell, detector signals over thickness
        _probe("probe_64", 64, 64, 40, 1, 10),
        # the reference's single-probe benchmark point: 256^2, 100 slices, detectors every 10 slices
        _probe("probe_256", 256, 256, 100, 1, 10),
        # position-averaged patterns and images (PACBED / probe images), position by position
        _probe("pacbed_512", 512, 512, 40, 8, 20, pacbed=True),
        # a small scan with the library's default batch: training pairs, quick looks, low resolution
        _scan("scan_128", 128, 128, 24, 64, 4, 32, ndetper=8),
        # an ordinary scan line: 256^2, configurations of the line in one batch, binned patterns too
        _scan("scan_256", 256, 256, 100, 32, 8, 256, nvar=8, bin=4),
        # the headline: one raster row of the 512^2 STEM scan, 16 configurations, 200 slices
        _scan("scan_512", 512, 512, 200, 64, 16, 1024, nvar=16, bin=4),
        # a specimen that does not fit a square power of two
        _scan("scan_720x384", 720, 384, 60, 24, 2, 64, ntype=2),
        # a wide field of view on device buffers, as a program that keeps its data on the GPU calls it
        _scan("scan_1024", 1024, 1024, 50, 16, 4, 64, ntype=2, ndetper=10, device=True),
        # the largest grid: high-angle scattering needs the reach, few positions fit a study
        _scan("scan_2048", 2048, 2048, 40, 4, 2, 32, ntype=2, nvar=2, ndetper=10),
        # a thin film whose every configuration is drawn afresh on the device
        {"name": "qep_512", "kind": "qep", "nx": 512, "ny": 512, "nobj": 10, "npos": 8, "npass": 8, "batch": 64,
         "ndetper": 5},
        # the control-variate scan of a weak phase object: 512^2 against its 192^2 coarse grid
        {"name": "mf_512_192", "kind": "mf", "nx": 512, "ny": 512, "low": 192, "nobj": 100, "npos": 32, "npass": 8,
         "batch": 256, "ntype": 4, "nvar": 8, "ndetper": 20},
        # one step of the surrogate's training: ten depth bins of 16 x 16 pixels, 30 signals
        {"name": "train_256", "kind": "train", "nbatch": 256, "cin": 10, "size": 16, "nout": 30, "relu": False},
    ]


def _unnamed(case):
    return {k: v for k, v in case.items() if k != "name"}


def draw(rng):
    """One more case: any kind, grid lengths from 48 to 2048 of every radix, specimens of 8 to 200 slices."""
    lengths = (48, 64, 80, 96, 120, 128, 160, 180, 192, 240, 256, 320, 384, 480, 512, 640, 720, 768, 960, 1024, 2048)
    kind = rng.choice(("probe", "probe", "scan", "scan", "scan", "scan", "qep", "mf", "train"))

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(most):
        nx = rng.choice([n for n in lengths if n <= most])
        ny = nx if rng.random() < 0.5 else rng.choice([n for n in lengths if n <= most and nx / 3 <= n <= 3 * nx])
        return nx, ny

    if kind == "probe":
        nx, ny = grid(1024)
        return _unnamed(_probe("", nx, ny, log_int(10, 120), rng.randint(1, 8), rng.choice((5, 10, 20)),
                               rng.random() < 0.3))
    if kind == "train":
        return {"kind": "train", "nbatch": log_int(32, 1024), "cin": rng.randint(3, 12),
                "size": rng.choice((16, 32)), "nout": rng.randint(3, 40), "relu": rng.random() < 0.5}
    if kind == "mf":
        nx = rng.choice((256, 384, 512))
        return {"kind": "mf", "nx": nx, "ny": nx, "low": rng.choice((96, 128, 192)),
                "nobj": log_int(20, 100), "npos": log_int(4, 40), "npass": rng.randint(2, 8), "batch": 256, "ntype": 2,
                "nvar": 4, "ndetper": rng.choice((5, 10, 20))}
    if kind == "qep":
        nx, ny = grid(768)
        return {"kind": "qep", "nx": nx, "ny": ny, "nobj": rng.randint(4, 14),
                "npos": log_int(2, 16), "npass": rng.randint(2, 8), "batch": rng.choice((32, 64, 128)), "ndetper": 5}
    nx, ny = grid(2048)
    npos, npass = log_int(3, 100), rng.randint(1, 8)
    # at most an eighth of the largest listed case
    nobj = log_int(8, 200)
    nobj = max(8, min(nobj, int(6.7e9 / (nx * ny * npos * npass))))
    while nobj * nx * ny * npos * npass > 6.7e9 and npos > 3:
        npos = npos * 2 // 3
    device = rng.random() < 0.3
    return _unnamed(_scan("", nx, ny, nobj, npos, npass, rng.choice((32, 64, 256)), ntype=rng.choice((2, 4)),
                          nvar=rng.randint(1, 4), ndetper=rng.choice((5, 10, 20)),
                          bin=0 if device else rng.choice((0, 2, 4)), device=device))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _freq(n, edge):
    """Spatial frequencies [1/nm] of a scrambled axis: 0, 1, ..., -n/2, ..., -1 over the cell edge."""
    f = np.arange(n)
    return np.where(f < n - n // 2, f, f - n) / edge


def _cells(n):
    return max(1, round(n / 85))


def _atoms(ncx, ncy, layer):
    """[natom, 3]: type, fractional x, y."""
    return np.array([(t, (ix + fx) / ncx, (iy + fy) / ncy) for iy in range(ncy) for ix in range(ncx)
                     for (t, fx, fy) in LAYERS[layer]])


def _atom_params(rng, weak):
    amp = rng.uniform(0.5, 5.0, (3, 2)) * (0.1 if weak else 4.0)      # V nm
    wid = rng.uniform(0.1, 0.4, (3, 2)) * (0.1 if weak else 0.07)     # nm
    return amp, wid


def _gratings(nx, ny, a, b, atoms, shift, amp, wid):
    """complex64 [nvar, ny, nx] host array: exp(i sigma V) of the displaced atoms (shift [nvar, natom, 2] nm)."""
    dev = "cuda"
    t = atoms[:, 0].astype(int)
    ca = torch.tensor(amp[t], dtype=torch.float64, device=dev).reshape(-1, 1)
    cw = torch.tensor(wid[t], dtype=torch.float64, device=dev).reshape(-1, 1)
    x = torch.arange(nx, dtype=torch.float64, device=dev) * (a / nx)
    y = torch.arange(ny, dtype=torch.float64, device=dev) * (b / ny)
    out = np.empty((len(shift), ny, nx), np.complex64)

    def gauss(coord, centre, period):
        d = coord[None, :] - torch.tensor(centre, dtype=torch.float64, device=dev).repeat_interleave(2)[:, None]
        d = torch.remainder(d + 0.5 * period, period) - 0.5 * period
        return torch.exp(-d * d / (2 * cw * cw))

    for v, s in enumerate(shift):
        gx, gy = gauss(x, atoms[:, 1] * a + s[:, 0], a), gauss(y, atoms[:, 2] * b + s[:, 1], b)
        phase = SIGMA * ((gy * ca).T @ gx)
        out[v] = torch.polar(torch.ones_like(phase), phase).to(torch.complex64).cpu().numpy()
    return out


def _optics(nx, ny, a, b, rng):
    """probe, propagator (complex64 [ny, nx]) and annular detectors (float32 [3, ny, nx])."""
    q2 = _freq(nx, a)[None, :] ** 2 + _freq(ny, b)[:, None] ** 2
    q = np.sqrt(q2)
    kmax = min((nx // 2) / a, (ny // 2) / b)
    theta = q * LAMBDA * 1e3                                          # mrad
    alpha = min(22.0, 0.6 * kmax * LAMBDA * 1e3)
    cs, df = 1000.0, float(rng.uniform(-5.0, 5.0))                    # spherical aberration, defocus [nm]
    chi = math.pi * LAMBDA * q2 * df + 0.5 * math.pi * cs * LAMBDA ** 3 * q2 * q2
    probe = np.where(theta <= alpha, np.exp(-1j * chi), 0)
    probe = (probe / np.sqrt((np.abs(probe) ** 2).sum())).astype(np.complex64)
    pro = np.where(q <= 0.6666667 * kmax, np.exp(-1j * math.pi * LAMBDA * DZ * q2) / (nx * ny), 0)
    det = np.stack([((theta >= lo) & (theta < hi)) for lo, hi in RINGS]).astype(np.float32)
    return probe, pro.astype(np.complex64), det


def _inputs(case, seed, grid=None):
    """Everything a pass reads, as host arrays; the same seed on another grid is the same specimen."""
    rng = np.random.default_rng([seed, 1])
    nx, ny = grid or (case["nx"], case["ny"])
    ncx, ncy = _cells(case["nx"]), _cells(case["ny"])
    a, b = ncx * CELL, ncy * CELL
    amp, wid = _atom_params(rng, case["kind"] == "mf")
    probe, pro, det = _optics(nx, ny, a, b, np.random.default_rng([seed, 2]))
    nobj, npos, npass = case["nobj"], case["npos"], case.get("npass", 1)
    p = {"nx": nx, "ny": ny, "a": a, "b": b, "probe": probe, "pro": pro, "det": det, "nobj": nobj}
    # positions: a raster row over the cell in the middle, with the scan's jitter
    line = np.stack([(ncx // 2 + (np.arange(npos) + 0.5) / npos) * CELL,
                     np.full(npos, (ncy // 2 + rng.uniform(0.0, 1.0)) * CELL)], 1)
    p["pos"] = (line + rng.normal(0.0, 0.003, line.shape)).astype(np.float32)
    if case["kind"] == "qep":
        # the generator holds one specimen's elements; only their displacements change from film to film
        amp, wid = _atom_params(np.random.default_rng(5), False)
        p["ntype"], p["nvar"] = nobj, npass
        p["atoms"] = [_atoms(ncx, ncy, s % 2) for s in range(2)]
        p["ff"], p["sk"] = _form_factors(nx, ny, a, b, amp, wid)
        p["seeds"] = [int(k) for k in rng.integers(1, 1 << 40, nobj)]
        p["varseq"] = np.repeat(np.arange(npass, dtype=np.int32)[:, None], nobj, 1)
    else:
        p["ntype"], p["nvar"] = case["ntype"], case.get("nvar", 1)
        p["gratings"] = []
        for s in range(p["ntype"]):
            at = _atoms(ncx, ncy, s % 2)
            p["gratings"].append(_gratings(nx, ny, a, b, at, rng.normal(0.0, PHONON, (p["nvar"], len(at), 2)), amp, wid))
        p["varseq"] = rng.integers(0, p["nvar"], (npass, nobj)).astype(np.int32)
    p["objslc"] = (np.arange(nobj) % p["ntype"]).astype(np.int32)
    return p


def _form_factors(nx, ny, a, b, amp, wid):
    """Radial tables [3, nk] complex64 whose grating phase equals sigma V of the Gaussian atoms."""
    nk = 12 * max(nx, ny)
    sk = float(np.float32(max(nx / a, ny / b) / nk))
    q = np.arange(nk) * sk
    k = 4 * math.pi * SIGMA / LAMBDA
    ff = [k * sum(amp[t, i] * 2 * math.pi * wid[t, i] ** 2 * np.exp(-2 * (math.pi * wid[t, i] * q) ** 2)
                  for i in range(2)) for t in range(3)]
    return np.asarray(ff).astype(np.complex64), sk


def _planes(ndetper, nobj):
    """Readout plane index of each of the nobj + 1 planes (entrance, every ndetper slices, exit), or -1."""
    marks = sorted(set(range(0, nobj + 1, ndetper)) | {nobj})
    return {p: k for k, p in enumerate(marks)}


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------
class _Context:
    """A library context with its setup, freed with the object."""

    def __init__(self, p, ndetper, imagedet, batch=None, stream=None):
        self.J = jb.JMS()
        self.L = self.J.L
        self.id = self.L.JMS_CreateContext()
        J = self.select()
        if stream is not None:
            J.set_stream(stream.cuda_stream)
        J.set_high_tension(KV)
        J.set_grid(p["nx"], p["ny"], p["a"], p["b"], DZ)
        e = J.setup(GPU, [p["nvar"]] * p["ntype"], p["objslc"], [0] * p["ntype"], ndetper, len(RINGS), imagedet)
        for s, g in enumerate(p.get("gratings", ())):
            e.append(J.set_phase_grating(GPU, s, g))
        e.append(J.set_propagator(GPU, 0, p["pro"]))
        for k in range(len(RINGS)):
            e.append(J.set_detector(GPU, k, p["det"][k]))
        e += [J.init_core(GPU), J.set_incident_wave(GPU, p["probe"])]
        if batch:
            e.append(self.L.JMS_SetScanBatch(batch))
        _ok(*e)

    def select(self):
        self.L.JMS_SelectContext(self.id)
        return self.J

    def __del__(self):
        try:
            self.L.JMS_SelectContext(0)
            self.L.JMS_DestroyContext(self.id)
        except Exception:
            pass


_streams = []


def _work_stream():
    """The program's one stream for generating gratings and scanning them (the generator is one per process)."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _ok(*codes):
    if any(codes):
        raise RuntimeError(f"the library returned {codes}")


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "train":
        from jmultislicelib_b200.surrogate import SurrogateNet

        g = torch.Generator(device="cuda").manual_seed(int(seed))
        shape = (case["nbatch"], case["cin"], case["size"], case["size"])
        s["net"] = SurrogateNet(case["nout"], case["nbatch"], seed=int(seed) % (1 << 31), cin=case["cin"],
                                size=case["size"], relu=case["relu"])
        s["x"] = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
        s["t"] = torch.randn((case["nbatch"], case["nout"]), generator=g, device="cuda")
        return s
    p = _inputs(case, seed)
    s["p"] = {k: p[k] for k in ("nx", "ny", "pos", "varseq")}
    nd = len(_planes(case["ndetper"], case["nobj"]))
    s["nd"] = nd
    if kind == "probe":
        # integrated detectors; with pacbed also the position-averaged images and diffraction patterns
        s["ctx"] = _Context(p, case["ndetper"], 1 | 32 | 64 if case["pacbed"] else 1)
    elif kind == "mf":
        low = _inputs(case, seed, (case["low"], case["low"]))
        s["low"] = _Context(low, case["ndetper"], 1, case["batch"])
        s["ctx"] = _Context(p, case["ndetper"], 1, case["batch"])
    elif kind == "qep":
        s["ctx"] = _Context(p, case["ndetper"], 1, case["batch"], _work_stream())
        J = s["ctx"].select()
        J.pgr_set_stream(_work_stream().cuda_stream)
        _ok(J.pgr_setup(p["nx"], p["ny"], p["a"], p["b"], KV, 2),
            J.pgr_set_form_factors(p["ff"], p["sk"], [8 * math.pi ** 2 * PHONON ** 2] * 3))
        s["seeds"] = p["seeds"]
        # atoms [natom, 5] of the two layers: fractional x, y, z, occupancy, type
        s["atoms"] = [np.column_stack([t[:, 1], t[:, 2], np.zeros(len(t)), np.ones(len(t)), t[:, 0]])
                      .astype(np.float32) for t in p["atoms"]]
    elif case["device"]:
        s["stream"] = torch.cuda.Stream()
        s["ctx"] = _Context(p, case["ndetper"], 1, case["batch"], s["stream"])
        s["d_pos"] = torch.from_numpy(p["pos"]).cuda()
    else:
        s["ctx"] = _Context(p, case["ndetper"], 1, case["batch"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        net = s["net"]
        loss = net.train_step(s["x"], s["t"], case["nbatch"], 2e-3)
        return {"loss": loss, "grads": list(net.grads), "params": list(net.params)}
    J, p = s["ctx"].select(), s["p"]
    nd, npos, npass = s["nd"], case["npos"], case.get("npass", 1)
    if kind == "probe":
        if case["pacbed"]:
            J.L.ResetImageAveraging(GPU, 0)
        sig = []
        for dx, dy in p["pos"]:
            _ok(J.offset(GPU, float(dx), float(dy)), J.gpu_multislice(0, 0, 1.0 / npos if case["pacbed"] else 1.0))
            sig.append(J.get_result(GPU, 1, nd * len(RINGS)))
        out = {"signals": np.stack(sig)}
        if case["pacbed"]:
            n = nd * p["nx"] * p["ny"]
            out["image"], _ = J.get_avg_result(GPU, 32, n)
            out["pattern"], _ = J.get_avg_result(GPU, 64, n)
        return out
    if kind == "mf":
        pos, var = p["pos"], p["varseq"]
        out = np.zeros((npos, nd, len(RINGS)), np.float32)
        _ok(J.L.JMS_ScanMultiFidelity(s["ctx"].id, s["low"].id, npos, pos.ctypes.data_as(C.POINTER(C.c_float)), 0.0,
                                      npass, var.ctypes.data_as(C.POINTER(C.c_int)),
                                      out.ctypes.data_as(C.POINTER(C.c_float))))
        return out
    if kind == "qep":
        for j in range(case["nobj"]):
            e, _ = J.pgr_calculate(s["atoms"][j % 2], DZ, ngr=npass, seed=s["seeds"][j], islc=j, ivar0=0, want=False)
            _ok(e)
        e, sig, _ = J.scan(p["pos"], npass, varseq=p["varseq"])
        _ok(e)
        return sig
    if case["device"]:
        with torch.cuda.stream(s["stream"]):
            out = torch.zeros((npos, nd, len(RINGS)), dtype=torch.float64, device="cuda")
            _ok(J.L.JMS_ScanGPUDevice(npos, s["d_pos"].data_ptr(), 0.0, npass,
                                      p["varseq"].ctypes.data_as(C.POINTER(C.c_int)), out.data_ptr(), None, 0))
        return out
    e, sig, pat = J.scan(p["pos"], npass, varseq=p["varseq"], bin=case["bin"])
    _ok(e)
    return {"signals": sig, "pattern": pat} if case["bin"] else sig


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------
def _multislice64(p, gratings, ndetper, varseq, bin=0, images=False):
    """Frozen-phonon averages over varseq [npass, nobj] for every position, in complex128: integrated signals
    [npos, nd, ndet]; with bin the exit pattern [npos, ny / bin, nx / bin]; with images the images and patterns
    of every plane summed over the positions."""
    c128, dev = torch.complex128, "cuda"
    nx, ny, nobj = p["nx"], p["ny"], p["nobj"]
    N, plane = nx * ny, _planes(ndetper, p["nobj"])
    probe, pro = (torch.from_numpy(p[k]).to(dev, c128) for k in ("probe", "pro"))
    det = torch.from_numpy(p["det"]).to(dev, torch.float64).reshape(len(RINGS), N)
    t = [g.to(dev) if torch.is_tensor(g) else torch.from_numpy(g).to(dev) for g in gratings]
    fx = torch.from_numpy(_freq(nx, p["a"])).to(dev)
    fy = torch.from_numpy(_freq(ny, p["b"])).to(dev)
    pos = torch.from_numpy(p["pos"].astype(np.float64)).to(dev)
    npos, npass, nd = len(pos), len(varseq), len(plane)
    sig = torch.zeros((npos, nd, len(RINGS)), dtype=torch.float64, device=dev)
    pat = torch.zeros((npos, ny // bin, nx // bin), dtype=torch.float64, device=dev) if bin else None
    img, dif = (torch.zeros((nd, ny, nx), dtype=torch.float64, device=dev) for _ in range(2)) if images else (None, None)
    group = max(1, (1 << 24) // N)
    for i in range(0, npos, group):
        k = slice(i, min(npos, i + group))
        ramp = torch.exp(-2j * math.pi * pos[k, 1].reshape(-1, 1, 1) * fy.reshape(1, -1, 1)) * \
            torch.exp(-2j * math.pi * pos[k, 0].reshape(-1, 1, 1) * fx.reshape(1, 1, -1))
        for var in varseq:
            psi = probe * ramp
            for j in range(nobj + 1):
                at = plane.get(j)
                if at is not None:
                    w = psi.real ** 2 + psi.imag ** 2
                    sig[k, at] += w.reshape(len(w), N) @ det.T
                    if images:
                        dif[at] += w.sum(0)
                        r = torch.fft.ifft2(psi, norm="forward")
                        img[at] += (r.real ** 2 + r.imag ** 2).sum(0)
                if j == nobj:
                    break
                psi = torch.fft.ifft2(psi, norm="forward")
                psi *= t[p["objslc"][j]][int(var[j])]
                psi = torch.fft.fft2(psi)
                psi *= pro
            if bin:
                u = torch.roll(psi.real ** 2 + psi.imag ** 2, (ny // 2, nx // 2), (1, 2))
                pat[k] += u.reshape(len(u), ny // bin, bin, nx // bin, bin).sum((2, 4))
    return sig / npass, pat / npass if bin else None, img, dif


def _mix64(seed, k):
    """Outputs k of the SplitMix64 stream of seed."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + k.astype(np.uint64) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _qep_gratings64(p, j):
    """complex128 [npass, ny, nx]: gratings of object slice j with the generator's displacement stream."""
    dev, nx, ny, a, b = "cuda", p["nx"], p["ny"], float(np.float32(p["a"])), float(np.float32(p["b"]))
    at = p["atoms"][j % 2].astype(np.float32)
    n, ngr = len(at), p["nvar"]
    c = np.arange(n * ngr)
    u1 = ((_mix64(p["seeds"][j], 2 * c + 1) >> np.uint64(11)) + np.uint64(1)).astype(np.float64) * 2.0 ** -53
    u2 = (_mix64(p["seeds"][j], 2 * c + 2) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
    u = math.sqrt(float(np.float32(8 * math.pi ** 2 * PHONON ** 2))) / math.sqrt(8 * math.pi ** 2)
    r = np.sqrt(-2 * np.log(u1))
    x = at[:, 1].astype(np.float64) + (u / a * r * np.cos(2 * math.pi * u2)).reshape(ngr, n)
    y = at[:, 2].astype(np.float64) + (u / b * r * np.sin(2 * math.pi * u2)).reshape(ngr, n)
    ix, iy = _freq(nx, 1.0), _freq(ny, 1.0)
    qx, qy = (ix / a)[None, :], (iy / b)[:, None]
    at_q = np.sqrt(qx * qx + qy * qy) / p["sk"]
    i0 = np.minimum(at_q.astype(np.int64), p["ff"].shape[1] - 2)
    w = at_q - i0
    pot = torch.zeros((ngr, ny, nx), dtype=torch.complex128, device=dev)
    for t in range(3):
        mine = np.nonzero(at[:, 0] == t)[0]
        if len(mine) == 0:
            continue
        f = p["ff"][t].astype(np.complex128)
        f = torch.from_numpy(f[i0] * (1 - w) + f[i0 + 1] * w).to(dev)
        ex = torch.exp(-2j * math.pi * torch.from_numpy(x[:, mine, None] * ix).to(dev))
        ey = torch.exp(-2j * math.pi * torch.from_numpy(y[:, mine, None] * iy).to(dev))
        pot += f * (ey.transpose(1, 2) @ ex)
    v = torch.fft.ifft2(pot, norm="forward") * (LAMBDA / (4 * math.pi * a * b))
    g = torch.exp(1j * v)
    # 2/3 band limit in the 32-bit arithmetic that defines it
    f32 = np.float32
    q = np.sqrt((ix.astype(f32) * (f32(1) / f32(a)))[None, :] ** 2 + (iy.astype(f32) * (f32(1) / f32(b)))[:, None] ** 2)
    kmax = min(f32(nx // 2) * (f32(1) / f32(a)), f32(ny // 2) * (f32(1) / f32(b)))
    return torch.fft.ifft2(torch.fft.fft2(g) * torch.from_numpy((q <= kmax * f32(0.6666667)).astype(np.float64)).to(dev))


def _train64(case, seed):
    """One training step in 64 bits, with weights and activations rounded to the BF16 they are stored in."""
    s = prepare(case, seed)
    net = s["net"]
    P = [q.detach().double() for q in net.params]
    nl, B = len(net.conv), case["nbatch"]
    w16 = [P[2 * k].to(torch.bfloat16).double().requires_grad_() for k in range(nl)]
    bias = [P[2 * k + 1].clone().requires_grad_() for k in range(nl)]
    wl, bl = P[-2].clone().requires_grad_(), P[-1].clone().requires_grad_()
    h = s["x"].double()
    for k in range(nl):
        h = torch.nn.functional.conv2d(h, w16[k], bias[k], stride=2, padding=1)
        h = torch.relu(h) if case["relu"] else h
        h = h + (h.detach().to(torch.bfloat16).double() - h.detach())
    out = h.mean((2, 3)) @ wl.T + bl
    loss = ((out - s["t"].double()) ** 2).sum() / (B * case["nout"])
    leaf = [v for k in range(nl) for v in (w16[k], bias[k])] + [wl, bl]
    grads = torch.autograd.grad(loss, leaf)
    b1, b2, lr, eps = (float(np.float32(v)) for v in (0.9, 0.999, 2e-3, 1e-8))
    new = []
    for q, g in zip(P, grads):
        m, v = (1 - b1) * g, (1 - b2) * g * g
        new.append(q - lr * (m / (1 - b1)) / (torch.sqrt(v / (1 - b2)) + eps))
    return {"loss": loss.detach().reshape(1), "grads": list(grads), "params": new}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train64(case, seed)
    p = _inputs(case, seed)
    if kind == "qep":
        gr = [_qep_gratings64(p, j) for j in range(case["nobj"])]
        return _multislice64(p, gr, case["ndetper"], p["varseq"])[0]
    if kind == "mf":
        low = _inputs(case, seed, (case["low"], case["low"]))
        f = _multislice64(p, p["gratings"], case["ndetper"], p["varseq"][:1])[0]
        g1 = _multislice64(low, low["gratings"], case["ndetper"], p["varseq"][:1])[0]
        gm = _multislice64(low, low["gratings"], case["ndetper"], p["varseq"])[0]
        return f - (g1 - gm)
    if kind == "probe":
        sig, _, img, dif = _multislice64(p, p["gratings"], case["ndetper"], p["varseq"], images=case["pacbed"])
        w = 1.0 / case["npos"] if case["pacbed"] else 1.0
        out = {"signals": sig.reshape(case["npos"], -1) * w}
        if case["pacbed"]:
            out["image"], out["pattern"] = img.reshape(-1) * w, dif.reshape(-1) * w
        return out
    sig, pat, _, _ = _multislice64(p, p["gratings"], case["ndetper"], p["varseq"], bin=case["bin"])
    return {"signals": sig, "pattern": pat} if case["bin"] else sig


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _scan_work(nx, ny, nobj, nwave, ngrating, nd, npos):
    """Operands once (gratings, propagator, detectors, probe), results once; per wave and slice a forward and an
    inverse 2-D transform and two complex products."""
    N = nx * ny
    return {"bytes": 8.0 * N * (ngrating + 2) + 4.0 * N * len(RINGS) + npos * (8.0 + 4.0 * nd * len(RINGS)),
            "flops": nwave * (nobj * N * (10.0 * math.log2(N) + 12.0) + nd * N * (3.0 + 2.0 * len(RINGS)))}


def work(case):
    kind = case["kind"]
    if kind == "train":
        h, macs, params = case["size"], 0, 0
        conv = ((case["cin"], 16), (16, 32), (32, 64), (64, 64))
        for ci, co in conv:
            h //= 2
            macs += case["nbatch"] * h * h * co * ci * 9
            params += co * (ci * 9 + 1)
        macs += case["nbatch"] * 64 * case["nout"]
        params += case["nout"] * 65
        x = case["nbatch"] * (2 * case["cin"] * case["size"] ** 2 + 4 * case["nout"])
        return {"bytes": float(x + params * 4 * 7), "flops": 6.0 * macs}
    nx, ny, nobj, npos, npass = case["nx"], case["ny"], case["nobj"], case["npos"], case.get("npass", 1)
    nd, N = len(_planes(case["ndetper"], nobj)), nx * ny
    if kind == "mf":
        used = min(case["ntype"], nobj)
        full = _scan_work(nx, ny, nobj, npos, used, nd, npos)
        low = _scan_work(case["low"], case["low"], nobj, npos * npass, used * min(case["nvar"], npass), nd, npos)
        return {k: full[k] + low[k] for k in full}
    if kind == "qep":
        w = _scan_work(nx, ny, nobj, npos * npass, 0, nd, npos)
        natom = _cells(nx) * _cells(ny) * 2.5
        # per grating: the Hermitian half of the structure factor, three transforms and the phase
        w["flops"] += nobj * npass * N * (4.0 * natom + 15.0 * math.log2(N) + 20.0)
        w["bytes"] += 8.0 * N * nobj * npass
        return w
    used = sum(min(case.get("nvar", 1), npass * (nobj // case["ntype"])) for _ in range(min(case["ntype"], nobj)))
    w = _scan_work(nx, ny, nobj, npos * npass, used, nd, npos)
    if case.get("bin"):
        w["bytes"] += 4.0 * npos * (nx // case["bin"]) * (ny // case["bin"])
    if case.get("pacbed"):
        w["bytes"] += 8.0 * N * nd
        w["flops"] += npos * nd * N * 10.0
    return w
