"""Performance cases of polybin3d_b200: what its users run, through its public entry points.

A case is a plain dict.  `kind` says which call is made; the other keys are its sizes and options:

  n0, n1, n2   grid (n2 even);  cell: grid spacing in Mpc/h, so boxes are n * cell
  lmax, nk     largest multipole and number of linear k-bins from the fundamental mode to
  frac         this fraction of the Nyquist frequency
  precision    'fp64' or 'mixed';  window: pixel window;  weight: 1/P_fid weighting or none
  mask         'none', 'sector' (a shell sector with holes: most of the box is empty) or
               'survey' (a ball with holes and varying completeness: most of the box is observed)
  sims         simulations of the linear term, or Monte Carlo realisations

kinds:
  pk           PSpec.Pk_ideal of a periodic box (simulation snapshots, one call per field)
  pk_masked    PSpec.Pk_numerator of a masked field, global or local sightline (survey data)
  bk           BSpec.Bk_ideal of a periodic box with the ideal Fisher matrix in hand
  bk_linear    BSpec.Bk_numerator of a masked field with the linear term's simulations loaded
  bk_setup     BSpec.compute_fisher_ideal for a new binning or fiducial spectrum
  fisher_pk    PSpec.compute_fisher with device noise (the unwindowed estimator's normalisation)
  fisher_bk    BSpec.compute_fisher with device noise
  pk_grad      power-spectrum numerator and its gradient (field-level inference, forward + backward)
  bk_grad      bispectrum numerator and its gradient

Fields of precision='mixed' are float32, and so are the spectra kept from them.
"""
import numpy as np
import torch

import polybin3d_b200 as pb
from polybin3d_b200.autograd import bk_numerator, pk_numerator

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _case(kind, n, **kw):
    c = {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "cell": 8.0, "lmax": 0, "nk": 10, "frac": 0.6,
         "precision": "fp64", "window": "none", "weight": False, "mask": "none", "local": False, "sims": 0}
    c.update(kw)
    return c


def listed():
    def named(name, *a, **kw):
        return dict(_case(*a, **kw), name=name)
    return [
        # one small snapshot after another: the smallest calls, bound by launches and latency
        named("pk_64", "pk", (64, 64, 64), cell=15.625, lmax=2, nk=10, frac=0.65),
        named("bk_64", "bk", (64, 64, 64), cell=15.625, lmax=0, nk=10, frac=0.65),
        # the largest grid a power spectrum is taken on, single precision
        named("pk_512", "pk", (512, 512, 512), lmax=4, nk=40, frac=0.9, precision="mixed"),
        # survey data about a varying line of sight, on a grid with an odd axis
        named("pk_local_150", "pk_masked", (150, 135, 144), cell=10.0, lmax=2, nk=20, frac=0.8, mask="survey",
              local=True),
        # the bispectrum of a large snapshot: 16 bins, quadrupoles, TSC window, split-precision contraction
        named("bk_256", "bk", (256, 256, 256), cell=7.8125, lmax=2, nk=16, frac=0.497, precision="mixed",
              window="tsc"),
        # double precision on an anisotropic grid
        named("bk_fp64_ragged", "bk", (120, 144, 100), cell=10.0, lmax=2, nk=9, frac=0.55, weight=True),
        # survey bispectrum: cubic and linear terms
        named("bk_linear_128", "bk_linear", (128, 128, 128), cell=11.71875, lmax=2, nk=10, frac=0.6,
              precision="mixed", window="tsc", mask="survey", sims=4),
        # a new binning: the ideal normalisation from scratch
        named("bk_setup_128", "bk_setup", (128, 128, 128), cell=11.71875, lmax=2, nk=12, frac=0.6, weight=True),
        # Monte Carlo Fisher matrices on a survey sector: 60 and 203 bins
        named("fisher_pk_128", "fisher_pk", (128, 128, 128), cell=11.71875, lmax=4, nk=20, frac=0.932, mask="sector",
              sims=8),
        named("fisher_bk_128", "fisher_bk", (128, 128, 128), cell=11.71875, lmax=0, nk=12, frac=0.746, mask="sector",
              sims=2),
        # gradients with respect to the field: small double precision, large single precision
        named("pk_grad_128", "pk_grad", (128, 128, 128), cell=11.71875, lmax=4, nk=20, frac=0.8, mask="survey"),
        named("bk_grad_256", "bk_grad", (256, 256, 256), cell=7.8125, lmax=2, nk=16, frac=0.497, precision="mixed",
              window="tsc"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))

    def grid(lo, hi, odd=False):
        n = size(lo, hi)
        ax = [max(lo, int(round(n * rng.uniform(0.8, 1.0)))) for _ in range(3)]
        if rng.random() < 0.4:
            ax = [n, n, n]
        return [a if odd and i < 2 else 2 * ((a + 1) // 2) for i, a in enumerate(ax)]

    kind = rng.choice(["pk", "pk", "pk_masked", "bk", "bk", "bk_linear", "bk_setup", "fisher_pk", "fisher_pk",
                       "fisher_bk", "pk_grad", "bk_grad"])
    precision = rng.choice(["fp64", "mixed"])
    window = rng.choice(["none", "tsc", "cic"])
    mask = rng.choice(["sector", "survey"])
    cell = round(rng.uniform(6.0, 16.0), 3)
    c = _drawn(rng, kind, grid, precision, window, mask, cell)
    # bins at least two fundamental modes wide: every bin holds modes and triangles
    c["nk"] = max(3, min(c["nk"], int((0.5 * c["frac"] * min(_dims(c)) - 1) / 2)))
    return c


def _drawn(rng, kind, grid, precision, window, mask, cell):
    if kind == "pk":
        n = grid(48, 384, odd=True)
        return _case(kind, n, cell=cell, lmax=rng.choice([0, 2, 4]), nk=rng.randint(5, 40), precision=precision,
                     frac=round(rng.uniform(0.4, 0.95), 3), window="none" if max(n) > 200 else window)
    if kind == "pk_masked":
        return _case(kind, grid(48, 160, odd=True), cell=cell, lmax=rng.choice([2, 4]), nk=rng.randint(5, 30),
                     frac=round(rng.uniform(0.4, 0.95), 3), window=window, mask=mask, local=rng.random() < 0.6)
    if kind == "bk":
        big = precision == "mixed"
        return _case(kind, grid(48, 256 if big else 160), cell=cell, lmax=rng.choice([0, 2]),
                     nk=rng.randint(6, 16 if big else 10), frac=round(rng.uniform(0.4, 0.62), 3),
                     precision=precision, window=window, weight=rng.random() < 0.3)
    if kind == "bk_linear":
        return _case(kind, grid(48, 128), cell=cell, lmax=rng.choice([0, 2]), nk=rng.randint(6, 10),
                     frac=round(rng.uniform(0.4, 0.62), 3), precision=precision, window=window, mask=mask,
                     sims=rng.randint(1, 5))
    if kind == "bk_setup":
        return _case(kind, grid(48, 144), cell=cell, lmax=rng.choice([0, 2]), nk=rng.randint(6, 12),
                     frac=round(rng.uniform(0.4, 0.62), 3), weight=True)
    if kind == "fisher_pk":
        return _case(kind, grid(48, 128, odd=rng.random() < 0.3), cell=cell, lmax=rng.choice([0, 2, 4]),
                     nk=rng.randint(6, 20), frac=round(rng.uniform(0.5, 0.95), 3), mask=mask, window=window,
                     sims=rng.randint(4, 8))
    if kind == "fisher_bk":
        return _case(kind, grid(48, 112), cell=cell, lmax=0, nk=rng.randint(6, 10),
                     frac=round(rng.uniform(0.5, 0.9), 3), mask=mask, window=window, sims=rng.randint(1, 2))
    if kind == "pk_grad":
        return _case(kind, grid(48, 192, odd=rng.random() < 0.3), cell=cell, lmax=rng.choice([0, 2, 4]),
                     nk=rng.randint(6, 30), frac=round(rng.uniform(0.4, 0.95), 3), mask=mask, window=window)
    return _case(kind, grid(64, 224), cell=cell, lmax=rng.choice([0, 2]), nk=rng.randint(6, 14),
                 frac=round(rng.uniform(0.4, 0.62), 3), precision=precision if rng.random() < 0.3 else "mixed",
                 window=window)


# --------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------
def _dims(c):
    return (c["n0"], c["n1"], c["n2"])


def _box(c):
    return np.asarray(_dims(c), dtype=np.float64) * c["cell"]


def _edges(c):
    kf = 2.0 * np.pi / _box(c)
    return np.linspace(np.max(kf), c["frac"] * np.pi / c["cell"], c["nk"] + 1)


def _centre(c):
    """Box centre of a survey seen from the origin (local sightline)."""
    return _box(c) * np.asarray([0.9, 0.7, 1.3]) if c["local"] else None


def _kgrids(c):
    """k-grids of the half spectrum, |k| and mode multiplicity (host, double precision)."""
    n, kf = _dims(c), 2.0 * np.pi / _box(c)
    ka = [np.fft.fftshift(np.arange(-n[i] // 2, n[i] // 2)) * kf[i] for i in range(2)]
    kx, ky, kz = np.meshgrid(ka[0], ka[1], np.arange(n[2] // 2 + 1) * kf[2], indexing="ij")
    return (kx, ky, kz), np.sqrt(kx ** 2 + ky ** 2 + kz ** 2), 1.0 + (kz > 0)


def _pk_table(c, seed):
    """Fiducial spectrum [k, P] when the case weights by it: a power law whose slope varies with the seed."""
    if not c["weight"]:
        return None
    k = np.linspace(0.0, 2.0 * np.pi / c["cell"], 2000)
    tilt = 0.1 * np.random.default_rng(seed).uniform(-1.0, 1.0)
    return np.asarray([k, 1e4 / (1.0 + (k / 0.05) ** (1.4 + tilt))])


def _fields(c, seed, count=1):
    """Lognormal fields of zero mean with a decaying spectrum, drawn on the device."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    n = _dims(c)
    k2 = 0
    for i in range(3):
        f = torch.fft.rfftfreq(n[i], device=DEV) if i == 2 else torch.fft.fftfreq(n[i], device=DEV)
        k2 = k2 + (2 * np.pi * f / c["cell"]).square().reshape([-1 if j == i else 1 for j in range(3)])
    amp = (1.0 + k2 / 0.05 ** 2) ** -0.4
    out = []
    for _ in range(count):
        d = torch.fft.irfftn(torch.fft.rfftn(torch.randn(n, generator=g, device=DEV)) * amp, s=n)
        d = 0.5 * d / d.std()
        d = torch.exp(d)
        out.append((d / d.mean() - 1.0).to(torch.float32 if c["precision"] == "mixed" else torch.float64))
    return out


def _mask(c, seed):
    """Survey mask (device, float32 values): see the head of this file; holes and completeness from the seed."""
    if c["mask"] == "none":
        return None
    n, box = _dims(c), _box(c)
    rng = np.random.default_rng(seed)
    ax = [torch.as_tensor((((np.arange(n[i]) + n[i] // 2) % n[i]) - n[i] // 2) * c["cell"], device=DEV).reshape(
        [-1 if j == i else 1 for j in range(3)]) for i in range(3)]
    r2 = ax[0] ** 2 + ax[1] ** 2 + ax[2] ** 2
    half = 0.5 * float(box.min())
    if c["mask"] == "sector":
        m = (r2 > (0.33 * half) ** 2) & (r2 < (0.93 * half) ** 2) & (ax[0] > 0) & (ax[1] > 0) & (ax[2] > 0)
    else:
        m = r2 < (0.95 * half) ** 2
    for _ in range(60):
        p, rad = rng.uniform(-half, half, 3), rng.uniform(0.01, 0.03) * 2 * half
        if c["mask"] == "sector":
            p = np.abs(p)
        m &= sum((ax[i] - p[i]) ** 2 for i in range(3)) > rad ** 2
    m = m.to(torch.float64)
    if c["mask"] == "survey":
        ph = rng.uniform(0, 2 * np.pi, 3)
        for i in range(3):
            m = m * (1.0 - 0.1 * (1.0 + torch.sin(6.0 * ax[i] / half + ph[i])))
    return m.to(torch.float32).contiguous()


def _cotangent(n, seed):
    return torch.as_tensor(np.random.default_rng(seed + 77).standard_normal(n), device=DEV)


def prepare(c, seed):
    kw = {} if c["kind"].startswith("fisher") else {"precision": c["precision"]}
    centre = _centre(c)
    base = pb.PolyBin3D(_box(c), _dims(c), Pk=_pk_table(c, seed), boxcenter=centre, pixel_window=c["window"],
                        sightline="local" if c["local"] else "global", verb=False, **kw)
    m = _mask(c, seed)
    mask = None if m is None else m.cpu().numpy()
    s = {"c": c, "base": base}
    if c["kind"] == "bk_setup":
        return s
    if c["kind"] in ("pk", "pk_masked", "fisher_pk", "pk_grad"):
        s["est"] = est = pb.PSpec(base, _edges(c), lmax=c["lmax"], mask=mask, verb=False)
    else:
        s["est"] = est = pb.BSpec(base, _edges(c), lmax=c["lmax"], mask=mask, Pk_fid="default", verb=False)
    if c["kind"].startswith("fisher"):
        return s
    fields = _fields(c, seed, 1 + c["sims"])
    if m is not None and not c["kind"].endswith("grad"):
        fields = [f * m.to(f.dtype) for f in fields]
    s["data"] = fields[0]
    if c["kind"] in ("pk", "bk"):
        est.compute_fisher_ideal()
    elif c["kind"] == "bk_linear":
        est.load_sims(lambda i: fields[1 + i], c["sims"])
        est._compute_symmetry_factor()
    elif c["kind"].endswith("grad"):
        if c["kind"] == "bk_grad":
            est._compute_symmetry_factor()
        s["v"] = _cotangent(est.N_bins, seed)
    return s


def _kept(c, x):
    """Spectra of float32 fields are kept in float32."""
    if isinstance(x, dict):
        return {k: _kept(c, v) for k, v in x.items()}
    if c["precision"] == "fp64":
        return x
    return x.to(torch.float32) if isinstance(x, torch.Tensor) else x.astype(np.float32)


def run(s):
    c, kind = s["c"], s["c"]["kind"]
    if kind == "pk":
        return _kept(c, s["est"].Pk_ideal(s["data"]))
    if kind == "pk_masked":
        return s["est"].Pk_numerator(s["data"])
    if kind == "bk":
        return _kept(c, s["est"].Bk_ideal(s["data"]))
    if kind == "bk_linear":
        return _kept(c, s["est"].Bk_numerator(s["data"]))
    if kind == "bk_setup":
        est = pb.BSpec(s["base"], _edges(c), lmax=c["lmax"], Pk_fid="default", verb=False)
        fish = est.compute_fisher_ideal()
        return {"fish": fish, "sym": est.sym_factor}
    if kind == "fisher_pk":
        return s["est"].compute_fisher(c["sims"], batch=min(8, c["sims"]), noise="philox")
    if kind == "fisher_bk":
        return s["est"].compute_fisher(c["sims"], noise="philox")
    d = s["data"].detach().requires_grad_(True)
    num = (pk_numerator if kind == "pk_grad" else bk_numerator)(s["est"], d)
    (grad,) = torch.autograd.grad(num, d, grad_outputs=s["v"])
    return {"num": _kept(c, num.detach()), "grad": grad}


def _triplets(c):
    """(b1, b2, b3) of the triangle bins whose centres satisfy the triangle condition, b1 <= b2 <= b3."""
    k = _edges(c)
    k = 0.5 * (k[1:] + k[:-1])
    r = range(len(k))
    return [(a, b, d) for a in r for b in r if b >= a for d in r if d >= b and not (k[d] < abs(k[a] - k[b]) or
                                                                               k[d] > k[a] + k[b])]


def work(c):
    """Bytes: the inputs read once and the outputs written once.  Operations: the real 3D transforms
    of the fields and of the maps (2.5 V log2 V each), the products and sums of the triangle bins on
    the smallest alias-free grid, and the binning of each spectrum once."""
    V = float(np.prod(_dims(c)))
    esz = 4 if c["precision"] == "mixed" else 8
    nl = c["lmax"] // 2 + 1
    fft = 2.5 * V * np.log2(V)
    trip = len(_triplets(c)) if c["kind"].startswith(("bk", "fisher_bk")) else 0
    nb = trip * nl if trip else c["nk"] * nl
    Vm = float(np.prod([min(n, 1.5 * c["frac"] * n) for n in _dims(c)]))
    maps = c["nk"] * nl
    cubic = maps * 2.5 * Vm * np.log2(Vm) + 2.0 * trip * nl * Vm
    kind = c["kind"]
    if kind == "pk":
        return {"bytes": V * esz + nb * 8, "flops": fft + 4 * V * nl}
    if kind == "pk_masked":
        extra = sum(2 * l + 1 for l in range(2, c["lmax"] + 1, 2)) if c["local"] else 0
        return {"bytes": V * esz + nb * 8, "flops": (1 + extra) * fft + 4 * V * nl}
    if kind == "bk":
        return {"bytes": V * esz + nb * 8, "flops": fft + cubic}
    if kind == "bk_linear":
        return {"bytes": V * esz * (1 + c["sims"]) + nb * 8, "flops": fft + (1 + c["sims"]) * cubic +
                4.0 * c["sims"] * trip * nl * Vm}
    if kind == "bk_setup":
        return {"bytes": V * 4 + nb * nb * 8.0, "flops": (maps * (1 + 5 * (c["lmax"] > 0))) * 2.5 * Vm * np.log2(Vm) +
                4.0 * trip * nl * (nl + 1) * Vm}
    if kind == "fisher_pk":
        return {"bytes": V * 8 + nb * nb * 8.0, "flops": c["sims"] * ((2 + 2 * nb) * fft + 4.0 * nb * V)}
    if kind == "fisher_bk":
        pairs = c["nk"] * (c["nk"] + 1) // 2
        return {"bytes": V * 8 + nb * nb * 8.0, "flops": c["sims"] * ((4 + 4 * c["nk"] + 2 * pairs + 2 * nb) * fft +
                                                                   8.0 * nb * nb / c["nk"] * V / 2)}
    if kind == "pk_grad":
        return {"bytes": V * esz * 2 + nb * 8, "flops": 3 * fft + 8 * V * nl}
    return {"bytes": V * esz * 2 + nb * 8, "flops": 3 * fft + 2 * cubic + 4.0 * trip * nl * Vm}


# --------------------------------------------------------------------------------------
# the same results in 64 bits, with torch alone
# --------------------------------------------------------------------------------------
class _Exact:
    """Grids of a case as double-precision tensors, its filters and the sums over them."""

    def __init__(self, c, seed):
        self.c, self.n, self.box = c, _dims(c), _box(c)
        self.N, self.V = float(np.prod(self.n)), float(self.box.prod())
        k, mod, deg = _kgrids(c)
        self.k = [torch.as_tensor(x, device=DEV) for x in k]
        self.mod = torch.as_tensor(mod, device=DEV)
        self.deg = torch.as_tensor(deg, device=DEV)
        self.unit = [torch.where(self.mod > 0, x / self.mod.clamp_min(1e-300), 0.0 * x) for x in self.k]
        self.mu = self.unit[2]
        self.edges = _edges(c)
        w = np.ones(self.n[:2] + (self.n[2] // 2 + 1,))
        if c["window"] != "none":
            s = [np.sin(np.pi / self.n[i] * k[i] / (2 * np.pi / self.box[i])) ** 2 for i in range(3)]
            for t in s:
                w = w * (np.sqrt(1 - 2.0 / 3 * t) if c["window"] == "cic" else np.sqrt(1 - t + 2.0 / 15 * t ** 2))
        self.W = torch.as_tensor(w, device=DEV)
        table = _pk_table(c, seed)
        inv = np.ones_like(mod) if table is None else 1.0 / np.interp(mod, table[0], table[1])
        inv[0, 0, 0] = 1.0
        self.invP = torch.as_tensor(inv, device=DEV)

    def fft(self, x):
        return torch.fft.rfftn(x.double(), dim=(-3, -2, -1))

    def ifft(self, x):
        return torch.fft.irfftn(x, s=self.n, dim=(-3, -2, -1))

    def theta(self, b):
        return ((self.mod >= self.edges[b]) & (self.mod < self.edges[b + 1])).double()

    def leg(self, l, mu=None):
        m = self.mu if mu is None else mu
        return {0: 1.0 + 0 * m, 2: 1.5 * m ** 2 - 0.5, 4: (35 * m ** 4 - 30 * m ** 2 + 3) / 8}[l]

    def bins(self, x, ls):
        """sum over the modes of each bin of deg L_l x, flattened (l, bin)."""
        nk = len(self.edges) - 1
        at = torch.bucketize(self.mod.reshape(-1), torch.as_tensor(self.edges, device=DEV), right=True)
        at = torch.where((at >= 1) & (at <= nk), at, 0 * at)
        return torch.cat([torch.zeros(nk + 1, dtype=torch.float64, device=DEV).index_add_(
            0, at, (self.deg * self.leg(l) * x).reshape(-1))[1:] for l in ls])

    def maps(self, x, ls, filt=None):
        """irfftn(Theta_b L_l filt x) for every (l, bin), (Nl nk, N^3)."""
        x = x if filt is None else x * filt
        return torch.stack([self.ifft(self.theta(b) * self.leg(l) * x).reshape(-1) for l in ls
                            for b in range(len(self.edges) - 1)])

    @staticmethod
    def sums(A, B, C, idx):
        """sum_x A[i] B[j] C[k] for the rows (i, j, k) of idx."""
        out = torch.zeros(len(idx), dtype=torch.float64, device=DEV)
        idx = np.asarray(idx)
        step = 1 << 21
        for a in np.unique(idx[:, 0]):
            rows = np.nonzero(idx[:, 0] == a)[0]
            bs, at = np.unique(idx[rows, 1], return_inverse=True)
            D = 0
            for v in range(0, A.shape[1], step):
                D = D + (A[a, v:v + step] * B[torch.as_tensor(bs, device=DEV), v:v + step]) @ C[:, v:v + step].T
            out[torch.as_tensor(rows, device=DEV)] = D[torch.as_tensor(at, device=DEV),
                                                      torch.as_tensor(idx[rows, 2], device=DEV)]
        return out

    def _addition(self, l):
        """Filters f and weights w with sum w f(k) f(k') = L_l(k.k')."""
        u = self.unit
        if l == 0:
            return [(1.0 + 0 * self.mod, 1.0)]
        assert l == 2
        return [(u[i] * u[j], 1.5 * (1 if i == j else 2)) for i in range(3) for j in range(i, 3)] + \
            [(1.0 * (self.mod > 0), -0.5)]

    def symmetry(self, trip):
        out = [6.0 if a == d else 2.0 if a == b or b == d else 1.0 for a, b, d in trip]
        ls = range(2, self.c["lmax"] + 1, 2)
        if not len(ls):
            return torch.as_tensor(out, dtype=torch.float64, device=DEV)
        u = self.maps(self.invP + 0j, [0])
        pairs = sorted({(a, d) for a, b, d in trip if b == d})
        den = self.sums(u, u, u, [(a, d, d) for a, d in pairs])
        for l in ls:
            num = sum(w * self.sums(u, y, y, [(a, d, d) for a, d in pairs])
                      for f, w in self._addition(l) for y in [self.maps(self.invP + 0j, [0], f)])
            ratio = dict(zip(pairs, (num / den).tolist()))
            out += [2 * (1 + 2 * ratio[a, d]) if a == d else 2.0 if a == b else 1 + ratio[a, d] if b == d else 1.0
                    for a, b, d in trip]
        return torch.as_tensor(out, dtype=torch.float64, device=DEV)

    def cubic(self, G, trip):
        nk, nl = len(self.edges) - 1, self.c["lmax"] // 2 + 1
        return self.sums(G, G, G, [(a, b, l * nk + d) for l in range(nl) for a, b, d in trip])

    def ideal_fisher(self, trip, sym):
        nk, ls = len(self.edges) - 1, range(0, self.c["lmax"] + 1, 2)
        n3, one = len(trip), self.invP + 0j
        u = self.maps(one, ls)
        F = torch.zeros(n3 * len(ls), n3 * len(ls), dtype=torch.float64, device=DEV)
        at = np.asarray(trip)
        same12, same23 = at[:, 0] == at[:, 1], at[:, 1] == at[:, 2]
        c1 = torch.as_tensor(np.where(same12 & ~same23, 2.0, np.where(same12 & same23, 2.0, 1.0)), device=DEV)
        c2 = torch.as_tensor(np.where(same12 & same23, 4.0, np.where(same23, 1.0, 0.0)), device=DEV)
        for i, l in enumerate(ls):
            for j, m in enumerate(ls):
                t1 = self.sums(u[:nk], u[:nk], self.maps(one, [0], self.leg(l) * self.leg(m)), trip)
                t2 = self.sums(u[:nk], u[i * nk:(i + 1) * nk], u[j * nk:(j + 1) * nk], trip)
                F[range(i * n3, i * n3 + n3), range(j * n3, j * n3 + n3)] = c1 * t1 + c2 * t2
        return F / torch.outer(sym, sym) * self.N ** 2 / self.V

    def multipole(self, x, l, r):
        """sum over monomials of L_l(k.r): the l-th multipole of x(r) about the direction of r."""
        u, out = self.unit, 0
        if l == 2:
            terms = [((i, j), 1.5 * (1 if i == j else 2)) for i in range(3) for j in range(i, 3)] + [((), -0.5)]
        else:
            terms = [((), 3 / 8.0)]
            for p, q in ((4, 35 / 8.0), (2, -30 / 8.0)):
                for a in range(p + 1):
                    for b in range(p + 1 - a):
                        f = [1, 1, 2, 6, 24]
                        terms.append(((0,) * a + (1,) * b + (2,) * (p - a - b), q * f[p] / f[a] / f[b] / f[p - a - b]))
        for at, w in terms:
            y, z = x, w
            for i in at:
                y, z = y * r[i], z * u[i]
            out = out + z * self.fft(y)
        return out

    def noise(self, seed):
        """Half spectrum of the Gaussian field whose white noise is the Box-Muller pair of the first two
        words of Philox4x32-10 with key = seed and counter = (voxel, 0x5A17, 0)."""
        p = torch.arange(int(self.N), dtype=torch.int64, device=DEV)
        M32, c = 0xFFFFFFFF, [p & 0xFFFFFFFF, p >> 32, 0 * p + 0x5A17, 0 * p]
        k0, k1 = seed & M32, seed >> 32
        for _ in range(10):
            a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
            c = [((b >> 32) & M32) ^ c[1] ^ k0, b & M32, ((a >> 32) & M32) ^ c[3] ^ k1, a & M32]
            k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
        u1, u2 = [(x.double() + 0.5) * 2.0 ** -32 for x in c[:2]]
        rad, ang = torch.sqrt(-2 * torch.log(u1)), 2 * np.pi * u2
        z = torch.complex(rad * torch.cos(ang), rad * torch.sin(ang)).reshape(self.n)
        mirror = z
        for i in range(3):
            mirror = torch.roll(torch.flip(mirror, [i]), 1, i)
        h = 0.5 * (z + mirror.conj())[..., :self.n[2] // 2 + 1]
        h[0, 0, 0] = 0
        return h * torch.sqrt(1.0 / self.invP) * self.W * self.N / np.sqrt(self.V)


def exact(c, seed):
    e = _Exact(c, seed)
    kind, ls, nk = c["kind"], range(0, c["lmax"] + 1, 2), c["nk"]
    m = _mask(c, seed)
    m = None if m is None else m.double()
    norm = e.V / e.N
    if kind in ("pk", "pk_masked", "pk_grad"):
        x = _fields(c, seed)[0].double()
        if m is not None:
            x = x * m
        X = e.fft(x) / e.W
        if kind == "pk":
            X = X * e.invP
            nums = 0.5 * norm / e.N * e.bins(X.abs() ** 2, ls)
            F = torch.zeros(len(nums), len(nums), dtype=torch.float64, device=DEV)
            for i, l in enumerate(ls):
                for j, q in enumerate(ls):
                    d = 0.5 * e.bins(e.invP ** 2 * e.leg(l) * e.leg(q), [0])
                    F[range(i * nk, i * nk + nk), range(j * nk, j * nk + nk)] = d
            p = torch.linalg.solve(F, nums)
            return {"p%d" % l: p[i * nk:(i + 1) * nk] for i, l in enumerate(ls)}
        if not c["local"]:
            nums = 0.5 * norm / e.N * e.bins(X.abs() ** 2, ls)
        else:
            centre = _centre(c)
            r = [torch.as_tensor(np.fft.fftshift(np.arange(-e.n[i] // 2, e.n[i] // 2)) * e.box[i] / e.n[i] + centre[i],
                                 device=DEV).reshape([-1 if j == i else 1 for j in range(3)]) for i in range(3)]
            rr = torch.sqrt(r[0] ** 2 + r[1] ** 2 + r[2] ** 2)
            r = [t / rr for t in r]
            real = e.ifft(X)
            nums = torch.cat([0.5 * norm / e.N * e.bins((X.conj() * (X if l == 0 else e.multipole(real, l, r))).real,
                                                       [0]) for l in ls])
        if kind == "pk_masked":
            return nums
        v = _cotangent(len(nums), seed)
        f = sum(v[i * nk + b] * e.leg(l) * e.theta(b) for i, l in enumerate(ls) for b in range(nk))
        return {"num": nums, "grad": norm * m * e.ifft(f * X / e.W)}
    trip = _triplets(c)
    if kind == "fisher_pk":
        F = 0
        for s in range(c["sims"]):
            a = e.noise(s + int(1e7))
            A, S = a * e.invP / e.W ** 2, e.fft(m * e.ifft(a))
            F = F + torch.stack([0.5 * norm / e.N * e.bins((A.conj() * e.fft(m * e.ifft(e.theta(b) * e.leg(l) * S)))
                                                           .real, ls) for l in ls for b in range(nk)])
        return F / c["sims"]
    sym = e.symmetry(trip)
    if kind == "bk_setup":
        return {"fish": e.ideal_fisher(trip, sym), "sym": sym}
    if kind == "fisher_bk":
        th = [e.theta(b) for b in range(nk)]
        F = 0

        def products(w):
            G = [[e.ifft(t * x) for t in th] for x in w]
            return {(a, b): e.fft(G[0][a] * G[0][b] - G[1][a] * G[1][b]) for a in range(nk) for b in range(a, nk)}
        for s in range(c["sims"]):
            a = [e.noise(s + int(1e7)), e.noise(s + int(2e7))]
            P = products([x * e.invP / e.W ** 2 for x in a])
            Q = torch.stack([e.fft(m * e.ifft(th[d] * P[a_, b] + th[a_] * P[b, d] + th[b] * P[a_, d]))
                             for a_, b, d in trip]).reshape(len(trip), -1)
            P = products([e.fft(m * e.ifft(x)) for x in a])
            rows = []
            for a_, b, d in trip:
                left = (e.deg * th[b] * P[a_, d].conj()).reshape(-1)
                rows.append(0.5 * norm / e.N * (Q @ left).real)
            F = F + torch.stack(rows) / torch.outer(sym, sym)
        return F / c["sims"]
    fields = [f.double() for f in _fields(c, seed, 1 + c["sims"])]
    if m is not None:
        fields = [(f.to(torch.float32) * m.to(torch.float32)).double() if c["precision"] == "mixed" else f * m
                  for f in fields]
    if kind == "bk":
        G = e.maps(e.fft(fields[0]) * e.invP / e.W, ls)
        num = e.cubic(G, trip) * norm / sym
        B = torch.linalg.solve(e.ideal_fisher(trip, sym), num)
        return {"b%d" % l: B[i * len(trip):(i + 1) * len(trip)] for i, l in enumerate(ls)}
    G = e.maps(e.fft(fields[0]) / e.W, ls)
    if kind == "bk_linear":
        tl = [(a, b, i * nk + d) for i in range(len(ls)) for a, b, d in trip]
        B = e.cubic(G, trip)
        for f in fields[1:]:
            S = e.maps(e.fft(f) / e.W, ls)
            B = B - (e.sums(G, S, S, tl) + e.sums(S, G, S, tl) + e.sums(S, S, G, tl)) / c["sims"]
        return B * norm / sym
    # bk_grad: the gradient of sum_t v_t num_t in the maps, gathered back through their filters
    num = e.cubic(G, trip) * norm / sym
    v = _cotangent(len(num), seed) * norm / sym
    T = torch.zeros((len(G),) * 3, dtype=torch.float64, device=DEV)
    for i in range(len(ls)):
        for t, (a, b, d) in enumerate(trip):
            for o, x, y in ((a, b, i * nk + d), (b, a, i * nk + d), (i * nk + d, a, b)):
                T[o, x, y] += v[i * len(trip) + t]
    spec = 0
    for o in range(len(G)):
        g = torch.cat([(x * (T[o] @ x)).sum(0) for x in G.split(1 << 21, 1)]).reshape(e.n)
        spec = spec + e.fft(g) * e.theta(o % nk) * e.leg(ls[o // nk]) / e.W
    return {"num": num, "grad": e.ifft(spec)}
