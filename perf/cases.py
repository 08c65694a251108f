"""Performance cases of the framework's main paths, through its public API.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` makes what a user's program holds before the call,
``run(state)`` is one pass, ``work(case)`` the bytes and operations it cannot
do without and ``exact(case, seed)`` the same outputs from plain torch in
64 bits.

Paths:

* ``expansion``  the spherical expansion as a featomic TensorMap;
* ``soap``       the power spectrum as a featomic TensorMap, with the explicit
                 gradients asked for;
* ``adjoint``    the dense power spectrum of the torch interface and its
                 backward pass to positions and cell;
* ``training``   a training step on energy and forces of a linear model: the
                 forward pass, the differentiable backward pass, and the double
                 backward to the weights;
* ``batch``      power spectrum, forces and energies of many molecules;
* ``lambda``     the Clebsch-Gordan product of two densities (lambda-SOAP);
* ``lode``       the long-range (LODE) spherical expansion.

Periodic boxes are jittered lattices at number density 0.1 A^-3 in a slightly
strained cube, molecules are jittered lattice balls of 7.2 A^3 per atom, in
the shapes of ``rascaline_b200.workloads``.
"""
import math

import numpy as np
import torch

DENSITY = 0.1
TYPES = (1, 6, 8, 7)
RADIALS = (3, 4, 5, 7, 8)


def listed():
    return [
        # featurising one small cell through the host API (the 216-atom
        # lattice configuration): latency, launches and labels
        dict(name="expansion_host_216", path="expansion", atoms=216, molecules=0, species=2, cutoff=5.0, radial=5,
             angular=4, gradients="", host=True),
        # expansion with positions gradients, the input of equivariant models
        # that differentiate explicitly
        dict(name="expansion_gradients_500", path="expansion", atoms=500, molecules=0, species=2, cutoff=5.5, radial=7,
             angular=6, gradients="positions", host=False),
        # the unit cell of a molecular-dynamics step: small and latency bound
        dict(name="soap_forces_64", path="soap", atoms=64, molecules=0, species=2, cutoff=4.0, radial=4, angular=3,
             gradients="positions", host=False),
        # the headline drop-in workload: a 1000-atom box with positions and
        # strain gradients
        dict(name="soap_forces_1000", path="soap", atoms=1000, molecules=0, species=3, cutoff=5.5, radial=7, angular=6,
             gradients="positions strain", host=False),
        # descriptors of a data set of molecules, no gradients
        dict(name="soap_values_molecules_512", path="soap", atoms=0, molecules=512, species=4, cutoff=5.0, radial=7,
             angular=6, gradients="", host=False),
        # one molecular-dynamics step of a small cell in the torch interface
        dict(name="adjoint_f32_64", path="adjoint", atoms=64, species=3, cutoff=4.5, radial=5, angular=4, precision=32),
        # forces and cell gradient of the large strained box (the adjoint's
        # headline configuration)
        dict(name="adjoint_f32_20000", path="adjoint", atoms=20000, species=4, cutoff=5.0, radial=7, angular=6,
             precision=32),
        # the same in double precision on an ordinary box
        dict(name="adjoint_f64_2000", path="adjoint", atoms=2000, species=4, cutoff=5.0, radial=7, angular=6,
             precision=64),
        # fitting a potential to forces
        dict(name="training_f32_1500", path="training", atoms=1500, species=3, cutoff=5.0, radial=7, angular=6,
             precision=32),
        # the batched headline configuration: 4096 molecules of 5 to 60 atoms
        dict(name="batch_4096", path="batch", molecules=4096, species=4, cutoff=5.0, radial=7, angular=6, pipeline=1),
        # every (l_1 <= l_2, lambda) block of a 2000-centre lambda-SOAP
        dict(name="lambda_soap_2000", path="lambda", atoms=2000, species=4, radial=7, angular=4, precision=64),
        # long-range descriptors of the 1000-atom box
        dict(name="lode_1000", path="lode", atoms=1000, species=3, radial=7, angular=6, smearing=1.0, gradients=""),
    ]


def _between(rng, low, high):
    """A whole number, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    path = rng.choice(["expansion", "soap", "soap", "adjoint", "adjoint", "training", "batch", "lambda", "lode"])
    case = dict(path=path)
    if path in ("expansion", "soap"):
        while True:
            molecules = rng.random() < 0.3
            gradients = rng.choice(["", "positions", "positions", "positions strain", "positions cell"])
            case.update(atoms=0 if molecules else _between(rng, 40, 1000),
                        molecules=_between(rng, 8, 512 if not gradients else 64) if molecules else 0,
                        species=rng.choice([1, 2, 3, 4]), cutoff=round(rng.uniform(3.5, 5.5), 2),
                        radial=rng.choice(RADIALS), angular=rng.choice([2, 3, 4, 5, 6, 8]), gradients=gradients,
                        host=rng.random() < 0.25 and not gradients)
            species = case["species"]
            blocks = (case["angular"] + 1) * species ** 2 if path == "expansion" else species ** 2 * (species + 1) // 2
            rows = 50.0 * max(case["atoms"], 33 * case["molecules"]) * species if gradients else 1.0
            props = (case["angular"] + 1) * (case["radial"] + 1) ** 2
            # as many outputs as can be looked at one by one, and no more
            # gradient rows than the headline workload's
            if blocks * (1 + len(gradients.split())) <= 64 and rows * props < 1.5e5 * 448:
                return case
    if path == "adjoint":
        precision = rng.choice([32, 32, 64])
        case.update(atoms=_between(rng, 40, 20000 if precision == 32 else 2000), species=rng.choice([1, 2, 3, 4]),
                    cutoff=round(rng.uniform(4.0, 5.0), 2), radial=rng.choice([3, 4, 5, 7]),
                    angular=rng.choice([3, 4, 5, 6]), precision=precision)
    elif path == "training":
        case.update(atoms=_between(rng, 40, 1500), species=rng.choice([1, 2, 3]), cutoff=round(rng.uniform(4.0, 5.0), 2),
                    radial=rng.choice([3, 4, 5, 7]), angular=rng.choice([3, 4, 5, 6]), precision=rng.choice([32, 64]))
    elif path == "batch":
        molecules = _between(rng, 8, 4096)
        case.update(molecules=molecules, species=rng.choice([2, 3, 4]), cutoff=round(rng.uniform(4.0, 5.0), 2),
                    radial=rng.choice([3, 5, 7]), angular=rng.choice([3, 4, 6]),
                    # one graph replay for small batches, the dense pipeline for large ones
                    pipeline=0 if molecules < 64 else 1)
    elif path == "lambda":
        case.update(atoms=_between(rng, 60, 2000), species=rng.choice([1, 2, 3, 4]), radial=rng.choice([3, 4, 5, 7]),
                    angular=rng.choice([2, 3, 4]), precision=rng.choice([32, 64]))
    else:
        gradients = rng.choice(["", "", "positions"])
        case.update(atoms=_between(rng, 40, 80 if gradients else 1000), species=2 if gradients else rng.choice([1, 2, 3]),
                    radial=rng.choice([3, 5, 7]), angular=rng.choice([3, 4, 6]), smearing=round(rng.uniform(1.0, 1.4), 2),
                    gradients=gradients)
    return case


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _soap_hypers(case):
    return {
        "cutoff": {"radius": case["cutoff"], "smoothing": {"type": "ShiftedCosine", "width": 0.5}},
        "density": {"type": "Gaussian", "width": 0.3},
        "basis": {"type": "TensorProduct", "max_angular": case["angular"],
                  "radial": {"type": "Gto", "max_radial": case["radial"]}},
    }


def _lode_hypers(case):
    return {
        "density": {"type": "SmearedPowerLaw", "smearing": case["smearing"], "exponent": 1},
        "basis": {"type": "TensorProduct", "max_angular": case["angular"],
                  "radial": {"type": "Gto", "max_radial": case["radial"], "radius": 5.5}},
    }


def _types(rng, n, species):
    """Every type about equally often, in random order."""
    return np.array(TYPES[:species], dtype=np.int32)[rng.permutation(n) % species]


def _turns(rng, count):
    return np.linalg.qr(rng.normal(size=(count, 3, 3)))[0]


def _box(case, seed):
    """(types, positions, cell) of one strained periodic box.  The structure
    belongs to the case; the seed turns it, moves it through the boundary and
    orders its atoms, so that another seed gives other inputs with as many
    pairs."""
    rng = np.random.default_rng(case["atoms"])
    n = case["atoms"]
    length = (n / DENSITY) ** (1.0 / 3.0)
    g = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    sites = np.stack(np.meshgrid(*[np.arange(g)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    sites = sites[rng.permutation(len(sites))[:n]]
    spacing = length / g
    jitter = max(0.1, 0.5 * (spacing - 0.95))
    fractional = ((sites + 0.5) * spacing + rng.uniform(-jitter, jitter, size=(n, 3))) / length
    cell = length * (np.eye(3) + rng.uniform(-0.02, 0.02, size=(3, 3)))
    types = _types(rng, n, case["species"])
    rng = np.random.default_rng(seed)
    order = rng.permutation(n)
    cell = cell @ _turns(rng, 1)[0]
    return types[order], ((fractional[order] + rng.uniform(size=3)) % 1.0) @ cell, cell


def _molecule_sizes(case):
    """Sizes spread evenly over 5 to 60 atoms."""
    m = case["molecules"]
    return 5 + np.arange(m) * 55 // max(1, m - 1)


def _molecules(case, seed):
    """(sizes, types, positions) of molecules: the lattice sites nearest to a
    random centre, jittered.  The seed turns each molecule and orders them."""
    rng = np.random.default_rng(case["molecules"])
    sizes = _molecule_sizes(case)
    m, spacing = len(sizes), 1.93
    grid = np.stack(np.meshgrid(*[np.arange(-3, 4)] * 3, indexing="ij"), axis=-1).reshape(-1, 3).astype(np.float64)
    sites = grid[None] + rng.uniform(-0.5, 0.5, size=(m, 1, 3))
    nearest = np.argsort((sites ** 2).sum(-1), axis=1)[:, :60]
    sites = np.take_along_axis(sites, nearest[:, :, None], axis=1) * spacing
    sites += rng.uniform(-0.45, 0.45, size=sites.shape)
    types = _types(rng, 60 * m, case["species"]).reshape(m, 60)
    rng = np.random.default_rng(seed)
    order = rng.permutation(m)
    sites = sites[order] @ _turns(rng, m)
    keep = np.arange(60)[None] < sizes[order][:, None]
    return sizes[order], types[order][keep], sites[keep]


def _structures(case, seed):
    """(sizes, types, positions, cells) of the structures of one call."""
    if case.get("molecules"):
        sizes, types, positions = _molecules(case, seed)
        return sizes, types, positions, np.zeros((len(sizes), 3, 3))
    types, positions, cell = _box(case, seed)
    return np.array([len(types)]), types, positions, cell[None]


def _normal(seed, shape, scale, dtype):
    generator = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=generator, dtype=torch.float64) * scale).to(dtype)


def _dtype(case):
    return torch.float32 if case.get("precision", 32) == 32 else torch.float64


def _property_count(case):
    return (case["angular"] + 1) * (case["radial"] + 1) ** 2


def _gradient_rows(case, seed, n):
    """dL/dP rows of the atoms, as a model's head gives them, on the GPU."""
    keys, props = case["species"] * (case["species"] + 1) // 2, _property_count(case)
    generator = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((n, keys, props), generator=generator, dtype=torch.float64,
                       device="cuda").div_(math.sqrt(keys * props)).to(_dtype(case))


def _weights(case, seed, dtype):
    """A linear model per centre species, [species, keys, properties]."""
    species = case["species"]
    keys, props = species * (species + 1) // 2, _property_count(case)
    return _normal(seed, (species, keys, props), 1.0 / math.sqrt(keys * props), dtype)


def _density_blocks(case, seed):
    """[samples, 2 l + 1, species * n] per l: normal values that fall off with l."""
    generator = torch.Generator(device="cuda").manual_seed(seed)
    width = case["species"] * (case["radial"] + 1)
    return [torch.randn((case["atoms"], 2 * l + 1, width), generator=generator, dtype=torch.float64,
                        device="cuda").div_(1.0 + l).to(_dtype(case)) for l in range(case["angular"] + 1)]


def prepare(case, seed):
    import rascaline_b200 as rb
    from rascaline_b200 import clebsch_gordan, torch_api

    path = case["path"]
    if path == "lambda":
        blocks = _density_blocks(case, seed)
        samples = rb.Labels(["system", "atom"], [[0, k] for k in range(case["atoms"])])
        radial = case["radial"] + 1
        properties = rb.Labels(["neighbor_type", "n"], [[t, n] for t in TYPES[:case["species"]] for n in range(radial)])
        density = clebsch_gordan.EquivariantTensorMap(
            rb.Labels(["o3_lambda", "o3_sigma", "center_type"], [[l, 1, 1] for l in range(len(blocks))]),
            [clebsch_gordan.Block(b, samples, [rb.Labels(["o3_mu"], [[m] for m in range(-l, l + 1)])], properties)
             for l, b in enumerate(blocks)])
        product = clebsch_gordan.DensityCorrelations(n_correlations=1, max_angular=2 * case["angular"])
        return dict(path=path, density=density, product=product)
    sizes, types, positions, cells = _structures(case, seed)
    on_gpu = torch.as_tensor(positions, device="cuda")
    if path == "batch":
        calculator = rb.SoapPowerSpectrum(**_soap_hypers(case))
        batch = torch_api.Batch(calculator, sizes, types, sorted(TYPES[:case["species"]]))
        if case["pipeline"] == 1:
            batch.config = dict(batch.config, pipeline=1)
        return dict(path=path, batch=batch, positions=on_gpu, out=batch.outputs(),
                    weights=_weights(case, seed + 1, torch.float32).cuda())
    if path in ("adjoint", "training"):
        calculator = torch_api.SoapPowerSpectrum(**_soap_hypers(case), precision=case["precision"])
        cell = torch.as_tensor(cells[0], device="cuda")
        state = dict(path=path, calculator=calculator, types=torch.as_tensor(types), positions=on_gpu, cell=cell)
        if path == "adjoint":
            state["gradient"] = _gradient_rows(case, seed + 1, len(types))
        else:
            species = np.unique(types)
            state["weights"] = _weights(case, seed + 1, _dtype(case)).cuda()
            state["species"] = torch.as_tensor(np.searchsorted(species, types), device="cuda")
            state["target"] = _normal(seed + 2, (len(types), 3), 1.0, torch.float64).cuda()
        return state
    if path == "lode":
        calculator = rb.LodeSphericalExpansion(**_lode_hypers(case))
    else:
        kind = rb.SphericalExpansion if path == "expansion" else rb.SoapPowerSpectrum
        calculator = kind(**_soap_hypers(case))
    state = dict(path=path, calculator=calculator, gradients=case["gradients"].split(), host=case.get("host", False))
    if state["host"]:
        starts = np.concatenate([[0], np.cumsum(sizes)])
        state["systems"] = [rb.System(types[a:b], positions[a:b], cell)
                            for a, b, cell in zip(starts[:-1], starts[1:], cells)]
    else:
        state.update(positions=on_gpu, types=types, cells=cells, sizes=sizes)
    return state


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(state):
    path = state["path"]
    if path == "lambda":
        return [block.values for block in state["product"].compute(state["density"]).blocks()]
    if path == "batch":
        return state["batch"].run(state["positions"], state["out"], weights=state["weights"])
    if path in ("adjoint", "training"):
        return _run_torch(state)
    if state["host"]:
        result = state["calculator"].compute(state["systems"], gradients=state["gradients"])
    else:
        result = state["calculator"].compute_device(state["positions"], state["types"], state["cells"], state["sizes"],
                                                    gradients=state["gradients"])
    outputs = []
    for block in result.blocks():
        outputs.append(block.values)
        outputs += [block.gradient(parameter).values for parameter in state["gradients"]]
    return outputs


def _run_torch(state):
    from rascaline_b200 import torch_api

    positions = state["positions"].detach().requires_grad_()
    if state["path"] == "adjoint":
        cell = state["cell"].detach().requires_grad_()
        values = state["calculator"].dense([torch_api.System(state["types"], positions, cell)])
        forces, virial = torch.autograd.grad(values, [positions, cell], state["gradient"])
        return [values.detach(), forces, virial]
    weights = state["weights"].detach().requires_grad_()
    values = state["calculator"].dense([torch_api.System(state["types"], positions, state["cell"])])
    energy = (values * weights[state["species"]]).sum()
    gradient, = torch.autograd.grad(energy, [positions], create_graph=True)
    loss = (gradient - state["target"]).square().sum() + energy.square() / len(positions)
    slope, = torch.autograd.grad(loss, [weights])
    return [energy.detach(), gradient.detach(), slope]


# --------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------
def work(case):
    """Inputs read once, outputs written once; multiply-adds of the expansion
    (per neighbour and coefficient), of the contractions and of the gradients."""
    path = case["path"]
    species, n = case["species"], case["radial"] + 1
    if path == "lambda":
        rows = sum((2 * a + 1) * (2 * b + 1) for a in range(case["angular"] + 1)
                   for b in range(a, case["angular"] + 1))
        outputs = case["atoms"] * rows * (species * n) ** 2
        inputs = case["atoms"] * (case["angular"] + 1) ** 2 * species * n
        return {"bytes": (outputs + inputs) * case["precision"] / 8, "flops": 2.0 * 2 * outputs}
    coefficients = (case["angular"] + 1) ** 2 * n
    if path == "lode":
        volume, k_cutoff = case["atoms"] / DENSITY, 1.2 * math.pi / case["smearing"]
        waves = 2.0 / 3.0 * math.pi * k_cutoff ** 3 * volume / (2 * math.pi) ** 3
        rows = case["atoms"] * species * (1 + (3.0 * case["atoms"] / species if case["gradients"] else 0))
        return {"bytes": 8.0 * (rows * coefficients + 3 * case["atoms"]), "flops": 2.0 * rows * coefficients * waves}
    if case.get("molecules"):
        atoms = int(_molecule_sizes(case).sum())
        neighbors = min(30.0, 0.6 * 4.0 / 3.0 * math.pi * case["cutoff"] ** 3 / 7.2)
    else:
        atoms = case["atoms"]
        neighbors = 4.0 / 3.0 * math.pi * case["cutoff"] ** 3 * DENSITY
    directions = atoms * neighbors
    keys, props = species * (species + 1) // 2, _property_count(case)
    contraction = 2.0 * atoms * keys * n * coefficients
    if path in ("adjoint", "training", "batch"):
        word = case.get("precision", 32) / 8
        rows = atoms * keys * props
        if path == "adjoint":
            words = 2 * rows  # the power spectrum written, dL/dP read
        elif path == "batch":
            words = rows + species * keys * props
        else:
            words = 2 * species * keys * props  # the weights and their gradient
        passes = 2 if path == "training" else 1
        return {"bytes": word * (words + 3 * atoms) + 24.0 * atoms,
                "flops": passes * (3 * contraction + directions * coefficients * (4 + 10))}
    gradients = case["gradients"].split()
    if path == "expansion":
        values = atoms * species * coefficients
        positions = 3.0 * (directions + atoms * species) * coefficients
        flops = 4.0 * directions * coefficients * (1 + 3 * bool(gradients))
    else:
        values = atoms * keys * props
        positions = 3.0 * (directions * species + atoms * keys) * props
        per_row = 2.0 * (2 * case["angular"] / 2 + 1)
        flops = 4.0 * directions * coefficients * (1 + 3 * bool(gradients)) + contraction
        flops += per_row * positions if "positions" in gradients else 0
    outputs = values * (1 + 9 * (len(gradients) - ("positions" in gradients)))
    outputs += positions if "positions" in gradients else 0
    return {"bytes": 8.0 * (outputs + 3 * atoms), "flops": flops}


# --------------------------------------------------------------------------
# the same outputs in 64 bits, plain torch
# --------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tensor(x, dtype=torch.float64):
    return torch.as_tensor(np.asarray(x), dtype=dtype, device=_device())


def _kummer(a, b, z):
    """1F1(a, b, z) for z >= 0 by its power series."""
    term = torch.ones_like(z)
    total = term.clone()
    for k in range(2000):
        term = term * ((a + k) / (b + k) / (k + 1.0)) * z
        total += term
        if k % 16 == 15 and bool((term.abs() <= 1e-17 * total.abs()).all()):
            break
    return total


def _gto(radial, radius):
    """Widths [n] and orthonormalisation [n, n] of the GTO basis."""
    n = radial + 1
    width = np.array([radius * max(math.sqrt(k), 1.0) / n for k in range(n)])
    norm = np.array([1.0 / math.sqrt(0.5 * width[k] ** (2 * k + 3) * math.gamma(k + 1.5)) for k in range(n)])
    overlap = np.zeros((n, n))
    for i in range(n):
        for j in range(n):
            e = 0.5 * (3 + i + j)
            overlap[i, j] = (0.5 / width[i] ** 2 + 0.5 / width[j] ** 2) ** -e * 0.5 * math.gamma(e) * norm[i] * norm[j]
    value, vector = np.linalg.eigh(overlap)
    return width, (vector / np.sqrt(value)) @ vector.T * norm


def _radial_integral(case, r):
    """R [pairs, l, n] and dR/dr of a Gaussian density in the GTO basis."""
    width, ortho = _gto(case["radial"], case["cutoff"])
    n = case["radial"] + 1
    c = 0.5 / 0.3 ** 2
    b = 0.5 / _tensor(width) ** 2
    z = (c * r[:, None]) ** 2 / (c + b)
    values, slopes = [], []
    for l in range(case["angular"] + 1):
        beta = l + 1.5
        alpha = _tensor([0.5 * (k + l + 3) for k in range(n)])
        ratio = _tensor([math.gamma(0.5 * (k + l + 3)) / math.gamma(beta) for k in range(n)])
        front = (math.pi / 0.3 ** 2) ** 0.75 * (torch.exp(-c * r * r) * (c * r) ** l)[:, None] * ratio * (c + b) ** -alpha
        value = front * _kummer(alpha, beta, z)
        slope = front * _kummer(alpha + 1, beta + 1, z) * (alpha / beta) * 2 * z / r[:, None]
        slope += value * (l / r - 2 * c * r)[:, None]
        values.append(value @ _tensor(ortho).T)
        slopes.append(slope @ _tensor(ortho).T)
    return torch.stack(values, 1), torch.stack(slopes, 1)


def _harmonics(direction, lmax):
    """Real spherical harmonics Y [pairs, (lmax + 1)^2] and the derivatives
    [pairs, 3, (lmax + 1)^2] that the path defines: r grad Y, except that
    directions within sin(theta) <= 0.1 of the z axis take m P / sin(theta)
    as -dP / (2 cos(theta))."""
    x, y, ct = direction.unbind(1)
    st = torch.hypot(x, y)
    off = st > 1e-15
    cp = torch.where(off, x / st.clamp_min(1e-300), torch.ones_like(x))
    sp = torch.where(off, y / st.clamp_min(1e-300), torch.zeros_like(x))
    cos, sin = [torch.ones_like(cp)], [torch.zeros_like(cp)]
    for m in range(lmax):
        # featomic leaves out the Condon-Shortley phase, so that P carries it
        cos.append(-(cos[m] * cp - sin[m] * sp))
        sin.append(-(sin[m] * cp + cos[m] * sp))
    P = {(0, 0): torch.full_like(ct, math.sqrt(0.5 / math.pi))}
    for l in range(1, lmax + 1):
        P[l, l] = -math.sqrt(1 + 0.5 / l) * st * P[l - 1, l - 1]
        for m in range(l):
            P[l, m] = math.sqrt((4 * l * l - 1) / (l * l - m * m)) * ct * P[l - 1, m]
            if m < l - 1:
                P[l, m] = P[l, m] - math.sqrt((4 * l * l - 1) / (l * l - m * m) * ((l - 1) ** 2 - m * m)
                                              / (4 * (l - 1) ** 2 - 1)) * P[l - 2, m]
    zero = torch.zeros_like(ct)
    Y, G = [], []
    for l in range(lmax + 1):
        row, grad = [None] * (2 * l + 1), [None] * (2 * l + 1)
        for m in range(l + 1):
            if m == 0:
                row[l] = P[l, 0] / math.sqrt(2)
                slope = math.sqrt(0.5 * l * (l + 1)) * P[l, 1] if l else zero
                grad[l] = torch.stack([cp * ct * slope, sp * ct * slope, -st * slope], 1)
                continue
            row[l + m], row[l - m] = P[l, m] * cos[m], P[l, m] * sin[m]
            # -2 dP/dtheta
            d = math.sqrt((l + m) * (l - m + 1)) * P[l, m - 1]
            if m < l:
                d = d - math.sqrt((l - m) * (l + m + 1)) * P[l, m + 1]
            over = torch.where(st > 0.1, m / st.clamp_min(1e-300) * P[l, m], -0.5 / ct * d)
            for sign, c, s in ((1, cos[m], -sin[m]), (-1, sin[m], cos[m])):
                theta, phi = -0.5 * c * d, over * s
                grad[l + sign * m] = torch.stack([cp * ct * theta - sp * phi, sp * ct * theta + cp * phi, -st * theta], 1)
        Y += row
        G += grad
    return torch.stack(Y, 1), torch.stack(G, 2)


def _pairs(sizes, positions, cells, cutoff):
    """Every directed pair: centre, neighbour, vector and cell shift."""
    found = []
    if not cells.any():
        sizes = torch.as_tensor(np.asarray(sizes), device=_device())
        starts = torch.cumsum(sizes, 0) - sizes
        of_atom = torch.repeat_interleave(sizes, sizes)
        i = torch.repeat_interleave(torch.arange(len(positions), device=_device()), of_atom)
        first = torch.repeat_interleave(torch.cumsum(of_atom, 0) - of_atom, of_atom)
        j = torch.repeat_interleave(torch.repeat_interleave(starts, sizes), of_atom) \
            + torch.arange(len(i), device=_device()) - first
        vector = positions[j] - positions[i]
        keep = (i != j) & ((vector ** 2).sum(1) < cutoff ** 2)
        return i[keep], j[keep], vector[keep], torch.zeros_like(vector[keep])
    cell = cells[0]
    heights = 1.0 / np.linalg.norm(np.linalg.inv(cell), axis=0)
    ranges = [range(-math.ceil(cutoff / h), math.ceil(cutoff / h) + 1) for h in heights]
    n = len(positions)
    chunk = max(1, 20_000_000 // n)
    for shift in np.array([[a, b, c] for a in ranges[0] for b in ranges[1] for c in ranges[2]], dtype=np.float64):
        move = _tensor(shift @ cell)
        for a in range(0, n, chunk):
            vector = positions[None] + move - positions[a:a + chunk, None]
            near = (vector ** 2).sum(-1) < cutoff ** 2
            if not shift.any():
                k = torch.arange(near.shape[0], device=near.device)
                near[k, a + k] = False
            i, j = near.nonzero(as_tuple=True)
            found.append((i + a, j, vector[i, j], _tensor(shift).expand(len(i), 3)))
    i, j, vector, shift = (torch.cat(x) for x in zip(*found))
    order = torch.argsort(i, stable=True)
    return i[order], j[order], vector[order], shift[order]


class _Expansion:
    """The spherical expansion of structures: coefficients [atoms, species,
    (l m), n] and the derivatives of every directed pair's term."""

    def __init__(self, case, seed):
        sizes, types, positions, cells = _structures(case, seed)
        self.case, self.sizes = case, sizes
        self.species = np.unique(types)
        self.n = len(types)
        self.kind = torch.as_tensor(np.searchsorted(self.species, types), device=_device())
        self.i, self.j, self.vector, self.shift = _pairs(sizes, _tensor(positions), cells, case["cutoff"])
        self.r = self.vector.norm(dim=1)
        self.spread = torch.as_tensor([l for l in range(case["angular"] + 1) for _ in range(2 * l + 1)],
                                      device=_device())
        self.segment = self.i * len(self.species) + self.kind[self.j]
        shape = (self.n * len(self.species), len(self.spread), case["radial"] + 1)
        total = torch.zeros(shape, dtype=torch.float64, device=_device())
        for part in self.parts():
            f, _, R, _, Y, _, _ = self.terms(part)
            total.index_add_(0, self.segment[part], (f[:, None] * Y)[:, :, None] * R[:, self.spread])
        total = total.reshape(self.n, len(self.species), *shape[1:])
        center = _radial_integral(case, _tensor([1e-160]))[0][0, 0] * math.sqrt(0.25 / math.pi)
        total[torch.arange(self.n, device=_device()), self.kind, 0] += center
        self.coefficients = total

    def parts(self):
        for a in range(0, len(self.r), 100_000):
            yield slice(a, a + 100_000)

    def terms(self, part):
        r, cutoff = self.r[part], self.case["cutoff"]
        s = math.pi * (r - cutoff + 0.5) / 0.5
        inside = r <= cutoff - 0.5
        f = torch.where(inside, torch.ones_like(r), 0.5 * (1 + torch.cos(s)))
        df = torch.where(inside, torch.zeros_like(r), -0.5 * math.pi / 0.5 * torch.sin(s))
        u = self.vector[part] / r[:, None]
        return (f, df) + _radial_integral(self.case, r) + _harmonics(u, self.case["angular"]) + (u,)

    def pair_gradients(self, part):
        """[pairs, 3, (l m), n]: the pair's term over the neighbour's position."""
        f, df, R, dR, Y, dY, u = self.terms(part)
        R, dR = R[:, self.spread], dR[:, self.spread]
        along = Y[:, :, None] * (df[:, None, None] * R + f[:, None, None] * dR)
        return u[:, :, None, None] * along[:, None] \
            + dY[:, :, :, None] * ((f / self.r[part])[:, None, None] * R)[:, None]

    def present(self):
        """[atoms, species]: whether the species is around (or is) the atom."""
        mask = torch.zeros((self.n, len(self.species)), dtype=torch.bool, device=_device())
        mask[self.i, self.kind[self.j]] = True
        mask[torch.arange(self.n, device=_device()), self.kind] = True
        return mask

    def rows(self, centres, kinds):
        """Gradient rows (sample, atom) of the centres towards the species in
        `kinds`: the selected pairs, the row of each pair, the row of each
        centre itself, and the number of rows."""
        sample = torch.full((self.n,), -1, dtype=torch.long, device=_device())
        sample[centres] = torch.arange(len(centres), device=_device())
        wanted = torch.zeros(len(self.species), dtype=torch.bool, device=_device())
        wanted[list(kinds)] = True
        pairs = ((sample[self.i] >= 0) & wanted[self.kind[self.j]]).nonzero()[:, 0]
        moving = pairs[self.i[pairs] != self.j[pairs]]
        key = torch.cat([sample[self.i[moving]] * self.n + self.j[moving], sample[centres] * self.n + centres])
        unique, row = torch.unique(key, return_inverse=True)
        return pairs, moving, sample, row[:len(moving)], row[len(moving):], len(unique)


def _normalisation(case):
    """(-1)^l / sqrt(2 l + 1) of every (l m)."""
    return _tensor([(-1) ** l / math.sqrt(2 * l + 1) for l in range(case["angular"] + 1) for _ in range(2 * l + 1)])


def _contract(case, a, b):
    """[..., (l m), n] x [..., (l m), n] -> [..., l n n]."""
    a = a * _normalisation(case)[:, None]
    out = [torch.einsum("...mp,...mq->...pq", a[..., l * l:(l + 1) ** 2, :], b[..., l * l:(l + 1) ** 2, :]).flatten(-2)
           for l in range(case["angular"] + 1)]
    return torch.cat(out, -1)


def _exact_blocks(case, seed):
    e = _Expansion(case, seed)
    gradients = case["gradients"].split()
    species, present, soap = len(e.species), e.present(), case["path"] == "soap"
    all_gradients = torch.cat([e.pair_gradients(part) for part in e.parts()]) if gradients else None
    outputs = []
    keys = [(c, a, b) for c in range(species) for a in range(species) for b in (range(a, species) if soap else (a,))]
    for c, a, b in keys:
        centres = ((e.kind == c) & present[:, a] & present[:, b]).nonzero()[:, 0]
        if len(centres) == 0:
            continue
        factor = math.sqrt(2) if a != b else 1.0
        both = e.coefficients[centres]
        if soap:
            results = {"values": _contract(case, both[:, a], both[:, b]) * factor}
        else:
            results = {"values": both[:, a]}
        if gradients:
            pairs, moving, sample, row, own, count = e.rows(centres, {a, b})
            for parameter in gradients:
                use = moving if parameter == "positions" else pairs
                if parameter == "positions":
                    out = torch.zeros((count, 3) + results["values"].shape[1:], dtype=torch.float64, device=_device())
                else:
                    out = torch.zeros((len(centres), 3, 3) + results["values"].shape[1:], dtype=torch.float64,
                                      device=_device())
                for at in range(0, len(use), 20_000):
                    p = use[at:at + 20_000]
                    g = all_gradients[p]
                    if soap:
                        ci = e.coefficients[e.i[p]][:, None]
                        kind = e.kind[e.j[p]]
                        g = factor * ((kind == a)[:, None, None] * _contract(case, g, ci[:, :, b].expand_as(g))
                                      + (kind == b)[:, None, None] * _contract(case, ci[:, :, a].expand_as(g), g))
                    if parameter == "positions":
                        out.index_add_(0, row[at:at + 20_000], g)
                        out.index_add_(0, own[sample[e.i[p]]], -g)
                    else:
                        v = (e.vector if parameter == "strain" else e.shift)[p]
                        g = v.reshape(v.shape + (1,) * (g.ndim - 1)) * g[:, None]
                        out.index_add_(0, sample[e.i[p]], g)
                results[parameter] = out
        if soap:
            outputs += list(results.values())
            continue
        for l in range(case["angular"] + 1):
            outputs += [x[..., l * l:(l + 1) ** 2, :] for x in results.values()]
    return outputs


def _keys(species):
    return [(a, b) for a in range(species) for b in range(a, species)]


def _power_spectrum(case, a, b):
    """[atoms, species, (l m), n] twice -> [atoms, keys, l n n]."""
    return torch.stack([_contract(case, a[:, s], b[:, t]) * (math.sqrt(2) if s != t else 1.0)
                        for s, t in _keys(case["species"])], 1)


def _exact_adjoint(e, gradient, cell):
    """dL/dpositions and dL/dcell (or dL/dstrain) for dL/dP."""
    c = e.coefficients.detach().requires_grad_()
    slope, = torch.autograd.grad(_power_spectrum(e.case, c, c), [c], gradient)
    forces = torch.zeros((e.n, 3), dtype=torch.float64, device=_device())
    virial = torch.zeros((3, 3), dtype=torch.float64, device=_device())
    for part in e.parts():
        i, j = e.i[part], e.j[part]
        g = torch.einsum("pxmn,pmn->px", e.pair_gradients(part), slope.flatten(0, 1)[e.segment[part]])
        if cell:
            virial += e.shift[part].T @ g
        g = g * (i != j)[:, None]
        forces.index_add_(0, j, g)
        forces.index_add_(0, i, -g)
    return forces, virial


def _exact_training(case, seed):
    e = _Expansion(case, seed)
    weights = _weights(case, seed + 1, _dtype(case)).double().to(_device())
    target = _normal(seed + 2, (e.n, 3), 1.0, torch.float64).to(_device())
    values = _power_spectrum(case, e.coefficients, e.coefficients)
    energy = (values * weights[e.kind]).sum()
    gradient, _ = _exact_adjoint(e, weights[e.kind], False)
    step = 2 * (gradient - target)
    tangent = torch.zeros_like(e.coefficients)
    for part in e.parts():
        delta = step[e.j[part]] - step[e.i[part]]
        tangent.flatten(0, 1).index_add_(0, e.segment[part], torch.einsum("pxmn,px->pmn", e.pair_gradients(part), delta))
    change = _power_spectrum(case, tangent, e.coefficients) + _power_spectrum(case, e.coefficients, tangent)
    change += values * (2 * energy / e.n)
    slope = torch.zeros_like(weights).index_add_(0, e.kind, change)
    return [energy, gradient, slope]


def _real_coupling(l1, l2, l):
    """Real Clebsch-Gordan coefficients [m1, m2, m], by Racah's formula and
    the unitary matrices from complex to real harmonics."""
    f = math.factorial
    table = np.zeros((2 * l1 + 1, 2 * l2 + 1, 2 * l + 1), dtype=complex)
    for m1 in range(-l1, l1 + 1):
        for m2 in range(-l2, l2 + 1):
            m = m1 + m2
            if abs(m) > l:
                continue
            total = 0.0
            for k in range(l1 + l2 - l + 1):
                parts = (k, l1 + l2 - l - k, l1 - m1 - k, l2 + m2 - k, l - l2 + m1 + k, l - l1 - m2 + k)
                if min(parts) >= 0:
                    total += (-1) ** k / math.prod(f(p) for p in parts)
            scale = (2 * l + 1) * f(l + l1 - l2) * f(l - l1 + l2) * f(l1 + l2 - l) / f(l1 + l2 + l + 1)
            scale *= f(l + m) * f(l - m) * f(l1 - m1) * f(l1 + m1) * f(l2 - m2) * f(l2 + m2)
            table[l1 + m1, l2 + m2, l + m] = total * math.sqrt(scale)

    def real(order):
        u = np.zeros((2 * order + 1, 2 * order + 1), dtype=complex)
        u[order, order] = 1.0
        for m in range(1, order + 1):
            u[order - m, order - m], u[order - m, order + m] = -1j * math.sqrt(0.5), 1j * (-1) ** m * math.sqrt(0.5)
            u[order + m, order - m], u[order + m, order + m] = math.sqrt(0.5), (-1) ** m * math.sqrt(0.5)
        return u

    table = np.einsum("ax,by,cz,xyz->abc", real(l1), real(l2), real(l).conj(), table)
    return table.real if (l1 + l2 + l) % 2 == 0 else table.imag


def _exact_lambda(case, seed):
    blocks = [b.double() for b in _density_blocks(case, seed)]
    outputs = []
    for l1 in range(len(blocks)):
        for l2 in range(l1, len(blocks)):
            for l in range(l2 - l1, l1 + l2 + 1):
                coupling = _tensor(_real_coupling(l1, l2, l))
                outputs.append(torch.einsum("xyz,sxp,syq->szpq", coupling, blocks[l1], blocks[l2]).flatten(2))
    return outputs


def _exact_lode(case, seed):
    types, positions, cell = _box(case, seed)
    species = np.unique(types)
    kind = np.searchsorted(species, types)
    lmax, n = case["angular"], case["radial"] + 1
    reciprocal = 2 * math.pi * np.linalg.inv(cell).T
    k_cutoff = 1.2 * math.pi / case["smearing"]
    reach = [math.ceil(k_cutoff * np.linalg.norm(row) / (2 * math.pi)) for row in cell]
    grid = np.stack(np.meshgrid(*[np.arange(-m, m + 1) for m in reach], indexing="ij"), axis=-1).reshape(-1, 3)
    waves = grid @ reciprocal
    norm = np.linalg.norm(waves, axis=1)
    keep = (norm < k_cutoff) & (norm > 0)
    waves, k = _tensor(waves[keep]), _tensor(norm[keep])
    width, ortho = _gto(case["radial"], 5.5)
    Y = _harmonics(waves / k[:, None], lmax)[0]
    projection = []
    for l in range(lmax + 1):
        raw = []
        for m in range(n):
            a, b, z = 0.5 * (m + l + 3), l + 1.5, 0.5 * (k * width[m]) ** 2
            front = math.sqrt(math.pi / 2) * width[m] ** (m + 3) * math.sqrt(2.0) ** m * math.gamma(a) / math.gamma(b)
            raw.append(front * (k * width[m] / math.sqrt(2)) ** l * torch.exp(-z) * _kummer(b - a, b, z))
        R = torch.stack(raw, 1) @ _tensor(ortho).T
        sign = (-1) ** (l // 2 if l % 2 == 0 else (l + 1) // 2)
        projection.append(sign * Y[:, l * l:(l + 1) ** 2, None] * R[:, None])
    weight = 4 * math.pi / abs(np.linalg.det(cell)) * 4 * math.pi * torch.exp(-0.5 * (k * case["smearing"]) ** 2) / k ** 2
    phase = _tensor(positions) @ waves.T
    cos, sin = torch.cos(phase), torch.sin(phase)
    kinds = torch.as_tensor(kind, device=_device())
    gradients = "positions" in case["gradients"]
    outputs = []
    for c in range(len(species)):
        centres = (kinds == c).nonzero()[:, 0]
        for t in range(len(species)):
            others = (kinds == t).nonzero()[:, 0]
            C, S = cos[others].sum(0), sin[others].sum(0)
            # half of the (k, -k) sums: twice the half space's terms
            parts = [cos[centres] * C + sin[centres] * S, sin[centres] * C - cos[centres] * S]
            for l in range(lmax + 1):
                outputs.append(torch.einsum("ik,kmn->imn", parts[l % 2] * weight, projection[l]))
                if not gradients:
                    continue
                rows = []
                for i in centres.tolist():
                    pair = [sin[i] * cos - cos[i] * sin, -(cos[i] * cos + sin[i] * sin)][l % 2]
                    pair = torch.where((kinds == t)[:, None], pair, torch.zeros_like(pair))
                    pair[i] = 0
                    pair[i] = -pair.sum(0)
                    wanted = (kinds == t)
                    wanted[i] = True
                    rows.append(torch.einsum("jk,kmn,kx->jxmn", pair[wanted] * weight, projection[l], waves))
                outputs.append(torch.cat(rows))
    return outputs


def exact(case, seed):
    path = case["path"]
    if path in ("expansion", "soap"):
        return _exact_blocks(case, seed)
    if path == "lambda":
        return _exact_lambda(case, seed)
    if path == "lode":
        return _exact_lode(case, seed)
    if path == "training":
        return _exact_training(case, seed)
    e = _Expansion(case, seed)
    if path == "adjoint":
        gradient = _gradient_rows(case, seed + 1, e.n).double()
        return [_power_spectrum(case, e.coefficients, e.coefficients), *_exact_adjoint(e, gradient, True)]
    weights = _weights(case, seed + 1, torch.float32).double().to(_device())
    values = _power_spectrum(case, e.coefficients, e.coefficients)
    forces, _ = _exact_adjoint(e, weights[e.kind], False)
    energies = torch.zeros(len(e.sizes), dtype=torch.float64, device=_device())
    structure = torch.repeat_interleave(torch.arange(len(e.sizes), device=_device()), _tensor(e.sizes, torch.long))
    energies.index_add_(0, structure, (values * weights[e.kind]).flatten(1).sum(1))
    return {"values": values, "gradients": forces, "energies": energies}
