"""Performance cases: the work users of this package have it do.

A case is a dict of plain values. Its "kind" says which public entry point it
goes through; the other fields are sizes, types and options:

  contract   one pairwise contraction of large labelled tensors whose axes
             interleave (capi.contract); also closing steps, whose output is a
             few values over a long contracted range
  gate       a q-site gate applied to a state-like tensor (capi.contract)
  transpose  an axis permutation (capi.permute)
  amplitude  a circuit amplitude, one TaskBasedContractor contracted repeatedly
  sliced     a circuit amplitude as the sum of all slices (SlicedContractor)
  gradient   an expectation value and its gradient in every angle
             (autograd.contract_network in an autograd.GraphedStep)

`listed` are the standing cases, `draw` gives more of the same ranges,
`prepare` what a program holds before the call, `run` one pass, `work` the
bytes and operations a pass cannot do without, `exact` the result in 64 bits
by plain torch and numpy."""
import functools
import math

import numpy as np
import torch

import jet_gb300 as jet
from jet_gb300 import autograd, capi, circuits, expectation

PRECISIONS = {"fp32": capi.PREC_FP32, "auto": capi.PREC_AUTO, "tf32x3": capi.PREC_TF32X3,
              "bf16x3": capi.PREC_BF16X3, "fp16x3": capi.PREC_FP16X3}
DEVICE = "cuda"


def listed():
    return [
        # The smallest whole network: a 16-qubit amplitude of a 4x4 grid, 8 cycles,
        # every step tiny, one contractor contracted again and again.
        {"name": "amplitude_16q", "kind": "amplitude", "sites": 2, "rows": 4, "cols": 4,
         "layers": 8},
        # Variational optimisation: the 6x6 grid with 10 layers and 720 angles,
        # loss and gradient per step.
        {"name": "gradient_720", "kind": "gradient", "rows": 6, "cols": 6, "layers": 10,
         "at": 3},
        # Sliced qutrit amplitude: 5x5 sites, 8 layers, 4 bonds (81 slices), 9 per batch.
        {"name": "sliced_qutrits", "kind": "sliced", "sites": 3, "rows": 5, "cols": 5,
         "layers": 8, "bonds": 4, "batch": 9, "precision": "auto"},
        # Sliced qubit amplitude whose large steps go to the tensor cores: 35 qubits,
        # 12 cycles, 4 bonds (16 slices) in one batch.
        {"name": "sliced_35q", "kind": "sliced", "sites": 2, "rows": 5, "cols": 7,
         "layers": 12, "bonds": 4, "batch": 16, "precision": "auto"},
        # The largest single contraction: rank 27 by rank 25 over 13 shared labels.
        {"name": "contract_27x25_bf16x3", "kind": "contract", "radix": 2, "m": 14, "n": 12,
         "k": 13, "precision": "bf16x3", "dtype": "complex64", "order": 1},
        # An ordinary step of a network in the AUTO form: 2048 x 1024 x 1024.
        {"name": "contract_mid_auto", "kind": "contract", "radix": 2, "m": 11, "n": 10, "k": 10,
         "precision": "auto", "dtype": "complex64", "order": 2},
        # The plain form (the default precision) on qutrits: 2187 x 2187 x 729.
        {"name": "contract_qutrit_fp32", "kind": "contract", "radix": 3, "m": 7, "n": 7, "k": 6,
         "precision": "fp32", "dtype": "complex64", "order": 3},
        # The default element type of the package, ragged extents.
        {"name": "contract_c128", "kind": "contract", "radix": 0, "m": 900, "n": 770, "k": 515,
         "precision": "fp32", "dtype": "complex128", "order": 4},
        # The closing step of a whole-network amplitude: 16 x 32 outputs over 2^21.
        {"name": "closing_16x32", "kind": "contract", "radix": 2, "m": 4, "n": 5, "k": 21,
         "precision": "fp32", "dtype": "complex64", "order": 5},
        # A two-qubit gate on a 26-qubit tensor: most steps of sliced benchmark networks.
        {"name": "gate_2of26", "kind": "gate", "radix": 2, "axes": 26, "on": 2,
         "dtype": "complex64", "order": 6},
        # A four-qubit block on a 24-qubit tensor (fused gates, 16 wide).
        {"name": "gate_4of24", "kind": "gate", "radix": 2, "axes": 24, "on": 4,
         "dtype": "complex64", "order": 7},
        # The transpose of a qutrit tensor (no bit permutation).
        {"name": "transpose_3x16", "kind": "transpose", "radix": 3, "axes": 16,
         "dtype": "complex64", "order": 8},
    ]


def draw(rng):
    kind = rng.choice(["contract", "contract", "contract", "closing", "gate", "gate", "transpose",
                       "amplitude", "sliced", "gradient"])
    order = rng.randrange(1 << 20)
    if kind == "contract":
        # Up to 2^37 multiply-adds on the tensor cores, 2^34 in the plain
        # form, 2^30 in complex128; operands up to 2^26 elements.
        form, top = rng.choice([("fp32", 34), ("auto", 37), ("bf16x3", 37), ("fp16x3", 37),
                                ("tf32x3", 36), ("c128", 30)])
        total = rng.uniform(18, top)
        cut = [rng.uniform(0.6, 1.4) for _ in range(3)]
        bits = [total * c / sum(cut) for c in cut]
        over = max(0.0, max(bits[0], bits[1]) + bits[2] - 26)
        bits = [max(2.0, b - over / 2) for b in bits]
        radix = rng.choice([2, 2, 3, 0])
        if radix:
            m, n, k = (max(1, int(b / math.log2(radix))) for b in bits)
        else:
            m, n, k = (max(2, int(2.0 ** b)) for b in bits)
        return {"kind": "contract", "radix": radix, "m": m, "n": n, "k": k,
                "precision": "fp32" if form == "c128" else form,
                "dtype": "complex128" if form == "c128" else "complex64", "order": order}
    if kind == "closing":
        dtype = rng.choice(["complex64", "complex64", "complex128"])
        return {"kind": "contract", "radix": 2, "m": rng.randint(0, 4), "n": rng.randint(0, 5),
                "k": rng.randint(10, 21 if dtype == "complex64" else 17), "precision": "fp32",
                "dtype": dtype, "order": order}
    if kind == "gate":
        radix = rng.choice([2, 2, 3])
        on = rng.randint(1, 4 if radix == 2 else 2)
        dtype = rng.choice(["complex64", "complex64", "complex128"])
        top = 26 if dtype == "complex64" else 22
        return {"kind": "gate", "radix": radix,
                "axes": int(rng.uniform(10, top) / math.log2(radix)), "on": on, "dtype": dtype,
                "order": order}
    if kind == "transpose":
        radix = rng.choice([2, 2, 3, 5])
        dtype = rng.choice(["complex64", "complex64", "complex128"])
        return {"kind": "transpose", "radix": radix,
                "axes": int(rng.uniform(10, 27 if dtype == "complex64" else 25)
                            / math.log2(radix)), "dtype": dtype, "order": order}
    if kind == "amplitude":
        sites = rng.choice([2, 2, 3])
        return {"kind": "amplitude", "sites": sites, "rows": rng.randint(3, 4),
                "cols": rng.randint(3, 5 if sites == 2 else 4), "layers": rng.randint(4, 9)}
    if kind == "sliced":
        sites = rng.choice([2, 3])
        return {"kind": "sliced", "sites": sites, "rows": 5 if sites == 2 else 4,
                "cols": rng.randint(4, 6) if sites == 2 else 4,
                "layers": rng.randint(8, 10) if sites == 2 else rng.randint(6, 8),
                "bonds": rng.randint(2, 4) if sites == 2 else 2, "batch": sites * sites,
                "precision": rng.choice(["auto", "fp32"])}
    rows, cols = rng.randint(3, 4), rng.randint(3, 5)
    return {"kind": "gradient", "rows": rows, "cols": cols, "layers": rng.randint(4, 7),
            "at": rng.randrange(rows) * cols + rng.randrange(cols - 1)}


# --- single contractions, gates and transposes -------------------------------


def _axes_of(case):
    """Operands of a contract or gate case: (A shape, A order, B shape, B
    order, m, n, k). An order lists the operand's axes as the product reads
    them: free then contracted for A, contracted then free for B. The axes lie
    in memory in an order seeded by the case."""
    rng = np.random.default_rng(case["order"])
    if case["kind"] == "gate":
        r, q = case["radix"], case["on"]
        on = [int(x) for x in rng.permutation(case["axes"])[:q]]
        rest = [x for x in range(case["axes"]) if x not in on]
        return ([r] * case["axes"], rest + on, [r] * (2 * q), list(range(2 * q)),
                r ** len(rest), r ** q, r ** q)
    if case["radix"] == 0:  # one axis each, both operands stored transposed
        m, n, k = case["m"], case["n"], case["k"]
        return [k, m], [1, 0], [n, k], [1, 0], m, n, k
    r, (m, n, k) = case["radix"], (case["m"], case["n"], case["k"])
    pa = [int(x) for x in rng.permutation(m + k)]
    pb = [int(x) for x in rng.permutation(k + n)]
    return [r] * (m + k), pa, [r] * (k + n), pb, r ** m, r ** n, r ** k


def _normal(gen, n, dtype, scale):
    """n complex values, real and imaginary parts N(0, scale^2)."""
    real = torch.float32 if dtype == "complex64" else torch.float64
    x = torch.randn(2 * n, generator=gen, device=DEVICE, dtype=real)
    return torch.view_as_complex(x.mul_(scale).reshape(n, 2))


def _operands(case, seed):
    a_shape, _, b_shape, _, _, _, _ = _axes_of(case)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    na, nb = math.prod(a_shape), math.prod(b_shape)
    if case["kind"] == "gate":  # a normalised state and a unitary
        d = math.isqrt(nb)
        a = _normal(gen, na, case["dtype"], math.sqrt(0.5 / na))
        b = torch.from_numpy(_unitary(np.random.default_rng(seed), d).reshape(-1))
        return a, b.to(DEVICE, a.dtype)
    scale = math.sqrt(0.5) * 2.0 ** -10
    return _normal(gen, na, case["dtype"], scale), _normal(gen, nb, case["dtype"], scale)


# --- circuits ----------------------------------------------------------------


def _grid_pairs(rows, cols, layer):
    """The coupled neighbours of a layer: horizontal pairs from even, then odd
    columns, vertical pairs from even, then odd rows."""
    p, out = layer % 4, []
    for r in range(rows):
        for c in range(cols):
            if p < 2 and c % 2 == p and c + 1 < cols:
                out.append((r * cols + c, r * cols + c + 1))
            if p >= 2 and r % 2 == p - 2 and r + 1 < rows:
                out.append((r * cols + c, (r + 1) * cols + c))
    return out


def _unitary(rng, d):
    q, r = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _circuit(case, seed):
    """The leaves (labels, shape, complex128 values) of <x| C |0...0> with a
    seeded output x: square roots of X, Y, W and fSim gates on qubits, random
    unitaries on qutrits."""
    rng = np.random.default_rng(seed)
    d, n = case["sites"], case["rows"] * case["cols"]
    w = np.array([[0, np.exp(-0.25j * np.pi)], [np.exp(0.25j * np.pi), 0]])
    singles = [(np.eye(2) - 1j * g) / math.sqrt(2)
               for g in (np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), w)]
    fsim = np.array([[1, 0, 0, 0], [0, 0, -1j, 0], [0, -1j, 0, 0],
                     [0, 0, 0, np.exp(-1j * np.pi / 6)]])
    at, leaves, last = [0] * n, [], [-1] * n

    def label(q):
        return "q%d_%d" % (q, at[q])

    def put(qs, matrix):
        ins = [label(q) for q in qs]
        for q in qs:
            at[q] += 1
        leaves.append(([label(q) for q in qs] + ins, [d] * (2 * len(qs)), matrix.reshape(-1)))

    for q in range(n):
        leaves.append(([label(q)], [d], np.eye(d, dtype=complex)[0]))
    for layer in range(case["layers"]):
        for q in range(n):
            if d == 2:
                last[q] = int(rng.choice([g for g in range(3) if g != last[q]]))
            put([q], singles[last[q]] if d == 2 else _unitary(rng, d))
        for pair in _grid_pairs(case["rows"], case["cols"], layer):
            put(list(pair), fsim if d == 2 else _unitary(rng, d * d))
    for q in range(n):
        leaves.append(([label(q)], [d], np.eye(d, dtype=complex)[int(rng.integers(d))]))
    return leaves


def _frozen(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "precision")))


@functools.lru_cache(maxsize=None)
def _circuit_plan(frozen):
    """(path, sliced bonds) of a circuit: the same for every seed, as the
    network's labels and shapes are."""
    case = dict(frozen)
    net = circuits.Network(_circuit(case, 0))
    path = circuits.best_gain_path(net, 16)
    return path, circuits.choose_slices(net, path, case["bonds"]) if "bonds" in case else []


def _network(case, seed):
    tn = jet.TensorNetwork(dtype="complex64")
    for labels, shape, values in _circuit(case, seed):
        tn.add_tensor(jet.Tensor(indices=labels, shape=shape,
                                 data=list(values.astype(np.complex64)), dtype="complex64"))
    return tn


@functools.lru_cache(maxsize=None)
def _gradient_plan(rows, cols, layers, at):
    """(leaves, path) of the light-cone network of <Z_i Z_j>, i = at, j = at + 1."""
    leaves = expectation.zz_network(rows, cols, layers, (at, at + 1))
    zero = np.zeros((layers, rows * cols))
    net = expectation.numeric_network(leaves, zero, zero)
    return leaves, circuits.find_path(net, restarts=8, seed=20240601)


def _angles(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    shape = (2, case["layers"], case["rows"] * case["cols"])
    return torch.rand(shape, generator=gen, device=DEVICE) * (2 * math.pi)


# --- the cases ---------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("contract", "gate"):
        a_shape, a_order, b_shape, b_order, m, n, k = _axes_of(case)
        a, b = _operands(case, seed)
        prec = PRECISIONS[case.get("precision", "fp32")]
        return kind, (a, a_shape, a_order, b, b_shape, b_order, m, n, k, prec)
    if kind == "transpose":
        shape = [case["radix"]] * case["axes"]
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        order = [int(x) for x in np.random.default_rng(case["order"]).permutation(case["axes"])]
        return kind, (_normal(gen, math.prod(shape), case["dtype"], 1.0), shape, order)
    if kind == "amplitude":
        path, _ = _circuit_plan(_frozen(case))
        tn = _network(case, seed)
        tbc = jet.TaskBasedContractor(dtype="complex64")
        tbc.add_contraction_tasks(tn, jet.PathInfo(tn, path))
        tbc.add_deletion_tasks()
        return kind, tbc
    if kind == "sliced":
        path, bonds = _circuit_plan(_frozen(case))
        sc = jet.SlicedContractorC64(_network(case, seed), path, bonds,
                                     PRECISIONS[case["precision"]])
        sc.set_batch_size(case["batch"])
        return kind, sc
    leaves, path = _gradient_plan(case["rows"], case["cols"], case["layers"], case["at"])
    labels = [leaf.labels for leaf in leaves]
    plan = autograd.ContractionPlan(labels, [leaf.shape for leaf in leaves], path)
    thetas, phis = (x.clone().requires_grad_() for x in _angles(case, seed))
    consts = {}

    def loss():
        tensors = expectation.build_leaves(leaves, thetas, phis, dtype=torch.complex64,
                                           device=DEVICE, const_cache=consts)
        return autograd.contract_network(tensors, labels, path, precision=capi.PREC_AUTO,
                                         plan=plan).real

    return kind, autograd.GraphedStep(loss, [thetas, phis])


def run(state):
    kind, s = state
    if kind in ("contract", "gate"):
        a, a_shape, a_order, b, b_shape, b_order, m, n, k, prec = s
        return capi.contract(a, a_shape, a_order, b, b_shape, b_order, m, n, k, precision=prec)
    if kind == "transpose":
        return capi.permute(*s)
    if kind == "amplitude":
        s.contract()
        return np.array(s.results[0].data, dtype=np.complex64)
    if kind == "sliced":
        return np.array(s.contract())
    loss = s.step()
    return [loss] + s.grads


def work(case):
    kind = case["kind"]
    if kind in ("contract", "gate"):
        a_shape, _, b_shape, _, m, n, k = _axes_of(case)
        size = 8 if case["dtype"] == "complex64" else 16
        return {"bytes": size * (math.prod(a_shape) + math.prod(b_shape) + m * n),
                "flops": 8 * m * n * k}
    if kind == "transpose":
        size = 8 if case["dtype"] == "complex64" else 16
        return {"bytes": 2 * size * case["radix"] ** case["axes"], "flops": 0}
    # Networks: eight operations per complex multiply-add of the path, every
    # slice of it; the leaves and the result are what must be read and written.
    if kind == "gradient":  # the value, and two contractions per step for the gradient
        leaves, path = _gradient_plan(case["rows"], case["cols"], case["layers"], case["at"])
        net = circuits.Network([(leaf.labels, leaf.shape, None) for leaf in leaves])
        angles = 2 * case["layers"] * case["rows"] * case["cols"]
        return {"bytes": 2 * 4 * angles, "flops": 3 * 4 * circuits.path_cost(net, path)[0]}
    path, bonds = _circuit_plan(_frozen(case))
    net = circuits.Network(_circuit(case, 0))
    flops = 4 * circuits.path_cost(net, path, bonds)[0] * case["sites"] ** len(bonds)
    return {"bytes": 8 * sum(math.prod(s) for _, s, _ in net.tensors), "flops": flops}


# --- 64-bit results ----------------------------------------------------------


def _greedy(labels, dims, seed):
    """A greedy order (pairs of node numbers) and its multiply-adds."""
    rng = np.random.default_rng(seed)
    nodes = {i: set(x) for i, x in enumerate(labels)}
    path, cost, new = [], 0.0, len(labels)

    def size(x):
        return math.prod(float(dims[i]) for i in x)

    def score(i, j):
        s = size(nodes[i] ^ nodes[j]) - size(nodes[i]) - size(nodes[j])
        return (math.copysign(math.log2(abs(s) + 1), s) - 0.2 * math.log(rng.exponential()), i, j)

    def next_to(i):
        return [j for j in nodes if j != i and nodes[i] & nodes[j]]

    todo = [score(i, j) for i in nodes for j in next_to(i) if i < j]
    while len(nodes) > 1:
        todo = [t for t in todo if t[1] in nodes and t[2] in nodes]
        # what is left may be scalars of separate pieces
        _, i, j = min(todo) if todo else (0, *list(nodes)[:2])
        cost += size(nodes[i] | nodes[j])
        nodes[new] = nodes.pop(i) ^ nodes.pop(j)
        path.append((i, j))
        todo += [score(x, new) for x in next_to(new)]
        new += 1
    return path, cost


def _contract64(labels, tensors):
    """The scalar that a closed network contracts to, in plain torch."""
    dims = {x: d for lab, t in zip(labels, tensors) for x, d in zip(lab, t.shape)}
    path, _ = min((_greedy(labels, dims, s) for s in range(8)), key=lambda p: p[1])
    nodes = {i: (list(lab), t) for i, (lab, t) in enumerate(zip(labels, tensors))}
    for new, (i, j) in enumerate(path, len(labels)):
        (la, a), (lb, b) = nodes.pop(i), nodes.pop(j)
        both = [x for x in la if x in lb]
        t = torch.tensordot(a, b, dims=([la.index(x) for x in both], [lb.index(x) for x in both]))
        nodes[new] = ([x for x in la + lb if x not in both], t)
    return nodes[len(labels) + len(path) - 1][1]


def _expectation64(case, angles):
    """Re <psi| Z_i Z_j |psi> of the circuit of RX, RZ and CZ layers, every
    gate outside the pair's light cone left out."""
    rows, cols, layers = case["rows"], case["cols"], case["layers"]
    pair = (case["at"], case["at"] + 1)
    cone, kept = set(pair), []
    for layer in reversed(range(layers)):
        pairs = [p for p in _grid_pairs(rows, cols, layer) if p[0] in cone or p[1] in cone]
        cone |= {q for p in pairs for q in p}
        kept.insert(0, (pairs, sorted(cone)))
    labels, tensors, at = [], [], {q: 0 for q in cone}
    zero = torch.tensor([1, 0], dtype=torch.complex128, device=DEVICE)
    cz = torch.diag(torch.tensor([1, 1, 1, -1], dtype=torch.complex128, device=DEVICE))
    off = torch.tensor([[0, 1], [1, 0]], dtype=torch.complex128, device=DEVICE)
    eye = torch.eye(2, dtype=torch.complex128, device=DEVICE)
    z = torch.diag(torch.tensor([1, -1], dtype=torch.complex128, device=DEVICE))

    def put(qs, t):
        for side, x in (("k", t), ("b", t.conj())):
            labels.append(["%s%d_%d" % (side, q, at[q] + 1) for q in qs]
                          + ["%s%d_%d" % (side, q, at[q]) for q in qs])
            tensors.append(x)
        for q in qs:
            at[q] += 1

    for q in cone:
        for side in "kb":
            labels.append(["%s%d_0" % (side, q)])
            tensors.append(zero)
    for layer, (pairs, active) in enumerate(kept):
        for q in active:
            t, p = angles[0][layer, q] / 2, angles[1][layer, q] / 2
            put([q], torch.cos(t) * eye - 1j * torch.sin(t) * off)
            put([q], torch.cos(p) * eye - 1j * torch.sin(p) * z)
        for p in pairs:
            put(list(p), cz.reshape(2, 2, 2, 2))
    for q in cone:
        labels.append(["b%d_%d" % (q, at[q]), "k%d_%d" % (q, at[q])])
        tensors.append(z if q in pair else eye)
    return _contract64(labels, tensors).real


def exact(case, seed):
    kind = case["kind"]
    if kind in ("contract", "gate"):
        a_shape, a_order, b_shape, b_order, m, n, k = _axes_of(case)
        a, b = _operands(case, seed)
        a = a.to(torch.complex128).reshape(a_shape).permute(a_order).reshape(m, k)
        b = b.to(torch.complex128).reshape(b_shape).permute(b_order).reshape(k, n)
        return (a @ b).reshape(-1)
    if kind == "transpose":
        _, (x, shape, order) = prepare(case, seed)
        return x.reshape(shape).permute(order).reshape(-1).to(torch.complex128)
    if kind == "gradient":
        angles = [x.double().requires_grad_() for x in _angles(case, seed)]
        value = _expectation64(case, angles)
        value.backward()
        return [value.detach()] + [x.grad for x in angles]
    leaves = _circuit(case, seed)
    # the values as the contraction gets them: rounded to complex64
    tensors = [torch.from_numpy(v.astype(np.complex64)).to(DEVICE, torch.complex128).reshape(s)
               for _, s, v in leaves]
    return _contract64([lab for lab, _, _ in leaves], tensors).reshape(1).cpu().numpy()
