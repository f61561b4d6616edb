"""Performance cases of the five operations, through the entry points a program calls.

A case is one operation with its sizes, the scalar type, the front end and what one pass does:

* ``api``: ``"torch"`` calls ``torch.ops.mops.*`` and takes gradients through autograd, as a
  model does; ``"plain"`` calls the functions of ``mops_b200`` on CUDA tensors; ``"plan"`` the
  same inside a ``Plan`` the program keeps for its graph (molecular dynamics, or an epoch over
  fixed structures).
* ``do``: ``"fwd"`` (inference), ``"vjp"`` (a backward call on its own), ``"both"`` (forward and
  backward: a training step, or energies with forces) and ``"second"`` (training on forces: the
  backward is itself differentiated; the torch operators that have second derivatives).
* ``sorted``: whether the scatter index is in ascending order, as a neighbour list by centre
  is, or in the order some other program left it.

Values are drawn as ``mops_b200.workloads`` draws them (but on the GPU, from the seed alone):
coefficients and operands of unit scale, scatter indices uniform over the output rows, so that
rows receive about Poisson-distributed numbers of entries and a few stay empty.
"""
import torch

import mops_b200
import mops_b200.torch  # noqa: F401  (registers torch.ops.mops)

OP = {"hpe": "homogeneous_polynomial_evaluation", "sap": "sparse_accumulation_of_products",
      "opsa": "outer_product_scatter_add", "opsaw": "outer_product_scatter_add_with_weights",
      "sasaw": "sparse_accumulation_scatter_add_with_weights"}
SECOND = ("hpe", "sap", "opsa")  # operations with second derivatives

# Work of one pass, in float operations, that a drawn case may have at most (the largest listed
# case has more), and entries of one operand, so that a state stays within a few GB.
MOST_FLOPS = 4e10
MOST_VALUES = 4e8




def listed():
    return [
        # an epoch over small batches: the benchmark size of the polynomial evaluation
        dict(name="hpe_train_small", op="hpe", api="torch", do="both", dtype="f64",
             I=1000, N=100, J=2000, K=4),
        # the same polynomials for every atom of a large cell
        dict(name="hpe_large", op="hpe", api="plain", do="both", dtype="f64",
             I=1 << 20, N=100, J=2000, K=4),
        # training on forces with the contraction of two features: first and second derivatives
        dict(name="sap_forces_small", op="sap", api="torch", do="second", dtype="f64",
             I=1000, nA=20, nB=6, nO=50, K=1000),
        # the contraction over every atom of a large batch
        dict(name="sap_large", op="sap", api="plain", do="both", dtype="f64",
             I=1 << 22, nA=20, nB=6, nO=50, K=1000),
        # one molecule in inference: nothing but latency
        dict(name="opsa_molecule", op="opsa", api="torch", do="fwd", dtype="f32",
             E=420, n=21, K=13, L=20, sorted=True),
        # a ragged batch of structures with odd channel counts, in double precision
        dict(name="opsa_ragged_f64", op="opsa", api="torch", do="both", dtype="f64",
             E=3000017, n=50021, K=7, L=25, sorted=True),
        # density expansion of a very large batch in single precision
        dict(name="opsa_large_f32", op="opsa", api="torch", do="both", dtype="f32",
             E=1 << 24, n=1 << 18, K=13, L=20, sorted=True),
        # message passing, one small batch of structures
        dict(name="opsaw_train_small", op="opsaw", api="torch", do="both", dtype="f64",
             E=60000, n=1000, K=13, L=32, sorted=True),
        # an edge list that nobody sorted, with the 4x4 spherical harmonics, single precision
        dict(name="opsaw_unsorted_f32", op="opsaw", api="plain", do="both", dtype="f32",
             E=300007, n=5003, K=16, L=32, sorted=False),
        # equivariant message passing: a molecular-dynamics step that keeps its plan
        dict(name="sasaw_md_plan", op="sasaw", api="plan", do="both", dtype="f64",
             E=60000, n=1000, nA=9, nW=9, nO=9, L=32, N=500, sorted=True),
        # its training in single precision with wider channels
        dict(name="sasaw_train_f32", op="sasaw", api="torch", do="both", dtype="f32",
             E=250001, n=4099, nA=9, nW=9, nO=9, L=64, N=500, sorted=True),
        # and over a graph whose weights are larger than the L2 cache
        dict(name="sasaw_large", op="sasaw", api="plain", do="both", dtype="f64",
             E=1 << 22, n=1 << 16, nA=9, nW=9, nO=9, L=32, N=500, sorted=True),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    while True:
        op = rng.choice(("hpe", "sap", "opsa", "opsaw", "sasaw"))
        api = rng.choice(("torch", "torch", "plain", "plan"))
        do = ["fwd", "both", "both"]
        if api == "torch" and op in SECOND:
            do.append("second")
        if api != "torch":
            do.append("vjp")
        c = dict(op=op, api=api, do=rng.choice(do), dtype=rng.choice(("f64", "f32")))
        if op == "hpe":
            c.update(I=log(30, 1 << 20), N=log(10, 200), J=log(50, 4000), K=rng.randint(1, 5))
        elif op == "sap":
            c.update(I=log(30, 1 << 22), nA=rng.randint(4, 32), nB=rng.randint(1, 16),
                     nO=log(5, 100), K=log(30, 2000))
        else:
            # 10 to 100 entries per output row; one index in eight is not sorted
            c.update(E=log(200, 1 << 24 if op == "opsa" else 1 << 22))
            c.update(n=max(2, int(c["E"] / rng.uniform(10, 100))))
            c.update(sorted=rng.random() >= 0.125)
            if op == "sasaw":
                # angular channels up to l = 1, 2, 3, or an odd count
                nA, nW, nO = (rng.choice((4, 9, 9, 16, rng.randint(2, 16))) for _ in range(3))
                c.update(nA=nA, nW=nW, nO=nO, L=rng.choice((8, 16, 32, 32, 64, rng.randint(5, 100))),
                         N=log(30, 1000))
            else:
                c.update(K=rng.randint(1, 18), L=rng.choice((rng.randint(2, 40), 32, 64)))
        w = work(c)
        if w["flops"] <= MOST_FLOPS and _values(c) <= MOST_VALUES:
            return c


def _values(c):
    """Scalars of the largest operand or result."""
    if c["op"] == "hpe":
        return c["I"] * c["N"]
    if c["op"] == "sap":
        return c["I"] * max(c["nA"], c["nB"], c["nO"])
    if c["op"] == "sasaw":
        return max(c["E"] * max(c["nA"], c["L"]), c["n"] * max(c["nW"], c["nO"]) * c["L"])
    return max(c["E"] * max(c["K"], c["L"]), c["n"] * c["K"] * c["L"])


class State:
    """What a program holds before the call: operands, index arrays, gradients, its plan."""

    def __init__(self, case, seed):
        self.op, self.api, self.do = case["op"], case["api"], case["do"]
        real = torch.float64 if case["dtype"] == "f64" else torch.float32
        g = torch.Generator(device="cuda").manual_seed(seed)

        def normal(*shape):
            return torch.randn(*shape, dtype=real, device="cuda", generator=g)

        def uniform(*shape):
            return torch.rand(*shape, dtype=real, device="cuda", generator=g).mul_(2).sub_(1)

        def index(n, *shape, ascending=False):
            i = torch.randint(n, shape, dtype=torch.int32, device="cuda", generator=g)
            return torch.sort(i).values if ascending else i

        c = case
        if self.op == "hpe":
            self.operands = [uniform(c["I"], c["N"])]
            self.args = self.operands + [normal(c["J"]), index(c["N"], c["J"], c["K"])]
            self.size = []
            out = (c["I"],)
        elif self.op == "sap":
            self.operands = [uniform(c["I"], c["nA"]), uniform(c["I"], c["nB"])]
            self.args = self.operands + [normal(c["K"]), index(c["nA"], c["K"]),
                                         index(c["nB"], c["K"]),
                                         index(c["nO"], c["K"], ascending=True)]
            self.size = [c["nO"]]
            out = (c["I"], c["nO"])
        elif self.op == "opsa":
            self.operands = [normal(c["E"], c["K"]), normal(c["E"], c["L"])]
            self.args = self.operands + [index(c["n"], c["E"], ascending=c["sorted"])]
            self.size = [c["n"]]
            out = (c["n"], c["K"], c["L"])
        elif self.op == "opsaw":
            self.operands = [normal(c["E"], c["K"]), normal(c["E"], c["L"]), normal(c["n"], c["L"])]
            self.args = self.operands + [index(c["n"], c["E"]),
                                         index(c["n"], c["E"], ascending=c["sorted"])]
            self.size = []
            out = (c["n"], c["K"], c["L"])
        else:
            A, B = normal(c["E"], c["nA"]), normal(c["E"], c["L"])
            W = normal(c["n"], c["nW"], c["L"])
            self.operands = [A, B, W]
            self.args = [A, B, normal(c["N"]), W, index(c["nA"], c["N"]), index(c["n"], c["E"]),
                         index(c["nW"], c["N"]), index(c["n"], c["E"], ascending=c["sorted"]),
                         index(c["nO"], c["N"], ascending=True)]
            self.size = [c["nO"]]
            out = (c["n"], c["nO"], c["L"])

        self.grad_output = normal(*out) if self.do != "fwd" else None
        self.second = [normal(*x.shape) for x in self.operands] if self.do == "second" else None
        if self.api == "torch":
            self.forward = getattr(torch.ops.mops, OP[self.op])
            if self.do != "fwd":
                for x in self.operands:
                    x.requires_grad_(True)
            if self.do == "second":
                self.grad_output.requires_grad_(True)
        else:
            self.forward = getattr(mops_b200, OP[self.op])
            self.backward = getattr(mops_b200, OP[self.op] + "_vjp")
            self.plan = mops_b200.Plan() if self.api == "plan" else None


def prepare(case, seed):
    return State(case, seed)


def _calls(s):
    out = []
    if s.do in ("fwd", "both"):
        out.append(s.forward(*s.args, *s.size))
    if s.do in ("vjp", "both"):
        grads = s.backward(s.grad_output, *s.args)
        out += grads if isinstance(grads, tuple) else [grads]
    return out


def run(s):
    if s.api == "plain":
        return _calls(s)
    if s.api == "plan":
        with s.plan:
            return _calls(s)
    out = s.forward(*s.args, *s.size)
    if s.do == "fwd":
        return [out]
    if s.do == "both":
        return [out, *torch.autograd.grad(out, s.operands, s.grad_output)]
    grads = torch.autograd.grad(out, s.operands, s.grad_output, create_graph=True)
    more = torch.autograd.grad(grads, [s.grad_output, *s.operands], s.second)
    return [out, *[x.detach() for x in grads], *more]


def work(case):
    """Bytes and float operations that the calls of one pass need: every call reads its operands
    once and writes its results once (the calls are separate, and their operands are in general
    larger than the caches), gathered rows of W counted once; multiplications of a product
    shared where the mathematics shares them (the gradients of a monomial cost three of it)."""
    c, op = case, case["op"]
    s = 8 if c["dtype"] == "f64" else 4
    if op == "hpe":
        I, N, J, K = c["I"], c["N"], c["J"], c["K"]
        inputs, table, outputs, terms = s * I * N, J * (s + 4 * K), s * I, I * J
        flops = [terms * (K + 1), terms * 3 * K, terms * 6 * K]
    elif op == "sap":
        I, K = c["I"], c["K"]
        inputs, table, outputs = s * I * (c["nA"] + c["nB"]), K * (s + 12), s * I * c["nO"]
        flops = [I * K * 3, I * K * 5, I * K * 9]
    elif op in ("opsa", "opsaw"):
        E, K, L, n = c["E"], c["K"], c["L"], c["n"]
        w = op == "opsaw"
        inputs = s * E * (K + L) + (s * n * L if w else 0)
        table, outputs = E * (8 if w else 4), s * n * K * L
        flops = [2 * E * K * L + (E * L if w else 0), 4 * E * K * L + (3 * E * L if w else 0),
                 8 * E * K * L]
    else:
        E, n, L, N, nA, nW, nO = (c[k] for k in ("E", "n", "L", "N", "nA", "nW", "nO"))
        inputs = s * E * (nA + L) + s * n * nW * L
        table, outputs = 8 * E + N * (s + 12), s * n * nO * L
        # the coupling contracted with the edge's A row first, then applied to its L channels
        cells = min(N, nW * nO)
        contract, product = 2 * min(N, cells * nA), 2 * cells * L
        flops = [E * (contract + product + nW * L),
                 E * (2 * contract + 2 * product + 3 * nW * L), 0]
    size = {"fwd": inputs + table + outputs, "vjp": 2 * inputs + table + outputs}
    # operands, directions and grad_output in; second gradients of all of them out
    second = 3 * inputs + table + 2 * outputs
    if c["do"] == "second":
        return {"bytes": float(size["fwd"] + size["vjp"] + second), "flops": float(sum(flops))}
    if c["do"] == "both":
        return {"bytes": float(size["fwd"] + size["vjp"]), "flops": float(flops[0] + flops[1])}
    return {"bytes": float(size[c["do"]]), "flops": float(flops[0 if c["do"] == "fwd" else 1])}


def tolerance(case):
    """Sums of some tens to thousands of products in another order, at the scalar's precision."""
    return {"rel": 1e-12} if case["dtype"] == "f64" else {"rel": 1e-5}
