"""What the ASE calculator keeps between calls (the descriptor's calculator, a captured step, the
results of the last structure) belongs to one force field and one periodicity: another of either
gives what a fresh calculator gives.  The host logic on the CPU against a stand-in for
SO4Calculator; the values on the GPU, bit for bit."""
import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import ase_calculator as A
from pyxtal_ff_gb300 import calculator as C
from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.ase_calculator import ForceField, PyXtalFFCalculator
from pyxtal_ff_gb300.nn import NeuralNetworkPotential

NB = 14  # components at lmax 2
DESC = {"type": "SNAP", "Rc": 4.0, "cutoff": "cosine", "weights": {"Si": 1.0}, "parameters": {"lmax": 2}}


def _potential(device, seed=0):
    torch.manual_seed(seed)
    nets = {"Si": torch.nn.Sequential(torch.nn.Linear(NB, 4), torch.nn.Tanh(), torch.nn.Linear(4, 1)).double()}
    return NeuralNetworkPotential(nets, {"Si": np.stack([np.zeros(NB), np.full(NB, 2.0)], 1)}, device=device)


def _si():
    return S.diamond_si(2, 1, 1, sigma=0.05, rng=np.random.default_rng(1))


class _Step:
    def __init__(self, calc):
        self.calc = calc

    def __call__(self, positions):
        return self.calc.result(len(positions))

    def check(self):
        return True


class _Fake:
    made = []

    def __init__(self, **kw):
        self.kw, self.log = kw, []
        _Fake.made.append(self)

    def result(self, n):
        return {"energies": torch.full((n,), float(self.kw["rcut"]), dtype=torch.float64),
                "forces": torch.zeros((n, 3), dtype=torch.float64), "stress": torch.zeros((1, 6), dtype=torch.float64)}

    def compute(self, batch, model):
        self.log.append("compute")
        return self.result(batch.natoms)

    def capture(self, batch, model):
        self.log.append("capture")
        return _Step(self)


CHANGES = {"Rc": {"Rc": 3.5}, "weights": {"weights": {"Si": 0.5}}, "cutoff": {"cutoff": "tanh"},
           "rfac": {"parameters": {"lmax": 2, "rfac": 0.9}}, "normalize_U": {"parameters": {"lmax": 2, "normalize_U": True}}}


@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("change", CHANGES)
def test_another_descriptor_drops_what_was_built_for_the_old(monkeypatch, change, in_place):
    monkeypatch.setattr(C, "SO4Calculator", _Fake)
    _Fake.made = []
    pot, atoms = _potential("cpu"), _si()
    calc = PyXtalFFCalculator(ff=ForceField(DESC, pot), route="adjoint")
    for _ in range(2):
        calc.calculate(atoms)
    assert _Fake.made[0].log == ["compute", "capture"]
    if in_place:
        calc.parameters["ff"]._descriptors.update(CHANGES[change])
    else:
        calc.parameters["ff"] = ForceField({**DESC, **CHANGES[change]}, pot)
    energy = calc.get_potential_energy(atoms)
    assert len(_Fake.made) == 2 and _Fake.made[1].log == ["compute"] and _Fake.made[1].kw != _Fake.made[0].kw
    assert energy == len(atoms) * CHANGES[change].get("Rc", 4.0)
    calc.calculate(atoms)
    assert _Fake.made[1].log == ["compute", "capture"] and _Fake.made[0].log == ["compute", "capture"]


def test_periodicity_or_networks_alone_are_a_change(monkeypatch):
    monkeypatch.setattr(C, "SO4Calculator", _Fake)
    _Fake.made = []
    atoms = _si()
    calc = PyXtalFFCalculator(ff=ForceField(DESC, _potential("cpu")), route="adjoint")
    calc.get_forces(atoms)
    calc.get_stress(atoms)
    assert _Fake.made[0].log == ["compute"]
    atoms.pbc = np.array([True, True, False])
    calc.get_forces(atoms)
    assert _Fake.made[0].log == ["compute"] * 2
    calc.parameters["ff"].model.models["Si"] = _potential("cpu", 1).models["Si"]
    calc.get_forces(atoms)
    assert _Fake.made[0].log == ["compute"] * 3
    held = calc._last_key  # the objects, not their ids
    assert any(m is calc.parameters["ff"].model for m in held) and (calc.parameters["ff"].model.models["Si"],) in held


@pytest.mark.parametrize("where", ["subclass", "instance"])
def test_plain_route_asks_a_model_of_its_own(monkeypatch, where):
    """A model whose calculate_properties is not NeuralNetworkPotential's, by its class or on the object
    alone, gets the descriptors (numpy) and gives the results."""
    class Mine(NeuralNetworkPotential):
        def calculate_properties(self, descriptor, bforce=True, bstress=False):
            return np.full(2, descriptor["x"]), np.ones((2, 3)), np.zeros(6)

    base = _potential("cpu")
    if where == "subclass":
        model = Mine(base.models, base.drange, device="cpu")
    else:
        model = base
        model.calculate_properties = lambda d, bforce=True, bstress=False: Mine.calculate_properties(model, d)
    monkeypatch.setattr(A, "compute_descriptor", lambda function, atoms: {"x": 3.5})
    calc, atoms = PyXtalFFCalculator(ff=ForceField(DESC, model)), S.Atoms([14] * 2, np.eye(3)[:2], 9 * np.eye(3))
    assert calc.get_potential_energy(atoms) == 7.0 and np.array_equal(calc.get_forces(atoms), np.ones((2, 3)))


@pytest.mark.gpu
@pytest.mark.parametrize("route", ["plain", "adjoint"])
def test_changes_equal_a_fresh_calculator(cuda_device, route):
    pot, atoms = _potential("cuda"), _si()
    calc = PyXtalFFCalculator(ff=ForceField(DESC, pot), route=route)

    def fresh_equal():
        got = calc.get_forces(atoms), calc.get_stress(atoms), calc.get_potential_energy(atoms)
        new = PyXtalFFCalculator(ff=calc.parameters["ff"], route=route)
        want = new.get_forces(atoms), new.get_stress(atoms), new.get_potential_energy(atoms)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
        return got[0]

    seen = [fresh_equal()]
    calc.calculate(atoms)
    calc.parameters["ff"] = ForceField({**DESC, "Rc": 4.5}, pot)
    seen.append(fresh_equal())
    calc.calculate(atoms)
    atoms.pbc = np.array([True, True, False])
    seen.append(fresh_equal())
    assert not np.array_equal(seen[0], seen[1]) and not np.array_equal(seen[1], seen[2])
