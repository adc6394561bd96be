"""The work that a user of this framework has it do, as measurable cases.

A case names one way into the framework (``"kind"``) and the sizes of one pass through it:

``ops``       the ``ani_mod`` operators on a device-resident batch: sort, features, coordinate gradient
``forces``    energies + forces of a resident batch through ``EnergyForces`` (molecular dynamics, screening)
``server``    one request of the energy server: one geometry in, energy + gradient out
``steps``     training steps over a pool of device-resident batches (``StepPipeline``)
``epoch``     one training epoch over a host data set (``feed_dataset`` as ``train()`` calls it)
``predict``   energies of a host data set (``TrainerMultiTower.predict``)
``gradients`` per-molecule energy gradients of a host data set (``coordinate_gradients``)
``fit_forces`` training on forces, which differentiates the gradient once more (``train_op_forces``)

Molecules are synthetic, of two shapes: ``gdb`` (random walks of up to ``heavy`` heavy atoms with the
hydrogens that fill their valences, bond lengths and angles of the ANI-1 GDB sets, coordinates
perturbed by 0.05 A) and ``large`` (64 to 256 atoms at 0.1 atoms per cubic Angstrom, no two closer
than 0.9 A).  The sizes and elements of the molecules belong to the case, so that its shapes do; the
coordinates, targets and weights come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from khan_b200 import EnergyForces, FlatNadam, FusedTrainStep, RawDataset, TrainerMultiTower, ani_mod, energy_server
from khan_b200.model import activations
from khan_b200.model.nn import MoleculeNN
from khan_b200.staged import StagedBatch
from khan_b200.training.fused_step import StepPipeline

FEATURES = 384
LAYERS = (128, 128, 64, 1)          # what TrainerMultiGPU and the energy server build
PARAMETERS = 4 * (384 * 128 + 128 + 128 * 128 + 128 + 128 * 64 + 64 + 64 + 1)
NETWORK_MACS = 384 * 128 + 128 * 128 + 128 * 64 + 64     # per atom and pass
DEVICE = "cuda:0"


# ---------------------------------------------------------------------------------------------- molecules
def _unit(rng, n):
    v = rng.normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _gdb(rng, kinds, n_mols, heavy):
    """(types, xyz, counts) of ``n_mols`` walks of 1..heavy heavy atoms (a single one has ``heavy``); heavy
    atoms first, then the hydrogens, as the loaders of the ANI-1 sets give them."""
    n_heavy = np.full(1, heavy) if n_mols == 1 else kinds.integers(1, heavy + 1, n_mols)
    elem = kinds.choice(np.array([1, 2, 3]), size=(n_mols, heavy), p=[0.72, 0.14, 0.14])
    pos = np.zeros((n_mols, heavy, 3))
    for k in range(1, heavy):
        todo = np.flatnonzero(n_heavy > k)
        for _ in range(40):                       # self-avoiding: draw again where atoms come too close
            if not len(todo):
                break
            prev, bond = pos[todo, k - 1], rng.uniform(1.38, 1.54, (len(todo), 1))
            turn = _unit(rng, len(todo))
            if k > 1:
                back = pos[todo, k - 2] - prev
                back /= np.linalg.norm(back, axis=1, keepdims=True)
                side = np.cross(back, turn)
                side /= np.linalg.norm(side, axis=1, keepdims=True)
                angle = np.deg2rad(rng.uniform(105.0, 120.0, (len(todo), 1)))
                turn = np.cos(angle) * back + np.sin(angle) * side
            pos[todo, k] = prev + bond * turn
            if k < 2:
                break
            gap = np.linalg.norm(pos[todo, :k - 1] - pos[todo, k][:, None], axis=2).min(axis=1)
            todo = todo[gap <= 1.9]
    index = np.arange(heavy)[None, :]
    real = index < n_heavy[:, None]
    bonds = (index > 0).astype(int) + (index < n_heavy[:, None] - 1)
    free = np.where(real, np.maximum(np.array([0, 4, 3, 2])[elem] - bonds, 0), 0)
    mol, atom = np.nonzero(real)
    h_of = np.repeat(np.arange(len(mol)), free[real])
    h_pos = pos[mol, atom][h_of] + rng.uniform(1.0, 1.1, (len(h_of), 1)) * _unit(rng, len(h_of))
    owner = np.concatenate([mol, mol[h_of]])
    order = np.argsort(owner, kind="stable")
    types = np.concatenate([elem[real], np.zeros(len(h_of), elem.dtype)])[order].astype(np.int32)
    xyz = np.concatenate([pos[real], h_pos])[order]
    return types, xyz + rng.normal(0.0, 0.05, xyz.shape), np.bincount(owner, minlength=n_mols)


def _large(rng, kinds, n_mols):
    """(types, xyz, counts) of molecules of 64..256 atoms: points drawn one after the other in a sphere,
    the first of eight candidates that keeps 0.9 A from all earlier ones (on the GPU, all molecules at once)."""
    counts = kinds.integers(64, 257, n_mols)
    gen = torch.Generator(device=DEVICE).manual_seed(int(rng.integers(1 << 31)))
    radius = torch.from_numpy((3.0 * counts / (4.0 * np.pi * 0.1)) ** (1.0 / 3.0)).to(DEVICE)[:, None]
    pos = torch.full((n_mols, 256, 3), 1e6, dtype=torch.float64, device=DEVICE)
    for k in range(256):
        way = torch.randn(n_mols, 8, 3, generator=gen, dtype=torch.float64, device=DEVICE)
        r = radius * torch.rand(n_mols, 8, generator=gen, dtype=torch.float64, device=DEVICE) ** (1.0 / 3.0)
        cand = way / way.norm(dim=2, keepdim=True) * r[:, :, None]
        ok = (torch.cdist(cand, pos[:, :max(k, 1)]) > 0.9).all(dim=2)
        pos[:, k] = cand[torch.arange(n_mols, device=DEVICE), ok.int().argmax(dim=1)]
    xyz = pos.cpu().numpy()[np.arange(256)[None, :] < counts[:, None]]
    types = kinds.choice(np.arange(4), size=len(xyz), p=[0.5, 0.35, 0.08, 0.07]).astype(np.int32)
    return types, xyz, counts


def _molecules(case, rng, batch=0):
    """(types int32[N], xyz float64[N, 3], counts[M]) of the case's molecules."""
    kinds = np.random.default_rng([case["mols"], case.get("heavy", 0), batch])
    if case.get("shape") == "large":
        return _large(rng, kinds, case["mols"])
    return _gdb(rng, kinds, case["mols"], case["heavy"])


def _dataset(case, rng, forces=False):
    """The molecules as the host data set that the loaders build: a list of (n, 4) arrays, with targets."""
    types, xyz, counts = _molecules(case, rng)
    rows = np.concatenate([types[:, None].astype(np.float64), xyz], axis=1)
    cuts = np.cumsum(counts)[:-1]
    grads = np.split(rng.normal(0.0, 0.05, xyz.shape), cuts) if forces else None
    return RawDataset(np.split(rows, cuts), list(rng.normal(0.0, 0.1, len(counts))), grads)


def _atoms(case):
    """Mean number of atoms of one pass, and the mean radial pairs and triplets of an atom."""
    if case.get("shape") == "large":
        return 160.0 * case["mols"], 13.4, 43.8
    heavy = case["heavy"]
    if case["mols"] == 1:
        return 2.58 * heavy + 2.0, 0.71 * heavy + 2.9, 6.3 * heavy + 17.0
    return (1.32 * heavy + 3.4) * case["mols"] * case.get("batches", 1), 0.59 * heavy + 2.1, 5.2 * heavy + 9.0


# -------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # one molecule advanced step by step: energy and forces of a single geometry, bound by latency
        {"name": "forces_one_molecule", "kind": "forces", "shape": "gdb", "mols": 1, "heavy": 8},
        # a geometry optimiser that asks the energy server, which computes in double precision
        {"name": "server_request", "kind": "server", "mols": 1, "heavy": 8, "dtype": "f64"},
        # the operators on a small batch: the CPU-runnable configuration, launches and call overhead count
        {"name": "ops_64_molecules", "kind": "ops", "shape": "gdb", "mols": 64, "heavy": 8, "dtype": "f32"},
        # the operators on the training batch, the benchmark's configuration
        {"name": "ops_batch", "kind": "ops", "shape": "gdb", "mols": 1024, "heavy": 8, "dtype": "f32"},
        # the same in double precision
        {"name": "ops_batch_f64", "kind": "ops", "shape": "gdb", "mols": 1024, "heavy": 8, "dtype": "f64"},
        # the operators on molecules of 64 to 256 atoms
        {"name": "ops_large_molecules", "kind": "ops", "shape": "large", "mols": 256, "dtype": "f32"},
        # energies + forces of a batch of conformations
        {"name": "forces_batch", "kind": "forces", "shape": "gdb", "mols": 1024, "heavy": 8},
        # training on batches that stay on the GPU
        {"name": "training_steps", "kind": "steps", "mols": 1024, "heavy": 8, "batches": 8},
        # one epoch of train(): shuffled, perturbed, exp(rmse) loss, max-norm hook
        {"name": "training_epoch", "kind": "epoch", "mols": 16384, "heavy": 8, "batch_size": 1024},
        # energies of a large data set at predict's default batch size
        {"name": "predict_data_set", "kind": "predict", "mols": 32768, "heavy": 8, "batch_size": 2048},
        # gradients of a data set at coordinate_gradients' default batch size
        {"name": "gradients_data_set", "kind": "gradients", "mols": 8192, "heavy": 8, "batch_size": 1024},
        # fitting forces
        {"name": "force_training", "kind": "fit_forces", "mols": 1024, "heavy": 8, "batch_size": 256},
    ]


def draw(rng):
    def size(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["ops", "ops", "ops", "forces", "forces", "server", "steps", "epoch", "predict", "gradients",
                       "fit_forces"])
    heavy = rng.choice([6, 7, 8, 9, 10])          # GDB-6 to GDB-10: the sets of the training and the test data
    if kind == "ops":
        dtype = rng.choice(["f32", "f32", "f64"])
        if rng.random() < 0.3:
            return {"kind": kind, "shape": "large", "mols": size(2, 256), "dtype": dtype}
        return {"kind": kind, "shape": "gdb", "mols": size(8, 8192 if dtype == "f32" else 2048), "heavy": heavy,
                "dtype": dtype}
    if kind == "forces":
        if rng.random() < 0.3:
            return {"kind": kind, "shape": "large", "mols": size(1, 128)}
        return {"kind": kind, "shape": "gdb", "mols": size(1, 4096), "heavy": heavy}
    if kind == "server":
        return {"kind": kind, "mols": 1, "heavy": rng.randint(2, 10), "dtype": rng.choice(["f64", "f32"])}
    if kind == "steps":
        return {"kind": kind, "mols": size(128, 2048), "heavy": heavy, "batches": rng.randint(2, 8)}
    if kind == "epoch":
        return {"kind": kind, "mols": size(1024, 16384), "heavy": heavy, "batch_size": size(256, 2048)}
    if kind == "predict":
        return {"kind": kind, "mols": size(64, 24576), "heavy": heavy, "batch_size": size(512, 4096)}
    if kind == "gradients":
        return {"kind": kind, "mols": size(64, 8192), "heavy": heavy, "batch_size": size(256, 2048)}
    return {"kind": kind, "mols": size(128, 1024), "heavy": heavy, "batch_size": size(64, 512)}


# -------------------------------------------------------------------------------------------- preparation
def _on_gpu(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a.astype(dtype))).to(DEVICE)


def _batch_tensors(case, rng, dtype, batch=0):
    types, xyz, counts = _molecules(case, rng, batch)
    coords = [_on_gpu(xyz[:, k], dtype) for k in range(3)]
    table = [_on_gpu(types, np.int32), _on_gpu(np.cumsum(counts) - counts, np.int32), _on_gpu(counts, np.int32)]
    return coords, table, np.bincount(types, minlength=4).astype(np.int32)


def _staged(case, rng, index=0):
    """The case's molecules in a StagedBatch, as a program that keeps its batches on the GPU holds them."""
    coords, table, acs = _batch_tensors(case, rng, np.float32, index)
    batch = StagedBatch(len(coords[0]), len(table[1]), device=DEVICE)
    batch.set_shape(len(coords[0]), len(table[1]), acs)
    for to, a in zip((batch.x, batch.y, batch.z, batch.types, batch.mol_offsets, batch.mol_counts), coords + table):
        to.copy_(a)
    return batch


def _trainer(case, seed):
    dtype = torch.float64 if case.get("dtype") == "f64" else torch.float32
    trainer = TrainerMultiTower(None, [torch.device(DEVICE)], precision=dtype, layer_sizes=LAYERS, seed=seed)
    trainer.set_learning_rate(1e-5)        # as late in the schedule of train(): small changes from pass to pass
    return trainer


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = {"kind": kind, "seed": seed % (1 << 31)}
    if kind == "ops":
        dtype = np.float64 if case["dtype"] == "f64" else np.float32
        coords, table, acs = _batch_tensors(case, rng, dtype)
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        state["upstream"] = [torch.randn(int(n) * FEATURES, generator=gen, dtype=coords[0].dtype, device=DEVICE)
                             for n in acs]
        state["batch"], state["acs"] = coords + table, acs
    elif kind == "forces":
        model = MoleculeNN(device=DEVICE, seed=seed)
        state["batch"] = _staged(case, rng)
        state["evaluator"] = EnergyForces(model, state["batch"].n_atoms, state["batch"].n_mols, device=DEVICE)
    elif kind == "server":
        types, xyz, _ = _molecules(case, rng)
        state["X"] = np.concatenate([types[:, None], xyz], axis=1).tolist()
        state["trainer"] = _trainer(case, seed)
    elif kind == "steps":
        model = MoleculeNN(activation_fn=activations.gaussian, device=DEVICE, seed=seed, init="he")
        optimizer = FlatNadam(model.get_parameters(), lr=1e-5, clip_norm=5.0)
        batches = [_staged(case, rng, k) for k in range(case["batches"])]
        labels = [_on_gpu(rng.normal(size=b.n_mols), np.float32) for b in batches]
        step = FusedTrainStep(model, optimizer, max(b.n_atoms for b in batches), case["mols"], device=DEVICE)
        warm = torch.cuda.Stream(device=DEVICE)
        warm.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(warm):
            for _ in range(2):
                step.step(batches[0], labels[0])
        torch.cuda.synchronize()
        state["pipeline"] = StepPipeline(step, batches, labels)
        state["pipeline"].prime()
        state["step"], state["batches"] = step, batches
    else:
        state["data"] = _dataset(case, rng, forces=kind == "fit_forces")
        state["trainer"], state["batch_size"] = _trainer(case, seed), case["batch_size"]
    return state


def _optimizer_state(optimizer):
    return {"weights": optimizer.flat_params, "m": optimizer.m, "v": optimizer.v, "average": optimizer.ema}


def run(state):
    kind = state["kind"]
    if kind == "ops":
        batch, acs = state["batch"], state["acs"]
        scatter, gather, counts = ani_mod.ani_sort(batch[3])
        features = ani_mod.featurize(*batch, scatter, acs)
        grads = ani_mod.featurize_grad(*batch, scatter, acs, *state["upstream"])
        return {"scatter": scatter, "gather": gather, "counts": counts, "features": features, "grads": grads}
    if kind == "forces":
        batch, evaluator = state["batch"], state["evaluator"]
        evaluator.run(batch)
        return {"energies": evaluator.mol_energy[:batch.n_mols], "gradients": batch.grads[:, :batch.n_atoms]}
    if kind == "server":
        answer = energy_server.evaluate(state["trainer"], state["X"])
        return {"energy": answer["energy"], "gradient": np.array(answer["gradient"])}
    if kind == "steps":
        step, batches = state["step"], state["batches"]
        for k in range(len(batches)):
            state["pipeline"].run(k)
        return dict(_optimizer_state(step.optimizer), errors=step.l2s[:batches[-1].n_mols],
                    gradients=[b.grads[:, :b.n_atoms] for b in batches])
    trainer, data, size = state["trainer"], state["data"], state["batch_size"]
    if kind == "predict":
        return np.array(trainer.predict(data, batch_size=size))
    if kind == "gradients":
        return np.concatenate(list(trainer.coordinate_gradients(data, batch_size=size)))
    np.random.seed(state["seed"])          # feed_dataset shuffles and perturbs with numpy's global generator
    if kind == "epoch":
        rounds = trainer.feed_dataset(data, True, [trainer.train_op], size, fuzz=1e-3,
                                      before_hooks=trainer.max_norm_ops)
    else:
        rounds = trainer.feed_dataset(data, True, [trainer.train_op_forces], size)
    for _ in rounds:
        pass
    return _optimizer_state(trainer.optimizer)


# ----------------------------------------------------------------------------------- what a pass has to do
def work(case):
    """Every input read once, every result written once; operations of the pair and triplet sums (125 and
    156 for the features, 201 and 417 for their gradient) and of the atomic networks."""
    kind, size = case["kind"], 8 if case.get("dtype") == "f64" else 4
    atoms, pairs, triplets = _atoms(case)
    mols = case["mols"] * case.get("batches", 1)
    features, gradient = 125 * pairs + 156 * triplets, 201 * pairs + 417 * triplets
    inputs = atoms * (3 * size + 4) + mols * 8
    if kind == "ops":
        return {"bytes": inputs + atoms * (8 + 2 * FEATURES * size + 3 * size), "flops": atoms * (features + gradient)}
    if kind == "predict":
        return {"bytes": inputs + 4 * mols + 4 * PARAMETERS, "flops": atoms * (features + 2 * NETWORK_MACS)}
    if kind in ("forces", "server", "gradients"):
        return {"bytes": inputs + size * (mols + 3 * atoms + PARAMETERS),
                "flops": atoms * (features + gradient + 4 * NETWORK_MACS)}
    steps = case.get("batches") or math.ceil(case["mols"] / case["batch_size"])
    state = steps * PARAMETERS * 4 * 8      # weights, two moments and the moving average, read and written
    if kind == "steps":
        return {"bytes": inputs + 4 * mols + 12 * atoms + state,
                "flops": atoms * (features + gradient + 6 * NETWORK_MACS)}
    if kind == "epoch":
        backward = NETWORK_MACS + NETWORK_MACS - FEATURES * 128
        return {"bytes": inputs + 4 * mols + state, "flops": atoms * (features + 2 * (NETWORK_MACS + backward))}
    return {"bytes": inputs + 12 * atoms + state, "flops": atoms * (features + 2 * gradient + 12 * NETWORK_MACS)}


def tolerance(case):
    """Sums of 32-bit (64-bit) values over pairs and triplets; the networks multiply in three TF32 products
    (2e-5 of the largest value), and training carries that error from step to step."""
    if case.get("dtype") == "f64":
        return {"rel": 1e-11 if case["kind"] == "server" else 1e-12}
    if case["kind"] == "ops":
        return {"rel": 1e-5}
    return {"rel": 1e-4}
