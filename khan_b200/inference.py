"""Energies and forces of staged batches through the C ABI only (no autograd):

    ani_sort -> featurize -> atomic networks (forward) -> molecule sums (ani_molecule_energy)
             -> atomic networks (backward to the features, dE_mol/dE_atom = 1) -> featurize_grad

which is what the reference evaluates for ``predict`` + ``coordinate_gradients``
(``khan/training/trainer_multi_tower.py:580-614,655-678``: ``tf.gradients(tower_pred, [x, y, z])``),
with every buffer pre-allocated so that a pass can be captured into a CUDA graph.
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import _lib
from .model import activations
from .staged import StagedBatch


class EnergyForces:
    """Pre-allocated evaluator for one model (the 384-128-128-64-1 networks, float32 or float64)."""

    def __init__(self, model, n_atoms: int, n_mols: int, device="cuda:0"):
        if not model.has_kernels:
            raise ValueError("EnergyForces needs the fused 384-128-128-64-1 networks")
        self.model = model
        self.device = torch.device(device)
        self.dtype = model.precision
        self.f64 = self.dtype == torch.float64
        _lib.same_device(self.device, *model.get_parameters(), where="EnergyForces")
        self.act_id = activations.KERNEL_ID[model.activation_fn]
        self.split = bool(model.split_precision)
        real = dict(dtype=self.dtype, device=self.device)
        self.energy_sorted = torch.empty(n_atoms, **real)
        self.mol_energy = torch.zeros(n_mols, **real)
        if not self.f64:
            self.ones = torch.ones(n_atoms, **real)
        self.n_atoms_cap, self.n_mols_cap = n_atoms, n_mols

    def _fixed_args(self, packed):
        """A new argument block with everything that does not change from batch to batch."""
        a = _lib.EnergyArgs64() if self.f64 else _lib.PassArgs()
        a.activation = self.act_id
        a.energy_sorted, a.mol_energy = self.energy_sorted.data_ptr(), self.mol_energy.data_ptr()
        if not self.f64:
            a.split_precision = int(self.split)
            a.grad_energy_sorted = self.ones.data_ptr()
        for t, ann in enumerate(self.model.anns):
            for k, (w, b) in enumerate(zip(ann.Ws, ann.bs)):
                getattr(a, f"w{k + 1}")[t], getattr(a, f"b{k + 1}")[t] = w.data_ptr(), b.data_ptr()
            if packed is not None:
                a.packed[t] = packed[t].data_ptr()
        return a

    def weights_place(self):
        """Changes when the model's weights have moved."""
        packed = None if self.f64 else self.model.packed_weights()
        return self.model.anns[0].Ws[0].data_ptr(), None if packed is None else packed.data_ptr()

    def _pass_args(self, sb: StagedBatch):
        """The argument block of the pass: everything that does not change from batch to batch is filled once
        (and again when the model's weights have moved), the batch's own fields per call."""
        packed, key = None if self.f64 else self.model.packed_weights(), self.weights_place()
        if getattr(self, "_pa_key", None) != key:
            self._pa, self._pa_key = self._fixed_args(packed), key
        a = self._pa
        a.n_atoms, a.n_mols, a.acs_host = sb.n_atoms, sb.n_mols, sb.acs_ptr
        a.xs, a.ys, a.zs = sb.x.data_ptr(), sb.y.data_ptr(), sb.z.data_ptr()
        a.atomic_numbers, a.mol_offsets, a.mol_atom_counts = (sb.types.data_ptr(), sb.mol_offsets.data_ptr(),
                                                              sb.mol_counts.data_ptr())
        a.scatter_idxs, a.gather_idxs, a.atom_counts = sb.scatter.data_ptr(), sb.gather.data_ptr(), sb.counts.data_ptr()
        a.features, a.feature_grads = sb.features.data_ptr(), sb.upstream.data_ptr()
        g, cap, esz = sb.grads.data_ptr(), sb.n_atoms_cap, sb.grads.element_size()
        a.x_grads, a.y_grads, a.z_grads = g, g + cap * esz, g + 2 * cap * esz
        return a

    def pass_block(self, sb: StagedBatch):
        """Argument block of passes over ``sb`` for a ``BatchDriver``, which fills in what describes the batch."""
        if not self.f64 and self.model.packed_weights() is None:
            self.model.pack_weights()                # allocates the packed copy (first use)
        a = self._pass_args(sb)
        return type(a).from_buffer_copy(a)

    def _call(self, sb: StagedBatch, phases: int, stream, where: str) -> None:
        if sb.n_atoms > self.n_atoms_cap or sb.n_mols > self.n_mols_cap or sb.dtype != self.dtype:
            raise ValueError("batch does not fit this evaluator")
        _lib.same_device(self.device, sb.features, sb.x, where=where)
        if stream is None:
            stream = torch.cuda.current_stream(self.device).cuda_stream
        if self.f64:
            phases &= ~_lib.PASS_PACK
        elif self.model.packed_weights() is None:
            self.model.pack_weights(ctypes.c_void_p(stream) if isinstance(stream, int) else stream)   # allocates the packed copy (first use)
            phases &= ~_lib.PASS_PACK
        a = self._pass_args(sb)
        a.phases = phases
        if self.f64:
            _lib.check(_lib.lib().ani_energy_pass_f64(ctypes.byref(a), stream), "ani_energy_pass_f64")
        else:
            _lib.check(_lib.lib().ani_network_pass_f32(ctypes.byref(a), stream), "ani_network_pass_f32")

    def featurize(self, sb: StagedBatch, stream: ctypes.c_void_p | None = None) -> None:
        """Sort + featurize of the batch staged in ``sb`` only (one C-ABI call): they need nothing but the
        coordinates, so a caller may run them for the NEXT batch on another stream beside the network kernels
        of this one and then call ``run(..., featurized=True)``."""
        self._call(sb, _lib.PASS_FEATURIZE, stream, "EnergyForces.featurize")

    def run(self, sb: StagedBatch, stream: ctypes.c_void_p | None = None, pack: bool = True,
            forces: bool = True, featurized: bool = False) -> None:
        """One pass over the batch staged in ``sb`` -- one C-ABI call (``ani_network_pass_f32`` or
        ``ani_energy_pass_f64``).  Afterwards
        ``self.mol_energy[:sb.n_mols]`` holds the molecule energies and ``sb.grads[:, :sb.n_atoms]`` dE/dx,
        dE/dy, dE/dz (forces are their negatives).  ``pack=False`` skips the refresh of the pre-packed
        weights: for a caller that packed them (``model.pack_weights``) after the last change of the
        weights, e.g. once before a series of passes that run side by side on several streams.
        ``forces=False`` stops after the molecule energies (``predict``); ``featurized=True`` leaves sort +
        featurize out (``featurize`` has run for this batch)."""
        self._call(sb, (_lib.PASS_PACK if pack else 0) | (0 if featurized else _lib.PASS_FEATURIZE) | _lib.PASS_FORWARD
                   | _lib.PASS_ENERGY | _lib.PASS_TRANSIENT
                   | ((_lib.PASS_BACKWARD | _lib.PASS_COORD_GRAD) if forces else 0), stream, "EnergyForces.run")

    KERNELS_PER_PASS = 5   # small molecules: weight packing (unless pack=False), sort, featurize, networks, featurize_grad + molecule sums


class PassTools:
    """What a pass over a data set (``predict``, ``coordinate_gradients``) keeps for the next one: two sets of device
    buffers, a stream for each, and pinned buffers for the results."""

    def __init__(self, model, cap_atoms: int, cap_mols: int, device):
        self.staged = [StagedBatch(cap_atoms, cap_mols, model.precision, device=device) for _ in range(2)]
        self.evaluators = [EnergyForces(model, cap_atoms, cap_mols, device=device) for _ in range(2)]
        self.streams = [torch.cuda.Stream(device=device) for _ in range(2)]
        self.ring, self.weights = [], []

    def fits(self, cap_atoms: int, cap_mols: int) -> bool:
        return self.staged[0].n_atoms_cap >= cap_atoms and self.staged[0].n_mols_cap >= cap_mols

    def blocks(self):
        return [ev.pass_block(sb) for ev, sb in zip(self.evaluators, self.staged)]

    def host_ring(self, size: int):
        if size and (not self.ring or self.ring[0].numel() < size):
            self.ring = [torch.empty(size, dtype=self.staged[0].dtype).pin_memory() for _ in range(_lib.DRIVER_RING)]
        return self.ring if size else []

    def weight_copies(self):
        if not self.weights:
            size = _lib.lib().ani_driver_weights_bytes(int(self.evaluators[0].f64))
            self.weights = [torch.empty(size, dtype=torch.uint8, device=self.evaluators[0].device)
                            for _ in range(_lib.DRIVER_RING)]
        return self.weights


class SingleGeometry:
    """Energy and gradient of one geometry at a time (the energy server's request): the inputs cross in one
    copy from a pinned arena, the results in one copy back, and nothing is allocated per call.  Calls must not
    overlap."""

    def __init__(self, model, capacity: int, device):
        self.capacity = capacity
        self.batch = StagedBatch(capacity, 1, model.precision, device=device)
        self.evaluator = EnergyForces(model, capacity, 1, device=device)
        size = self.batch.xyz.element_size()
        nbytes = 3 * capacity * size + 4 * capacity + 8      # x, y, z | elements | offset, count of the molecule
        self.host_in = torch.zeros(nbytes, dtype=torch.uint8).pin_memory()
        self.dev_in = torch.zeros(nbytes, dtype=torch.uint8, device=device)

        def views(arena):
            ints = arena[3 * capacity * size:].view(torch.int32)
            return arena[:3 * capacity * size].view(model.precision).view(3, capacity), ints[:capacity], ints[capacity:]

        xyz, types, table = views(self.host_in)
        self._xyz, self._types, self._table = xyz.numpy(), types.numpy(), table.numpy()
        b = self.batch
        b.xyz, b.types, table = views(self.dev_in)
        b.x, b.y, b.z = b.xyz[0], b.xyz[1], b.xyz[2]
        b.mol_offsets, b.mol_counts = table[:1], table[1:]
        # the gradient (padded to the capacity) and the energy in one array each side
        self.dev_out = torch.zeros(3 * capacity + 1, dtype=model.precision, device=device)
        self.host_out = torch.zeros(3 * capacity + 1, dtype=model.precision).pin_memory()
        self._out = self.host_out.numpy()
        b.grads = self.dev_out[:3 * capacity].view(3, capacity)
        self.evaluator.mol_energy = self.dev_out[3 * capacity:]

        self._request = r = _lib.RequestArgs()
        r.in_host, r.in_dev, r.in_bytes = self.host_in.data_ptr(), self.dev_in.data_ptr(), nbytes
        r.out_host, r.out_dev = self.host_out.data_ptr(), self.dev_out.data_ptr()
        r.out_bytes = self.dev_out.numel() * size
        self._weights = self._block = None

    def _prepare(self):
        """The argument block of the pass, again when the weights have moved."""
        weights = self.evaluator.model.anns[0].Ws[0].data_ptr()
        if self._weights != weights:
            block = self._block = self.evaluator.pass_block(self.batch)
            block.n_mols = 1
            block.phases = (_lib.PASS_FEATURIZE | _lib.PASS_FORWARD | _lib.PASS_ENERGY | _lib.PASS_BACKWARD
                            | _lib.PASS_COORD_GRAD)
            if self.evaluator.f64:
                self._request.pass64 = ctypes.pointer(block)
            else:
                block.phases |= _lib.PASS_PACK | _lib.PASS_TRANSIENT
                self._request.pass_ = ctypes.pointer(block)
            self._weights = weights
        return self._block

    def evaluate(self, arr):
        """``arr``: float64 ``(n, 4)`` array, n up to the capacity.  Returns (energy, (n, 3) gradient)."""
        n = len(arr)
        self._xyz[:, :n] = arr[:, 1:].T
        self._types[:n] = arr[:, 0]
        self._table[1] = n
        self.batch.set_shape(n, 1, np.bincount(self._types[:n], minlength=4))
        with torch.cuda.device(self.batch.device):
            self._prepare().n_atoms = n
            _lib.check(_lib.lib().ani_request(ctypes.byref(self._request), torch.cuda.current_stream().cuda_stream),
                       "ani_request")
        return float(self._out[-1]), self._out[:-1].reshape(3, self.capacity)[:, :n].T.copy()
