"""The fused tensor-core atomic-network kernel against a plain float64 torch evaluation of the
same four 384-128-128-64-1 stacks.  Tolerances (relative to the largest energy): 2e-5 with the
split-precision products (float32-grade), 5e-3 with plain tf32."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(model, feats64, acs):
    import torch
    starts = np.concatenate([[0], np.cumsum(acs)])
    out = []
    for t, ann in enumerate(model.anns):
        a = feats64[int(starts[t]):int(starts[t + 1])]
        last = len(ann.Ws) - 1
        for k, (w, b) in enumerate(zip(ann.Ws, ann.bs)):
            a = a @ w.detach().double() + b.detach().double()
            if k != last:
                a = model.activation_fn(a)
        out.append(a.reshape(-1))
    return torch.cat(out)


@pytest.mark.parametrize("act", ["celu", "gaussian", "normal", "softplus"])
@pytest.mark.parametrize("split,tol", [(True, 2e-5), (False, 5e-3)])
def test_fused_forward_matches_dense_float64(act, split, tol):
    import torch
    from khan_b200.model import activations, nn
    torch.manual_seed(0)
    acs = np.array([300, 129, 0, 7])          # a full tile + remainder, an exact edge, empty, tiny
    n = int(acs.sum())
    model = nn.MoleculeNN(activation_fn=activations.get_fn_by_name(act), seed=1, split_precision=split)
    for ann in model.anns:                     # non-zero biases so that they are exercised
        for b in ann.bs:
            b.data.normal_(0.0, 0.1)
    feats = (torch.rand((n, 384), device="cuda") * 2.0).float()
    got = model.atom_energies_sorted(feats, acs)
    from khan_b200 import ani_mod
    ani_mod.check_device_status("mlp")
    ref = _reference(model, feats.double(), acs)
    scale = ref.abs().max().item()
    assert (got.double() - ref).abs().max().item() < tol * scale


def _interleaved(model):
    out = []
    for ann in model.anns:
        for w, b in zip(ann.Ws, ann.bs):
            out.extend([w, b])
    return out


def _dense64(model, feats64, acs, params64):
    import torch
    starts = np.concatenate([[0], np.cumsum(acs)])
    out = []
    for t in range(4):
        a = feats64[int(starts[t]):int(starts[t + 1])]
        w1, b1, w2, b2, w3, b3, w4, b4 = params64[8 * t: 8 * t + 8]
        for w, b in ((w1, b1), (w2, b2), (w3, b3)):
            a = model.activation_fn(a @ w + b)
        out.append((a @ w4 + b4).reshape(-1))
    return torch.cat(out)


@pytest.mark.parametrize("act", ["celu", "gaussian", "normal", "softplus"])
def test_backward_kernel_matches_dense_float64(act):
    """Feature gradient (from the backward kernel) and all weight gradients against float64
    autograd of the same networks; tolerance 5e-5 of the largest entry of each gradient."""
    import torch
    from khan_b200.model import activations, nn
    acs = np.array([300, 129, 0, 7])
    n = int(acs.sum())
    model = nn.MoleculeNN(activation_fn=activations.get_fn_by_name(act), seed=3, init="he")
    for ann in model.anns:
        for b in ann.bs:
            b.data.normal_(0.0, 0.1)
    gen = torch.Generator(device="cuda").manual_seed(5)
    feats = torch.rand((n, 384), device="cuda", generator=gen).requires_grad_(True)
    w = torch.randn(n, device="cuda", generator=gen)
    (model.atom_energies_sorted(feats, acs) * w).sum().backward()
    fused = [feats.grad.clone()] + [None if p.grad is None else p.grad.clone() for p in _interleaved(model)]
    feats64 = feats.detach().double().requires_grad_(True)
    params64 = [p.detach().double().requires_grad_(True) for p in _interleaved(model)]
    (_dense64(model, feats64, acs, params64) * w.double()).sum().backward()
    plain = [feats64.grad] + [p.grad for p in params64]
    from khan_b200 import ani_mod
    ani_mod.check_device_status("mlp backward")
    for k, (a, b) in enumerate(zip(fused, plain)):
        if b is None or b.abs().max().item() == 0.0:      # the empty element
            assert a is None or a.abs().max().item() == 0.0
            continue
        assert (a.double() - b).abs().max().item() < 5e-5 * b.abs().max().item(), k


def test_double_backward_keeps_the_second_derivative():
    """Force-training path: the gradient of a function of dE/dfeatures with respect to the
    weights (create_graph=True) against float64 autograd."""
    import torch
    from khan_b200.model import activations, nn
    acs = np.array([70, 20, 9, 5])
    n = int(acs.sum())
    model = nn.MoleculeNN(activation_fn=activations.celu, seed=4, init="he")
    gen = torch.Generator(device="cuda").manual_seed(6)
    feats = torch.rand((n, 384), device="cuda", generator=gen).requires_grad_(True)
    e = model.atom_energies_sorted(feats, acs)
    (gf,) = torch.autograd.grad(e.sum(), feats, create_graph=True)
    (gf ** 2).sum().backward()
    fused = [None if p.grad is None else p.grad.clone() for p in _interleaved(model)]
    feats64 = feats.detach().double().requires_grad_(True)
    params64 = [p.detach().double().requires_grad_(True) for p in _interleaved(model)]
    (gf64,) = torch.autograd.grad(_dense64(model, feats64, acs, params64).sum(), feats64, create_graph=True)
    (gf64 ** 2).sum().backward()
    for a, p in zip(fused, params64):
        b = p.grad
        if b is None or b.abs().max().item() == 0.0:     # the output bias does not reach dE/dfeatures
            assert a is None or a.abs().max().item() == 0.0
            continue
        assert (a.double() - b).abs().max().item() < 1e-3 * b.abs().max().item()


def test_weight_gradients_accumulate_into_existing_buffers():
    """Second backward pass: the parameters already have gradient buffers, so the kernel adds
    into them directly; the result must be exactly twice the first pass up to rounding."""
    import torch
    from khan_b200.model import activations, nn
    acs = np.array([140, 0, 33, 600])
    n = int(acs.sum())
    model = nn.MoleculeNN(activation_fn=activations.celu, seed=8, init="he")
    model.accumulate_into_grad = True
    gen = torch.Generator(device="cuda").manual_seed(9)
    feats = torch.rand((n, 384), device="cuda", generator=gen)
    w = torch.randn(n, device="cuda", generator=gen)
    (model.atom_energies_sorted(feats, acs) * w).sum().backward()
    params = [p for p in _interleaved(model) if p.grad is not None]
    first = [p.grad.clone() for p in params]
    ptrs = [p.grad.data_ptr() for p in params]
    (model.atom_energies_sorted(feats, acs) * w).sum().backward()
    for p, f, ptr in zip(params, first, ptrs):
        assert p.grad.data_ptr() == ptr
        assert (p.grad - 2 * f).abs().max().item() <= 1e-5 * f.abs().max().item()
    # without the flag torch.autograd.grad still gets its gradients returned
    model.accumulate_into_grad = False
    got = torch.autograd.grad((model.atom_energies_sorted(feats, acs) * w).sum(), params)
    for g, f in zip(got, first):
        assert (g - f).abs().max().item() <= 1e-5 * f.abs().max().item()


def test_packed_and_unpacked_weight_paths_agree(monkeypatch):
    """The kernels fetch pre-packed weight chunks with bulk copies by default; without a packed
    copy they stage the weights themselves.  Same operands, same MMAs: identical energies, and
    gradients equal up to the order of the floating-point reductions."""
    import torch
    from khan_b200.model import activations, nn
    acs = np.array([300, 129, 0, 7])
    n = int(acs.sum())
    gen = torch.Generator(device="cuda").manual_seed(12)
    base = torch.rand((n, 384), device="cuda", generator=gen)
    w = torch.randn(n, device="cuda", generator=gen)
    results = []
    for packed in (True, False):
        model = nn.MoleculeNN(activation_fn=activations.gaussian, seed=13, init="he")
        if not packed:
            monkeypatch.setattr(nn.MoleculeNN, "pack_weights", lambda self, stream=None: None)
        feats = base.clone().requires_grad_(True)
        e = model.atom_energies_sorted(feats, acs)
        (e * w).sum().backward()
        results.append((e.detach().clone(), feats.grad.clone(),
                        [p.grad.clone() for p in _interleaved(model) if p.grad is not None]))
    (e0, f0, g0), (e1, f1, g1) = results
    assert torch.equal(e0, e1)
    assert torch.equal(f0, f1)
    for a, b in zip(g0, g1):
        assert (a - b).abs().max().item() <= 1e-5 * b.abs().max().item()


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("n_mols,heavy", [(1, 1), (1, 8), (7, 2), (40, 8), (90, 8)])
def test_few_atom_networks_match_the_autograd_path(precision, n_mols, heavy):
    """The 16-atom-tile kernel (float64: any size; float32: up to a limit that 90 molecules exceed): energies
    and coordinate gradients against the dense differentiable path, tiles of 1 to 16 atoms, absent elements."""
    import torch
    from khan_b200 import RawDataset, TrainerMultiTower
    from khan_b200.model import activations
    from khan_b200.data import synthetic as syn
    mols = syn.gdb_like_batch(n_mols, seed=n_mols, heavy_min=heavy, heavy_max=heavy).molecules()
    ds = RawDataset(mols)
    for act in (activations.celu, activations.gaussian, activations.normal, activations.softplus):
        tr = TrainerMultiTower(None, [torch.device("cuda", 0)], precision=precision, layer_sizes=(128, 128, 64, 1),
                               activation_fn=act, seed=3)
        got_e, got_g = np.array(tr.predict(ds)), np.concatenate(list(tr.coordinate_gradients(ds)))
        dense = TrainerMultiTower(None, [torch.device("cuda", 0)], precision="float64", layer_sizes=(128, 128, 64, 1),
                                  activation_fn=act, seed=3)
        with torch.no_grad():      # the same (float32) weights in the dense double-precision path
            for a, b in zip(dense.parameters, tr.parameters):
                a.copy_(b)
        dense._evaluator_usable = lambda dataset: False
        want_e = np.array(dense.predict(ds))
        want_g = np.concatenate(list(dense.coordinate_gradients(ds, use_evaluator=False)))
        tol = 1e-4 if precision == "float32" else 1e-10
        assert np.abs(got_e - want_e).max() <= tol * np.abs(want_e).max()
        assert np.abs(got_g - want_g).max() <= tol * np.abs(want_g).max()
        e1, g1 = tr.energy_and_gradient(mols[0])
        assert abs(e1 - want_e[0]) <= tol * np.abs(want_e).max()
        assert np.abs(g1 - want_g[:len(mols[0])]).max() <= tol * np.abs(want_g).max()


@pytest.mark.parametrize("counts,width", [((1, 0, 0, 0), 4), ((5, 0, 3, 70), 64), ((300, 31, 0, 1), 128)])
def test_bias_and_celu_between_layers(counts, width):
    """ani_bias_celu_f32 against float64: one addition (half an ulp of z) and exp in float32 (at most 1e-6 off, times 0.1)."""
    import torch
    from khan_b200 import _lib
    n, rng = sum(counts), np.random.default_rng(width)
    z0, b = rng.normal(size=(n, width)).astype(np.float32), rng.normal(size=(4, width)).astype(np.float32)
    z, bias = torch.from_numpy(z0).cuda(), torch.from_numpy(b).cuda()
    a = torch.empty_like(z)
    where = (ctypes.c_void_p * 4)(*[bias[t].data_ptr() if counts[t] else None for t in range(4)])
    acs = (ctypes.c_int * 4)(*counts)
    _lib.check(_lib.lib().ani_bias_celu_f32(z.data_ptr(), a.data_ptr(), where, acs, width, None), "ani_bias_celu_f32")
    want = z0.astype(np.float64) + np.repeat(b.astype(np.float64), counts, axis=0)
    assert np.abs(z.cpu().numpy() - want).max() <= 6e-8 * np.abs(want).max()
    zs = z.cpu().numpy().astype(np.float64)
    celu = np.where(zs >= 0, zs, 0.1 * np.expm1(10.0 * np.minimum(zs, 0.0)))
    assert np.abs(a.cpu().numpy() - celu).max() < 2e-7
    last = torch.from_numpy(z0).cuda()                # without an activation
    _lib.check(_lib.lib().ani_bias_celu_f32(last.data_ptr(), None, where, acs, width, None), "ani_bias_celu_f32")
    assert torch.equal(last, z)
