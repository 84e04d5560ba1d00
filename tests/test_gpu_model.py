"""GPU: sub-block and end-to-end E/F/S/M parity.

Sub-blocks are compared with the oracle's functions (forward and data gradients);
whole evaluations with the committed results of the reference's own float32 run,
inside the gates  |dE| <= 1e-5 eV/atom, |dF| <= 1e-4 eV/A, |dS| <= 1e-5 eV/A^3,
|dm| <= 1e-4 mu_B."""
import numpy as np
import pytest
import torch

from conftest import GOLDEN_CASES, GPA, TOL, golden_config, load_golden
from functools import partial

from gpu_util import dev, report
from matris_b200 import workloads
from matris_b200.weights import full_config, random_checkpoint

pytestmark = pytest.mark.gpu
report_feat = partial(report, scaled=True)  # feature tensors: bound scales with the reference's magnitude


def rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).float()


@pytest.fixture(scope="module")
def setup():
    from matris_b200.graph import build_batched_graph
    from matris_b200.model import pack_parameters, row_graphs
    crystals = [workloads.demo_pu4si6(), workloads.random_crystals(2, seed=21)[1]]
    g = build_batched_graph([c.numbers for c in crystals], [c.cart for c in crystals], [c.lattice for c in crystals])
    ck = random_checkpoint(dict(num_layers=1, reference_energy="mpa"), seed=3, jitter=0.1)
    P = pack_parameters(ck["state_dict"], full_config(ck["config"]), g.cart32.device)
    return g, ck, P, row_graphs(g)


def _oracle_dicts(g):
    lg = g.line_graph.cpu().long()
    atom = dict(source_index=g.neighbor.cpu().long(), target_index=g.center.cpu().long())
    line = dict(atom_list=lg[:, 0], target_index=lg[:, 1], source_index=lg[:, 3])
    return atom, line, g.d2u.cpu().long()


@pytest.mark.parametrize("which", ["atom", "line"])
def test_attention_layer_forward_backward(setup, which):
    from matris_b200.model import AttentionFn
    from oracle.model import _P, attention_layer
    g, ck, P, (atom_rg, line_rg) = setup
    atom_d, line_d, d2u = _oracle_dicts(g)
    sd = {k: v.double() for k, v in ck["state_dict"].items()}
    if which == "atom":
        rg, gd, emap, nn_, ne = atom_rg, atom_d, d2u, g.n_atoms, g.n_bonds
    else:
        rg, gd, emap, nn_, ne = line_rg, line_d, None, g.n_bonds, g.n_triplets
    node, edge = rnd(nn_, 128, seed=1), rnd(ne, 128, seed=2)
    dn, de = rnd(nn_, 128, seed=3), rnd(ne, 128, seed=4)
    N, E = node.double().requires_grad_(True), edge.double().requires_grad_(True)
    rn, re_ = attention_layer(_P(sd, f"interaction_block.0.attn_block_{which}_graph."), N, E, gd, emap)
    gn, ge = torch.autograd.grad((rn * dn.double()).sum() + (re_ * de.double()).sum(), [N, E])
    n_in, e_in = dev(node).requires_grad_(True), dev(edge).requires_grad_(True)
    on, oe = AttentionFn.apply(n_in, e_in, getattr(P.layers[0], "attn_" + which), rg)
    report_feat(f"attention[{which}] node", on, rn, 3e-5)
    report_feat(f"attention[{which}] edge", oe, re_, 3e-5)
    dn_, de_ = torch.autograd.grad([on, oe], [n_in, e_in], [dev(dn), dev(de)])
    report_feat(f"attention[{which}] d node", dn_, gn, 2e-4)
    report_feat(f"attention[{which}] d edge", de_, ge, 2e-4)


@pytest.mark.parametrize("which", ["atom", "line"])
def test_refinement_layer_forward_backward(setup, which):
    from matris_b200.model import RefineFn
    from oracle.model import _P, refinement_layer
    g, ck, P, (atom_rg, line_rg) = setup
    atom_d, line_d, d2u = _oracle_dicts(g)
    sd = {k: v.double() for k, v in ck["state_dict"].items()}
    rbf = rnd(g.n_bonds, 7, seed=5, scale=0.3)
    if which == "atom":
        rg, gd, emap, nn_, ne, af = atom_rg, atom_d, d2u, g.n_atoms, g.n_bonds, None
    else:
        rg, gd, emap, nn_, ne, af = line_rg, line_d, None, g.n_bonds, g.n_triplets, rnd(g.n_atoms, 128, seed=6)
    node, edge = rnd(nn_, 128, seed=1), rnd(ne, 128, seed=2)
    dn, de = rnd(nn_, 128, seed=3), rnd(ne, 128, seed=4)
    N, E, Rb = node.double().requires_grad_(True), edge.double().requires_grad_(True), rbf.double().requires_grad_(True)
    A = None if af is None else af.double().requires_grad_(True)
    rn, re_ = refinement_layer(_P(sd, f"interaction_block.0.refine_block_{which}_graph."), N, E, Rb, gd, emap, A)
    leaves = [N, E, Rb] + ([A] if A is not None else [])
    grads = torch.autograd.grad((rn * dn.double()).sum() + (re_ * de.double()).sum(), leaves, retain_graph=True)
    n_in, e_in, r_in = dev(node).requires_grad_(True), dev(edge).requires_grad_(True), dev(rbf).requires_grad_(True)
    a_in = None if af is None else dev(af).requires_grad_(True)
    on, oe = RefineFn.apply(n_in, e_in, r_in, a_in, getattr(P.layers[0], "refine_" + which), rg)
    report_feat(f"refine[{which}] node", on, rn, 3e-5)
    report_feat(f"refine[{which}] edge", oe, re_, 3e-5)
    mine = torch.autograd.grad([on, oe], [n_in, e_in, r_in] + ([a_in] if a_in is not None else []), [dev(dn), dev(de)])
    for name, a, b in zip(["node", "edge", "rbf", "atom"], mine, grads):
        report_feat(f"refine[{which}] d {name}", a, b, 2e-4)
    # the last layer's form: the edge update is not computed (a placeholder comes back) and sends no gradient
    grads = torch.autograd.grad((rn * dn.double()).sum(), leaves)
    rg.skip_edge_out = True
    try:
        on, oe = RefineFn.apply(n_in, e_in, r_in, a_in, getattr(P.layers[0], "refine_" + which), rg)
        assert oe.numel() == 0 and not oe.requires_grad
        report_feat(f"refine[{which}] node, no edge update", on, rn, 3e-5)
        mine = torch.autograd.grad([on], [n_in, e_in, r_in] + ([a_in] if a_in is not None else []), [dev(dn)])
    finally:
        rg.skip_edge_out = False
    for name, a, b in zip(["node", "edge", "rbf", "atom"], mine, grads):
        report_feat(f"refine[{which}] d {name}, no edge update", a, b, 2e-4)


def _evaluate(ck, crystals, task, keep=None):
    from matris_b200 import MatRIS
    model = MatRIS.from_dict(ck).to("cuda")
    model.keep_activations = keep
    out = model.predict(crystals, task)
    res = {"e": out["e"].cpu().double().numpy(), "ref_energy": out["ref_energy"].cpu().double().numpy()}
    if "f" in out:
        res["f"] = torch.cat(list(out["f"])).cpu().double().numpy()
    if "s" in out:
        res["s"] = torch.stack(out["s"]).cpu().double().numpy()
    if "m" in out:
        res["m"] = torch.cat(out["m"]).cpu().double().numpy()
    return res, out, model


@pytest.mark.parametrize("mode", ["simt", "tcgen05_tile", "tcgen05_tf32"])
def test_other_contraction_modes_match_reference(mode):
    """A whole evaluation in the cross-check modes, whose bond gradients are summed by a launch of their own into the buffer of dz2."""
    from matris_b200 import ops
    meta, crystals, z = load_golden("random2_L2")
    ck = random_checkpoint(golden_config(meta), seed=meta["seed"], jitter=meta["jitter"])
    try:
        ops.set_gemm_mode(mode)
        res = _evaluate(ck, crystals, "efs")[0]
        assert ops.gemm_status() == 0
    finally:
        ops.set_gemm_mode("tcgen05")
    for k, unit in (("e", 1.0), ("f", 1.0), ("s", GPA)):
        report(f"mode {mode} {k}", res[k] / unit, z[f"ref32_{k}"] / unit, TOL[k])
    report(f"mode {mode} F vs fp64 (2e-3 relative)", res["f"], z["ref64_f"], 2e-3 * np.abs(z["ref64_f"]).max())


@pytest.mark.parametrize("keep", [True, False], ids=["keep", "recompute"])
@pytest.mark.parametrize("case", GOLDEN_CASES)
def test_end_to_end_matches_reference(case, keep):
    """Whole evaluations against the reference's own float32 results; the gates are ABSOLUTE.  Both memory
    policies run every case (the reference itself recomputes above 60,000 triplets; fe432_L2 is above that)."""
    meta, crystals, z = load_golden(case)
    ck = random_checkpoint(golden_config(meta), seed=meta["seed"], jitter=meta["jitter"])
    res, out, _ = _evaluate(ck, crystals, meta["task"], keep=keep)
    tag = f"e2e[{case},{'keep' if keep else 'recompute'}]"
    report(f"{tag} E (eV/atom)", res["e"], z["ref32_e"], TOL["e"])
    # the model's own energy, before the (much larger) tabulated reference energy is added
    report(f"{tag} E model part (eV/atom)", res["e"] - res["ref_energy"], z["ref32_e_model"], TOL["e"])
    report(f"{tag} E model part vs fp64", res["e"] - res["ref_energy"], z["ref64_e_model"], TOL["e"])
    report(f"{tag} F (eV/A)", res["f"], z["ref32_f"], TOL["f"])
    report(f"{tag} S (eV/A^3)", res["s"] / GPA, z["ref32_s"] / GPA, TOL["s"])
    if "m" in meta["task"]:
        report(f"{tag} M (mu_B)", res["m"], z["ref32_m"], TOL["m"])
    report(f"{tag} reference energy", res["ref_energy"], z["ref32_ref_energy"], 1e-6)
    # tighter checks against the reference's float64 run, relative to the largest component (random-init forces are
    # small, so the absolute gate alone is blunt), with a floor at the float32 rounding noise of the reference
    # itself (forces that vanish by symmetry have nothing but that noise to compare)
    report(f"{tag} F vs fp64 (2e-3 relative)", res["f"], z["ref64_f"], max(2e-3 * np.abs(z["ref64_f"]).max(), 1e-6))
    report(f"{tag} S vs fp64 (2e-3 relative, GPa)", res["s"], z["ref64_s"], max(2e-3 * np.abs(z["ref64_s"]).max(), 1e-4))
    # result dictionary layout of MatRIS.forward
    assert out["atoms_per_graph"].dtype == torch.int32 and len(out["f"]) == len(crystals)
    assert out["s"][0].shape == (3, 3) and out["f"][0].shape == (len(crystals[0].numbers), 3)


def test_tasks_and_keys():
    meta, crystals, z = load_golden("pu4si6_L2")
    ck = random_checkpoint(dict(num_layers=2, reference_energy="mpa"), seed=0, jitter=0.1)
    for task, keys in (("e", {"e"}), ("em", {"e", "m"}), ("ef", {"e", "f"}), ("efs", {"e", "f", "s"})):
        res, out, _ = _evaluate(ck, crystals, task)
        assert set(out) == keys | {"atoms_per_graph", "ref_energy"}
        report(f"task={task} E", res["e"], z["ref32_e"], TOL["e"])


def test_batch_equals_single_structures():
    crystals = workloads.random_crystals(4, seed=5)
    ck = random_checkpoint(dict(num_layers=2, reference_energy="mpa"), seed=1)
    batch, _, model = _evaluate(ck, crystals, "efs")
    ofs = 0
    for b, cr in enumerate(crystals):
        single, _, _ = _evaluate(ck, [cr], "efs")
        n = len(cr.numbers)
        report(f"batch-vs-single E[{b}]", batch["e"][b:b + 1], single["e"], 2e-6)
        report(f"batch-vs-single F[{b}]", batch["f"][ofs:ofs + n], single["f"], 2e-6)
        report(f"batch-vs-single S[{b}]", batch["s"][b] / GPA, single["s"][0] / GPA, 2e-7)
        ofs += n


def test_forces_are_energy_derivatives():
    """Finite differences of the CUDA energy against the CUDA forces (no oracle involved)."""
    from matris_b200 import MatRIS
    from matris_b200.workloads import Crystal
    cr = workloads.demo_pu4si6()
    ck = random_checkpoint(dict(num_layers=2, reference_energy="mpa"), seed=2)
    model = MatRIS.from_dict(ck).to("cuda")
    out = model.predict([cr], "ef")
    f = out["f"][0].cpu().double().numpy()
    n = len(cr.numbers)
    h = 2e-2
    for (i, k) in ((0, 0), (5, 2)):
        e = []
        for sgn in (+1, -1):
            cart = cr.cart.copy()
            cart[i, k] += sgn * h
            e.append(float(model.predict([Crystal(cr.numbers, cart, cr.lattice)], "e")["e"][0]) * n)
        fd = -(e[0] - e[1]) / (2 * h)
        assert abs(fd - f[i, k]) < 5e-3 * max(1.0, abs(f[i, k])) + 2e-3, (fd, f[i, k])


def test_state_dict_roundtrip_and_from_dict():
    from matris_b200 import MatRIS
    ck = random_checkpoint(dict(num_layers=1, reference_energy="mpa"), seed=4)
    model = MatRIS.from_dict(ck)
    assert list(model.state_dict().keys()) == list(ck["state_dict"].keys())
    assert model.config["num_layers"] == 1 and model.is_intensive
    with pytest.raises(RuntimeError):
        model([workloads.demo_pu4si6()])  # still on CPU: no fallback


def test_recompute_equals_kept_activations():
    """The memory policies (keep sub-block internals / recompute them in backward / keep those of the last n layers
    only) agree."""
    from matris_b200 import MatRIS
    crystals = workloads.random_crystals(3, seed=9)
    ck = random_checkpoint(dict(num_layers=3, reference_energy="mpa"), seed=5)
    model = MatRIS.from_dict(ck).to("cuda")
    res = {}
    for keep, kept in ((True, 3), (False, 0), (1, 1), (2, 2), (None, 3)):
        model.keep_activations = keep
        out = model.predict(crystals, "efs")
        assert model.last_kept_layers == kept, (keep, model.last_kept_layers)
        res[keep] = (torch.cat(list(out["f"])).cpu(), torch.stack(out["s"]).cpu())
    for keep in (False, 1, 2, None):
        report(f"keep all vs keep_activations={keep}: F", res[True][0], res[keep][0], 2e-6)
        report(f"keep all vs keep_activations={keep}: S", res[True][1] / GPA, res[keep][1] / GPA, 2e-7)


def test_predict_in_sub_batches_equals_one_batch():
    """With little memory to plan with, predict evaluates a list of structures as contiguous sub-batches that keep
    every layer's internals; the results are those of the single batch (which then recomputes), in order."""
    from matris_b200 import MatRIS
    crystals = workloads.random_crystals(12, seed=13)
    ck = random_checkpoint(dict(num_layers=3, reference_energy="mpa"), seed=5)
    model = MatRIS.from_dict(ck).to("cuda")
    g = model.graph_converter.batch(crystals)
    assert model.split_for_memory(g) == [(0, 12)]
    one = model.predict(crystals, "efsm")
    assert model.last_kept_layers == 3
    # room for the internals of about a third of the batch: 45 % of the limit = a third of what all layers take
    model.memory_limit_bytes = 3 * (6.7e3 * g.n_triplets + 6.2e3 * g.n_edges) / 0.45 / 3
    ranges = model.split_for_memory(g)
    assert len(ranges) >= 3 and ranges[0][0] == 0 and ranges[-1][1] == 12
    assert all(a[1] == b[0] and a[0] < a[1] for a, b in zip(ranges, ranges[1:]))
    graphs = model.plan_batches(crystals)
    assert [x.n_struct for x in graphs] == [b - a for a, b in ranges]
    parts = model.predict(crystals, "efsm")
    assert model.last_kept_layers == 3  # the last sub-batch kept everything
    assert torch.equal(parts["atoms_per_graph"].cpu(), one["atoms_per_graph"].cpu())
    report("sub-batches vs one batch: E", parts["e"], one["e"], 1e-6, rel=True)
    # a float32 matrix product over the batch's composition table: rounding depends on the batch shape
    report("sub-batches vs one batch: reference energy", parts["ref_energy"], one["ref_energy"], 1e-6, rel=True)
    assert len(parts["f"]) == len(parts["s"]) == len(parts["m"]) == 12
    report("sub-batches vs one batch: F", torch.cat(list(parts["f"])), torch.cat(list(one["f"])), 2e-6)
    report("sub-batches vs one batch: S", torch.stack(parts["s"]) / GPA, torch.stack(one["s"]) / GPA, 2e-7)
    report("sub-batches vs one batch: M", torch.cat(parts["m"]), torch.cat(one["m"]), 2e-6)
    model.keep_activations = False       # an explicit policy is taken as given: no split
    assert model.split_for_memory(g) == [(0, 12)]


def test_forward_raises_once_after_an_expired_wait_and_recovers():
    """An expired bounded wait surfaces as one exception (at the next forward, or at check_status once the stream
    has been synchronised) and the model then works again."""
    from matris_b200 import MatRIS, ops
    from matris_b200._lib import MbError
    ck = random_checkpoint(dict(num_layers=1, reference_energy="mpa"), seed=6)
    model = MatRIS.from_dict(ck).to("cuda")
    cr = [workloads.demo_pu4si6()]
    first = model.predict(cr, "ef")
    e0 = first["e"].cpu()
    model.check_status()                 # nothing expired
    ops.selftest_wait_expiry()           # a wait runs out on this device
    out = model.predict(cr, "ef")        # this call's status copy carries the bit
    torch.cuda.synchronize()
    with pytest.raises(MbError, match="bounded wait expired"):
        model.check_status()
    again = model.predict(cr, "ef")      # the word was cleared on raising: no second exception
    report("energy after recovery", again["e"].cpu(), e0, 1e-6)
    torch.cuda.synchronize()
    model.check_status()
    ops.selftest_wait_expiry()
    model.predict(cr, "e")
    with pytest.raises(MbError):         # ... or the next forward raises
        torch.cuda.synchronize()
        model.predict(cr, "e")
    model.predict(cr, "e")
