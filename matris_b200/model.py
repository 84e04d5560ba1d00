"""MatRIS energy / force / stress / magmom evaluation on B200.

Host-side mirror of the reference's ``MatRIS`` module
(matris/model/model.py:30-317): same constructor arguments, ``config``,
``state_dict`` key names, ``from_dict`` / ``load`` checkpoint interface,
``graph_converter`` attribute and ``forward(graphs, task, is_training)`` result
dictionary.  All arithmetic runs in the CUDA kernels behind the C ABI, and the sequence of
kernels of an evaluation - forward and the hand-written backward pass (data
gradients only: weights are frozen at inference) that gives forces = -dE/dr and
stress = (1/V) dE/d(strain), the reference's conservative head
(matris/model/readout.py:202-224) - is queued by one library call.
``AttentionFn`` / ``RefineFn`` expose the two sub-blocks to torch.autograd.

Memory policy: a sub-block always keeps its inputs for the backward pass.  Its
internals are kept too for as many of the last layers as fit in memory; those of
the earlier layers are recomputed in the backward pass (the reference switches to
recomputation above 60,000 triplets, matris/model/interaction_block.py:15, 400-403).
"""
from __future__ import annotations

import ctypes as C
import os
from collections.abc import Sequence
from types import SimpleNamespace

import numpy as np
import torch
from torch import nn
from torch.autograd.function import once_differentiable

from . import _lib, ops
from ._lib import MbError
from .graph import BatchedGraph, GraphConverter, RadiusGraph, build_batched_graph, as_arrays
from .weights import BUFFER_KEYS, check_supported, full_config, random_state_dict, schema

GPA_PER_EV_A3 = 160.21766208  # matris/model/readout.py:215
# Evaluations that need at most this much memory take it as one block: one allocation, and a block the allocator can place
# again at the next call.  Larger ones ask for their buffers one by one, so that a block of a large part of the device is
# never wanted in one piece; just above the limit (256 atoms) that is 830 calls and 3 ms of host time under 9 ms of device time.
WORKSPACE_LIMIT = 4 << 30
# An evaluation plans with this much of the memory that is left: the rest is for what the allocator cannot place.
MEMORY_SHARE = 0.9


# ------------------------------------------------------------------ packed parameters
class _Packer:
    """Parameters as the library's structs of device pointers.  The tensors behind the pointers are kept in ``alive``."""

    def __init__(self, sd: dict, device):
        self.sd, self.device, self.alive = sd, device, []

    def get(self, key) -> torch.Tensor:
        return self.sd[key].detach().to(device=self.device, dtype=torch.float32)

    def vec(self, t) -> int | None:
        """Device address of a contiguous copy (None for a parameter the configuration does not have)."""
        if t is None:
            return None
        t = t.reshape(-1).contiguous()
        self.alive.append(t)
        return t.data_ptr()

    def weight(self, t) -> _lib.MbWeight:
        sw = ops.SplitWeight(t)
        self.alive.append(sw)
        return _lib.MbWeight(*sw.ptrs, sw.ldw)

    def gated(self, prefix, roles=()) -> _lib.MbUpdate:
        """GatedMLP: first layers of core|gate stacked to [256,K], second layers to [256,128], plus the transposes the
        backward products contract with.  ``roles`` names the origin of each 128 columns of layer 1 for an edge update
        ("edge", "ctr", "tgt", "src"): the library then forms the node terms once per node."""
        get, c, g = self.get, prefix + "mlp_core.layers.", prefix + "mlp_gate.layers."
        w1 = torch.cat([get(c + "0.weight"), get(g + "0.weight")], 0)
        w2c, w2g = get(c + "3.weight"), get(g + "3.weight")
        if roles:
            part = {r: w1[:, 128 * i:128 * i + 128] for i, r in enumerate(roles)}
            ts = torch.cat([part["tgt"], part["src"]], 0)
            first = dict(we=self.weight(part["edge"]), wet=self.weight(part["edge"].t()), wts=self.weight(ts),
                         wtst=self.weight(ts.t()))
            if "ctr" in part:
                first.update(wc=self.weight(part["ctr"]), wct=self.weight(part["ctr"].t()))
        else:
            first = dict(w1=self.weight(w1), w1t=self.weight(w1.t()))
        return _lib.MbUpdate(
            kind=0, k=w1.shape[1], **first, w2=self.weight(torch.cat([w2c, w2g], 0)),
            w2t=self.weight(torch.cat([w2c.t(), w2g.t()], 0)), b1=self.vec(torch.cat([get(c + "0.bias"), get(g + "0.bias")])),
            b2=self.vec(torch.cat([get(c + "3.bias"), get(g + "3.bias")])), nc=self.vec(get(prefix + "core_norm.weight")),
            ng=self.vec(get(prefix + "gate_norm.weight")))

    def mlp(self, prefix, bias, roles=()) -> _lib.MbUpdate:
        """The plain-MLP variant of an update block (graph_conv_mlp = "MLP"): nn.Sequential(MLP, RMSNorm)
        (matris/model/interaction_block.py:39-62, 172-184)."""
        get = self.get
        w1, w2 = get(prefix + "0.layers.0.weight"), get(prefix + "0.layers.3.weight")
        return _lib.MbUpdate(
            kind=1, k=w1.shape[1], w1=self.weight(w1), w2=self.weight(w2), w1t=self.weight(w1.t()), w2t=self.weight(w2.t()),
            b1=self.vec(get(prefix + "0.layers.0.bias")) if bias else None,
            b2=self.vec(get(prefix + "0.layers.3.bias")) if bias else None, nc=self.vec(get(prefix + "1.weight")))

    def ffn(self, prefix, bias) -> _lib.MbFfn:
        """node_FFN / edge_FFN (matris/model/interaction_block.py:197-210): two linear layers, biases only with use_bias."""
        w1, w2 = self.get(prefix + "layers.0.weight"), self.get(prefix + "layers.3.weight")
        return _lib.MbFfn(
            w1=self.weight(w1), w2=self.weight(w2), w1t=self.weight(w1.t()), w2t=self.weight(w2.t()),
            b1=self.vec(self.get(prefix + "layers.0.bias")) if bias else None,
            b2=self.vec(self.get(prefix + "layers.3.bias")) if bias else None)

    def attention(self, prefix, update) -> _lib.MbAttnParams:
        wst = torch.cat([self.get(prefix + "source_weight_linear.weight"), self.get(prefix + "target_weight_linear.weight")], 0)
        edge, more = update(prefix + "edge_nonlinear_update.", ("edge", "tgt", "src")), {}
        if edge.kind == 0:
            c, g = (self.get(f"{prefix}edge_nonlinear_update.mlp_{b}.layers.0.weight")[:, :128] for b in ("core", "gate"))
            more["welt"] = self.weight(torch.cat([c.t(), g.t(), wst.t()], 1))
        return _lib.MbAttnParams(
            node=update(prefix + "node_nonlinear_update."), edge=edge, **more,
            wst=self.weight(wst), wstt=self.weight(wst.t()), wn=self.vec(self.get(prefix + "node_res_weight")),
            we=self.vec(self.get(prefix + "edge_res_weight")))

    def refinement(self, prefix, update, bias, smoothed, line) -> _lib.MbRefineParams:
        return _lib.MbRefineParams(
            edge=update(prefix + "edge_nonlinear_update.", ("edge", "ctr", "tgt", "src") if line else ("edge", "tgt", "src")), nffn=self.ffn(prefix + "node_FFN.", bias),
            effn=self.ffn(prefix + "edge_FFN.", bias), wenv=self.vec(self.get(prefix + "learnable_envelope.weight")),
            wn=self.vec(self.get(prefix + "node_res_weight")), we=self.vec(self.get(prefix + "edge_res_weight")),
            smoothed_edge=int(smoothed))


def pack_parameters(sd: dict, cfg: dict, device) -> SimpleNamespace:
    """``.model``: the whole model as mb_model_params; ``.layers[i].attn_atom`` etc.: the sub-blocks' structs in it."""
    k = _Packer(sd, device)
    get, vec, weight = k.get, k.vec, k.weight
    n_layers, bias = int(cfg["num_layers"]), bool(cfg["use_bias"])
    M, layers = _lib.MbModelParams(), (_lib.MbLayerParams * n_layers)()
    M.layers, M.n_layers = layers, n_layers
    M.gaussian = str(cfg["distance_expansion"]).lower() == "gaussian"
    M.fourier = str(cfg["three_body_expansion"]).lower() == "fourier"
    M.envelope_exponent, M.cut2, M.cut3 = cfg["envelope_exponent"], cfg["pairwise_cutoff"], cfg["three_body_cutoff"]
    M.emb_table = vec(get("atom_embedding.embedding.weight"))
    M.emb_w = weight(get("atom_embedding.atom_swish_layer.linear.weight"))
    e = "edge_embedding."
    if M.gaussian:
        # GaussianExpansion: the offsets are a buffer, the coefficient is derived from them at construction
        # (matris/model/basis_function.py:203-205: float32 spacing, then Python float arithmetic)
        off = [get(e + n + "_rbf_expansion.offset") for n in ("pairwise", "threebody")]
        M.freq2, M.freq3 = vec(off[0]), vec(off[1])
        M.coeff2, M.coeff3 = (-0.5 / (2.0 * (o[1] - o[0])).item() ** 2 for o in (off[0].cpu(), off[1].cpu()))
    else:
        M.freq2, M.freq3 = (vec(get(e + n + "_rbf_expansion.frequencies")) for n in ("pairwise", "threebody"))
    M.e_w1 = vec(get(e + "edge_linear1.weight"))
    w2, w3 = get(e + "edge_linear2.weight"), get(e + "swish_layer.linear.weight")
    M.e_w2, M.e_w3, M.e_w2t, M.e_w3t = weight(w2), weight(w3), weight(w2.t()), weight(w3.t())
    M.e_lnw, M.e_lnb = vec(get(e + "edge_init_norm.weight")), vec(get(e + "edge_init_norm.bias"))
    t = "three_body_embedding."
    if M.fourier:
        M.t_freq = vec(get(t + "expansion.frequencies"))
    else:
        M.sph_factor = float(sd[t + "expansion.factor"])
    M.t_wa, wb = vec(get(t + "angle_embedding.weight")), get(t + "swish_layer.linear.weight")
    M.t_wb, M.t_wbt = weight(wb), weight(wb.t())
    update = (lambda p, roles=(): k.mlp(p, bias, roles)) if str(cfg["graph_conv_mlp"]).lower() == "mlp" else k.gated
    for i, L in enumerate(layers):
        p = f"interaction_block.{i}."
        for g in ("atom", "line"):
            setattr(L, "attn_" + g, k.attention(f"{p}attn_block_{g}_graph.", update))
            smoothed = bool(cfg["use_smoothed_for_delta_edge"]) and g == "atom"
            setattr(L, "refine_" + g, k.refinement(f"{p}refine_block_{g}_graph.", update, bias, smoothed, g == "line"))
    M.out_norm = vec(get("readout_norm.weight"))
    h = "energy_head.energy_head.layers."
    w0, w3 = get(h + "0.weight"), get(h + "3.weight")
    M.h_w0, M.h_w3, M.h_w0t, M.h_w3t = weight(w0), weight(w3), weight(w0.t()), weight(w3.t())
    M.h_b0, M.h_b3, M.h_w6, M.h_b6 = (vec(get(h + n)) for n in ("0.bias", "3.bias", "6.weight", "6.bias"))
    m = "magmom_head.magmom_head.layers."
    M.m_w0 = weight(get(m + "0.weight"))
    M.m_b0, M.m_w3, M.m_b3 = (vec(get(m + n)) for n in ("0.bias", "3.weight", "3.bias"))
    if cfg["reference_energy"] is not None:
        table = get("reference_energy.fc.weight")
        M.ref_table, M.n_species = vec(table), table.numel()
    M.is_intensive = int(bool(cfg["is_intensive"]))
    return SimpleNamespace(model=M, layers=layers, alive=k.alive)


# ------------------------------------------------------------------ sub-blocks as autograd functions
def row_graphs(g: BatchedGraph):
    """The two message-passing graphs of a batch as the library takes them (rows grouped by target node, the source side
    as a permutation)."""
    p = _lib.ptr
    atom = SimpleNamespace(n_bonds=g.n_bonds, skip_edge_out=False, alive=g, c=_lib.MbRowGraph(
        n_rows=g.n_edges, n_nodes=g.n_atoms, n_edge_rows=g.n_bonds, is_atom=1, tgt=p(g.center), src=p(g.neighbor),
        tgt_ptr=p(g.edge_ptr), src_ptr=p(g.edge_ptr), src_perm=p(g.rev), emap=p(g.d2u), u2d=p(g.u2d), rev=p(g.rev)))
    line = None
    if g.n_triplets:
        cols = g.lg_cols
        line = SimpleNamespace(n_bonds=g.n_bonds, skip_edge_out=False, alive=g, c=_lib.MbRowGraph(
            n_rows=g.n_triplets, n_nodes=g.n_bonds, n_edge_rows=g.n_triplets, n_ctr=g.n_atoms, ctr=p(cols[0]),
            tgt=p(cols[1]), src=p(cols[3]), tgt_ptr=p(g.trip_ptr), src_ptr=p(g.trip_src_ptr), src_perm=p(g.trip_src_perm)))
    return atom, line


def _layer_call(entry, like, *args):
    """Call a sub-block entry point with a workspace of the size it asks for."""
    need = C.c_size_t(0)
    _lib.call(entry, *args, None, C.byref(need), None)
    ws = torch.empty(need.value, dtype=torch.uint8, device=like.device)
    _lib.call(entry, *args, ws.data_ptr(), C.byref(need), ops._stream())


class AttentionFn(torch.autograd.Function):
    """Graph_Attention_Layer.forward (matris/model/interaction_block.py:87-143) and its data gradients."""

    @staticmethod
    def forward(ctx, node, edge, P, rg):
        node, edge = node.contiguous(), edge.contiguous()
        node_out, edge_out = torch.empty_like(node), torch.empty_like(edge)
        p = _lib.ptr
        _layer_call("mb_attention_layer", node, C.byref(P), C.byref(rg.c), p(node), p(edge), p(node_out), p(edge_out), None,
                    None, None, None)
        ctx.save_for_backward(node, edge)
        ctx.P, ctx.rg = P, rg
        return node_out, edge_out

    @staticmethod
    @once_differentiable
    def backward(ctx, d_node_out, d_edge_out):
        node, edge = ctx.saved_tensors
        d_node_out, d_edge_out = d_node_out.contiguous(), d_edge_out.contiguous()
        d_node, d_edge = torch.empty_like(node), torch.empty_like(edge)
        p = _lib.ptr
        _layer_call("mb_attention_layer", node, C.byref(ctx.P), C.byref(ctx.rg.c), p(node), p(edge), None, None,
                    p(d_node_out), p(d_edge_out), p(d_node), p(d_edge))
        return d_node, d_edge, None, None


class RefineFn(torch.autograd.Function):
    """Refinement.forward (matris/model/interaction_block.py:218-278) and its data gradients.  With ``rg.skip_edge_out``
    the edge update is not computed; a placeholder nobody reads keeps the signature (node, edge)."""

    @staticmethod
    def forward(ctx, node, edge, rbf, atom_feat, P, rg):
        node, edge, rbf = node.contiguous(), edge.contiguous(), rbf.contiguous()
        if atom_feat is not None:
            atom_feat = atom_feat.contiguous()
        want_edge = not rg.skip_edge_out
        node_out = torch.empty_like(node)
        edge_out = torch.empty_like(edge) if want_edge else edge.new_empty(0)
        p = _lib.ptr
        _layer_call("mb_refine_layer", node, C.byref(P), C.byref(rg.c), p(node), p(edge), p(rbf), p(atom_feat), p(node_out),
                    p(edge_out) if want_edge else None, None, None, None, None, None, None)
        ctx.save_for_backward(node, edge, rbf, atom_feat)
        ctx.P, ctx.rg, ctx.want_edge = P, rg, want_edge
        if not want_edge:
            ctx.mark_non_differentiable(edge_out)
        return node_out, edge_out

    @staticmethod
    @once_differentiable
    def backward(ctx, d_node_out, d_edge_out):
        node, edge, rbf, atom_feat = ctx.saved_tensors
        d_node_out, d_edge_out = d_node_out.contiguous(), d_edge_out.contiguous() if ctx.want_edge else None
        d_node, d_edge, d_rbf = torch.empty_like(node), torch.empty_like(edge), torch.zeros_like(rbf)
        d_atom = None if atom_feat is None else torch.zeros_like(atom_feat)
        p = _lib.ptr
        _layer_call("mb_refine_layer", node, C.byref(ctx.P), C.byref(ctx.rg.c), p(node), p(edge), p(rbf), p(atom_feat), None,
                    None, p(d_node_out), p(d_edge_out), p(d_node), p(d_edge), p(d_rbf), p(d_atom))
        return d_node, d_edge, d_rbf, d_atom, None, None


# ------------------------------------------------------------------ the module
class _Node(nn.Module):
    """Anonymous container so that parameters sit under the reference's dotted key names."""


def kept_layers_for(n_layers: int, n_triplets: int, n_edges: int, avail: float) -> int:
    """The estimate of ``MatRIS.kept_layers`` as a function of the available bytes."""
    per_layer = 6.7e3 * n_triplets + 6.2e3 * n_edges
    budget = 0.45 * avail
    n_keep = n_layers if per_layer * n_layers < budget else max(0, int(budget // max(per_layer, 1.0)))
    # Second bound, on the peak of the backward pass (saved inputs of all layers + the temporaries of one recomputed
    # layer + gradients).  Measured on three graph shapes (4.1 M - 6.6 M triplets, 1.0 M - 1.7 M directed edges):
    # 17.4 KB per triplet + 13.8 KB per directed edge with nothing kept, growing by 2.5 KB per triplet + 4.3 KB per
    # directed edge per kept layer; that peak must stay below 92 % of the memory.
    base = 18.0e3 * n_triplets + 14.2e3 * n_edges
    step = 2.6e3 * n_triplets + 4.4e3 * n_edges
    # Third bound, on the end of the forward pass (saved inputs of all layers, about 17 KB per triplet, + the kept
    # internals).
    inputs = 17.0e3 * n_triplets + 2.0e3 * n_edges
    while 0 < n_keep < n_layers and max(base + step * n_keep, inputs + per_layer * n_keep) > 0.92 * avail:
        n_keep -= 1
    return n_keep


def split_ranges(triplets, edges, fits) -> list[tuple[int, int]]:
    """Cut a list of structures (per-structure triplet and directed-edge counts) into contiguous ranges with
    ``fits(sum of triplets, sum of edges)`` true for every range, as few as a greedy walk needs and then balanced
    by triplet + edge rows.  A structure that does not fit alone gets a range of its own."""
    triplets, edges = np.asarray(triplets, dtype=np.int64), np.asarray(edges, dtype=np.int64)
    return _split(triplets + edges, lambda a, b: fits(int(triplets[a:b].sum()), int(edges[a:b].sum())))


def _split(rows, fits) -> list[tuple[int, int]]:
    """``split_ranges`` for a predicate of the range itself, ``fits(a, b)``; whatever is part of a range that fits fits too, so
    the longest range from a structure on is found by bisection."""
    n, greedy, a = len(rows), [], 0
    while a < n:
        lo, hi = a + 1, n + 1  # the range [a, lo) is taken, [a, hi) is too long
        while hi - lo > 1:
            mid = (lo + hi) // 2
            lo, hi = (mid, hi) if fits(a, mid) else (lo, mid)
        greedy.append((a, lo))
        a = lo
    if len(greedy) == 1:
        return greedy
    cum = np.cumsum(rows, dtype=np.float64)
    for parts in range(len(greedy), min(n, len(greedy) + 2) + 1):
        cuts = [0] + [int(np.searchsorted(cum, cum[-1] * k / parts, side="left")) + 1 for k in range(1, parts)] + [n]
        ranges = [(cuts[k], cuts[k + 1]) for k in range(parts)]
        if all(b > a for a, b in ranges) and all(b - a == 1 or fits(a, b) for a, b in ranges):
            return ranges
    return greedy


class MatRIS(nn.Module):
    """Drop-in for the reference's ``MatRIS`` (matris/model/model.py:30-317)."""

    def __init__(self, num_layers: int = 6, node_feat_dim: int = 128, edge_feat_dim: int = 128,
                 three_body_feat_dim: int = 128, mlp_hidden_dims=(128, 128), dropout: float = 0.0,
                 use_bias: bool = False, distance_expansion: str = "Bessel", three_body_expansion: str = "SH",
                 num_radial: int = 7, num_angular: int = 7, max_l: int = 4, max_n: int = 4,
                 envelope_exponent: int = 8, graph_conv_mlp: str = "GateMLP", activation_type: str = "silu",
                 norm_type: str = "rms", pairwise_cutoff: float = 6, three_body_cutoff: float = 4,
                 use_smoothed_for_delta_edge: bool = False, learnable_basis: bool = True, is_intensive: bool = True,
                 is_conservation: bool = True, reference_energy: str | None = None, seed: int = 0):
        super().__init__()
        self.config = {k: v for k, v in locals().items() if k not in ("self", "__class__", "seed")}
        cfg = full_config(self.config)
        check_supported(cfg)
        self.is_intensive = is_intensive
        self.graph_converter = GraphConverter(atom_graph_cutoff=pairwise_cutoff, line_graph_cutoff=three_body_cutoff)
        for key, value in random_state_dict(cfg, seed=seed).items():
            self._register(key, value, buffer=key in BUFFER_KEYS, trainable=not key.startswith("reference_energy"))
        self._packed = None
        self._packed_device = None
        self.last_batch = None
        # None: decide per call from free memory; True / False: keep / recompute all; n: keep the last n layers' internals
        self.keep_activations = None
        # plan as if at most this many bytes of device memory were available (None: what the device has left)
        self.memory_limit_bytes = None

    # -- parameter tree -------------------------------------------------------------------
    def _register(self, key, value, buffer, trainable):
        mod = self
        parts = key.split(".")
        for p in parts[:-1]:
            if not hasattr(mod, p):
                mod.add_module(p, _Node())
            mod = getattr(mod, p)
        if buffer:
            mod.register_buffer(parts[-1], value.clone())
        else:
            mod.register_parameter(parts[-1], nn.Parameter(value.clone(), requires_grad=False))

    def get_params(self) -> int:
        return sum(p.numel() for p in self.parameters())

    def _apply(self, fn, *a, **k):
        self._packed = None
        out = super()._apply(fn, *a, **k)
        # graphs are built where the weights live: a batch on another GPU would be read through peer pointers
        # (or fault without peer access) by kernels launched on this one
        dev = self.device
        self.graph_converter.device = dev if dev.type == "cuda" else None
        return out

    def load_state_dict(self, state_dict, strict: bool = True, **kw):
        self._packed = None
        return super().load_state_dict(state_dict, strict=strict, **kw)

    def packed(self, device):
        if self._packed is None or self._packed_device != device:
            self._packed = pack_parameters(self.state_dict(), full_config(self.config), device)
            self._packed_device = device
        return self._packed

    @property
    def device(self):
        return next(self.parameters()).device

    # -- checkpoint interface ---------------------------------------------------------------
    @classmethod
    def from_dict(cls, dct: dict):
        model = MatRIS(**dct["config"])
        model.load_state_dict(dct["state_dict"])
        return model

    @classmethod
    def load(cls, model_name: str = "matris_10m_oam", device: str | None = None, path: str | None = None):
        """Load a checkpoint ``{"config", "state_dict"}``.  ``model_name`` resolves to
        ``~/.cache/matris/MatRIS_10M_{OAM,MP}.pth.tar`` exactly like the reference
        (matris/model/model.py:262-317); ``path`` (an extension) names the file directly."""
        if path is None:
            model_name = model_name.lower()
            supported = ["matris_10m_oam", "matris_10m_mp"]
            if os.path.isfile(model_name):
                path = model_name
            elif model_name not in supported:
                raise ValueError(f"Unsupported model_name: {model_name}. Supported models are: {supported}")
            else:
                files = {"matris_10m_oam": "MatRIS_10M_OAM.pth.tar", "matris_10m_mp": "MatRIS_10M_MP.pth.tar"}
                urls = {"matris_10m_oam": "https://figshare.com/ndownloader/files/59142728",
                        "matris_10m_mp": "https://figshare.com/ndownloader/files/59143058"}
                cache_dir = os.path.expanduser("~/.cache/matris")
                os.makedirs(cache_dir, exist_ok=True)
                path = os.path.join(cache_dir, files[model_name])
                if not os.path.exists(path):
                    print(f"Checkpoint not found, downloading to {path} ...")
                    torch.hub.download_url_to_file(urls[model_name], path)
        if device is None:
            device = "cuda"
        ckpt = torch.load(path, map_location=torch.device("cpu"), weights_only=False)
        model = MatRIS.from_dict(ckpt).to(device)
        print(f"Loading {model_name} successfully, running on {device}.")
        return model

    # -- evaluation -------------------------------------------------------------------------
    def _as_batch(self, graphs) -> BatchedGraph:
        if isinstance(graphs, BatchedGraph):
            if graphs.device != self.device:
                raise ValueError(f"the batch lives on {graphs.device} but the model on {self.device}: build it with "
                                 "model.graph_converter (which follows the model) or pass device= to "
                                 "build_batched_graph")
            return graphs
        if isinstance(graphs, RadiusGraph):
            graphs = [graphs]
        graphs = list(graphs)
        if not graphs:
            raise ValueError("no graphs")
        b0 = getattr(graphs[0], "_batch", None)
        if (b0 is not None and len(graphs) == b0.n_struct and b0.device == self.device
                and all(getattr(g, "_batch", None) is b0 and g._index == i for i, g in enumerate(graphs))):
            return b0
        arrays = [g.source_arrays() if isinstance(g, RadiusGraph) else as_arrays(g) for g in graphs]
        return build_batched_graph([a[0] for a in arrays], [a[1] for a in arrays], [a[2] for a in arrays],
                                   self.config["pairwise_cutoff"], self.config["three_body_cutoff"], self.device)

    def _check_elements(self, g: BatchedGraph) -> None:
        """The kernels look atoms up in tables by their number without a test of their own."""
        n = self.atom_embedding.embedding.weight.shape[0]
        lo, hi = g.number_range
        if lo < 1 or hi > n:
            raise IndexError(f"atomic numbers from {lo} to {hi}: the model knows the elements 1 to {n}")

    def forward(self, graphs: Sequence[RadiusGraph] | BatchedGraph, task: str = "ef", is_training: bool = False):
        """Same result dictionary as the reference's ``MatRIS.forward`` (model.py:183-250): ``e`` [B] energy per
        atom including the reference energy, ``f`` tuple of [n_i,3], ``s`` list of [3,3] in GPa, ``m`` list of
        [n_i], ``atoms_per_graph``, ``ref_energy``.  ``graphs`` may also be a ``BatchedGraph``."""
        if is_training:
            raise NotImplementedError("matris_b200 evaluates frozen models only (no parameter gradients)")
        if self.device.type != "cuda":
            raise RuntimeError("matris_b200 runs on a CUDA device only: move the model with .to('cuda')")
        g = self._as_batch(graphs)
        self._check_elements(g)
        self.last_batch = g
        with torch.cuda.device(g.device):
            # The GEMM kernels bound every wait and raise a status word instead of hanging.  The word of the previous
            # evaluation was copied to pinned memory in stream order; it is read here, so a failure surfaces at the
            # latest one call later and costs no synchronisation.
            flag = getattr(self, "_gemm_flag", None)
            if flag is None:
                flag = self._gemm_flag = torch.zeros(1, dtype=torch.int32).pin_memory()
            self.check_status()
            out = self._evaluate(g, task)
            ops.gemm_status_async(flag)
            return out

    def check_status(self) -> None:
        """Raise if a bounded wait of a tensor-core kernel expired in an evaluation whose status word has reached
        the host (``forward`` enqueues the copy; it is valid once the stream has been synchronised, e.g. by reading
        a result).  The word is cleared on raising, so that one expiry does not disable the model."""
        flag = getattr(self, "_gemm_flag", None)
        if flag is not None and int(flag[0]) != 0:
            status = int(flag[0])
            flag.zero_()
            with torch.cuda.device(self.device):
                ops.gemm_status_clear()
            raise MbError(f"a tensor-core kernel's bounded wait expired (status {status}): the results of that "
                          "evaluation are invalid")

    # -- memory policy -----------------------------------------------------------------------
    def _available_bytes(self) -> float:
        """Memory the allocator can still hand out = device total - what lives outside this allocator - what it has
        allocated (capped by ``memory_limit_bytes`` when set).  The driver query behind the middle term costs
        milliseconds (during which the GPU idles at the start of an evaluation), so it is refreshed every 64th call
        only; the last term is a counter."""
        st = getattr(self, "_mem_state", None)
        if st is None:
            st = self._mem_state = {"calls": 0, "total": 0, "outside": 0}
        if st["calls"] % 64 == 0:
            free, total = torch.cuda.mem_get_info(self.device)
            st["total"], st["outside"] = total, total - free - torch.cuda.memory_reserved(self.device)
        st["calls"] += 1
        # (the one counter: torch.cuda.memory_allocated would flatten all of them on every call, while the device idles)
        counters = torch.cuda.memory_stats_as_nested_dict(self.device)
        allocated = counters["allocated_bytes"]["all"]["current"] if counters else 0
        avail = st["total"] - st["outside"] - allocated
        if self.memory_limit_bytes is not None:
            avail = min(avail, float(self.memory_limit_bytes))
        return avail

    def _fixed_layers(self) -> int | None:
        """The number of layers ``keep_activations`` names (None: it leaves the choice to the memory policy)."""
        n_layers, keep = int(self.config["num_layers"]), self.keep_activations
        if keep is None or isinstance(keep, bool):
            return None if keep is None else n_layers * keep
        return max(0, min(n_layers, int(keep)))

    def kept_layers(self, n_triplets: int, n_edges: int, avail: float | None = None) -> int:
        """An estimate, without a graph in hand, of how many (last) layers keep their internals for the backward pass on a
        batch with that many triplet rows and directed edges, on the safe side of what ``forward`` finds out from the
        exact need of the evaluation.  ``avail``: bytes to plan with (None: what the device has left); ``keep_activations``
        overrides."""
        fixed = self._fixed_layers()
        if fixed is not None:
            return fixed
        return kept_layers_for(int(self.config["num_layers"]), n_triplets, n_edges,
                               self._available_bytes() if avail is None else avail)

    def _need(self, e: _lib.MbEval, keep: int) -> int:
        """Bytes the evaluation ``e`` has in use at most when its last ``keep`` layers keep their internals."""
        size, e.keep_layers = C.c_size_t(0), keep
        _lib.check(_lib.load().mb_evaluate_workspace(C.byref(e), C.byref(size)), "mb_evaluate_workspace")
        return size.value

    def _plan_memory(self, e: _lib.MbEval) -> int:
        """Decide how many (last) layers keep their internals for the backward pass - as many as fit in memory, or what
        ``keep_activations`` says - and set it in ``e``; returns the bytes the evaluation will use."""
        n_layers, fixed = e.model.contents.n_layers, self._fixed_layers()
        if fixed is not None:
            return self._need(e, fixed)
        budget = MEMORY_SHARE * self._available_bytes()
        # the need grows with the number of kept layers: the largest that fits, by bisection
        best = self._need(e, n_layers)
        if best <= budget:
            return best
        lo, hi = 0, n_layers
        while hi - lo > 1:
            mid = (lo + hi) // 2
            lo, hi = (mid, hi) if self._need(e, mid) <= budget else (lo, mid)
        return self._need(e, lo)

    def split_for_memory(self, g: BatchedGraph, headroom: float = 0.93) -> list[tuple[int, int]]:
        """Contiguous ranges of the structures of batch ``g`` such that every range, evaluated as a batch of its own,
        keeps the internals of all layers (no recomputation in the backward pass): ``[(0, n_struct)]`` when the
        whole batch does.  Structures are independent, so evaluating the ranges one after another gives the same
        results; on a batch that would recompute most layers it is about a fifth faster.  ``headroom`` scales the
        available memory the plan may count on (the ranges' own graphs and results take some)."""
        if g.n_struct <= 1 or self.keep_activations is not None:
            return [(0, g.n_struct)]
        P, n_layers = self.packed(g.device), int(self.config["num_layers"])
        budget = MEMORY_SHARE * self._available_bytes()
        e = _lib.MbEval()
        e.model = C.pointer(P.model)
        e.f = e.s = e.m = 256  # all outputs (the counts alone matter to a dry run; nothing is read)

        def need(n_atoms, n_struct, n_edges, n_triplets):
            e.n_atoms, e.n_struct, e.n_edges, e.n_bonds, e.n_triplets = n_atoms, n_struct, n_edges, n_edges // 2, n_triplets
            return self._need(e, n_layers)

        if need(g.n_atoms, g.n_struct, g.n_edges, g.n_triplets) <= budget:
            return [(0, g.n_struct)]
        ap, ep, _, tp = (np.asarray(p, dtype=np.int64) for p in g.structure_slices())
        return _split(np.diff(tp) + np.diff(ep), lambda a, b: need(int(ap[b] - ap[a]), b - a, int(ep[b] - ep[a]),
                                                                   int(tp[b] - tp[a])) <= headroom * budget)

    def _evaluate(self, g: BatchedGraph, task: str):
        dev, n_struct, n_atoms = g.device, g.n_struct, g.n_atoms
        P = self.packed(dev)
        want = {"f": 3 * n_atoms if "f" in task else 0, "s": 9 * n_struct if "s" in task else 0,
                "m": n_atoms if "m" in task else 0}
        e, p = _lib.MbEval(), _lib.ptr
        e.model = C.pointer(P.model)
        e.n_atoms, e.n_struct, e.n_edges, e.n_bonds, e.n_triplets = n_atoms, n_struct, g.n_edges, g.n_bonds, g.n_triplets
        e.cart, e.lattice, e.volume = p(g.cart32), p(g.lattice32), p(g.volume)
        e.atom_struct, e.atom_ptr, e.numbers = p(g.atom_struct), p(g.atom_ptr), p(g.numbers)
        e.center, e.neighbor, e.image, e.edge_ptr = p(g.center), p(g.neighbor), p(g.image), p(g.edge_ptr)
        e.rev, e.d2u, e.u2d = p(g.rev), p(g.d2u), p(g.u2d)
        e.trip_ptr, e.trip_src_ptr, e.trip_src_perm = p(g.trip_ptr), p(g.trip_src_ptr), p(g.trip_src_perm)
        e.line_graph, e.lg_cols = p(g.line_graph), p(g.lg_cols)
        energy, ref = (torch.empty(n_struct, dtype=torch.float32, device=dev) for _ in range(2))
        apg = torch.empty(n_struct, dtype=torch.int32, device=dev)
        res = {k: torch.empty(n, dtype=torch.float32, device=dev) for k, n in want.items() if n}
        e.e, e.ref, e.atoms_per_struct = p(energy), p(ref), p(apg)
        e.f, e.s, e.m = (p(res.get(k)) for k in ("f", "s", "m"))
        size = self._plan_memory(e)
        self.last_kept_layers = e.keep_layers
        if size <= WORKSPACE_LIMIT:
            # sizes in steps of an eighth of their power of two, so that the slightly different graphs of successive steps
            # find the block of the step before in the allocator's cache
            step = 1 << max(12, size.bit_length() - 4)
            size = (size + step - 1) // step * step
            ws = torch.empty(size, dtype=torch.uint8, device=dev)
            e.ws, e.ws_bytes = ws.data_ptr(), size
        else:
            stream = torch.cuda.current_stream(dev)

            def alloc(n):
                try:
                    return torch.cuda.caching_allocator_alloc(n, dev, stream)
                except torch.cuda.OutOfMemoryError:  # comes back as a status code
                    return None
            e.alloc, e.release = _lib.ALLOC_FN(alloc), _lib.FREE_FN(torch.cuda.caching_allocator_delete)
        _lib.evaluate(e, ops._stream())
        out = {}
        if "f" in res:
            out["f"] = torch.split(res["f"].view(n_atoms, 3), g.atoms_per_graph)
        if "s" in res:
            out["s"] = list(torch.unbind(res["s"].view(n_struct, 3, 3), dim=0))
        if "m" in res:
            out["m"] = list(torch.split(res["m"], g.atoms_per_graph))
        out["e"], out["atoms_per_graph"] = energy, apg
        out["ref_energy"] = ref if self.config["reference_energy"] is not None else 0
        return out

    # -- convenience ------------------------------------------------------------------------
    def plan_batches(self, structures) -> list[BatchedGraph]:
        """The device-resident graphs ``predict`` evaluates for a list of structures: one batch when the internals of
        every layer fit in memory beside it, otherwise the contiguous sub-batches of ``split_for_memory``."""
        structures = list(structures)
        g = self.graph_converter.batch(structures)
        ranges = self.split_for_memory(g)
        if len(ranges) == 1:
            return [g]
        del g
        return [self.graph_converter.batch(structures[a:b]) for a, b in ranges]

    def forward_batches(self, graphs: Sequence[BatchedGraph], task: str = "efsm") -> dict:
        """Evaluate sub-batches one after another and join the results in order: the dictionary ``forward`` returns
        for the concatenated list of structures."""
        outs = [self.forward(g, task=task) for g in graphs]
        if len(outs) == 1:
            return outs[0]
        res = {"e": torch.cat([o["e"] for o in outs]), "atoms_per_graph": torch.cat([o["atoms_per_graph"] for o in outs])}
        ref = [o["ref_energy"] for o in outs]
        res["ref_energy"] = torch.cat(ref) if torch.is_tensor(ref[0]) else ref[0]
        if "f" in outs[0]:
            res["f"] = tuple(t for o in outs for t in o["f"])
        for k in ("s", "m"):
            if k in outs[0]:
                res[k] = [t for o in outs for t in o[k]]
        return res

    def predict(self, structures, task: str = "efsm"):
        """Evaluate a list of structures (any accepted structure type): as one batch, or, when the backward pass of
        that batch would have to recompute layers for lack of memory, as the sub-batches of ``plan_batches``."""
        return self.forward_batches(self.plan_batches(structures), task=task)

    def predict_sharded(self, structures, task: str = "efsm", group=None, dst: int = 0):
        """``predict`` over all ranks of a ``torch.distributed`` group (one process per GPU, every rank passes the
        same list): structures are assigned to ranks by predicted cost, evaluated locally, and E / F / S / M are
        gathered to rank ``dst`` (see matris_b200.parallel.evaluate).  Returns the full result there, None elsewhere."""
        from .parallel import evaluate
        return evaluate(self, structures, task, group=group, dst=dst)
