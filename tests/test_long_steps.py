"""Steps of many rows through the kernels that only they reach: latent attention over heads made for the step, experts'
products in tiles of 128 entries, selective scans and recurrences over pieces.  At the edges of tiles and pieces, against the
plain implementation (tests/plain_vunelix.py) or the sums written out."""
import json
import os

import numpy as np
import pytest
import torch

from conftest import random_tokens
from infinicore_infer_b200.kernels.host import conv_walks_rows, experts_take_tiles
import plain_vunelix as plain

pytestmark = pytest.mark.gpu
F = torch.float64


@pytest.fixture(scope="module")
def K():
    from infinicore_infer_b200 import kernels
    return kernels


@pytest.mark.parametrize("heads,dim,rank", [(3, 64, 72), (2, 128, 64), (16, 128, 512)])
def test_latent_attention_over_heads_made_for_the_step(tmp_path, heads, dim, rank):
    """Prompts and portions of one and several requests, tiles of 128 rows and keys at their edges.  The other way of running the
    same records, over the latent rows, has the same operands and one rounding to bfloat16 more or less at each of its
    products: both lie within a few units of 2^-8 of the float64 model, and of each other."""
    from infinicore_infer_b200.config import config_class_for
    from infinicore_infer_b200.engine import Engine, StepEntry
    from infinicore_infer_b200.weights import index_directory, read_tensor, write_model_folder
    cfg = {"architecture": "Vunelix", "norm": {"eps": 1e-5}, "vocab": 97, "width": 64, "logit_softcap": None, "layers": [
        {"type": "latent_attention", "mlp": None, "mixer": {"heads": heads, "dim": dim, "rot_dim": 64, "vdim": dim, "kv_rank": rank,
                                                            "scale": (dim + 64) ** -0.5, "rot": {"base": 1e3, "dims": 32}}}]}
    write_model_folder(config_class_for(cfg).from_dict(cfg), str(tmp_path), seed=5, std=0.16, norm_std=0.2)
    with open(os.path.join(tmp_path, "config.json")) as f:
        disk = json.load(f)
    weights = {n: read_tensor(i).float() for n, i in index_directory(str(tmp_path)).items()}
    engine = Engine.from_folder(str(tmp_path), max_tokens=640, cache_tokens=1280, page_size=16, max_requests=3, max_step_tokens=512)
    toks = [random_tokens(s, 400, 97) for s in range(3)]
    want = [plain.forward(t, disk, weights) for t in toks]
    scale = want[0].std()
    # (request, from, to) of every step's entries; the last step decodes
    steps = [[(0, 0, 128)], [(0, 128, 148), (1, 0, 129)], [(0, 148, 400)], [(1, 129, 385), (2, 0, 64)], [(2, 64, 200)], [(1, 385, 386), (2, 200, 201)]]
    logits = {}
    for other_way in (False, True):
        engine.runtime.plain_attention = other_way
        rows = []
        for step in steps:
            out = engine.step([StepEntry((other_way, r), toks[r][a:b], list(range(b - a))) for r, a, b in step])
            rows.append(out.double().cpu())
            ref = torch.cat([want[r][a:b] for r, a, b in step])
            err = (rows[-1] - ref).square().mean().sqrt() / scale
            assert err <= 0.03, f"{step}, over the latent rows: {other_way}: {err:.4f} of the logits' spread"
        logits[other_way] = torch.cat(rows)
        for r in range(3):
            engine.end((other_way, r))
    engine.check()
    engine.runtime.plain_attention = False
    assert (logits[False] - logits[True]).square().mean().sqrt() <= 0.03 * scale
    assert not torch.equal(logits[False], logits[True])         # both ways ran


def _one_layer(family, mixer):
    extra = {"vunelix": dict(logit_softcap=None), "fupapel": dict(residual_mult=1.0),
             "fapenex": dict(max_positions=640, logit_scale=1.0, logit_softcap=None)}[family]
    return dict(architecture=family.capitalize(), norm=dict(eps=1e-5), vocab=97, width=64, layers=[dict(type="latent_attention", mlp=None, mixer=mixer)], **extra)


@pytest.mark.parametrize("family,heads,dim,rot,rank,q_rank,window", [
    ("fapenex", 2, 128, 0, 128, 40, 100), ("fapenex", 3, 64, 0, 136, 40, 100), ("fapenex", 2, 128, 0, 128, 40, 600),       # queries through a latent, a window
    ("fupapel", 2, 128, 64, 72, 48, 0), ("fupapel", 3, 64, 64, 64, 40, 0),      # and rotated parts, learned sinks, a gate per head
    ("vunelix", 2, 128, 64, 64, 0, 0)])                                         # neither; a gate per element
def test_every_form_of_latent_attention_over_heads_and_who_goes_which_way(tmp_path, family, heads, dim, rot, rank, q_rank, window):
    """Every instance and option, prompts and portions whose tiles end inside other requests' rows (with a query latent the output lies
    where the plain queries lay), windows that cross key tiles.  A step goes over heads as a whole: one request of eight rows or fewer
    keeps all of it on the latent rows, where the bits are those of an engine that knows no other way.  Both ways round operands and
    results to bfloat16 (2^-9 each, about ten on the way to a logit): within 0.03 of the logits' spread of float64."""
    import importlib
    from infinicore_infer_b200.config import config_class_for
    from infinicore_infer_b200.engine import Engine, StepEntry
    from infinicore_infer_b200.weights import index_directory, read_tensor, write_model_folder
    mixer = dict(heads=heads, dim=dim, vdim=dim, kv_rank=rank, scale=(dim + rot) ** -0.5)
    mixer.update(dict(rot_dim=rot, rot=dict(base=1e3, dims=64 if q_rank else 32)) if rot else {}, **(dict(q_rank=q_rank) if q_rank else {}),
                 **(dict(mask=dict(size=window)) if window else {}))
    cfg = _one_layer(family, mixer)
    write_model_folder(config_class_for(cfg).from_dict(cfg), str(tmp_path), seed=heads + dim, std=0.16, norm_std=0.2)
    with open(os.path.join(tmp_path, "config.json")) as f:
        disk = json.load(f)
    index = index_directory(str(tmp_path))
    toks = [random_tokens(s, 400, 97) for s in range(3)]
    reference = importlib.import_module("plain_" + family)
    if family == "vunelix":
        weights = {n: read_tensor(i).float() for n, i in index.items()}
        want = [reference.forward(t, disk, weights) for t in toks]
    else:
        weights = {n: read_tensor(i).double().numpy() for n, i in index.items()}
        want = [torch.from_numpy(np.asarray(reference.forward(disk, weights, t))) for t in toks]
    engine = Engine.from_folder(str(tmp_path), max_tokens=640, cache_tokens=1280, page_size=16, max_requests=3, max_step_tokens=512)
    # (over heads, (request, from, to) of every entry); a step that has a request of at most eight rows is not
    steps = [(True, [(0, 0, 150)]), (True, [(0, 150, 190), (1, 0, 129)]), (False, [(1, 129, 321), (0, 190, 191)]), (False, [(2, 0, 8), (1, 321, 395)]),
             (True, [(2, 8, 200), (0, 191, 400)]), (False, [(1, 395, 396), (2, 200, 201)])]
    got = {}
    for other_way in (False, True):
        engine.runtime.plain_attention = other_way
        got[other_way] = [engine.step([StepEntry((other_way, r), toks[r][a:b], list(range(b - a))) for r, a, b in step]).double().cpu() for _, step in steps]
        for r in range(3):
            engine.end((other_way, r))
    engine.check()
    engine.runtime.plain_attention = False
    for (over_heads, step), one, other in zip(steps, got[False], got[True]):
        ref = torch.cat([want[r][a:b] for r, a, b in step])
        for out in (one, other):
            err = (out - ref).square().mean().sqrt() / want[0].std()
            assert err <= 0.03, f"{step}: {err:.4f} of the logits' spread"
        assert torch.equal(one, other) == (not over_heads), step


@pytest.mark.parametrize("dh,rotated,tile_keys", [(64, False, 128), (64, True, 128), (128, False, 64), (128, False, 128), (128, True, 128)])
def test_weights_of_an_attention_over_laid_heads_are_float32_accurate(K, dh, rotated, tile_keys):
    """Each instance, with values that pick single weights: row t has scores -a_t b_j (exact in float32) over 64 keys and far lower ones
    over the rest, and column j of its output is key j's weight, rounded to bfloat16 as an operand, over the float32 sum of the weights,
    rounded once more.  Scores in [-8, 0]: the exponent's factor and product err by 8 x 1.5 x 2^-24, the special-function unit by 2^-22, the sum
    and the quotient by another 2^-22; each of the two roundings moves by at most twice that over the spacing 2^-8: 2^-10 of them
    in all."""
    dev, g, T, before = torch.device("cuda:0"), torch.Generator().manual_seed(dh), 1000, 200
    C = T + before
    a = (torch.rand(T, generator=g) * 1.5 + 0.5).to(torch.bfloat16)
    b = (torch.rand(64, generator=g) * 4).to(torch.bfloat16)
    b[0] = 0
    q, kv, out = torch.zeros(T, dh), torch.zeros(C, 2 * dh), torch.empty(T, dh, dtype=torch.bfloat16, device=dev)
    q[:, 3] = a.float()
    kv[:64, 3], kv[64:, 3] = -b.float(), -256.0
    kv[:64, dh:dh + 64] = torch.eye(64)
    q, kv = q.to(torch.bfloat16).to(dev), kv.to(torch.bfloat16).to(dev)
    q_rot, k_rot = torch.zeros(T, 72, dtype=torch.bfloat16, device=dev), torch.zeros(C, 64, dtype=torch.bfloat16, device=dev)
    n = (T + 127) // 128
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    tiles, start, pos, status = ints([[0, 128 * i, 0] for i in reversed(range(n))]), ints([0, T]), ints([before]), K.gemm_status(dev)
    i, p = K._c_int, K._ptr
    K._check("attention_tcgen05", K._build.load("attention_tcgen05").jk_attention_laid_tcgen05(
        p(q), p(q_rot if rotated else None), i(72), i(8), p(kv), p(k_rot if rotated else None), K._c_ll(C), p(out), p(tiles), i(n), i(T), p(start), p(pos),
        i(1), i(dh), K._c_float(1.0), i(0), p(status), p(None), p(None), i(0), i(0), i(tile_keys), K._stream()))
    K.check_gemm_status(dev)
    e = torch.exp(-a.double()[:, None] * b.double())
    want = e.to(torch.bfloat16).double() / e.sum(1, keepdim=True)
    got = out[:, :64].double().cpu()
    assert ((got - want).abs() <= 2.0 ** -6 * want).all()
    assert (got != want.to(torch.bfloat16).double()).double().mean() <= 2.0 ** -10


@pytest.mark.parametrize("T,d,ff,experts,top,act", [(128, 1024, 256, 1, 1, "silu"), (129, 1032, 264, 2, 2, "swish_clamp"), (300, 1096, 264, 5, 2, "silu"),
                                                    (600, 32776, 8, 3, 1, "silu")])
def test_expert_products_in_tiles_of_entries(K, T, d, ff, experts, top, act):
    """Entries that fill tiles of 128 exactly, by one more and by part, an expert without rows (the router's bias shuns it), widths
    that end inside a tile and inside a step of K.  A product's operands are exact, its sums float32, the inner activations
    rounded to bfloat16: 2^-9 of each, averaged over ff of them."""
    dev, g = torch.device("cuda:0"), torch.Generator().manual_seed(T + d)
    assert experts_take_tiles(T * top, experts, d, ff)
    h = torch.randn(T, d, generator=g).to(torch.bfloat16)
    w_gu, w_dn = (torch.randn(experts * n, k, generator=g).div(k ** 0.5).to(torch.bfloat16) for n, k in ((2 * ff, d), (d, ff)))
    router = torch.randn(experts, d, generator=g)
    bias = torch.zeros(experts)
    if experts > 2:
        bias[1] = -1e3
    code = {"silu": K.ACT_SILU, "swish_clamp": 6}[act]
    delta = torch.full((T, d), 9.0, device=dev)
    K.routed_experts(h.to(dev), router.to(dev), w_gu.to(dev), w_dn.to(dev), delta, False, experts, top, code, score_form=1, limit=1.5,
                     router_bias=bias.to(dev))
    K.check_gemm_status(dev)
    z = h.double() @ router.double().T + bias.double()
    score = torch.softmax(z, -1)
    chosen = z.topk(top, -1).indices
    want = torch.zeros(T, d, dtype=F)
    for e in range(experts):
        rows = (chosen == e).any(-1)
        gu = h[rows].double() @ w_gu[e * 2 * ff: (e + 1) * 2 * ff].double().T
        a, u = gu[:, :ff], gu[:, ff:]
        if act == "silu":
            inner = plain.silu(a) * u
        else:
            a, u = a.clamp(max=1.5), u.clamp(-1.5, 1.5)
            inner = a * torch.sigmoid(1.702 * a) * (u + 1)
        share = score[rows, e] / (score[rows].gather(1, chosen[rows]).sum(-1) + 1e-20)
        want[rows] += share.unsqueeze(-1) * (inner @ w_dn[e * d: (e + 1) * d].double().T)
    err = (delta.double().cpu() - want).abs().max()
    assert err <= 2.0 ** -8 * want.abs().max(), float(err)


@pytest.mark.parametrize("act", ["none", "silu", "gelu_tanh", "sigmoid", "relu", "swish_clamp"])
def test_expert_products_of_groups_of_rows_that_are_part_full(K, act):
    """Experts with 1, 31, 33, 63 and 142 entries: the groups of 32 rows that a warp of the products finishes are full, part full and
    empty, over 208 and 1,288 features, so that a warp comes back for more columns after a pass in which some of its rows had nothing
    to store.  Every activation; scores that multiply the units' inputs.  The bound of the test above."""
    dev, g = torch.device("cuda:0"), torch.Generator().manual_seed(len(act))
    counts, d, ff, limit = [1, 31, 33, 63, 142], 1288, 208, 1.5
    T, E = sum(counts), len(counts)
    assert experts_take_tiles(T, E, d, ff)
    owner = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T, generator=g)]
    h = torch.randn(T, d, generator=g)
    h[:, :E] = 20.0 * torch.nn.functional.one_hot(owner, E)         # the router reads the owner
    h = h.to(torch.bfloat16)
    router = torch.zeros(E, d)
    router[:, :E] = torch.eye(E)
    w_gu, w_dn = (torch.randn(E * n, k, generator=g).div(k ** 0.5).to(torch.bfloat16) for n, k in ((2 * ff, d), (d, ff)))
    w_gu[:, :E] = 0.0
    delta = torch.full((T, d), 9.0, device=dev)
    code = {"none": 0, "silu": 1, "gelu_tanh": 2, "sigmoid": 3, "relu": 4, "swish_clamp": 6}[act]
    K.routed_experts(h.to(dev), router.to(dev), w_gu.to(dev), w_dn.to(dev), delta, False, E, 1, code, limit=limit)
    K.check_gemm_status(dev)
    score = 1.0 / (1.0 + np.exp(-20.0))                             # the default form: sigmoid of the router's output, times the inputs
    want = torch.zeros(T, d, dtype=F)
    for e in range(E):
        rows = owner == e
        gu = score * (h[rows].double() @ w_gu[e * 2 * ff: (e + 1) * 2 * ff].double().T)
        a, u = gu[:, :ff], gu[:, ff:]
        if act == "swish_clamp":
            a, u = a.clamp(max=limit), u.clamp(-limit, limit)
            inner = a * torch.sigmoid(1.702 * a) * (u + 1)
        else:
            f = {"none": lambda x: x, "silu": plain.silu, "sigmoid": torch.sigmoid, "relu": torch.relu,
                 "gelu_tanh": lambda x: torch.nn.functional.gelu(x, approximate="tanh")}[act]
            inner = f(a) * u
        want[rows] = inner @ w_dn[e * d: (e + 1) * d].double().T
    err = (delta.double().cpu() - want).abs().max()
    assert err <= 2.0 ** -8 * want.abs().max(), float(err)


@pytest.mark.parametrize("act,code,least", [("silu", 1, -88.5), ("sigmoid", 3, -80.0), ("gelu_tanh", 2, -9.9), ("swish_clamp", 6, -52.0),
                                            ("none", 5, -88.5), ("none", 7, -88.5)])
def test_experts_units_are_float32_accurate_over_the_gates_range(K, act, code, least):
    """One expert whose rows of W pick single elements of a row: gates and ups arrive exactly, from where the unit vanishes on, and what
    leaves is the unit rounded to bfloat16.  A rounding is 2^-8 at most; what float32 adds before it (e^-s to one unit in the last place, a
    sum, a quotient, a product: 2.5 x 2^-23; three roundings of s where it is not the gate) seldom moves one: by at most twice that
    over the spacing 2^-8, 2^-12 where s is the gate.  Codes that name no unit of an expert leave the gate as it is."""
    dev, g, T, ff, limit = torch.device("cuda:0"), torch.Generator().manual_seed(code), 300, 1024, 4.0
    z = (least + (8.0 - least) * torch.rand(T, ff, generator=g)).to(torch.bfloat16)
    z[:, :3] = torch.tensor([-88.5, -88.0, -87.5]).clamp(min=least)
    up = torch.randn(T, ff, generator=g).abs().add(1.0).to(torch.bfloat16)
    h, w_gu, w_dn = torch.cat([z, up], 1).to(dev), torch.eye(2 * ff, dtype=torch.bfloat16, device=dev), torch.zeros(2 * ff, ff, dtype=torch.bfloat16, device=dev)
    w_dn[:ff] = torch.eye(ff)
    delta = torch.empty(T, 2 * ff, device=dev)
    K.routed_experts(h, torch.zeros(1, 2 * ff, device=dev), w_gu, w_dn, delta, False, 1, 1, code, score_form=1, limit=limit)        # a score of 1
    K.check_gemm_status(dev)
    z, up, got = z.double(), up.double(), delta[:, :ff].double().cpu()
    if act == "swish_clamp":
        z, up = z.clamp(max=limit), up.clamp(-limit, limit) + 1
    s = {"gelu_tanh": 2 * (2 / np.pi) ** 0.5 * (z + 0.044715 * z ** 3), "swish_clamp": 1.702 * z}.get(act, z)
    want = {"sigmoid": torch.sigmoid(s), "none": z}.get(act, z * torch.sigmoid(s)) * up
    exact = act in ("silu", "sigmoid", "none")
    before = 2.5 * 2.0 ** -23 + (0 if exact else 3 * 2.0 ** -24 * s.abs())
    assert ((got - want).abs() <= (2.0 ** -8 + before) * want.abs()).all()
    if exact:
        assert (got != want.to(torch.bfloat16).double()).double().mean() <= 2.0 ** -12


@pytest.mark.parametrize("states", [5, 16, 20])
@pytest.mark.parametrize("lens", [(768,), (1793, 1, 513), (1475, 64), (900, 640), (896,), (1921, 1, 769), (2500, 65)])
def test_selective_scan_over_pieces(K, states, lens):
    """Requests of exactly one piece, of one row more, and of several, from states that are not zero; 130 channels.  Float32
    throughout: rounding of 2^-24 a step over a chain whose decays are below 1."""
    dev, g, E, rank = torch.device("cuda:0"), torch.Generator().manual_seed(states), 130, 3
    T = sum(lens)
    x, z = torch.randn(T, E, generator=g), torch.randn(T, E, generator=g)
    low = torch.randn(T, rank + 2 * states, generator=g)
    w_dt, b_dt = torch.randn(E, rank, generator=g) * 0.3, torch.randn(E, generator=g) - 3.0
    A, skip = -torch.exp(torch.randn(E, states, generator=g)), torch.randn(E, generator=g)
    first = torch.randn(len(lens) + 1, E, states, generator=g)
    state, slots = first.clone().to(dev), torch.arange(len(lens), 0, -1, dtype=torch.int32)
    starts = torch.tensor([0] + list(lens)).cumsum(0).to(torch.int32)
    out = torch.empty(T, E, device=dev)
    K.selective_scan(x.to(dev), low.to(dev), rank, states, z.to(dev), E, w_dt.to(dev), b_dt.to(dev), A.to(dev), skip.to(dev), state, starts.to(dev),
                     slots.to(dev), out, dt_buf=torch.empty(T, E, device=dev))
    dt = torch.nn.functional.softplus(low[:, :rank].double() @ w_dt.double().T + b_dt.double())
    for i, s in enumerate(slots.tolist()):
        a, b = int(starts[i]), int(starts[i + 1])
        S = first[s].double()
        want = torch.empty(b - a, E, dtype=F)
        for t in range(a, b):
            S = torch.exp(dt[t].unsqueeze(1) * A.double()) * S + (dt[t] * x[t].double()).unsqueeze(1) * low[t, rank: rank + states].double()
            want[t - a] = (S @ low[t, rank + states:].double() + skip.double() * x[t].double()) * plain.silu(z[t].double())
        assert (out[a:b].double().cpu() - want).abs().max() <= 2e-5 * want.abs().max()
        assert (state[s].double().cpu() - S).abs().max() <= 2e-5 * S.abs().max()
    assert torch.equal(state[0].cpu(), first[0])


@pytest.mark.parametrize("dk,dv,rank,form,act,w2_type", [(128, 128, 16, 0, 0, torch.bfloat16), (64, 160, 5, 1, 1, torch.float32), (4, 12, 3, 0, 0, torch.float32),
                                                         (100, 36, 24, 0, 1, torch.bfloat16), (68, 64, 1, 1, 0, torch.float32)])
def test_projected_decay_recurrence_as_products_within_pieces(K, dk, dv, rank, form, act, w2_type):
    """Portions that end at the edges of quarters and halves of a piece, beside one that runs in one go, from states that are not
    zero; the same rows laid so that vectors of four do not fit walk the pieces row by row.  Float32 sums of at most dk + 64 terms
    whose decays are below 1: rounding of 2^-24 a step."""
    from infinicore_infer_b200.parts import LinearAttention
    dev, g, H = torch.device("cuda:0"), torch.Generator().manual_seed(dk + dv), 2
    lens = [65, 80, 3, 97, 160, 127]
    T, n = sum(lens), len(lens)
    u = torch.randn(T, 2 * H * dk + H * dv + rank, generator=g)
    w2 = (torch.randn(H * dk, rank, generator=g) * 0.7).to(w2_type)
    b2 = torch.randn(H * dk, generator=g) - (2.0 if form else -2.0)
    first = torch.randn(n + 1, H, dk, dv, generator=g)
    starts, slots = torch.tensor([0] + lens).cumsum(0).to(torch.int32), torch.arange(n, 0, -1, dtype=torch.int32)
    caps = LinearAttention.step_list_capacity(T, n)
    arrays = {name: np.zeros(max(1, c), dtype=np.int32) for name, c in caps.items()}
    counts = LinearAttention.fill_step_lists(n, n, lens, [0] * n, arrays)
    lists = {name: torch.from_numpy(arrays[name][:max(1, counts[name][0] * w)]).to(dev) for name, w in (("direct", 1), ("pieces", 2), ("piece_reqs", 3))}
    got = []
    for shift in (0, 1):        # 1: offsets that are no multiples of four
        rows = torch.cat([torch.zeros(T, shift), u, torch.zeros(T, -(u.shape[1] + shift) % 4)], 1).contiguous().to(dev)
        state, out = first.clone().to(dev), torch.empty(T, H * dv, device=dev)
        K.linear_scan(rows, (shift, shift + H * dk, shift + 2 * H * dk), H, dk, dv, act, 0.5, None, w2.to(dev), b2.to(dev), shift + 2 * H * dk + H * dv,
                      6.0, state, starts.to(dev), slots.to(dev), out, decay_form=form, **lists)
        got.append((out.double().cpu(), state.double().cpu()))
    f = plain.silu if act else (lambda x: x)
    U = u.double()
    q, k = f(U[:, :H * dk]).view(T, H, dk) * 0.5, f(U[:, H * dk: 2 * H * dk]).view(T, H, dk)
    v = f(U[:, 2 * H * dk: 2 * H * dk + H * dv]).view(T, H, dv)
    z = (U[:, 2 * H * dk + H * dv:] @ w2.double().T + b2.double()).view(T, H, dk)
    a = torch.exp(-torch.exp(z)) if form else torch.exp(torch.nn.functional.logsigmoid(z) / 6.0)
    for i, s in enumerate(slots.tolist()):
        S, want = first[s].double(), []
        for t in range(int(starts[i]), int(starts[i + 1])):
            S = a[t].unsqueeze(-1) * S + k[t].unsqueeze(-1) * v[t].unsqueeze(1)
            want.append(torch.einsum("hkv,hk->hv", S, q[t]).reshape(-1))
        want = torch.stack(want)
        for out, state in got:
            assert (out[int(starts[i]): int(starts[i + 1])] - want).abs().max() <= 2e-5 * want.abs().max(), f"request {i}"
            assert (state[s] - S).abs().max() <= 2e-5 * S.abs().max(), f"state of request {i}"
    assert torch.equal(got[0][1][0], first[0].double()) and not torch.equal(got[0][0], got[1][0])


@pytest.mark.parametrize("taps,C,lens", [(4, 8196, [128]), (3, 7044, [7, 1, 2, 1, 140]), (2, 8192, [1, 129]), (4, 7304, [9, 3, 1, 1, 130]), (4, 8196, [1] * 257)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_causal_convolution_of_many_rows(K, taps, C, lens, dtype):
    """Requests shorter than the taps, of one row and across the blocks' eight rows; the same rows laid so that vectors of four do not
    fit take a thread an element.  Both add the taps in the same order: the same bits."""
    dev, g, T, n = torch.device("cuda:0"), torch.Generator().manual_seed(C), sum(lens), len(lens)
    assert conv_walks_rows(T, n, C)
    u, w, b, ib = (torch.randn(*s, generator=g) for s in ((T, C), (C, taps), (C,), (C,)))
    tail = torch.randn(n + 1, taps - 1, C, generator=g)
    starts, slots = torch.tensor([0] + lens).cumsum(0).to(torch.int32), torch.arange(n, 0, -1, dtype=torch.int32)
    row_req = torch.repeat_interleave(torch.arange(n, dtype=torch.int32), torch.tensor(lens))
    got = []
    for shift in (0, 1):
        rows = torch.cat([torch.zeros(T, shift), u, torch.zeros(T, 4 - shift)], 1).contiguous().to(dev)
        state, y32, yT = tail.clone().to(dev), torch.empty(T, C, device=dev), torch.empty(T, C, dtype=dtype, device=dev)
        K.causal_conv(rows, shift, C, w.to(dev), b.to(dev), K.ACT_SILU, state, row_req.to(dev), starts.to(dev), slots.to(dev), y32, yT, in_bias=ib.to(dev))
        got.append((y32.cpu(), yT.cpu(), state.cpu()))
    assert all(torch.equal(x, y) for x, y in zip(*got))
    for r, s in enumerate(slots.tolist()):
        a, e = int(starts[r]), int(starts[r + 1])
        x = torch.cat([tail[s].double(), u[a:e].double() + ib.double()])
        want = plain.silu(b.double() + sum(w[:, j].double() * x[j: j + e - a] for j in range(taps)))
        assert (got[0][0][a:e].double() - want).abs().max() <= 2.0 ** -20 * want.abs().max()
        assert (got[0][2][s].double() - x[-(taps - 1):]).abs().max() <= 2.0 ** -22 * x.abs().max()
