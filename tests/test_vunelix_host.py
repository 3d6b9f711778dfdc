"""Vunelix without a GPU: the configuration, the run order of a looped span, the manifest, the rotation's frequencies."""
import ctypes
import math

import pytest
import torch

import plain_vunelix as plain
from infinicore_infer_b200.config import ConfigError, FrequencyRampSpec, PairRotarySpec, VunelixConfig, config_class_for
from infinicore_infer_b200.kernels import _build
from infinicore_infer_b200.parts import cache_needs, model_manifest, state_needs


def cfg(loop=None, cap=7.5):
    layers = [
        {"type": "mamba1", "mixer": {"inner": 24, "state": 6, "dt_rank": 2, "conv": 3}, "mlp": {"kind": "dense", "ff": 20}},
        {"type": "latent_attention", "mlp": {"kind": "moe", "router": {"experts": 3, "top": 2}, "expert": {"ff": 8}, "shared": {"ff": 12}},
         "mixer": {"heads": 2, "dim": 6, "rot_dim": 4, "vdim": 10, "kv_rank": 14, "scale": 0.3,
                   "rot": {"base": 100.0, "dims": 4, "scaling": {"factor": 2.0, "original": 16, "fast": 4.0, "slow": 1.0}}}},
        {"type": "latent_attention", "mlp": None,
         "mixer": {"heads": 1, "dim": 4, "rot_dim": 6, "vdim": 4, "kv_rank": 5, "scale": 0.5, "rot": {"base": 50.0, "dims": 2}}},
    ]
    out = {"architecture": "Vunelix", "norm": {"eps": 1e-5}, "vocab": 40, "width": 16, "layers": layers, "logit_softcap": cap}
    if loop:
        out["loop"] = dict(zip(("start", "stop", "times"), loop))
    return out


def test_the_registry_finds_the_configuration_and_it_reads_back():
    c = config_class_for(cfg())
    assert c is VunelixConfig
    typed = c.from_dict(cfg(loop=(1, 3, 2)), max_tokens=99)
    assert typed.max_positions == 99 and typed.loop == (1, 3, 2) and typed.logit_softcap == 7.5
    again = VunelixConfig.from_dict(typed.to_dict(), max_tokens=99)
    assert again == typed
    assert VunelixConfig.from_dict(cfg(cap=None)).logit_softcap == 0.0


def test_run_order_of_a_span_that_runs_several_times():
    spec = VunelixConfig.from_dict(cfg(loop=(1, 3, 2))).model_spec()
    assert [e.layer for e in spec.order] == [0, 1, 2, 1, 2]
    assert [e.cache for e in spec.order] == [0, 1, 2, 3, 4]
    assert [(e.before.step_index, e.before.steps) if e.before else None for e in spec.order] == [None, (0, 2), None, (1, 2), None]
    assert [(i, t, first) for i, t, first in plain.run_order(cfg(loop=(1, 3, 2)))] == \
        [(i, t, first) for i, t, first in VunelixConfig.from_dict(cfg(loop=(1, 3, 2))).run_order()]
    plain_order = VunelixConfig.from_dict(cfg()).model_spec().order
    assert [e.layer for e in plain_order] == [0, 1, 2] and all(e.before is None for e in plain_order)
    needs, tails = cache_needs(spec), state_needs(spec)
    assert needs[0].shape == (24, 6) and tails[0].shape == (2, 24)
    assert needs[1] == needs[3] and needs[1].head_dim == 18 and needs[1].v_head_dim == 14 and needs[1].values_in_keys
    assert needs[2].head_dim == 11 and tails[1] is None


def test_manifest_names_every_tensor_once():
    names = model_manifest(VunelixConfig.from_dict(cfg(loop=(0, 2, 3))).model_spec())
    assert names["loop.in"].shape == (16, 32) and names["loop.step"].shape == (3, 16)
    assert names["l0.mix.A_log"].shape == (24, 6) and names["l0.mix.x"].shape == (2 + 12, 24) and names["l0.mix.conv.b"].shape == (24,)
    assert names["l1.mix.dkv"].shape == (18, 16) and names["l1.mix.uk"].shape == (12, 14) and names["l1.mix.g"].shape == (20, 16)
    assert names["l1.mlp.e2.down"].shape == (16, 8) and names["l1.mlp.shared.up"].shape == (12, 16) and names["l1.mlp.router"].shape == (3, 16)
    assert "l2.norm2" not in names and "l2.norm1b" in names and names["head"].optional
    assert "loop.in" not in model_manifest(VunelixConfig.from_dict(cfg()).model_spec())


@pytest.mark.parametrize("dims,base,scaling", [(8, 1e4, None), (32, 5e5, (4.0, 256, 16.0, 2.0)), (6, 300.0, (16.0, 8, 2.0, 0.25))])
def test_stretched_frequencies(dims, base, scaling):
    spec = PairRotarySpec(dims=dims, base=base, scaling=None if scaling is None else FrequencyRampSpec(*scaling))
    f, m = spec.frequencies()
    names = None if scaling is None else dict(zip(("factor", "original", "fast", "slow"), scaling))
    pf, pm = plain.rotary_frequencies(dims, base, names)
    assert all(abs(a - b) <= 1e-12 * b for a, b in zip(f, pf.tolist())) and abs(m - pm) < 1e-12
    if scaling:
        assert abs(m - (0.1 * math.log(scaling[0]) + 1.0)) < 1e-12
        plainf = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
        assert all(p / scaling[0] - 1e-15 <= a <= p + 1e-15 for a, p in zip(f, plainf))


@pytest.mark.parametrize("change,what", [
    (lambda c: c["layers"][1]["mixer"]["rot"].update(dims=6), "rot.dims"),
    (lambda c: c["layers"][0].update(type="mamba2"), "type"),
    (lambda c: c["layers"][1]["mlp"]["router"].update(top=4), "experts"),
    (lambda c: c.update(loop={"start": 2, "stop": 5, "times": 2}), "loop"),
    (lambda c: c["layers"][0]["mixer"].pop("state"), "state"),
])
def test_what_the_configuration_refuses(change, what):
    c = cfg()
    change(c)
    with pytest.raises(ConfigError, match=what):
        VunelixConfig.from_dict(c)


def latent_program(heads=16, dim=128, rot=64, rank=512, window=0, num_pages=65, page_size=16, max_positions=640):
    """The record of a latent attention that may run over heads made for the step, and the environment of an engine that holds
    ``num_pages`` pages (the null page among them)."""
    from infinicore_infer_b200.kernels import dtype_code
    from infinicore_infer_b200.parts import program
    op = program.record("latent_attention", "q", "o", heads=heads, rank=rank, rot_width=rot, softmax_scale=0.1, window=window, num_pages=num_pages,
                        max_positions=max_positions, fold=2, head_dim=dim, v_head_dim=dim, in2_slot="o", out2_slot="act")
    env = program.RunnerEnv(dtype=dtype_code(torch.bfloat16), page_size=page_size, max_blocks=max_positions // page_size)
    env.routing.sms = 148
    return program, (program.RunnerOp * 1)(op), env


def slot_bytes(program, ops, env, rows):
    sizes = (ctypes.c_longlong * len(program.SLOTS))()
    assert _build.load("runner").jk_runner_slot_bytes(ctypes.byref(env), ops, len(ops), rows, rows, sizes) == 0
    return dict(zip(program.SLOTS, sizes))


def test_room_for_heads_is_bounded_by_the_positions_a_step_can_see():
    """16 heads of 128 + 64 over a latent of 512 take 2 (512 + 64 + 4,096) bytes a position."""
    per = 2 * (512 + 64 + 16 * 256)
    for rows, pages, window, max_positions, positions in ((2048, 65, 0, 640, 64 * 16),             # the cache holds fewer positions
                                                         (2048, 100000, 0, 100000, 4 * 2048),      # four times the step's rows
                                                         (2048, 65, 100, 100000, 4 * 2048),        # a window: pages come and go
                                                         (64, 100000, 0, 48, 4 * 48),              # four requests at most, of 48 positions
                                                         (40, 65, 0, 112, 112 + 48)):              # two requests would not meet the rule with more
        program, ops, env = latent_program(num_pages=pages, window=window, max_positions=max_positions)
        got = slot_bytes(program, ops, env, rows)["heads"]
        assert got <= per * positions + 4096 + 12 * (rows // 128 + rows // 16), (rows, pages, window, got)
        assert got >= per * min(positions, 2 * max_positions if rows == 40 else positions) - per * 48, (rows, pages, window, got)


@pytest.mark.parametrize("switch", ["", "legacy_tensor_cores", "library_only"])
@pytest.mark.parametrize("rows", [1, 31, 32, 63, 64, 4096])
def test_an_engine_has_room_for_heads_exactly_where_it_binds_the_kernels(rows, switch):
    """The table of entry points is shared by all engines of a process: an engine that keeps room without binding both modules would go
    over heads or not by what another engine has bound."""
    program, ops, env = latent_program()
    if switch:
        setattr(env if switch in dict(env._fields_) else env.routing, switch, 1)
    needed = program.modules_needed(env, ops, len(ops), rows)
    room = slot_bytes(program, ops, env, rows)["heads"] > 0
    assert needed["attention_tcgen05"] == needed["gemm_tcgen05"] == room == (rows >= 32 and not switch)
    assert needed["blocks"] and not needed["mixers"]


@pytest.mark.parametrize("left", [0, -1])
def test_an_engine_leaves_the_room_for_heads_out_where_memory_is_short(monkeypatch, left):
    """The buffer is optional: it is made where enough stays free after it, and is else too small for any step."""
    module, ops, env = latent_program()
    sizes = slot_bytes(module, ops, env, 64)
    monkeypatch.setattr(module, "free_bytes", lambda device: module.LEAVE_FREE + sizes["heads"] + left)
    slots = module.allocate_slots(list(sizes.values()), torch.device("cpu"))
    assert [t.numel() for t in slots] == [16 if n == "heads" and left < 0 else max(16, b) for n, b in sizes.items()]


@pytest.mark.parametrize("dtype,dim,twice", [(torch.float32, 64, False), (torch.bfloat16, 48, False), (torch.bfloat16, 64, True)])
def test_the_key_map_is_kept_as_stored_only_where_heads_can_be_made_from_it(dtype, dim, twice):
    """Beside its transpose; elsewhere (float32, sizes outside the rule) the layer holds one copy of each map and no more."""
    from infinicore_infer_b200.parts import LatentAttention
    from infinicore_infer_b200.parts.base import Runtime
    layer = dict(type="latent_attention", mlp=None, mixer=dict(heads=2, dim=dim, rot_dim=64, vdim=dim, kv_rank=72, scale=0.1, rot=dict(base=1e3, dims=32)))
    c = dict(architecture="Vunelix", norm=dict(eps=1e-5), vocab=40, width=16, logit_softcap=None, layers=[layer])
    spec = VunelixConfig.from_dict(c).model_spec()
    names = model_manifest(spec)

    class Weights:
        def get(self, name, role):
            return torch.zeros(names[name].shape, dtype=dtype)

        def get_rows(self, wanted, role):
            return torch.cat([self.get(n, role) for n in wanted])

    part = LatentAttention(spec.layers[0].mixer, Weights(), "l0.mix.", Runtime(dtype, "cpu"))
    held = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes() for t in (part.w_heads, part.w_q_latent, part.w_v) if t is not None}
    one = 2 * dim * 72 * dtype.itemsize
    assert sum(held.values()) == (3 if twice else 2) * one
