"""The rules that choose between two forms of a kernel, at sizes where both were timed: a rule that sends a call to the slower form
fails here.  Host code only."""
import pytest

from infinicore_infer_b200.kernels import host


@pytest.mark.parametrize("heads,requests,window,keys", [
    # (rows, position of the first) of every request; microseconds on a B200 with tiles of 128 and of 64 keys
    (8, [(128, 4000)], 0, 128),                 # 72, 87
    (32, [(128, 4000)], 0, 128),                # 72, 88
    (64, [(128, 4000)], 0, 128),                # 73, 88
    (8, [(1000, 7000)], 0, 128),                # 125, 158
    (16, [(1024, 4000)], 0, 128),               # 87, 106
    (16, [(2048, 0)], 0, 128),                  # 45, 52
    (32, [(512, 0)], 0, 128),                   # 18, 20
    (32, [(1024, 0)], 0, 128),                  # 32, 34
    (32, [(1000, 0), (64, 3000)], 0, 128),      # 56, 72
    (32, [(1000, 0), (200, 0), (1, 3000)], 0, 64),      # the short request's row is no tile; 39, 34
    (16, [(2048, 4000)], 0, 64),                # 164, 138
    (16, [(2048, 0)], 1024, 64),                # 43, 37
    (16, [(1536, 0)], 512, 64),                 # 30, 26
    (32, [(768, 1000)], 0, 64),                 # 54, 50
    (32, [(1536, 0)], 0, 64),                   # 55, 48
    (32, [(100, 2000)] * 6, 0, 64),             # 81, 60
    (32, [(60, 0)] * 10, 0, 64),                # 28, 19
    (32, [(833, 0), (1667, 0), (2503, 0)], 0, 64)])     # 207, 152
def test_keys_a_tile_of_the_prefill_attention(heads, requests, window, keys):
    start = [0]
    for n, _ in requests:
        start.append(start[-1] + n)
    assert host.attention_tile_keys(heads, start, [p for _, p in requests], window) == keys


@pytest.mark.parametrize("rows,requests,channels,walks", [
    # microseconds, two and four taps: an element a thread, eight rows a thread
    (128, 1, 64, False), (2048, 1, 64, False),          # 9 and 11, 13
    (128, 128, 64, False), (256, 256, 512, False),      # 8, 16 and 17
    (512, 1, 512, False), (640, 16, 512, False),        # 11 and 13, 13; 13, 13 and 15
    (256, 1, 2048, False), (128, 128, 4096, False), (256, 256, 4096, False),    # 13 and 15, 15; 12 and 15, 16 and 19; 18 and 21, 19 and 23
    (2048, 1, 512, True), (512, 1, 2048, True),         # 17 and 20, 15 both
    (640, 16, 2048, True), (256, 1, 4096, True),        # 20 and 24, 15 and 17; 17 and 20, 15
    (256, 256, 8192, True), (2048, 1, 4096, True)])     # 27 and 36, 21 and 26; 75 and 95, 36 and 42
def test_rows_a_thread_of_the_causal_convolution(rows, requests, channels, walks):
    assert host.conv_walks_rows(rows, requests, channels) == walks


@pytest.mark.parametrize("elem,heads,kv_heads,size,requests,rows,context,walks", [
    # (rows of each request, bound on the histories); microseconds by warps and by blocks
    (2, 4, 4, 16, 512, 1, 256, True), (2, 4, 4, 16, 1, 1, 1001, False), (2, 7, 7, 30, 512, 1, 256, True), (2, 7, 7, 30, 1, 300, 300, True),     # 18, 70; 96, 70; 38, 194; 40, 66
    (2, 7, 7, 30, 1, 2048, 2048, False), (2, 4, 1, 32, 1024, 1, 512, False),        # 744, 567; 216, 116
    (2, 8, 8, 96, 512, 1, 256, True), (2, 36, 36, 64, 64, 1, 512, False), (2, 16, 16, 256, 64, 1, 512, True), (2, 1, 1, 512, 1, 500, 500, False),     # 284, 310; -; 585, 676; 699, 406
    (4, 4, 4, 16, 512, 1, 256, True), (4, 16, 16, 256, 512, 1, 256, True), (4, 36, 36, 64, 512, 1, 256, False),      # 37, 61; 1,134, 1,603; 713, 556
    (4, 36, 36, 64, 1, 17, 17, True), (4, 24, 8, 64, 1, 17, 17, False), (4, 16, 16, 256, 1, 17, 17, True),        # 9, 12; 8, 7; 18, 26
    (4, 24, 8, 64, 1, 301, 301, False), (4, 24, 8, 64, 8, 1, 4096, False), (4, 36, 36, 128, 64, 4, 4, True), (4, 4, 4, 16, 8, 1, 0, False)])     # -; -; 27, 78; not known
def test_kernel_of_the_float32_row_attention(elem, heads, kv_heads, size, requests, rows, context, walks):
    assert host.attention_rows_walk(rows * requests, requests, context, heads, kv_heads, size, elem) == walks


@pytest.mark.parametrize("lens,channels,states,cuts", [
    # microseconds end to end and over pieces
    ([512], 4096, 16, False), ([768], 4096, 16, True), ([2048], 4096, 16, True),        # 148 twice; 589, 360
    ([768] * 8, 64, 16, False), ([768] * 2, 512, 16, False), ([1000], 512, 16, True), ([1024] * 4, 64, 16, True),      # 104, 113; 127, 133; 149, 111; 132, 113
    ([896], 130, 5, True), ([1921, 1, 769], 130, 16, True), ([895], 130, 16, False), ([2500, 65], 130, 20, True),
    ([768], 512, 32, False), ([1024] * 4, 512, 32, False), ([2048], 512, 32, True), ([2048] * 4, 512, 32, True),     # 135, 178; 279, 302; 548, 276; 647, 374
    ([2048] * 2, 4096, 32, True), ([2048] * 4, 4096, 32, False), ([4096], 64, 33, False)])      # 989, 768; 1,161, 1,357; more states than a thread keeps
def test_pieces_of_the_selective_scan(lens, channels, states, cuts):
    assert host.selective_scan_cuts(sum(lens), len(lens), channels, states) == cuts


@pytest.mark.parametrize("rows,experts,top,width,ff,tiles", [
    # microseconds of a layer in tiles of 64 entries and of 128
    (65, 1, 1, 64, 64, False), (512, 4, 2, 64, 64, False), (64, 32, 2, 64, 64, False),      # 26, 31; 30, 37; 30, 33
    (33, 2, 2, 256, 64, False), (512, 4, 2, 256, 256, False), (2048, 8, 2, 256, 64, False),     # 30, 33; 36, 49; 42, 47
    (512, 4, 2, 128, 512, False), (64, 4, 2, 512, 128, False), (65, 1, 1, 512, 512, False),     # 38, 43; 34, 39; 38, 41
    (512, 4, 2, 512, 512, False),           # 48, 49 to 52
    (128, 128, 1, 2048, 1408, False),       # one entry an expert: not measured
    (2048, 8, 2, 512, 512, True), (64, 32, 2, 512, 512, True), (64, 16, 2, 512, 512, True),     # 87, 61; 60, 49; 48, 43
    (2048, 8, 2, 128, 512, True), (64, 64, 2, 512, 128, True),      # 59, 49; 54, 46
    (65, 1, 1, 1024, 256, True), (33, 2, 2, 1024, 1024, True), (64, 4, 2, 2048, 512, True),     # 44, 43; 56, 47; 69, 54
    (48, 8, 2, 2048, 1408, True), (128, 64, 2, 2048, 1408, True)])      # 102, 72; 367, 223
def test_tiles_of_the_routed_experts(rows, experts, top, width, ff, tiles):
    assert host.experts_take_tiles(rows * top, experts, width, ff) == tiles


@pytest.mark.parametrize("dim,rot,rank,requests,window,heads", [
    # (rows, position of the first) of every request; microseconds over the latent rows and over heads made for the step
    (64, 0, 64, [(32, 0)], 0, False), (64, 0, 64, [(16, 0)] * 2, 0, False), (64, 0, 64, [(20, 100)] * 16, 0, False),    # 17, 24 twice; 26, 30
    (64, 0, 64, [(100, 100)] * 4, 64, False), (64, 64, 160, [(32, 0)], 0, False), (64, 64, 160, [(16, 0)] * 2, 0, False),   # 24, 28; 22, 24 twice
    (128, 64, 512, [(1, 500)] * 8, 0, False), (128, 64, 512, [(31, 0)], 0, False),
    (64, 0, 64, [(32, 500)], 0, True), (64, 0, 64, [(256, 0)], 0, True), (64, 64, 160, [(20, 100)] * 16, 0, True),      # 52, 28; 34, 24; 34, 30
    (64, 64, 160, [(100, 100)] * 4, 64, True), (128, 64, 512, [(16, 0)] * 2, 0, True), (128, 64, 512, [(2048, 0)], 0, True)])   # 30, 28; 36, 28; 887, 75
def test_way_of_a_latent_attention(dim, rot, rank, requests, window, heads):
    rows, keys = sum(n for n, _ in requests), sum(n + p for n, p in requests)
    assert host.latent_takes_heads(rows, len(requests), keys, window, dim, rot, dim, rank) == heads


@pytest.mark.parametrize("rows,n,k,tensor", [
    # microseconds: on the CUDA cores, on the tensor cores
    (16, 2560, 1536, True), (23, 7680, 1536, True),                 # 16, 13; 26, 21: below 256 rows K alone decides
    (24, 1536, 1536, True), (32, 11264, 2048, True),                # 20, 10; 52, 45
    (301, 7680, 1536, True), (301, 1536, 3840, True),               # 199, 45; 108, 33
    (64, 64, 2048, True), (2048, 512, 512, True),                   # 19, 9; 35, 14
    (32, 512, 512, True), (64, 512, 512, True), (64, 512, 508, False),      # 7, 7; 7, 7
    (301, 288, 96, False), (640, 1024, 256, False)])                # 3, 5; 15, 9: short sums stay
def test_float32_products_on_the_tensor_cores(rows, n, k, tensor):
    tile, cuts = host.f32_plan(rows, n, k)
    assert (tile != 0) == tensor
    # the blocks of clusters that run at once on 148 SMs, one a block: 33 of four, 14 of eight
    blocks = -(-rows // tile) * -(-n // 128) * cuts if tile else 0
    assert cuts in (1, 2, 4, 8) and (cuts == 1 or blocks <= {2: 148, 4: 132, 8: 112}[cuts])


@pytest.mark.parametrize("n,k,cuts", [(2560, 1536, 4), (1536, 1536, 8), (7680, 1536, 2), (1536, 3840, 8), (11520, 2304, 1), (4096, 16384, 4), (64, 2048, 8),
                                      (512, 512, 4), (73440, 1536, 1), (1, 512, 4), (300, 511, 0)])
def test_float32_products_of_few_rows_add_in_one_order(n, k, cuts):
    """Below 256 rows neither the way nor the cuts of K, which set the order of a row's sums, depend on the rows; the tile may."""
    plans = [host.f32_plan(rows, n, k) for rows in range(1, 256)]
    assert {c if t else 0 for t, c in plans} == {cuts}


@pytest.mark.parametrize("kind,k,dtype,library,needs", [("linear", 512, "float32", 0, True), ("residual", 511, "float32", 0, False), ("gate_up", 2048, "float32", 0, True),
                                                        ("norm_add", 2048, "float32", 0, False), ("linear", 2048, "float32", 1, False), ("linear", 2048, "bfloat16", 0, False)])
@pytest.mark.parametrize("rows", [1, 23, 4096])
def test_a_model_binds_the_split_float32_product_where_its_records_reach_it(kind, k, dtype, library, needs, rows):
    """By the records alone, as the product's way: an engine of small steps would else run it or not by what another engine has bound."""
    import torch

    from infinicore_infer_b200.kernels import dtype_code
    from infinicore_infer_b200.parts import program
    env = program.RunnerEnv(dtype=dtype_code(getattr(torch, dtype)), page_size=16, max_blocks=4)
    env.routing.sms, env.routing.library_only = 148, library
    ops = (program.RunnerOp * 1)(program.record(kind, "h", "act", n=256, k=k))
    assert program.modules_needed(env, ops, 1, rows)["gemm_f32_tcgen05"] == needs


@pytest.mark.parametrize("rows,short,tiles,page,takes", [(31, 0, 1, 16, False), (32, 0, 1, 16, True), (32, 1, 1, 16, False), (300, 0, 0, 16, False), (300, 0, 3, 24, False),
                                                         (300, 0, 3, 1, True), (300, 0, 3, 256, True)])
def test_float32_attention_in_tiles(rows, short, tiles, page, takes):
    assert host.attention_f32_takes(rows, short, tiles, page) == takes


@pytest.mark.parametrize("blocks,dh,tall", [(349, 64, False), (350, 64, True), (119, 128, False), (120, 128, True)])
def test_tiles_of_the_float32_attention(blocks, dh, tall):
    assert host.attention_f32_tall(blocks, dh) == tall


@pytest.mark.parametrize("rows,k,takes", [(64, 512, True), (65, 512, False), (1, 16, True), (1, 24, False), (16, 1040, True), (16, 1072, False)])
def test_heads_products_of_few_rows(rows, k, takes):
    """Whole steps of 16 columns, and two blocks an SM."""
    assert host.head_takes_rows(rows, k) == takes


@pytest.mark.parametrize("k,elem,blocks,groups", [(2048, 2, 10 ** 6, 1), (512, 2, 1183, 1), (512, 2, 1184, 2), (256, 2, 2368, 4), (256, 2, 2367, 2), (64, 4, 10 ** 6, 4), (512, 4, 10 ** 6, 1)])
def test_groups_of_an_experts_rows_a_block(k, elem, blocks, groups):
    """More than one only where that many rows of 16 are 2 KB at most and the grid stays at four blocks an SM."""
    assert host.expert_row_groups(k, elem, blocks) == groups


@pytest.mark.parametrize("code,words", [(1, "gemm_tcgen05: a bounded wait ran out (TMA"), (4, "linear_small: a row's sum of squares"), (14, "attention_tcgen05"),
                                        (23, "routed_experts of many rows"), (24, "routed_experts of few rows: a bounded wait ran out (copies"),
                                        (25, "head_linear of few rows: a bounded wait ran out (copies"), (33, "gemm_f32_tcgen05: a bounded wait ran out (weights and sums"),
                                        (99, "status code 99")])
def test_a_status_word_names_its_kernel(monkeypatch, code, words):
    """The word as a kernel leaves it: the check raises with the kernel's own name, and clears it."""
    import torch

    from infinicore_infer_b200 import kernels
    word = torch.tensor([code], dtype=torch.int32)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    monkeypatch.setattr(kernels._build, "_loaded", {})
    monkeypatch.setitem(kernels._tg_status, "a device", word)
    with pytest.raises(kernels.KernelError) as e:
        kernels.check_gemm_status("a device")
    assert words in str(e.value) and int(word) == 0
    kernels.check_gemm_status("a device")


def test_sampling_parameters_beyond_their_types_are_clamped(monkeypatch):
    """A top-k beyond 32 bits or infinite reaches the draw as the largest whole number."""
    import torch

    from infinicore_infer_b200 import kernels
    from infinicore_infer_b200.sampling.sampler import Sampler, SamplingParams
    seen = []
    monkeypatch.setattr(kernels, "sample", lambda logits, t, k, p, u, out: (seen.append(k.tolist()), out.zero_()))
    params = [SamplingParams(temperature=1.0, topk=k, topp=0.5) for k in (7, 2 ** 40, float("inf"), -2 ** 40)]
    Sampler("cpu").sample(torch.zeros(4, 8), params, range(4))
    assert seen == [[7, 2 ** 31 - 1, 2 ** 31 - 1, 1 - 2 ** 31]]


@pytest.mark.filterwarnings("error")
def test_sampling_parameters_beyond_float32_are_infinite(monkeypatch):
    import torch

    from infinicore_infer_b200 import kernels
    from infinicore_infer_b200.sampling.sampler import Sampler, SamplingParams
    seen = []
    monkeypatch.setattr(kernels, "sample", lambda logits, t, k, p, u, out: (seen.append(t.tolist()), out.zero_()))
    Sampler("cpu").sample(torch.zeros(2, 8), [SamplingParams(temperature=t, topk=5, topp=0.5) for t in (1e300, 0.5)], range(2))
    assert seen == [[float("inf"), 0.5]]
