"""Latent attention of long prompt portions, whose keys and values are formed: the kernels against float64, and steps in which
such portions stand beside decoded tokens and short portions that attend over the latents."""

import pytest
import torch

import helpers as H
import zupilorn_cases as Z

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("sink", [False, True], ids=["", "sink"])
@pytest.mark.parametrize("dim,rot,rank", [(128, 64, 128), (128, 16, 64), (64, 32, 64)], ids=str)
@pytest.mark.parametrize("lengths", [((0, 1), (0, 97)), ((95, 128), (1, 129), (0, 33)), ((300, 200),)], ids=str)
def test_formed_keys_and_values(dim, rot, rank, lengths, sink):
    """Requests of (cached, new) tokens around the tiles' edges over shuffled pages, pages of others filled with NaN. Against
    float64 over the same formed keys and values, the probabilities and the result are rounded to bfloat16 (8 bits: 2^-8 each at
    most) and the scores' sums and exponentials are float32: within 2^-7 (1 + 1/8) of the weighted sum of the values' sizes."""
    from llm_pipeline_b200.ops import kernels
    heads, page, gen = 3, 16, torch.Generator().manual_seed(dim + rot + len(lengths))
    R, dk = len(lengths), rank + rot
    ctx = [s + n for s, n in lengths]
    N = sum(n for _s, n in lengths)
    need = [-(-c // page) for c in ctx]
    order = torch.randperm(sum(need) + 3, generator=gen).tolist()
    pages = torch.full((sum(need) + 3, page, dk), float("nan"))
    tables = torch.full((R, max(need)), -1, dtype=torch.int32)
    latents = [torch.randn(c, dk, generator=gen).to(torch.bfloat16).float() for c in ctx]
    for r, c in enumerate(ctx):
        for i in range(need[r]):
            tables[r, i] = order.pop()
            part = latents[r][i * page:(i + 1) * page]
            pages[tables[r, i], :part.shape[0]] = part
    q = torch.randn(N, heads, dim + rot, generator=gen).to(torch.bfloat16)
    w = (torch.randn(heads * 2 * dim, rank, generator=gen) * rank ** -0.5).to(torch.bfloat16)
    sinks = torch.randn(heads, generator=gen) if sink else None
    keys = kernels.latent_prompt_keys(dim, rot, dim, rank)
    blocks = [(r, t) for r in range(R) for t in range(0, ctx[r], keys)]
    base = [next(i for i, b in enumerate(blocks) if b[0] == r) * keys for r in range(R)]
    rows = torch.empty(len(blocks) * keys, dk, dtype=torch.bfloat16, device=DEV)
    ctx_len = _i32(ctx)
    kernels.latent_gather(pages.to(DEV, torch.bfloat16), tables.to(DEV), ctx_len, _i32([r for r, _t in blocks]), _i32([t for _r, t in blocks]), keys, rows)
    for r in range(R):
        padded = rows[base[r]:base[r] + -(-ctx[r] // keys) * keys].float().cpu()
        assert torch.equal(padded[:ctx[r]], latents[r]) and (padded[ctx[r]:] == 0).all()
    kv = (rows[:, :rank].float() @ w.to(DEV).float().T).to(torch.bfloat16)
    out = torch.full((N, heads, dim), 7.0, dtype=torch.bfloat16, device=DEV)
    tiles = [(r, t) for r, (_s, n) in enumerate(lengths) for t in range(0, n, kernels.LATENT_PROMPT_TOKENS)]
    starts = [0]
    for _s, n in lengths:
        starts.append(starts[-1] + n)
    scale = (dim + rot) ** -0.5 * 3.0
    kernels.latent_prompt_attention(q.to(DEV), kv, rows, _i32(starts), ctx_len, _i32([r for r, _t in tiles]), _i32([t for _r, t in tiles]),
                                    _i32([base[r] for r, _t in tiles]), out, dim, rank, scale, sink=sinks.to(DEV) if sink else None)
    torch.cuda.synchronize()
    kernels.check_error_flag()
    kv, got = kv.double().cpu(), out.double().cpu()
    for r, (s, n) in enumerate(lengths):
        mine = kv[base[r]:base[r] + ctx[r]].view(ctx[r], 2 * heads, dim)
        k, v = mine[:, :heads], mine[:, heads:]
        qr = q[starts[r]:starts[r + 1]].double()
        score = (torch.einsum("nhd,thd->hnt", qr[..., :dim], k) + torch.einsum("nhd,td->hnt", qr[..., dim:], latents[r][:, rank:].double())) * scale
        score = score.masked_fill(torch.arange(ctx[r]) > s + torch.arange(n)[:, None], float("-inf"))
        if sink:
            score = torch.cat([score, sinks.double()[:, None, None].expand(heads, n, 1)], dim=2)
        p = torch.softmax(score, dim=2)[:, :, :ctx[r]]
        want, sizes = torch.einsum("hnt,thd->nhd", p, v), torch.einsum("hnt,thd->nhd", p, v.abs())
        assert ((got[starts[r]:starts[r + 1]] - want).abs() <= 1.125 * 2.0 ** -7 * sizes).all(), r


def test_formed_portions_beside_decoded_tokens_and_short_portions(tmp_path, monkeypatch):
    """Whole models in bfloat16 with portions of 40 tokens and more formed, cut and mixed so that steps hold both kinds (and ones
    that join), over contexts of several key segments; and a bound on the formed rows' memory that sends every request to the latents."""
    from llm_pipeline_b200.ops import kernels
    from llm_pipeline_b200.parts.latent_attention import LatentAttention
    for name, value in (("FORMED_MIN_TOKENS", 40), ("FORMED_JOIN_KEYS", 30), ("FORMED_MIN_GAIN_US", 0.0)):
        monkeypatch.setattr(LatentAttention, name, value)
    cfg = Z.config([Z.latent_layer(3, 64, 32, 64, 128, None), Z.latent_layer(3, 64, 32, 64, 128, None)], width=96, vocab=61)
    W = Z.weights_for(cfg, 21)
    folder = Z.write_model(str(tmp_path), cfg, W)
    seg = kernels.LATENT_SEGMENT_KEYS
    requests = {f"r{i}": H.random_tokens(61, n, 40 + i) for i, n in enumerate([2 * seg + 60, 130, 2 * seg + 90, 3])}
    want = Z.oracle(cfg, W, requests)
    runner = H.make_runner(folder, torch.bfloat16, page_size=16, num_pages=100, max_request_tokens=3 * seg, max_requests=4)
    calls = {"formed": 0, "both": 0}
    formed, attend = kernels.latent_prompt_attention, kernels.latent_attention_mma

    def counting(*args, **kwargs):
        calls["formed"] += 1
        return formed(*args, **kwargs)

    def beside(*args, **kwargs):
        calls["both"] += kwargs.get("rows") is not None
        return attend(*args, **kwargs)

    monkeypatch.setattr(kernels, "latent_prompt_attention", counting)
    monkeypatch.setattr(kernels, "latent_attention_mma", beside)
    Z.assert_matches(H.replay(runner, H.cut_whole(requests)), want, torch.bfloat16, "whole")
    Z.assert_matches(H.replay(runner, H.cut_portions(requests, (39, 70, 3, 128, 129, 41))), want, torch.bfloat16, "portions")
    Z.assert_matches(H.replay(runner, H.cut_mixed(requests, (60, 2, 131, 90, 7), max_live=4, decode_tail=30)), want, torch.bfloat16, "mixed")
    assert calls["formed"] and calls["both"]
    monkeypatch.setattr(LatentAttention, "FORMED_MAX_BYTES", 1)
    calls["formed"] = 0
    Z.assert_matches(H.replay(runner, H.cut_whole(requests)), want, torch.bfloat16, "nothing formed")
    assert calls["formed"] == 0


def _mixer(heads, rank, seed=1):
    from llm_pipeline_b200.parts import lookup
    part = lookup("mixer", "latent_attention")("p", hidden_size=64, num_heads=heads, dim=64, rot_dim=32, vdim=64, kv_rank=rank,
                                               scale=96 ** -0.5, norm_eps=1e-5)
    gen = torch.Generator().manual_seed(seed)
    weights = {name: torch.randn(spec.shape, generator=gen).to(DEV, torch.bfloat16) for name, spec in part.param_specs().items()}
    part.load(lambda name, role: weights[name])
    return part, weights


def test_the_maps_of_the_values_are_held_once():
    part, weights = _mixer(4, 128)
    assert part.formed_keys
    assert torch.equal(part.w_ukv, torch.cat([weights["p.uk"], weights["p.uv"]]))
    assert torch.equal(part.w_uv, weights["p.uv"].view(4, 64, 128)) and part.w_uv.is_contiguous()
    assert part.w_uv.untyped_storage().data_ptr() == part.w_ukv.untyped_storage().data_ptr()


def test_layers_of_other_sizes_choose_for_themselves():
    """A portion worth a second path beside a long context in a layer of large latents and not in one of small: each layer of a step
    chooses by its own sizes, whichever comes first."""
    from llm_pipeline_b200.engine.context import StepContext
    large, small = _mixer(16, 1024)[0], _mixer(16, 128)[0]

    def context():
        ctx = StepContext(torch.device(DEV), torch.bfloat16)
        ctx.q_lens, ctx.starts, ctx.max_q_len = [1100, 100], [0, 5000], 1100
        return ctx

    alone = [part._formed_plan(context()) is not None for part in (large, small)]
    assert alone == [True, False]
    for order in ((large, small), (small, large)):
        ctx = context()
        assert [part._formed_plan(ctx) is not None for part in order] == [part is large for part in order]


@pytest.mark.parametrize("sink", [False, True], ids=["", "sink"])
@pytest.mark.parametrize("heads,rank,rot", [(16, 512, 64), (3, 128, 16), (17, 256, 32), (33, 384, 64)], ids=str)
@pytest.mark.parametrize("ctx", [(1, 127, 128, 129), (64, 65, 4096), (777,)], ids=str)
def test_single_tokens(ctx, heads, rank, rot, sink):
    """Contexts around the edges of 128 keys and their halves beside long ones (ranges that end before others begin), heads of one
    tile and more, in one step, for a bound above every context too. Against float64 over the same rows, the probabilities and the
    result are rounded to bfloat16 (8 bits: 2^-8 each at most) and the scores' sums and exponentials are float32: within
    2^-7 (1 + 1/8) of the weighted sum of the values' sizes. Pages of others and rows past a context are NaN."""
    from llm_pipeline_b200.ops import kernels
    page, gen = 16, torch.Generator().manual_seed(sum(ctx) + heads + rank)
    assert kernels.latent_decode_supports(rank, rot, page)
    need = [-(-c // page) for c in ctx]
    order = torch.randperm(sum(need) + 3, generator=gen).tolist()
    pages = torch.full((sum(need) + 3, page, rank + rot), float("nan"))
    tables = torch.full((len(ctx), max(need)), -1, dtype=torch.int32)
    rows = [torch.randn(c, rank + rot, generator=gen).to(torch.bfloat16).float() for c in ctx]
    for r in range(len(ctx)):
        for i in range(need[r]):
            tables[r, i] = order.pop()
            part = rows[r][i * page:(i + 1) * page]
            pages[tables[r, i], :part.shape[0]] = part
    q = torch.randn(len(ctx), heads, rank + rot, generator=gen).to(torch.bfloat16)
    sinks = torch.randn(heads, generator=gen) if sink else None
    on = q.to(DEV)
    scale = (rank + rot) ** -0.5 * 3.0
    for longest in (max(ctx), max(ctx) + 1000):
        out = torch.full((len(ctx), heads, rank), 7.0, dtype=torch.bfloat16, device=DEV)
        kernels.latent_decode(on[..., :rank], on[..., rank:], pages.to(DEV, torch.bfloat16), tables.to(DEV), _i32(ctx), out, scale, longest,
                              sink=sinks.to(DEV) if sink else None)
        torch.cuda.synchronize()
        kernels.check_error_flag()
        for r in range(len(ctx)):
            score = (q[r].double() @ rows[r].double().T) * scale
            if sink:
                score = torch.cat([score, sinks.double()[:, None]], dim=1)
            p = torch.softmax(score, dim=1)[:, :ctx[r]]
            v = rows[r][:, :rank].double()
            assert ((out[r].double().cpu() - p @ v).abs() <= 2.0 ** -7 * (1 + 1 / 8) * (p @ v.abs())).all(), (r, longest)


@pytest.mark.parametrize("batch,rows,n,k", [(3, 1, 16, 8), (2, 8, 64, 128), (2, 9, 65, 136), (4, 16, 512, 256), (3, 7, 130, 264), (2, 16, 15, 512), (1, 3, 17, 1048)], ids=str)
def test_few_rows_of_several_heads(batch, rows, n, k):
    """The heads' maps of a decode step's rows around the tiles of 16 weight rows and 8 rows, runs of 32 of K and the split of a long K, on
    transposed views with other entries between; float64 within bfloat16's rounding of the result (half of the last of 7 stored bits: 2^-8) and float32 sums. A row has the bits
    that it has alone."""
    from llm_pipeline_b200.ops import kernels
    gen = torch.Generator().manual_seed(rows * n + k)
    x = torch.randn(rows, batch, k + 8, generator=gen).to(torch.bfloat16).to(DEV)
    w = torch.randn(batch, n, k, generator=gen).to(torch.bfloat16).to(DEV)
    out = torch.full((rows, batch, n + 3), 7.0, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_batched(x[:, :, :k].transpose(0, 1), w, out[:, :, :n].transpose(0, 1))
    want = torch.einsum("mbk,bnk->mbn", x[:, :, :k].double(), w.double())
    scale = torch.einsum("mbk,bnk->mbn", x[:, :, :k].double().abs(), w.double().abs())
    assert ((out[:, :, :n].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * scale).all()
    assert (out[:, :, n:] == 7.0).all()
    for m in {0, rows - 1}:
        alone = torch.empty(1, batch, n, dtype=torch.bfloat16, device=DEV)
        kernels.gemm_batched(x[m:m + 1, :, :k].transpose(0, 1), w, alone.transpose(0, 1))
        assert torch.equal(alone[0], out[m, :, :n])


@pytest.mark.parametrize("rows,n,k", [(16, 512, 128), (8, 64, 256), (8, 64, 1048), (1, 128, 512)], ids=str)
def test_few_rows_of_several_heads_hold_float32_sums(rows, n, k):
    """Entries of one sign, where every rounding of a sum shows: the result is the nearest bfloat16 but for sums within 4 x 2^-24 of their
    terms' sizes of the middle between two (float32 sums by a tree over 32 lanes reach 2.2, a chain of MMAs on one accumulator 5 to 7)."""
    from llm_pipeline_b200.ops import kernels
    for seed in range(60):
        gen = torch.Generator(device=DEV).manual_seed(seed)
        x = (torch.randn(16, rows, k, generator=gen, device=DEV) + 1).to(torch.bfloat16)
        w = ((torch.randn(16, n, k, generator=gen, device=DEV) + 1) * k ** -0.5).to(torch.bfloat16)
        out = torch.empty(16, rows, n, dtype=torch.bfloat16, device=DEV)
        kernels.gemm_batched(x, w, out)
        want = x.double() @ w.double().transpose(1, 2)
        least = (want.to(torch.bfloat16).double() - want).abs()
        sizes = x.double().abs() @ w.double().abs().transpose(1, 2)
        assert ((out.double() - want).abs() <= least + 4 * 2.0 ** -24 * sizes).all(), seed


@pytest.mark.parametrize("k", [128, 512])
def test_few_rows_of_several_heads_by_weights_just_made(k):
    """Weights that the kernel launched before writes, other ones every time: the product is of those, as after a pause. A layer's own
    weights, which may be read sooner, give the same bits."""
    from llm_pipeline_b200.ops import kernels
    gen = torch.Generator().manual_seed(k)
    x = torch.randn(4, 8, k, generator=gen).to(torch.bfloat16).to(DEV)
    made = [torch.randn(4 * 512, k, generator=gen).to(DEV) for _ in range(8)]
    w = torch.zeros(4, 512, k, dtype=torch.bfloat16, device=DEV)
    outs = torch.empty(8, 4, 8, 512, dtype=torch.bfloat16, device=DEV)
    for rows, out in zip(made, outs):
        kernels.convert_rows(rows, w.view(4 * 512, k))
        kernels.gemm_batched(x, w, out)
    for rows, out in zip(made, outs):
        paused, held = torch.empty_like(out), torch.empty_like(out)
        whole = rows.to(torch.bfloat16).view(4, 512, k)
        torch.cuda.synchronize()
        kernels.gemm_batched(x, whole, paused)
        torch.cuda.synchronize()
        kernels.gemm_batched(x, whole, held, held=True)
        assert torch.equal(out, paused) and torch.equal(held, paused)
