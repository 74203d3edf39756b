"""Paged decode attention, KV append and the serving engine on the GPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dh,splits", [(4, 128, 1), (4, 128, 5), (6, 64, 3), (16, 128, 0)])
def test_paged_decode_matches_reference(heads, dh, splits):
    from llm_systems_from_scratch_b200.ops import serving_ops, torch_impl
    d, page, n_pages, r = heads * dh, 16, 64, 5
    g = torch.Generator(device="cuda").manual_seed(0)
    kc = torch.randn(n_pages, page, d, device="cuda", generator=g).bfloat16()
    vc = torch.randn(n_pages, page, d, device="cuda", generator=g).bfloat16()
    qkv = torch.randn(r, 3 * d, device="cuda", generator=g).bfloat16()
    lens = torch.tensor([1, 16, 17, 100, 191], dtype=torch.int32, device="cuda")
    tables = torch.stack([torch.randperm(n_pages, device="cuda", generator=g)[:12] for _ in range(r)]).int()
    out = serving_ops.paged_decode_attention(qkv, kc, vc, tables, lens, heads, splits)
    ref = torch_impl.paged_decode_attention(qkv[:, :d].float(), kc.float(), vc.float(), tables.cpu(), lens.cpu(), heads)
    assert (out.float() - ref).abs().max().item() < 2e-2


def test_kv_append_writes_only_selected_slots():
    from llm_systems_from_scratch_b200.ops import serving_ops
    d = 512
    kc = torch.zeros(8, 16, d, device="cuda", dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    qkv = torch.randn(4, 3 * d, device="cuda").bfloat16()
    slots = torch.tensor([5, -1, 127, 16], device="cuda")
    serving_ops.kv_append(kc, vc, qkv, slots)
    kf, vf = kc.view(-1, d), vc.view(-1, d)
    for i, s in enumerate(slots.tolist()):
        if s >= 0:
            assert torch.equal(kf[s], qkv[i, d:2 * d]) and torch.equal(vf[s], qkv[i, 2 * d:])
    assert int((kf.abs().sum(-1) > 0).sum()) == 3


def test_paged_kernels_report_bad_tables_instead_of_reading_them():
    """A page id beyond the cache, a length beyond the table and a slot beyond the cache are skipped and recorded in
    the status word; good rows of the same launch are unaffected and the context stays usable."""
    from llm_systems_from_scratch_b200.ops import native, serving_ops, torch_impl
    heads, dh, page, n_pages, r = 4, 128, 16, 32, 3
    d = heads * dh
    g = torch.Generator(device="cuda").manual_seed(0)
    kc = torch.randn(n_pages, page, d, device="cuda", generator=g).bfloat16()
    vc = torch.randn(n_pages, page, d, device="cuda", generator=g).bfloat16()
    qkv = torch.randn(r, 3 * d, device="cuda", generator=g).bfloat16()
    tables = torch.stack([torch.randperm(n_pages, device="cuda", generator=g)[:4] for _ in range(r)]).int()
    good_lens = torch.tensor([10, 33, 64], dtype=torch.int32, device="cuda")
    ref = torch_impl.paged_decode_attention(qkv[:, :d].float(), kc.float(), vc.float(), tables.cpu(), good_lens.cpu(), heads)
    native.status_word().zero_()
    for bad_tables, bad_lens in ((tables.clone().index_put_((torch.tensor([1]), torch.tensor([0])), torch.tensor(n_pages + 7, dtype=torch.int32, device="cuda")), good_lens),
                                 (tables, torch.tensor([10, 33, 4 * page + 1], dtype=torch.int32, device="cuda"))):
        out = serving_ops.paged_decode_attention(qkv, kc, vc, bad_tables, bad_lens, heads, 2)
        torch.cuda.synchronize()
        with pytest.raises(native.KernelError):
            native.check_status()
        assert (out[0].float() - ref[0]).abs().max().item() < 2e-2       # the untouched row is still right
        assert torch.isfinite(out.float()).all()
    before = kc.clone()
    serving_ops.kv_append(kc, vc, qkv, torch.tensor([3, n_pages * page, -1], device="cuda"))
    torch.cuda.synchronize()
    with pytest.raises(native.KernelError):
        native.check_status()
    changed = (kc.view(-1, d) != before.view(-1, d)).any(-1).nonzero().flatten().tolist()
    assert changed == [3]
    native.check_status()                                                 # cleared; nothing pending


@pytest.mark.parametrize("graphs", [False, True])
def test_engine_matches_full_recompute_on_gpu(graphs):
    from llm_systems_from_scratch_b200.models.transformer import TransformerLM
    from llm_systems_from_scratch_b200.ops import native
    from llm_systems_from_scratch_b200.serving import ServingEngine
    torch.manual_seed(0)
    cfg = dict(vocab_size=503, context_length=256, d_model=256, num_layers=2, num_heads=4, d_ff=688, rope_theta=10000.0)
    model = TransformerLM(**cfg, use_custom_triton=True).cuda().eval()
    g = torch.Generator().manual_seed(1)
    prompts = [torch.randint(0, 503, (n,), generator=g).tolist() for n in (5, 130, 33, 64, 17)]
    eng = ServingEngine(model, page_size=16, max_batch=4, max_context=256, use_cuda_graphs=graphs)
    got = eng.generate(prompts, 12)
    native.check_status()
    # oracle: greedy decoding by re-running the same bf16 kernels on the whole context each time
    agree = total = 0
    for p, out in zip(prompts, got):
        ids = torch.tensor([p], device="cuda")
        for tok in out:
            logits = model(ids)[0, -1].float()
            top2 = logits.topk(2).values
            if (top2[0] - top2[1]).item() > 0.05:          # skip numerically tied positions
                total += 1
                agree += int(int(logits.argmax()) == tok)
            ids = torch.cat((ids, torch.tensor([[tok]], device="cuda")), dim=1)
    assert total > 20 and agree == total, (agree, total)
    assert eng.cache.allocator.free == eng.cache.num_pages


@pytest.mark.parametrize("graphs", [False, True])
def test_engine_with_programmatic_dependent_launch_gives_the_same_tokens(graphs):
    """The decode-path kernels launched as programmatic dependents (each starts while the kernel before it drains and
    waits for it before touching global memory) must produce exactly the tokens of ordinary launches, eagerly and in
    captured graphs, and leave the status word clean."""
    from llm_systems_from_scratch_b200.models.transformer import TransformerLM
    from llm_systems_from_scratch_b200.ops import native
    from llm_systems_from_scratch_b200.serving import ServingEngine
    torch.manual_seed(0)
    cfg = dict(vocab_size=503, context_length=256, d_model=256, num_layers=3, num_heads=4, d_ff=688, rope_theta=10000.0)
    model = TransformerLM(**cfg, use_custom_triton=True).cuda().eval()
    g = torch.Generator().manual_seed(2)
    prompts = [torch.randint(0, 503, (n,), generator=g).tolist() for n in (7, 120, 40, 64, 19, 90)]
    outs = {}
    prev = native.set_pdl(False)
    try:
        for pdl in (False, True):
            native.set_pdl(pdl)
            eng = ServingEngine(model, page_size=16, max_batch=4, max_context=256, use_cuda_graphs=graphs)
            outs[pdl] = eng.generate(prompts, 24)
            torch.cuda.synchronize()
            native.check_status()
            assert eng.cache.allocator.free == eng.cache.num_pages
    finally:
        native.set_pdl(prev)
    assert outs[True] == outs[False]


@pytest.mark.parametrize("heads,dh", [(4, 128), (6, 64), (16, 128)])
def test_rope_kv_append_equals_the_two_separate_kernels(heads, dh):
    from llm_systems_from_scratch_b200.models.transformer import RotaryEmbedding
    from llm_systems_from_scratch_b200.ops import native, serving_ops
    d, page, n_pages, r = heads * dh, 16, 12, 37
    g = torch.Generator(device="cuda").manual_seed(3)
    cache = RotaryEmbedding._build_cache(300, dh, 10000.0).cuda().contiguous()
    qkv = torch.randn(r, 3 * d, device="cuda", generator=g).bfloat16()
    pos = torch.randint(0, 300, (r,), device="cuda", generator=g).int()
    slots = torch.randperm(n_pages * page, device="cuda", generator=g)[:r].long()
    slots[3] = -1
    slots[11] = -1
    a_qkv, b_qkv = qkv.clone(), qkv.clone()
    ka, va = (torch.zeros(n_pages, page, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    kb, vb = torch.zeros_like(ka), torch.zeros_like(va)
    native.rope_(a_qkv, cache, pos, heads)
    serving_ops.kv_append(ka, va, a_qkv, slots)
    serving_ops.rope_kv_append(b_qkv, cache, pos, kb, vb, slots, heads)
    torch.cuda.synchronize()
    native.check_status()
    assert torch.equal(a_qkv, b_qkv) and torch.equal(ka, kb) and torch.equal(va, vb)
    # a slot beyond the cache is reported and not written; the row is still rotated
    bad = slots.clone()
    bad[5] = n_pages * page + 9
    c_qkv, kc, vc = qkv.clone(), torch.zeros_like(ka), torch.zeros_like(va)
    serving_ops.rope_kv_append(c_qkv, cache, pos, kc, vc, bad, heads)
    torch.cuda.synchronize()
    with pytest.raises(native.KernelError):
        native.check_status()
    assert torch.equal(c_qkv, a_qkv)
    keep = torch.ones(r, dtype=torch.bool, device="cuda")
    keep[5] = False
    keep &= slots >= 0
    assert torch.equal(kc.view(-1, d)[slots[keep]], ka.view(-1, d)[slots[keep]])
    assert float(kc.view(-1, d)[slots[5]].abs().sum()) == 0.0


@pytest.mark.parametrize("rows", [1, 7, 33, 64, 65, 1024, 1030, 129, 200, 256, 257, 1023])
@pytest.mark.parametrize("heads,dh", [(16, 128), (12, 64), (2, 32), (3, 40), (32, 128)])
def test_qkv_projection_that_rotates_and_appends(rows, heads, dh, monkeypatch):
    """Against the three steps one after the other, whichever the rule on rows and widths would take: rows of one and two short tiles and of whole
    ones, contractions that are sliced (4096 columns, up to 256 rows); rows without a slot, and a slot beyond the cache, which is reported."""
    from llm_systems_from_scratch_b200.ops import native, serving_ops
    monkeypatch.setattr(serving_ops, "APPEND_MAX_WORK", float("inf"))
    d, ctx, pages, page = heads * dh, 300, 70, 16
    g = torch.Generator("cuda").manual_seed(rows)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    h, w = rand(rows, d).bfloat16(), (rand(3 * d, d) / d ** 0.5).bfloat16()
    angle = torch.arange(ctx)[:, None] * 100.0 ** -(torch.arange(dh // 2) / (dh / 2))
    table = torch.stack((angle.cos(), angle.sin())).float().cuda()
    positions = torch.randint(0, ctx, (rows,), generator=g, device="cuda", dtype=torch.int32)
    slots = torch.randperm(pages * page, generator=g, device="cuda")[:rows]
    slots[rows // 2] = -1
    k, v = (rand(pages, page, d).bfloat16() for _ in range(2))
    k0, v0 = k.clone(), v.clone()
    native.status_word().zero_()
    got = serving_ops.qkv_rope_append(h, w, table, positions, k, v, slots, heads)
    native.check_status()
    want = h.double() @ w.double().T
    turn = want[:, :2 * d].reshape(rows, 2 * heads, dh // 2, 2)
    c, s = (t[positions.long()].double()[:, None] for t in table)
    want[:, :2 * d] = torch.stack((turn[..., 0] * c - turn[..., 1] * s, turn[..., 0] * s + turn[..., 1] * c), -1).reshape(rows, 2 * d)
    assert ((got.double() - want).norm() / want.norm()).item() < 2.0 ** -8             # two roundings to bf16 of at most 2^-9
    three, k3, v3 = native.gemm(h, w, "nt", b_stable=True), k0.clone(), v0.clone()
    serving_ops.rope_kv_append(three, table, positions, k3, v3, slots, heads)
    assert torch.equal(got, three) and torch.equal(k, k3) and torch.equal(v, v3)
    on = slots >= 0
    for cache, old, cols in ((k, k0, got[:, d:2 * d]), (v, v0, got[:, 2 * d:])):
        assert torch.equal(cache.view(-1, d)[slots[on]], cols[on])
        rest = torch.ones(pages * page, dtype=torch.bool, device="cuda").index_fill_(0, slots[on], False)
        assert torch.equal(cache.view(-1, d)[rest], old.view(-1, d)[rest])
    slots[0] = pages * page
    k.copy_(k0)
    serving_ops.qkv_rope_append(h, w, table, positions, k, v, slots, heads)
    torch.cuda.synchronize()
    with pytest.raises(native.KernelError):
        native.check_status()
    on = (slots >= 0) & (slots < pages * page)
    rest = torch.ones(pages * page, dtype=torch.bool, device="cuda").index_fill_(0, slots[on], False)
    assert torch.equal(k.view(-1, d)[rest], k0.view(-1, d)[rest])


@pytest.mark.parametrize("rows", [100, 129, 200])
def test_decode_steps_of_any_size_round_gate_and_up(rows, monkeypatch):
    """Logits of a step of single tokens, and tokens of the captured step of its bucket (128 or 256 rows), against the four launches one after
    the other: the same bits, below and above the rows that a tile has."""
    from llm_systems_from_scratch_b200 import ops
    from llm_systems_from_scratch_b200.models.transformer import TransformerLM
    from llm_systems_from_scratch_b200.ops import mixer_ops as mo, native
    from llm_systems_from_scratch_b200.serving import ServingEngine
    torch.manual_seed(0)
    cfg = dict(vocab_size=503, context_length=64, d_model=256, num_layers=2, num_heads=4, d_ff=704, rope_theta=10000.0)
    model = TransformerLM(**cfg, use_custom_triton=True).cuda().eval()
    g = torch.Generator().manual_seed(rows)
    prompts, singles = torch.randint(0, 503, (2, rows, 3), generator=g).tolist()

    def steps():
        eng = ServingEngine(model, page_size=16, max_batch=256, max_context=64)
        reqs = [eng.open(i) for i in range(rows)]
        eng.extend([(r, p, []) for r, p in zip(reqs, prompts)])
        # from here on there are single tokens only
        with monkeypatch.context() as at:
            if plain:
                at.setattr(mo, "glu", lambda h, w, n, act: ops.silu_mul_fwd(ops.gemm(h, w, "nt", b_stable=True)))
            logits = [eng.extend([(r, [t[i]], [0]) for r, t in zip(reqs, singles)]) for i in range(2)]
            for r in reqs:
                r.output, r.prompt = [7], list(range(r.fed))
                eng.sched.grow(r, r.fed + 2)
            return logits, eng.decode(reqs)
    plain = False
    got, tokens = steps()
    plain = True
    want, expected = steps()
    native.check_status()
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and tokens == expected


@pytest.mark.parametrize("rows,width,fused", [(1, 2048, True), (256, 2048, True), (381, 2048, True), (382, 2048, False), (512, 2048, False),
                                              (8192, 2048, False), (1525, 1024, True), (1526, 1024, False), (300, 4096, False)])
def test_long_steps_leave_rotation_and_append_to_a_launch_of_their_own(rows, width, fused, monkeypatch):
    """Rotating and appending in the product's epilogue takes the device longer than a pass of its own (512 rows of 2048 columns 27.7 us, 20.3)."""
    from llm_systems_from_scratch_b200.ops import serving_ops
    apart = []
    monkeypatch.setattr(serving_ops, "rope_kv_append", lambda *a: apart.append(len(a)))
    h, w = (torch.randn(n, width, device="cuda").bfloat16() for n in (rows, 3 * width))
    cache = torch.zeros(1, 16, width, device="cuda", dtype=torch.bfloat16)
    serving_ops.qkv_rope_append(h, w, torch.ones(2, 4, 32, device="cuda"), torch.zeros(rows, device="cuda", dtype=torch.int32), cache, cache.clone(),
                                torch.full((rows,), -1, device="cuda"), width // 64)
    assert bool(apart) != fused


@pytest.mark.parametrize("page", [1, 5, 8, 12, 16])
@pytest.mark.parametrize("heads,dh", [(1, 64), (5, 64), (3, 128), (32, 128)])
@pytest.mark.parametrize("splits", [1, 2, 7])
def test_paged_decode_forms(page, heads, dh, splits):
    """Pages that chunks of eight tokens straddle and ones that they do not, rows of columns that are no multiple of a warp's 256, contexts of
    more pages than a warp holds ids for, of none, one, a chunk and its edges; a query with a row pitch of its own."""
    from llm_systems_from_scratch_b200.ops import native, serving_ops, torch_impl
    d, lens = heads * dh, [0, 1, 7, 8, 9, 64, 100, 33 * page + 1, 65 * page]
    per, r = 65 * page if page > 1 else 100, len(lens)
    g = torch.Generator(device="cuda").manual_seed(page)
    n_pages = -(-per // page) + 40
    kc, vc = (torch.randn(n_pages, page, d, device="cuda", generator=g).bfloat16() for _ in "kv")
    tables = torch.stack([torch.randperm(n_pages, device="cuda", generator=g)[:-(-per // page)] for _ in range(r)]).int()
    lens = torch.tensor([min(n, tables.shape[1] * page) for n in lens], dtype=torch.int32, device="cuda")
    q = torch.randn(r, 3 * d, device="cuda", generator=g).bfloat16()
    out = serving_ops.paged_decode_attention(q, kc, vc, tables, lens, heads, splits)
    assert not out[0].any()
    ref = torch_impl.paged_decode_attention(q[1:, :d].double(), kc.double(), vc.double(), tables[1:], lens[1:], heads)
    assert (out[1:].double() - ref).norm() <= 2.0 ** -8 * ref.norm()          # one rounding to bf16 is at most 2^-9
    assert torch.equal(serving_ops.paged_decode_attention(q[:, :d].contiguous(), kc, vc, tables, lens, heads, splits), out)
    native.check_status()


@pytest.mark.parametrize("heads,dh,ff", [(4, 64, 704), (2, 128, 688), (16, 128, 5504)])
def test_all_layers_from_one_call(heads, dh, ff, monkeypatch):
    """Prompts (short, and long enough for CTA pairs), a portion that continues beside single tokens, steps of single tokens and a captured
    step: logits and caches are those of the ops one by one, bit for bit, with as many launches; what only the ops take is left to them."""
    from llm_systems_from_scratch_b200.models.transformer import TransformerLM
    from llm_systems_from_scratch_b200.ops import native, serving_ops
    from llm_systems_from_scratch_b200.serving import ServingEngine
    torch.manual_seed(0)
    model = TransformerLM(503, 1088, heads * dh, 2, heads, ff, 10000.0, use_custom_triton=True).cuda().eval()
    g = torch.Generator().manual_seed(heads)
    ids = lambda n: torch.randint(0, 503, (n,), generator=g).tolist()
    lengths = [1, 70, 200, 1030]
    prompts, more, singles = [ids(n) for n in lengths], ids(40), ids(4)
    taken = []
    real = serving_ops.transformer_layers

    def steps():
        eng = ServingEngine(model, page_size=16, max_batch=8, max_context=1088)
        native.reset_launch_count()
        reqs = [eng.open(i) for i in range(4)]
        logits = [eng.extend([(reqs[i], prompts[i], [lengths[i] - 1])]) for i in range(3)]
        logits.append(eng.extend([(reqs[3], prompts[3], [0, 1029])]))
        logits.append(eng.extend([(reqs[1], more, [39]), (reqs[2], [singles[2]], [0])]))
        logits.append(eng.extend([(r, [t], [0]) for r, t in zip(reqs, singles)]))
        for r in reqs:
            r.output, r.prompt = [7], list(range(r.fed))
            eng.sched.grow(r, r.fed + 2)
        return logits, eng.decode(reqs), [eng.cache.k.clone(), eng.cache.v.clone()], native.launch_count()
    monkeypatch.setattr(serving_ops, "transformer_layers", lambda *a, **k: taken.append(real(*a, **k)) or taken[-1])
    got = steps()
    assert taken and all(t is not None for t in taken)
    monkeypatch.setattr(serving_ops, "transformer_layers", lambda *a, **k: None)
    want = steps()
    assert all(torch.equal(a, b) for a, b in zip(got[0] + got[2], want[0] + want[2])) and got[1] == want[1] and got[3] == want[3]
    narrow = torch.zeros(3, heads * 8, dtype=torch.bfloat16, device="cuda")
    assert real(narrow, [None], heads, ff, 1e-5, None, None, None, None, None, False) is None           # heads of 8 columns
    native.check_status()
