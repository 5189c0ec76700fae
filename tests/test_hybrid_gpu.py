"""Hybrid Gated-DeltaNet model on the sm_100a kernel chain (needs a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _hybrid_cfg(gdn_dim: int = 64):
    from smcsd_b200.models.config import ModelConfig
    lt = ["linear_attention", "linear_attention", "linear_attention", "full_attention"] * 2
    return ModelConfig(arch="hybrid_gdn", vocab_size=8192, hidden_size=512, n_layers=8, n_heads=4, n_kv_heads=2,
                       head_dim=128, ffn_size=1024, rope_theta=10000.0, max_position=2048, layer_types=lt,
                       gdn_n_k_heads=2, gdn_n_v_heads=4, gdn_head_k_dim=gdn_dim, gdn_head_v_dim=gdn_dim, gdn_conv_width=4,
                       partial_rotary=0.25, attn_output_gate=True, qk_norm=True, norm_plus_one=True, rms_eps=1e-6,
                       name="hybrid-test")


def _dense_draft():
    from smcsd_b200.models.config import ModelConfig
    return ModelConfig(arch="llama", vocab_size=8192, hidden_size=256, n_layers=2, n_heads=4, n_kv_heads=2,
                       head_dim=64, ffn_size=768, max_position=2048, tie_embeddings=True, name="dense-draft")


def test_native_hybrid_forward_matches_torch():
    from smcsd_b200 import SMCEngine
    from smcsd_b200.models.layers import ExtendBatch
    eng = SMCEngine(_hybrid_cfg(), _dense_draft(), n_particles=4, gamma=4, max_running_requests=2, context_length=512,
                    device="cuda", max_total_tokens=8192, backend="native", cycle_graph=False)
    s = eng._sched
    m, nm = s.target, s.native_runner.target
    dev = "cuda"
    bs, P = 4, 19
    g = torch.Generator(device=dev).manual_seed(0)
    rows = torch.arange(bs, dtype=torch.int32, device=dev)
    for b in range(bs):
        s.bt.table[b, :P + 8] = s.alloc.alloc(P + 8)
    ids = torch.randint(0, 8192, (bs * P,), generator=g, device=dev)
    pre = ExtendBatch(ids, torch.arange(P, device=dev).repeat(bs), s.bt.table[:bs, :P].reshape(-1), rows,
                      torch.zeros(bs, dtype=torch.int32, device=dev), extend_len=0, extend_lens=[P] * bs,
                      prefix_lens_host=[0] * bs)
    m.forward_torch(pre, s.kv_t, s.bt.table, s.state_t)
    conv0, temp0 = s.state_t.conv.clone(), s.state_t.temporal.clone()
    kk, vv = s.kv_t.k.clone(), s.kv_t.v.clone()
    for E in (5, 1, 2):
        ids2 = torch.randint(0, 8192, (bs * E,), generator=g, device=dev, dtype=torch.int32)
        pos2 = (torch.arange(E, device=dev) + P).repeat(bs).to(torch.int32)
        locs2 = s.bt.table[:bs, P:P + E].reshape(-1).contiguous()
        pref = torch.full((bs,), P, dtype=torch.int32, device=dev)
        ext = ExtendBatch(ids2.long(), pos2.long(), locs2, rows, pref, extend_len=E, prefix_lens_host=[P] * bs)
        ref = m.logits_torch(m.forward_torch(ext, s.kv_t, s.bt.table, s.state_t))
        conv_ref, temp_ref = s.state_t.conv.clone(), s.state_t.temporal.clone()
        # rewind the recurrent state and the cache, then run the kernel chain on the same inputs
        s.state_t.conv.copy_(conv0); s.state_t.temporal.copy_(temp0); s.kv_t.k.copy_(kk); s.kv_t.v.copy_(vv)
        nm.forward(ids2, pos2, locs2, rows, pref, bs, E)
        got = nm.lm_head(bs * E)[: bs * E].clone()
        torch.cuda.synchronize()
        assert s.native_runner.check_status() == 0
        scale = ref.abs().max().item()
        assert (got - ref).abs().max().item() < 0.08 * scale, E
        assert (s.state_t.temporal[:, :bs] - temp_ref[:, :bs]).abs().max().item() < 0.05 * max(1.0, temp_ref.abs().max().item())
        assert (s.state_t.conv[:, :bs] - conv_ref[:, :bs]).abs().max().item() < 0.05 * max(1.0, conv_ref.abs().max().item())
        s.state_t.conv.copy_(conv0); s.state_t.temporal.copy_(temp0); s.kv_t.k.copy_(kk); s.kv_t.v.copy_(vv)


def test_engine_hybrid_target_dense_draft_native():
    from smcsd_b200 import SMCEngine
    g = torch.Generator().manual_seed(0)
    prompts = [torch.randint(0, 8192, (30,), generator=g).tolist() for _ in range(3)]
    outs = {}
    for graph in (False, True):
        eng = SMCEngine(_hybrid_cfg(), _dense_draft(), n_particles=4, gamma=4, max_running_requests=2,
                        context_length=512, device="cuda", max_total_tokens=8192, backend="native", cycle_graph=graph,
                        draft_temperature=0.7, target_temperature=0.7, random_seed=2)
        o = eng.generate(input_ids=prompts, sampling_params={"max_new_tokens": 31, "ignore_eos": True})
        assert [x["completion_tokens"] for x in o] == [31] * 3
        assert eng._sched.native_runner.check_status() == 0
        eng._sched.check_idle_invariants()
        outs[graph] = o
    for a, b in zip(outs[False], outs[True]):
        assert a["output_ids"] == b["output_ids"]


def test_hybrid_state_follows_resampling_native():
    from smcsd_b200.config import EngineArgs
    from smcsd_b200.io_types import GenerateRequest, ParticleOutput, SamplingParams
    from smcsd_b200.models import build_model
    from smcsd_b200.runtime.scheduler import SMCScheduler
    cfg = _hybrid_cfg()
    model = build_model(cfg, torch.bfloat16, "cuda", seed=0)
    args = EngineArgs(model_path=cfg, draft_model_path=cfg, n_particles=4, gamma=3, max_running_requests=1,
                      context_length=512, device="cuda", max_total_tokens=8192, backend="native",
                      draft_temperature=0.8, target_temperature=0.8, resample_threshold=2.0).finalize()
    sched = SMCScheduler(args, target=model, draft=model)
    g = torch.Generator().manual_seed(3)
    sched.add_request(GenerateRequest("r", torch.randint(0, 8192, (17,), generator=g).tolist(),
                                      SamplingParams(max_new_tokens=25, ignore_eos=True)))
    outs = sched.run_until_idle()
    po = [o for o in outs if isinstance(o, ParticleOutput)][0]
    assert int(sched.state.counters[2]) > 0
    # the draft advances its state token by token, the target in gamma+1-token passes; bf16 noise only
    assert max(abs(w) for w in po.log_w_tilde) < 0.6, po.log_w_tilde
    assert sched.native_runner.check_status() == 0


@pytest.mark.parametrize("gdn_dim,lens", [(64, [37, 16, 5, 70]), (128, [137, 16, 5, 270])])
def test_native_hybrid_prefill_matches_torch_prefill(gdn_dim, lens):
    """Prompt pass of a hybrid target and a hybrid draft through the kernel chains (attention layers over 16-token
    blocks, Gated-DeltaNet layers walking each prompt once) vs the plain PyTorch forward: same cache contents and
    the same recurrent state, the draft's one token short under the deferred schedule.  With 128 x 128 heads and
    long prompts the Gated-DeltaNet layers take the chunk-parallel tcgen05 kernel."""
    from smcsd_b200.config import EngineArgs
    from smcsd_b200.models import build_model
    from smcsd_b200.runtime.scheduler import SMCScheduler
    from smcsd_b200.runtime.worker import PrefillItem
    cfg = _hybrid_cfg(gdn_dim)
    model = build_model(cfg, torch.bfloat16, "cuda", seed=0)
    args = EngineArgs(model_path=cfg, draft_model_path=cfg, n_particles=4, gamma=3, max_running_requests=4,
                      context_length=512, device="cuda", max_total_tokens=8192, backend="native",
                      cycle_graph=False).finalize()
    s = SMCScheduler(args, target=model, draft=model)
    r = s.native_runner
    if gdn_dim == 128:
        assert r.target.gdn_chunked
    g = torch.Generator().manual_seed(4)
    items = []
    for L in lens:
        row = s.bt.alloc_parent_row()
        s.bt.table[row, :L] = s.alloc.alloc(L)
        items.append(PrefillItem(row, torch.randint(0, 8192, (L,), generator=g).tolist()))
    rows = torch.tensor([it.row for it in items], device="cuda")
    for pool in (s.state_t, s.state_d):
        pool.clear_rows(rows)
    r.prefill(s.worker, items)
    torch.cuda.synchronize()
    assert r.check_status() == 0
    got = [x.clone() for x in (s.kv_t.k, s.kv_t.v, s.kv_d.k, s.state_t.temporal, s.state_t.conv, s.state_d.temporal,
                               s.state_d.conv)]
    s.kv_t.k.zero_(); s.kv_t.v.zero_(); s.kv_d.k.zero_()
    for pool in (s.state_t, s.state_d):
        pool.clear_rows(rows)
    native, s.worker.native = s.worker.native, None
    s.worker.prefill(items)
    s.worker.native = native
    ref = [s.kv_t.k, s.kv_t.v, s.kv_d.k, s.state_t.temporal, s.state_t.conv, s.state_d.temporal, s.state_d.conv]
    names = ["target K", "target V", "draft K", "target temporal", "target conv", "draft temporal", "draft conv"]
    for it, L in zip(items, lens):
        for a, b, name in zip(got[:3], ref[:3], names):
            # the stateful draft stops one token short, so its last prompt page is only written by the kernel path
            n = L - 1 if name.startswith("draft") else L
            pages = s.bt.table[it.row, :n].long()
            x = b[:, pages].float()
            err = (a[:, pages].float() - x).abs().max().item()
            assert err < 0.06 * max(1.0, x.abs().max().item()), (name, L, err)
    for a, b, name in zip(got[3:], ref[3:], names[3:]):
        x = b[:, rows].float()
        err = (a[:, rows].float() - x).abs().max().item()
        assert err < 0.05 * max(1.0, x.abs().max().item()), (name, err)
    # the two pools must differ: the draft's state stops one token before the target's
    assert (s.state_t.temporal[:, rows] - s.state_d.temporal[:, rows]).abs().max().item() > 0


@pytest.mark.parametrize("lens", [[150, 64, 1, 300], [512, 37]])
def test_gdn_chunked_prefill_kernel_matches_recurrence(lens):
    """Chunk-parallel delta rule on tcgen05 (64 tokens per step, dk = dv = 128) against the token-by-token recurrence in
    fp32 PyTorch and against the token-serial kernel: outputs after the gated RMSNorm and the final recurrent state,
    from a non-zero initial state, rows of different lengths (partial last chunks, a single-token row)."""
    import torch.nn.functional as F
    from smcsd_b200.models.hybrid_gdn import gdn_recurrent_step
    from smcsd_b200.ops import native as K
    torch.manual_seed(5)
    dev = "cuda"
    Hk, Hv, dk, dv, W, eps = 2, 4, 128, 128, 4, 1e-6
    key_dim, value_dim = Hk * dk, Hv * dv
    conv_dim = 2 * key_dim + value_dim
    ldp = conv_dim + value_dim + 2 * Hv
    ldp += (-ldp) % 8
    T, bs = sum(lens), len(lens)
    proj = torch.randn(T, ldp, device=dev)
    proj[:, conv_dim + value_dim:] *= 2.0                        # spread the gates
    conv_w = (torch.randn(conv_dim, W, device=dev) * 0.3).bfloat16()
    dt_bias = torch.ones(Hv, device=dev)
    A_log = torch.log(torch.empty(Hv, device=dev).uniform_(0.5, 8.0))
    gnorm_w = (1.0 + 0.1 * torch.randn(dv, device=dev)).bfloat16()
    rows = torch.tensor([3, 0, 2, 5][:bs], dtype=torch.int32, device=dev)
    conv0 = torch.randn(8, conv_dim, W - 1, device=dev) * 0.5
    temp0 = torch.randn(8, Hv, dk, dv, device=dev) * 0.2
    off = torch.tensor([sum(lens[:i]) for i in range(bs)], dtype=torch.int32, device=dev)
    ln = torch.tensor(lens, dtype=torch.int32, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)

    # fp32 reference
    ref_out = torch.zeros(T, value_dim, device=dev)
    ref_temp = temp0.clone()
    rep = Hv // Hk
    for b, n in enumerate(lens):
        t0, r = int(off[b]), int(rows[b])
        seq = torch.cat([conv0[r], proj[t0:t0 + n, :conv_dim].t()], dim=1)
        conv = F.silu(F.conv1d(seq.unsqueeze(0), conv_w.float().unsqueeze(1), groups=conv_dim).squeeze(0)).t()
        q = conv[:, :key_dim].reshape(n, Hk, dk)
        k = conv[:, key_dim:2 * key_dim].reshape(n, Hk, dk)
        v = conv[:, 2 * key_dim:].reshape(n, Hv, dv)
        q = (q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5).repeat_interleave(rep, dim=1)
        k = (k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(rep, dim=1)
        z = proj[t0:t0 + n, conv_dim:conv_dim + value_dim].view(n, Hv, dv)
        beta = torch.sigmoid(proj[t0:t0 + n, conv_dim + value_dim:conv_dim + value_dim + Hv])
        g = -A_log.exp() * F.softplus(proj[t0:t0 + n, conv_dim + value_dim + Hv:conv_dim + value_dim + 2 * Hv] + dt_bias)
        S = ref_temp[r].clone()
        for t in range(n):
            S, o = gdn_recurrent_step(S, q[t], k[t], v[t], g[t], beta[t])
            y = o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + eps)
            ref_out[t0 + t] = (y.bfloat16().float() * gnorm_w.float() * F.silu(z[t])).reshape(-1)
        ref_temp[r] = S

    got = {}
    for chunked in (False, True):
        conv_s, temp_s = conv0.clone(), temp0.clone()
        conv_out = torch.zeros(T, conv_dim, device=dev)
        out = torch.zeros(T, value_dim, device=dev, dtype=torch.bfloat16)
        K.gdn_step(proj, conv_s, temp_s, rows, conv_w, dt_bias, A_log, gnorm_w, conv_out, out, bs=bs, E=0, Hk=Hk, Hv=Hv,
                   dk=dk, dv=dv, W=W, eps=eps, tok_off=off, tok_len=ln, chunked=chunked, status=status,
                   max_len=max(lens) if chunked else 0)
        torch.cuda.synchronize()
        assert int(status) == 0
        got[chunked] = (out.float(), temp_s)
    o_scale, s_scale = ref_out.abs().max().item(), ref_temp.abs().max().item()
    for chunked in (False, True):
        o, s = got[chunked]
        tol = 2e-2 if chunked else 1e-2                           # bf16 operands in the chunked form, fp32 otherwise
        assert (o - ref_out).abs().max().item() < tol * o_scale, (chunked, (o - ref_out).abs().max().item(), o_scale)
        assert (s - ref_temp).abs().max().item() < tol * s_scale, (chunked, (s - ref_temp).abs().max().item(), s_scale)
    used = [int(r) for r in rows]
    untouched = [r for r in range(8) if r not in used]
    assert torch.equal(got[True][1][untouched], temp0[untouched])


@pytest.mark.parametrize("lens", [[1], [63, 65], [64, 128, 2], [129, 0, 191, 33]])
def test_gdn_chunks_match_the_token_serial_kernel(lens):
    """Rows at the edges of chunks, one of them empty, and scratch memory of exactly their chunks (one chunk less is refused by status)."""
    from smcsd_b200.ops import native as K
    torch.manual_seed(9)
    dev, Hk, Hv, d, W = "cuda", 2, 4, 128, 4
    conv_dim = 2 * Hk * d + Hv * d
    ldp = conv_dim + Hv * d + 2 * Hv
    T, bs = sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    proj, conv_w = torch.randn(T, ldp, device=dev), (torch.randn(conv_dim, W, device=dev) * 0.3).bfloat16()
    dt, A_log, gw = torch.ones(Hv, device=dev), torch.log(torch.empty(Hv, device=dev).uniform_(0.5, 8.0)), torch.ones(d, device=dev).bfloat16()
    rows, off, ln = i32(list(range(bs))), i32([sum(lens[:i]) for i in range(bs)]), i32(lens)
    state0 = torch.randn(bs, Hv, d, d, device=dev) * 0.2
    got, chunks = [], sum((n + 63) // 64 for n in lens)

    def run(chunked, slots):
        conv_s, state, out = torch.zeros(bs, conv_dim, W - 1, device=dev), state0.clone(), torch.zeros(T, Hv * d, device=dev).bfloat16()
        status, room = torch.zeros(1, dtype=torch.int32, device=dev), torch.empty(K.gdn_scratch_bytes(0, max(slots, 1), Hv), dtype=torch.uint8, device=dev)
        K.gdn_step(proj, conv_s, state, rows, conv_w, dt, A_log, gw, torch.zeros(T, conv_dim, device=dev), out, bs=bs, E=0, Hk=Hk, Hv=Hv, dk=d,
                   dv=d, W=W, eps=1e-6, tok_off=off, tok_len=ln, chunked=chunked, status=status, max_len=max(lens), scratch=room)
        torch.cuda.synchronize()
        return out.float(), state, int(status)
    ref, exact_state, _ = run(False, 1)
    out, state, status = run(True, chunks)
    assert status == 0
    # operands rounded to bf16 (2^-9 each, some ten of them a chunk) against fp32 ones
    assert (out - ref).abs().max() < 2e-2 * ref.abs().max() and (state - exact_state).abs().max() < 2e-2 * exact_state.abs().max()
    if chunks > 1:
        assert run(True, chunks - 1)[2] == K.ERR_BOUNDS


@pytest.mark.parametrize("held,new,chunked", [(0, [50], True), (0, [48], False), (0, [100, 20], True), (5, [100], False), (10, [300], False),
                                              (8, [500], True), (1, [130], True), (3, [130], False)])
def test_delta_rule_in_chunks_is_for_rows_long_on_average(monkeypatch, held, new, chunked):
    """Sequences under way beside new prompts: batches whose rows average 64 tokens (in blocks of 16) take the chunk kernels, which round
    operands to bf16; all others keep fp32, also where one of their rows is long."""
    from smcsd_b200 import SMCEngine
    from smcsd_b200.ops import native as K
    eng = SMCEngine(_hybrid_cfg(128), _dense_draft(), n_particles=1, gamma=1, max_running_requests=16, context_length=1024, device="cuda",
                    max_total_tokens=8192, backend="native")
    some = lambda n: torch.arange(n).mul(37).remainder(8192).tolist()
    if held:
        eng.feed([(f"h{i}", some(20 + i), []) for i in range(held)])
    seen, step = [], K.gdn_step
    monkeypatch.setattr(K, "gdn_step", lambda *a, **kw: (seen.append(kw.get("chunked", False)), step(*a, **kw))[1])
    eng.feed([(f"h{i}", [7], [0]) for i in range(held)] + [(f"p{i}", some(n), [n - 1]) for i, n in enumerate(new)])
    assert len(seen) == 6 and set(seen) == {chunked}


def _chunk_case(lens, seed=9):
    torch.manual_seed(seed)
    dev, Hk, Hv, d, W = "cuda", 2, 4, 128, 4
    conv_dim, T, bs = (2 * Hk + Hv) * d, sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    args = [torch.randn(T, conv_dim + Hv * d + 2 * Hv, device=dev), torch.zeros(bs, conv_dim, W - 1, device=dev), torch.randn(bs, Hv, d, d, device=dev) * 0.2,
            i32(list(range(bs))), (torch.randn(conv_dim, W, device=dev) * 0.3).bfloat16(), torch.ones(Hv, device=dev), torch.zeros(Hv, device=dev),
            torch.ones(d, device=dev).bfloat16(), torch.zeros(T, conv_dim, device=dev), torch.zeros(T, Hv * d, device=dev).bfloat16()]
    return args, dict(bs=bs, E=0, Hk=Hk, Hv=Hv, dk=d, dv=d, W=W, eps=1e-6, tok_off=i32([sum(lens[:i]) for i in range(bs)]), tok_len=i32(lens),
                      status=i32([0]))


def test_gdn_chunks_without_a_bound_of_the_rows():
    """The bound of the rows' lengths is optional: the same bits without it (the window of a row by the serial form of the convolution)."""
    from smcsd_b200.ops import native as K
    got = []
    for bound in (130, 0):
        a, kw = _chunk_case([130, 5, 64])
        K.gdn_step(*a, chunked=True, max_len=bound, **kw)
        torch.cuda.synchronize()
        assert int(kw["status"]) == 0
        got.append((a[9], a[2], a[1]))
    assert all(torch.equal(x, y) for x, y in zip(*got))


def test_gdn_chunks_report_a_row_longer_than_its_bound():
    from smcsd_b200.ops import native as K
    a, kw = _chunk_case([40, 200, 65])
    want, kw2 = _chunk_case([40, 200, 65])
    before = a[2].clone()
    K.gdn_step(*a, chunked=True, max_len=100, **kw)
    K.gdn_step(*want, chunked=True, max_len=200, **kw2)
    torch.cuda.synchronize()
    assert int(kw["status"]) == K.ERR_BOUNDS and int(kw2["status"]) == 0
    assert torch.equal(a[2][1], before[1]) and torch.equal(a[2][[0, 2]], want[2][[0, 2]]) and torch.equal(a[9][240:], want[9][240:])


def test_gdn_scratch_is_allocated_once():
    """Batches of more and more rows, up to as many as run in chunks: one allocation (the caching allocator would keep every earlier one)."""
    from smcsd_b200 import SMCEngine
    from smcsd_b200.ops import native as K
    eng = SMCEngine(_hybrid_cfg(128), _dense_draft(), n_particles=1, gamma=1, max_running_requests=64, context_length=512, device="cuda",
                    max_total_tokens=8192, backend="native")
    places = set()
    for n, length in ((1, 100), (2, 64), (40, 70), (60, 64), (60, 49)):
        eng.feed([(str(i), list(range(length)), []) for i in range(n)], [str(i) for i in range(n)])
        room = eng._sched.native_runner._prefill_chain("target")._gdn_scratch
        places.add((room.data_ptr(), room.numel()))
    assert len(places) == 1
    most = K.gdn_most_rows(4096)                                     # every row 49 tokens, 64 in blocks of 16
    assert K.gdn_takes_chunks(K.gdn_padded([49] * most), most) and not K.gdn_takes_chunks(K.gdn_padded([48] * most), most)
    assert (most + 1) * 49 > 4096


def test_gdn_chunks_count_cycles_per_phase():
    from smcsd_b200.ops import native as K
    (a, kw), (b, kw2) = _chunk_case([200, 70]), _chunk_case([200, 70])
    trace = torch.zeros(10, dtype=torch.int64, device="cuda")
    K.gdn_step(*a, chunked=True, max_len=200, trace=trace, **kw)
    K.gdn_step(*b, chunked=True, max_len=200, **kw2)
    torch.cuda.synchronize()
    assert int(kw["status"]) == 0 and bool((trace > 0).all()) and int(trace.sum()) < 10 ** 7
    assert torch.equal(a[9], b[9]) and torch.equal(a[2], b[2])
