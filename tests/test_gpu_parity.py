"""CUDA path against the CPU oracle, through the C ABI, on seeded inputs.

Tolerances (from the parity rules of this path):
  * selected index set: identical to the oracle except indices whose vote lies within 1e-4
    (relative) of the k-th vote; ascending order; init / local windows exact;
  * attention output: <= 2e-2 absolute for bf16, <= 1e-5 absolute in fp32 check mode;
  * scoring-query rotation: bit-exact; logits: 2e-3 absolute (fp32 summation order).
"""
import numpy as np
import pytest
import torch

from oracle import synth
from oracle import tokenselect_oracle as orc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

BF16, F32 = torch.bfloat16, torch.float32
ATTN_TOL = {BF16: 2e-2, F32: 1e-5}

# name, hq, hkv, d, N, n_init, n_local, top_k, rope_base, dtype, extra engine kwargs
SHAPES = [
    ("llama_tp1_bf16", 32, 8, 128, 8192, 128, 512, 1024, 5e5, BF16, {}),
    ("qwen_tp1_bf16", 28, 4, 128, 4096, 128, 512, 512, 1e6, BF16, {}),
    ("llama_tp4_bf16", 8, 2, 128, 3000, 16, 64, 256, 5e5, BF16, {}),
    ("llama_tp8_bf16", 4, 1, 128, 5000, 16, 64, 256, 5e5, BF16, {}),
    ("qwen_tp4_bf16", 7, 1, 128, 3001, 16, 64, 300, 1e6, BF16, {}),
    ("divmap_bf16", 8, 2, 128, 2500, 16, 64, 256, 5e5, BF16, {"gqa_map": "div"}),
    # the two bf16 scoring paths forced against their default row sizes
    ("direct_llama_tp1", 32, 8, 128, 8192, 128, 512, 1024, 5e5, BF16, {"score_path": "direct"}),
    ("direct_qwen_tp1", 28, 4, 128, 4096, 128, 512, 512, 1e6, BF16, {"score_path": "direct"}),
    ("direct_llama_tp4", 8, 2, 128, 3000, 16, 64, 256, 5e5, BF16, {"score_path": "direct"}),
    ("direct_llama_tp8", 4, 1, 128, 5000, 16, 64, 256, 5e5, BF16, {"score_path": "direct"}),
    ("plain_bf16", 8, 2, 128, 2048, 16, 64, 256, 5e5, BF16, {"plain_score": True}),
    # the general selection kernel followed by the stand-alone attention kernels (TS_CFG_SPLIT_ATTEND) at shapes
    # that default to the single layer-step kernel
    ("split_attend_llama_tp1", 32, 8, 128, 8192, 128, 512, 1024, 5e5, BF16, {"extra_flags": 256}),
    ("split_attend_qwen_tp4", 7, 1, 128, 3001, 16, 64, 300, 1e6, BF16, {"extra_flags": 256}),
    ("softcap_bf16", 8, 2, 128, 1500, 16, 64, 256, 5e5, BF16, {"logit_cap": 30.0}),
    ("fp32_check", 32, 8, 128, 8192, 128, 512, 1024, 5e5, F32, {}),
    ("fp32_d64_mha", 4, 4, 64, 1024, 8, 32, 128, 1e4, F32, {}),
    ("softcap_fp32", 8, 2, 128, 1500, 16, 64, 256, 5e5, F32, {"logit_cap": 30.0}),
]


@pytest.mark.parametrize("shape", SHAPES, ids=[s[0] for s in SHAPES])
def test_layer_step_matches_oracle(shape):
    name, hq, hkv, d, n, n_init, n_local, k, base, dtype, kw = shape
    seed = 100 + SHAPES.index(shape)
    case = synth.make_layer_case(seed, n, hq, hkv, d, n_init, n_local, base, dtype=dtype,
                                 gqa_map=kw.get("gqa_map", "mod"))
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, dtype, max_ctx=n + 8, **kw)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    out, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens)

    o = orc.DecodeOracle(gu.oracle_config(eng))
    ref = o.decode_layer(0, q, None, None, None, kp, vp, rtt, ridx, lens)
    info = ref["info"][0]
    assert int(res["flags"][0]) == orc.FLAG_RECOMPUTE == ref["flags"][0]

    # scoring query: bit-exact
    nc = n - n_init - n_local
    q_rot = eng.debug_read(0, hq * d, dtype)
    assert torch.equal(q_rot.view(hq, d), info["q_rot"]), "rotated scoring query differs"

    # logits
    lg = eng.debug_read(1, nc * hq, F32).view(nc, hq).numpy()
    want_lg = orc.score_logits(info["q_rot"], kp, rtt[case.req_pool_idx][n_init: n - n_local], eng.cfg.gqa_map)
    cols = gu.logits_columns_to_heads(eng)
    np.testing.assert_allclose(lg, want_lg.numpy()[cols].T, rtol=1e-5, atol=2e-3)

    # votes
    votes = eng.debug_read(2, nc, F32).numpy()
    np.testing.assert_allclose(votes, info["votes"].numpy(), rtol=2e-3, atol=1e-30)
    assert abs(votes.sum() - hq) < 1e-2 * hq

    # selection
    pos = gu.check_selection(eng, res, 0, ref["positions"][0], info["votes"], n)
    slots = res["slots"][0, : eng.cfg.n_sel]
    assert torch.equal(slots, rtt[case.req_pool_idx][torch.from_numpy(pos).long()])

    # attention over the rows the CUDA path selected
    want = orc.sparse_attention(q.view(hq, d), kp, vp, slots, eng.cfg.sm_scale or d ** -0.5, base, 1.0,
                                eng.cfg.logit_cap, torch.float64).reshape(-1)
    err = (out[0].double() - want).abs().max().item()
    assert err <= ATTN_TOL[dtype], f"attention error {err}"
    if np.array_equal(pos, ref["positions"][0].numpy()):
        err2 = (out[0].float() - ref["out"][0]).abs().max().item()
        assert err2 <= ATTN_TOL[dtype] + 1e-6


def _multi_request(seed, lens, hq, hkv, d, dtype, pool_rows, max_ctx, max_reqs, req_slots):
    """Several requests sharing one pool, rows scattered by a seeded permutation."""
    perm = synth.permutation(seed, 50, pool_rows)
    k_pool = synth.normal(seed, 51, (pool_rows, hkv, d)).to(dtype)
    v_pool = synth.normal(seed, 52, (pool_rows, hkv, d)).to(dtype)
    rtt = torch.full((max_reqs, max_ctx), -1, dtype=torch.int32)
    at = 0
    for n, slot in zip(lens, req_slots):
        rtt[slot, :n] = perm[at: at + n].to(torch.int32)
        at += n
    q = synth.normal(seed, 53, (len(lens), hq * d)).to(dtype)
    return q, k_pool, v_pool, rtt


@pytest.mark.parametrize("dtype,flags", [(BF16, 0), (BF16, 1024), (F32, 0)], ids=["bf16", "bf16_inline_attention", "fp32"])
def test_ragged_batch_with_dense_requests(dtype, flags):
    """Requests of different lengths in one call, some below the guard (attend to everything), at
    the guard boundary (N == n_sel and N == n_sel + 1), and one shorter than n_init.  Batches take the
    selection kernel followed by the attention kernels by default; TS_CFG_INLINE_ATTEND (1024) keeps the
    attention inside the layer-step kernel."""
    hq, hkv, d, n_init, n_local, k, base = 8, 2, 128, 16, 64, 256, 5e5
    n_sel = n_init + k + n_local
    lens = [2000, n_sel, n_sel + 1, 5, 1177, 40]
    slots = [3, 0, 5, 1, 2, 4]
    q, kp, vp, rtt = _multi_request(7, lens, hq, hkv, d, dtype, 6000, 2100, 6, slots)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, dtype, max_ctx=2100, max_reqs=6, max_batch=6,
                         extra_flags=flags)
    ridx, sl = torch.tensor(slots), torch.tensor(lens)
    out, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, sl)
    ref = orc.DecodeOracle(gu.oracle_config(eng)).decode_layer(0, q, None, None, None, kp, vp, rtt, ridx, sl)
    for b, n in enumerate(lens):
        assert int(res["flags"][b]) == ref["flags"][b]
        if ref["flags"][b] == orc.FLAG_DENSE:
            assert int(res["count"][b]) == n
            assert torch.equal(res["positions"][b, :n], torch.arange(n, dtype=torch.int32))
            assert torch.equal(res["slots"][b, :n], rtt[slots[b], :n])
        else:
            gu.check_selection(eng, res, b, ref["positions"][b], ref["info"][b]["votes"], n)
        cnt = int(res["count"][b])
        want = orc.sparse_attention(q[b].view(hq, d), kp, vp, res["slots"][b, :cnt], d ** -0.5, base, 1.0, 0.0,
                                    torch.float64).reshape(-1)
        assert (out[b].double() - want).abs().max().item() <= ATTN_TOL[dtype]


def test_exact_ties_take_lowest_positions():
    """All candidate keys equal -> all votes equal -> the k lowest candidate positions win."""
    hq, hkv, d, n_init, n_local, k, base, n = 8, 2, 128, 16, 64, 256, 5e5, 3000
    case = synth.make_layer_case(11, n, hq, hkv, d, n_init, n_local, base, dtype=BF16, planted_frac=0.0)
    rows = case.req_to_token[case.req_pool_idx][:n].long()
    case.k_pool[rows] = case.k_pool[rows[0]].clone()
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    out, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens)
    pos = res["positions"][0, : eng.cfg.n_sel]
    assert torch.equal(pos[: n_init + k], torch.arange(n_init + k, dtype=torch.int32))
    assert torch.isfinite(out.float()).all()


def test_pairwise_ties_break_by_position():
    """Every candidate key appears twice (positions p and p + Nc/2): votes tie in pairs, and where the
    k-th vote's pair straddles the boundary the lower position must be the one taken."""
    hq, hkv, d, n_init, n_local, k, base = 8, 2, 128, 16, 64, 255, 5e5
    nc = 2000
    n = n_init + nc + n_local
    case = synth.make_layer_case(12, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    row = case.req_to_token[case.req_pool_idx]
    lo = row[n_init: n_init + nc // 2].long()
    hi = row[n_init + nc // 2: n_init + nc].long()
    case.k_pool[hi] = case.k_pool[lo]
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    _, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens)
    ref = orc.DecodeOracle(gu.oracle_config(eng)).decode_layer(0, q, None, None, None, kp, vp, rtt, ridx, lens)
    votes = eng.debug_read(2, nc, F32).numpy()
    assert np.array_equal(votes[: nc // 2], votes[nc // 2:]), "duplicated keys must give identical votes"
    got = res["positions"][0, n_init: n_init + k].numpy() - n_init
    # exact rule on the CUDA path's own votes: sort by (-vote, position)
    order = np.lexsort((np.arange(nc), -votes.astype(np.float64)))[:k]
    assert np.array_equal(got, np.sort(order))
    gu.check_selection(eng, res, 0, ref["positions"][0], ref["info"][0]["votes"], n)


@pytest.mark.parametrize("ks", [5, 6, 1, 32])
def test_vote_max_pool(ks):
    hq, hkv, d, n_init, n_local, k, base, n = 8, 2, 128, 16, 64, 256, 5e5, 2048
    case = synth.make_layer_case(20 + ks, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8, kernel_size=ks)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    _, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens)
    ref = orc.DecodeOracle(gu.oracle_config(eng)).decode_layer(0, q, None, None, None, kp, vp, rtt, ridx, lens)
    pooled = ref["info"][0]["votes"]
    nc = n - n_init - n_local
    assert pooled.numel() == (nc if ks % 2 else nc - 1)
    got = eng.debug_read(2, pooled.numel(), F32).numpy()
    np.testing.assert_allclose(got, pooled.numpy(), rtol=2e-3, atol=1e-30)
    # max-pooling creates runs of equal votes; compare with the exact rule on the CUDA path's own votes
    sel = res["positions"][0, n_init: n_init + k].numpy() - n_init
    order = np.lexsort((np.arange(got.size), -got.astype(np.float64)))[:k]
    assert np.array_equal(sel, np.sort(order))


def test_kv_append_then_attend():
    """k_new / v_new are written to the pools at out_cache_loc before selection and attention."""
    hq, hkv, d, n_init, n_local, k, base, n = 8, 2, 128, 16, 64, 256, 5e5, 1500
    case = synth.make_layer_case(31, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    loc = rtt[case.req_pool_idx, n - 1: n].clone()
    k_new = synth.normal(31, 60, (1, hkv * d)).to(BF16)
    v_new = synth.normal(31, 61, (1, hkv * d)).to(BF16)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8)
    out, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens, k_new, v_new, loc)
    assert torch.equal(res["k_pool"][loc.long()].reshape(1, -1), k_new)
    assert torch.equal(res["v_pool"][loc.long()].reshape(1, -1), v_new)
    kp2, vp2 = kp.clone(), vp.clone()
    ref = orc.DecodeOracle(gu.oracle_config(eng)).decode_layer(0, q, k_new, v_new, loc, kp2, vp2, rtt, ridx, lens)
    gu.check_selection(eng, res, 0, ref["positions"][0], ref["info"][0]["votes"], n)
    want = orc.sparse_attention(q.view(hq, d), kp2, vp2, res["slots"][0, : eng.cfg.n_sel], d ** -0.5, base, 1.0,
                                0.0, torch.float64).reshape(-1)
    assert (out[0].double() - want).abs().max().item() <= ATTN_TOL[BF16]


def test_bad_pool_row_is_reported_not_dereferenced():
    hq, hkv, d, n_init, n_local, k, base, n = 8, 2, 128, 16, 64, 256, 5e5, 1200
    case = synth.make_layer_case(41, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    rtt = rtt.clone()
    rtt[case.req_pool_idx, 500] = kp.shape[0] + 123
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8)
    dev = eng.device
    eng.decode_layer(0, q.to(dev), None, None, None, kp.to(dev), vp.to(dev), rtt.to(dev),
                     ridx.to(device=dev, dtype=torch.int32), lens.to(device=dev, dtype=torch.int32))
    torch.cuda.synchronize()
    code, detail = eng.last_error()
    assert code == 6 and detail == kp.shape[0] + 123
    # the error word is cleared by the read; the handle keeps working
    out, _ = gu.run_gpu(eng, 0, q, kp, vp, case.req_to_token, ridx, lens)
    assert torch.isfinite(out.float()).all()


def test_workspace_capacity_is_checked_on_the_device():
    hq, hkv, d, n_init, n_local, k, base, n = 8, 2, 128, 16, 64, 256, 5e5, 3000
    case = synth.make_layer_case(42, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8, max_batch=1, max_total=1024)
    dev = eng.device
    eng.decode_layer(0, q.to(dev), None, None, None, kp.to(dev), vp.to(dev), rtt.to(dev),
                     ridx.to(device=dev, dtype=torch.int32), lens.to(device=dev, dtype=torch.int32))
    torch.cuda.synchronize()
    code, _ = eng.last_error()
    assert code == 4


def test_invalid_arguments_are_rejected_on_the_host():
    eng = gu.make_engine(8, 2, 128, 16, 64, 256, 5e5, BF16, max_ctx=4096, max_batch=2)
    dev = eng.device
    q = torch.zeros(3, 8 * 128, dtype=BF16, device=dev)
    pool = torch.zeros(64, 2, 128, dtype=BF16, device=dev)
    rtt = torch.zeros(4, 4096, dtype=torch.int32, device=dev)
    idx = torch.zeros(3, dtype=torch.int32, device=dev)
    from tokenselect_b200 import TokenSelectError
    with pytest.raises(TokenSelectError) as ei:
        eng.decode_layer(0, q, None, None, None, pool, pool.clone(), rtt, idx, idx)   # batch 3 > max_batch 2
    assert ei.value.status == 4
    with pytest.raises(TokenSelectError):
        eng.decode_layer(7, q[:1], None, None, None, pool, pool.clone(), rtt, idx[:1], idx[:1])  # layer out of range
    with pytest.raises(ValueError):
        eng.decode_layer(0, q[:1].float(), None, None, None, pool, pool.clone(), rtt, idx[:1], idx[:1])


@pytest.mark.parametrize("gain", [6.0, 20.0], ids=["peaked", "very_peaked"])
def test_underflowing_votes(gain):
    """A query scaled until almost every softmax term underflows: most votes are denormal or exactly zero.
    Votes in the normal fp32 range must select exactly as in the oracle; where the k-th vote itself is
    denormal or zero, the two evaluations (division folded into the exponent here, exp then divide in the
    oracle) may disagree only among candidates whose oracle vote is below 2^-120, and zeros are taken from
    the lowest positions."""
    hq, hkv, d, n_init, n_local, k, base, n = 8, 2, 128, 16, 64, 256, 5e5, 3000
    case = synth.make_layer_case(61, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    case.q.mul_(gain)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8)
    out, res = gu.run_gpu(eng, 0, *gu.case_tensors(case))
    o = orc.DecodeOracle(gu.oracle_config(eng))
    flag, pos, info = o.select(0, case.req_pool_idx, case.q.view(hq, d), case.k_pool,
                               case.req_to_token[case.req_pool_idx], n)
    votes = info["votes"].double().numpy()
    got = res["positions"][0, n_init:n_init + k].numpy() - n_init
    want = pos[n_init:n_init + k].numpy() - n_init
    assert int(res["count"][0]) == eng.cfg.n_sel and np.all(np.diff(got) > 0)
    kth = np.sort(votes)[::-1][k - 1]
    diff = set(got.tolist()) ^ set(want.tolist())
    tiny = 2.0 ** -120
    if kth >= tiny:
        ok, why = orc.index_sets_match(got, want, votes, k, rel_tol=1e-4)
        assert ok, why
    else:
        assert all(votes[i] < tiny for i in diff), sorted(votes[list(diff)])[-3:]
        # everything in the normal range is in
        assert set(np.nonzero(votes >= tiny)[0].tolist()) <= set(got.tolist())
    assert torch.isfinite(out.float()).all()


def test_phase_stamps_only_with_the_diagnostic_flag():
    """TS_CFG_PHASE_STAMPS (32): CTA 0 records nanosecond timestamps at the selection kernel's phase boundaries,
    read back with ts_debug_read(3).  Without the flag the kernels read no timer and the slots stay zero; the
    results are the same either way."""
    hq, hkv, d, n_init, n_local, top_k, base, n = 8, 2, 128, 16, 64, 256, 5e5, 3000
    case = synth.make_layer_case(97, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    outs = []
    for flags in (0, 32):
        eng = gu.make_engine(hq, hkv, d, n_init, n_local, top_k, base, BF16, max_ctx=n + 8, max_batch=1,
                             extra_flags=flags)
        out, dbg = gu.run_gpu(eng, 0, *gu.case_tensors(case))
        eng.raise_on_device_error()
        ts = eng.debug_read(3, 64, torch.int64)
        if flags == 0:
            assert int(ts.abs().sum()) == 0
        else:
            phase = ts[:9]                        # start, plan, score, barrier, vote, barrier, filter, barrier, emit
            assert int(phase.min()) > 0 and bool((phase[1:] >= phase[:-1]).all())
        outs.append((out, dbg["slots"]))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("hq,hkv,d,n,dtype,kw", [
    (8, 8, 128, 337, F32, {}),                       # one head a KV head; a single candidate more than top_k
    (6, 3, 64, 1001, F32, {}),                       # three KV heads: warps left over
    (40, 20, 64, 700, F32, {}),                      # more KV heads than warps
    (7, 1, 128, 901, F32, {}),                       # a full and a partial block of four heads, all warps on one KV head
    (8, 1, 64, 1200, BF16, {}),
    (12, 4, 64, 1111, BF16, {"gqa_map": "div"}),
], ids=lambda v: str(v))
def test_cuda_core_scoring_shapes(hq, hkv, d, n, dtype, kw):
    """Head-block, warp and row-step edges of the scoring without tensor cores.  Logits: fp32 sums of d products of
    magnitude ~1 in another order than the oracle's, held to the 2e-3 absolute stated above."""
    n_init, n_local, k, base = 16, 64, 256, 5e5
    case = synth.make_layer_case(200 + n, n, hq, hkv, d, n_init, n_local, base, dtype=dtype, gqa_map=kw.get("gqa_map", "mod"))
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, dtype, max_ctx=n + 8, **kw)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    out, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens)
    ref = orc.DecodeOracle(gu.oracle_config(eng)).decode_layer(0, q, None, None, None, kp, vp, rtt, ridx, lens)
    info, nc = ref["info"][0], n - n_init - n_local
    lg = eng.debug_read(1, nc * hq, F32).view(nc, hq).numpy()
    want = orc.score_logits(info["q_rot"], kp, rtt[case.req_pool_idx][n_init: n - n_local], eng.cfg.gqa_map)
    np.testing.assert_allclose(lg, want.numpy()[gu.logits_columns_to_heads(eng)].T, rtol=1e-5, atol=2e-3)
    gu.check_selection(eng, res, 0, ref["positions"][0], info["votes"], n)
    want = orc.sparse_attention(q.view(hq, d), kp, vp, res["slots"][0, : eng.cfg.n_sel], d ** -0.5, base, 1.0, 0.0,
                                torch.float64).reshape(-1)
    assert (out[0].double() - want).abs().max().item() <= ATTN_TOL[dtype]


@pytest.mark.parametrize("hq,hkv,lens,kw,ties", [
    (4, 1, [262145], {}, False),                     # more candidates a CTA than its shared-memory copies hold
    (7, 1, [240003], {}, False),                     # logit rows that are no multiple of 16 bytes
    (8, 1, [250001], {"kernel_size": 4}, False),     # pooled votes; an even window drops the last candidate
    (4, 1, [240000], {}, True),                      # every vote equal: lists instead of records, full radix descent
    (8, 2, [400 + 37 * i for i in range(40)], {}, False),   # several requests a CTA
    (28, 4, [60001, 900, 150000, 343], {}, False),   # blocks of logits through two buffers, across requests
    (14, 2, [30000, 8000], {"score_path": "direct"}, False),   # votes from global memory only
], ids=["long", "odd_heads", "pooled_even", "ties", "many_requests", "two_buffers", "direct"])
def test_votes_and_exact_top_k_at_scale(hq, hkv, lens, kw, ties):
    """Votes against the 64-bit softmax of the kernel's own logits (relative 1e-4: a logit of magnitude 100 times log2 e
    has 1e-5 absolute error in fp32, and so has its exponential, relatively), and the list against the exact rule on
    the kernel's own votes: the k largest, lowest position first among equals, in position order.  The output against the
    64-bit attention over the rows the kernel listed."""
    d, n_init, n_local, k, base = 128, 16, 64, 256, 5e5
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(sum(lens) + hq)
    total = sum(lens)
    kp = torch.randn(total, hkv, d, generator=g, device=dev, dtype=BF16)
    if ties:
        kp[:] = kp[:1].clone()
    vp = torch.randn(total, hkv, d, generator=g, device=dev, dtype=BF16)
    q = torch.randn(len(lens), hq * d, generator=g, device=dev, dtype=BF16)
    perm = torch.randperm(total, generator=g, device=dev).to(torch.int32)
    rtt = torch.zeros(len(lens), max(lens), dtype=torch.int32, device=dev)
    at = 0
    for b, n in enumerate(lens):
        rtt[b, :n] = perm[at:at + n]
        at += n
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=max(lens), max_reqs=len(lens),
                         max_batch=len(lens), max_total=total, **kw)
    dbg = eng.new_debug_buffers(len(lens))
    out = eng.decode_layer(0, q, None, None, None, kp, vp, rtt, torch.arange(len(lens), dtype=torch.int32, device=dev),
                           torch.tensor(lens, dtype=torch.int32, device=dev), debug=dbg)
    torch.cuda.synchronize()
    eng.raise_on_device_error()
    region = [(max(n - n_init - n_local, 0) + 127) // 128 * 128 if n > n_init + n_local + k else 0 for n in lens]
    logits = eng.debug_read(1, sum(region) * hq, F32).view(-1, hq).to(dev).double()
    votes = eng.debug_read(2, sum(region), F32).to(dev)
    ks = kw.get("kernel_size", -1)
    off = 0
    for b, n in enumerate(lens):
        if not region[b]:
            assert int(dbg["count"][b]) == n
            continue
        nc = n - n_init - n_local
        want = torch.softmax(logits[off:off + nc], 0).sum(1)
        if ks > 0:
            want = torch.nn.functional.max_pool1d(want[None], ks, stride=1, padding=(ks - 1) // 2)[0]
        got = votes[off:off + want.numel()]
        torch.testing.assert_close(got.double(), want, rtol=1e-4, atol=1e-30)
        best = torch.sort(got, descending=True, stable=True).indices[:k].sort().values
        pos = dbg["positions"][b]
        assert torch.equal(pos[n_init:n_init + k].long(), best + n_init)
        assert torch.equal(dbg["slots"][b], rtt[b][pos.long()])
        off += region[b]
    for b in range(len(lens)):                       # the attention over the rows the kernel listed, the window's last among them
        slots = dbg["slots"][b, :int(dbg["count"][b])].cpu()
        rows, at = slots.long().unique(return_inverse=True)
        want = orc.sparse_attention(q[b].cpu().view(hq, d), kp[rows.to(dev)].cpu(), vp[rows.to(dev)].cpu(), at.to(torch.int32),
                                    d ** -0.5, base, 1.0, 0.0, torch.float64).reshape(-1)
        assert (out[b].cpu().double() - want).abs().max().item() <= ATTN_TOL[BF16], b


@pytest.mark.parametrize("hq,hkv,batch,k", [(32, 8, 48, 256), (28, 4, 40, 256), (8, 2, 100, 100), (7, 1, 130, 100), (8, 1, 2, 17)])
def test_batched_attention_shares_blocks(hq, hkv, batch, k):
    """Batches whose list blocks outnumber the attention kernel's CTAs (a CTA then covers several requests, or part of
    one), with lists of one row, of a whole block, of one row more and of the full budget, against the oracle on the
    rows the kernel listed (2e-2, the bf16 output's rounding)."""
    d, n_init, n_local, base = 128, 16, 64, 5e5
    lens = [(1, 16, 17, 5, n_init + n_local + k, 700 + i, 40 + i)[i % 7] for i in range(batch)]
    slots = list(range(batch))
    q, kp, vp, rtt = _multi_request(90 + hq, lens, hq, hkv, d, BF16, sum(lens) + 64, 900, batch, slots)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=900, max_reqs=batch, max_batch=batch)
    out, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, torch.tensor(slots), torch.tensor(lens))
    for b, n in enumerate(lens):
        cnt = int(res["count"][b])
        assert cnt == min(n, eng.cfg.n_sel)
        want = orc.sparse_attention(q[b].view(hq, d), kp, vp, res["slots"][b, :cnt], d ** -0.5, base, 1.0, 0.0,
                                    torch.float64).reshape(-1)
        assert (out[b].double() - want).abs().max().item() <= ATTN_TOL[BF16], (b, n)


@pytest.mark.parametrize("n", [2500, 900], ids=["selects", "all_tokens"])
@pytest.mark.parametrize("hq", [40, 48, 56, 64])
def test_one_request_with_wide_groups_over_eight_kv_heads(hq, n):
    """Five to eight query heads on each of eight KV heads, lists of 32 rows a CTA (all tokens) and of 16 or more (windows
    of 720 rows beside the winners): the widest partial outputs, inside the layer-step kernel up to six heads a KV head and
    in the attention kernels beyond."""
    hkv, d, n_init, n_local, k, base = 8, 128, 128, 592, 1024, 5e5
    case = synth.make_layer_case(500 + hq + n, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8, max_batch=1)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    out, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens)
    ref = orc.DecodeOracle(gu.oracle_config(eng)).decode_layer(0, q, None, None, None, kp, vp, rtt, ridx, lens)
    assert int(res["flags"][0]) == ref["flags"][0] == (orc.FLAG_RECOMPUTE if n > eng.cfg.n_sel else orc.FLAG_DENSE)
    cnt = int(res["count"][0])
    assert cnt == min(n, eng.cfg.n_sel)
    if n > eng.cfg.n_sel:
        gu.check_selection(eng, res, 0, ref["positions"][0], ref["info"][0]["votes"], n)
    want = orc.sparse_attention(q.view(hq, d), kp, vp, res["slots"][0, :cnt], d ** -0.5, base, 1.0, 0.0,
                                torch.float64).reshape(-1)
    assert (out[0].double() - want).abs().max().item() <= ATTN_TOL[BF16]


@pytest.mark.parametrize("hq,nc", [(40, 6784), (40, 7200), (48, 8200), (32, 6160), (56, 7200)])
def test_equal_votes_beside_the_copies_of_the_own_candidates(hq, nc):
    """Every candidate key equal, so that all candidates are members of the threshold bin and are staged together in shared
    memory: as many as the staging area holds, and more than lie between its start and the CTA's copies of its own votes
    and pool rows, which the emission still reads.  The k lowest positions win."""
    hkv, d, n_init, n_local, k, base = 8, 128, 16, 64, 256, 5e5
    n = n_init + nc + n_local
    case = synth.make_layer_case(600 + hq, n, hq, hkv, d, n_init, n_local, base, dtype=BF16, planted_frac=0.0)
    rows = case.req_to_token[case.req_pool_idx][:n].long()
    case.k_pool[rows] = case.k_pool[rows[0]].clone()
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8, max_batch=1)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    out, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens)
    pos, slots = res["positions"][0], res["slots"][0]
    assert torch.equal(pos[: n_init + k], torch.arange(n_init + k, dtype=torch.int32))
    assert torch.equal(slots, rtt[case.req_pool_idx][pos.long()])
    want = orc.sparse_attention(q.view(hq, d), kp, vp, slots, d ** -0.5, base, 1.0, 0.0, torch.float64).reshape(-1)
    assert (out[0].double() - want).abs().max().item() <= ATTN_TOL[BF16]


@pytest.mark.parametrize("hq,hkv,batch,flags", [(8, 2, 2, 0), (32, 8, 3, 0), (7, 1, 1, 256), (8, 2, 1, 0)],
                         ids=["batch2", "batch3", "split_attention", "layer_step"])
def test_query_may_start_at_any_element(hq, hkv, batch, flags):
    """A contiguous query that starts at an odd element of its storage gives the bits of an aligned one, wherever the
    attention runs."""
    d, n_init, n_local, k, base = 128, 16, 64, 256, 5e5
    lens, slots = [900, 300, 1200][:batch], list(range(batch))
    q, kp, vp, rtt = _multi_request(97, lens, hq, hkv, d, BF16, 2600, 1300, 3, slots)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=1300, max_reqs=3, max_batch=batch, extra_flags=flags)
    dev = eng.device
    store = torch.zeros(q.numel() + 1, dtype=BF16, device=dev)
    odd = store[1:].view(batch, -1)
    odd.copy_(q)
    assert odd.is_contiguous() and odd.data_ptr() % 4 == 2
    rest = (None, None, None, kp.to(dev), vp.to(dev), rtt.to(dev), torch.tensor(slots, dtype=torch.int32, device=dev),
            torch.tensor(lens, dtype=torch.int32, device=dev))
    want, got = eng.decode_layer(0, q.to(dev), *rest), eng.decode_layer(0, odd, *rest)
    torch.cuda.synchronize()
    eng.raise_on_device_error()
    assert torch.equal(want, got)


def test_bases_off_the_copies_grid_are_rejected_on_the_host():
    """Pools, new rows and a chunk's queries and output move in 16-byte pieces: a base that is not a multiple of 16 bytes
    is refused before anything is launched."""
    from tokenselect_b200 import TokenSelectError
    hq, hkv, d, n_init, n_local, k, base, n = 8, 2, 128, 16, 64, 256, 5e5, 200
    case = synth.make_layer_case(98, n, hq, hkv, d, n_init, n_local, base, dtype=BF16)
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=n + 8, max_batch=1)
    dev = eng.device

    def off(t):
        store = torch.zeros(t.numel() + 1, dtype=t.dtype, device=dev)
        store[1:].copy_(t.reshape(-1))
        return store[1:].view(t.shape)

    q, kp, vp, rtt = (t.to(dev) for t in (case.q[None].contiguous(), case.k_pool, case.v_pool, case.req_to_token))
    new = torch.zeros(1, hkv * d, dtype=BF16, device=dev)
    loc = rtt[case.req_pool_idx, n - 1:n].clone()
    where = (rtt, torch.tensor([case.req_pool_idx], dtype=torch.int32, device=dev), torch.tensor([n], dtype=torch.int32, device=dev))
    before = eng.launch_count
    for args in ((None, None, None, off(kp), vp), (None, None, None, kp, off(vp)), (off(new), new, loc, kp, vp), (new, off(new), loc, kp, vp)):
        with pytest.raises(TokenSelectError) as ei:
            eng.decode_layer(0, q, *args, *where)
        assert ei.value.status == 1
    chunk = (rtt, case.req_pool_idx, n)
    for qc, pools, out in ((off(q), (kp, vp), None), (q, (off(kp), vp), None), (q, (kp, off(vp)), None), (q, (kp, vp), off(q))):
        with pytest.raises(TokenSelectError) as ei:
            eng.extend_chunk(0, qc, None, None, None, *pools, *chunk, out=out)
        assert ei.value.status == 1
    assert eng.launch_count == before
    eng.extend_chunk(0, q, None, None, None, kp, vp, *chunk)
    eng.raise_on_device_error()


@pytest.mark.parametrize("hq,hkv,d", [(8, 2, 128), (12, 4, 64)])
def test_a_nan_key_makes_its_heads_statistics_nan(hq, hkv, d):
    """fp32 scoring: a softmax over logits of which one is NaN is NaN everywhere, and so are the votes; the selection still
    names k distinct candidates."""
    n_init, n_local, k, base, n = 16, 64, 256, 5e5, 900
    case = synth.make_layer_case(99, n, hq, hkv, d, n_init, n_local, base, dtype=F32)
    q, kp, vp, rtt, ridx, lens = gu.case_tensors(case)
    kp[int(rtt[case.req_pool_idx, 500]), 0, 3] = float("nan")
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, F32, max_ctx=n + 8, max_batch=1)
    _, res = gu.run_gpu(eng, 0, q, kp, vp, rtt, ridx, lens)
    nc = n - n_init - n_local
    logits = eng.debug_read(1, nc * hq, F32).view(nc, hq)
    assert torch.isnan(logits).sum() == hq // hkv and torch.isnan(logits[500 - n_init]).sum() == hq // hkv
    assert torch.isnan(torch.softmax(logits, 0).sum(1)).all()
    assert torch.isnan(eng.debug_read(2, nc, F32)).all()
    pos = res["positions"][0, n_init:n_init + k]
    assert bool((pos[1:] > pos[:-1]).all()) and int(pos[0]) >= n_init and int(pos[-1]) < n - n_local


@pytest.mark.parametrize("hq,hkv,lens,kw", [
    (32, 8, [700], {}), (8, 2, [336], {}), (7, 1, [1], {}), (28, 4, [333], {}),
    (8, 2, [300, 17, 336], {}), (8, 2, [300, 17, 336], {"extra_flags": 1024}),      # batches; attention inside the layer-step kernel
    (8, 2, [336], {"query_cache": True}),
], ids=lambda v: str(v))
def test_new_rows_are_attended_by_requests_below_the_guard(hq, hkv, lens, kw):
    """Requests that attend to every token, with this step's K/V rows: one CTA appends a request's row and another attends
    to it.  Before every step the row holds large values, which a read that came too early would bring into the output.
    Forty steps over fresh rows, the last four checked against the 64-bit attention, all against their repetition."""
    d, n_init, n_local, k, base = 128, 16, 64, 256 if max(lens) <= 336 else 1024, 5e5
    batch = len(lens)
    q, kp, vp, rtt = _multi_request(96, lens, hq, hkv, d, BF16, sum(lens) + 8, max(lens), batch, list(range(batch)))
    eng = gu.make_engine(hq, hkv, d, n_init, n_local, k, base, BF16, max_ctx=max(lens), max_reqs=batch, max_batch=batch, **kw)
    dev = eng.device
    kd, vd, rd = kp.to(dev), vp.to(dev), rtt.to(dev)
    ridx, sl = torch.arange(batch, dtype=torch.int32, device=dev), torch.tensor(lens, dtype=torch.int32, device=dev)
    loc = torch.stack([rtt[b, n - 1] for b, n in enumerate(lens)])
    locd, rows = loc.to(dev), loc.long()
    for t in range(40):
        k_new, v_new = synth.normal(96, 100 + t, (batch, hkv * d)).to(BF16), synth.normal(96, 200 + t, (batch, hkv * d)).to(BF16)
        qt = synth.normal(96, 300 + t, (batch, hq * d)).to(BF16)
        kn, vn, qd = k_new.to(dev), v_new.to(dev), qt.to(dev)
        kd[rows.to(dev)], vd[rows.to(dev)] = 30.0, 1000.0
        out = eng.decode_layer(0, qd, kn, vn, locd, kd, vd, rd, ridx, sl)
        again = eng.decode_layer(0, qd, None, None, None, kd, vd, rd, ridx, sl)
        assert torch.equal(out, again), t                # the rows are in place in the second call
        kp[rows], vp[rows] = k_new.view(batch, hkv, d), v_new.view(batch, hkv, d)
        if t < 36:
            continue
        assert torch.equal(kd.cpu(), kp) and torch.equal(vd.cpu(), vp)
        for b, n in enumerate(lens):
            want = orc.sparse_attention(qt[b].view(hq, d), kp, vp, rtt[b, :n], d ** -0.5, base, 1.0, 0.0, torch.float64).reshape(-1)
            assert (out[b].cpu().double() - want).abs().max().item() <= ATTN_TOL[BF16], (t, b)
    torch.cuda.synchronize()
    eng.raise_on_device_error()
