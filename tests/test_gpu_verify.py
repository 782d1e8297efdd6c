"""Parity of the CUDA verify/decode attention with the reference's known answers and with the CPU oracle,
through the C ABI (all_quant_b200.uq_cuda -> libuq_b200.so).  Needs a B200."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from all_quant_b200 import uq_cuda
from oracle import uq_oracle as O
from tests.cases import check_close, check_harness_rule, load_cases

pytestmark = pytest.mark.gpu
CASES = load_cases()


def dev(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t if dtype is None else t.view(dtype)


def run_case(c, **kw):
    q = dev(c.q.view(np.int16), torch.bfloat16)
    out = uq_cuda.uq_decode_cuda(q, dev(c.kc), dev(c.ks), dev(c.vc), dev(c.vs), dev(c.bt), dev(c.sl), sm_scale=c.sm_scale, **kw)
    torch.cuda.synchronize()
    assert uq_cuda.last_status()[0] == 0
    return out.float().cpu().numpy()


@pytest.mark.parametrize("c", CASES, ids=repr)
def test_known_answers(c):
    got = run_case(c)
    check_close(got, c.ref, c.name)
    check_harness_rule(got, c.ref, c.name)
    for b in range(c.B):            # rows that see no key are exact zeros
        for j in range(c.K):
            if c.sl[b] - c.K + j + 1 <= 0:
                assert not got[b, j].any()


@pytest.mark.parametrize("c", [x for x in CASES if x.name in ("ref_cuda_main_K8", "gen_k8g8_K8", "ref_cuda_p16_g4_K3", "gen_d256_K8")], ids=repr)
@pytest.mark.parametrize("nsplit", [1, 2, 3, 7, 16])
def test_nsplit_invariance(c, nsplit):
    check_close(run_case(c, nsplit=nsplit), c.ref, f"{c.name} nsplit={nsplit}")


@pytest.mark.parametrize("c", [x for x in CASES if x.name in ("ref_cuda_main_K4", "gen_cfg0_K4", "gen_g7_K3")], ids=repr)
def test_fused_equals_no_sharing(c):
    a = run_case(c, fused=True)
    b = run_case(c, fused=False)
    check_close(b, c.ref, c.name + " no-sharing")
    assert np.abs(a - b).max() <= 2e-2 * max(1.0, np.abs(c.ref).max())


@pytest.mark.parametrize("path", ["fma", "tc"])
def test_both_kernels_on_the_same_case(path, monkeypatch):
    c = [x for x in CASES if x.name == "ref_cuda_main_K8"][0]
    monkeypatch.setenv("UQ_B200_CFG", f"path={path}")
    try:
        got = run_case(c)
    except RuntimeError as e:   # a forced kernel that does not serve the shape answers invalid value, never garbage
        assert "InvalidValue" in str(e)
        pytest.skip(f"{path} kernel does not serve this shape")
    assert uq_cuda.last_path() == (1 if path == "fma" else 2)
    check_close(got, c.ref, f"{c.name} {path}")


def test_caller_workspace_int64_tables_and_out_argument():
    c = [x for x in CASES if x.name == "ref_cuda_main_K4"][0]
    q = dev(c.q.view(np.int16), torch.bfloat16)
    ns = 5
    ws = torch.full((uq_cuda.workspace_floats(c.B, c.K, c.HQ, c.HKV, c.D, ns),), float("nan"), device="cuda")
    out = torch.full_like(q, float("nan"))
    r = uq_cuda.uq_decode_cuda(q, dev(c.kc), dev(c.ks), dev(c.vc), dev(c.vs), dev(c.bt).long(), dev(c.sl).long(), nsplit=ns,
                               workspace=ws, out=out)
    assert r.data_ptr() == out.data_ptr()
    check_close(out.float().cpu().numpy(), c.ref, "workspace")


def test_poisoned_tail_and_unused_table_entries():
    """Bytes after seq_len in the last page and page-table entries past the sequence may hold anything."""
    c = [x for x in CASES if x.name == "gen_cfg0_K4"][0]
    kc, ks, vc, vs, bt = (a.copy() for a in (c.kc, c.ks, c.vc, c.vs, c.bt))
    for b in range(c.B):
        n = int(c.sl[b])
        last = bt[b, (n - 1) // c.PAGE]
        t = n % c.PAGE
        if t:
            for a in (kc, ks, vc, vs):
                a[last, :, t:] = 0xFF
        bt[b, (n + c.PAGE - 1) // c.PAGE:] = -1
    q = dev(c.q.view(np.int16), torch.bfloat16)
    out = uq_cuda.uq_decode_cuda(q, dev(kc), dev(ks), dev(vc), dev(vs), dev(bt), dev(c.sl))
    check_close(out.float().cpu().numpy(), c.ref, "poisoned tail")


def test_scale_extremes():
    """Scale bytes far from 127 (2^+-20): outputs follow the oracle on the same bytes."""
    c = [x for x in CASES if x.name == "ref_cuda_main_K2"][0]
    ks = (c.ks.astype(np.int32) - 20).clip(0, 255).astype(np.uint8)
    vs = (c.vs.astype(np.int32) + 20).clip(0, 255).astype(np.uint8)
    ref = O.reference(c.q, c.kc, ks, c.vc, vs, c.bt, c.sl, c.sm_scale)
    q = dev(c.q.view(np.int16), torch.bfloat16)
    out = uq_cuda.uq_decode_cuda(q, dev(c.kc), dev(ks), dev(c.vc), dev(vs), dev(c.bt), dev(c.sl))
    mx = np.abs(ref).max()      # outputs are ~2^20 here: apply the acceptance rule to outputs normalised to O(1)
    check_close(out.float().cpu().numpy() / mx, ref / mx, "scale extremes")


@pytest.mark.parametrize("K,HQ,HKV,D", [(16, 16, 2, 128), (12, 16, 2, 128), (8, 32, 2, 64), (16, 8, 1, 256), (13, 14, 2, 128)])
def test_more_than_64_query_rows_run_as_draft_chunks_on_the_tensor_core_kernel(K, HQ, HKV, D):
    """K * group between 65 and 128 rows: consecutive drafts are verified in chunks of at most 64 rows; answers follow the oracle, short sequences (fewer tokens than drafts) included."""
    rng = np.random.default_rng(K * 100 + HQ)
    B, PAGE = 3, 32
    sl = np.array([900, 5, 333], np.int32)       # 5 < K: some drafts see nothing or only part of the tokens
    npg = -(-int(sl.max()) // PAGE)
    pages = B * npg
    k = rng.standard_normal((pages, HKV, PAGE, D)).astype(np.float32) * np.exp(0.5 * rng.standard_normal((1, HKV, 1, D))).astype(np.float32)
    v = rng.standard_normal((pages, HKV, PAGE, D)).astype(np.float32)
    kc, ks = O.quantize_fp4(k)
    vc, vs = O.quantize_fp4(v)
    bt = rng.permutation(pages).astype(np.int32).reshape(B, npg)
    qb = O.bf16_bits(rng.standard_normal((B, K, HQ, D)).astype(np.float32))
    ref = O.reference(qb, kc, ks, vc, vs, bt, sl)
    q = dev(qb.view(np.int16), torch.bfloat16)
    args = (dev(kc), dev(ks), dev(vc), dev(vs), dev(bt), dev(sl))
    for nsplit in (None, 2):
        out = uq_cuda.uq_decode_cuda(q, *args, nsplit=nsplit)
        assert uq_cuda.last_path() == 2 and uq_cuda.last_status() == (0, 0, 0, 0)
        check_close(out.float().cpu().numpy(), ref, f"K={K} nsplit={nsplit}")
    # the context-split form writes its partial rows through the same mapping
    o, lse = uq_cuda.uq_decode_partial(q, *args)
    merged = uq_cuda.uq_merge(o.unsqueeze(0), lse.unsqueeze(0))
    check_close(merged.float().cpu().numpy(), ref, f"K={K} partial")


@pytest.mark.parametrize("nsplit", [1, 2, None])
@pytest.mark.parametrize("K,HQ,HKV,D", [(16, 16, 2, 128), (9, 8, 1, 256), (5, 28, 2, 64)])
def test_two_chunks_of_drafts_share_one_launch(K, HQ, HKV, D, nsplit):
    """65..128 query rows: both chunks are work items of one attention launch and one combine (two launches in all), rows that
    divide unevenly between them, a sequence without keys, and one slot per item (whole items per CTA) included."""
    rng = np.random.default_rng(K + D)
    B, PAGE = 5, 16
    sl = np.array([700, 0, 3, 128, 129], np.int32)
    npg = -(-int(sl.max()) // PAGE)
    kc, ks = O.quantize_fp4(rng.standard_normal((B * npg, HKV, PAGE, D)).astype(np.float32))
    vc, vs = O.quantize_fp4(rng.standard_normal((B * npg, HKV, PAGE, D)).astype(np.float32))
    bt = rng.permutation(B * npg).astype(np.int32).reshape(B, npg)
    qb = O.bf16_bits(rng.standard_normal((B, K, HQ, D)).astype(np.float32))
    n0 = uq_cuda.launch_count()
    out = uq_cuda.uq_decode_cuda(dev(qb.view(np.int16), torch.bfloat16), *(dev(a) for a in (kc, ks, vc, vs, bt, sl)), nsplit=nsplit)
    assert uq_cuda.launch_count() == n0 + 2 and uq_cuda.last_path() == 2 and uq_cuda.last_status() == (0, 0, 0, 0)
    check_close(out.float().cpu().numpy(), O.reference(qb, kc, ks, vc, vs, bt, sl), f"K={K} nsplit={nsplit}")



@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("D,PAGE", [(64, 16), (64, 32), (64, 48), (64, 64), (64, 128), (128, 16), (128, 32), (256, 16), (256, 32)])
@pytest.mark.parametrize("rows", [8, 32, 64])
def test_scale_slices_of_small_copies_come_by_a_third_warp(D, PAGE, rows, fmt):
    """Small copy units: the scale bytes arrive 16 bytes per lane (1 .. 8 keys each, up to four pieces per lane), units past a
    sequence's end are left out; lengths that end inside a unit, on its edge and one key past a tile."""
    rng = np.random.default_rng(D + PAGE + rows)
    B, HKV, G = 4, 2, 8
    K = rows // G
    sl = np.array([1, 128 + PAGE, 129, 5 * 128 - 3], np.int32)
    npg = -(-int(sl.max()) // PAGE)
    shape = lambda row: (B * npg, HKV, PAGE, row)
    kc, vc = (rng.integers(0, 256, shape(D // 2), dtype=np.uint8) for _ in range(2))
    # Scales and queries for which every key counts: with the 16 bytes of a neighbour in the place of any one piece, K or V, some row of
    # the oracle's answer moves by more than 1.5 % of its largest entry (98 % of the pieces or more, by format and head size).
    per, kr, vr, qs = (32, (124, 128), (125, 129), 0.4) if fmt == 0 else (16, (0x28, 0x48), (0x28, 0x48), 0.3)
    ks, vs = (rng.integers(*r, shape(D // per)).astype(np.uint8) for r in (kr, vr))
    bt = rng.permutation(B * npg).astype(np.int32).reshape(B, npg)
    qb = O.bf16_bits(qs * rng.standard_normal((B, K, HKV * G, D)).astype(np.float32))
    ref = O.reference(qb, kc, ks, vc, vs, bt, sl) if fmt == 0 else O.reference_nvfp4(qb, kc, ks, vc, vs, bt, sl, 0.5, 0.5)
    out = uq_cuda.uq_decode_cuda(dev(qb.view(np.int16), torch.bfloat16), *(dev(a) for a in (kc, ks, vc, vs, bt, sl)),
                                 **(dict(fmt=1, k_ts=0.5, v_ts=0.5) if fmt else {}))
    assert uq_cuda.last_path() == 2 and uq_cuda.last_status() == (0, 0, 0, 0)
    # row by row relative to the row's largest: a sequence of one key returns values up to 24, one of 637 keys small sums, and the
    # rounding of bf16 (2^-9 of an entry) is far below the rule's 1 % in each
    mx = np.abs(ref).max(-1, keepdims=True)
    mx[mx == 0] = 1
    check_close(out.float().cpu().numpy() / mx, ref / mx, f"PAGE={PAGE}")


@pytest.mark.parametrize("PAGE,D,fmt", [(16, 128, 0), (256, 128, 0), (512, 128, 0), (256, 64, 0), (1024, 256, 0), (256, 128, 1), (48, 128, 0),
                                         (96, 128, 0), (80, 64, 0), (192, 256, 0), (48, 128, 1), (144, 128, 0), (24, 128, 0), (40, 64, 0)])
def test_page_sizes_from_16_to_1024_tokens(PAGE, D, fmt):
    """Pages smaller than the 128-key tile are copied whole, larger ones in 128-token parts, and a page size that neither
    divides 128 nor is a multiple of it (48, 80, 96, 144, 192 ...) in parts of gcd(PAGE, 128) tokens, three to eight copies per
    stream and tile; only a page size that is not a multiple of 16 runs on the CUDA-core kernel.  Ragged lengths that end
    inside a page and inside a part of a page."""
    rng = np.random.default_rng(PAGE + D)
    B, K, HQ, HKV = 3, 4, 8, 2
    sl = np.array([2 * PAGE + 77, 130, 3 * PAGE], np.int32)
    npg = -(-int(sl.max()) // PAGE)
    pages = B * npg
    kc = rng.integers(0, 256, (pages, HKV, PAGE, D // 2), dtype=np.uint8)
    vc = rng.integers(0, 256, (pages, HKV, PAGE, D // 2), dtype=np.uint8)
    if fmt == 0:
        ks = rng.integers(125, 130, (pages, HKV, PAGE, D // 32)).astype(np.uint8)
        vs = rng.integers(125, 130, (pages, HKV, PAGE, D // 32)).astype(np.uint8)
    else:
        ks = rng.integers(0x30, 0x40, (pages, HKV, PAGE, D // 16)).astype(np.uint8)
        vs = rng.integers(0x30, 0x40, (pages, HKV, PAGE, D // 16)).astype(np.uint8)
    bt = rng.permutation(pages).astype(np.int32).reshape(B, npg)
    qb = O.bf16_bits(0.3 * rng.standard_normal((B, K, HQ, D)).astype(np.float32))
    ref = O.reference(qb, kc, ks, vc, vs, bt, sl) if fmt == 0 else O.reference_nvfp4(qb, kc, ks, vc, vs, bt, sl, 0.5, 0.5)
    q = dev(qb.view(np.int16), torch.bfloat16)
    kw = dict(fmt=1, k_ts=0.5, v_ts=0.5) if fmt else {}
    for nsplit in (None, 3):
        out = uq_cuda.uq_decode_cuda(q, dev(kc), dev(ks), dev(vc), dev(vs), dev(bt), dev(sl), nsplit=nsplit, **kw)
        assert uq_cuda.last_status() == (0, 0, 0, 0)
        assert uq_cuda.last_path() == (2 if PAGE % 16 == 0 else 1)
        mx = np.abs(ref).max()      # random codes and scales give outputs of order ten: the rule is applied to outputs normalised to O(1)
        check_close(out.float().cpu().numpy() / mx, ref / mx, f"PAGE={PAGE} D={D} fmt={fmt} nsplit={nsplit}")


@pytest.mark.parametrize("B,HKV,G,K", [(700, 8, 2, 2), (1000, 4, 8, 1), (300, 8, 8, 8)])
def test_many_short_sequences_put_more_segments_on_a_cta_than_its_list_holds(B, HKV, G, K):
    """Hundreds of sequences of one or two tiles (some empty): a CTA's share of the work list then spans more items than the 32
    candidates listed at set-up, so every role goes on with the walker from where the list ends; with one partial slot per item
    (nsplit 1) the items are dealt out by index, the list's other form."""
    rng = np.random.default_rng(B + HKV)
    D, PAGE = 128, 64
    HQ = HKV * G
    sl = rng.integers(1, 4 * PAGE, B).astype(np.int32)
    sl[rng.random(B) < 0.05] = 0
    sl[rng.random(B) < 0.05] = K
    npg = -(-int(sl.max()) // PAGE)
    pages = B * npg
    kc = rng.integers(0, 256, (pages, HKV, PAGE, D // 2), dtype=np.uint8)
    vc = rng.integers(0, 256, (pages, HKV, PAGE, D // 2), dtype=np.uint8)
    ks = rng.integers(125, 130, (pages, HKV, PAGE, D // 32)).astype(np.uint8)
    vs = rng.integers(125, 130, (pages, HKV, PAGE, D // 32)).astype(np.uint8)
    bt = rng.permutation(pages).astype(np.int32).reshape(B, npg)
    qb = O.bf16_bits(0.3 * rng.standard_normal((B, K, HQ, D)).astype(np.float32))
    ref = O.reference(qb, kc, ks, vc, vs, bt, sl)
    q = dev(qb.view(np.int16), torch.bfloat16)
    mx = np.abs(ref).max()
    for nsplit in (None, 1, 2):
        out = uq_cuda.uq_decode_cuda(q, dev(kc), dev(ks), dev(vc), dev(vs), dev(bt), dev(sl), nsplit=nsplit)
        assert uq_cuda.last_status() == (0, 0, 0, 0) and uq_cuda.last_path() == 2
        check_close(out.float().cpu().numpy() / mx, ref / mx, f"B={B} HKV={HKV} nsplit={nsplit}")


def test_late_outliers_take_the_second_pass():
    """Keys whose scores (and V scales) dwarf those of a segment's first tile arrive late in every sequence: the quick path
    marks the segment and the careful pass redoes it; outputs follow the oracle on the same bytes."""
    c = [x for x in CASES if x.name == "ref_cuda_main_K8"][0]
    ks, vs = c.ks.copy(), c.vs.copy()
    for b in range(c.B):
        npg = -(-int(c.sl[b]) // c.PAGE)
        first, late = c.bt[b, : max(1, 128 // c.PAGE)], c.bt[b, npg // 2]
        ks[first] = (ks[first].astype(np.int32) - 10).clip(0, 255).astype(np.uint8)
        ks[late] = (ks[late].astype(np.int32) + 3).clip(0, 255).astype(np.uint8)
        vs[late] = (vs[late].astype(np.int32) + 5).clip(0, 255).astype(np.uint8)
    ref = O.reference(c.q, c.kc, ks, c.vc, vs, c.bt, c.sl, c.sm_scale)
    q = dev(c.q.view(np.int16), torch.bfloat16)
    for nsplit in (1, 4):
        out = uq_cuda.uq_decode_cuda(q, dev(c.kc), dev(ks), dev(c.vc), dev(vs), dev(c.bt), dev(c.sl), nsplit=nsplit)
        assert uq_cuda.last_status() == (0, 0, 0, 0)
        mx = np.abs(ref).max()
        check_close(out.float().cpu().numpy() / mx, ref / mx, f"late outliers nsplit={nsplit}")


def test_repeated_calls_are_bitwise_identical():
    """No result depends on which warp or CTA got somewhere first: the same call gives the same bits."""
    c = [x for x in CASES if x.name == "ref_cuda_main_K8"][0]
    q = dev(c.q.view(np.int16), torch.bfloat16)
    args = (dev(c.kc), dev(c.ks), dev(c.vc), dev(c.vs), dev(c.bt), dev(c.sl))
    outs = [uq_cuda.uq_decode_cuda(q, *args, nsplit=4).clone() for _ in range(6)]
    assert all(torch.equal(outs[0], o) for o in outs[1:])


def test_unserved_shapes_answer_invalid_value_before_any_work():
    c = [x for x in CASES if x.name == "ref_cuda_main_K1"][0]
    q = dev(c.q.view(np.int16), torch.bfloat16)
    args = (dev(c.kc), dev(c.ks), dev(c.vc), dev(c.vs), dev(c.bt), dev(c.sl))
    with pytest.raises(RuntimeError, match="InvalidValue"):
        uq_cuda.uq_decode_cuda(q, *args, fmt=2)
    with pytest.raises(RuntimeError, match="scale"):   # an NVFP4 call needs D/16 scale bytes per row
        uq_cuda.uq_decode_cuda(q, *args, fmt=1)
    with pytest.raises(RuntimeError, match="InvalidValue"):
        uq_cuda.uq_decode_cuda(q, *args, nsplit=129)
    with pytest.raises(RuntimeError, match="InvalidValue"):
        uq_cuda.uq_decode_cuda(q, *args, nsplit=0)
    with pytest.raises(RuntimeError, match="bf16"):
        uq_cuda.uq_decode_cuda(q.float(), *args)
    # the tuning hints of the reference's kernels are accepted and ignored
    out = uq_cuda.uq_decode_cuda(q, *args, variant=4, mb=2, nwarps=8, stages=4)
    check_close(out.float().cpu().numpy(), c.ref, "hints")


@pytest.mark.parametrize("R", [2, 4, 8])
def test_context_split_partials_merge_to_the_unsplit_answer(R):
    c = [x for x in CASES if x.name == "gen_d256_K8"][0]
    q = dev(c.q.view(np.int16), torch.bfloat16)
    per = -(-c.max_pages // R)
    os_, ls_ = [], []
    for r in range(R):
        lo, hi = min(r * per, c.max_pages), min((r + 1) * per, c.max_pages)
        bt = np.zeros((c.B, max(per, 1)), np.int32)
        bt[:, : hi - lo] = c.bt[:, lo:hi]
        off = np.full(c.B, lo * c.PAGE, np.int32)
        o, l = uq_cuda.uq_decode_partial(q, dev(c.kc), dev(c.ks), dev(c.vc), dev(c.vs), dev(bt), dev(c.sl), dev(off))
        # each shard's partial against the oracle's partial on the same shard
        nloc = np.clip(c.sl - lo * c.PAGE, 0, (hi - lo) * c.PAGE).astype(np.int32)
        ro, rl = O.reference(c.q, c.kc, c.ks, c.vc, c.vs, bt, c.sl, pos_offset=off, n_local=nloc, return_lse=True)
        check_close(o.cpu().numpy(), ro, f"shard {r} o")
        lse = l.cpu().numpy() * np.log(2.0)
        fin = np.isfinite(rl)
        assert np.array_equal(np.isfinite(lse), fin)
        assert np.abs(lse[fin] - rl[fin]).max(initial=0) <= 2e-3
        os_.append(o)
        ls_.append(l)
    out = uq_cuda.uq_merge(torch.stack(os_), torch.stack(ls_))
    check_close(out.float().cpu().numpy(), c.ref, f"merge R={R}")
    # the packed form (what one all-gather of per-rank buffers gives): same shards, same bits
    B, K, HQ, D = q.shape
    n = B * K * HQ * (D + 1)
    packed = torch.empty(R, n, dtype=torch.float32, device="cuda")
    for r in range(R):
        lo, hi = min(r * per, c.max_pages), min((r + 1) * per, c.max_pages)
        bt = np.zeros((c.B, max(per, 1)), np.int32)
        bt[:, : hi - lo] = c.bt[:, lo:hi]
        off = np.full(c.B, lo * c.PAGE, np.int32)
        uq_cuda.uq_decode_partial(q, dev(c.kc), dev(c.ks), dev(c.vc), dev(c.vs), dev(bt), dev(c.sl), dev(off), into=packed[r])
    out2 = uq_cuda.uq_merge_packed(packed, B * K * HQ, D, torch.empty_like(q))
    assert torch.equal(out2, out)


def test_a_wait_that_runs_out_is_reported_and_the_next_call_is_unaffected(monkeypatch):
    """The give-up path of the tcgen05 kernel on a healthy GPU: with UQ_B200_CFG=expire=30 the softmax role never announces a
    segment's query tile (an arrival that nothing makes), so the issuing thread's wait for it - barrier id 30, bounded at one
    second like every wait of the kernel - runs out.  The kernel must return (every role drains to the common exit, the copy
    warps wait for their copies in flight, TMEM goes back), the status record must name a wait that ran out (code 1; the
    issuing thread's, or the softmax role's own wait for scores that were never computed, ids 62-64, whichever CTA reports
    first), and the next ordinary calls on the device must be right."""
    c = [x for x in CASES if x.name == "gen_cfg0_K4"][0]
    q = dev(c.q.view(np.int16), torch.bfloat16)
    args = (dev(c.kc), dev(c.ks), dev(c.vc), dev(c.vs), dev(c.bt), dev(c.sl))
    monkeypatch.setenv("UQ_B200_CFG", "path=tc,expire=30")
    bad = uq_cuda.uq_decode_cuda(q, *args)     # not an answer: the combine writes NaN rows while the status code is set
    assert torch.isnan(bad.float()).all()
    st = uq_cuda.last_status()
    assert st[0] == 1 and st[2] in (30, 62, 63, 64), st
    monkeypatch.delenv("UQ_B200_CFG")
    for _ in range(2):
        out = uq_cuda.uq_decode_cuda(q, *args)
        assert uq_cuda.last_status() == (0, 0, 0, 0) and uq_cuda.last_path() == 2
        check_close(out.float().cpu().numpy(), c.ref, "call after a wait that ran out")


@pytest.mark.parametrize("mode", ["together", "graph"])
@pytest.mark.parametrize("chain,fmt,ctx,K", [("append verify", 0, 900, 2), ("append verify", 1, 900, 2), ("append rotate verify", 0, 900, 2), ("append append verify", 0, 900, 2),
                                             ("verify verify", 0, 900, 8), ("append verify", 0, 9000, 1), ("append rotate verify", 0, 300, 16)])
def test_a_chain_of_calls_needs_no_synchronisation(chain, fmt, ctx, K, mode):
    """Every kernel is set up while the one before it on the stream still runs and waits for it before it touches memory.  Calls that
    write what the next one reads - cache, queries, scratch - follow each other with nothing of torch's in between, eagerly and replayed
    from a graph, and give the bits of the same calls run apart.  Every step rewrites the whole cache with other tokens (from 9000 per
    sequence on in several thousand blocks of the bulk kernel), so that anything read too early is another step's."""
    B, HQ, HKV, D, PAGE, steps = 4, 16, 4, 128, 64, 4 if ctx > 4000 else 10
    g = torch.Generator(device="cuda").manual_seed(5)
    npg = -(-ctx // PAGE)
    bt = torch.randperm(B * npg, generator=g, device="cuda").to(torch.int32).view(B, npg)
    pos = torch.arange(ctx, device="cuda").repeat(B)
    slots = bt.long().repeat_interleave(ctx, 0)[torch.arange(B * ctx, device="cuda"), pos // PAGE] * PAGE + pos % PAGE
    sl = torch.full((B,), ctx, dtype=torch.int32, device="cuda")
    key, value = ([torch.randn(B * ctx, HKV, D, generator=g, device="cuda").bfloat16() for _ in range(steps)] for _ in range(2))
    q = [torch.randn(B, K, HQ, D, generator=g, device="cuda").bfloat16() for _ in range(steps)]
    cache = [torch.zeros(B * npg, HKV, PAGE, w, dtype=torch.uint8, device="cuda") for w in (D // 2, D // (16 if fmt else 32)) * 2]
    ws = torch.empty(uq_cuda.workspace_floats(B, K, HQ, HKV, D, 8), device="cuda")
    rot, outs = torch.empty_like(q[0]), [torch.empty_like(q[0]) for _ in range(2 * steps)]
    ts = dict(fmt=1, k_ts=0.01, v_ts=0.01) if fmt else {}

    def append(k, v, rotate):
        if fmt:
            uq_cuda.append_kv_nvfp4(*cache, k, v, slots, 0.01, 0.01)
        else:
            uq_cuda.append_kv(*cache, k, v, slots, rotate_k=rotate)

    def run(after):
        for s in range(steps):
            n, last = 0, q[s]
            for what in chain.split():
                if what == "append":
                    append(key[(s + n) % steps], value[s], "rotate" in chain)
                elif what == "rotate":
                    last = uq_cuda.fwht(q[s], out=rot)
                else:
                    uq_cuda.uq_decode_cuda(last, *cache, bt, sl, nsplit=8, workspace=ws, out=outs[2 * s + n % 2], **ts)
                    last = q[(s + 1) % steps]
                n += 1
                after()

    def result(how):
        for t in (*cache, *outs, rot, ws):
            t.zero_()
        if "append" not in chain:
            append(key[0], value[0], False)
        torch.cuda.synchronize()
        how()
        torch.cuda.synchronize()
        return [t.clone() for t in (*outs, *cache)]

    def graph():
        graphs = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs):
            run(lambda: None)
        graphs.replay()

    apart = result(lambda: run(torch.cuda.synchronize))
    assert uq_cuda.last_path() == 2
    for a, b in zip(apart, result(graph if mode == "graph" else lambda: run(lambda: None))):
        assert torch.equal(a, b)
    assert any(bool(t.any()) for t in apart[:2]) and uq_cuda.last_status() == (0, 0, 0, 0)


@pytest.mark.parametrize("nsplit", [2, 3])
@pytest.mark.parametrize("B,HKV,long_ones,longest,width", [(40, 4, 3, 3000, 3000), (40, 4, 3, 3000, 40000), (150, 1, 1, 9000, 9000), (33, 8, 33, 1500, 1500), (3, 1, 3, 20000, 20000)])
def test_items_cut_into_no_more_pieces_than_they_have_slots(B, HKV, long_ones, longest, width, nsplit):
    """Few partial slots and lengths far apart: the CTAs' equal share would cut the long items into more pieces than there are
    slots, so a larger chunk is chosen (the smallest of a row of candidates that fits, or the one that always does).  The
    scratch is exactly nsplit slots; a guard behind it stays untouched.  `width`: a page table far wider than the sequences."""
    rng = np.random.default_rng(B + HKV)
    K, G, D, PAGE = 2, 2, 64, 64
    sl = rng.integers(1, 200, B).astype(np.int32)
    sl[rng.permutation(B)[:long_ones]] = longest - rng.integers(0, 100, long_ones)
    npg = -(-sl // PAGE)
    pages = int(npg.sum())
    kc, ks = O.quantize_fp4(rng.standard_normal((pages, HKV, PAGE, D)).astype(np.float32))
    vc, vs = O.quantize_fp4(rng.standard_normal((pages, HKV, PAGE, D)).astype(np.float32))
    bt = np.zeros((B, -(-width // PAGE)), np.int32)
    perm, at = rng.permutation(pages).astype(np.int32), 0
    for b in range(B):
        bt[b, :npg[b]] = perm[at:at + npg[b]]
        at += npg[b]
    qb = O.bf16_bits(rng.standard_normal((B, K, HKV * G, D)).astype(np.float32))
    n = uq_cuda.workspace_floats(B, K, HKV * G, HKV, D, nsplit)
    ws = torch.full((n + 4096,), 7.0, device="cuda")
    out = uq_cuda.uq_decode_cuda(dev(qb.view(np.int16), torch.bfloat16), *(dev(a) for a in (kc, ks, vc, vs, bt, sl)), nsplit=nsplit, workspace=ws)
    assert uq_cuda.last_path() == 2 and uq_cuda.last_status() == (0, 0, 0, 0)
    check_close(out.float().cpu().numpy(), O.reference(qb, kc, ks, vc, vs, bt, sl), f"nsplit={nsplit}")
    assert bool((ws[n:] == 7.0).all())


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("K", [1, 4])
@pytest.mark.parametrize("PAGE", [64, 128, 256, 96])
def test_searching_launches_take_the_third_copy_warp_at_every_page_size(PAGE, K, fmt):
    """head_dim 128, up to 32 rows, few slots per item and a table wide enough for the chunk search: whole pages, 128-token parts and
    common parts of them as copy units, scale slices 16 bytes per lane; every row against its own largest."""
    rng = np.random.default_rng(PAGE + K)
    B, HKV, G, D, nsplit = 40, 4, 8, 128, 3
    sl = rng.integers(1, 300, B).astype(np.int32)
    sl[:3] = (2100, 129, 1)
    npg = -(-sl // PAGE)
    pages = int(npg.sum())
    per, kr, vr, qs = (32, (124, 128), (125, 129), 0.4) if fmt == 0 else (16, (0x28, 0x48), (0x28, 0x48), 0.3)
    kc, vc = (rng.integers(0, 256, (pages, HKV, PAGE, D // 2), dtype=np.uint8) for _ in range(2))
    ks, vs = (rng.integers(*r, (pages, HKV, PAGE, D // per)).astype(np.uint8) for r in (kr, vr))
    bt, perm, at = np.zeros((B, -(-3000 // PAGE)), np.int32), rng.permutation(pages).astype(np.int32), 0
    for b in range(B):
        bt[b, :npg[b]] = perm[at:at + npg[b]]
        at += npg[b]
    qb = O.bf16_bits(qs * rng.standard_normal((B, K, HKV * G, D)).astype(np.float32))
    ref = O.reference(qb, kc, ks, vc, vs, bt, sl) if fmt == 0 else O.reference_nvfp4(qb, kc, ks, vc, vs, bt, sl, 0.5, 0.5)
    out = uq_cuda.uq_decode_cuda(dev(qb.view(np.int16), torch.bfloat16), *(dev(a) for a in (kc, ks, vc, vs, bt, sl)), nsplit=nsplit,
                                 **(dict(fmt=1, k_ts=0.5, v_ts=0.5) if fmt else {}))
    assert uq_cuda.last_path() == 2 and uq_cuda.last_status() == (0, 0, 0, 0)
    mx = np.abs(ref).max(-1, keepdims=True)
    mx[mx == 0] = 1
    check_close(out.float().cpu().numpy() / mx, ref / mx, f"PAGE={PAGE}")


CAPTURED_CHAIN = """
import ctypes, torch
from all_quant_b200 import uq_cuda
B, K, HQ, HKV, D, PAGE, T = 2, 2, 8, 2, 64, 16, 40
dev = dict(device="cuda")
new = lambda row: torch.zeros(8, HKV, PAGE, row, dtype=torch.uint8, **dev)
uq, nv = (new(D // 2), new(D // 32), new(D // 2), new(D // 32)), (new(D // 2), new(D // 16), new(D // 2), new(D // 16))
key, slots = torch.randn(T, HKV, D, **dev).bfloat16(), torch.arange(T, **dev)
q, r, out = (torch.randn(B, K, HQ, D, **dev).bfloat16() for _ in range(3))
bt, sl = torch.arange(8, dtype=torch.int32, **dev).view(B, 4), torch.tensor([33, 7], dtype=torch.int32, **dev)
ws = torch.empty(uq_cuda.workspace_floats(B, K, HQ, HKV, D, 4), **dev)

def chain():
    for kernel in ("rows", "bulk"):
        uq_cuda.append_kv(*uq, key, key, slots, kernel=kernel)
        uq_cuda.append_kv_nvfp4(*nv, key, key, slots, 0.1, 0.1, kernel=kernel)
    uq_cuda.fwht(q, out=r)
    uq_cuda.uq_decode_cuda(r, *uq, bt, sl, nsplit=4, workspace=ws, out=out)

chain()
torch.cuda.synchronize()
cu, s, g, n = ctypes.CDLL("libcuda.so.1"), torch.cuda.Stream(), ctypes.c_void_p(), ctypes.c_size_t()
assert cu.cuStreamBeginCapture_v2(ctypes.c_void_p(s.cuda_stream), 2) == 0
with torch.cuda.stream(s):
    chain()
assert cu.cuStreamEndCapture(ctypes.c_void_p(s.cuda_stream), ctypes.byref(g)) == 0
assert cu.cuGraphGetEdges_v2(g, None, None, None, ctypes.byref(n)) == 0
ends, kind = [(ctypes.c_void_p * n.value)() for _ in range(2)], (ctypes.c_uint8 * (8 * n.value))()   # kind: 8 bytes per edge, byte 2 its type
assert cu.cuGraphGetEdges_v2(g, ends[0], ends[1], kind, ctypes.byref(n)) == 0
print("edges", n.value, "programmatic", sum(kind[8 * i + 2] == 1 for i in range(n.value)))
"""


@pytest.mark.parametrize("cfg,programmatic", [("", 6), ("pdl=0", 0)])
def test_the_switch_makes_every_launch_an_ordinary_one(cfg, programmatic):
    """Four appends, a rotation and a verify call with its combine, captured: all six edges between the seven kernels are
    programmatic, and none with the switch off (read once per process, so each side is a process of its own)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CAPTURED_CHAIN], cwd=root, env={**os.environ, "UQ_B200_CFG": cfg}, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and f"edges 6 programmatic {programmatic}" in r.stdout, r.stdout + r.stderr


def test_a_launch_that_fails_leaves_no_error_for_the_next_one():
    """Launches into a capture that has been invalidated (a synchronisation inside it) fail with the runtime's error; the next
    ones, on a healthy stream, succeed: the failed launch's error is returned once and not left for a later launch check."""
    B, K, HQ, HKV, D, PAGE, T = 2, 2, 8, 2, 64, 16, 40
    kc, ks = (torch.zeros(8, HKV, PAGE, w, dtype=torch.uint8, device="cuda") for w in (D // 2, D // 32))
    vc, vs = torch.zeros_like(kc), torch.zeros_like(ks)
    key, slots = torch.randn(T, HKV, D, device="cuda").bfloat16(), torch.arange(T, device="cuda")
    q, r, out = (torch.randn(B, K, HQ, D, device="cuda").bfloat16() for _ in range(3))
    bt, sl = torch.arange(8, dtype=torch.int32, device="cuda").view(B, 4), torch.tensor([33, 7], dtype=torch.int32, device="cuda")
    ws = torch.empty(uq_cuda.workspace_floats(B, K, HQ, HKV, D, 4), device="cuda")
    o1, l1, m1 = torch.randn(2, B, K, HQ, D, device="cuda"), torch.randn(2, B, K, HQ, device="cuda"), torch.empty_like(q)
    calls = [lambda: uq_cuda.uq_decode_cuda(q, kc, ks, vc, vs, bt, sl, nsplit=4, workspace=ws, out=out), lambda: uq_cuda.fwht(q, out=r),
             lambda: uq_cuda.append_kv(kc, ks, vc, vs, key, key, slots, kernel="rows"), lambda: uq_cuda.append_kv(kc, ks, vc, vs, key, key, slots, kernel="bulk")]
    after = calls + [lambda: uq_cuda.uq_merge(o1, l1, out=m1)]   # (the merge's launch check reads the runtime's last error)
    for call in after:
        call()
    torch.cuda.synchronize()
    cu, s, g = ctypes.CDLL("libcuda.so.1"), torch.cuda.Stream(), ctypes.c_void_p()
    handle = ctypes.c_void_p(s.cuda_stream)
    for failing in calls:
        assert cu.cuStreamBeginCapture_v2(handle, 2) == 0
        assert cu.cuStreamSynchronize(handle) != 0          # not allowed here: the capture is invalid from now on
        with torch.cuda.stream(s), pytest.raises(RuntimeError):
            failing()
        assert cu.cuStreamEndCapture(handle, ctypes.byref(g)) != 0
        for call in reversed(after):
            call()
    torch.cuda.synchronize()
    assert uq_cuda.last_status() == (0, 0, 0, 0)
