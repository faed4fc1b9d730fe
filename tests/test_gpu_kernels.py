"""sm_100a select/apply kernels against the plain-PyTorch oracle, one GPU."""
import numpy as np
import pytest
import torch

from stellatrain_b200.ops import oracle as O
from stellatrain_b200.parallel import buckets as B

pytestmark = pytest.mark.gpu

SIZES = [1, 15, 16, 17, 1000, 4096, 65535, 65536, 70001, 300000]


def make_bucket(compressor, ratio, optimizer="sgd", sizes=SIZES, chunk=4096, narrow=False, debug=False, **kw):
    from stellatrain_b200.parallel.gpu_bucket import GpuBucket

    dev = torch.device("cuda:0")
    layout = B.BucketLayout([f"t{i}" for i in range(len(sizes))], sizes, chunk_elems=chunk, narrow_wire=narrow)
    b = GpuBucket(0, layout, dev, compressor=compressor, ratio=ratio, optimizer=optimizer, **kw)
    b.wire_local(debug_checks=debug)
    return b


def seg_slices(b):
    return [(s, slice(s.off, s.off + s.numel), slice(s.off, s.off + s.n_pad)) for s in b.layout.segments]


def read_stream(b, epoch):
    idx, val = b.stream_of(epoch & 1, 0)
    return idx.cpu().numpy().view(np.uint32).astype(np.int64), val.cpu()


def oracle_states(b):
    st = b.seg_state()
    return [O.ThresholdState(float(s["tau"]), float(s["tau_inc"]), bool(s["inited"])) for s in st]


def fill_grads(b, gen, scale=1e-2, mode="normal"):
    for s, sl, _ in seg_slices(b):
        if mode == "normal":
            g = torch.randn(s.numel, generator=gen, device="cuda") * scale
        elif mode == "ties":
            g = torch.randint(-3, 4, (s.numel,), generator=gen, device="cuda").float() * scale
        elif mode == "zero":
            g = torch.zeros(s.numel, device="cuda")
        b.grad[sl] = g


@pytest.mark.parametrize("compressor", ["topk", "thresholdv", "thresholdv16"])
@pytest.mark.parametrize("mode", ["normal", "ties", "zero", "shrinking"])
@pytest.mark.parametrize("fused", [True, False])
def test_select_matches_oracle(compressor, mode, fused):
    """Bit-equal entries, residuals and thresholds against the plain-PyTorch rule, for the four-kernel chain and for the
    one-pass chain that takes over once every tensor has been through one select.  "shrinking" halves the gradient scale
    every step, so the threshold (top-k: the cut under the previous one) is far too high and the one-pass chain has to
    complete the stream from the whole tensor; "zero" leaves top-k a previous threshold of zero."""
    torch.manual_seed(0)
    gen = torch.Generator(device="cuda").manual_seed(1234)
    b = make_bucket(compressor, 0.99, fused_select=fused)
    resid_ref = torch.zeros_like(b.resid)
    steps = 3 if mode in ("ties", "zero") else 6
    for step in range(steps):
        epoch = step + 1
        if mode == "shrinking":
            fill_grads(b, gen, scale=1e-2 * 0.5 ** step)
        else:
            fill_grads(b, gen, mode=mode if not (mode == "zero" and step == 1) else "normal")
        grad = b.grad.clone()
        states = oracle_states(b)
        b.select()
        torch.cuda.synchronize()
        b.check_status()
        one_pass = fused and step > 0
        assert b.last_select_fused == one_pass
        assert float(b.grad.abs().max()) == 0.0, "consumed gradients must be zeroed"
        idx_all, val_all = read_stream(b, epoch)
        new_states = b.seg_state()
        for si, (s, sl, slp) in enumerate(seg_slices(b)):
            k = s.k
            got_idx = idx_all[s.out_off : s.out_off + k]
            got_val = val_all[s.out_off : s.out_off + k]
            st = states[si]
            pad = compressor == "thresholdv16"
            g = grad[slp] if pad else grad[sl]
            r = resid_ref[slp] if pad else resid_ref[sl]
            want_idx, want_val, new_r = O.compress_step(compressor, g, r, k, st, one_pass=one_pass)
            want_idx = want_idx.cpu().numpy() + s.off
            valid = got_idx != O.SENTINEL
            order_g = np.argsort(got_idx[valid], kind="stable")
            order_w = np.argsort(want_idx, kind="stable")
            assert np.array_equal(got_idx[valid][order_g], want_idx[order_w]), (compressor, mode, step, s.name)
            assert torch.equal(got_val[torch.from_numpy(valid)][torch.from_numpy(order_g)],
                               want_val.cpu()[torch.from_numpy(order_w)])
            if pad:
                resid_ref[slp] = new_r
            else:
                resid_ref[sl] = new_r
            if compressor != "topk":
                assert bool(new_states[si]["inited"])
                assert new_states[si]["tau"] == pytest.approx(st.tau, rel=1e-5, abs=1e-30)
        assert torch.equal(b.resid, resid_ref), (compressor, mode, step)


@pytest.mark.parametrize("compressor", ["topk", "thresholdv", "thresholdv16"])
@pytest.mark.parametrize("mode", ["steady", "jumps", "ties", "mostly_zero", "huge"])
@pytest.mark.parametrize("ratio,chunk,narrow,piece_runs", [(0.99, 8192, False, 8), (0.5, 1024, False, 32), (0.999, 1 << 18, False, 128),
                                                           (0.5, 8192, False, 128), (0.99, 8192, True, 128), (0.5, 1024, True, 8)])
def test_one_pass_select_at_its_edges(compressor, mode, ratio, chunk, narrow, piece_runs, monkeypatch):
    """The one-pass chain against the plain rule at the edges of its runs (1024 elements), pieces (of the named number of runs) and chunks:
    the same entries bit for bit.  "jumps" moves the gradient scale up and down by large factors, so that top-k's
    candidates fall short and the refill kernel selects; "mostly_zero" leaves fewer entries than the budget; "huge"
    holds values far outside the histogram window.  ``narrow``: tensors of fewer than 65536 elements send bf16 values and keep
    the rounding error."""
    sizes = [1, 16, 1023, 1024, 1025, 8192, 9001, 32769, 65519, 131071, 131072, 131073, 400001]
    monkeypatch.setattr(B, "MIN_PIECE_RUNS", piece_runs)
    monkeypatch.setattr(B, "MAX_PIECE_RUNS", piece_runs)
    gen = torch.Generator(device="cuda").manual_seed(99)
    b = make_bucket(compressor, ratio, sizes=sizes, chunk=chunk, narrow=narrow)
    resid_ref = torch.zeros_like(b.resid)
    for step in range(7):
        scale = [1.0, 1.0, 0.02, 0.02, 50.0, 0.5, 0.4][step] if mode == "jumps" else 1.0
        fill_grads(b, gen, scale=1e-2 * scale, mode="ties" if mode == "ties" else "normal")
        for s, sl, _ in seg_slices(b):
            if mode == "mostly_zero":
                b.grad[sl] *= (torch.rand(s.numel, generator=gen, device="cuda") < 0.2 * (1 - ratio)).float()
            if mode == "huge" and step in (1, 4):
                b.grad[s.off + s.numel // 2] = 1e30
        grad, states = b.grad.clone(), oracle_states(b)
        b.select()
        torch.cuda.synchronize()
        b.check_status()
        assert b.last_select_fused == (step > 0)
        idx_all, val_all = read_stream(b, step + 1)
        for si, (s, sl, slp) in enumerate(seg_slices(b)):
            own = slp if compressor == "thresholdv16" else sl
            # top-k of a tensor with fewer entries than the budget sends zeros, lowest index first
            want_idx, want_val, new_r = O.compress_step(compressor, grad[own], resid_ref[own], s.k, states[si], one_pass=step > 0)
            if b.layout.is_narrow(s):
                sent = want_val.bfloat16().float()
                new_r[want_idx] = want_val - sent
                want_val = sent
            got = torch.from_numpy(idx_all[s.out_off : s.out_off + s.k])
            valid = got != O.SENTINEL
            got, order = got[valid].sort()
            want, worder = (want_idx.cpu() + s.off).sort()
            assert torch.equal(got, want), (s.numel, step)
            assert torch.equal(val_all[s.out_off : s.out_off + s.k][valid][order], want_val.cpu()[worder]), (s.numel, step)
            resid_ref[own] = new_r
            if compressor != "topk":
                assert b.seg_state()[si]["tau"] == pytest.approx(states[si].tau, rel=1e-5, abs=1e-30)
        assert torch.equal(b.resid, resid_ref), step
    # the chain leaves its counters as it found them
    assert int(b.hist.abs().max()) == 0 and int(b.hist_top.abs().max()) == 0 and int(b.hist_rest.abs().max()) == 0 and int(b.piece_cnt.abs().max()) == 0
    work = b.work.view(len(sizes), B.SEG_WORK_WORDS)
    assert int(work[:, 4:6].abs().max()) == 0 and int(work[:, 10:].abs().max()) == 0 and int(b.counters[4]) == 0


@pytest.mark.parametrize("compressor", ["thresholdv", "thresholdv16"])
@pytest.mark.parametrize("where", ["everywhere", "one piece", "first piece"])
@pytest.mark.parametrize("over", [0.7, 1.1, 3.0])
def test_items_over_the_threshold_in_all_pieces_or_in_one(compressor, where, over):
    """A CTA sends the listed items of its own piece unless one piece holds most of them; then the positions are shared out.
    ``over``: items over the threshold, as a multiple of the budget."""
    n, ratio = 3_000_003, 0.97
    b = make_bucket(compressor, ratio, sizes=[n, 70_001], chunk=8192)
    assert b.n_pieces > 20
    gen = torch.Generator(device="cuda").manual_seed(5)
    resid_ref = torch.zeros_like(b.resid)
    per_piece = b.layout.piece_runs * B.RUN_ELEMS
    for step in range(3):
        fill_grads(b, gen)
        if where != "everywhere":
            at = per_piece * (0 if where == "first piece" else 7)
            b.grad[at : at + per_piece] *= 1000.0
        grad = b.grad.clone()
        if step > 0:        # a threshold that lets so many pass
            block = compressor == "thresholdv16"
            state = b.seg_state()
            for si, (s, _, slp) in enumerate(seg_slices(b)):
                key = (grad[slp] + b.resid[slp]).abs()
                key = key.view(-1, 16).sum(1) if block else key
                state["tau"][si] = float(key.sort(descending=True).values[int(over * (s.k // 16 if block else s.k))])
            b.state.copy_(torch.from_numpy(state.view(np.uint8).reshape(-1)))
        states = oracle_states(b)
        b.select()
        torch.cuda.synchronize()
        b.check_status()
        idx_all, val_all = read_stream(b, step + 1)
        for si, (s, sl, slp) in enumerate(seg_slices(b)):
            own = slp if compressor == "thresholdv16" else sl
            want_idx, want_val, new_r = O.compress_step(compressor, grad[own], resid_ref[own], s.k, states[si], one_pass=step > 0)
            got = torch.from_numpy(idx_all[s.out_off : s.out_off + s.k])
            valid = got != O.SENTINEL
            got, order = got[valid].sort()
            want, worder = (want_idx.cpu() + s.off).sort()
            assert torch.equal(got, want), (s.numel, step)
            assert torch.equal(val_all[s.out_off : s.out_off + s.k][valid][order], want_val.cpu()[worder]), (s.numel, step)
            resid_ref[own] = new_r
        assert torch.equal(b.resid, resid_ref), step


def set_seg_state(b, **fields):
    state = b.seg_state()
    for k, v in fields.items():
        state[k] = v
    b.state.copy_(torch.from_numpy(state.view(np.uint8).reshape(-1)))


@pytest.mark.parametrize("tau", [-0.5, -0.0, float("nan"), float("inf")])
def test_a_block_threshold_that_no_block_reaches(tau):
    """A restored threshold may be anything.  One that no block reaches, also by its sign bit, leaves the whole stream to the
    fill: the best blocks of the tensor, few (searched in shared memory) or many."""
    sizes = [1000, 30_000, 70_001]
    b = make_bucket("thresholdv16", 0.97, sizes=sizes)
    gen = torch.Generator(device="cuda").manual_seed(8)
    for step in range(4):
        fill_grads(b, gen)
        if step >= 2:
            set_seg_state(b, tau=np.float32(tau))
        a = b.grad + b.resid
        b.select()
        torch.cuda.synchronize()
        b.check_status()
        if step < 2:
            continue
        idx, val = read_stream(b, step + 1)
        for s, _, slp in seg_slices(b):
            key = a[slp].view(-1, 4).abs()
            key = ((key[:, 0] + key[:, 1]) + (key[:, 2] + key[:, 3])).view(-1, 4)
            key = (key[:, 0] + key[:, 1]) + (key[:, 2] + key[:, 3])
            blocks = key.sort(descending=True, stable=True).indices[: (s.k + 15) // 16]
            want = (blocks[:, None] * 16 + torch.arange(16, device="cuda")).reshape(-1)[: s.k] + s.off      # the last one is cut off
            got = torch.from_numpy(idx[s.out_off : s.out_off + s.k])
            assert torch.equal(got.sort().values, want.cpu().sort().values), (s.numel, step)
            assert torch.equal(val[s.out_off : s.out_off + s.k], a[got.cuda()].cpu())
            left = a[slp].clone()
            left[want - s.off] = 0.0
            assert torch.equal(b.resid[slp], left)


@pytest.mark.parametrize("threshold", [-0.5, -0.0, float("nan"), float("inf")])
def test_an_element_threshold_that_no_element_reaches(threshold):
    """The same for elements: threshold-v then sends nothing and keeps everything, top-k (whose state is its previous k-th
    largest value) finds its entries in the whole tensor."""
    sizes = [1000, 30_000, 300_000]
    v, top = make_bucket("thresholdv", 0.97, sizes=sizes), make_bucket("topk", 0.97, sizes=sizes)
    gen = torch.Generator(device="cuda").manual_seed(10)
    for step in range(4):
        for b in (v, top):
            fill_grads(b, gen)
        if step >= 2:
            set_seg_state(v, tau=np.float32(threshold))
            set_seg_state(top, r1=np.float32(threshold).view(np.uint32))
        a_v, a_top = v.grad + v.resid, top.grad + top.resid
        for b in (v, top):
            b.select()
            torch.cuda.synchronize()
            b.check_status()
        if step < 2:
            continue
        idx, _ = read_stream(v, step + 1)
        assert np.all(idx == O.SENTINEL) and torch.equal(v.resid, a_v)
        idx, val = read_stream(top, step + 1)
        for s, sl, slp in seg_slices(top):
            want = a_top[sl].abs().sort(descending=True, stable=True).indices[: s.k] + s.off
            got = torch.from_numpy(idx[s.out_off : s.out_off + s.k])
            assert torch.equal(got.sort().values, want.cpu().sort().values), (s.numel, step)
            assert torch.equal(val[s.out_off : s.out_off + s.k], a_top[got.cuda()].cpu())
            left = a_top[slp].clone()
            left[want - s.off] = 0.0
            assert torch.equal(top.resid[slp], left)


def test_a_fill_whose_candidates_are_not_there_is_reported():
    """The fill's candidates and their count come from counters that every select leaves at zero.  Were they ever wrong, the
    search for the cut must end: with an error, and nothing stored past it."""
    n, ratio = 300_000, 0.99
    b = make_bucket("thresholdv16", ratio, sizes=[n], chunk=8192)
    assert b.n_pieces > 1
    gen = torch.Generator(device="cuda").manual_seed(9)
    for _ in range(2):
        fill_grads(b, gen)
        b.select()
    torch.cuda.synchronize()
    b.check_status()
    # as many blocks with something in them as the budget has: the fill wants every candidate
    wanted = (b.layout.segments[0].k + 15) // 16
    b.resid.zero_()
    b.grad.zero_()
    b.grad.view(-1)[: wanted * 96 : 96] = 1.0
    set_seg_state(b, tau=np.float32(1e30), r0=np.float32(1.0).view(np.uint32))
    lists = b.scratch.buf.view(-1, 2)
    first = b.layout.n_total // 16
    lists[first : first + 5] = torch.tensor([0, 0x7F000000], dtype=torch.int32, device="cuda")      # five leftovers over the threshold
    b.work.view(1, B.SEG_WORK_WORDS)[0, 4] = 5                                                       # in front of the candidates
    b.select()
    torch.cuda.synchronize()
    assert int(b.status.item()) == 4


@pytest.mark.parametrize("compressor", ["topk", "thresholdv", "thresholdv16"])
def test_a_ratio_change_cuts_the_bucket_anew(compressor):
    """More entries want smaller pieces; thresholds and residuals stay."""
    b = make_bucket(compressor, 0.995, sizes=[70001, 17_000_003], chunk=8192, min_ratio=0.9)
    gen, resid_ref = torch.Generator(device="cuda").manual_seed(6), torch.zeros_like(b.resid)
    cuts = []
    for step, ratio in enumerate([0.995, 0.995, 0.9, 0.9, 0.97]):
        if ratio != b.ratio:
            b.set_ratio(ratio)
        cuts.append(b.n_pieces)
        fill_grads(b, gen)
        grad, states = b.grad.clone(), oracle_states(b)
        b.select()
        torch.cuda.synchronize()
        b.check_status()
        idx_all, _ = b.stream_of((step + 1) & 1, 0)
        for si, (s, sl, slp) in enumerate(seg_slices(b)):
            own = slp if compressor == "thresholdv16" else sl
            want, _, new_r = O.compress_step(compressor, grad[own], resid_ref[own], s.k, states[si], one_pass=step > 0)
            got = idx_all[s.out_off : s.out_off + s.k]
            assert torch.equal(got[got != -1].long().sort().values, want.sort().values + s.off), (step, s.name)
            resid_ref[own] = new_r
        assert torch.equal(b.resid, resid_ref), step
    assert cuts[0] == cuts[1] < cuts[4] < cuts[2] == cuts[3]


@pytest.mark.parametrize("compressor", ["topk", "thresholdv", "thresholdv16", "randomk"])
@pytest.mark.parametrize("n", [17, 1000, 4097, 131089])
@pytest.mark.parametrize("form", ["plain", "unaligned", "strided"])
def test_compress_reads_the_tensor_in_place(compressor, n, form):
    """Single-tensor compression takes the caller's tensor as the gradient of a bucket without a residual: the pairs of the
    plain rule, for aligned, unaligned and strided tensors, a ratio that changes from call to call, and NaNs dropped."""
    import stellatrain_b200 as st

    gen = torch.Generator(device="cuda").manual_seed(n)
    name, state = f"{compressor} {n} {form}", O.ThresholdState()
    st.configure_compression(compressor)
    try:
        for call in range(5):
            store = torch.randn(2 * n + 1, generator=gen, device="cuda") * 1e-2
            store[5] = float("nan")
            x = {"plain": store[:n], "unaligned": store[1 : n + 1], "strided": store[: 2 * n : 2]}[form]
            before = store.clone()
            ratio = 0.9 if call < 3 else 0.75
            k = int((1.0 - ratio) * n)
            idx, val = st.compress(name, x, ratio)
            assert torch.equal(store.nan_to_num(7.0), before.nan_to_num(7.0)) and idx.dtype == torch.int32
            x = x.nan_to_num(0.0)
            assert torch.equal(val, x[idx.long()]) and len(torch.unique(idx)) == len(idx)
            if compressor == "randomk":
                assert len(idx) == k
                continue
            want, _, _ = O.compress_step(compressor, x, torch.zeros_like(x), k, state, one_pass=call > 0)
            want = want[want < n].sort().values
            assert torch.equal(idx.long().sort().values, want), call
    finally:
        st.configure_compression("thresholdv16")


@pytest.mark.parametrize("compressor", ["topk", "thresholdv", "thresholdv16"])
@pytest.mark.parametrize("n", [4095, 400_003])
def test_compress_of_values_that_change_in_scale(compressor, n):
    """The ways of the chain that read the tensor once more (too few candidates, the fill from all blocks), at its ragged end and
    with NaN in it: the pairs of the plain rule, and the tensor as it was."""
    import stellatrain_b200 as st

    gen = torch.Generator(device="cuda").manual_seed(n)
    name, state = f"{compressor} {n} scales", O.ThresholdState()
    st.configure_compression(compressor)
    try:
        for call, scale in enumerate([1.0, 1.0, 0.01, 0.01, 30.0, 0.2, 0.0]):
            x = torch.randn(n, generator=gen, device="cuda") * (1e-2 * scale)
            if call == 5:
                x[: n - 100] = 0.0
            x[n - 2] = float("nan")
            before = x.clone()
            idx, val = st.compress(name, x, 0.97)
            assert torch.equal(x.nan_to_num(7.0), before.nan_to_num(7.0))
            x = x.nan_to_num(0.0)
            assert torch.equal(val, x[idx.long()]) and len(torch.unique(idx)) == len(idx)
            want, _, _ = O.compress_step(compressor, x, torch.zeros_like(x), int((1.0 - 0.97) * n), state, one_pass=call > 0)
            want = want[want < n].sort().values
            assert torch.equal(idx.long().sort().values, want), call
    finally:
        st.configure_compression("thresholdv16")


@pytest.mark.parametrize("compressor", ["topk", "thresholdv", "thresholdv16"])
@pytest.mark.parametrize("n", [2, 3, 6, 16_385, 16_386, 140_001, 140_002])
def test_compress_reads_the_last_elements_however_many_there_are(compressor, n):
    """A tensor in place is read four elements at a time, and its end by itself: tensors shorter than that, and one or two
    elements behind the last four, which are the largest of all, on the ways that read the tensor once more."""
    import stellatrain_b200 as st

    gen = torch.Generator(device="cuda").manual_seed(n)
    name, state = f"{compressor} {n} end", O.ThresholdState()
    st.configure_compression(compressor)
    try:
        for call, scale in enumerate([1.0, 1.0, 0.01, 30.0, 0.2]):
            x = torch.randn(n, generator=gen, device="cuda") * (1e-2 * scale)
            x[-2:] = 5e-2 * scale
            k = max(1, int((1.0 - 0.9) * n)) if n > 16 else n // 2
            idx, val = st.compress(name, x, 0.9 if n > 16 else 0.5)
            assert torch.equal(val, x[idx.long()]) and len(torch.unique(idx)) == len(idx)
            want, _, _ = O.compress_step(compressor, x, torch.zeros_like(x), k, state, one_pass=call > 0)
            want = want[want < n].sort().values
            assert torch.equal(idx.long().sort().values, want), call
    finally:
        st.configure_compression("thresholdv16")


@pytest.mark.parametrize("compressor", ["topk", "thresholdv", "thresholdv16"])
def test_compress_under_capture_is_refused_and_leaves_no_trace(compressor):
    """The refused call must not count as the tensor's first select, which is the one that measures the threshold."""
    import stellatrain_b200 as st

    n, name = 5000, f"captured {compressor}"
    gen, state = torch.Generator(device="cuda").manual_seed(2), O.ThresholdState()
    st.configure_compression(compressor)
    try:
        for call in range(4):
            x = torch.randn(n, generator=gen, device="cuda")
            if call in (0, 2):
                with pytest.raises(RuntimeError, match="captured"), torch.cuda.graph(torch.cuda.CUDAGraph()):
                    st.compress(name, x, 0.9)
            idx, val = st.compress(name, x, 0.9)
            want, _, _ = O.compress_step(compressor, x, torch.zeros_like(x), int((1 - 0.9) * n), state, one_pass=call > 0)
            assert torch.equal(idx.long().sort().values, want[want < n].sort().values), call
            assert torch.equal(val, x[idx.long()])
    finally:
        st.configure_compression("thresholdv16")


def test_select_drops_nan():
    b = make_bucket("topk", 0.9, sizes=[1000, 5000])
    g = torch.randn(b.layout.n_total, device="cuda")
    g[3] = float("nan")
    g[1500] = float("nan")
    b.grad.copy_(g)
    # padding must stay zero
    for s, sl, slp in seg_slices(b):
        b.grad[s.off + s.numel : s.off + s.n_pad] = 0
    b.select()
    torch.cuda.synchronize()
    b.check_status()
    assert not torch.isnan(b.resid).any()
    idx, val = read_stream(b, 1)
    assert 3 not in idx and 1500 not in idx
    assert not torch.isnan(val).any()


@pytest.mark.parametrize("optimizer", ["sgd", "adam"])
def test_apply_matches_oracle(optimizer):
    gen = torch.Generator(device="cuda").manual_seed(7)
    b = make_bucket("topk", 0.95, optimizer=optimizer)
    if optimizer == "sgd":
        b.set_optimizer_options(lr=0.1, momentum=0.9, weight_decay=1e-4)
        cfg, st = O.SGDConfig(lr=0.1, momentum=0.9, weight_decay=1e-4), O.SGDState()
    else:
        b.set_optimizer_options(lr=1e-3, weight_decay=1e-2)
        cfg, st = O.AdamConfig(lr=1e-3, weight_decay=1e-2), O.AdamState()
    b.param.copy_(torch.randn(b.layout.n_total, generator=gen, device="cuda"))
    p_ref = b.param.clone()
    for step in range(4):
        epoch = step + 1
        fill_grads(b, gen)
        b.select()
        b.apply()
        torch.cuda.synchronize()
        b.check_status()
        idx, val = read_stream(b, epoch)
        g, touched = O.merge_streams(b.layout.n_total, [(torch.from_numpy(idx).cuda(), val.cuda())], [1.0])
        if optimizer == "sgd":
            O.sparse_sgd(p_ref, g, touched, cfg, st)
        else:
            O.sparse_adam(p_ref, g, touched, cfg, st)
        torch.testing.assert_close(b.param, p_ref, rtol=2e-5, atol=1e-6)
        assert float(b.acc.abs().max()) == 0.0, "accumulator must be clean after apply"
    if optimizer == "sgd":
        torch.testing.assert_close(b.m, st.b, rtol=2e-5, atol=1e-7)
    else:
        torch.testing.assert_close(b.m, st.m, rtol=2e-5, atol=1e-7)
        torch.testing.assert_close(b.v, st.v, rtol=2e-5, atol=1e-10)


def test_apply_options_nesterov_smart_amsgrad():
    gen = torch.Generator(device="cuda").manual_seed(11)
    b = make_bucket("topk", 0.9, optimizer="sgd", sizes=[5000, 33], smart_momentum=True)
    b.set_optimizer_options(lr=0.05, momentum=0.8, nesterov=1, dampening=0.1)
    cfg, st = O.SGDConfig(lr=0.05, momentum=0.8, nesterov=True, dampening=0.1, smart_momentum=True), O.SGDState()
    p_ref = b.param.clone()
    for step in range(4):
        fill_grads(b, gen)
        b.select(); b.apply()
        torch.cuda.synchronize()
        idx, val = read_stream(b, step + 1)
        g, touched = O.merge_streams(b.layout.n_total, [(torch.from_numpy(idx).cuda(), val.cuda())], [1.0])
        O.sparse_sgd(p_ref, g, touched, cfg, st)
        torch.testing.assert_close(b.param, p_ref, rtol=1e-4, atol=1e-6)

    b = make_bucket("topk", 0.9, optimizer="adam", sizes=[5000, 33], amsgrad=True)
    b.set_optimizer_options(lr=1e-2, maximize=1)
    cfg, st = O.AdamConfig(lr=1e-2, amsgrad=True, maximize=True), O.AdamState()
    p_ref = b.param.clone()
    for step in range(4):
        fill_grads(b, gen)
        b.select(); b.apply()
        torch.cuda.synchronize()
        idx, val = read_stream(b, step + 1)
        g, touched = O.merge_streams(b.layout.n_total, [(torch.from_numpy(idx).cuda(), val.cuda())], [1.0])
        O.sparse_adam(p_ref, g, touched, cfg, st)
        torch.testing.assert_close(b.param, p_ref, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("compressor", ["topk", "thresholdv", "thresholdv16"])
@pytest.mark.parametrize("optimizer", ["sgd", "adam"])
@pytest.mark.parametrize("narrow,infinite", [(True, False), (False, False), (False, True)])
def test_a_stream_names_an_element_once(compressor, optimizer, narrow, infinite):
    """What the single-source apply rests on.  Gradients that are dense at first and then live in a few blocks only (an
    embedding, a mostly frozen tensor) leave the near misses short of the budget, so that threshold-v16 fills its stream from
    all blocks; neither the remainders of the narrow format's rounding nor inf - inf in the residual may be sent again in the
    same stream.  Against the merging apply, which would add such entries up."""
    sizes = [5, 3000, 40000, 65000, 200000, 300001]
    pair = [make_bucket(compressor, 0.9, optimizer, sizes=sizes, chunk=8192, narrow=narrow, debug=d) for d in (False, True)]
    assert [b.apply_kernels for b in pair] == [1, 2]
    gen = torch.Generator(device="cuda").manual_seed(17)
    start = torch.randn(pair[0].layout.n_total, generator=gen, device="cuda")
    live = (torch.rand(pair[0].layout.n_total // 16, generator=gen, device="cuda") < 0.01).repeat_interleave(16)
    for b in pair:
        b.set_optimizer_options(lr=1e-2, momentum=0.9)
        b.param.copy_(start)
    for step in range(50):
        fill_grads(pair[0], gen)
        if step >= 5:
            pair[0].grad *= live
        if infinite and step in (10, 30):
            for s, _, _ in seg_slices(pair[0]):
                pair[0].grad[s.off + s.numel // 2] = float("inf")
        pair[1].grad.copy_(pair[0].grad)
        for b in pair:
            a = b.grad + b.resid
            b.select()
            idx, val = b.stream_of((step + 1) & 1, 0)
            there = idx != -1
            idx, val = idx[there].long(), val[there]
            assert len(torch.unique(idx)) == len(idx), step
            if not infinite:
                # the wire format's rounding error is a float32 value, so nothing gets lost
                assert torch.equal(b.resid.index_add(0, idx, val), a), step
            b.apply()
    for b in pair:
        torch.cuda.synchronize()
        b.check_status()
    for name in ("param", "rec", "resid"):
        torch.testing.assert_close(getattr(pair[0], name), getattr(pair[1], name), rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("optimizer,options,extra", [
    ("sgd", dict(lr=0.1, momentum=0.9, weight_decay=1e-4), {}),
    ("sgd", dict(lr=0.05, momentum=0.8, nesterov=1, dampening=0.1), dict(smart_momentum=True)),
    ("adam", dict(lr=1e-3, weight_decay=1e-2), {}),
    ("adam", dict(lr=1e-2, maximize=1), dict(amsgrad=True)),
])
@pytest.mark.parametrize("compressor,narrow", [("topk", False), ("thresholdv", True), ("randomk", False)])
@pytest.mark.parametrize("ctas", [1, 148 * 16])
def test_single_source_apply_equals_the_merging_one(optimizer, options, extra, compressor, narrow, ctas):
    """The one-kernel apply of a single source against scatter + apply (which debug checks keep): the same bits, with one
    entry per thread and with a grid that walks the stream.  Both do the same operations in the same order."""
    from stellatrain_b200.parallel.gpu_bucket import GpuBucket

    pair = []
    for debug in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(21)
        layout = B.BucketLayout([f"t{i}" for i in range(4)], [1, 300, 5000, 70001], chunk_elems=4096, narrow_wire=narrow)
        b = GpuBucket(0, layout, torch.device("cuda:0"), compressor=compressor, ratio=0.9, optimizer=optimizer, **extra)
        b.wire_local(debug_checks=debug)
        assert b.apply_kernels == (2 if debug else 1)
        b.handle.max_ctas_per_source = ctas
        b.set_optimizer_options(**options)
        b.param.copy_(torch.randn(layout.n_total, generator=gen, device="cuda"))
        for _ in range(5):
            fill_grads(b, gen)
            b.select()
            b.apply()
        b.apply()                      # nothing selected: leaves everything alone
        torch.cuda.synchronize()
        b.check_status()
        pair.append(b)
    one, two = pair
    assert torch.equal(one.param, two.param) and torch.equal(one.rec, two.rec)
    assert torch.equal(one.opt, two.opt) and torch.equal(one.counters[:4], two.counters[:4])
    for name in ("vmax", "last"):
        if getattr(one, name) is not None:
            assert torch.equal(getattr(one, name), getattr(two, name))


@pytest.mark.parametrize("compressor,n,narrow", [("topk", 378_881, False), ("topk", 3_031_039, False), ("topk", 3_031_051, False),
                                                 ("thresholdv16", 378_897, False), ("thresholdv16", 3_200_003, False),
                                                 ("thresholdv", 640_000, True)])
@pytest.mark.parametrize("ctas", [3, 148 * 16])
def test_single_source_apply_at_the_edges_of_its_grid(compressor, n, narrow, ctas):
    """More entries than one per thread on every SM (37,888): four of them a thread, and scattered ones one a thread again past
    303,104; the last CTA is not full.  The same bits as scatter + apply, which debug checks keep."""
    pair = []
    for debug in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(22)
        sizes = [n // 10] * 10 if narrow else [n]
        b = make_bucket(compressor, 0.9, "adam", sizes=sizes, chunk=8192, narrow=narrow, debug=debug)
        b.handle.max_ctas_per_source = ctas
        for _ in range(3):
            fill_grads(b, gen)
            b.select()
            b.apply()
        torch.cuda.synchronize()
        b.check_status()
        pair.append(b)
    assert torch.equal(pair[0].param, pair[1].param) and torch.equal(pair[0].rec, pair[1].rec)


@pytest.mark.parametrize("sizes,ratio", [([1, 1025, 131072, 131073, 400_001], 0.5), ([3_000_003, 17], 0.97)])
def test_randomk_positions_of_a_tensor_in_pieces(sizes, ratio):
    """The pieces of a tensor share its positions out: position j holds element (start + j stride) mod n, as one CTA wrote it."""
    b = make_bucket("randomk", ratio, sizes=sizes, chunk=8192)
    gen = torch.Generator(device="cuda").manual_seed(4)
    for step in range(2):
        fill_grads(b, gen)
        a = b.grad + b.resid
        b.select()
        torch.cuda.synchronize()
        b.check_status()
        idx, val = read_stream(b, step + 1)
        for s, _, _ in seg_slices(b):
            i = idx[s.out_off : s.out_off + s.k] - s.off
            assert (i >= 0).all() and (i < s.numel).all()
            assert s.k < 3 or (np.diff(i) % s.numel == np.diff(i)[0] % s.numel).all()
            assert torch.equal(val[s.out_off : s.out_off + s.k], a[torch.from_numpy(i + s.off).cuda()].cpu())
        a[torch.from_numpy(idx).cuda()] = 0.0
        assert torch.equal(b.resid, a)


def test_randomk_stream_is_valid():
    b = make_bucket("randomk", 0.9, sizes=[1000, 4096, 17])
    gen = torch.Generator(device="cuda").manual_seed(3)
    fill_grads(b, gen)
    grad = b.grad.clone()
    b.select()
    torch.cuda.synchronize()
    b.check_status()
    idx, val = read_stream(b, 1)
    for s, sl, _ in seg_slices(b):
        i = idx[s.out_off : s.out_off + s.k]
        assert len(np.unique(i)) == s.k
        assert (i >= s.off).all() and (i < s.off + s.numel).all()
        assert torch.equal(val[s.out_off : s.out_off + s.k], grad[torch.from_numpy(i).cuda()].cpu())
    assert float(b.resid[torch.from_numpy(idx).cuda()].abs().max()) == 0.0


def test_change_ratio_between_steps():
    gen = torch.Generator(device="cuda").manual_seed(5)
    b = make_bucket("topk", 0.99, sizes=[20000, 300], min_ratio=0.9)
    fill_grads(b, gen); b.select(); b.apply(); torch.cuda.synchronize(); b.check_status()
    cap0 = b.layout.cap
    b.set_ratio(0.9)
    assert b.layout.cap > cap0
    fill_grads(b, gen)
    a = b.grad + b.resid
    b.select(); torch.cuda.synchronize(); b.check_status()
    idx, val = read_stream(b, 2)
    s = b.layout.segments[0]
    want = O.select_topk(a[: s.numel], s.k).cpu().numpy()
    assert np.array_equal(np.sort(idx[: s.k]), np.sort(want))


def test_peer_copy_and_max_abs_diff():
    from stellatrain_b200 import _build

    C = _build.load_extension("_C")
    a = torch.randn(4096, device="cuda")
    bb = torch.empty_like(a)
    s = torch.cuda.current_stream().cuda_stream
    C.peer_copy(bb.data_ptr(), a.data_ptr(), a.numel(), s)
    out = torch.zeros(1, dtype=torch.int32, device="cuda")
    bb[17] += 0.5
    C.max_abs_diff(a.data_ptr(), bb.data_ptr(), a.numel(), out.data_ptr(), s)
    torch.cuda.synchronize()
    assert out.view(torch.float32).item() == pytest.approx(0.5, rel=1e-6)
