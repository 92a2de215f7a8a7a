"""The continuous-batching decoder step (int4 weights, paged KV cache, mixed prefill + decode)
against per-sequence execution on the CPU oracle: every sequence of a packed step must come out as
if it had been run alone through the causal forward, lm_head and greedy argmax."""
import numpy as np
import pytest

import oracle_lib as O
from gpu_util import TOL, max_rel
from logismos_b200.decoder import BlockAllocator, DecoderModel
from logismos_b200.embed import ComputeError
from stella_weights import TINY, make_weights, quantize_weights

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup():
    w = make_weights(TINY, 77)
    qw, deq = quantize_weights(TINY, w)
    oracle = O.OracleStella(TINY, deq)
    return qw, deq, oracle


def oracle_last(oracle, deq, ids):
    h = oracle.forward(np.asarray(ids, np.uint32), causal=True)[-1]
    logits = O.linear_t(h, deq["lm_head"], None, 1, TINY["vocab"], TINY["hidden"])
    return h, logits


def check_step(model, oracle, deq, histories, order):
    hs, lg, toks = model.last_hidden(), model.last_logits(), model._toks
    for row, sid in enumerate(order):
        h_ref, l_ref = oracle_last(oracle, deq, histories[sid])
        assert max_rel(hs[row], h_ref) <= TOL, (sid, len(histories[sid]))
        assert max_rel(lg[row], l_ref) <= TOL
        # greedy is exact on the GPU's own logits (first maximum wins) ...
        assert toks[row] == O.greedy(lg[row])
        # ... and agrees with the oracle's choice up to the logit tolerance
        assert l_ref[toks[row]] >= l_ref.max() - TOL * np.abs(l_ref).max()


def test_mixed_prefill_and_decode_steps_equal_per_sequence_execution(setup):
    qw, deq, oracle = setup
    rng = np.random.default_rng(1)
    alloc = BlockAllocator(64, 16, seed=3)
    model = DecoderModel(TINY, qw, n_pool_blocks=64, max_blocks_per_seq=16, max_step_tokens=512, max_step_seqs=8)
    hist = {}

    def run(entries):
        """entries: list of (seq id, new ids)."""
        ids, cached, new, tabs, order = [], [], [], [], []
        for sid, toks in entries:
            prev = hist.setdefault(sid, [])
            cached.append(len(prev)); new.append(len(toks)); ids.extend(toks)
            prev.extend(int(t) for t in toks)
            tabs.append(alloc.ensure(sid, len(prev))); order.append(sid)
        model._toks = model.step(ids, cached, new, np.stack(tabs))
        assert model.device_status() == 0
        check_step(model, oracle, deq, hist, order)
        return dict(zip(order, model._toks.tolist()))

    # step 1: three prefill chunks
    nxt = run([(0, rng.integers(0, 1000, 40)), (1, rng.integers(0, 1000, 7)), (2, rng.integers(0, 1000, 100))])
    # steps 2..: decode the three (crossing 16-token block boundaries), a new prefill joins in step 2,
    # caller order mixes decode and prefill entries
    nxt = run([(0, [nxt[0]]), (3, rng.integers(0, 1000, 33)), (1, [nxt[1]]), (2, [nxt[2]])])
    for _ in range(10):
        nxt = run([(sid, [nxt[sid]]) for sid in (2, 0, 3, 1)])
    assert len(hist[1]) == 18 and model.launches_last_step() > 0
    # a single-token sequence is a decode against an empty cache
    run([(9, [5])])
    # a prompt fed in chunks: every chunk after the first continues a cached prefix (positions, cache
    # slots, keys and values read through the block table), mixed with decode rows and with a chunk that
    # starts another sequence; every step is compared with the oracle run on the whole history, so
    # chunked == whole prompt == oracle
    prompt = rng.integers(0, 1000, 150)
    run([(11, prompt[:64]), (0, [nxt[0]])])
    run([(2, [nxt[2]]), (11, prompt[64:129]), (12, rng.integers(0, 1000, 20))])
    last = run([(11, prompt[129:])])
    h_chunked = model.last_hidden()[0].copy()
    whole = run([(13, prompt)])
    assert max_rel(model.last_hidden()[0], h_chunked) <= TOL and whole[13] == last[11]
    model.close()


def test_step_rejects_what_it_cannot_run(setup):
    qw, _, _ = setup
    model = DecoderModel(TINY, qw, n_pool_blocks=8, max_blocks_per_seq=8, max_step_tokens=64, max_step_seqs=2)
    tab = np.array([[0, 1, 2, 3, 4, 5, 6, 7]], np.int32)
    with pytest.raises(ComputeError):   # block table row with a missing entry
        model.step([1] * 20, [0], [20], np.array([[0, -1, -1, -1, -1, -1, -1, -1]], np.int32))
    with pytest.raises(ComputeError):   # more tokens than the step workspace
        model.step([1] * 65, [0], [65], tab)
    with pytest.raises(Exception):      # beyond the block table
        model.step([1], [128], [1], tab)
    model.close()


def test_turbo3_cache_mode_runs_the_same_steps_at_the_codec_accuracy(setup):
    """kv_turbo3: the cache holds TurboQuant 3-bit rows (4.57 times smaller) and every sequence attends
    through the decoding gather. The K/V rows carry the codec's error (3 bits per value), so the stack is
    compared with the fp32 oracle at the codec's accuracy, not at the bf16 bar: the kernel-level tests
    (test_gpu_paged, test_gpu_attention) hold the cache bytes and the attention over them to the oracle."""
    from gpu_util import cosine
    qw, deq, oracle = setup
    rng = np.random.default_rng(4)
    alloc = BlockAllocator(64, 16, seed=3)
    model = DecoderModel(TINY, qw, n_pool_blocks=64, max_blocks_per_seq=16, max_step_tokens=256, max_step_seqs=4, kv_turbo3=True)
    hist = {0: rng.integers(0, 1000, 60).tolist(), 1: rng.integers(0, 1000, 130).tolist()}
    # sequence 1 enters in two chunks (the second continues a cached, quantised prefix), sequence 0 whole
    toks = model.step(hist[0] + hist[1][:64], [0, 0], [60, 64], np.stack([alloc.ensure(0, 60), alloc.ensure(1, 64)]))
    assert model.device_status() == 0
    hist[0].append(int(toks[0]))
    toks = model.step([hist[0][-1]] + hist[1][64:], [60, 64], [1, 66], np.stack([alloc.ensure(0, 61), alloc.ensure(1, 130)]))
    assert model.device_status() == 0
    hist[1].append(int(toks[1])); hist[0].append(int(toks[0]))
    for _ in range(3):
        toks = model.step([hist[0][-1], hist[1][-1]], [len(hist[0]) - 1, len(hist[1]) - 1], [1, 1],
                          np.stack([alloc.ensure(0, len(hist[0])), alloc.ensure(1, len(hist[1]))]))
        assert model.device_status() == 0
        hs = model.last_hidden()
        for row, sid in enumerate((0, 1)):
            h_ref, _ = oracle_last(oracle, deq, hist[sid])
            assert np.isfinite(hs[row]).all() and cosine(hs[row], h_ref) >= 0.9, (sid, cosine(hs[row], h_ref))
        hist[0].append(int(toks[0])); hist[1].append(int(toks[1]))
    model.close()


@pytest.mark.parametrize("n_seqs", [1, 2, 3, 4, 5])
def test_decode_steps_of_few_sequences(n_seqs):
    """Up to four rows the projections run as one launch each with the norm in front and rotation, cache store or SwiGLU behind;
    five rows take the general route. Widths that leave uneven slices of k (20 and 44 groups of 32), contexts on both sides
    of a decode chunk."""
    cfg = dict(TINY, hidden=640, n_heads=5, n_kv_heads=1, intermediate=1408, vocab=700)
    w = make_weights(cfg, 31)
    qw, deq = quantize_weights(cfg, w)
    oracle = O.OracleStella(cfg, deq)
    rng = np.random.default_rng(n_seqs)
    alloc = BlockAllocator(128, 32, seed=3)
    model = DecoderModel(cfg, qw, n_pool_blocks=128, max_blocks_per_seq=32, max_step_tokens=512, max_step_seqs=9)
    lens = [127, 40, 16, 1, 130, 3, 20, 8, 5][:n_seqs]
    hist = [rng.integers(0, cfg["vocab"], n).tolist() for n in lens]
    toks = model.step(sum(hist, []), [0] * n_seqs, lens, np.stack([alloc.ensure(i, n) for i, n in enumerate(lens)]))
    for _ in range(3):
        for i in range(n_seqs):
            hist[i].append(int(toks[i]))
        toks = model.step([h[-1] for h in hist], [len(h) - 1 for h in hist], [1] * n_seqs, np.stack([alloc.ensure(i, len(h)) for i, h in enumerate(hist)]))
        assert model.device_status() == 0
        hs, lg = model.last_hidden(), model.last_logits()
        for i, ids in enumerate(hist):
            h_ref = oracle.forward(np.asarray(ids, np.uint32), causal=True)[-1]
            assert max_rel(hs[i], h_ref) <= TOL and max_rel(lg[i], O.linear_t(h_ref, deq["lm_head"], None, 1, cfg["vocab"], cfg["hidden"])) <= TOL, i
            assert toks[i] == O.greedy(lg[i])
    model.close()


@pytest.mark.parametrize("heads,kv,inter", [(2, 1, 256), (6, 3, 1280), (8, 1, 512), (12, 1, 512), (16, 2, 2048), (12, 2, 8960)])
@pytest.mark.parametrize("n_seqs", [1, 2, 3, 4])
def test_decode_steps_whose_layers_are_one_launch(heads, kv, inter, n_seqs):
    """Widths at which the layers of a decode step of up to four rows run as one launch (and two, of 16 heads and of 12 to a key head, at which they do not): two to twelve warps,
    CTAs without a share of a matrix, shares that end in part of a tile, one to eight tiles a CTA, groups of 2 to 8 query heads. Contexts that
    end a cache block, begin one, are one token and need further rounds of blocks; 3 layers, so that every place in shared memory is filled
    again and the parity of its barrier comes back."""
    cfg = dict(TINY, hidden=128 * heads, n_heads=heads, n_kv_heads=kv, intermediate=inter, vocab=520, n_layers=3, max_pos=2048)
    qw, deq = quantize_weights(cfg, make_weights(cfg, 31))
    oracle = O.OracleStella(cfg, deq)
    rng = np.random.default_rng([n_seqs, heads])
    alloc = BlockAllocator(300, 100, seed=3)
    model = DecoderModel(cfg, qw, n_pool_blocks=300, max_blocks_per_seq=100, max_step_tokens=1024, max_step_seqs=4)
    lens = [(130, 1, 47, 16), (15, 700, 30, 1), (1, 31, 128, 97), (250, 16, 3, 5)][n_seqs - 1][:n_seqs]
    hist = [rng.integers(0, cfg["vocab"], n).tolist() for n in lens]
    step = lambda ids, cached, new: model.step(ids, cached, new, np.stack([alloc.ensure(i, c + n) for i, (c, n) in enumerate(zip(cached, new))]))
    for i in range(n_seqs):  # a sequence at a time, so that one of a single token is a decode step as well
        model.step(hist[i], [0], [lens[i]], alloc.ensure(i, lens[i])[None])
    for _ in range(5):
        for h in hist:
            h.append(int(rng.integers(0, cfg["vocab"])))
        toks = step([h[-1] for h in hist], [len(h) - 1 for h in hist], [1] * n_seqs)
        assert model.device_status() == 0 and (model.launches_last_step() <= 7) == (heads <= 12 and heads // kv <= 8)
    hs, lg = model.last_hidden(), model.last_logits()
    again = step([h[-1] for h in hist], [len(h) - 1 for h in hist], [1] * n_seqs)
    assert np.array_equal(hs, model.last_hidden()) and np.array_equal(lg, model.last_logits()) and np.array_equal(toks, again)
    for i, ids in enumerate(hist):
        h_ref = oracle.forward(np.asarray(ids, np.uint32), causal=True)[-1]
        assert max_rel(hs[i], h_ref) <= TOL and max_rel(lg[i], O.linear_t(h_ref, deq["lm_head"], None, 1, cfg["vocab"], cfg["hidden"])) <= TOL, i
        assert toks[i] == O.greedy(lg[i])
    model.close()


def test_one_launch_and_one_per_projection_on_long_contexts():
    """Contexts of up to 3000 tokens (several rounds of cache blocks per warp): the layers as one launch against the general route of the
    deterministic switch. Bound: as the tests against the oracle. Two sequences whose tables share the block of a new token do not take the one launch, which reads blocks
    ahead of the stores into them."""
    from logismos_b200._lib import lib
    cfg = dict(TINY, hidden=768, n_heads=6, n_kv_heads=2, intermediate=1024, vocab=512, max_pos=4096)
    qw, _ = quantize_weights(cfg, make_weights(cfg, 5))
    model = DecoderModel(cfg, qw, n_pool_blocks=512, max_blocks_per_seq=200, max_step_tokens=3072, max_step_seqs=4)
    rng, alloc = np.random.default_rng(1), BlockAllocator(512, 200, seed=2)
    lens = [3000, 1537, 512]
    tables = np.stack([alloc.ensure(i, n + 1) for i, n in enumerate(lens)])
    for i, n in enumerate(lens):
        model.step(rng.integers(0, 512, n), [0], [n], tables[i:i + 1])
    out = []
    for det in (0, 1):
        lib.logismos_set_deterministic(det)
        try:
            model.step([5, 6, 7], lens, [1] * 3, tables)
            out.append((model.last_hidden().copy(), model.last_logits().copy(), model.launches_last_step()))
        finally:
            lib.logismos_set_deterministic(0)
    assert out[0][2] < out[1][2] and max_rel(out[0][0], out[1][0]) <= TOL and max_rel(out[0][1], out[1][1]) <= TOL
    model.step([5, 5], [3000, 3000], [1, 1], tables[[0, 0]])
    assert model.launches_last_step() > 7 and max_rel(model.last_hidden(), out[1][0][[0, 0]]) <= TOL
    model.close()


@pytest.mark.parametrize("heads,kv,inter", [(10, 2, 3840), (10, 5, 512), (10, 10, 1024), (6, 2, 1024), (2, 1, 256)])
@pytest.mark.parametrize("n_seqs", [1, 2, 3, 4])
def test_one_launch_with_warps_that_are_no_multiple_of_four(heads, kv, inter, n_seqs):
    """Ten, six and two warps, few tiles a CTA and contexts of one to many chunks, so that a CTA puts chunks together and holds weight rows as well: the layers as one launch against
    the general route of the deterministic switch. Bound: as the tests against the oracle."""
    from logismos_b200._lib import lib
    cfg = dict(TINY, hidden=128 * heads, n_heads=heads, n_kv_heads=kv, intermediate=inter, vocab=520, n_layers=3, max_pos=2048)
    qw, _ = quantize_weights(cfg, make_weights(cfg, 13))
    model = DecoderModel(cfg, qw, n_pool_blocks=300, max_blocks_per_seq=100, max_step_tokens=1536, max_step_seqs=4)
    rng, alloc = np.random.default_rng([heads, n_seqs]), BlockAllocator(300, 100, seed=2)
    lens = [400, 900, 20, 150]
    tables = np.stack([alloc.ensure(i, n + 1) for i, n in enumerate(lens)])
    for i, n in enumerate(lens):
        model.step(rng.integers(0, 520, n), [0], [n], tables[i:i + 1])
    for first in range(4):
        which = [(first + i) % 4 for i in range(n_seqs)]
        out = []
        for det in (0, 1):
            lib.logismos_set_deterministic(det)
            try:
                model.step([5 + i for i in which], [lens[i] for i in which], [1] * n_seqs, tables[which])
                out.append((model.last_hidden().copy(), model.last_logits().copy()))
                assert (model.launches_last_step() <= 7) == (det == 0)
            finally:
                lib.logismos_set_deterministic(0)
        for i in range(n_seqs):
            assert max_rel(out[0][0][i], out[1][0][i]) <= TOL and max_rel(out[0][1][i], out[1][1][i]) <= TOL, (first, i)
    model.close()


def test_long_contexts_of_many_key_heads_do_not_take_the_one_launch():
    """Six key heads and four rows leave six chunks per context: a step at 1500 tokens needs 8 rounds of cache blocks and takes the one launch, at 3000 tokens 16 and does not. Bound:
    as the tests against the oracle."""
    from logismos_b200._lib import lib
    cfg = dict(TINY, hidden=768, n_heads=6, n_kv_heads=6, intermediate=1024, vocab=512, max_pos=4096)
    qw, _ = quantize_weights(cfg, make_weights(cfg, 5))
    model = DecoderModel(cfg, qw, n_pool_blocks=512, max_blocks_per_seq=200, max_step_tokens=3072, max_step_seqs=4)
    rng, alloc = np.random.default_rng(1), BlockAllocator(512, 200, seed=2)
    tables = np.stack([alloc.ensure(i, n + 1) for i, n in enumerate((3000, 70, 33, 5))])
    for i, n in enumerate((3000, 70, 33, 5)):
        model.step(rng.integers(0, 512, n), [0], [n], tables[i:i + 1])
    for ctx, one in ((1500, True), (3000, False)):
        out = []
        for det in (0, 1):
            lib.logismos_set_deterministic(det)
            try:
                model.step([5, 6, 7, 8], [ctx, 70, 33, 5], [1] * 4, tables)
                out.append(model.last_logits().copy())
                assert (model.launches_last_step() <= 7) == (one and det == 0), (ctx, det, model.launches_last_step())
            finally:
                lib.logismos_set_deterministic(0)
        assert max_rel(out[0], out[1]) <= TOL
    model.close()


@pytest.mark.parametrize("before", [62, 63, 64, 65])
def test_numbers_of_the_one_launch_start_again(before):
    """The words that CTAs exchange carry numbers of 32 bits. A model's count starts 64 launches short of where they end: steps of one row up to there, then one of four rows, whose words
    have not all been written before, and two more. Bound: as the tests against the oracle."""
    from logismos_b200._lib import lib
    cfg = dict(TINY, hidden=512, n_heads=4, n_kv_heads=2, intermediate=512, vocab=512, n_layers=3, max_pos=1024)
    qw, _ = quantize_weights(cfg, make_weights(cfg, 9))
    model = DecoderModel(cfg, qw, n_pool_blocks=128, max_blocks_per_seq=32, max_step_tokens=512, max_step_seqs=4)
    rng, alloc = np.random.default_rng(4), BlockAllocator(128, 32, seed=2)
    lens = [17, 300, 129, 64]
    tables = np.stack([alloc.ensure(i, n + 1) for i, n in enumerate(lens)])
    for i, n in enumerate(lens):
        model.step(rng.integers(0, 512, n), [0], [n], tables[i:i + 1])

    def step(rows, det):
        lib.logismos_set_deterministic(det)
        try:
            model.step(list(range(rows)), lens[:rows], [1] * rows, tables[:rows])
            assert (model.launches_last_step() <= 7) == (det == 0)
            return model.last_logits().copy()
        finally:
            lib.logismos_set_deterministic(0)

    want = step(4, 1)
    for _ in range(before):
        first = step(1, 0)
    assert max_rel(first, want[:1]) <= TOL
    for rows in (4, 1, 3):
        got = step(rows, 0)
        assert max_rel(got, want[:rows]) <= TOL, rows
    model.close()


def test_numbers_start_again_where_some_ctas_have_no_part():
    """Two heads and one row: 18 of 148 CTAs have no weight rows, no chunk and nothing to put together. They read the count of launches and clear words with the others. Steps over the point
    where the numbers start again and beyond. Bound: as the tests against the oracle."""
    from logismos_b200._lib import lib
    cfg = dict(TINY, hidden=256, n_heads=2, n_kv_heads=1, intermediate=256, vocab=512, n_layers=2, max_pos=1024)
    qw, _ = quantize_weights(cfg, make_weights(cfg, 9))
    model = DecoderModel(cfg, qw, n_pool_blocks=64, max_blocks_per_seq=32, max_step_tokens=512, max_step_seqs=4)
    rng, alloc = np.random.default_rng(4), BlockAllocator(64, 32, seed=2)
    tables = np.stack([alloc.ensure(0, 200)])
    model.step(rng.integers(0, 512, 190), [0], [190], tables)
    out = []
    for det in [1] + 100 * [0]:
        lib.logismos_set_deterministic(det)
        try:
            model.step([7], [190], [1], tables)
            assert (model.launches_last_step() <= 7) == (det == 0)
            out.append(model.last_logits().copy())
        finally:
            lib.logismos_set_deterministic(0)
        assert max_rel(out[-1], out[0]) <= TOL, len(out)
    model.close()


def test_one_launch_steps_replay_from_a_graph():
    """A step's device work captured in a CUDA graph: the layers as one launch count their launches on the device, so each replay is the step again, bit for bit, also where the numbers
    of the words start again."""
    import torch
    cfg = dict(TINY, hidden=512, n_heads=4, n_kv_heads=2, intermediate=512, vocab=512, n_layers=3, max_pos=1024)
    qw, _ = quantize_weights(cfg, make_weights(cfg, 9))
    model = DecoderModel(cfg, qw, n_pool_blocks=64, max_blocks_per_seq=32, max_step_tokens=512, max_step_seqs=4)
    rng, alloc = np.random.default_rng(4), BlockAllocator(64, 32, seed=2)
    tables = np.stack([alloc.ensure(i, n + 1) for i, n in enumerate((300, 17))])
    for i, n in enumerate((300, 17)):
        model.step(rng.integers(0, 512, n), [0], [n], tables[i:i + 1])
    model.step([7, 9], [300, 17], [1, 1], tables)
    want, stream, graph = model.last_logits().copy(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        model.replay_device(torch.cuda.current_stream().cuda_stream)
    assert model.launches_last_step() <= 7
    for _ in range(80):
        graph.replay()
    torch.cuda.synchronize()
    assert model.device_status() == 0 and np.array_equal(model.last_logits(), want)
    model.close()


def test_deterministic_switch_keeps_a_row_independent_of_its_step():
    """With the switch on, a sequence's decode steps have the same bits alone and beside 3, 4 and 29 others: the same projections and the
    same pieces of its context of 1000 tokens."""
    from logismos_b200._lib import lib
    cfg = dict(TINY, max_pos=1024)
    qw, _ = quantize_weights(cfg, make_weights(cfg, 77))
    model = DecoderModel(cfg, qw, n_pool_blocks=2048, max_blocks_per_seq=64, max_step_tokens=1024, max_step_seqs=32)
    prompt = np.random.default_rng(4).integers(0, cfg["vocab"], 1000)
    lib.logismos_set_deterministic(1)
    try:
        seen = {}
        for n in (1, 4, 5, 30):
            alloc = BlockAllocator(2048, 64, seed=n)
            tables = np.stack([alloc.ensure(i, 1003) for i in range(n)])
            for i in range(n):
                model.step(np.roll(prompt, i), [0], [1000], tables[i:i + 1])
            for t in range(3):
                model.step([7 + t] * n, [1000 + t] * n, [1] * n, tables)
                seen.setdefault(t, []).append((n, model.last_hidden()[0].copy(), model.last_logits()[0].copy() if n <= 5 else None))
        for t, rows in seen.items():
            for n, h, l in rows[1:]:
                assert np.array_equal(h, rows[0][1]) and (l is None or np.array_equal(l, rows[0][2])), (t, n)
        assert model.device_status() == 0
    finally:
        lib.logismos_set_deterministic(0)
        model.close()


def in_two_threads(work):
    """work(i) in threads 0 and 1, which begin together; what they raise."""
    import threading
    start, errors = threading.Barrier(2), []

    def run(i):
        try:
            start.wait()
            work(i)
        except Exception as e:  # reported by the caller
            errors.append(repr(e))
    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def test_models_of_different_widths_step_in_two_threads():
    """Models on one GPU are stepped from threads of their own. Their launches of the same kernel ask for different amounts of shared
    memory (80 and 46 KB for four rows); none may narrow what another is about to launch with."""
    models, tables = [], np.arange(8, dtype=np.int32).reshape(4, 2)
    for i in (8960, 5120):
        cfg = dict(TINY, intermediate=i, vocab=512)
        qw, _ = quantize_weights(cfg, make_weights(cfg, 3))
        models.append(DecoderModel(cfg, qw, n_pool_blocks=8, max_blocks_per_seq=2, max_step_tokens=8, max_step_seqs=4))
        models[-1].step([1, 2, 3, 4], [0] * 4, [1] * 4, tables)

    def work(i):
        for t in range(3000):
            models[i].step([5, 6, 7, 8], [1] * 4, [1] * 4, tables)
    assert in_two_threads(work) == []
    for m in models:
        assert m.device_status() == 0
        m.close()
