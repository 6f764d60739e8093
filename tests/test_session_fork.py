"""Forking a live session at a position that is NOT block-aligned, then appending on both branches: the shared partial
tail block must be replaced by a private copy of its valid rows (copy-on-write) on each side.

Reference: PagedKvBlockTable::fork_prefix (crates/macllm-kv/src/cache.rs:1565-1571), the copy-on-write reservation
(cache.rs:2252-2280,2376-2418), copy_paged_prefix (cache.rs:3042-3089) and the reference's own cases
paged_copy_on_write_* (cache.rs:4632-4747).  The host bookkeeping is compared with the oracle on the fake model (no GPU);
the device page copy is compared with the oracle's logits on a GPU."""
import importlib

import numpy as np
import pytest


@pytest.fixture(scope="module")
def eng(mk):
    return importlib.import_module("macllm_infer_b200.engine")


@pytest.mark.parametrize("start", [0.0, 1.5, "0", None, [0]])
def test_a_start_position_is_a_whole_number(eng, start):
    model = eng.Model.fake(vocab=32, kv_capacity_tokens=1024)
    session = model.new_session()
    with pytest.raises(TypeError):
        model.forward_batch([(session, [1, 2, 3], start)])
    model.forward_batch([(session, [1, 2, 3], 0)])   # nothing was reserved or run by the refused call


def oracle_fork(om, s, n):
    return dict(table=s["table"].fork_prefix(n), len=n)


def test_fork_of_a_partial_tail_copies_on_write_on_both_branches_host_side(eng):
    from oracle import engine as oe
    model = eng.Model.fake(vocab=32, kv_capacity_tokens=1024)
    om = oe.OracleModel(32, 4096, 16, 8, 1024, 0)
    a, oa = model.new_session(), om.new_session()
    prompt = list(range(1, 22))                       # 21 tokens: one full block and 5 rows of a second one
    model.forward_batch([(a, prompt, 0)])
    om.forward([(oa, prompt, 0)], om.reserve_batch([(oa, 0, 21)]))
    b, ob = a.fork_prefix(21), oracle_fork(om, oa, 21)
    assert len(b) == 21
    assert [int(x) for x in b.block_table()[0]] == [int(x) for x in a.block_table()[0]] == [blk[0] for blk in oa["table"].blocks]
    assert model.pool_stats() == om.pool.stats()
    # both branches append: each replaces the shared tail by a private block (replacement first, then growth)
    model.forward_batch([(a, [5], 21), (b, [7, 8], 21)])
    om.forward([(oa, [5], 21), (ob, [7, 8], 21)], om.reserve_batch([(oa, 21, 1), (ob, 21, 2)]))
    ta, tb = [int(x) for x in a.block_table()[0]], [int(x) for x in b.block_table()[0]]
    assert ta == [blk[0] for blk in oa["table"].blocks] and tb == [blk[0] for blk in ob["table"].blocks]
    assert ta[0] == tb[0] and ta[1] != tb[1]        # the full block stays shared, the tails are private now
    assert model.pool_stats() == om.pool.stats()
    # a fork beyond the source's length, or of another model's session, is refused
    capi = importlib.import_module("macllm_infer_b200._capi")
    with pytest.raises(capi.MkError):
        a.fork_prefix(23)
    other = eng.Model.fake(vocab=32)
    with pytest.raises(capi.MkError):
        import ctypes as C
        h = C.c_void_p()
        capi.check(capi.lib().mk_session_fork_prefix(other._h, a._h, 4, C.byref(h)))


@pytest.mark.gpu
@pytest.mark.parametrize("kv_dtype,matmul_path,layers,fork_at", [("f32", 1, 1, 21), ("f16", 0, 1, 21), ("f32", 1, 2, 37), ("f16", 0, 2, 5)])
def test_copy_on_write_page_copy_matches_the_oracle(mk, eng, tmp_path_factory, kv_dtype, matmul_path, layers, fork_at):
    """cow_copy_kernel on the device: after the fork both branches attend to the prefix rows their private tail
    blocks received by copy, so their logits match the oracle only if the copy moved the right rows of every layer and
    head."""
    from oracle import decoder, engine as oe
    seed = importlib.import_module("macllm_infer_b200.seed_gguf")
    spec = seed.scaled("tinyllama-1.1b", layers=layers, vocab=2048)
    path = tmp_path_factory.mktemp("fork") / "llama.gguf"
    seed.write_seed_gguf(path, spec, seed=0)
    model = eng.Model.load_gguf(path, kv_dtype=kv_dtype, matmul_path=matmul_path, max_batch_tokens=128, max_batch_lanes=4)
    dec = decoder.Decoder(path, kv_dtype="f32", matmul_mode=1)
    om = oe.OracleModel(dec.vocab, dec.max_context, 16, 8, 4096, 0, decoder=dec)
    rng = np.random.default_rng(fork_at)
    prompt = [int(x) for x in rng.integers(3, spec.vocab, size=fork_at)]
    a, oa = model.new_session(), om.new_session()
    model.forward_batch([(a, prompt, 0)])
    om.forward([(oa, prompt, 0)], om.reserve_batch([(oa, 0, fork_at)]))
    b, ob = a.fork_prefix(fork_at), oracle_fork(om, oa, fork_at)
    ta = [int(x) for x in rng.integers(3, spec.vocab, size=1)]
    tb = [int(x) for x in rng.integers(3, spec.vocab, size=3)]
    # control sessions that never fork: the same tokens through private blocks only
    ca, cb = model.new_session(), model.new_session()
    model.forward_batch([(ca, prompt, 0)])
    model.forward_batch([(cb, prompt, 0)])
    for step in range(2):
        pa, pb = fork_at + step * 1, fork_at + step * 3
        got, _ = model.forward_batch([(a, ta, pa), (b, tb, pb)])
        ctl, _ = model.forward_batch([(ca, ta, pa), (cb, tb, pb)])
        want = om.forward([(oa, ta, pa), (ob, tb, pb)], om.reserve_batch([(oa, pa, 1), (ob, pb, 3)]))
        assert np.isfinite(got).all()
        # the copied rows are the rows the private blocks of the control hold: the same kernels on the same values,
        # only the block numbers differ, so the logits are bit-identical.  A missing or misplaced row would show here.
        assert np.array_equal(got, ctl)
        err = float(np.abs(got - want).max())
        cos = min(float(g @ w / np.sqrt((g @ g) * (w @ w))) for g, w in zip(got, want))
        print("step", step, "max-abs vs oracle", err, "cos", cos)
        # against the oracle: the envelope of the end-to-end tests (a flipped 8-bit rounding moves a logit by a few 1e-2)
        assert err <= 0.25 and cos >= 0.999
        # block ids differ from the oracle's here (the control sessions take blocks in between; the host-side test
        # above compares ids); the shape of the sharing is the same: full prefix blocks shared, tails private
        ba, bb = [int(x) for x in a.block_table()[0]], [int(x) for x in b.block_table()[0]]
        full = fork_at // 16
        assert ba[:full] == bb[:full] and len(ba) == len(oa["table"].blocks) and len(bb) == len(ob["table"].blocks)
        assert not set(ba[full:]) & set(bb[full:])
    # the control sessions hold blocks the oracle never allocated, so pool counters are compared without them
    for c in (ca, cb):
        c.clear()
        c.close()
    model.synchronize()
    ps, os_ = model.pool_stats(), om.pool.stats()
    assert ps["live_blocks"] == os_["live_blocks"] and ps["reserved_blocks"] == os_["reserved_blocks"] == 0


@pytest.mark.gpu
def test_lanes_that_share_more_pages_than_the_pool_has(mk, eng, tmp_path_factory):
    """64 lanes over one prefix name its pages 64 times: 7808 table entries with a pool of 256 pages.  The results are those of a pool that could
    hold every lane's pages."""
    seed = importlib.import_module("macllm_infer_b200.seed_gguf")
    spec = seed.scaled("tinyllama-1.1b", layers=1, vocab=512)
    path = tmp_path_factory.mktemp("fork") / "llama.gguf"
    seed.write_seed_gguf(path, spec, seed=0)
    prefix = 1936
    got = []
    for capacity in (4096, 64 * (prefix + 32)):
        model = eng.Model.load_gguf(path, kv_dtype="f16", max_batch_tokens=64, max_batch_lanes=64, kv_capacity_tokens=capacity)
        rng = np.random.default_rng(0)
        prompt = rng.integers(3, spec.vocab, prefix)
        first = model.new_session()
        for at in range(0, prefix, 64):
            model.forward_batch([(first, prompt[at:at + 64], at)])
        sessions = [first] + [first.fork_prefix(prefix) for _ in range(63)]
        rows = []
        for step in range(3):
            ids = rng.integers(3, spec.vocab, 64)
            logits, _ = model.forward_batch([(s, [int(t)], prefix + step) for s, t in zip(sessions, ids)])
            rows.append(logits)
        got.append(np.stack(rows))
    assert np.isfinite(got[0]).all() and np.array_equal(got[0], got[1])
