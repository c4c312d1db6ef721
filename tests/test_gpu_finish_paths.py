"""The branches of a row's finish and the warp-per-row kernel, at the sizes where they change: tokens,
statuses, kept lists and probabilities bit for bit against the oracle."""
import numpy as np
import pytest

from born_b200 import workloads as W
from tests.test_gpu_parity import assert_parity, run_both

pytestmark = pytest.mark.gpu


def _logits(seed, B, V, dtype, scale=3.0):
    z = (W.normal(seed, 11, B * V) * scale).astype(np.float32).reshape(B, V)
    if dtype == "f32":
        return z
    return (z.view(np.uint32) >> 16).astype(np.uint16)  # (truncated: any bf16 values will do, ties included)


# either side of 32, 64, 128, 256 candidates (threads per candidate, then the counting sort), of 128 (bisection
# over thread maxima, then bins) and up to the candidate limit; top-p off and on
@pytest.mark.parametrize("k", [1, 31, 32, 33, 64, 65, 128, 129, 255, 256, 257, 600, 1000])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_candidate_counts_either_side_of_every_split(sampler, oracle, k, dtype):
    B, V = 6, 20011 if dtype == "f32" else 20008
    z, u = _logits(k, B, V, dtype), W.uniform_f32(k, 2, B)
    for top_p in (0.0, 0.93):
        got, ref = run_both(sampler, oracle, z, dict(temperature=4.0, top_k=k, top_p=top_p), u, want_kept=1024)
        assert_parity(got, ref)


# min-p and top-p alone leave their own numbers of candidates
@pytest.mark.parametrize("params", [dict(temperature=3.0, min_p=0.02), dict(temperature=1.5, top_p=0.9),
                                    dict(temperature=2.0, min_p=0.005, top_p=0.97)])
def test_candidate_counts_of_rows_without_top_k(sampler, oracle, params):
    B, V = 12, 32000
    z = _logits(5, B, V, "f32") * np.linspace(0.6, 1.6, B, dtype=np.float32)[:, None]
    got, ref = run_both(sampler, oracle, z, params, W.uniform_f32(5, 2, B), want_kept=1024)
    assert_parity(got, ref)


# every live group belongs to one thread: its maxima cannot tell the k-th key
def test_fewer_live_maxima_than_top_k(sampler, oracle):
    B, V = 3, 131072
    z = _logits(9, B, V, "f32")
    live = (np.arange(V) // 32) % 256 == 7
    mask = np.packbits(np.tile(live, (B, 1)), axis=1, bitorder="little").view(np.uint32)
    got, ref = run_both(sampler, oracle, z, dict(temperature=1.0, top_k=50), W.uniform_f32(9, 2, B), mask=mask)
    assert_parity(got, ref)


# top-k above 128 (bins over the keys) where the k-th value is tiny beside the maximum: one unit in the last
# place of the maximum spans many steps of its key.  Rows of one value beside one outlier (all ties: the exact
# search) and of small normal values
@pytest.mark.parametrize("k", [100, 150, 200, 600])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("segments", [1, 4])
def test_kth_value_tiny_beside_the_maximum(sampler, oracle, k, dtype, segments):
    if segments > 1 and k > 256:
        pytest.skip("a segment's top-k is limited to 256")
    V, outlier = 32768, [17.0, 40.0, 11.0, 21.5, 20.5, 48.7, 50.2]
    z = (W.normal(30, 1, len(outlier) * V) * 1e-6).astype(np.float32).reshape(-1, V)
    for b, v in enumerate([1e-6, 1e-5, -1e-5, 1e-6, 3e-5]):
        z[b] = v
    z[:, 3] = outlier
    logits = z if dtype == "f32" else W.f32_to_bf16_bits(z).reshape(z.shape)
    u = W.uniform_f32(30, 2, len(outlier))
    for params in (dict(temperature=4.0, top_k=k), dict(temperature=4.0, top_k=k, top_p=0.999)):
        got, ref = run_both(sampler, oracle, logits, params, u, segments=segments, want_kept=1024)
        assert_parity(got, ref)


# ... and the way a smaller top-k gets there: a mask leaves all live groups to one thread
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_kth_value_tiny_beside_the_maximum_with_few_live_maxima(sampler, oracle, dtype):
    B, V, k = 3, 131072, 10
    z = (W.normal(31, 1, B * V) * 1e-6).astype(np.float32).reshape(B, V)
    live = (np.arange(V) // 32) % 256 == 7
    z[:, 7 * 32] = [48.7, 17.0, 21.5]
    mask = np.packbits(np.tile(live, (B, 1)), axis=1, bitorder="little").view(np.uint32)
    logits = z if dtype == "f32" else W.f32_to_bf16_bits(z).reshape(z.shape)
    got, ref = run_both(sampler, oracle, logits, dict(temperature=4.0, top_k=k), W.uniform_f32(31, 2, B), mask=mask)
    assert_parity(got, ref)


# history tokens among the candidates, beside them, and such as share a bit of the 4096-bit map with one
@pytest.mark.parametrize("B", [2, 40])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_history_tokens_among_the_candidates(sampler, oracle, B, dtype):
    V, H = 50176, 300
    z = _logits(3, B, V, dtype)
    val = z if dtype == "f32" else (z.astype(np.uint32) << 16).view(np.float32)
    order = np.argsort(-val, axis=1)
    hist = np.empty((B, H), np.int32)
    hist[:, :60] = order[:, :120:2]
    hist[:, 60:120] = (order[:, 1:121:2] + 4096) % V
    hist[:, 120:] = W.randint(3, 4, B * (H - 120), V).reshape(B, -1)
    for params in (dict(temperature=0.9, top_k=50, top_p=0.95, repetition_penalty=1.2),
                   dict(temperature=0.9, min_p=0.05, top_p=0.9, frequency_penalty=0.5, presence_penalty=-0.4),
                   dict(temperature=0.0, frequency_penalty=0.7)):
        got, ref = run_both(sampler, oracle, z, params, W.uniform_f32(3, 2, B), hist=hist)
        assert_parity(got, ref)


# the history list by bits (up to the longest segment whose bits fit the ring) and by the hash table (beyond it,
# and in ranges of long rows): few tokens many times each, tokens that share a hash, ids outside the row
@pytest.mark.parametrize("B,V,dtype", [(2, 1000, "f32"), (40, 32001, "f32"), (150, 229376, "bf16"), (150, 229377, "bf16"), (150, 262144, "f32"),
                                       (300, 180000, "bf16")])
def test_history_list_by_bits_and_by_hash(sampler, oracle, B, V, dtype):
    H = 700
    z = _logits(V, B, V, dtype)
    val = z if dtype == "f32" else (z.astype(np.uint32) << 16).view(np.float32)
    hist = W.randint(V, 4, B * H, V).astype(np.int32).reshape(B, H)
    top = np.argpartition(-val, 50, axis=1)[:, :50]
    hist[:, :50] = top
    hist[:, 50:100] = top[:, ::-1]                   # repeats
    hist[:, 100:400] = hist[:, 300:600]              # ... of tokens all over the row, many with a common hash
    hist[:, 600:680] = top[:, :1]                    # one token many times
    hist[:, 680:690], hist[:, 690:] = -1, V
    for params in (dict(temperature=0.9, top_k=40, repetition_penalty=1.2, frequency_penalty=0.02),
                   dict(temperature=0.9, min_p=0.05, top_p=0.9, frequency_penalty=0.05, presence_penalty=0.3)):
        got, ref = run_both(sampler, oracle, z, params, W.uniform_f32(V, 2, B), hist=hist)
        assert_parity(got, ref)


# a cluster whose rows are too long for their group keys to stay in shared memory
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_cluster_with_keys_in_global_memory(oracle, dtype):
    from born_b200 import Sampler
    B, V, H = 2, 450000, 100
    z, u = _logits(45, B, V, dtype, 4.0), W.uniform_f32(45, 2, B)
    val = z if dtype == "f32" else (z.astype(np.uint32) << 16).view(np.float32)
    hist = W.randint(45, 4, B * H, V).astype(np.int32).reshape(B, H)
    hist[:, :40] = np.argsort(-val, axis=1)[:, :80:2]
    s = Sampler(device=0, max_batch=B, max_vocab=V)
    try:
        for params in (dict(temperature=1.0, top_k=50), dict(temperature=1.0, top_k=200, top_p=0.9), dict(temperature=0.8, min_p=0.05),
                       dict(temperature=0.5, top_p=0.8), dict(temperature=0.0)):
            for h in (None, hist):
                p = dict(params, **({} if h is None else dict(repetition_penalty=1.2)))
                got, ref = run_both(s, oracle, z, p, u, hist=h)
                assert_parity(got, ref)
    finally:
        s.close()


# top-p alone over penalised values: from the group keys (peaked rows), from the groups' tokens or by the exact search
# (flat ones); history tokens above the penalised maximum,
# raised by a penalty below zero, masked, and beside the nucleus
@pytest.mark.parametrize("B,V,masked", [(1, 50176, False), (24, 50176, False), (24, 50176, True), (200, 16384, False), (301, 50176, False),
                                        (400, 8192, True)])
def test_nucleus_of_penalised_rows(sampler, oracle, B, V, masked):
    H = 200
    rank = np.argsort(W.uniform_f32(B, 4, B * V).reshape(B, V), axis=1).argsort(axis=1)
    z = _logits(B + V, B, V, "f32", 1.0) - np.float32(1.6) * np.log(rank + 1.0).astype(np.float32)
    flat = np.arange(B) % 8 == 7
    z[flat] = _logits(B + V, B, V, "f32", 2.2)[flat]
    order = np.argsort(-z, axis=1)
    hist = W.randint(B, 5, B * H, V).astype(np.int32).reshape(B, H)
    hist[:, :40] = order[:, :80:2]
    hist[:, 40:60] = order[:, :40:2]
    mask = None
    if masked:
        bits = W.uniform_f32(B, 6, B * V).reshape(B, V) < 0.7
        bits[:, 0] = True
        mask = np.packbits(bits, axis=1, bitorder="little").view(np.uint32)
    u = W.uniform_f32(B, 2, B)
    for params in (dict(temperature=0.8, top_p=0.9, repetition_penalty=1.2), dict(temperature=1.1, top_p=0.6, frequency_penalty=-0.7),
                   dict(temperature=0.6, top_p=0.97, repetition_penalty=1.1, frequency_penalty=0.5, presence_penalty=0.3)):
        sampler.fallback_rows
        got, ref = run_both(sampler, oracle, z, params, u, mask=mask, hist=hist, want_kept=1024)
        assert_parity(got, ref)
        # only the flat rows, whose nucleus or its bound may not fit the selection, take the exact search
        assert sampler.fallback_rows <= flat.sum()


# more rows than CTAs fit at once: a CTA per row in waves, and ranges for long rows with a nearly empty second wave
@pytest.mark.parametrize("B,V,dtype", [(297, 1000, "f32"), (301, 50176, "f32"), (303, 50001, "bf16"), (375, 50176, "bf16"), (600, 1031, "bf16")])
def test_more_rows_than_fit_at_once(sampler, oracle, B, V, dtype):
    z, u = _logits(B, B, V, dtype), W.uniform_f32(B, 2, B)
    hist = W.randint(B, 3, B * 40, V).astype(np.int32).reshape(B, 40)
    for params in (dict(temperature=0.8, top_k=40, top_p=0.9, repetition_penalty=1.3), dict(temperature=0.0)):
        got, ref = run_both(sampler, oracle, z, params, u, hist=hist)
        assert_parity(got, ref)
    got, ref = run_both(sampler, oracle, z, dict(temperature=0.7, top_p=0.8), u)
    assert_parity(got, ref, check_kept=False)


# a warp per row: one block, a block and a granule, ragged tails, the largest top-k; and the rows that leave
# its path: equal values beyond its candidate list, nothing alive, NaN and infinity
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("V,G,k", [(520, 8, 8), (1024, 8, 16), (1032, 8, 16), (8200, 8, 64), (9216, 8, 128), (9016, 4, 1)])
def test_warp_per_row_segments(sampler, oracle, V, G, k, dtype):
    import torch
    # (a CTA per row would take more than two waves and a half of two per SM)
    B = -(-(5 * torch.cuda.get_device_properties(0).multi_processor_count + 8) // G)
    z = _logits(V + k, B, V * G, dtype)
    ninf, pinf, nan, one = ((np.float32(x) for x in (-np.inf, np.inf, np.nan, 1.0)) if dtype == "f32" else
                            (np.uint16(x) for x in (0xFF80, 0x7F80, 0x7FC0, 0x3F80)))
    z[0] = ninf
    z[1, V:2 * V] = one        # one segment all equal
    z[2, V * G - 1] = nan
    z[3, 5] = pinf
    z[4, 7:] = ninf            # fewer tokens than top-k
    z[5] = ninf
    z[5, V * G - 3:] = one
    got, ref = run_both(sampler, oracle, z, dict(temperature=1.3, top_k=k, top_p=0.95), W.uniform_f32(V, 2, B), segments=G,
                        want_kept=min(1024, k * G))
    assert_parity(got, ref)
    # (the oracle's own log-sum-exp adds in fp32 one term after another: float64 is the measure)
    val = z if dtype == "f32" else (z.astype(np.uint32) << 16).view(np.float32)
    for b in np.nonzero(ref["status"] == 0)[0]:
        x = val[b].astype(np.float64) / float(np.float32(1.3))
        truth = x.max() + np.log(np.exp(x - x.max()).sum())
        # 1e-5 relative on sum(exp) is 1e-5 absolute on its logarithm
        assert abs(got["lse"][b] - truth) <= 1e-5 + 1e-6 * abs(truth), (b, got["lse"][b], truth)


# a wait that runs out in every work decomposition leaves the right rows failed (the hook checks the statuses)
# and nothing behind: records, tickets, deferred rows
def test_expired_waits_of_every_decomposition(sampler, oracle, lib):
    from born_b200 import _lib as L
    rc = lib.born_debug_expire_wait(sampler._h, None)
    assert rc == L.ERR_DEVICE_TIMEOUT, (rc, lib.born_last_error(sampler._h))
    for B, V, G in ((2, 49152, 1), (301, 50176, 1), (100, 2048 * 8, 8)):
        z = _logits(B, B, V, "f32")
        got, ref = run_both(sampler, oracle, z, dict(temperature=1.0, top_k=16), W.uniform_f32(B, 2, B), segments=G)
        assert_parity(got, ref)
    sampler.check_error()


# a gathered record of a pass that failed fails its row; a count beyond the record reads no further than it
def test_merge_of_failed_and_overlong_records(sampler):
    import torch
    from born_b200 import _lib as L
    B, V, K, G = 5, 4096, 16, 2
    z = torch.from_numpy(_logits(77, B, V * G, "f32")).cuda()
    u = torch.from_numpy(W.uniform_f32(77, 2, B)).cuda()
    gathered = torch.stack([sampler.shard_local(z[:, g * V:(g + 1) * V], g, G, K) for g in range(G)])
    want = {k: v.clone() for k, v in sampler.shard_merge(gathered, u, V, 0, G, K).items()}
    words = gathered.view(torch.int32)
    words[1, 2, 2] = 0x7FFFFFFF
    words[0, 3, 2] = -1
    words[1, 4, 3] |= 2
    got = sampler.shard_merge(gathered, u, V, 0, G, K)
    assert (want["status"] == L.ROW_OK).all()
    for k in ("token", "status", "prob", "lse"):
        assert torch.equal(got[k][:4], want[k][:4]), k
    assert got["status"][4] == 100 + L.ERR_DEVICE_TIMEOUT and got["token"][4] == -1 and torch.isnan(got["lse"][4])
