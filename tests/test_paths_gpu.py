"""Dispatch edges of the CUDA engine against the CPU oracle: merges taken together, streams that widen, merges the
host gives, many equal counts, tables that are rebuilt, the row seam's table sizes.  Every comparison is exact."""
import time

import numpy as np
import pytest
import torch

from oracle import oracle as O
from supertoken_b200 import ops
from supertoken_b200.engine import CapacityError, Engine

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, params=["policy", "filter_always"])
def filter_mode(request, monkeypatch):
    if request.param == "filter_always":
        monkeypatch.setenv("STBPE_FILTER_DENSITY", "1e30")
    return request.param


def _engine(ids, off, base_vocab, target, slots=1 << 18):
    e = Engine(max(len(ids), 1), base_vocab=base_vocab, max_merges=max(target, 1), table_slots=slots)
    e.append_ids(ids, off)
    e.count_initial()
    return e


def _check(e, ids, off, base_vocab, target):
    """A finished run: merges, counts, stream and histogram as the oracle's."""
    m, cnt, _ = e.merges()
    om, oc, _ = O.train_flat(ids, off, base_vocab, target, 1)
    assert m == om and cnt.tolist() == oc
    ids2, off2 = ids.copy(), off.copy()
    for i, (a, b) in enumerate(om):
        O.apply_merge_flat(ids2, off2, a, b, base_vocab + i)
    gi, _ = e.export_stream()
    assert np.array_equal(gi, ids2[:off2[-1]])
    _check_histogram(e, ids2[:off2[-1]].copy(), off2)


def _check_histogram(e, ids, off):
    k, c = e.export_histogram()
    ok, oc = O.count_pairs_flat(ids, off, 1)
    assert np.array_equal(k.cpu().numpy().astype(np.uint64), ok) and np.array_equal(c.cpu().numpy(), oc)


def _rows(ids, rng, mean):
    cuts = np.unique(rng.randint(1, len(ids), max(len(ids) // mean, 1)))
    return np.concatenate([[0], cuts, [len(ids)]]).astype(np.int64)


@pytest.mark.parametrize("seed", range(6))
def test_merges_that_share_a_token_or_touch(seed):
    # words over few tokens: pairs with a common first or second token, chains, runs, matches side by side on tile seams
    rng = np.random.RandomState(seed)
    words = [[1, 2], [1, 3], [4, 2], [5, 6], [6, 7], [8, 8, 8], [2, 1], [9]]
    ids = np.array([t for w in rng.choice(len(words), 9000, p=rng.dirichlet(np.ones(len(words)))) for t in words[w]], dtype=np.int32)
    off = _rows(ids, rng, 700 if seed % 2 else 40)
    e = _engine(ids, off, 16, 60)
    e.train(60)
    _check(e, ids, off, 16, 60)
    e.close()


@pytest.mark.parametrize("top", [32764, 65534])
def test_stream_widens_while_training_and_while_appending(top):
    # new ids pass the largest of a 16-bit stream in mid-run; ids of a later piece do so at once; exports beyond 65 535
    rng = np.random.RandomState(top)
    ids = rng.choice([1, 2, 3, 4], 6000).astype(np.int32)
    off = _rows(ids, rng, 300)
    e = _engine(ids, off, top, 12)
    e.train(12)
    _check(e, ids, off, top, 12)
    e.close()
    more = np.concatenate([ids, rng.choice([5, top, top + 1], 3000).astype(np.int32)])
    off2 = np.concatenate([off, [len(more)]]).astype(np.int64)
    e = Engine(len(more), base_vocab=top + 2, max_merges=12, table_slots=1 << 18)
    e.append_ids(ids, off)
    e.append_ids(more[len(ids):].copy())
    e.count_initial()
    e.train(12)
    _check(e, more, off2, top + 2, 12)
    e.close()


@pytest.mark.parametrize("base_vocab,largest,tiles", [(505, 504, 8193), (511, 510, 8192), (509, 510, 8192), (505, 511, 8192), (505, 504, 8191)])
def test_new_ids_pass_nine_bits(base_vocab, largest, tiles, filter_mode):
    # long streams without the pair filter look at nine bits of an id while all lie below 511: the new ids reach that in
    # mid-run, at once, or an id of the stream is there already
    if filter_mode == "filter_always":
        pytest.skip("streams without the filter")
    rng = np.random.RandomState(base_vocab + largest + tiles)
    n = tiles * 1024 - 100
    ids = rng.choice(np.array([1, 2, 3, 255, 256, largest], dtype=np.int32), n, p=[0.3, 0.25, 0.2, 0.15, 0.06, 0.04])
    off = _rows(ids, rng, 4000)
    e = _engine(ids, off, base_vocab, 12)
    e.train(12)
    _check(e, ids, off, base_vocab, 12)
    e.close()


@pytest.mark.parametrize("base_vocab,largest", [(2041, 2040), (2047, 2046), (2045, 2046), (2041, 2047), (8185, 8184), (8191, 8190), (8185, 8191),
                                                (2041, 8190)])
def test_new_ids_pass_eleven_and_thirteen_bits(base_vocab, largest):
    # with and without the filter: the new ids need another bit in mid-run or at once, or an id of the stream is above them
    rng = np.random.RandomState(base_vocab + largest)
    ids = rng.choice(np.array([1, 2, 3, 1023, 1024, largest], dtype=np.int32), 70000, p=[0.3, 0.25, 0.2, 0.15, 0.06, 0.04])
    off = _rows(ids, rng, 700)
    e = _engine(ids, off, base_vocab, 24)
    e.train(24)
    _check(e, ids, off, base_vocab, 24)
    e.close()


@pytest.mark.parametrize("above,wide", [(1, False), (0, True), (-1000, True)])
def test_counts_that_16_bit_tokens_leave_no_room_for(above, wide, monkeypatch):
    # the limit, 2^34 in earnest, one above the largest count, at it and below it
    rng = np.random.RandomState(4)
    ids = rng.choice([1, 2, 3], 20000, p=[0.5, 0.3, 0.2]).astype(np.int32)
    off = _rows(ids, rng, 300)
    top = int(O.count_pairs_flat(ids, off, 1)[1].max())
    monkeypatch.setenv("STBPE_NARROW_COUNTS", str(top + above))
    e = _engine(ids, off, 16, 30)
    e.train(1)
    st = e.state()
    assert (st.tile_bytes_in > st.n_tiles * 1024 * 4) == wide
    e.train(29)
    _check(e, ids, off, 16, 30)
    e.close()


@pytest.mark.parametrize("n", [1, 2, 9, 40])
def test_merges_given_by_the_host(n):
    # absent pairs, a pair twice in a row, pairs of the new ids, pairs that share tokens
    rng = np.random.RandomState(n)
    ids = rng.randint(0, 12, 20000).astype(np.int32)
    off = _rows(ids, rng, 500)
    pairs = [(1, 2), (1, 3), (1, 2), (16, 4), (5, 5), (5, 6), (900, 901), (17, 18)]
    pairs = (pairs + [(int(a), int(b)) for a, b in rng.randint(0, 30, (40, 2))])[:n]
    e = _engine(ids, off, 16, n)
    e.apply_merges(pairs, 16)
    ids2, off2 = ids.copy(), off.copy()
    for i, (a, b) in enumerate(pairs):
        O.apply_merge_flat(ids2, off2, a, b, 16 + i)
    gi, _ = e.export_stream()
    assert np.array_equal(gi, ids2[:off2[-1]]) and e.merges()[0] == pairs
    _check_histogram(e, ids2[:off2[-1]].copy(), off2)
    e.close()


def _apply_checked(e, ids, off, merges, first):
    for i, (a, b) in enumerate(merges):
        O.apply_merge_flat(ids, off, a, b, first + i)
    gi, _ = e.export_stream()
    assert np.array_equal(gi, ids[:off[-1]])
    _check_histogram(e, ids[:off[-1]].copy(), off)


OVERTAKEN = [[0, 1, 2]] * 50 + [[0, 1]] * 50 + [[3, 4]] * 60 + [[5, 2]] * 40  # (0,1) -> 5 takes (5,2) past (3,4)


@pytest.mark.parametrize("as_bytes", [False, True])
@pytest.mark.parametrize("base_vocab", [5, 6])
def test_merge_that_lifts_a_pair_with_an_id_of_the_stream(as_bytes, base_vocab):
    ids, off = O.flatten_rows(OVERTAKEN)
    e = Engine(len(ids), base_vocab=base_vocab, max_merges=3)
    e.append_bytes(ids.astype(np.uint8), off) if as_bytes else e.append_ids(ids, off)
    e.count_initial()
    e.train(3)
    assert (e.merges()[0][1] == (5, 2)) == (base_vocab == 5)
    _check(e, ids, off, base_vocab, 3)
    e.close()


@pytest.mark.parametrize("seed", range(8))
def test_new_ids_that_occur_in_the_stream(seed):
    # bytes and ids at and above base_vocab: the first new ids are among them, the later ones are not
    rng = np.random.RandomState(seed)
    top = (14, 40, 200, 256, 300)[seed % 5]
    ids = rng.choice(top, 12000, p=rng.dirichlet(np.full(top, 0.3))).astype(np.int32)
    off = _rows(ids, rng, 60)
    base = int(rng.randint(3, top))
    e = Engine(len(ids), base_vocab=base, max_merges=60, table_slots=1 << 18)
    half = int(off[len(off) // 2])
    if top <= 256 and seed % 2:
        e.append_bytes(ids.astype(np.uint8), off)
    elif top <= 256 and seed % 4 == 0:  # bytes, counted, then ids
        e.append_bytes(ids[:half].astype(np.uint8), off[:len(off) // 2 + 1])
        e.count_initial()
        e.append_ids(ids[half:].copy(), off[len(off) // 2:] - half)
    else:
        e.append_ids(ids, off)
    e.count_initial()
    for n in (7, 53):
        e.train(n)
    _check(e, ids, off, base, 60)
    e.close()


def test_best_pairs_after_merges_that_the_host_numbers():
    # the host's new ids lie above, among and below those of the loop, which must not take them for unused
    ids, off = O.flatten_rows([[0, 1, 2]] * 50 + [[0, 1]] * 50 + [[3, 4]] * 60 + [[7, 8, 2]] * 40)
    e = _engine(ids, off, 4, 8)
    e.apply_merge(7, 8, 5)  # the stream's (5,2) has 40, as in OVERTAKEN
    ids2, off2 = ids.copy(), off.copy()
    O.apply_merge_flat(ids2, off2, 7, 8, 5)
    om, oc, _ = O.train_flat(ids2[:off2[-1]].copy(), off2, 5, 7, 1)  # merge 1 of the log gets id 5
    e.train(7)
    got, counts, _ = e.merges()
    assert got[1:] == om and counts.tolist()[1:] == oc and (5, 2) in om[:2]
    _apply_checked(e, ids2, off2, om, 5)
    e.close()


@pytest.mark.parametrize("new_id", [8, 20])
def test_tie_with_a_pair_that_was_lifted_again(new_id):
    # (5,2) falls to nothing and comes back, so the candidate list, which holds every pair here, names it twice and far
    # apart; (10,11) has as many
    ids, off = O.flatten_rows([[5, 2]] * 10 + [[7, 8, 2]] * 60 + [[10, 11]] * 60 + [[12, 13]] * 90 +
                              [[i, i + 1] for i in range(100, 1300, 2)] * 2)
    e = _engine(ids, off, 16, 8)
    e.apply_merge(5, 2, 9)
    e.apply_merge(7, 8, 5)
    assert e.next_tied(None, new_id, 5) == (1, 60, [5 << 32 | 2, 10 << 32 | 11])  # (12,13) is alone with its count
    e.close()


@pytest.mark.parametrize("seed", range(6))
def test_untied_runs_with_ids_of_the_stream(seed):
    # pairs that are lifted again and again by merges into ids that were there before, then runs with unused ids
    rng = np.random.RandomState(seed)
    ids = rng.choice(10, 6000, p=rng.dirichlet(np.ones(10))).astype(np.int32)
    off = _rows(ids, rng, 50)
    e = _engine(ids, off, 6, 60)
    ids2, off2 = ids.copy(), off.copy()
    made, drawn, new = [], None, 6
    for _ in range(6):
        a, b = (int(x) for x in rng.randint(0, 10, 2))
        e.apply_merge(a, b, 3)
        O.apply_merge_flat(ids2, off2, a, b, 3)
        made.append((a, b))
    for most in (0, 2, 9, 9, 9):
        done, count, tied = e.next_tied(drawn, new, most)
        for j in range(done):
            k, c = O.count_pairs_flat(ids2[:off2[-1]].copy(), off2, 1)
            best = np.sort(k[c == c.max()])
            pair = drawn if drawn is not None and j == 0 else (int(best[0]) >> 32, int(best[0]) & 0xFFFFFFFF)
            assert (drawn is not None and j == 0) or len(best) == 1
            O.apply_merge_flat(ids2, off2, *pair, new + j)
            made.append(pair)
        k, c = O.count_pairs_flat(ids2[:off2[-1]].copy(), off2, 1)
        assert count == c.max() and tied == np.sort(k[c == c.max()]).tolist()
        drawn = (tied[-1] >> 32, tied[-1] & 0xFFFFFFFF)
        new = new + done if most < 9 else 20 + len(made)
    assert e.merges()[0] == made
    _apply_checked(e, ids2, off2, [], 0)
    e.close()


def test_timed_merges_are_the_merges_of_train():
    rng = np.random.RandomState(7)
    ids = rng.choice(12, 150000, p=rng.dirichlet(np.ones(12))).astype(np.int32)
    off = _rows(ids, rng, 500)
    e = _engine(ids, off, 12, 40)
    choose, merge, none, repack = e.train_timed(25)
    assert choose > 0 and merge > 0 and none == 0 and repack >= 0
    e.train(15)
    _check(e, ids, off, 12, 40)
    e.close()


def test_matches_reported_for_each_host_given_merge():
    # whatever ran before: the matches of this merge alone
    rng = np.random.RandomState(2)
    ids = rng.randint(0, 9, 30000).astype(np.int32)
    off = _rows(ids, rng, 400)
    e = _engine(ids, off, 16, 30)
    ids2, off2 = ids.copy(), off.copy()
    for n in (0, 3, 1, 0, 6):
        e.train(n)
        for i, (a, b) in enumerate(e.merges()[0][len(e.merges()[0]) - n:] if n else []):
            O.apply_merge_flat(ids2, off2, a, b, e.state().merges_done + 16 - n + i)
        a, b = (int(x) for x in rng.randint(0, 9, 2))
        live = int(off2[-1])
        O.apply_merge_flat(ids2, off2, a, b, 16 + e.state().merges_done)
        assert e.apply_merge(a, b, 16 + e.state().merges_done) == live - int(off2[-1])
    e.close()


@pytest.mark.parametrize("most", [0, 3, 50])
def test_ties_are_left_to_the_host(most):
    rng = np.random.RandomState(5)
    ids = rng.randint(0, 40, 4000).astype(np.int32)
    off = _rows(ids, rng, 200)
    e = _engine(ids, off, 64, 60)
    ids2, off2 = ids.copy(), off.copy()
    made, drawn, draws = [], None, 0
    while len(made) < 50:
        room = min(most, 50 - len(made) - (drawn is not None))
        done, count, tied = e.next_tied(drawn, 64 + len(made), room)
        assert done <= (drawn is not None) + room
        for j in range(done):
            k, c = O.count_pairs_flat(ids2[:off2[-1]].copy(), off2, 1)
            best = np.sort(k[c == c.max()])
            pair = drawn if drawn is not None and j == 0 else (int(best[0]) >> 32, int(best[0]) & 0xFFFFFFFF)
            assert (drawn is not None and j == 0) or len(best) == 1
            O.apply_merge_flat(ids2, off2, *pair, 64 + len(made))
            made.append(pair)
        k, c = O.count_pairs_flat(ids2[:off2[-1]].copy(), off2, 1)
        assert count == c.max() and tied == np.sort(k[c == c.max()]).tolist()
        drawn = (tied[-1] >> 32, tied[-1] & 0xFFFFFFFF)
        draws += 1
    assert e.merges()[0] == made and (most == 0 or draws < 50)
    e.close()


@pytest.mark.parametrize("n", [300, 1025, 5000, 20000])
def test_more_equal_counts_than_candidates(n):
    # n pairs of count 2: the threshold has to be found among the keys
    ids = np.tile(np.random.RandomState(n).permutation(n).astype(np.int32), 2)
    off = np.array([0, n, 2 * n], dtype=np.int64)
    e = _engine(ids, off, n, 20, 1 << 17)
    e.train(20)
    _check(e, ids, off, n, 20)
    e.close()


@pytest.mark.parametrize("slots,n", [(1 << 10, 3), (1 << 13, 1025), (1 << 18, 8193), (1 << 21, 400001),
                                     (1 << 28, 90001), (1 << 30, 150001)])
def test_partitioned_count_builds_tables_of_any_size(slots, n, monkeypatch):
    monkeypatch.setenv("STBPE_DENSE32_MIN_TOKENS", "1")
    rng = np.random.RandomState(n)
    ids = (rng.zipf(1.3, n) % 65536).astype(np.int32)
    off = _rows(ids, rng, 97)
    e = _engine(ids, off, 65536, 4, slots)
    _check_histogram(e, ids, off)
    e.close()


@pytest.mark.parametrize("slots,max_tokens,batches", [(1 << 18, 3 * 10**8, 2), (1 << 28, 10**9, 4)])
def test_partitioned_count_with_several_pieces_per_region(slots, max_tokens, batches, monkeypatch):
    # four pairs only, so that regions fill beyond a piece (8 192 or 16 384 words; about 0.3 of a CTA's 16 384 tokens a batch)
    monkeypatch.setenv("STBPE_DENSE32_MIN_TOKENS", "1")
    n = torch.cuda.get_device_properties(0).multi_processor_count * 16384 * batches
    ids = np.random.RandomState(batches).choice([300, 301], n, p=[0.55, 0.45]).astype(np.int32)
    off = np.arange(0, n + 1, n // 8, dtype=np.int64)
    e = Engine(max_tokens, base_vocab=512, max_merges=1, table_slots=slots)
    e.append_ids(ids, off)
    e.count_initial()
    assert e.state().count_convert_ms > 0
    _check_histogram(e, ids, off)
    e.close()


@pytest.mark.parametrize("partitioned", [False, True])
def test_full_pair_table_is_reported_at_once(partitioned, monkeypatch):
    # some 4 million distinct pairs, 65 536 slots: an add that walked the whole table each time would take half a minute
    monkeypatch.setenv("STBPE_DENSE32_MIN_TOKENS", "1" if partitioned else str(1 << 40))
    ids = np.random.RandomState(1).randint(0, 65536, 1 << 22).astype(np.int32)
    e = Engine(len(ids), base_vocab=65536, max_merges=1, table_slots=1 << 16)
    e.append_ids(ids)
    t = time.perf_counter()
    with pytest.raises(CapacityError):
        e.count_initial()
    assert time.perf_counter() - t < 10
    e.close()


@pytest.mark.parametrize("lg,vocab,slots", [(15, 65536, 1 << 20), (22, 65536, 1 << 24), (22, 256, 1 << 20), (22, 1500, 1 << 22),
                                            (26, 65536, 1 << 27)])
def test_automatic_table_of_a_stream_of_ids(lg, vocab, slots):
    # uniform ids: nearly every pair is another one, so 2^22 of them do not fit 2^22 slots, 2^26 not the 2^25 they get first
    n = 1 << lg
    ids = torch.randint(0, vocab, (n,), dtype=torch.int32, device="cuda", generator=torch.Generator("cuda").manual_seed(lg))
    e = Engine(2 * n, base_vocab=65536, max_merges=4)
    for _ in range(2):
        e.reset()
        e.append_ids(ids)
        e.count_initial()
        assert e.state().table_slots == slots
        k, c = e.export_histogram()
        ref, rc = torch.unique((ids[:-1].to(torch.int64) << 32) | ids[1:], return_counts=True)
        assert torch.equal(k, ref) and torch.equal(c, rc)
    e.train(4)  # (of the shortest stream every pair is alone: nothing to merge)
    k, c = e.export_histogram()
    e.count_initial()
    k2, c2 = e.export_histogram()
    assert torch.equal(k, k2) and torch.equal(c, c2)
    e.close()


@pytest.mark.parametrize("n,top,partitioned", [((1 << 21) - 1, 65535, False), (1 << 21, 65535, True), ((1 << 21) + 1025, 30000, True),
                                               (1 << 21, 65536, False), (1 << 21, 4094, False), (1 << 21, 4095, True),
                                               ((1 << 23) - 1, 511, False), ((1 << 23) + 3, 511, True)])
def test_streams_on_both_sides_of_the_partitioned_count(n, top, partitioned):
    # rows of one token among long ones, ids up to `top`, most of them small
    g = torch.Generator("cuda").manual_seed(n + top)
    ids = (torch.rand(n, device="cuda", generator=g) ** 4 * (top + 1)).to(torch.int32).clamp_(max=top)
    ids[n // 2] = top
    starts = torch.unique(torch.cat([torch.randint(1, n, (n // 900,), device="cuda", generator=g), torch.arange(1, 40, device="cuda")]))
    off = np.concatenate([[0], starts.cpu().numpy(), [n]]).astype(np.int64)
    e = Engine(n + 77, base_vocab=65536, max_merges=1)
    e.append_ids(ids, off)
    e.count_initial()
    assert (e.state().count_convert_ms > 0) == partitioned
    keep = torch.ones(n - 1, dtype=torch.bool, device="cuda")
    keep[starts - 1] = False  # a pair does not reach into the next row
    ref, rc = torch.unique(((ids[:-1].to(torch.int64) << 32) | ids[1:])[keep], return_counts=True)
    k, c = e.export_histogram()
    assert torch.equal(k, ref) and torch.equal(c, rc)
    e.close()


def test_pair_table_grows_in_mid_run():
    # random bytes: every merge makes some hundred pairs that were not there before
    n = 16 << 20
    data = torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    e = Engine(n, max_merges=1000)
    e.append_bytes(data, np.arange(0, n + 1, n // 64))
    e.count_initial()
    slots = e.state().table_slots
    e.train(1000)
    assert e.state().table_slots > slots
    k, n = e.export_histogram()
    e.count_initial()  # recount of the rewritten stream
    k2, n2 = e.export_histogram()
    assert torch.equal(k, k2) and torch.equal(n, n2)
    e.close()


@pytest.mark.parametrize("rows,width,alphabet", [(1, 2, 4), (64, 1024, 1), (64, 1024, 300), (65, 1009, 2), (65, 1008, 70000), (64, 4095, 128), (64, 4096, 128), (64, 4096, 129), (16, 16385, 70000),
                                                 (40, 4000, 70000)])
def test_seam_count_at_its_table_and_rank_limits(rows, width, alphabet):
    # both shared-memory tables (from 2^18 cells on the large one), up to and beyond 16 384 pairs, and a repeated count
    g = np.random.RandomState(rows * width)
    t = g.randint(0, alphabet, (rows, width)).astype(np.int32)
    v = (np.arange(width)[None, :] < g.randint(width // 2, width + 1, (rows, 1))).astype(np.uint8)
    cap = rows * width
    keys = torch.empty((cap, 2), dtype=torch.int32, device="cuda")
    counts = torch.empty(cap, dtype=torch.int64, device="cuda")
    length = torch.empty(1, dtype=torch.int64, device="cuda")
    ops.count_pairs(torch.from_numpy(t).cuda(), torch.from_numpy(v).cuda(), keys, counts, length)
    ok, oc = O.count_pairs_rows(t, v)
    n = int(length.item())
    got = (keys[:n, 0].to(torch.int64) << 32) | keys[:n, 1].to(torch.int64)
    assert np.array_equal(got.cpu().numpy().astype(np.uint64), ok) and np.array_equal(counts[:n].cpu().numpy(), oc)
    best = ops.select_best_pair(ops.PairHistogramResult(got.contiguous(), counts[:n]))
    assert tuple(best[:2]) == O.select_best(ok, oc)


@pytest.mark.parametrize("per", [1, 2, 16, 17, 32, 33, 340])
def test_tiles_by_their_number_of_matches(per):
    # few matches per tile go through the lanes one side at a time, more than sixteen with both sides; at a tile's ends the
    # neighbours come out of the next tile's record
    rng = np.random.RandomState(per)
    tiles = 70
    ids = rng.randint(10, 200, tiles * 1024).astype(np.int32)
    for t in range(tiles):
        at = rng.choice(341, per, replace=False) * 3
        if t % 3 == 0:
            at[0] = 1022  # ends with the tile ...
        if t % 3 == 1:
            at[0] = 1023  # ... or goes over its end
        for p in t * 1024 + at:
            ids[p:p + 2] = (1, 2)[:len(ids) - p]
    off = _rows(ids, rng, 3000)
    e = _engine(ids, off, 256, 40)
    e.train(40)
    _check(e, ids, off, 256, 40)
    e.close()


@pytest.mark.parametrize("kind", ["bytes", "constant", "byte_rows_then_ids", "ids_then_byte_rows", "mixed_ids", "negative_and_large"])
@pytest.mark.parametrize("rows,width,shift", [(512, 513, 0), (300, 1777, 1), (148 * 17, 4099, 0)])
def test_seam_count_of_byte_pairs_and_others(kind, rows, width, shift, filter_mode):
    # every CTA decides by its first cells how it counts; a pair counted both ways is one entry; the 16-bit counters are
    # emptied in time (a constant batch of more than 15 turns)
    if filter_mode == "filter_always":
        pytest.skip("no stream")
    g = np.random.RandomState(rows + width)
    t = g.randint(0, 256, (rows, width)).astype(np.int32)
    if kind == "constant":
        t[:] = 255
    elif kind == "byte_rows_then_ids":
        t[rows // 2:] += g.randint(0, 300, (rows - rows // 2, width)).astype(np.int32)
    elif kind == "ids_then_byte_rows":
        t[:rows // 2] = t[:rows // 2] % 40 + 240
    elif kind == "mixed_ids":
        t = g.randint(200, 312, (rows, width)).astype(np.int32)
    elif kind == "negative_and_large":
        t = np.where(g.rand(rows, width) < 0.1, g.choice([-2, -2**31, 2**31 - 1, 65536], (rows, width)), t % 8).astype(np.int32)
    v = (g.rand(rows, width) < 0.97).astype(np.uint8)
    flat_t, flat_v = torch.zeros(rows * width + 4, dtype=torch.int32, device="cuda"), torch.zeros(rows * width + 4, dtype=torch.uint8, device="cuda")
    flat_t[shift:shift + rows * width] = torch.from_numpy(t.ravel()).cuda()
    flat_v[shift:shift + rows * width] = torch.from_numpy(v.ravel()).cuda()
    dt, dv = flat_t[shift:shift + rows * width].view(rows, width), flat_v[shift:shift + rows * width].view(rows, width)
    cap = 1 << 20
    keys, counts = torch.empty((cap, 2), dtype=torch.int32, device="cuda"), torch.empty(cap, dtype=torch.int64, device="cuda")
    length = torch.empty(1, dtype=torch.int64, device="cuda")
    ops.count_pairs(dt, dv, keys, counts, length)
    a, b = t[:, :-1].astype(np.int64) & 0xFFFFFFFF, t[:, 1:].astype(np.int64) & 0xFFFFFFFF
    both = (v[:, :-1] & v[:, 1:]).astype(bool)
    ok, oc = np.unique((a.astype(np.uint64)[both] << np.uint64(32)) | b.astype(np.uint64)[both], return_counts=True)
    n = int(length.item())
    got = (keys[:n, 0].to(torch.int64) << 32) | (keys[:n, 1].to(torch.int64) & 0xFFFFFFFF)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), ok) and np.array_equal(counts[:n].cpu().numpy(), oc)
    assert bool((keys[n:] == -1).all()) and not bool(counts[n:].any())


def _drawn_run(ids, off, base_vocab, target, seed, device, start=None, slots=1 << 18):
    """Merges of a loop that breaks ties by random.Random(seed), drawn on the host or on the device, and the generator's state."""
    import random
    rng, merge, done = random.Random(seed), start, 0
    e = _engine(ids, off, base_vocab, target, slots)
    trips = 0
    while done < target:
        n, count, cands = e.next_tied(merge, base_vocab + done, target - done - (merge is not None), rng if device else None)
        done, merge, trips = done + n, None, trips + 1
        if done >= target or not cands or count < 2:
            break
        key = cands[rng.randrange(len(cands))] if len(cands) > 1 else cands[0]
        merge = (key >> 32, key & 0xFFFFFFFF)
        if done == target - 1:
            e.apply_merge(*merge, base_vocab + done)
            done += 1
    m, c, live = e.merges()
    stream = e.export_stream()[0]
    e.close()
    return m, c.tolist(), live.tolist(), stream.tolist(), rng.getstate(), trips


@pytest.mark.parametrize("seed,n,alphabet,target", [(0, 3000, 6, 90), (1, 3000, 40, 150), (2, 40000, 300, 120), (3, 200, 200, 30), (4, 9000, 1000, 60),
                                                    (5, 70000, 12, 200), (6, 2500, 3, 400)])
def test_ties_drawn_on_the_device_as_on_the_host(seed, n, alphabet, target):
    # few and many tied pairs, counts that fall to the threshold and below 2; the device breaks every tie, in one call
    rng = np.random.RandomState(seed)
    ids = rng.randint(0, alphabet, n).astype(np.int32)
    off = _rows(ids, rng, 90)
    host, dev = (_drawn_run(ids, off, 1000, target, seed, d) for d in (False, True))
    assert host[:5] == dev[:5]
    assert dev[5] == 1 < host[5]


@pytest.mark.parametrize("few", [None, 1, 3])
@pytest.mark.parametrize("base_vocab", [508, 2040, 32760])
def test_ties_drawn_while_the_ids_pass_a_number_of_bits(base_vocab, few, monkeypatch):
    # The device looks at all bits of an id while it holds outputs of the generator, and may look at fewer once they have run
    # out (few: as many per call).  From 32 767 on the tokens are 32 bits wide and the host breaks the ties.
    rng = np.random.RandomState(base_vocab)
    ids = rng.choice([1, 2, 3, 4, 5], 30000).astype(np.int32)
    off = _rows(ids, rng, 60)
    if few is not None:
        init = Engine.__init__

        class Few:
            def __init__(self, lib):
                self.lib = lib

            def __getattr__(self, name):
                return getattr(self.lib, name)

            def stbpe_next_drawn(self, h, a, b, new_id, most, words, n, *rest):
                return self.lib.stbpe_next_drawn(h, a, b, new_id, most, words, min(n, few), *rest)

        def with_few(self, *args, **kwargs):
            init(self, *args, **kwargs)
            self._lib = Few(self._lib)

        monkeypatch.setattr(Engine, "__init__", with_few)
    host, dev = (_drawn_run(ids, off, base_vocab, 40, 7, d, start=(1, 2)) for d in (False, True))
    assert host[:5] == dev[:5]
    if few is None and base_vocab < 32760:
        assert dev[5] == 1 < host[5]


def _crowded(pairs, tiles_per_cta, seed):
    """Matches of the pairs (0, 1), (2, 3), ... in turn, each behind a token out of 30 000: every CTA meets more distinct
    neighbours than its histogram has entries, so some go to the pair table while tiles are still being worked on."""
    rng = np.random.RandomState(seed)
    ctas = torch.cuda.get_device_properties(0).multi_processor_count
    ids = rng.randint(16, 30000, tiles_per_cta * ctas * 1024).astype(np.int32)
    n = len(ids) // 3 // pairs * pairs
    k = rng.permutation(np.arange(n) % pairs)
    ids[1:3 * n:3], ids[2:3 * n:3] = 2 * k, 2 * k + 1
    keys = set()
    for t in ids.reshape(-1, 1024)[::ctas]:  # the tiles of CTA 0
        at = np.flatnonzero((t[:-1] < 16) & (t[:-1] % 2 == 0) & (t[1:] == t[:-1] + 1))
        at = at[(at > 0) & (at < 1022)]
        keys |= {(x, k, 0) for x, k in zip(t[at - 1].tolist(), t[at].tolist())} | {(y, k, 1) for y, k in zip(t[at + 2].tolist(), t[at].tolist())}
    return ids, keys


def test_more_neighbours_than_the_histogram_of_a_cta_has_entries():
    ids, keys = _crowded(8, 9, 1)
    assert len(keys) > 4096  # in one step, as all eight pairs go together
    off = np.array([0, len(ids)], dtype=np.int64)
    e = _engine(ids, off, 30000, 24, 1 << 23)
    e.train(24)
    _check(e, ids, off, 30000, 24)
    e.close()


def test_more_neighbours_than_entries_while_ties_are_drawn():
    ids, keys = _crowded(2, 14, 2)
    assert min(sum(k == p for _, k, _ in keys) for p in (0, 2)) > 4096  # for the one pair that is drawn
    off = np.array([0, len(ids)], dtype=np.int64)
    host, dev = (_drawn_run(ids, off, 30000, 6, 3, d, slots=1 << 23) for d in (False, True))
    assert host[:5] == dev[:5]
    assert dev[5] < host[5]  # the tie was broken on the device


@pytest.mark.parametrize("density,timed", [("0", False), ("0", True), ("1e30", False)])
def test_tiles_that_the_last_step_visited(density, timed, monkeypatch):
    # below zero: every tile; with the pair filter their number, here those of one pair in one tile
    monkeypatch.setenv("STBPE_FILTER_DENSITY", density)
    ids = np.random.RandomState(0).randint(10, 10000, 64 * 1024).astype(np.int32)
    ids[5 * 1024 + 100:5 * 1024 + 300] = np.tile([1, 2], 100)
    e = _engine(ids, np.array([0, len(ids)], dtype=np.int64), 10000, 1)
    (e.train_timed if timed else e.train)(1)
    assert e.merges()[0] == [(1, 2)]
    visited = e.state().work_tiles
    assert visited < 0 if density == "0" else 1 <= visited < 64
    e.close()


@pytest.mark.parametrize("n", [60, 130, 256])
def test_seam_count_of_pairs_that_start_at_one_slot(n):
    # rows of one pair each, whose keys all begin their search at the same slot of the table (1024 slots for up to 512 pairs)
    g = np.random.RandomState(n)
    ab = g.randint(0, 1 << 30, (600000, 2)).astype(np.int32)
    h = (ab[:, 0].astype(np.uint64) << np.uint64(32)) | ab[:, 1].astype(np.uint64)
    for mul in (0xff51afd7ed558ccd, 0xc4ceb9fe1a85ec53, 1):
        h = (h ^ (h >> np.uint64(33))) * np.uint64(mul)
    t = torch.from_numpy(np.ascontiguousarray(ab[(h & np.uint64(1023)) == 1000][:n])).cuda()
    assert t.shape[0] == n
    keys, counts = torch.empty((n, 2), dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.int64, device="cuda")
    length = torch.empty(1, dtype=torch.int64, device="cuda")
    ops.count_pairs(t, torch.ones_like(t, dtype=torch.uint8), keys, counts, length)
    assert int(length) == n and sorted(map(tuple, keys.tolist())) == sorted(map(tuple, t.tolist())) and bool((counts == 1).all())


@pytest.mark.parametrize("base_vocab,tied,calls", [(40000, 50, 0), (10000, 1100, 4), (10000, 50, 2)])
def test_outputs_are_taken_ahead_only_where_the_device_may_draw(base_vocab, tied, calls):
    # 32-bit tokens, and more tied pairs than the device keeps: rows of one pair each, all pairs twice
    import random

    class Counted(random.Random):
        ahead = 0

        def getrandbits(self, k):
            self.ahead += k > 32
            return super().getrandbits(k)

    pairs = np.stack([np.arange(tied), np.arange(tied) + tied], 1).astype(np.int32)
    ids = np.concatenate([pairs, pairs]).ravel()
    e = _engine(ids, np.arange(0, len(ids) + 1, 2).astype(np.int64), base_vocab, 20)
    rng, merge, left, want, plain = Counted(3), None, list(map(tuple, pairs.tolist())), [], random.Random(3)
    if tied <= 1024 and base_vocab < 32767:  # the device breaks them all: the outputs are taken ahead once, and once for good
        assert e.next_tied(None, base_vocab, 20, rng)[0] == 20 and rng.ahead == calls
        e.close()
        return
    for done in range(20):  # (after 1, 3, 7 and 15 calls the device is asked again)
        want.append(left.pop(plain.randrange(len(left))))
        _, count, cands = e.next_tied(merge, base_vocab + max(done - 1, 0), 20 - done, rng)
        assert count == 2 and len(cands) == len(left) + 1
        key = cands[rng.randrange(len(cands))]
        merge = (key >> 32, key & 0xFFFFFFFF)
        assert merge == want[-1]
    assert rng.ahead == calls
    e.close()


def _loop_launches(run):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    return sum("loop_kernel" in ev.name for ev in prof.events())


@pytest.mark.parametrize("base_vocab,tiles", [(2047, 40), (2040, 40), (8191, 40), (505, 8192), (2047, 8192)])
def test_no_launch_that_leaves_for_the_bits_of_its_first_ids(base_vocab, tiles, filter_mode, monkeypatch):
    if filter_mode == "policy":
        monkeypatch.setenv("STBPE_FILTER_DENSITY", "0")
    rng = np.random.RandomState(base_vocab)
    data = rng.randint(0, 200, tiles * 1024, dtype=np.uint8)
    e = Engine(len(data), base_vocab=base_vocab, max_merges=20)
    e.append_bytes(data, np.array([0, len(data)], dtype=np.int64))
    e.count_initial()
    # (with the filter, the first launch returns for the host to build it)
    assert _loop_launches(lambda: e.train(20)) == (1 if filter_mode == "policy" else 2)
    assert len(e.merges()[0]) == 20
    e.close()


@pytest.mark.parametrize("base_vocab,target", [(441, 90), (1917, 150), (7676, 530)])
def test_long_streams_pass_nine_eleven_and_thirteen_bits_in_mid_run(base_vocab, target, filter_mode, monkeypatch):
    # enough merges before the bound to look at fewer bits up to it: 64 below 511, 128 below 2 047, 512 below 8 191
    if filter_mode == "policy":
        if target == 530:
            pytest.skip("thirteen bits only with the filter")
        monkeypatch.setenv("STBPE_FILTER_DENSITY", "0")
    rng = np.random.RandomState(target)
    ids = rng.randint(0, 200, 8192 * 1024 - 100).astype(np.int32)
    off = _rows(ids, rng, 4000)
    e = _engine(ids, off, base_vocab, target, 1 << 20)
    e.train(target)
    _check(e, ids, off, base_vocab, target)
    e.close()
